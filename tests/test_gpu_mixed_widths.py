"""Served jobs of different widths: the distance kernel of their shared rounds
goes by how wide most of them are, and is chosen anew when jobs end.  Every
job's result is the one that it has alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _input(ctx, j, frames, bins, generations, pop=24):
    import part_conc_spt_abc_gb300.workloads as W
    inp, _ = W.make_problem(ctx, [150.0 + 40 * j], [10.0], 5e13, [1.0], 3, frames, bins, pop, generations, seed=j)
    inp.params.avg_trial_count = 50
    return inp


def _out(sim):
    o, i = sim.output(), sim.info()
    return [o.m, o.s, o.c, o.dist, o.w, i.gamma, i.trials, i.accepted, i.iterations, i.converged]


@pytest.mark.parametrize("frames,bins,first,last", [
    (200, [1024, 64, 64, 64], b"k_distance_strip", b"k_distance_rows"),
    (200, [64, 64, 256], b"k_distance_rows", b"k_distance_rows"),
    (200, [256, 64, 64, 64], b"k_distance_strip", b"k_distance_rows"),
    (200, [320, 320, 64, 64], b"k_distance_rows", b"k_distance_rows"),
    (60, [320, 32, 32], b"k_distance_rows", b"k_distance_rows"),
    (200, [160, 128, 64], b"k_distance_strip", b"k_distance_strip"),
    (1700, [300, 33, 33, 33], b"k_distance_rows", b"k_distance_rows")])
def test_served_widths(pcs, ctx, frames, bins, first, last):
    # the widest job ends last
    inputs = [_input(ctx, j, frames if b == max(bins) else frames // 2, b, 3 if b == max(bins) else 1)
              for j, b in enumerate(bins)]
    alone = []
    for j, inp in enumerate(inputs):
        sim = pcs.make_simulation(ctx, inp, 70 + j)
        sim.run()
        alone.append(_out(sim))
        sim.close()
    with pcs.Context(0) as c:
        srv = pcs.Server(c)
        sims = [pcs.make_simulation(c, inp, 70 + j) for j, inp in enumerate(inputs)]
        for sim in sims:
            srv.submit(sim)
        srv.step()
        seen = [pcs.lib().pcs_debug_last_kernel(1)]
        while srv.step():
            seen.append(pcs.lib().pcs_debug_last_kernel(1))
        got = [_out(sim) for sim in sims]
        for sim in sims:
            sim.close()
    assert seen[0] == first and seen[-1] == last
    for a, b in zip(got, alone):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
