"""Jobs with double distances (accel -dt d) beside and after jobs without, on one
context and of one shape: every job's result is the one that it has on a
context of its own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _input(ctx, j, double):
    import part_conc_spt_abc_gb300.workloads as W
    inp, _ = W.make_problem(ctx, [150.0 + 30 * j], [10.0], 3e14, [1.0], 6, 60, 300, 48, 2, seed=j)
    inp.params.avg_trial_count = 50
    inp.params.distance_double = double
    return inp


def _out(sim):
    o, i = sim.output(), sim.info()
    return [o.m, o.s, o.c, o.dist, o.w, i.gamma, i.trials, i.accepted, i.iterations, i.converged]


def _alone(pcs, inp, seed):
    with pcs.Context(0) as c:
        sim = pcs.make_simulation(c, inp, seed)
        sim.run()
        r = _out(sim)
        sim.close()
    return r


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


def test_one_after_another(pcs, ctx):
    inputs = [_input(ctx, j, double) for j, double in enumerate([0, 1, 0, 1])]
    want = [_alone(pcs, inp, 50 + j) for j, inp in enumerate(inputs)]
    other = _input(ctx, 1, 0)
    assert not _same(_alone(pcs, other, 51), want[1])  # the two distances are told apart
    with pcs.Context(0) as c:
        for j, inp in enumerate(inputs):
            sim = pcs.make_simulation(c, inp, 50 + j)
            sim.run()
            assert _same(_out(sim), want[j]), j
            sim.close()


@pytest.mark.parametrize("doubles", [[1, 0, 0], [0, 0, 1]])
def test_in_shared_rounds(pcs, ctx, doubles):
    inputs = [_input(ctx, j, double) for j, double in enumerate(doubles)]
    want = [_alone(pcs, inp, 60 + j) for j, inp in enumerate(inputs)]
    with pcs.Context(0) as c:
        srv = pcs.Server(c)
        sims = [pcs.make_simulation(c, inp, 60 + j) for j, inp in enumerate(inputs)]
        for sim in sims:
            srv.submit(sim)
        while srv.step():
            pass
        for j, sim in enumerate(sims):
            assert _same(_out(sim), want[j]), j
            sim.close()
