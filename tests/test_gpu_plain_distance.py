"""The distance kernel that each plain form launches: strips of one CTA in the
reference's geometry; in the persistent one, too, but the row kernel where
there are eight strips or more.  Both give the same estimation, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frames,bins,persistent", [(60, 100, b"k_distance_strip"), (700, 64, b"k_distance_strip"),
                                                    (60, 30, b"k_distance_strip"), (60, 300, b"k_distance_rows")])
def test_plain_forms(pcs, ctx, frames, bins, persistent):
    import part_conc_spt_abc_gb300.workloads as W
    inp, _ = W.make_problem(ctx, [150.0], [10.0], 5e13, [1.0], 3, frames, bins, 24, 1, seed=bins)
    inp.params.avg_trial_count = 50
    got = []
    try:
        for launch, kernel in ((1, b"k_distance_strip"), (2, persistent)):
            ctx.set_tuning(plain_launch=launch)
            sim = pcs.make_simulation(ctx, inp, 7)
            sim.run_plain(0, 5)
            assert pcs.lib().pcs_debug_last_kernel(1) == kernel
            o, i = sim.output(), sim.info()
            got.append([o.m, o.s, o.c, o.dist, o.w, i.gamma, i.trials, i.accepted])
            sim.close()
    finally:
        ctx.set_tuning(plain_launch=1)
    for a, b in zip(*got):
        assert np.array_equal(a, b)
