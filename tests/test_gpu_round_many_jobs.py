"""More jobs in a round than a warp has lanes: the round plan's threads and
the proposals' job lookup past job 32 give each job what it gets alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [1, 2])
def test_forty_jobs_alone_equals_mix(pcs, ctx, order):
    import part_conc_spt_abc_gb300.workloads as W
    inputs = []
    for j in range(40):
        inp, _ = W.make_problem(ctx, [150.0 + 10 * j], [10.0], 5e13, [1.0], 2 + j % 3, 10 + j, 32 + j % 7, 8 + j % 5,
                                1 + j % 2, seed=j)
        inp.params.avg_trial_count = 50
        inputs.append(inp)

    def out(sim):
        o, i = sim.output(), sim.info()
        return [o.m, o.s, o.c, o.dist, o.w, i.gamma, i.trials, i.accepted, i.iterations, i.converged]

    alone = {}
    for j in (0, 7, 31, 32, 33, 39):
        sim = pcs.make_simulation(ctx, inputs[j], 100 + j)
        sim.run()
        alone[j] = out(sim)
        sim.close()
    ctx.set_tuning(job_order=order, round_capacity=333)  # the jobs compete for the round
    try:
        srv = pcs.Server(ctx)
        sims = [pcs.make_simulation(ctx, inp, 100 + j) for j, inp in enumerate(inputs)]
        for sim in sims:
            srv.submit(sim)
        while srv.step():
            pass
        for j, want in alone.items():
            for a, b in zip(out(sims[j]), want):
                assert np.array_equal(a, b), j
        for sim in sims:
            sim.close()
    finally:
        ctx.set_tuning(job_order=2, round_capacity=2048)
