"""Rounds of one proposal to more than the work-item scan has threads, odd
numbers of them, few and many particles per video (both Poisson samplers),
every model: a job's result is the one of rounds of the default size."""
import numpy as np
import pytest

from test_gpu_pmc import small_input

pytestmark = pytest.mark.gpu


def _out(pcs, ctx, inp):
    sim = pcs.make_simulation(ctx, inp, 31)
    sim.run()
    o, i = sim.output(), sim.info()
    sim.close()
    return [o.m, o.s, o.c, o.dist, o.w, i.gamma, i.trials, i.accepted, i.iterations, i.converged]


@pytest.mark.parametrize("capacity,pop", [(1, 33), (2, 33), (3, 64), (33, 65), (1023, 1300), (1025, 1300), (1999, 1300)])
@pytest.mark.parametrize("conc,C,cholesky", [(2e13, 1, False), (1e15, 2, True)])
def test_round_sizes(pcs, ctx, capacity, pop, conc, C, cholesky):
    inp, _ = small_input(pcs, C=C, pop=pop, videos=33, frames=12)
    p = inp.params
    p.lb_c, p.ub_c = conc * 1e-6 * 0.5, conc * 1e-6 * 2.0
    p.perturbation = pcs.PERTURB_CHOLESKY if cholesky else pcs.PERTURB_DIAGONAL
    p.max_generations = 2
    want = _out(pcs, ctx, inp)
    try:
        ctx.set_tuning(round_capacity=capacity)
        got = _out(pcs, ctx, inp)
    finally:
        ctx.set_tuning(round_capacity=2048)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
