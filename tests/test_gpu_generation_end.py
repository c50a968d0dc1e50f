"""The end of a generation, spread over a cluster of CTAs, at population sizes
around its warps, CTA width and chunks: normalised and cumulative weights,
epsilon, the perturbation factor, the committed population and the reset slots
against numpy on the engine's own populations (read from checkpoints)."""
import numpy as np
import pytest

from test_gpu_pmc import small_input
from test_gpu_pmc_parity import parse

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pop", [9, 31, 32, 33, 255, 1023, 1024, 1025, 2057])
@pytest.mark.parametrize("cholesky,weighting,schedule", [(False, 0, 1), (True, 0, 1), (True, 1, 0), (False, 1, 0)])
def test_generation_end(pcs, ctx, pop, cholesky, weighting, schedule):
    C = 2 if cholesky else 1
    inp, _ = small_input(pcs, C=C, pop=pop, weighting=weighting, videos=2, frames=20)
    p = inp.params
    p.perturbation = pcs.PERTURB_CHOLESKY if cholesky else pcs.PERTURB_DIAGONAL
    p.schedule = pcs.SCHEDULE_QUANTILE if schedule else pcs.SCHEDULE_DELTA
    p.quantile, p.delta_gamma = 0.37, 0.01
    P = 3 * C + 1
    sim = pcs.make_simulation(ctx, inp, 23)
    for generation in range(3):
        if sim.step():
            break
        info, blob = sim.info(), sim.checkpoint()
        s = parse(blob, pop, P)
        if generation:
            assert np.array_equal(s["theta"], s["theta_new"]) and np.array_equal(s["dist"], s["dist_new"])
            if weighting:
                d = 1.0 / (s["dist"] * s["dist"])
                np.testing.assert_allclose(s["w"], d / d.sum(), rtol=1e-12)
            assert abs(s["w"].sum() - 1.0) < 1e-12
        assert np.array_equal(s["wcum"], np.cumsum(s["w"]))  # added in order
        rank = min(pop - 1, int(0.37 * pop)) if schedule else pop // 2
        eps = np.sort(s["dist_new"])[rank]
        if schedule:
            assert info.gamma == eps
        elif generation == 0:
            assert info.gamma == eps - 0.01
        free = [q for q in range(P) if q != P - 1]
        th = s["theta"][:, free]
        if not cholesky:
            np.testing.assert_allclose(np.diag(s["factor"])[free], np.sqrt(2.0 * th.var(axis=0)), rtol=1e-9, atol=1e-300)
            assert np.count_nonzero(s["factor"] - np.diag(np.diag(s["factor"]))) == 0
        elif pop > 30:
            x = th - s["w"] @ th
            want = np.linalg.cholesky(2.0 * (x * s["w"][:, None]).T @ x)
            np.testing.assert_allclose(s["factor"][np.ix_(free, free)], want, rtol=1e-7, atol=1e-9 * np.abs(want).max())
        tail = np.frombuffer(blob[len(blob) - 12 * pop:], np.uint32).reshape(3, pop)
        assert not tail[0].any() and np.array_equal(tail[1], np.arange(pop)) and not tail[2].any()
    sim.close()
