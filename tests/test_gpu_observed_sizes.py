"""Observed cumulative histograms at the edges of the row and column passes:
a warp's 32 and 256 cells, a CTA's 8 columns and 128 shares of the rows, and
shapes below all of them; both conventions, and through a job's distances the
column-major copy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,B", [(1, 1), (2, 7), (7, 9), (8, 8), (9, 31), (127, 32), (128, 33), (129, 255), (257, 256),
                                 (40, 257), (2001, 3), (3, 2001), (1001, 513)])
def test_observed_sat_sizes(pcs, ctx, oracle, R, B):
    rng = np.random.default_rng(R * 4096 + B)
    n = 5000
    K = rng.integers(0, R, n)
    DE = rng.uniform(0.0, 6.0, n)  # a sixth of the tracks above the range
    np.testing.assert_array_equal(pcs.observed_sat(ctx, K, DE, R, B, 5.0), oracle.observed_sat(K, DE, R, B, 5.0))
    K = rng.integers(1, R + 1, n)
    np.testing.assert_array_equal(pcs.observed_sat(ctx, K, DE, R, B, 5.0, julia=True),
                                  oracle.observed_sat_julia(K, DE, R, B, 5.0))


@pytest.mark.parametrize("frames,B", [(60, 33), (140, 64), (20, 31)])
def test_column_major_copy(pcs, ctx, oracle, frames, B):
    """A round's distances use the job's column-major copy."""
    import part_conc_spt_abc_gb300.workloads as W
    inp, _ = W.make_problem(ctx, [175.0], [10.0], 1e14, [1.0], 4, frames, B, 24, 1, seed=3)
    sim = pcs.make_simulation(ctx, inp, 7)
    srv = pcs.Server(ctx)
    srv.submit(sim)
    srv.step()
    props, theta, counts = sim.round_proposals()
    setup = W.forward_setup(inp.frames.astype(np.uint32), B)
    runs = [pcs.ForwardRun(c, p.half_az, p.pre_comp_prob, p.sd_scale, p.sd_shape, p.slot, p.trial, p.generation)
            for p, c in zip(props, counts)]
    hist = pcs.simulate_hist(ctx, setup, runs, seed=7)
    ref = oracle.observed_sat(inp.K, inp.DE, frames + 1, B, W.UB_DE)
    for p, h in zip(props, hist):
        assert np.float32(p.distance).tobytes() == np.float32(oracle.distance_kdist(h, ref)[0]).tobytes()
    while srv.step():
        pass
    sim.close()
