"""Clusters of CTAs with every output (double and exact integer sums, prefix
sums): two to eight strips, lone last columns, more histograms than clusters
fit at once, strips that are past the integer form while others are not,
heights with two tiles, one tile and none."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,B,count", [(33, 33, 2), (97, 64, 3), (301, 128, 37), (997, 255, 19), (1001, 256, 40), (1400, 96, 2),
                                       (1, 40, 3), (1600, 250, 1)])
@pytest.mark.parametrize("f64,ssd,cum", [(True, True, True), (True, False, False), (False, True, True), (False, False, True)])
@pytest.mark.parametrize("big", [0, 2**22 - 1, 2**22, 2**31])
def test_cluster_sums(pcs, ctx, oracle, R, B, count, f64, ssd, cum, big):
    rng = np.random.default_rng(R + B)
    hist = rng.poisson(0.6, (count, R, B)).astype(np.uint32)
    ref = np.cumsum(np.cumsum(rng.poisson(0.6, (R, B)), 0), 1).astype(np.uint32)
    if big:  # one histogram: small to the left of the last strip, large from there on
        hist[count - 1] = 0
        hist[count - 1, R // 2, 32 * ((B - 1) // 32)] = big
    r = pcs.scan_distance(ctx, hist, ref, want_f64=f64, want_ssd=ssd, want_cum=cum)
    for q in sorted({0, count // 2, count - 1}):
        d32, want_cum, want_ssd = oracle.distance_kdist(hist[q], ref)
        assert r["dist_f32"][q].tobytes() == np.float32(d32).tobytes(), q
        if cum:
            assert np.array_equal(r["cum"][q], want_cum), q
        if ssd:
            assert r["ssd"][q] == want_ssd, q
        if f64:
            assert r["dist_f64"][q] == oracle.distance_kdist_f64(hist[q], ref), q
