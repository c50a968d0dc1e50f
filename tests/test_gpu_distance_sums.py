"""The strip kernel's double and exact integer sums at the edge of its integer
form: cumulative counts just below, at and just above 2^22, the largest
differences there are (an observed histogram of zeros, or a simulated one), on
the tallest strips, odd and even column counts, with the prefix sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,B", [(1664, 34), (1664, 33), (33, 1), (201, 65)])
@pytest.mark.parametrize("total", [2**22 - 1, 2**22, 2**22 + 1])
@pytest.mark.parametrize("observed", [False, True])
def test_sums_at_the_integer_edge(pcs, ctx, oracle, R, B, total, observed):
    h = np.zeros((R, B), np.uint32)
    h[0, 0] = 3 if observed else total - 2
    h[R - 1, B - 1] += 2  # the last cell holds the largest cumulative count
    ref = np.full((R, B), total if observed else 0, np.uint32)
    r = pcs.scan_distance(ctx, h, ref, want_cum=True, want_f64=True, want_ssd=True)
    d32, _, ssd = oracle.distance_kdist(h, ref)
    assert r["ssd"][0] == ssd
    assert r["dist_f64"][0] == oracle.distance_kdist_f64(h, ref)
    assert r["dist_f32"][0].tobytes() == np.float32(d32).tobytes()
    assert np.array_equal(r["cum"][0], np.cumsum(np.cumsum(h, 0, dtype=np.uint64), 1).astype(np.uint32))
