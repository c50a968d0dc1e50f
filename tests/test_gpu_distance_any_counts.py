"""Distances of arrays that are no cumulative histogram of a few million
tracks: an observed array that falls, so that its last cell is not its largest,
and prefix sums that wrap around 2^32.  The kernels' integer forms hold below
2^22 only; where the last cell does not tell, the sums are the oracle's all the
same -- by strips, clusters, rows and blocks of rows, with and without the
double sums, the exact sums and the prefix sums.  (Strips and clusters that are
asked for the float alone go by the last cell.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EVERY = [(True, True, True), (True, False, False), (False, True, False), (False, False, True)]
SHAPES = [(b"k_distance_strip", 40, 30, 3), (b"k_distance_strip", 52, 33, 400), (b"k_distance_cluster", 301, 70, 3),
          (b"k_distance_cluster", 900, 128, 2), (b"k_distance_rows", 65, 1024, 2), (b"k_distance_rows", 33, 513, 3),
          (b"k_distance_rows", 1700, 100, 2), (b"k_distance", 1700, 40, 2)]


def _ref(kind, R, B):
    ref = np.arange(R * B, dtype=np.uint32).reshape(R, B) % 1000
    if kind == "first cell":
        ref[0, 0] = 2**23
    elif kind == "a middle row":
        ref[R // 2, B // 2] = 3 * 2**22
    elif kind == "falling":
        ref = (2**31 - 2**31 // (R * B) * np.arange(R * B, dtype=np.uint64)).astype(np.uint32).reshape(R, B)
        ref[R - 1] = 7
    elif kind == "all but the last rows":
        ref[:max(1, R - 8)] += np.uint32(2**32 - 2000)
    return ref


def _check(pcs, ctx, oracle, kernel, hist, ref, f64, ssd, cum):
    r = pcs.scan_distance(ctx, hist, ref, want_f64=f64, want_ssd=ssd, want_cum=cum)
    assert kernel is None or pcs.lib().pcs_debug_last_kernel(1) == kernel
    for q in sorted({0, len(hist) // 2, len(hist) - 1}):
        d32, want_cum, want_ssd = oracle.distance_kdist(hist[q], ref)
        assert r["dist_f32"][q].tobytes() == np.float32(d32).tobytes(), q
        if cum:
            assert np.array_equal(r["cum"][q], want_cum), q
        if ssd:
            assert r["ssd"][q] == want_ssd, q
        if f64:
            assert r["dist_f64"][q] == oracle.distance_kdist_f64(hist[q], ref), q


@pytest.mark.parametrize("kernel,R,B,count", SHAPES)
@pytest.mark.parametrize("f64,ssd,cum", EVERY)
@pytest.mark.parametrize("kind", ["first cell", "a middle row", "falling", "all but the last rows"])
def test_observed_arrays_that_fall(pcs, ctx, oracle, kernel, R, B, count, f64, ssd, cum, kind):
    hist = np.random.default_rng(R).poisson(0.6, (count, R, B)).astype(np.uint32)
    kernel = None if f64 and kernel == b"k_distance_rows" else kernel  # a leftover launch may follow
    _check(pcs, ctx, oracle, kernel, hist, _ref(kind, R, B), f64, ssd, cum)


@pytest.mark.parametrize("kernel,R,B,count", [s for s in SHAPES if s[0] in (b"k_distance_rows", b"k_distance")])
@pytest.mark.parametrize("kind", ["a middle row", "falling", "all but the last rows"])
def test_float_alone(pcs, ctx, oracle, kernel, R, B, count, kind):
    hist = np.random.default_rng(B).poisson(0.6, (count, R, B)).astype(np.uint32)
    _check(pcs, ctx, oracle, kernel, hist, _ref(kind, R, B), False, False, False)


@pytest.mark.parametrize("kernel,R,B,count", SHAPES)
@pytest.mark.parametrize("f64,ssd,cum", EVERY)
def test_sums_that_wrap(pcs, ctx, oracle, kernel, R, B, count, f64, ssd, cum):
    hist = np.random.default_rng(R + B).poisson(0.6, (count, R, B)).astype(np.uint32)
    hist[:, R // 3, B // 2] += np.uint32(2**31)  # large from here on,
    hist[:, R - 2, B // 3] += np.uint32(2**31)   # and past 2^32 in the last rows
    ref = np.cumsum(np.cumsum(np.random.default_rng(1).poisson(0.6, (R, B)), 0), 1).astype(np.uint32)
    _check(pcs, ctx, oracle, None, hist, ref, f64, ssd, cum)
