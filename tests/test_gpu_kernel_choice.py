"""Sizes near the lines between the distance kernels and between the forward
model's, with the kernel that they are meant for asserted: a rule that moves
fails here instead of leaving a kernel untested.  (The lines depend on the
number of SMs; these are for 152.)"""
import numpy as np
import pytest

from test_gpu_screen import CASES, VIDEOS, _both, _runs

pytestmark = pytest.mark.gpu

SUMS = [(False, False, False), (True, True, True), (True, False, False), (False, True, True)]


def _distances(pcs, ctx, oracle, kernel, R, B, count, f64, ssd, cum, big):
    rng = np.random.default_rng(R + B)
    hist = rng.poisson(0.6, (count, R, B)).astype(np.uint32)
    ref = np.cumsum(np.cumsum(rng.poisson(0.6, (R, B)), 0), 1).astype(np.uint32)
    if big:  # one histogram: small to the left of the last strip, large from there on
        hist[count - 1] = 0
        hist[count - 1, R // 2, 32 * ((B - 1) // 32)] = big
    r = pcs.scan_distance(ctx, hist, ref, want_f64=f64, want_ssd=ssd, want_cum=cum)
    assert pcs.lib().pcs_debug_last_kernel(1) == kernel
    for q in sorted({0, count // 2, count - 1}):
        d32, want_cum, want_ssd = oracle.distance_kdist(hist[q], ref)
        assert r["dist_f32"][q].tobytes() == np.float32(d32).tobytes(), q
        if cum:
            assert np.array_equal(r["cum"][q], want_cum), q
        if ssd:
            assert r["ssd"][q] == want_ssd, q
        if f64:
            assert r["dist_f64"][q] == oracle.distance_kdist_f64(hist[q], ref), q


@pytest.mark.parametrize("R,B,count", [(171, 33, 2), (200, 64, 3), (201, 40, 5), (1, 97, 3), (7, 130, 2), (31, 255, 2),
                                       (2, 225, 3), (1, 256, 2)])  # two strips; few rows
@pytest.mark.parametrize("f64,ssd,cum", SUMS)
@pytest.mark.parametrize("big", [0, 2**22 - 1, 2**22])
def test_clusters(pcs, ctx, oracle, R, B, count, f64, ssd, cum, big):
    _distances(pcs, ctx, oracle, b"k_distance_cluster", R, B, count, f64, ssd, cum, big)


@pytest.mark.parametrize("R,B,count", [(9, 4, 4000), (33, 257, 310), (1700, 129, 3), (1700, 1, 460), (1665, 3, 460),
                                       (17, 132, 920)])  # a last warp with one column, with four; lanes with one, with three
@pytest.mark.parametrize("f64,ssd,cum", SUMS)
@pytest.mark.parametrize("big", [0, 2**22])
def test_rows(pcs, ctx, oracle, R, B, count, f64, ssd, cum, big):
    _distances(pcs, ctx, oracle, b"k_distance_rows", R, B, count, f64, ssd, cum, big)


@pytest.mark.parametrize("kernel,R,B,count", [(b"k_distance_strip", 170, 33, 2), (b"k_distance_strip", 97, 64, 3),
                                              (b"k_distance_strip", 65, 129, 900), (b"k_distance_strip", 7, 1, 3800),
                                              (b"k_distance", 1665, 64, 100)])
@pytest.mark.parametrize("f64,ssd,cum", SUMS)
def test_beside_the_lines(pcs, ctx, oracle, kernel, R, B, count, f64, ssd, cum):
    _distances(pcs, ctx, oracle, kernel, R, B, count, f64, ssd, cum, 0)


@pytest.mark.parametrize("name", ["lognormal", "ragged", "kmin-1", "box-edge", "long-steps", "one-frame"])
@pytest.mark.parametrize("block", [64, 256, 512, 1024])
def test_walks_without_screening(pcs, ctx, name, block):
    """120000 particles: more than k_simulate_few takes, and about one slice
    per warp, so that k_simulate_walk walks each slice at once."""
    model, C, F, kmin, sd, depth, half_l, half_a = CASES[name]
    frames = np.random.default_rng(5).integers(1, 140, VIDEOS) if F == "ragged" else np.full(VIDEOS, F)
    setup = pcs.ForwardSetup(model, C, frames.astype(np.uint32), kmin, 0.2, half_l, half_a, 0.125, int(frames.max()) + 1, 64)
    runs = _runs(pcs, C, sd, depth, model == 1, -0.2 if model == 2 else None, per_video=1500)
    want, got = _both(pcs, ctx, setup, runs, block_size=block)
    assert pcs.lib().pcs_debug_last_kernel(0) == b"k_simulate_walk"
    assert want.sum() > 0 and np.array_equal(got, want)


@pytest.mark.parametrize("per_video", [1, 90])
def test_few_particles_with_kmin_0(pcs, ctx, per_video):
    """kmin 0 records a track for every frame that does not find the particle:
    not k_simulate_few's."""
    model, C, F, kmin, sd, depth, half_l, half_a = CASES["kmin-0"]
    setup = pcs.ForwardSetup(model, C, np.full(VIDEOS, F, np.uint32), kmin, 0.2, half_l, half_a, 0.125, F + 1, 64)
    want, got = _both(pcs, ctx, setup, _runs(pcs, C, sd, depth, False, per_video=per_video))
    assert pcs.lib().pcs_debug_last_kernel(0) == b"k_simulate_walk"
    assert want.sum() > 0 and np.array_equal(got, want)
