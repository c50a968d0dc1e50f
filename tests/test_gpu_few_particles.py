"""Few particles (four or eight lanes per particle, a lane per coordinate): the
histogram is the item-by-item kernel's, count for count -- every model and
edge of the walk, track lengths and frame counts around the blocks of 16 and
32 frames, particle counts around a warp's 4 or 8 and an item's 32, and
launches just below and above the rules' lines."""
import numpy as np
import pytest

from test_gpu_screen import CASES, VIDEOS, _both, _runs

pytestmark = pytest.mark.gpu


def _setup(pcs, model, C, frames, kmin, half_l, half_a):
    return pcs.ForwardSetup(model, C, frames.astype(np.uint32), kmin, 0.2, half_l, half_a, 0.125, int(frames.max()) + 1, 64)


@pytest.mark.parametrize("per_video", [90, 300])  # 7200 particles: eight lanes; 24000: four
@pytest.mark.parametrize("name", list(CASES))
def test_walks(pcs, ctx, name, per_video):
    model, C, F, kmin, sd, depth, half_l, half_a = CASES[name]
    frames = np.random.default_rng(5).integers(1, 140, VIDEOS) if F == "ragged" else np.full(VIDEOS, F)
    runs = _runs(pcs, C, sd, depth, model == 1, -0.2 if model == 2 else None, per_video=per_video)
    want, got = _both(pcs, ctx, _setup(pcs, model, C, frames, kmin, half_l, half_a), runs)
    assert np.array_equal(got, want), (name, int(want.sum()), int(np.abs(got.astype(np.int64) - want).sum()))
    assert want.sum() > 0 or name == "never-in"


@pytest.mark.parametrize("frames", [1, 2, 16, 17, 18, 32, 33, 34, 65, 100])
@pytest.mark.parametrize("kmin", [1, 2, 16, 17, 33])
@pytest.mark.parametrize("per_video", [90, 150])
def test_blocks_of_frames(pcs, ctx, frames, kmin, per_video):
    setup = _setup(pcs, 0, 1, np.full(VIDEOS, frames), kmin, (20.0, 20.0, 4.0), (15.0, 15.0))  # tracks of all lengths
    want, got = _both(pcs, ctx, setup, _runs(pcs, 1, 0.7, 5.0, False, per_video=per_video))
    assert np.array_equal(got, want)


@pytest.mark.parametrize("counts", [[0], [1], [7], [8], [9], [31], [32], [33], [0, 5, 0, 40], [1] * 700])
def test_counts(pcs, ctx, counts):
    setup = _setup(pcs, 0, 1, np.full(2, 40), 1, (20.0, 20.0, 4.0), (15.0, 15.0))
    pre = np.array([2.0], np.float32)
    runs = [pcs.ForwardRun(np.array([n - n // 2, n // 2], np.uint32), np.array([2.5], np.float32), pre,
                           np.array([0.7], np.float32), None, slot=q) for q, n in enumerate(counts)]
    want, got = _both(pcs, ctx, setup, runs)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("items", [255, 256, 257, 2047, 2048, 2049])
def test_around_the_line(pcs, ctx, items):
    setup = _setup(pcs, 0, 1, np.full(1, 30), 2, (20.0, 20.0, 4.0), (15.0, 15.0))
    run = pcs.ForwardRun(np.array([32 * items], np.uint32), np.array([1.0], np.float32), np.array([2.0], np.float32),
                         np.array([0.7], np.float32), None)
    want, got = _both(pcs, ctx, setup, [run])
    assert np.array_equal(got, want) and want.sum() > 0
