"""The tile-less walk kernel (k_simulate_walk): screened particles, particles
walked in step by a warp and tracks binned in batches give the histogram of
the item-by-item kernel (a shared-memory tile), count for count."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PER_VIDEO, VIDEOS, RUNS = 3300, 20, 4  # 264000 particles: more than two slices for every warp, so the launch screens


def _runs(pcs, C, sd, depth, variable, shape=None, per_video=PER_VIDEO):
    rng = np.random.default_rng(C)
    pre = (np.arange(1, C + 1) / C).astype(np.float32)
    pre[-1] = 2.0
    sds = (np.float32(sd) * np.linspace(1.0, 0.4, C)).astype(np.float32)
    haz = (0.5 * depth * np.linspace(1.0, 1.4, C if variable else 1)).astype(np.float32)
    return [pcs.ForwardRun(rng.poisson(per_video, VIDEOS).astype(np.uint32), haz, pre, sds,
                           None if shape is None else np.full(C, shape, np.float32), slot=q, trial=1, generation=2)
            for q in range(RUNS)]


def _both(pcs, ctx, setup, runs, **tuning):
    keep = ctx.tuning
    try:
        ctx.set_tuning(hist_tile_rows=16, block_size=256, particles_per_thread=1)
        want = pcs.simulate_hist(ctx, setup, runs, seed=11)
        ctx.set_tuning(hist_tile_rows=0xFFFFFFFF, **tuning)
        return want, pcs.simulate_hist(ctx, setup, runs, seed=11)
    finally:
        ctx.set_tuning(hist_tile_rows=keep.hist_tile_rows or 0xFFFFFFFF, block_size=keep.block_size)


CASES = {
    # model, C, frames, kmin, step sd, depth, half box, half area
    "lognormal": (2, 2, 60, 2, 0.4, 2.0, (100.0, 80.0, 10.0), (50.0, 40.0)),
    "ragged": (2, 3, "ragged", 2, 0.5, 2.0, (100.0, 80.0, 10.0), (50.0, 40.0)),
    "variable-depth": (1, 3, 75, 3, 0.3, 2.0, (40.0, 40.0, 10.0), (30.8, 30.8)),
    "kmin-0": (0, 1, 50, 0, 0.4, 2.0, (100.0, 80.0, 10.0), (50.0, 40.0)),
    "kmin-1": (0, 2, 51, 1, 0.4, 2.0, (100.0, 80.0, 10.0), (50.0, 40.0)),
    "z-only": (0, 1, 52, 2, 0.3, 1.0, (100.0, 80.0, 10.0), (100.0, 80.0)),
    "always-in": (0, 1, 53, 2, 0.3, 100.0, (100.0, 80.0, 10.0), (100.0, 80.0)),
    "never-in": (0, 1, 54, 2, 0.3, 2.0, (100.0, 80.0, 10.0), (-1.0, 40.0)),
    "long-steps": (0, 2, 55, 2, 12.0, 2.0, (100.0, 80.0, 10.0), (50.0, 40.0)),
    "no-steps": (0, 1, 56, 2, 0.0, 2.0, (100.0, 80.0, 10.0), (50.0, 40.0)),
    "edge": (0, 1, 48, 2, 2.5, 2.0, (100.0, 80.0, 10.0), (98.0, 79.0)),
    "box-edge": (0, 1, 90, 2, 0.8, 4.0, (20.0, 19.0, 10.0), (1.0, 0.5)),  # groups with and without x, y wraps
    "tiny-steps": (0, 1, 64, 2, 1e-6, 4.0, (100.0, 80.0, 10.0), (99.0, 79.0)),  # steps near one rounding of x
    "short": (0, 2, 47, 2, 0.4, 2.0, (100.0, 80.0, 10.0), (50.0, 40.0)),
    "one-step": (2, 1, 2, 1, 0.4, 2.0, (100.0, 80.0, 10.0), (50.0, 40.0)),
    "one-frame": (2, 1, 1, 1, 0.4, 2.0, (100.0, 80.0, 10.0), (50.0, 40.0)),
}


@pytest.mark.parametrize("name", list(CASES))
def test_walk_kernel_equals_tile_kernel(pcs, ctx, name):
    model, C, F, kmin, sd, depth, half_l, half_a = CASES[name]
    frames = np.random.default_rng(5).integers(1, 140, VIDEOS) if F == "ragged" else np.full(VIDEOS, F)
    setup = pcs.ForwardSetup(model, C, frames.astype(np.uint32), kmin, 0.2, half_l, half_a, 0.125, int(frames.max()) + 1, 64)
    want, got = _both(pcs, ctx, setup, _runs(pcs, C, sd, depth, model == 1, -0.2 if model == 2 else None))
    assert np.array_equal(got, want), (name, int(want.sum()), int(np.abs(got.astype(np.int64) - want).sum()))
    assert want.sum() > 0 or name == "never-in"


@pytest.mark.parametrize("block,per_video", [(64, PER_VIDEO), (512, PER_VIDEO), (1024, 2 * PER_VIDEO), (256, 300), (256, 1)])
def test_walk_kernel_launch_shapes(pcs, ctx, block, per_video):
    """Other CTA sizes, and launches too small to screen."""
    setup = pcs.ForwardSetup(0, 2, np.full(VIDEOS, 64, np.uint32), 2, 0.2, (100.0, 80.0, 10.0), (50.0, 40.0), 0.125, 65, 64)
    want, got = _both(pcs, ctx, setup, _runs(pcs, 2, 0.4, 2.0, False, per_video=per_video), block_size=block)
    assert np.array_equal(got, want)
