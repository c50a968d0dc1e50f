"""A negative step sd (pcs_simulate_hist takes it) mirrors the steps: the
tile-less kernels wrap such particles at the box's edge like the tile kernel,
above and below the number of particles that k_simulate_few takes."""
import numpy as np
import pytest

from test_gpu_screen import PER_VIDEO, VIDEOS, _both, _runs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_video,kernel", [(PER_VIDEO, b"k_simulate_walk"), (90, b"k_simulate_few")])
@pytest.mark.parametrize("model,sd", [(0, -0.8), (0, -3.0), (2, -0.8)])
def test_negative_step_sd(pcs, ctx, per_video, kernel, model, sd):
    setup = pcs.ForwardSetup(model, 1, np.full(VIDEOS, 90, np.uint32), 2, 0.2, (20.0, 19.0, 10.0), (1.0, 0.5), 0.125, 91, 64)
    runs = _runs(pcs, 1, sd, 4.0, False, -0.2 if model == 2 else None, per_video=per_video)
    want, got = _both(pcs, ctx, setup, runs)
    assert pcs.lib().pcs_debug_last_kernel(0) == kernel
    assert want.sum() > 0 and np.array_equal(got, want), int(np.abs(got.astype(np.int64) - want).sum())
