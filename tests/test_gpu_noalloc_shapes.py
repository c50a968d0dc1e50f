"""pcs_scan_distance_noalloc over the launches it takes: tensor maps and cell
copies (bins not a multiple of 4, rows or bins below 32, a buffer that is not
16-byte aligned), clusters and strip walks, histograms taller than a strip."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,R,B,offset", [(3, 32, 32, 0), (5, 31, 64, 0), (4, 64, 31, 0), (6, 301, 128, 1),
                                              (340, 120, 96, 0), (20, 640, 70, 0), (130, 600, 64, 0), (2, 1001, 256, 2),
                                              (3, 201, 1000, 0), (2, 1800, 40, 0), (1, 1, 1, 3)])
def test_noalloc_shapes(pcs, ctx, oracle, count, R, B, offset):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(count * 7 + R)
    hist = rng.poisson(0.8, (count, R, B)).astype(np.uint32)
    ref = np.cumsum(np.cumsum(rng.poisson(0.8, (R, B)), 0), 1).astype(np.uint32)
    buf = torch.full((count * R * B + 8,), 77, dtype=torch.int32, device="cuda")
    buf[offset:offset + hist.size] = torch.from_numpy(hist.view(np.int32).reshape(-1)).cuda()
    d_ref = torch.from_numpy(ref.view(np.int32).copy()).cuda()
    dist = torch.full((count,), -1.0, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    st = pcs.lib().pcs_scan_distance_noalloc(C.c_void_p(buf.data_ptr() + 4 * offset), C.c_void_p(d_ref.data_ptr()), R, B,
                                             count, C.c_void_p(dist.data_ptr()), None)
    assert st == 0, pcs.lib().pcs_last_error()
    got, after = dist.cpu().numpy(), buf.cpu().numpy()
    for q in range(count):
        assert got[q].tobytes() == np.float32(oracle.distance_kdist(hist[q], ref)[0]).tobytes(), q
    assert not after[offset:offset + hist.size].any()
    assert (after[:offset] == 77).all() and (after[offset + hist.size:] == 77).all()
