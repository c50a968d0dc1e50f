"""The row kernel (many turns of strips: many histograms, many columns, tall
ones) against the oracle, bit for bit: remainders of rows, columns, lanes and
warps, rows that are not 16-byte aligned, histograms zeroed, cumulative counts
around 2^22 in some histograms of a launch, double sums around 2^53, rounds
that mix narrow and wide jobs."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(9, 4, 2500), (7, 1, 3800), (8, 128, 700), (33, 127, 1000), (65, 129, 900), (16, 132, 640), (1, 256, 650),
          (201, 255, 310), (40, 1024, 2), (31, 1023, 3), (9, 1025, 2), (1700, 96, 2), (1665, 132, 3), (301, 640, 1)]


def _check(r, oracle, hist, ref, q):
    d32, cum, ssd = oracle.distance_kdist(hist, ref)
    assert r["dist_f32"][q].tobytes() == np.float32(d32).tobytes(), q
    if r.get("cum") is not None:
        assert np.array_equal(r["cum"][q], cum), q
    if r.get("ssd") is not None:
        assert r["ssd"][q] == ssd, q
    if r.get("dist_f64") is not None:
        assert r["dist_f64"][q] == oracle.distance_kdist_f64(hist, ref), q


@pytest.mark.parametrize("R,B,count", SHAPES)
@pytest.mark.parametrize("f64,ssd,cum", [(False, False, False), (True, False, True), (False, True, False), (True, True, True)])
def test_shapes(pcs, ctx, oracle, R, B, count, f64, ssd, cum):
    rng = np.random.default_rng(R * 7 + B)
    hist = rng.poisson(0.7, (count, R, B)).astype(np.uint32)
    ref = np.cumsum(np.cumsum(rng.poisson(0.7, (R, B)), 0), 1).astype(np.uint32)
    hist[count // 2, R // 2, B // 2] = 2**22  # one histogram past the integer form from this row on
    r = pcs.scan_distance(ctx, hist, ref, want_f64=f64, want_ssd=ssd, want_cum=cum)
    for q in range(count):
        _check(r, oracle, hist[q], ref, q)


@pytest.mark.parametrize("R,B,count", [(40, 1024, 3), (33, 999, 3)])
@pytest.mark.parametrize("observed", [False, True])
def test_integer_and_double_edges(pcs, ctx, oracle, R, B, count, observed):
    below = int(np.sqrt(2**53 / (R * B))) - 1  # a sum of squares just below 2^53
    for total in (below, below + 2, 2**22 - 1, 2**22, 2**22 + 1, 2**32 - 1):
        hist = np.zeros((count, R, B), np.uint32)
        hist[0, 0, 0] = hist[1, R - 1, B - 1] = total
        hist[2, R - 1, 0] = 5
        if observed:
            hist[0], hist[2] = hist[2].copy(), hist[0].copy()
        ref = np.full((R, B), total if observed else 0, np.uint32)
        r = pcs.scan_distance(ctx, hist, ref, want_f64=True, want_ssd=True, want_cum=True)
        one = pcs.scan_distance(ctx, hist, ref)
        for q in range(count):
            _check(r, oracle, hist[q], ref, q)
            assert one["dist_f32"][q].tobytes() == r["dist_f32"][q].tobytes(), q


@pytest.mark.parametrize("count,R,B,offset", [(700, 40, 128, 0), (900, 33, 128, 1), (900, 33, 127, 2), (3, 50, 1024, 3),
                                              (2, 1700, 132, 0)])
def test_buffers(pcs, ctx, oracle, count, R, B, offset):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(count)
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


@pytest.mark.parametrize("double", [0, 1])
def test_mixed_rounds(pcs, ctx, double):
    import part_conc_spt_abc_gb300.workloads as W
    inputs = []
    for j, bins in enumerate([33, 300, 128, 999, 64, 1024]):
        inp, _ = W.make_problem(ctx, [150.0 + 40 * j], [10.0], 5e13, [1.0], 3, 20 + 9 * j, bins, 24, 2, seed=j)
        inp.params.avg_trial_count = 50
        inp.params.distance_double = double
        inputs.append(inp)

    def out(sim):
        o, i = sim.output(), sim.info()
        return [o.m, o.s, o.c, o.dist, o.w, i.gamma, i.trials, i.accepted, i.iterations, i.converged]

    alone = []
    for j, inp in enumerate(inputs):
        sim = pcs.make_simulation(ctx, inp, 100 + j)
        sim.run()
        alone.append(out(sim))
        sim.close()
    srv = pcs.Server(ctx)
    sims = [pcs.make_simulation(ctx, inp, 100 + j) for j, inp in enumerate(inputs)]
    for sim in sims:
        srv.submit(sim)
    while srv.step():
        pass
    for j, want in enumerate(alone):
        for a, b in zip(out(sims[j]), want):
            assert np.array_equal(a, b), j
    for sim in sims:
        sim.close()
