"""The standalone entry points' kept workspace: calls of very different sizes
in turn (larger ones than it keeps among them), and several threads on one
context, give what a call on its own gives."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _calls(pcs, ctx):
    import part_conc_spt_abc_gb300.workloads as W
    rng = np.random.default_rng(3)
    out = []
    for R, B, n in [(5, 3, 1), (301, 128, 40), (201, 100, 1), (1001, 256, 70), (33, 40, 900)]:  # 70 x 1001 x 256: 72 MB
        h = rng.poisson(0.5, (n, R, B)).astype(np.uint32)
        ref = np.cumsum(np.cumsum(rng.poisson(0.5, (R, B)), 0), 1).astype(np.uint32)
        out.append(lambda h=h, ref=ref: pcs.scan_distance(ctx, h, ref, want_f64=True, want_ssd=True)["dist_f64"])
    for n, R, B in [(10, 20, 20), (60000, 301, 128)]:
        K, DE = rng.integers(0, R, n), rng.uniform(0, 6, n)
        out.append(lambda K=K, DE=DE, R=R, B=B: pcs.observed_sat(ctx, K, DE, R, B, 5.0))
    for frames, count in [(30, 1), (80, 300)]:
        setup = W.forward_setup(np.full(6, frames, np.uint32), 64)
        runs = [W.lognormal_run(rng.poisson(40, 6), [200.0], [10.0], [1.0], slot=q) for q in range(count)]
        out.append(lambda setup=setup, runs=runs: pcs.simulate_hist(ctx, setup, runs, seed=5))
    return out


def test_sizes_in_turn(pcs, ctx):
    calls = _calls(pcs, ctx)
    want = [f() for f in calls]
    for i in [4, 0, 3, 1, 8, 5, 3, 2, 6, 7, 0]:
        assert np.array_equal(calls[i](), want[i]), i
    with pytest.raises(pcs.PcsError):  # a call that fails leaves the workspace usable
        pcs.observed_sat(ctx, np.array([9]), np.array([1.0]), 4, 4, 5.0)
    assert np.array_equal(calls[1](), want[1])


def test_several_threads(pcs, ctx):
    calls = _calls(pcs, ctx)
    want = [f() for f in calls]
    wrong = []

    def work(k):
        for i in range(3 * len(calls)):
            j = (i * 5 + k) % len(calls)
            try:
                same = np.array_equal(calls[j](), want[j])
            except Exception as e:  # noqa: BLE001 -- a thread's exception would be lost
                same, j = False, (j, repr(e))
            if not same:
                wrong.append((k, j))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
