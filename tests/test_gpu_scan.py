"""The pruned scan (automatic kernel choice) against the rows-per-lane scorer,
which evaluates every pair: identical selections and, at one of the pruned
steps, identical neighbour lists.  Sizes sit at the edges of the scan's shapes:
512-column passes, 32-candidate groups, heaps of 1 to 256 entries, the 4,096
columns from which outlying candidates are scanned on their own."""
import ctypes

import numpy as np
import pytest

from speedynn_b200 import _lib, datagen
from speedynn_b200._lib import _i32p, ptr
from speedynn_b200.selector import Selector

pytestmark = pytest.mark.gpu


def _data(n, m, p, seed, kind):
    s = datagen.generate(n, max(m, 1), p, n_mag=min(5, (p + 1) // 2), n_heavy=max(0, min(3, p - 9)), seed=seed,
                         dup_frac=0.3 if kind == "dup" else 0.0)
    if kind == "ties":  # integer-valued features: many equal distances
        for X in (s.Xtrain, s.Xval):
            X[:] = np.rint(X)
    if kind == "binary":  # two-valued features: most columns stay open, the dense scorer takes over
        for X in (s.Xtrain, s.Xval):
            X[:] = X > np.median(X, axis=0)
    if kind == "wild":  # outlying rows, non-finite values, a constant feature
        rng = np.random.default_rng(seed)
        for X in (s.Xtrain, s.Xval):
            X[rng.integers(0, X.shape[0], 8), rng.integers(0, p, 8)] *= 1e4
            X[rng.integers(0, X.shape[0], 3), 1] = (np.nan, np.inf, -np.inf)
        s.Xtrain[:, 2] = s.Xval[:, 2] = 1.0
    return s


CASES = [
    # n_train, n_val (0: CV), p, k_vals, method, steps to run, data
    (511, 65, 34, [1], "forward", 4, "plain"),
    (512, 40, 35, [16, 3], "forward", 4, "ties"),
    (513, 33, 67, [17], "forward", 4, "dup"),
    (1025, 0, 12, [64, 5], "forward", 5, "plain"),
    (700, 0, 33, [9], "forward", 4, "wild"),
    (2000, 50, 14, [150, 65], "forward", 4, "plain"),
    (600, 90, 12, [256], "forward", 4, "dup"),
    (4095, 130, 40, [10], "forward", 5, "plain"),
    (4096, 130, 40, [10], "forward", 5, "wild"),
    (5000, 300, 37, [10], "forward", 6, "wild"),  # 32 candidates at the sixth step: a full group
    (4100, 300, 35, [50], "forward", 4, "wild"),
    (9001, 301, 66, [5, 20], "forward", 5, "wild"),
    (8192, 120, 40, [10, 1], "forward", 5, "ties"),
    (4500, 4300, 12, [10], "forward", 4, "binary"),
    (4500, 4300, 12, [70], "forward", 4, "binary"),
    (511, 65, 34, [1], "backward", 4, "plain"),
    (513, 0, 33, [16, 3], "backward", 4, "ties"),
    (1000, 70, 65, [5], "backward", 5, "dup"),
    (3000, 0, 32, [9], "backward", 20, "plain"),
    (1500, 64, 31, [40], "backward", 10, "wild"),
    (900, 64, 12, [200], "backward", 8, "plain"),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(str(x) for x in c[:3]) + f"-k{max(c[3])}-{c[4]}-{c[6]}")
def test_scan_equals_scoring_every_pair(case):
    n, m, p, kv, method, steps, kind = case
    s = _data(n, m, p, n + p, kind)
    Xv, yv = (s.Xval, s.yval) if m else (None, None)
    out = {}
    for kernel in (0, 1):
        with Selector(s.Xtrain, s.ytrain, Xv, yv, k_vals=kv, num_features=steps if method == "forward" else p - steps,
                      method=method, k_fold=3) as sel:
            sel.set_kernel(kernel)
            r = sel.run()
            sel.reset()
            for _ in range(steps - 1):
                assert sel.step()
            sel.keep_neighbours(True)
            assert sel.step()
            out[kernel] = (r, sel.neighbours())
    (ra, na), (rb, nb) = out[0], out[1]
    for k in ("ordering", "mask", "errors", "errors64", "step_best_k", "best_k", "num_final"):
        np.testing.assert_array_equal(ra[k], rb[k], err_msg=k)
    for a, b in zip(na, nb):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("shape", [(1500, 400, 14, 3), (4500, 4300, 12, 0), (4500, 4300, 12, 2), (2500, 300, 40, 5)])
@pytest.mark.parametrize("k", [7, 80])
def test_device_step_equals_a_handles(shape, k):
    """snn_score_step_noalloc against a handle that scores every pair, after
    `steps` committed features (none: every distance is zero, and the larger
    problem goes to the dense scorer)."""
    import torch

    n, m, p, steps = shape
    s = _data(n, m, p, n + k, "plain")
    prefix = list(range(1, steps + 1))
    with Selector(s.Xtrain, s.ytrain, s.Xval, s.yval, k_vals=[k], num_features=steps + 1, method="forward") as sel:
        sel.set_kernel(1)
        sel.commit_sequence(prefix)
        assert sel.step()
        rows = np.arange(m, dtype=np.int32)
        cands, pred = sel.predictions(rows)
    e = (s.yval[None, :] - pred[:, 0]).astype(np.float32)
    sq = (e * e).astype(np.float32)
    want = np.sqrt((np.add.accumulate(sq, axis=1, dtype=np.float32)[:, -1] / np.float32(m)).astype(np.float64)).astype(np.float32)
    dev = torch.device("cuda", 0)
    ld = (n + 63) // 64 * 64
    XT = torch.zeros((p, ld), dtype=torch.float32, device=dev)
    XT[:, :n] = torch.from_numpy(np.ascontiguousarray(s.Xtrain.T)).to(dev)
    XV = torch.from_numpy(np.ascontiguousarray(s.Xval.T)).to(dev)
    D = torch.zeros((m, ld), dtype=torch.float32, device=dev)
    for f in prefix:
        t = XV[f][:, None] - XT[f][None, :]
        D += t.mul_(t)
    D[:, n:] = float("inf")
    yt, yv = torch.from_numpy(s.ytrain).to(dev), torch.from_numpy(s.yval).to(dev)
    out = torch.zeros((cands.size, 1), dtype=torch.float32, device=dev)
    out64 = torch.zeros((cands.size, 1), dtype=torch.float64, device=dev)
    kv = np.array([k], np.int32)
    rc = _lib.lib().snn_score_step_noalloc(
        D.data_ptr(), ld, XT.data_ptr(), XV.data_ptr(), m, yt.data_ptr(), yv.data_ptr(), m, n, p, ptr(cands, _i32p), cands.size,
        ptr(kv, _i32p), 1, 0, out.data_ptr(), out64.data_ptr(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, _lib.lib().snn_last_error()
    np.testing.assert_array_equal(out.cpu().numpy()[:, 0], want)
