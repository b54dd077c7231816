"""The probe that leaves a backward run to the dense scorer counts its warps
right for any number of candidates: 1,020 are 32 groups of a warp's lanes,
1,056 are 33 and 2,052 are 65.  All features but one are constant, so half of
all distances are equal and pruning does not pay."""
import numpy as np
import pytest

from speedynn_b200.selector import Selector

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [1020, 1056, 2052])
def test_dense_scorer_takes_over(p):
    n, m = 1100, 140
    rng = np.random.default_rng(p)
    X, Xv = np.ones((n, p), np.float32), np.ones((m, p), np.float32)
    X[:, 7], Xv[:, 7] = rng.random(n) < 0.5, rng.random(m) < 0.5
    y, yv = rng.random(n, dtype=np.float32), rng.random(m, dtype=np.float32)
    out = []
    for kernel in (0, 3):
        with Selector(X, y, Xv, yv, k_vals=[5], num_features=p - 1, method="backward") as sel:
            sel.set_kernel(kernel)
            out.append((sel.run(), sel.timing()["launches"]))
    # the scan would pack the candidates first
    assert out[0][1] == out[1][1]
    for key in ("ordering", "errors", "errors64"):
        np.testing.assert_array_equal(out[0][0][key], out[1][0][key], err_msg=key)
