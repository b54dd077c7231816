"""Features with many missing (NaN) training values: a missing value's distance
never enters a list, and a pruned step's starting bound must not count it as a
column.  The automatic choice against the rows-per-lane scorer, which evaluates
every pair: the neighbour lists and predictions of every candidate after every
step (a mostly missing feature rarely wins, so selections alone say little)."""
import numpy as np
import pytest

from speedynn_b200 import datagen
from speedynn_b200.selector import Selector

pytestmark = pytest.mark.gpu

SHARES = (0.5, 0.7, 0.95, 1.0)  # of the last four features' training values


def _data(n, m, p, seed):
    s = datagen.generate(n, max(m, 1), p, n_mag=5, seed=seed)
    rng = np.random.default_rng(seed)
    for j, share in zip(range(p - len(SHARES), p), SHARES):
        s.Xtrain[rng.random(n) < share, j] = np.nan
        s.Xval[rng.random(s.Xval.shape[0]) < 0.1, j] = np.nan
    return s


@pytest.mark.parametrize("k", [1, 5, 8, 9, 10, 16, 20])
@pytest.mark.parametrize("n,m,p,method,steps", [
    (1500, 90, 12, "forward", 4),
    (900, 0, 12, "forward", 4),
    (4200, 4150, 10, "forward", 4),  # more than one wave of warps
    (1500, 70, 36, "forward", 3),  # two groups of candidates
    (16500, 60, 11, "forward", 6),  # steps with listed near columns
    (1200, 80, 12, "backward", 5),
    (800, 0, 12, "backward", 5),
])
def test_missing_values_never_tighten_a_bound(n, m, p, method, steps, k):
    s = _data(n, m, p, n + k)
    Xv, yv = (s.Xval, s.yval) if m else (None, None)
    sels = []
    try:
        for kernel in (0, 1):
            sel = Selector(s.Xtrain, s.ytrain, Xv, yv, k_vals=[k], num_features=steps if method == "forward" else p - steps,
                           method=method, k_fold=3)
            sels.append(sel)
            sel.set_kernel(kernel)
            sel.keep_neighbours(True)
        rows = np.arange(m or n, dtype=np.int32)
        for t in range(steps):
            got, want = ((sel.step(), *sel.neighbours(), *sel.predictions(rows)) for sel in sels)
            for a, b in zip(got, want):
                np.testing.assert_array_equal(a, b, err_msg=f"step {t}")
        ra, rb = (sel.results() for sel in sels)
        for key in ("ordering", "errors", "errors64"):
            np.testing.assert_array_equal(ra[key], rb[key], err_msg=key)
    finally:
        for sel in sels:
            sel.close()
