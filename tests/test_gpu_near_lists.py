"""Steps that the pruned scan takes from the near columns listed by the commit:
every candidate's neighbour lists and predictions against the rows-per-lane
scorer, after every step, and that the lists were there to be used."""
import numpy as np
import pytest

from speedynn_b200 import datagen
from speedynn_b200.selector import Selector, release_memory

pytestmark = pytest.mark.gpu

STEPS = 6


def _steps(s, k, holdout, check):
    sels = []
    try:
        for kernel in (0, 1):
            sel = Selector(s.Xtrain, s.ytrain, s.Xval if holdout else None, s.yval if holdout else None, k_vals=[k],
                           num_features=STEPS, method="forward", k_fold=5)
            sels.append(sel)
            sel.set_kernel(kernel)
            sel.keep_neighbours(True)
        n_rows = (s.Xval if holdout else s.Xtrain).shape[0]
        rows = np.arange(0, n_rows, max(1, n_rows // 500), dtype=np.int32)
        for t in range(STEPS):
            near = sels[0].near_lists()  # of the commit before this step
            got, want = ((sel.step(), *sel.neighbours_rows(rows), *sel.predictions(rows)) for sel in sels)
            for a, b in zip(got, want):
                np.testing.assert_array_equal(a, b, err_msg=f"step {t}")
            check(t, near, n_rows)
    finally:
        for sel in sels:
            sel.close()


@pytest.mark.parametrize("k", [1, 9, 16, 17, 50, 150])
@pytest.mark.parametrize("n,m,p", [(16384, 300, 11), (17001, 4400, 9)])
@pytest.mark.parametrize("kind", ["plain", "dup", "integers", "wild"])
def test_lists_of_listed_steps(n, m, p, k, kind):
    s = datagen.generate(n, m, p, n_mag=5, seed=n + k, dup_frac=0.3 if kind == "dup" else 0.0)
    for X in (s.Xtrain, s.Xval):
        if kind == "integers":
            X[:] = np.rint(X)
        if kind == "wild":
            rng = np.random.default_rng(n)
            X[rng.integers(0, X.shape[0], 8), rng.integers(0, p, 8)] *= 1e4
            X[rng.integers(0, X.shape[0], 3), 1] = (np.nan, np.inf, -np.inf)

    def check(t, near, n_rows):
        assert near["kept"]
        if t < 2:  # the first commit has no earlier one to go by
            assert near["usable"] == 0
        elif kind == "plain":
            assert near["usable"] > n_rows // 4

    _steps(s, k, True, check)


def test_lists_of_listed_steps_across_folds():
    s = datagen.generate(16390, 1, 9, n_mag=5, seed=8)

    def check(t, near, n_rows):
        assert near["kept"] and (t < 2 or near["usable"] > n_rows // 4)

    _steps(s, 10, False, check)


def test_fewer_columns_keep_no_lists():
    s = datagen.generate(16383, 64, 9, n_mag=5, seed=9)

    def check(t, near, n_rows):
        assert near == {"kept": False, "usable": 0}

    _steps(s, 5, True, check)


def test_nearly_full_device_keeps_no_lists():
    import torch

    s = datagen.generate(16384, 20000, 9, n_mag=5, seed=3)

    def run():
        with Selector(s.Xtrain, s.ytrain, s.Xval, s.yval, k_vals=[5], num_features=5, method="forward") as sel:
            took = free - torch.cuda.mem_get_info(0)[0]
            return sel.run(), sel.near_lists(), took

    release_memory()  # what earlier handles left would make room for the lists
    free, _ = torch.cuda.mem_get_info(0)
    want, near, took = run()
    assert near["kept"] and near["usable"] > 5000
    free, _ = torch.cuda.mem_get_info(0)
    hog = torch.empty(free - took + 200 * 10**6, dtype=torch.uint8, device="cuda:0")  # of 328 MB of lists
    try:
        got, near, _ = run()
    finally:
        del hog
        torch.cuda.empty_cache()
    assert near == {"kept": False, "usable": 0}
    for key in ("ordering", "errors", "errors64"):
        np.testing.assert_array_equal(got[key], want[key], err_msg=key)
