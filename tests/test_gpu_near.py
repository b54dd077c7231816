"""Pruned scan over the near columns that a commit lists (forward, 16,384
training columns and more) against the rows-per-lane scorer, which evaluates
every pair: identical selections.  Data decide how long the lists get: two-valued
ones overflow or stay empty, duplicates and integers tie at their edge, and
outlying rows leave most columns beyond it."""
import numpy as np
import pytest

from speedynn_b200 import datagen
from speedynn_b200.selector import Selector

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,p", [(16384, 300, 12), (16385, 4300, 11), (20011, 700, 40)])
@pytest.mark.parametrize("k", [3, 10, 16, 20, 50, 200])
@pytest.mark.parametrize("kind", ["plain", "dup", "integers", "binary", "wild"])
def test_listed_columns_equal_every_pair(n, m, p, k, kind):
    s = datagen.generate(n, m, p, n_mag=5, n_heavy=2, seed=n + k, dup_frac=0.3 if kind == "dup" else 0.0)
    for X in (s.Xtrain, s.Xval):
        if kind == "integers":
            X[:] = np.rint(X)
        if kind == "binary":
            X[:] = X > np.median(X, axis=0)
        if kind == "wild":
            rng = np.random.default_rng(n)
            X[rng.integers(0, X.shape[0], 8), rng.integers(0, p, 8)] *= 1e4
            X[rng.integers(0, X.shape[0], 3), 1] = (np.nan, np.inf, -np.inf)
    runs = []
    for kernel in (0, 1):
        with Selector(s.Xtrain, s.ytrain, s.Xval, s.yval, k_vals=[k], num_features=9, method="forward") as sel:
            sel.set_kernel(kernel)
            runs.append(sel.run())
    np.testing.assert_array_equal(runs[0]["ordering"], runs[1]["ordering"])
    np.testing.assert_array_equal(runs[0]["errors64"], runs[1]["errors64"])


@pytest.mark.parametrize("k", [5, 50])
def test_listed_columns_across_folds(k):
    """The same with folds, whose own columns (+inf in D) no list may hold."""
    s = datagen.generate(16390, 1, 9, n_mag=5, seed=k)
    runs = []
    for kernel in (0, 1):
        with Selector(s.Xtrain, s.ytrain, k_vals=[k], num_features=6, method="forward", k_fold=7) as sel:
            sel.set_kernel(kernel)
            runs.append(sel.run())
    np.testing.assert_array_equal(runs[0]["ordering"], runs[1]["ordering"])
    np.testing.assert_array_equal(runs[0]["errors64"], runs[1]["errors64"])


def test_without_memory_for_the_lists():
    """A problem that fits the device only without its lists runs without them."""
    import torch

    n, m = 16384, 20000
    s = datagen.generate(n, m, 9, n_mag=5, seed=3)

    def run():
        with Selector(s.Xtrain, s.ytrain, s.Xval, s.yval, k_vals=[5], num_features=5, method="forward") as sel:
            return sel.run()

    want = run()
    # D 1.31 GB, everything else but the 0.33 GB of lists below 0.1 GB
    free, _ = torch.cuda.mem_get_info(0)
    hog = torch.empty(free - 1560 * 10**6, dtype=torch.uint8, device="cuda:0")
    try:
        got = run()
    finally:
        del hog
        torch.cuda.empty_cache()
    np.testing.assert_array_equal(got["ordering"], want["ordering"])
    np.testing.assert_array_equal(got["errors64"], want["errors64"])
