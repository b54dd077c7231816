"""Warm starts: several features committed at once against the same features
committed one per step (commit_sequence of a prefix against the run it is from)."""
import numpy as np
import pytest

from speedynn_b200 import datagen
from speedynn_b200.selector import Selector

pytestmark = pytest.mark.gpu


# columns around the 512 that a block stages, rows around its sixteen; prefixes around the sixteen features of a launch
@pytest.mark.parametrize("n,m", [(97, 15), (511, 16), (512, 17), (1540, 33), (4700, 300)])
@pytest.mark.parametrize("cut", [1, 2, 16, 17, 36])
@pytest.mark.parametrize("method", ["forward", "backward"])
@pytest.mark.parametrize("cv", [False, True])
def test_prefix_at_once_equals_steps(n, m, cut, method, cv):
    p, k = 38, [3]
    s = datagen.generate(n, m, p, n_mag=5, seed=n + cut)
    data = (s.Xtrain, s.ytrain) if cv else (s.Xtrain, s.ytrain, s.Xval, s.yval)
    kw = dict(k_vals=k, num_features=36 if method == "forward" else 2, method=method, k_fold=4 if cv else 0)
    if cv and n > 1600:
        pytest.skip("the smaller ones cover the folds")
    with Selector(*data, **kw) as sel:
        full = sel.run()
    steps = 36  # forward fills the slots from the front, backward from the back
    slots = np.arange(steps) if method == "forward" else p - 1 - np.arange(steps)
    with Selector(*data, **kw) as sel:
        for _ in range(2):  # a fresh handle, then one that has run
            sel.commit_sequence(full["ordering"][slots[:cut]])
            while sel.step():
                pass
            res = sel.results()
            np.testing.assert_array_equal(res["ordering"], full["ordering"])
            np.testing.assert_array_equal(res["mask"], full["mask"])
            np.testing.assert_array_equal(res["errors"][slots[cut:]], full["errors"][slots[cut:]])
            np.testing.assert_array_equal(res["errors64"][slots[cut:]], full["errors64"][slots[cut:]])
