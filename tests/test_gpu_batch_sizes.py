"""Batches whose problems have many (candidate, k) errors: a wave's memory is
sized to all of its problems' buffers."""
import numpy as np
import pytest

from speedynn_b200 import datagen
from speedynn_b200.batch import Batch
from speedynn_b200.selector import Selector

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,p,nk,method,nf", [
    (1024, 512, 500, 256, "forward", 2),
    (600, 0, 500, 200, "backward", 498),
    (64, 64, 300, 1, "forward", 3),
])
@pytest.mark.parametrize("copies", [1, 2])
def test_many_errors_fit_their_wave(n, m, p, nk, method, nf, copies):
    s = datagen.generate(n, max(m, 1), p, n_mag=5, seed=n)
    q = dict(Xtrain=s.Xtrain, ytrain=s.ytrain, k_vals=list(range(1, nk + 1)), num_features=nf, method=method, k_fold=3)
    if m:
        q.update(Xval=s.Xval, yval=s.yval)
    with Selector(**q) as sel:
        want = sel.run()
    with Batch([q] * copies) as b:
        got = b.run()
        waves = b.timing()["waves"]
    assert waves == 1 and len(got) == copies
    for r in got:
        for key in ("ordering", "errors", "errors64", "step_best_k"):
            np.testing.assert_array_equal(r[key], want[key], err_msg=key)
