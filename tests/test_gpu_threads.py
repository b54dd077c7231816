"""Handles of different list lengths used from several threads at once: their
launches share kernel instances (and those instances' limits), their results
are the ones they have alone."""
import threading

import numpy as np
import pytest

from speedynn_b200 import datagen
from speedynn_b200.selector import Selector

pytestmark = pytest.mark.gpu

KS = (9, 12, 20, 60, 200, 256)


@pytest.mark.parametrize("kernel,runs", [(0, 150), (1, 10)])
@pytest.mark.parametrize("method", ["forward", "backward"])
def test_list_lengths_from_several_threads(kernel, runs, method):
    s = datagen.generate(600, 60, 9, n_mag=5, seed=17)

    def run(k):
        with Selector(s.Xtrain, s.ytrain, s.Xval, s.yval, k_vals=[k], num_features=4, method=method) as sel:
            sel.set_kernel(kernel)
            return [sel.run() for _ in range(runs)]

    want = {k: run(k)[-1] for k in KS}
    errors = []

    def work(k):
        try:
            for r in run(k):
                for key in ("ordering", "errors64"):
                    np.testing.assert_array_equal(r[key], want[k][key], err_msg=f"k = {k}")
        except Exception as e:  # noqa: BLE001 -- reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in KS * 2]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
