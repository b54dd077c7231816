"""Loss lists at the edges of what snn_set_model takes: longer than a launch
grid is high, and too long for the device's memory."""
import numpy as np
import pytest

from speedynn_b200 import _lib, datagen
from speedynn_b200._lib import _i32p, ptr
from speedynn_b200.selector import Selector

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_losses", [65535, 65536, 131071])
def test_long_loss_lists(n_losses):
    s = datagen.generate(60, 40, 9, n_mag=5, seed=n_losses)
    ids = np.resize([2, 0, 4, 5], n_losses)  # the first decides
    out = []
    for lf in (ids, ids[:4]):
        with Selector(s.Xtrain, s.ytrain, s.Xval, s.yval, k_vals=[3], num_features=2, method="forward", loss_functions=lf) as sel:
            out.append(sel.run())
    np.testing.assert_array_equal(out[0]["ordering"], out[1]["ordering"])
    np.testing.assert_array_equal(out[0]["errors_all"], out[1]["errors_all"][np.arange(n_losses) % 4])


def test_list_without_memory_leaves_a_plain_handle():
    s = datagen.generate(300, 64, 500, n_mag=5, seed=7)
    ids = np.ones(2_000_000, np.int32)  # x 500 candidates x 64 list lengths: 256 GB of losses
    with Selector(s.Xtrain, s.ytrain, s.Xval, s.yval, k_vals=range(1, 65), num_features=3, method="forward") as sel:
        want = sel.run()
        assert _lib.lib().snn_set_model(sel._h, ptr(ids, _i32p), ids.size, 1) == _lib.SNN_ERR_NOMEM
        got = sel.run()
    for key in ("ordering", "errors", "errors64", "step_best_k", "errors_all"):
        np.testing.assert_array_equal(got[key], want[key], err_msg=key)
