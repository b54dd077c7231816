"""Loss lists at the edges of what snn_set_model takes: longer than a launch
grid is high."""
import numpy as np
import pytest

from speedynn_b200 import datagen
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
