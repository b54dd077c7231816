"""Handles on a device that is nearly full: what only makes a problem faster is
left out before the problem is refused."""
import numpy as np
import pytest

from speedynn_b200 import datagen
from speedynn_b200.selector import Selector

pytestmark = pytest.mark.gpu


def test_without_memory_for_the_scan():
    """More scored rows than training columns: the list of walks is the largest
    thing that the pruned scan keeps (160 MB), and 80 MB are missing."""
    import torch

    s = datagen.generate(4096, 200000, 200, n_mag=5, seed=4)

    def make():
        return Selector(s.Xtrain, s.ytrain, s.Xval, s.yval, k_vals=[10], num_features=3, method="forward")

    torch.cuda.synchronize()
    free, _ = torch.cuda.mem_get_info(0)
    with make() as sel:
        took = free - torch.cuda.mem_get_info(0)[0]
        want = sel.run()
    assert took > 2 * 10**9  # a block of that size is not kept
    free, _ = torch.cuda.mem_get_info(0)
    hog = torch.empty(free - took + 80 * 10**6, dtype=torch.uint8, device="cuda:0")
    try:
        with make() as sel:
            got = sel.run()
    finally:
        del hog
        torch.cuda.empty_cache()
    for key in ("ordering", "errors", "errors64"):
        np.testing.assert_array_equal(got[key], want[key], err_msg=key)
