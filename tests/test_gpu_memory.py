"""Handles on a device that is nearly full: what only makes a problem faster is
left out before the problem is refused; and memory that closed handles keep."""
import numpy as np
import pytest

from speedynn_b200 import datagen
from speedynn_b200.selector import Selector, release_memory

pytestmark = pytest.mark.gpu


def test_without_memory_for_the_scan():
    """More scored rows than training columns: the list of walks is the largest
    thing that the pruned scan keeps (160 MB), and 80 MB are missing."""
    import torch

    s = datagen.generate(4096, 200000, 200, n_mag=5, seed=4)

    def make():
        return Selector(s.Xtrain, s.ytrain, s.Xval, s.yval, k_vals=[10], num_features=3, method="forward")

    torch.cuda.synchronize()
    release_memory()  # what earlier handles left would make room
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


@pytest.mark.parametrize("device", [0, -1])
def test_closed_handles_memory_is_given_back(device):
    import torch

    s = datagen.generate(4096, 4096, 9, n_mag=5, seed=5)

    def run():
        with Selector(s.Xtrain, s.ytrain, s.Xval, s.yval, k_vals=[5], num_features=2, method="forward") as sel:
            return sel.run()

    run()  # kernels are loaded
    release_memory(device)
    free, _ = torch.cuda.mem_get_info(0)
    want = run()
    kept = free - torch.cuda.mem_get_info(0)[0]
    assert 67 * 10**6 < kept <= 256 * 2**20
    with Selector(s.Xtrain, s.ytrain, k_vals=[5], num_features=2, method="forward") as sel:
        release_memory(device)  # a handle in use keeps its own
        in_use = sel.run()
        release_memory(device)
        np.testing.assert_array_equal(sel.run()["errors64"], in_use["errors64"])
    release_memory(device)
    assert torch.cuda.mem_get_info(0)[0] == free
    np.testing.assert_array_equal(run()["errors64"], want["errors64"])
