"""The radix sort where its tile size changes (512 keys up to 303,104 pairs,
2560 beyond) and at the edges of both tiles: the stable order, to the bit."""
import numpy as np
import pytest

import ggb200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("noalloc", [False, True])
@pytest.mark.parametrize("n", [2, 511, 512, 513, 1025, 303103, 303104, 303105, 305665])
def test_stable_order_at_tile_edges(n, noalloc):
    import torch
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 1 << 62, size=n, dtype=np.uint64)
    keys[::3] &= np.uint64(0xFF000000FF)      # many equal keys
    dk = torch.from_numpy(keys.view(np.int64).copy()).cuda()
    dv = torch.arange(n, dtype=torch.int32, device="cuda")
    (ggb200.radix_sort_pairs_noalloc if noalloc else ggb200.radix_sort_pairs)(dk, dv, n, 63)
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(dv.cpu().numpy(), order)
    assert np.array_equal(dk.cpu().numpy().view(np.uint64), keys[order])
