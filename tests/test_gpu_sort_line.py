"""Sorts of device arrays around the size from which they take larger tiles
(5 * 2^17 pairs), against numpy's stable sort: exact."""
import numpy as np
import pytest
import torch

from cindergs_b200.pipeline import radix_sort_u32_pairs, radix_sort_u64_pairs

pytestmark = pytest.mark.gpu
LINE = 5 * 2**17


def device(a):
    return torch.from_numpy(a.view(np.int32).copy()).cuda()


@pytest.mark.parametrize("spread", [2**32, 2**9, 1])  # equal digits take another course per warp
@pytest.mark.parametrize("n", [LINE - 1, LINE, LINE + 1])
def test_pairs(gpu_state, n, spread):
    keys = np.random.default_rng(n).integers(0, spread, n, dtype=np.uint64).astype(np.uint32)
    dk, dv = device(keys), device(np.arange(n, dtype=np.uint32))
    torch.cuda.synchronize()
    radix_sort_u32_pairs(gpu_state, dk.data_ptr(), dv.data_ptr(), n, 32)
    gpu_state.synchronize()
    order = np.argsort(keys, kind="stable")
    np.testing.assert_array_equal(dk.cpu().numpy().view(np.uint32), keys[order])
    np.testing.assert_array_equal(dv.cpu().numpy(), order)


@pytest.mark.parametrize("n", [LINE, LINE + 1])
def test_two_word_keys(gpu_state, n):
    rng = np.random.default_rng(n)
    tiles = rng.integers(0, 2**13, n, dtype=np.uint32)
    depths = rng.integers(0, 2**20, n, dtype=np.uint32)
    dt, dd, di = device(tiles), device(depths), device(np.arange(n, dtype=np.uint32))
    torch.cuda.synchronize()
    radix_sort_u64_pairs(gpu_state, dt.data_ptr(), dd.data_ptr(), di.data_ptr(), n, 13)
    gpu_state.synchronize()
    order = np.lexsort((depths, tiles))
    np.testing.assert_array_equal(dt.cpu().numpy().view(np.uint32), tiles[order])
    np.testing.assert_array_equal(dd.cpu().numpy().view(np.uint32), depths[order])
    np.testing.assert_array_equal(di.cpu().numpy(), order)
