"""Pair sort around the edges of its tiles (2,048 keys up to 3 * 2^19 keys,
4,096 above) against numpy's stable sort: exact."""
import ctypes

import numpy as np
import pytest
import torch

from cindergs_b200 import _abi
from cindergs_b200.pipeline import radix_sort_u32_pairs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("digit_bits", [8, 4])
@pytest.mark.parametrize("n", [2047, 2048, 2049, 3 * 2**19 - 1, 3 * 2**19, 3 * 2**19 + 1])
def test_pairs_at_tile_edges(gpu_state, n, digit_bits):
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 2**17, n, dtype=np.uint32)
    vals = np.arange(n, dtype=np.uint32)
    dk = torch.from_numpy(keys.view(np.int32).copy()).cuda()
    dv = torch.from_numpy(vals.view(np.int32).copy()).cuda()
    torch.cuda.synchronize()
    radix_sort_u32_pairs(gpu_state, dk.data_ptr(), dv.data_ptr(), n, 17, digit_bits)
    gpu_state.synchronize()
    order = np.argsort(keys, kind="stable")
    np.testing.assert_array_equal(dk.cpu().numpy().view(np.uint32), keys[order])
    np.testing.assert_array_equal(dv.cpu().numpy().view(np.uint32), vals[order])


def test_noalloc_scratch_at_its_largest(gpu_state):
    # its fixed look-back area holds 4,096-key tiles at every size
    lib = _abi.load()
    n = 1 << 20
    keys = np.random.default_rng(7).integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32)
    dk = torch.from_numpy(keys.view(np.int32).copy()).cuda()
    dv = torch.arange(n, dtype=torch.int32, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    rc = lib.cgs_sort_pairs_u32_noalloc(ctypes.c_void_p(dk.data_ptr()),
                                        ctypes.c_void_p(dv.data_ptr()), n, 32, 8, stream)
    assert rc == _abi.CGS_OK
    order = np.argsort(keys, kind="stable")
    np.testing.assert_array_equal(dk.cpu().numpy().view(np.uint32), keys[order])
    np.testing.assert_array_equal(dv.cpu().numpy(), order.astype(np.int32))
