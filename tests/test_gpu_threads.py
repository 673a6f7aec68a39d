"""Contexts of two threads launching the same kernels with different amounts of
shared memory: no launch is refused because the other thread's opt-in came
between, and the results are those of one thread alone."""
import ctypes
import threading

import numpy as np
import pytest
import torch

from cindergs_b200 import GpuPipelineState, PolyCageMesh, _abi, radix_sort_u32_pairs

pytestmark = pytest.mark.gpu


def together(*work):
    errors = []

    def guarded(f):
        try:
            f()
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=guarded, args=(f,)) for f in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_field_projection_of_two_cages():
    states = []
    try:
        for level in (1, 3):
            st = GpuPipelineState(0)
            states.append(st)
            st.mvc_cage_upload(PolyCageMesh.icosphere([0, 0, 0], 1.15, level))
            st.mvc_field_create(seed=level)
        pts = torch.rand(64, 3, device="cuda") - 0.5
        want = [st.mvc_field_infer(pts)[0].clone() for st in states]

        def infer(k):
            for _ in range(2000):
                got = states[k].mvc_field_infer(pts)[0]
            assert torch.equal(got, want[k])

        together(lambda: infer(0), lambda: infer(1))
    finally:
        for st in states:
            st.close()


def test_sorts_with_and_without_a_context():
    lib = _abi.load()
    st = GpuPipelineState(0)
    stream = torch.cuda.Stream()
    try:
        big, small = 1_600_000, 300_000  # both in 4,096-key tiles
        keys = torch.randint(0, 2**31 - 1, (big,), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()

        def with_context():
            for _ in range(300):
                k, v = keys.clone(), torch.arange(big, dtype=torch.int32, device="cuda")
                torch.cuda.synchronize()
                radix_sort_u32_pairs(st, k.data_ptr(), v.data_ptr(), big, 32)
            st.synchronize()
            assert torch.equal(k, keys.sort(stable=True).values)

        def without():
            with torch.cuda.stream(stream):
                for _ in range(2000):
                    k, v = keys[:small].clone(), torch.arange(small, dtype=torch.int32, device="cuda")
                    rc = lib.cgs_sort_pairs_u32_noalloc(
                        ctypes.c_void_p(k.data_ptr()), ctypes.c_void_p(v.data_ptr()), small, 32, 8,
                        ctypes.c_void_p(stream.cuda_stream))
                    assert rc == _abi.CGS_OK
                stream.synchronize()
                np.testing.assert_array_equal(k.cpu(), keys[:small].sort(stable=True).values.cpu())

        together(with_context, without)
    finally:
        st.close()
