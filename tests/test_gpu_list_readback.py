"""Reading the tile lists back costs what its bytes cost, not a pass over every
entry on the host: the ranges (8 bytes a tile) and the offsets (4 bytes a
splat) of a frame with millions of entries take a fraction of the entries
themselves."""
import time

import numpy as np
import pytest

from cindergs_b200 import GpuPipelineState, _abi, random_scene
from helpers import compositor, config0_camera

pytestmark = pytest.mark.gpu


def test_small_buffers_read_fast():
    w, h = 1920, 1080
    scene = random_scene(400_000, seed=1, box=1.0)
    cam = config0_camera(w, h)
    st = GpuPipelineState(0)
    try:
        st.upload_scene(scene)
        t = st.execute_frame_gpu(scene, None, cam, compositor(w, h, cam), force_stage3=True)
        assert t.total_tile_entries > 5_000_000

        def fastest(which):
            times = []
            for _ in range(5):
                t0 = time.perf_counter()
                st.read_buffer(which, np.uint32)
                times.append(time.perf_counter() - t0)
            return min(times)

        ids = fastest(_abi.BUF_SORTED_IDS)
        assert fastest(_abi.BUF_TILE_RANGES) < 0.1 * ids
        assert fastest(_abi.BUF_TILE_OFFSETS) < 0.5 * ids
    finally:
        st.close()
