"""Viewports of so many tiles that a block composites several: ragged sizes just
above the line of each tile shape, most tiles empty, some with lists past one
batch, against the oracle's frame; and the background of empty tiles against a
viewport of few tiles, for backgrounds outside [0, 1] too."""
import numpy as np
import pytest

from cindergs_b200 import GpuPipelineState, _abi, random_scene
from helpers import compositor, config0_camera, oracle_frame

pytestmark = pytest.mark.gpu


# 64 x resident blocks (592, 2,368, 296 on 148 SMs): 37,888, 151,552 and 18,944 tiles
@pytest.mark.parametrize("wh,shape", [((6151, 1607), _abi.TILE_16X16), ((4999, 1951), _abi.TILE_8X8),
                                      ((4993, 1953), _abi.TILE_32X16)])
@pytest.mark.parametrize("sort", [_abi.SORT_AUTO, _abi.SORT_RADIX])
def test_image(wh, shape, sort):
    scene = random_scene(1500, seed=12)
    scene.positions *= np.float32(0.3)
    cam = config0_camera(*wh)
    comp = compositor(*wh, cam, deg=1)
    st = GpuPipelineState(0)
    try:
        st.upload_scene(scene)
        t = st.execute_frame_gpu(scene, None, cam, comp, force_stage3=True, write_f32=True,
                                 tile_shape=shape, entry_sort=sort)
        img = st.readback_framebuffer_f32(*wh)
        ranges = st.read_buffer(_abi.BUF_TILE_RANGES, np.uint32).reshape(-1, 2)
        bytes8 = st.readback_framebuffer_rgba8(*wh)
    finally:
        st.close()
    o = oracle_frame(scene, cam, comp, tile=_abi.TILE_SHAPES[shape])
    assert t.total_tile_entries == o["entries"]
    count = ranges[:, 1] - ranges[:, 0]
    assert (count == 0).mean() > 0.3 and count.max() > 128  # one batch
    assert np.abs(img - o["rgba_f32"]).max() <= 2e-3
    np.testing.assert_array_equal(bytes8, np.clip(np.rint(img * np.float32(255)), 0, 255).astype(np.uint8))


@pytest.mark.parametrize("bg", [(0.02, 0.03, 0.05, 1.0), (-0.5, 2.0, 0.5, 0.25), (0.0, 1.0, 0.499, -3.0),
                                (float("nan"), float("inf"), 0.1, 7.0)])
def test_background(bg):
    scene = random_scene(1, seed=1)
    scene.positions[:] = (0, 0, 50)  # behind the camera
    st = GpuPipelineState(0)
    try:
        st.upload_scene(scene)
        for w, h in ((33, 17), (6151, 1607)):
            cam = config0_camera(w, h)
            st.execute_frame_gpu(scene, None, cam, compositor(w, h, cam, bg=bg), write_f32=True)
            want = np.array([*np.nan_to_num(np.clip(np.float32(bg[:3]), 0, 1)), bg[3]], np.float32)
            np.testing.assert_array_equal(st.readback_framebuffer_f32(w, h),
                                          np.broadcast_to(want, (h, w, 4)))
            w8 = np.clip(np.rint(want * np.float32(255)), 0, 255).astype(np.uint8)
            np.testing.assert_array_equal(st.readback_framebuffer_rgba8(w, h),
                                          np.broadcast_to(w8, (h, w, 4)))
    finally:
        st.close()
