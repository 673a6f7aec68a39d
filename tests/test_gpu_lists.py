"""Stage 3 through screen-block lists (CGS_SORT_AUTO): every Stage 3 integer
bit-exact against the oracle at the edges of the screen blocks (8x4 tiles),
of the pairing tiles (1,024 slots), of the groups of 32 pairs and of the pair
sort's digits, with pair buffers that overflow, and equal to the entry sorts'."""
import numpy as np
import pytest

from cindergs_b200 import GpuPipelineState, _abi, random_scene

from helpers import assert_stage23_exact, compositor, config0_camera, gpu_buffers, oracle_frame

pytestmark = pytest.mark.gpu


def run(st, scene, w, h, tile_shape=0, entry_sort=0):
    cam = config0_camera(w, h)
    comp = compositor(w, h, cam, deg=1)
    t = st.execute_frame_gpu(scene, None, cam, comp, force_stage3=True, write_f32=True,
                             tile_shape=tile_shape, entry_sort=entry_sort)
    g = gpu_buffers(st, key64=t.used_64bit_keys)
    g["f32"] = st.readback_framebuffer_f32(w, h)
    return t, g, cam, comp


@pytest.mark.parametrize("n", [1, 33, 1025])
@pytest.mark.parametrize("wh", [(1, 1), (16, 16), (127, 63), (128, 64), (129, 65)])
def test_block_edges(n, wh):
    st = GpuPipelineState(0)
    try:
        scene = random_scene(n, seed=n)
        st.upload_scene(scene)
        t, g, cam, comp = run(st, scene, *wh)
        o = oracle_frame(scene, cam, comp)
        assert t.total_tile_entries == o["entries"]
        assert_stage23_exact(g, o)
        assert np.abs(g["f32"] - o["rgba_f32"]).max() <= 2e-3
    finally:
        st.close()


# faint splats: lists of thousands of entries that no pixel saturates before,
# so the compositor goes past the 1,024 written ones (one group and four
# groups per chunk, blocks of 64, 256 and 512 threads)
@pytest.mark.parametrize("n,wh,shape,grow", [(6_000, (64, 48), _abi.TILE_16X16, 40.0),
                                             (60_000, (200, 130), _abi.TILE_32X16, 4.0),
                                             (60_000, (100, 70), _abi.TILE_8X8, 20.0),
                                             (90_000, (300, 200), _abi.TILE_16X16, 4.0)])
def test_beyond_the_written_entries(n, wh, shape, grow):
    st = GpuPipelineState(0)
    try:
        scene = random_scene(n, seed=9)
        scene.covariances_3d[:] *= np.float32(grow)
        scene.opacities[:] = np.random.default_rng(1).uniform(0.0042, 0.008, n).astype(np.float32)
        st.upload_scene(scene)
        t, g, cam, comp = run(st, scene, *wh, tile_shape=shape)
        o = oracle_frame(scene, cam, comp, tile=_abi.TILE_SHAPES[shape])
        assert int((g["ranges"][1::2] - g["ranges"][0::2]).max()) > 2048
        assert_stage23_exact(g, o)
        assert np.abs(g["f32"] - o["rgba_f32"]).max() <= 2e-3
        _, r, _, _ = run(st, scene, *wh, tile_shape=shape, entry_sort=_abi.SORT_RADIX)
        np.testing.assert_array_equal(g["f32"], r["f32"])
    finally:
        st.close()


# (n, viewport, tile shape, covariance scale): more than 2^18 pairs (four groups
# per chunk), two pair-sort passes (460 and 1,020 blocks), splats over whole
# screens (the pair buffers overflow on the first frame), 64-bit keys
@pytest.mark.parametrize("n,wh,shape,grow", [(120_000, (1920, 1080), _abi.TILE_16X16, 1.0),
                                             (20_000, (1280, 720), _abi.TILE_8X8, 1.0),
                                             (3_000, (1920, 1080), _abi.TILE_8X8, 4.0),
                                             (2_000, (1920, 1080), _abi.TILE_16X16, 400.0),
                                             (2_000, (1283, 717), _abi.TILE_32X16, 100.0),
                                             (1_500, (4100, 4099), _abi.TILE_16X16, 30.0)])
def test_lists_equal_oracle_and_entry_sorts(n, wh, shape, grow):
    st = GpuPipelineState(0)
    try:
        scene = random_scene(n, seed=5)
        scene.covariances_3d[:] *= np.float32(grow)
        st.upload_scene(scene)
        t, g, cam, comp = run(st, scene, *wh, tile_shape=shape)
        o = oracle_frame(scene, cam, comp, tile=_abi.TILE_SHAPES[shape])
        assert t.total_tile_entries == o["entries"]
        assert_stage23_exact(g, o, key64=t.used_64bit_keys)
        assert np.abs(g["f32"] - o["rgba_f32"]).max() <= 2e-3
        _, r, _, _ = run(st, scene, *wh, tile_shape=shape, entry_sort=_abi.SORT_RADIX)
        for k in ("offsets", "sorted_keys", "sorted_ids", "ranges", "f32"):
            np.testing.assert_array_equal(g[k], r[k], err_msg=k)
    finally:
        st.close()
