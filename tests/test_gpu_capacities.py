"""Buffers that turn out too small: frames are rendered again with grown ones,
copies of them made again, and what cannot be grown stays refused."""
import numpy as np
import pytest
import torch

from cindergs_b200 import (CameraUniforms, CompositorUniforms, GaussianSceneSoa, GpuPipelineState,
                           _abi, random_scene)
from helpers import assert_stage23_exact, compositor, config0_camera, gpu_buffers, oracle_frame

pytestmark = pytest.mark.gpu


def look(z, w, h):
    return CameraUniforms.from_look_at((0.0, 0.3, z), (0, 0, 0), (0, 1, 0), np.deg2rad(60), w, h, 0.2)


def test_copies_of_two_overflowed_frames():
    """Two frames in a row overflow, each rendered again when the next is
    enqueued, with copies of both begun before: both copies hold the whole
    frames."""
    w, h = 1280, 720
    scene = random_scene(40_000, seed=2, box=1.0)
    scene.covariances_3d[:] *= np.float32(30.0)
    cams = [look(z, w, h) for z in (60.0, 12.0, 3.0)]

    def frame(st, cam):
        st.execute_frame_gpu(scene, None, cam, compositor(w, h, cam, deg=1), force_stage3=True,
                             stage_timings=False)

    ref = GpuPipelineState(0)
    st = GpuPipelineState(0)
    try:
        ref.upload_scene(scene)
        want = []
        for cam in cams[1:]:
            frame(ref, cam)
            want.append(ref.readback_framebuffer_rgba8(w, h))
        st.upload_scene(scene)
        frame(st, cams[0])
        st.synchronize()
        outs, tickets = [np.zeros((h, w, 4), np.uint8) for _ in range(2)], []
        for out, cam in zip(outs, cams[1:]):
            frame(st, cam)
            tickets.append(st.readback_framebuffer_rgba8_async(out))
            torch.cuda.synchronize()  # the next call finds the frame finished
        frame(st, cams[0])
        for t, out, img in zip(tickets, outs, want):
            st.readback_wait(t)
            np.testing.assert_array_equal(out, img)
    finally:
        st.close()
        ref.close()


def test_copy_outlives_its_frames_slot():
    """An overflowed frame's copy is made again before a later frame takes the
    place of the frame's arguments, however many frames follow."""
    w, h = 1280, 720
    scene = random_scene(40_000, seed=2, box=1.0)
    scene.covariances_3d[:] *= np.float32(30.0)
    far, near = look(60.0, w, h), look(3.0, w, h)
    st = GpuPipelineState(0)
    try:
        st.upload_scene(scene)
        st.execute_frame_gpu(scene, None, far, compositor(w, h, far, deg=1), force_stage3=True)
        out = np.zeros((h, w, 4), np.uint8)
        st.execute_frame_gpu(scene, None, near, compositor(w, h, near, deg=1), force_stage3=True,
                             stage_timings=False)
        ticket = st.readback_framebuffer_rgba8_async(out)
        for _ in range(6):
            st.execute_frame_gpu(scene, None, far, compositor(w, h, far, deg=1), force_stage3=True,
                                 stage_timings=False)
        st.readback_wait(ticket)
        st.execute_frame_gpu(scene, None, near, compositor(w, h, near, deg=1), force_stage3=True)
        np.testing.assert_array_equal(out, st.readback_framebuffer_rgba8(w, h))
    finally:
        st.close()


def test_failed_growth_is_not_reused():
    """A frame whose lists do not fit the device budget fails; the same frame
    again fails too instead of reusing what was listed, and renders once the
    budget allows it."""
    w, h = 1280, 720
    scene = random_scene(20_000, seed=4, box=1.0)
    scene.covariances_3d[:] *= np.float32(100.0)
    far, near = look(100.0, w, h), look(2.5, w, h)
    st = GpuPipelineState(0)
    try:
        st.upload_scene(scene)
        comp = compositor(w, h, near, deg=1)
        st.execute_frame_gpu(scene, None, far, compositor(w, h, far, deg=1), write_f32=True)
        st.set_device_budget(st.device_bytes() + (64 << 10))
        for _ in range(3):
            with pytest.raises(_abi.CgsError) as e:
                st.execute_frame_gpu(scene, None, near, comp, write_f32=True)
            assert e.value.code == _abi.CGS_E_OOM
        st.set_device_budget(0)
        t = st.execute_frame_gpu(scene, None, near, comp, write_f32=True)
        o = oracle_frame(scene, near, comp)
        assert t.total_tile_entries == o["entries"]
        assert_stage23_exact(gpu_buffers(st), o)
    finally:
        st.close()


def test_no_view_twice_after_a_smaller_viewport_or_scene():
    """A viewport or scene after a smaller one fits where it fits a new context."""
    def views(st, scene, sizes):
        cams = [config0_camera(*wh) for wh in sizes]
        comps = [CompositorUniforms(*wh) for wh in sizes]
        return st.execute_views(scene, None, cams, comps, st.view_images(comps), use_graph=False)

    st = GpuPipelineState(0)
    try:
        scene = random_scene(60_000, seed=6, box=1.0)
        st.upload_scene(scene)
        st.upload_cages(None)
        assert views(st, scene, [(1280, 720)])["views_rerendered"] == 0
    finally:
        st.close()
    st = GpuPipelineState(0)
    try:
        st.upload_scene(random_scene(10, seed=6, box=1.0))
        st.upload_cages(None)
        views(st, random_scene(10, seed=6, box=1.0), [(16, 16)])
        st.upload_scene(scene)
        st.upload_cages(None)
        assert views(st, scene, [(32, 32), (1280, 720)])["views_rerendered"] == 0
    finally:
        st.close()


@pytest.mark.parametrize("sort", [_abi.SORT_AUTO, _abi.SORT_RADIX, _abi.SORT_TRANSPOSE])
def test_overflow_is_listed_again(sort):
    """Each way to make the lists starts a fresh context with buffers below this
    frame's needs (2^20 entries, max(4 n, 2^16) pairs of a splat and an 8x4-tile
    block): the views are rendered again, and a frame equals the oracle."""
    w, h = 1920, 1080
    scene = random_scene(4000, seed=13)
    scene.covariances_3d[:] = np.array([0.09, 0.0, 0.0, 0.09, 0.0, 0.09], np.float32)
    scene.positions *= np.float32(0.4)
    cam = config0_camera(w, h)
    comp = compositor(w, h, cam, deg=1)
    o = oracle_frame(scene, cam, comp)
    # the splats' tile boxes from the oracle's extents and centres
    ext = o["ext"]
    mu = o["attrs"].reshape(-1, 10)[:, :2]
    ex, ey = (ext & 0xFFFF).astype(np.float32), (ext >> 16).astype(np.float32)
    tiles = [np.clip(np.floor(np.stack([mu[:, k] - e, mu[:, k] + e]) / 16), 0, n - 1).astype(np.int64)
             for k, e, n in ((0, ex, 120), (1, ey, 68))]
    blocks = np.prod([(t[1] >> s) - (t[0] >> s) + 1 for t, s in zip(tiles, (3, 2))], 0)
    assert blocks[ext != 0].sum() > 1 << 16 and o["entries"] > 1 << 20
    st = GpuPipelineState(0)
    try:
        st.upload_scene(scene)
        st.upload_cages(None)
        images = st.view_images([comp])
        assert st.execute_views(scene, None, [cam], [comp], images, use_graph=False,
                                entry_sort=sort)["views_rerendered"] > 0
        st.close()
        st = GpuPipelineState(0)
        st.upload_scene(scene)
        t = st.execute_frame_gpu(scene, None, cam, comp, force_stage3=True, write_f32=True,
                                 entry_sort=sort)
        assert t.total_tile_entries == o["entries"]
        assert_stage23_exact(gpu_buffers(st), o)
        assert np.abs(st.readback_framebuffer_f32(w, h) - o["rgba_f32"]).max() <= 2e-3
    finally:
        st.close()


def test_more_entries_than_a_frame_may_have():
    """More than 2^32 - 2^16 tile entries are refused, however the lists are
    made: 80,000 splats over 65,536 tiles each."""
    w, h, n = 7680, 4320, 80_000
    scene = random_scene(n, seed=3)
    scene.positions[:] = np.random.default_rng(3).uniform(-0.3, 0.3, (n, 3)).astype(np.float32)
    scene.covariances_3d[:] = np.array([4.0, 0.0, 0.0, 4.0, 0.0, 4.0], np.float32)
    scene.opacities[:] = 0.9
    cam = look(4.0, w, h)
    st = GpuPipelineState(0)
    try:
        st.upload_scene(scene)
        with pytest.raises(_abi.CgsError) as e:
            st.execute_frame_gpu(scene, None, cam, compositor(w, h, cam, deg=0), force_stage3=True,
                                 tile_shape=_abi.TILE_8X8)
        assert e.value.code == _abi.CGS_E_CAPACITY
        far = look(60.0, 320, 180)  # the context goes on
        small = compositor(320, 180, far, deg=0)
        assert st.execute_frame_gpu(scene, None, far, small, force_stage3=True).total_tile_entries > 0
    finally:
        st.close()


@pytest.mark.parametrize("sort", [_abi.SORT_RADIX, _abi.SORT_TRANSPOSE, _abi.SORT_AUTO])
def test_graph_of_views_of_different_widths(sort):
    """The pass before a capture may raise the capacities without a re-render
    (entries past 80% of them): the buffers then fit every view's digit width
    when the graph is captured, and its replay equals the views one by one."""
    w, h = 1920, 1080
    scene = random_scene(4000, seed=13)
    scene.covariances_3d[:] = np.array([0.09, 0.0, 0.0, 0.09, 0.0, 0.09], np.float32)
    scene.positions *= np.float32(0.4)
    cam = config0_camera(w, h)
    st = GpuPipelineState(0)
    st.upload_scene(scene)
    all_entries = st.execute_frame_gpu(scene, None, cam, compositor(w, h, cam)).total_tile_entries
    st.close()
    n = int(scene.count * 0.92 * 2**20 / all_entries)
    part = GaussianSceneSoa(scene.positions[:n], scene.covariances_3d[:n], scene.opacities[:n],
                            scene.sh_coeffs[:n])
    sizes = [(w, h), (640, 360), (64, 48)]  # 13, 10 and 4 tile bits
    cams = [config0_camera(*s) for s in sizes]
    comps = [compositor(*s, c, deg=1) for s, c in zip(sizes, cams)]
    st = GpuPipelineState(0)
    try:
        st.upload_scene(part)
        st.upload_cages(None)
        images = st.view_images(comps)
        stats = [st.execute_views(part, None, cams, comps, images, entry_sort=sort) for _ in range(3)]
        assert stats[0]["views_rerendered"] == 0 or sort == _abi.SORT_AUTO
        assert stats[-1]["graph_replayed"] == 1
        torch.cuda.synchronize()
        got = [im.cpu().numpy().view(np.uint8).reshape(s[1], s[0], 4) for im, s in zip(images, sizes)]
        for s, c, q, im in zip(sizes, cams, comps, got):
            t = st.execute_frame_gpu(part, None, c, q, force_stage3=True)
            np.testing.assert_array_equal(im, st.readback_framebuffer_rgba8(*s))
            if s == (w, h):
                assert 0.8 * 2**20 < t.total_tile_entries <= 2**20
    finally:
        st.close()
