"""Buffers that turn out too small: frames are rendered again with grown ones,
copies of them made again, and what cannot be grown stays refused."""
import numpy as np
import pytest
import torch

from cindergs_b200 import CameraUniforms, CompositorUniforms, GpuPipelineState, _abi, random_scene
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
