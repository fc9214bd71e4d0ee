"""Renders given to the legacy stream (NULL) run after everything that stream orders itself behind: its own work and
that of every blocking stream, whatever thread queued it."""
import ctypes

import pytest
import torch

import mypbr_gb300 as mp
from conftest import scene_path

CYCLES = 100_000_000  # about 50 ms


@pytest.fixture
def blocking_stream():
    handle = ctypes.c_void_p()
    rt = torch.cuda.cudart()
    assert int(rt.cudaStreamCreate(ctypes.addressof(handle))) == 0
    yield torch.cuda.ExternalStream(handle.value)
    torch.cuda.synchronize()
    rt.cudaStreamDestroy(handle.value)


@pytest.mark.gpu
@pytest.mark.parametrize("null", [0, 1])  # NULL and cudaStreamLegacy
@pytest.mark.parametrize("where", ["legacy", "blocking"])
def test_a_render_on_the_legacy_stream_waits_for(where, null, blocking_stream):
    scene = mp.load_scene(scene_path("cornell_c1.scene"))
    gpu = mp.GpuScene(scene)
    cam = scene.camera
    cam.image_width, cam.samples_per_pixel, cam.max_depth = 32, 1, 4
    c, o = cam.structs()
    plane = torch.zeros(cam.height(), 32, 3, dtype=torch.float64, device="cuda:0")

    def render():
        mp.check(mp.lib().mypbr_gpu_render_device(gpu.handle, ctypes.byref(c), ctypes.byref(o),
                                                  ctypes.c_void_p(plane.data_ptr()), None, None, None,
                                                  ctypes.c_void_p(null), None))

    render()
    torch.cuda.synchronize()
    want = plane.clone()
    torch.cuda.synchronize()
    stream = blocking_stream if where == "blocking" else torch.cuda.default_stream()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(CYCLES)
        plane.fill_(7.0)  # before the render, by the legacy stream's order
    render()
    torch.cuda.synchronize()
    assert torch.equal(plane, want)
