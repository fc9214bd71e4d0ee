"""What a kernel's own check finds is reported by the call it ran in, not by a later one."""
import ctypes

import pytest
import torch

import mypbr_gb300 as mp
from conftest import scene_path


@pytest.mark.gpu
@pytest.mark.parametrize("stats", [False, True])
@pytest.mark.parametrize("null", [False, True])
@pytest.mark.parametrize("code,status", [(1, 10), (2, 10), (3, 4)])
def test_device_render_reports_its_own_error(code, status, null, stats):
    scene = mp.load_scene(scene_path("cornell_c1.scene"))
    gpu = mp.GpuScene(scene)
    cam = scene.camera
    cam.image_width, cam.samples_per_pixel, cam.max_depth = 16, 1, 2
    c, o = cam.structs()
    plane = torch.zeros(cam.height(), 16, 3, dtype=torch.float64, device="cuda:0")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()

    def render():
        st = mp.RenderStatsStruct()
        return mp.lib().mypbr_gpu_render_device(gpu.handle, ctypes.byref(c), ctypes.byref(o),
                                                ctypes.c_void_p(plane.data_ptr()), None, None, None,
                                                ctypes.c_void_p(0 if null else stream.cuda_stream),
                                                ctypes.byref(st) if stats else None)

    mp.check(mp.lib().mypbr_gpu_test_device_error(gpu.handle, code))
    assert render() == status
    assert render() == 0


@pytest.mark.gpu
def test_every_handle_has_an_error_word_of_its_own():
    scene = mp.load_scene(scene_path("cornell_c1.scene"))
    cam = scene.camera
    cam.image_width, cam.samples_per_pixel, cam.max_depth = 16, 1, 2
    gpus = [mp.GpuScene(scene) for _ in range(3)]
    mp.check(mp.lib().mypbr_gpu_test_device_error(gpus[1].handle, 2))
    cam.render(gpus[0])
    cam.render(gpus[2])
    gpus[1].close()  # its error goes with it
    gpus[1] = mp.GpuScene(scene)
    for gpu in gpus:
        cam.render(gpu)
    mp.release_memory()  # handles are alive: their words stay
    mp.check(mp.lib().mypbr_gpu_test_device_error(gpus[0].handle, 2))
    with pytest.raises(Exception):
        cam.render(gpus[0])
    cam.render(gpus[0])
