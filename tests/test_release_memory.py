"""Device memory that calls without a scene handle keep, given back on request."""
import ctypes

import numpy as np
import pytest
import torch

import mypbr_gb300 as mp
from conftest import scene_path


def test_release_without_a_gpu():
    if torch.cuda.is_available():
        pytest.skip("a GPU is present")
    mp.release_memory()


@pytest.mark.gpu
def test_denoise_memory_is_given_back():
    h, w = 1000, 1000
    plane = np.ones((h, w, 3))

    def denoise():
        out = np.empty_like(plane)
        mp.denoise(plane, plane, plane, np.ones((h, w)), w, h, out)
        return out

    want = denoise()
    mp.release_memory()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    assert np.array_equal(denoise(), want)
    # 148 bytes a pixel are kept
    assert torch.cuda.mem_get_info()[0] <= free - 140 * h * w
    mp.release_memory()
    assert torch.cuda.mem_get_info()[0] >= free - (2 << 20)
    assert np.array_equal(denoise(), want)


@pytest.mark.gpu
def test_a_very_large_frame_is_not_kept():
    """A narrow band of an image whose planes take 1.5 GB: the host render leaves no more memory taken than the same
    render into device memory does."""
    scene = mp.load_scene(scene_path("cornell_c1.scene"))
    gpu = mp.GpuScene(scene)
    cam = scene.camera
    cam.image_width, cam.aspect_ratio, cam.samples_per_pixel, cam.max_depth = 8192, 1.0, 1, 1
    cam.first_row, cam.row_count = 4096, 1
    c, o = cam.structs()
    plane = torch.empty(cam.height(), 8192, 3, dtype=torch.float64, device="cuda:0")
    torch.cuda.synchronize()
    mp.check(mp.lib().mypbr_gpu_render_device(gpu.handle, ctypes.byref(c), ctypes.byref(o),
                                              ctypes.c_void_p(plane.data_ptr()), None, None, None, None, None))
    free = torch.cuda.mem_get_info()[0]
    frame = cam.render(gpu)
    assert torch.cuda.mem_get_info()[0] >= free - (64 << 20)
    assert np.array_equal(frame.radiance[4096], plane[4096].cpu().numpy())
