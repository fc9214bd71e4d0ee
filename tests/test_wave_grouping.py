"""The wave's bookkeeping: paths queued, classified, shaded and summed into the film must give the same
frame however the passes are grouped into waves, at sizes around the tiles of the kernels that do it
(8 entries a thread and 2048 a block in the classification, 1 to 32 lanes a pixel in the film sums)."""
import os

import numpy as np
import pytest

import mypbr_gb300 as mp

SCENES = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "scenes")


def _render(scene, gpu, width, height, spp, per_wave, first_row=0, rows=0):
    cam = mp.Camera(*scene.camera.structs())
    cam.image_width, cam.aspect_ratio = width, width / (height + 0.5)
    cam.samples_per_pixel, cam.samples_per_wave = spp, per_wave
    cam.max_depth, cam.collect_features, cam.seed = 6, 1, 11
    cam.first_row, cam.row_count = first_row, rows
    f = cam.render(gpu)
    return [f.radiance, f.albedo, f.normal, f.variance]


# pixels x passes: a single path, one short of and past a thread's 8 entries, past a block's 2048, more
# passes than lanes, and a film larger than one round of the summing kernel
@pytest.mark.gpu
@pytest.mark.parametrize("width,height,spp,per_wave", [
    (1, 1, 1, 1), (7, 1, 1, 1), (3, 3, 5, 2), (17, 1, 33, 32), (31, 33, 4, 3), (23, 89, 7, 4), (640, 401, 3, 1)])
@pytest.mark.parametrize("name", ["materials", "fog_box"])
def test_waves_do_not_change_the_frame(name, width, height, spp, per_wave):
    scene = mp.load_scene(os.path.join(SCENES, name + ".scene"))
    gpu = mp.GpuScene(scene)
    whole = _render(scene, gpu, width, height, spp, spp)
    parts = _render(scene, gpu, width, height, spp, per_wave)
    # every path is the same; only the order of spp FP64 additions differs: spp units in the last place of
    # the sums (2^-53 each), and for the variance of its two cancelling terms
    tol = 4 * spp * 2.0 ** -53
    for a, b in zip(whole[:3], parts[:3]):
        assert np.all(np.abs(a - b) <= tol * np.abs(a) + 1e-300 + tol)
    second = whole[3] * max(spp - 1, 1) + (whole[0] @ np.array([0.2126, 0.7152, 0.0722])) ** 2
    assert np.all(np.abs(whole[3] - parts[3]) <= 4 * tol * second + 1e-300)


@pytest.mark.gpu
@pytest.mark.parametrize("first_row,rows", [(0, 1), (5, 7), (20, 13)])
def test_a_band_holds_the_frame_s_rows(first_row, rows):
    scene = mp.load_scene(os.path.join(SCENES, "materials.scene"))
    gpu = mp.GpuScene(scene)
    whole = _render(scene, gpu, 41, 33, 6, 6)
    band = _render(scene, gpu, 41, 33, 6, 4, first_row, rows)
    tol = 24 * 2.0 ** -53
    for a, b in zip(whole[:3], band[:3]):
        cut = a[first_row:first_row + rows]
        assert np.all(np.abs(cut - b[first_row:first_row + rows]) <= tol * np.abs(cut) + tol)
        assert not b[:first_row].any() and not b[first_row + rows:].any()


# The sum of a pixel's passes against the passes rendered one at a time (one slot a pixel, no lanes to join)
@pytest.mark.gpu
@pytest.mark.parametrize("spp", [2, 5, 31, 64])
def test_film_sums_the_passes(spp):
    scene = mp.load_scene(os.path.join(SCENES, "materials.scene"))
    gpu = mp.GpuScene(scene)
    got = _render(scene, gpu, 9, 7, spp, spp)[0]
    one = _render(scene, gpu, 9, 7, spp, 1)[0]
    assert np.all(np.abs(got - one) <= 2 * spp * 2.0 ** -53 * (np.abs(one) + 1))
