"""Lamps at the same distance along a ray as another surface: overlapping or doubled lamps, lamps back to back, lamps
flush with a ceiling. What a shadow ray brings there is what its closest hit emits, by the order of that walk's tests,
however the shadow rays are traced."""
import numpy as np
import pytest

import mypbr_gb300 as mp
import oracle as orc
from conftest import scene_path

ROOM = """
image_width 48
aspect_ratio 1
max_depth 4
background 0 0 0
camera lookfrom 0 0 3.9  lookat 0 0 0  vup 0 1 0  vfov 70
material white lambertian 0.7 0.7 0.7
material shiny metal 0.8 0.7 0.6 0.3
material clear dielectric 1.5
material red emissive 5 1 1
material blue emissive 1 1 5
quad -2 -2 -4  4 0 0  0 0 8  white
quad -2 2 -4  4 0 0  0 0 8  white
quad -2 -2 -4  4 0 0  0 4 0  white
quad -2 -2 -4  0 4 0  0 0 8  white
quad 2 -2 -4  0 4 0  0 0 8  white
sphere 0.6 -1.2 0.5 0.8 shiny
box -1.4 -2 -1  -0.4 -0.4 0  white
box 40 40 40  44 44 44  white
sphere 42 42 42 1 clear
"""
# edges in this order face down (-y)
LAMPS = {
    "overlapping": "quad -1 1.5 -1  2 0 0  0 0 0.6  red\nquad -0.3 1.5 -1.7  0.6 0 0  0 0 2  blue",
    "doubled": "quad -1 1.5 -1  2 0 0  0 0 1  red\nquad -1 1.5 -1  2 0 0  0 0 1  red",
    "back_to_back": "quad -1 1.5 -1  0 0 1  2 0 0  blue\nquad -1 1.5 -1  2 0 0  0 0 1  red",
    "flush_ceiling": "quad -1 2 -1  2 0 0  0 0 1  red",
    "flush_box": "box -1 1 -1  1 1.5 0  white\nquad -0.8 1 -0.8  1.6 0 0  0 0 0.6  red",
    "doubled_sphere": "sphere 0 1.2 0 0.3 red\nsphere 0 1.2 0 0.3 blue",
    "turned": "quad -1 1.1 -1  1.6 0.5 0.1  0.1 0.2 1.1  red\nquad -1 1.1 -1  1.6 0.5 0.1  0.1 0.2 1.1  blue",
}
# enough spheres that they fill most leaves (the walks then differ), out of sight
SPHERES = "".join(f"sphere {50 + 3 * k} 50 50 1 white\n" for k in range(40))


def _scene(lamps, spheres=False, extra=""):
    return mp.parse_scene(ROOM + LAMPS[lamps] + "\n" + (SPHERES if spheres else "") + extra)


def _same_light(gpu, cam, traversals=(0, 2, 3, 4, 5)):
    for traversal in traversals:
        mp.set_launch(gpu, 0, 0, traversal)
        for seed in (3, 4):
            cam.seed = seed
            # transparent shadows ask for closest hits; the clear sphere is sealed in a box, so nothing shines through it
            cam.transparent_shadows = 1
            want = cam.render(gpu).radiance
            cam.transparent_shadows = 0
            got = cam.render(gpu).radiance
            assert want.any()
            # the same paths, lit by the same surfaces: FP32 sums of a few terms, whose last bits may differ
            np.testing.assert_allclose(got, want, rtol=1e-5, atol=1e-7, err_msg=f"traversal {traversal}")


@pytest.mark.gpu
@pytest.mark.parametrize("spheres", [False, True])
@pytest.mark.parametrize("lamps", LAMPS)
def test_ties_are_settled_by_the_closest_hit(lamps, spheres):
    scene = _scene(lamps, spheres)
    cam = scene.camera
    cam.samples_per_pixel = 2
    _same_light(mp.GpuScene(scene), cam)


@pytest.mark.gpu
def test_ties_with_voxels_and_with_the_ground():
    """A lamp lying on the ground plane, under a voxel model's lower face."""
    scene = mp.parse_scene(ROOM + f"ground height -3 white\nvox {scene_path('voxels_default.vox')} scale 0.1 translate 0 1 0\n"
                           "quad -1 1 -1  2 0 0  0 0 2  red\nquad -9 -3 -9  0 0 18  18 0 0  blue\n")
    cam = scene.camera
    cam.samples_per_pixel = 4
    _same_light(mp.GpuScene(scene), cam)


@pytest.mark.gpu
@pytest.mark.parametrize("lamps", ["overlapping", "doubled", "turned"])
def test_tied_lamps_light_the_room_as_the_oracle_says(lamps):
    scene = _scene(lamps)
    cam = scene.camera
    cam.image_width, cam.samples_per_pixel, cam.max_depth = 24, 256, 3
    rad, var, _ = mp.render_ex(cam, mp.GpuScene(scene))
    ref_rad, ref_var, _ = orc.OracleScene(scene).render(cam, threads=0)
    # two Monte Carlo estimates: channel means within 4 sigma of their combined error
    n = rad.shape[0] * rad.shape[1]
    sigma = np.sqrt(var.sum(axis=(0, 1)) + ref_var.sum(axis=(0, 1))) / n
    z = (rad.mean(axis=(0, 1)) - ref_rad.mean(axis=(0, 1))) / sigma
    assert np.all(np.abs(z) < 4), z


# (lamps, leaf references) measured faster one way or the other
@pytest.mark.parametrize("lamps,refs,few", [(1, 6, 1), (3, 8, 1), (4, 9, 0), (16, 21, 0), (12, 41, 0), (8, 109, 1), (12, 401, 1),
                                            (16, 405, 0), (16, 1557, 1), (16, 300016, 1), (17, 300017, 0)])
def test_which_scenes_look_for_emitters_first(lamps, refs, few):
    assert mp.lib().mypbr_gpu_test_few_emitters(lamps, refs) == few


# 1 to 16 lamps, with enough other surfaces that they are tested one by one, under skies that shine and do not
@pytest.mark.gpu
@pytest.mark.parametrize("sky", ["background 0 0 0", "background 0.3 0.4 0.5",
                                 "background 0 0 0\nsun elevation 40 azimuth 30 intensity 3 angle 3"])
@pytest.mark.parametrize("lamps", [1, 2, 5, 16])
def test_every_path_has_the_light_of_its_closest_hit(lamps, sky):
    rng = np.random.default_rng(lamps)
    text = ROOM.replace("background 0 0 0\n", "")
    for k in range(lamps):  # under the ceiling, facing down, up and sideways, some behind others
        edges = ["0.5 0 0  0 0 0.5", "0 0 0.5  0.5 0 0", "0 0.5 0  0 0 0.5"][k % 3]
        text += f"quad {-1.6 + 0.8 * (k % 5)} {1.9 - 0.05 * (k % 4)} {-3 + 1.5 * (k // 5)}  {edges}  {['red', 'blue'][k % 2]}\n"
    for x, y, z, r in zip(*rng.uniform(-1.8, 1.8, (3, 170)), rng.uniform(0.02, 0.1, 170)):
        text += f"box {x - r} {y - r} {z - r}  {x + r} {y + r} {z + r}  white\n"
    scene = mp.parse_scene(text + sky + "\n")
    assert mp.lib().mypbr_gpu_test_few_emitters(lamps, 19 + 6 * 170 + lamps) == 1
    cam = scene.camera
    cam.samples_per_pixel = 2
    _same_light(mp.GpuScene(scene), cam)
