"""Shadow rays three ways: whether anything is in the way, the nearest of few emitters first, and the closest
hit through clear glass. Where a scene's answer does not depend on the way, its frames must not either."""
import numpy as np
import pytest

import mypbr_gb300 as mp

ROOM = """
image_width 60
aspect_ratio 1
max_depth 5
camera lookfrom 0 0 3.9  lookat 0 0 0  vup 0 1 0  vfov 70
material white lambertian 0.7 0.7 0.7
material shiny metal 0.8 0.7 0.6 0.3
material clear dielectric 1.5
quad -2 -2 -4  4 0 0  0 0 8  white
quad -2 2 -4  4 0 0  0 0 8  white
quad -2 -2 -4  4 0 0  0 4 0  white
quad -2 -2 -4  0 4 0  0 0 8  white
quad 2 -2 -4  0 4 0  0 0 8  white
sphere 0.6 -1.2 0.5 0.8 shiny
box -1.4 -2 -1  -0.4 0.4 0  white
box 40 40 40  44 44 44  white
sphere 42 42 42 1 clear
"""


def _lamps(n):
    """n lamps under the ceiling facing down, up (dark from below) and sideways, some behind others."""
    out = []
    for k in range(n):
        out.append(f"material lamp{k} emissive {1 + k % 3} {2 - k % 2} {1 + 0.1 * k}")
        x, z = -1.6 + 0.8 * (k % 5), -3 + 1.5 * (k // 5)
        edges = ["0.5 0 0  0 0 0.5", "0 0 0.5  0.5 0 0", "0 0.5 0  0 0 0.5"][k % 3]
        out.append(f"quad {x} {1.9 - 0.05 * (k % 4)} {z}  {edges}  lamp{k}")
    if n > 2:
        out.append("sphere -1.2 1.2 1 0.2 lamp1")
    return "\n".join(out) + "\n"


# 1 emitter, the largest count tested one by one (15 quads and a sphere), one past it, under a black and a lit sky
@pytest.mark.gpu
@pytest.mark.parametrize("lamps", [1, 2, 15, 16])
@pytest.mark.parametrize("sky", ["background 0 0 0", "background 0.3 0.4 0.5",
                                 "background 0 0 0\nsun elevation 40 azimuth 30 intensity 3 angle 3",
                                 "background 0 0 0\nmaterial haze volume 0.9 0.9 0.9 g 0.4\nfog 0.05 haze"])
def test_emitters_first_is_the_closest_hit(lamps, sky):
    scene = mp.parse_scene(ROOM + _lamps(lamps) + sky + "\n")
    gpu = mp.GpuScene(scene)
    cam = scene.camera
    cam.samples_per_pixel, cam.seed = 8, 5
    frames = []
    # transparent shadows ask for closest hits (the clear sphere is sealed in a box, so nothing shines through it)
    for transparent in (0, 1):
        cam.transparent_shadows = transparent
        for traversal in (0, 1, 2, 3, 4, 5):
            mp.set_launch(gpu, 0, 0, traversal)
            frames.append(cam.render(gpu).radiance)
    assert frames[0].any()  # the scene is lit
    for f in frames[1:]:
        # FP32 path arithmetic is the same in all; a walk whose last bit differs may turn single paths
        off = np.abs(f - frames[0]) > 1e-5 * np.abs(frames[0]) + 1e-7
        assert off.any(axis=2).mean() < 0.002


@pytest.mark.gpu
@pytest.mark.parametrize("rays", [1, 31, 33, 129, 4097])
def test_lanes_take_every_ray(rays):
    """Queues around the sizes of a warp and of the runs its lanes take rays from."""
    scene = mp.parse_scene(ROOM + _lamps(3) + "background 0.2 0.2 0.2\n")
    gpu = mp.GpuScene(scene)
    cam = scene.camera
    cam.image_width, cam.aspect_ratio, cam.samples_per_pixel = 1, 1.0, rays
    out = []
    for traversal in (1, 4):
        mp.set_launch(gpu, 0, 0, traversal)
        out.append(mp.render_ex(cam, gpu))
    assert out[0][2]["extension_rays"] == out[1][2]["extension_rays"]
    assert np.allclose(out[0][0], out[1][0], rtol=1e-5)
