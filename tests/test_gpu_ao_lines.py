"""The AO march by line maxima, bit-exact with the oracle: frames whose inner
pixels (every tap inside) are none, one and a few; a frame size change in one
context (the tap tables follow it); and a close view whose steep depths end
pixels early (black)."""
import numpy as np
import pytest

from helpers import Pair, assert_bitexact, options
from polyred_gb300 import procedural, scene as sc

pytestmark = pytest.mark.gpu


def _scene(W, H, near_by):
    m = sc.BlinnPhong(diffuse=sc.color_from_value(0.8, 0.8, 0.8), specular=sc.color_from_value(0.5, 0.5, 0.5),
                      shininess=16, ambient_occlusion=True)
    rng = np.random.default_rng(7)
    s = sc.Scene(sc.Geometry(procedural.ground_plane(30.0, -1.0, material_id=0), m).translate(0.0, 0.0, -14.0))
    for _ in range(30):
        r = float(rng.uniform(0.2, 1.2))
        s.add(sc.Geometry(procedural.uv_sphere(24, 12, r), m).translate(float(rng.uniform(-6, 6)), r - 1.0,
                                                                        float(rng.uniform(-9, 2))))
    s.add(sc.Point(position=(4, 6, 3)), sc.Ambient(intensity=0.3))
    eye, target = ((0.3, -0.2, 3.4), (0.0, -0.6, 0.0)) if near_by else ((2.0, 2.0, 6.0), (0, -0.5, -2))
    cam = sc.Perspective(position=eye, target=target, up=(0, 1, 0), fov=60, aspect=W / H, near=0.1, far=100)
    return s, cam


@pytest.mark.parametrize("near_by", [False, True])
@pytest.mark.parametrize("W,H", [(200, 200), (201, 201), (239, 210), (333, 204)])
def test_inner_pixels(device, W, H, near_by):
    s, cam = _scene(W, H, near_by)
    p = Pair(device, options(s, cam, W, H))
    gpu, cpu = p.frame()
    assert_bitexact(gpu, cpu)
    assert p.stats["n_ao_pixels"] > W * H // 3
    if near_by:
        lit = gpu["tri_id"] != 0xFFFFFFFF
        assert (gpu["rgba"][lit][:, :3].max(1) == 0).sum() > 100
