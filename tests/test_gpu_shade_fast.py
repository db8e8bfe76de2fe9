"""Shading by certified float32 lighting (frames that ask for colours, ids and
depths alone), bit-exact with the oracle: exponents at and past the ends of
its range, flat and smooth normals under uneven scales, an ambient term that
is exactly a half, lights of both kinds, far, close to a surface, of negative
and zero intensity, many at once, none casting, and triangles from pixel size
to the whole frame. The same frame with every fragment output gives the same
colours."""
import numpy as np
import pytest

from helpers import ALL_OUTPUTS, Pair, assert_bitexact, options
from polyred_gb300 import procedural, scene as sc

pytestmark = pytest.mark.gpu
IMAGE = ("rgba", "tri_id", "depth")
W, H = 211, 147


def _scene(shininess, lights, ambient, seed):
    rng = np.random.default_rng(seed)
    s = sc.Scene()
    for k in range(24):
        m = sc.BlinnPhong(diffuse=tuple(int(v) for v in rng.integers(0, 256, 4)), specular=tuple(int(v) for v in rng.integers(0, 256, 4)),
                          texture=tuple(int(v) for v in rng.choice([0, 1, 128, 255], 4)), shininess=shininess,
                          flat_shading=bool(k % 3 == 0), receive_shadow=bool(k % 2))
        g = sc.Geometry(procedural.uv_sphere(int(rng.integers(4, 40)), int(rng.integers(3, 20)), 1.0), m)
        g.scale(*(float(v) for v in rng.uniform(0.1, 1.3, 3))).translate(*(float(v) for v in rng.uniform(-3, 3, 3)))
        s.add(g)
    s.add(sc.Geometry(procedural.ground_plane(30.0, -3.0, material_id=0), m).translate(0.0, 0.0, -10.0))
    for l in lights:
        s.add(l)
    for a in ambient:
        s.add(sc.Ambient(intensity=a))
    cam = sc.Perspective(position=(0.3, 0.8, 7.0), target=(0, 0, 0), up=(0, 1, 0), fov=55, aspect=W / H, near=0.1, far=100)
    return s, cam


LIGHTS = {
    "point": [sc.Point(position=(4, 6, 3), intensity=3.0, cast_shadow=True)],
    "near": [sc.Point(position=(0.5, 0.2, 0.4), intensity=0.4), sc.Point(position=(0, 0, 0), intensity=-0.2)],
    "directional": lambda: [sc.Directional(direction=(-1, -1, -0.5), intensity=0.7), sc.Directional(direction=(0, 1, 0), intensity=0.0)],
    "many": [sc.Point(position=(8 * np.cos(a), 3, 8 * np.sin(a)), intensity=0.5, color=(255, 200, 40, 255)) for a in range(16)],
}


@pytest.mark.parametrize("lights", sorted(LIGHTS))
@pytest.mark.parametrize("shininess,ambient", [(1.0, (0.1,)), (32.0, (0.1, 0.5)), (1024.0, ()), (0.5, (0.25,)), (2000.0, (0.1,)),
                                               (7.3, (-0.1, 0.3))])
def test_image_frames(device, lights, shininess, ambient):
    ls = LIGHTS[lights]
    s, cam = _scene(shininess, ls() if callable(ls) else ls, ambient, seed=hash((len(lights), shininess)) % 1000)
    shadow = lights == "point"
    o = options(s, cam, W, H, shadow_map=shadow)
    fast, cpu = Pair(device, o, outputs=IMAGE).frame()
    assert_bitexact(fast, cpu)
    assert (fast["tri_id"] != 0xFFFFFFFF).mean() > 0.3
    full, _ = Pair(device, o, outputs=ALL_OUTPUTS).frame()
    assert_bitexact(full, fast, IMAGE)
