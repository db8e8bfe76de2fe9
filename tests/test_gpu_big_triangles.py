"""Rasterisation of large records by 32 x 32 blocks, bit-exact with the oracle
(colours, ids, depths and shadow maps): triangles whose boxes end on, before
and past block and tile edges, slivers of any slope, triangles that reach past
the frame or the map, collinear ones (NaN depths, the fix-up passes), a few
(shared by several warps each) and many."""
import math

import numpy as np
import pytest

from helpers import Pair, assert_bitexact, options
from polyred_gb300 import scene as sc

pytestmark = pytest.mark.gpu
W, H = 331, 269


def _mesh(px, depth):
    """Screen-space triangles (n, 3, 2) unprojected from a 60-degree camera at the origin to view depths (n, 3)."""
    n = len(px)
    t = math.tan(math.radians(60) / 2)
    pos, nor = np.ones((n, 3, 4), np.float32), np.zeros((n, 3, 4), np.float32)
    pos[..., 0] = (px[..., 0] / W * 2 - 1) * t * (W / H) * depth
    pos[..., 1] = (px[..., 1] / H * 2 - 1) * t * depth
    pos[..., 2] = -depth
    nor[..., 2] = 1
    return sc.Mesh(pos, nor)


def _triangles(kind, seed):
    g = np.random.default_rng(seed)
    if kind == "edges":  # right triangles with legs about multiples of the tile and block sizes
        legs = [60, 63, 64, 65, 71, 96, 97, 127, 128, 129, 200]
        at = [(0.5, 0.5), (3, 2), (31.9, 33.1), (17.25, 64)]
        return np.array([[(x, y), (x + a, y), (x, y + b)] for a in legs for b in (a, 70) for x, y in at], float)
    if kind == "slivers":
        a = g.uniform((0, 0), (W, H), (120, 2))
        b = g.uniform((0, 0), (W, H), (120, 2))
        return np.stack([a, b, (a + b) / 2 + g.normal(0, 1, (120, 2)) * g.choice([0.01, 0.3, 2.0], (120, 1))], 1)
    if kind == "past":
        return g.uniform((-W, -H), (2 * W, 2 * H), (80, 3, 2))
    n = 3 if kind == "few" else 900
    return g.uniform((0, 0), (W, H), (n, 3, 2))


@pytest.mark.parametrize("kind", ["edges", "slivers", "past", "few", "many"])
@pytest.mark.parametrize("degenerate", [False, True])
def test_blocks(device, kind, degenerate):
    px = _triangles(kind, 11)
    u, v = px[:, 1] - px[:, 0], px[:, 2] - px[:, 0]
    flip = u[:, 0] * v[:, 1] - u[:, 1] * v[:, 0] < 0
    px[flip] = px[flip][:, ::-1]
    g = np.random.default_rng(5)
    if degenerate:  # whole pixels on one line: zero area, 0 / 0 barycentrics
        line = np.array([[(10, 20), (150, 160), (290, 20 + 280)], [(5, 200), (300, 200), (150, 200)]], float)
        px = np.concatenate([px[: len(px) // 2], line, px[len(px) // 2:]])
    depth = g.uniform(2, 30, (len(px), 1)) * np.ones((1, 3)) if kind != "past" else g.uniform(2, 30, (len(px), 3))
    m = sc.BlinnPhong(diffuse=(200, 90, 40, 255), specular=(90, 90, 90, 255), shininess=16, receive_shadow=True)
    s = sc.Scene(sc.Geometry(_mesh(px, depth), m), sc.Point(position=(3, 5, 4), cast_shadow=True), sc.Ambient(intensity=0.2))
    cam = sc.Perspective(position=(0, 0, 0), target=(0, 0, -1), up=(0, 1, 0), fov=60, aspect=W / H, near=0.1, far=60)
    p = Pair(device, options(s, cam, W, H, shadow_map=True, shadow_size=(257, 190)))
    for _ in range(2):
        gpu, cpu = p.frame(with_shadow_maps=True)
        assert_bitexact(gpu, cpu)
    assert (gpu["tri_id"] != 0xFFFFFFFF).any()
