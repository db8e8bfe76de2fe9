"""The frame's chain of overlapped launches, bit-exact with the oracle: frames
of one pixel, of odd pixel counts (the last key of the cleared range) and of a
few rows; scenes whose triangles all, partly or never reach the clipper; no
light, lights that cast and do not, several casting lights (their passes share
records and tasks); each frame drawn twice with another size between, so that
keys, counters and work lists of the one before are there to be cleared."""
import pytest

from helpers import Pair, assert_bitexact, options
from polyred_gb300 import procedural, scene as sc

pytestmark = pytest.mark.gpu

LIGHTS = {"none": (), "plain": (False,), "cast": (True,), "mixed": (False, True, False, True, True)}
CAMERA = {"inside": (0, 0.2, 0.4), "edge": (0, 1, 2.5), "far": (0, 2, 9)}


@pytest.mark.parametrize("size", [(1, 1), (7, 3), (45, 31), (641, 5), (257, 255)])
@pytest.mark.parametrize("lights", sorted(LIGHTS))
@pytest.mark.parametrize("camera", sorted(CAMERA))
def test_chain(device, size, lights, camera):
    m = sc.BlinnPhong(diffuse=(200, 90, 40, 255), specular=(90, 90, 90, 255), shininess=16, receive_shadow=True)
    parts = [sc.Geometry(procedural.uv_sphere(24, 12), m), sc.Ambient(intensity=0.3)]
    parts += [sc.Point(position=(3 - k, 4, 2 + k), cast_shadow=c) for k, c in enumerate(LIGHTS[lights])]
    s = sc.Scene(*parts)
    for W, H in (size, (64, 33), size):
        cam = sc.Perspective(position=CAMERA[camera], target=(0, 0, 0), up=(0, 1, 0), fov=60, aspect=W / H, near=0.1, far=40)
        p = Pair(device, options(s, cam, W, H, shadow_map=True, shadow_size=(61, 47)))
        for _ in range(2):
            gpu, cpu = p.frame(with_shadow_maps=True)
            assert_bitexact(gpu, cpu)
