"""The anti-aliasing resize by tiles of 32 x 8 output pixels, bit-exact with
the oracle: images of one pixel, one short of, equal to and one past a tile,
at the smallest and largest factors."""
import numpy as np
import pytest

from helpers import Pair, options
from polyred_gb300 import procedural

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [2, 3, 7, 16])
@pytest.mark.parametrize("size", [(1, 1), (31, 7), (32, 8), (33, 9), (97, 5)])
def test_tiles(device, m, size):
    s, cam = procedural.small_scene(width=size[0], height=size[1])
    p = Pair(device, options(s, cam, *size, msaa=m), outputs=("rgba",))
    gpu, cpu = p.frame()
    assert gpu["rgba"].shape == (size[1], size[0], 4) and np.array_equal(gpu["rgba"], cpu["rgba"])
