"""Image textures sampled in float32 with certified level weights, bit-exact
with the oracle: one-texel, one-column, odd and power-of-two images, with and
without mipmaps, magnified to far past the last level, wrapped and negative
coordinates, coordinates whose derivatives overflow, and no numbers."""
import numpy as np
import pytest

from helpers import Pair, assert_bitexact, options
from polyred_gb300 import scene as sc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mipmap", [False, True])
@pytest.mark.parametrize("w,h", [(1, 1), (1, 9), (2, 2), (7, 3), (64, 64), (300, 37)])
def test_sampling(device, w, h, mipmap):
    g = np.random.default_rng(w * 1000 + h)
    image = g.integers(0, 256, (h, w, 4), np.uint8)
    image[: h // 2] = image[0, 0]  # equal neighbours too
    pos, uv = [], []
    scales = list(10.0 ** np.linspace(-4, 5, 44)) + [1e30, 3e38, np.inf, np.nan]
    for k, s in enumerate(scales):
        x, y = (k % 8 - 4) * 1.0, (k // 8 - 3) * 1.0
        c = np.array([[x, y], [x + 0.9, y], [x + 0.9, y + 0.9], [x, y + 0.9]])
        z = -g.uniform(6, 9, 4)
        with np.errstate(invalid="ignore", over="ignore"):
            t = (g.uniform(-1, 1, (4, 2)) * s).astype(np.float32)
        for tri in ((0, 1, 2), (0, 2, 3)):
            pos.append([[c[i, 0], c[i, 1], z[i], 1.0] for i in tri])
            uv.append([t[i] for i in tri])
    nor = np.zeros((len(pos), 3, 4), np.float32)
    nor[..., 2] = 1
    m = sc.BlinnPhong(diffuse=(200, 220, 240, 255), specular=(9, 9, 9, 255), shininess=16,
                      texture=sc.ImageTexture(image, mipmap=mipmap))
    s = sc.Scene(sc.Geometry(sc.Mesh(np.array(pos, np.float32), nor, np.array(uv, np.float32)), m),
                 sc.Point(position=(1, 2, 4)), sc.Ambient(intensity=0.9))
    cam = sc.Perspective(position=(0, 0, 0), target=(0, 0, -1), up=(0, 1, 0), fov=60, aspect=1.3, near=0.1, far=40)
    for outputs in (("rgba", "tri_id", "depth"), ("rgba", "uvd")):
        p = Pair(device, options(s, cam, 390, 300), outputs=outputs)
        gpu, cpu = p.frame()
        assert_bitexact(gpu, cpu)
    assert len(np.unique(gpu["rgba"].reshape(-1, 4), axis=0)) > 2
