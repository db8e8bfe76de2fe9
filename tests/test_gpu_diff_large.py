"""The backward pass's shared gradients over many pixels: float32 partial sums
stay short. A flat plane that faces its light, whose terms are whole numbers
below 2^12: sums of 4096 of them are exact in float32 (and the totals in
float64), longer ones are not. And spheres of several materials under a gradient
of either sign, against the FP64 adjoint on the same G-buffer."""
import ctypes as C

import numpy as np
import pytest

import oracle
from polyred_gb300 import _abi, diff, native, scene as sc
from test_gpu_diff_sums import _renderer

pytestmark = pytest.mark.gpu
LIT, FLAT = 1, 2  # G-buffer pixel flags


@pytest.mark.parametrize("W,H", [(3840, 2160), (2051, 1999)])
def test_partial_sums(W, H):
    import torch
    pos = np.array([[[-9, -9, 0, 1], [9, -9, 0, 1], [0, 9, 0, 1]]], np.float32)
    nor = np.tile(np.float32([0, 0, 1, 0]), (1, 3, 1))
    mat = sc.BlinnPhong(diffuse=(255, 255, 255, 255), specular=(0, 0, 0, 255), shininess=1.0, texture=(1, 1, 1, 255), flat_shading=True)
    s = sc.Scene(sc.Geometry(sc.Mesh(pos, nor), mat), sc.Directional(direction=(0, 0, -1), intensity=1.0), sc.Ambient(intensity=0.5))
    cam = sc.Perspective(position=(0, 0, 4), target=(0, 0, 0), up=(0, 1, 0), fov=50, aspect=W / H, near=0.1, far=100)
    r = diff.DiffRenderer(s, [diff.View(cam, W, H)], shadow_map=False)
    p = r.initial_params()
    pixel = torch.zeros(16)
    pixel.view(torch.int32)[2] = LIT | FLAT
    pixel[3] = 1.0                                      # factor
    pixel[7], pixel[11], pixel[14] = 255.0, 1.0, 1.0    # alpha, position (0, 0, 0, 1), face normal (0, 0, 1)
    gbuf = pixel.cuda().expand(H, W, 16).contiguous()
    k = torch.randint(0, 4096, (H, W), generator=torch.Generator().manual_seed(W))
    total = int(k.sum())
    grad = torch.zeros((H, W, 4), device="cuda")
    grad[..., 0] = k.cuda()
    fd = r.frame(0, p["light_pos"].numpy(), p["light_intensity"].numpy(), p["ambient"].numpy())
    d, keep = r._params_struct(p)
    g = _abi.pr_diff_grads()
    g.size = C.sizeof(_abi.pr_diff_grads)
    host = {n: np.zeros(c, np.float64) for n, c in (("kd", 3), ("light_intensity", 1), ("ambient", 1))}
    for n, a in host.items():
        setattr(g, n, a.ctypes.data_as(_abi.DP))
    torch.cuda.synchronize()
    native.check(r.lib.pr_diff_backward(r.device.handle, C.byref(fd.desc), C.byref(d), gbuf.data_ptr(), grad.data_ptr(), C.byref(g)))
    assert host["ambient"][0] == host["light_intensity"][0] == host["kd"][0] == total, ({n: a[0] - total for n, a in host.items()})


def test_all_shared_gradients(W=2600, H=1701):
    import torch
    r = _renderer(W, H, 3)
    p = r.initial_params()
    _, gbuf = r.forward_raw(0, p)
    grad = torch.randn(H, W, 4, generator=torch.Generator().manual_seed(5)).cuda()
    got = r.backward_raw(0, p, gbuf, grad)
    fd = r.frame(0, p["light_pos"].numpy(), p["light_intensity"].numpy(), p["ambient"].numpy())
    npp = {k: v.detach().cpu().numpy().astype(np.float64) for k, v in p.items()}
    inp = oracle.DiffInputs(r.flat, gbuf.cpu().numpy(), npp, fd.desc, oracle.normal_matrices(r.flat))
    g64 = grad.cpu().numpy().astype(np.float64)
    want, scale = oracle.diff_backward64(inp, g64), oracle.diff_backward64(inp, g64, absolute=True)
    for k in ("kd", "ks", "shininess", "light_pos", "light_intensity", "ambient"):
        a, b = got[k].cpu().numpy().astype(np.float64).reshape(-1), want[k].reshape(-1)
        # each pixel's float32 terms within 2^-17 of their magnitudes (as in the central-difference checks)
        assert (np.abs(a - b) <= 2.0 ** -17 * scale[k].reshape(-1)).all(), (k, np.abs(a - b) / scale[k].reshape(-1))
        assert np.abs(b).max() > 0
