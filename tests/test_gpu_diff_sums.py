"""The backward pass's warp sums and vertex atomics: gradient arrays that are
and are not 16-byte aligned, image widths that leave lanes idle, warps of one
and of several materials, no light and sixteen, against the FP64 adjoint on
the same G-buffer."""
import ctypes as C

import numpy as np
import pytest

import oracle
from polyred_gb300 import _abi, diff, native, procedural, scene as sc

pytestmark = pytest.mark.gpu


def _renderer(W, H, lights):
    rng = np.random.default_rng(3)
    s = sc.Scene()
    for k in range(9):  # three materials side by side, one of them flat, and a vertex-coloured sphere
        mats = [] if k == 4 else [sc.BlinnPhong(diffuse=(200, 120, 60 + 20 * k, 255), specular=(120, 120, 120, 255), shininess=5.0 + 7 * (k % 3),
                                                flat_shading=k % 3 == 2)]
        mesh = procedural.uv_sphere(12, 7, 0.6)
        if not mats:
            mesh = sc.Mesh(mesh.pos, mesh.nor, mesh.uv, rng.integers(0, 256, mesh.col.shape).astype(np.uint8), np.full(mesh.n_tris, -1))
        s.add(sc.Geometry(mesh, *mats).translate(float(k % 3) - 1.0, float(k // 3) - 1.0, 0.0))
    for k in range(lights):
        s.add(sc.Directional(direction=(-1, -1, -2), intensity=0.3) if k % 3 == 1 else
              sc.Point(position=(3 * np.cos(k), 2 + 0.1 * k, 3), intensity=1.5 / lights))
    s.add(sc.Ambient(intensity=0.1), sc.Ambient(intensity=0.07))
    cam = sc.Perspective(position=(0, 0, 4), target=(0, 0, 0), up=(0, 1, 0), fov=50, aspect=W / H, near=0.1, far=100)
    return diff.DiffRenderer(s, [diff.View(cam, W, H)], shadow_map=False)


@pytest.mark.parametrize("W,H,lights", [(97, 61, 2), (33, 40, 0), (64, 33, 16)])
def test_sums_and_alignment(W, H, lights):
    import torch
    r = _renderer(W, H, lights)
    p = r.initial_params()
    rad, gbuf = r.forward_raw(0, p)
    grad = torch.randn(H, W, 4, generator=torch.Generator().manual_seed(1)).cuda()
    got = {k: v.cpu().numpy() for k, v in r.backward_raw(0, p, gbuf, grad).items()}
    fd = r.frame(0, p["light_pos"].numpy(), p["light_intensity"].numpy(), p["ambient"].numpy())
    npp = {k: v.detach().cpu().numpy().astype(np.float64) for k, v in p.items()}
    inp = oracle.DiffInputs(r.flat, gbuf.cpu().numpy(), npp, fd.desc, oracle.normal_matrices(r.flat))
    want = oracle.diff_backward64(inp, grad.cpu().numpy().astype(np.float64))
    for k in diff.PARAM_NAMES:
        a, b = got[k].astype(np.float64).reshape(-1), np.asarray(want[k], np.float64).reshape(-1)
        # float32 terms of some hundred roundings each (a power amplifies by up to 19), of either sign: 2e-4 of the largest
        assert np.abs(a - b).max(initial=0) <= 2e-4 * max(np.abs(b).max(initial=0), 1e-3), k
    # the same gradients into arrays 4 bytes off
    d, keep = r._params_struct(p)
    nt = r.flat.n_tris * 12
    bufs = [torch.full((nt + 1,), 7.0, device="cuda") for _ in range(2)]
    g = _abi.pr_diff_grads()
    g.size = C.sizeof(_abi.pr_diff_grads)
    g.vertex_color, g.vertex_normal = (b.data_ptr() + 4 for b in bufs)
    torch.cuda.synchronize()
    native.check(r.lib.pr_diff_backward(r.device.handle, C.byref(fd.desc), C.byref(d), gbuf.data_ptr(), grad.data_ptr(), C.byref(g)))
    for b, k in zip(bufs, ("vertex_color", "vertex_normal")):
        b = b.cpu().numpy()
        assert b[0] == 7.0
        np.testing.assert_allclose(b[1:].reshape(-1, 3, 4), got[k], rtol=1e-4, atol=1e-4 * np.abs(got[k]).max())
