"""pr_depth_map_noalloc against the oracle's drawDepth: vertices so far out that
the reference's int64 pixel bounds overflow."""
import ctypes as C

import numpy as np
import pytest

import oracle
from helpers import THREADS, same_bits
from polyred_gb300 import _abi, native, pmath, render, scene as sc
from test_zz_no_alloc import _desc, _objects, _ortho, _soup

pytestmark = pytest.mark.gpu


def both_windings(tris):
    t = np.asarray(tris, np.float32).reshape(-1, 3, 3)
    return np.stack([t, t[:, ::-1]], 1).reshape(-1, 3, 3)


def oracle_map(soup, w, h, view, proj, parts=None):
    """The light's depth map after one frame of triangles `soup` (n, 3, 4), from zero; parts: (count, model) per object."""
    s = sc.Scene()
    at = 0
    for n, model in parts or [(len(soup), None)]:
        pos = np.ascontiguousarray(soup[at:at + n])
        g = sc.Geometry(sc.Mesh(pos, np.tile(np.float32([0, 0, 1, 0]), (n, 3, 1))), sc.BlinnPhong())
        s.add(g if model is None else g.translate(*model))
        at += n
    s.add(sc.Point(position=(0, 0, 5), cast_shadow=True))
    cam = sc.Orthographic(position=(0, 0, 5), target=(0, 0, 0), up=(0, 1, 0), left=-2, right=2, bottom=-2, top=2, near=1, far=-20)
    opts = dict(width=8, height=8, camera=cam, scene=s, perspective=False, shadow_map=True, gamma=False,
                background=(0, 0, 0, 0), shadow_size=(w, h))
    flat = render.FlatScene(s)
    fd = render.FrameDesc(opts, {0: (view, proj)})
    out = render.Outputs(8, 8, ("rgba",))
    state = np.zeros((1, h, w), np.float32)
    oracle.render(flat.desc(), fd.desc, out.desc, shadow_state=state, threads=THREADS)
    return state[0], flat


def device_map(lib, flat, w, h, view, proj, init=None):
    import torch
    pos = torch.from_numpy(np.ascontiguousarray(flat.pos)).cuda()
    depth = torch.zeros((h, w), dtype=torch.float32, device="cuda") if init is None else torch.from_numpy(init.copy()).cuda()
    nd = _desc(flat.n_tris, flat.objects, w, h, view, proj, pos.data_ptr(), depth.data_ptr())
    nd.n_objects = flat.n_objects
    torch.cuda.synchronize()
    rc = lib.pr_depth_map_noalloc(C.byref(nd))
    return rc, depth.cpu().numpy()


def check(lib, soup, w, h, parts=None):
    view, proj = _ortho()
    want, flat = oracle_map(soup, w, h, view, proj, parts)
    rc, got = device_map(lib, flat, w, h, view, proj)
    native.check(rc)
    eq = same_bits(np.where(got == 0, np.float32(0), got), np.where(want == 0, np.float32(0), want))
    assert eq.all(), (int((~eq).sum()), np.argwhere(~eq)[:3])
    return want


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("sign", [-1, 1])
def test_far_vertices(native_lib, axis, sign):
    """A vertex 2^k pixels out, on both sides of 2^62 and 2^63: beyond the
    latter the reference's upper bound int(x) is the smallest int64 and it draws
    nothing."""
    tris = []
    for n, k in enumerate(range(54, 64)):  # 16 pixels a unit: 2^58 to 2^67 pixels
        y = -1.8 + 0.36 * n
        t = np.array([[-0.5, y, -0.3 - 0.1 * n], [sign * 2.0 ** k, y, -0.3 - 0.1 * n], [-0.5, y + 0.3, -0.3 - 0.1 * n]])
        tris.append(t if axis == 0 else t[:, [1, 0, 2]])
    want = check(native_lib, _soup(both_windings(tris)), 64, 64)
    assert 50 < (want != 0).sum() < 64 * 64
