"""pr_depth_map_noalloc against the oracle's drawDepth: vertices so far out that
the reference's int64 pixel bounds overflow; maps up to 2^20 texels long, whose
corners do not fit 16 bits; as many objects as travel with the launch, one more,
and the most."""
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


def long_triangles(w, h):
    """Small and long triangles along the whole map and past its ends; every 16th edge-on along a line of texel
    centres (0 / 0 barycentrics: NaN depths)."""
    g = np.random.default_rng(w + 3 * h)
    long, short = max(w, h), min(w, h)
    k = 400
    at = g.uniform(-2.05, 2.05, (k, 1)) + np.where(g.random((k, 3)) < 0.5, 6.0 / long, g.choice([1e-3, 3e-2, 0.5], (k, 1))) * g.normal(0, 1, (k, 3))
    across = g.uniform(-2, 2, (k, 1)) + g.normal(0, 0.8, (k, 3))
    across[::16] = -2 + 4 * (g.integers(0, short, (k // 16, 1)) + 0.5) / short
    z = g.uniform(-2, 2, (k, 1)) + g.normal(0, 0.3, (k, 3))
    return np.stack([at, across, z] if w > h else [across, at, z], 2)


@pytest.mark.parametrize("w,h", [(1 << 20, 1), (1, 1 << 20), (131072, 8), (8, 131072), (65537, 15), (65001, 16), (65000, 16), (16, 65000), (16385, 60)])
def test_long_maps(native_lib, w, h):
    want = check(native_lib, _soup(both_windings(long_triangles(w, h))), w, h)
    row = want.any(0) if w > h else want.any(1)
    n = len(row)
    assert row[: n // 16].any() and row[-(n // 16):].any()
    if min(w, h) & (min(w, h) - 1) == 0:  # texel centres are float32 numbers
        assert np.isnan(want).any()


def test_long_map_overflow_leaves_the_map_unchanged(native_lib):
    """260 triangles that cover 131072 x 8 texels need 1024 tasks apiece: refused as on a square map; 200 are not."""
    tris = [[[-9, -9, -1 + k / 260], [9, -9, -1 + k / 260], [0, 12, -1 + k / 260]] for k in range(260)]
    soup = _soup(both_windings(tris))
    view, proj = _ortho()
    init = np.random.default_rng(7).uniform(-1, 1, (8, 131072)).astype(np.float32)
    init.view(np.uint32)[:, ::13] = 0x7FA00001
    for n, ok in ((260, False), (200, True)):
        _, flat = oracle_map(soup[: 2 * n], 4, 4, view, proj)
        rc, got = device_map(native_lib, flat, 131072, 8, view, proj, init)
        same = np.array_equal(got.view(np.uint32), init.view(np.uint32))
        assert (rc, same) == ((_abi.PR_OK, False) if ok else (_abi.PR_ERR_OVERFLOW, True))


@pytest.mark.parametrize("w,h", [(200, 120), (70000, 9)])
@pytest.mark.parametrize("n", [31, 32, 33, 256])
def test_objects(native_lib, n, w, h):
    """Objects of 0 to 3 hundred triangles (several to a block of 128, and more than a block) with models of their own."""
    g = np.random.default_rng(n)
    counts = g.choice([0, 2, 14, 130, 300], n, p=[0.2, 0.4, 0.3, 0.07, 0.03])
    counts[[0, -1]] = 2
    parts, tris = [], []
    for c in counts:
        parts.append((int(c), tuple(g.uniform(-1.5, 1.5, 3))))
        at = g.uniform(-0.3, 0.3, (c // 2, 1, 3)) + g.normal(0, 0.15, (c // 2, 3, 3))
        tris.append(both_windings(at))
    want = check(native_lib, _soup(np.concatenate(tris)), w, h, [p for p in parts])
    assert (want != 0).sum() > 0.05 * w * h
