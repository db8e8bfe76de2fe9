"""Submitted frames whose shading outlasts the next upload: a scene's triangle
arrays are overwritten as soon as the frame that read them has nothing left but
shading, so shading may read none of them. Two scenes of the same layout and
different contents, with image textures, AO, many lights and every G-buffer
output, alternate; every output equals the synchronous frame's, bit for bit."""
import ctypes as C

import numpy as np
import pytest

from helpers import ALL_OUTPUTS, options, shadow_cams
from polyred_gb300 import _abi, native, procedural, render, scene as sc

pytestmark = pytest.mark.gpu
W, H = 1600, 900


def _scene(seed):
    g = np.random.default_rng(seed)
    tex = sc.ImageTexture(g.integers(0, 256, (64, 64, 4)).astype(np.uint8))
    s = sc.Scene()
    for k in range(6):
        mesh = procedural.uv_sphere(24, 12, 1.0 + 0.2 * g.random())
        mesh = sc.Mesh(mesh.pos, mesh.nor, mesh.uv + g.random(2).astype(np.float32), g.integers(0, 256, mesh.col.shape).astype(np.uint8),
                       np.full(mesh.n_tris, -1 if k == 5 else 0))
        m = sc.BlinnPhong(diffuse=tuple(g.integers(50, 256, 4)), specular=tuple(g.integers(50, 256, 4)), shininess=float(2 + 9 * k),
                          texture=tex if k % 2 else tuple(g.integers(50, 256, 4)), flat_shading=k == 2, ambient_occlusion=True,
                          receive_shadow=True)
        s.add(sc.Geometry(mesh, m).translate(*(g.uniform(-1.5, 1.5, 3))))
    for k in range(16):
        s.add(sc.Point(position=tuple(g.uniform(-4, 4, 3)), intensity=0.4, cast_shadow=k < 2))
    s.add(sc.Ambient(intensity=0.2))
    cam = sc.Perspective(position=(0, 0.5, 3.2), target=(0, 0, 0), up=(0, 1, 0), fov=60, aspect=W / H, near=0.1, far=40)
    o = options(s, cam, W, H, shadow_map=True, shadow_size=(256, 256))
    flat = render.FlatScene(s)
    return flat, flat.desc(), render.FrameDesc(o, shadow_cams(o))


def test_uploads_during_shading(device):
    import torch
    lib = native.load()
    scenes = [_scene(k) for k in (1, 2)]
    assert scenes[0][0].n_tris == scenes[1][0].n_tris
    ref = []
    for flat, d, fd in scenes:  # also sizes the capacities
        native.check(lib.pr_scene_upload(device.handle, C.byref(d)))
        o = render.Outputs(W, H, ALL_OUTPUTS)
        native.check(lib.pr_render(device.handle, C.byref(fd.desc), C.byref(o.desc)))
        ref.append(o.arrays)
    assert all((r["tri_id"] != 0xFFFFFFFF).mean() > 0.3 for r in ref)
    dt = {np.dtype(np.float32): torch.float32, np.dtype(np.uint8): torch.uint8, np.dtype(np.uint32): torch.int32, np.dtype(np.int32): torch.int32}
    sent = []
    for k in range(12):
        _, d, fd = scenes[k % 2]
        t = {n: torch.zeros(ref[0][n].shape, dtype=dt[ref[0][n].dtype], device="cuda") for n in ALL_OUTPUTS}
        od = _abi.pr_outputs()
        od.size = C.sizeof(_abi.pr_outputs)
        od.flags = _abi.PR_OUT_DEVICE_PTRS
        for n, a in t.items():
            setattr(od, n, a.data_ptr())
        sent.append((d, fd, t, od))
    torch.cuda.synchronize()
    for d, fd, _, od in sent:  # nothing between the calls: the uploads run beside the shading before them
        native.check(lib.pr_frame_submit(device.handle, C.byref(d), C.byref(fd.desc), C.byref(od)))
    native.check(lib.pr_sync(device.handle))
    for k, (_, _, t, _) in enumerate(sent):
        for n, a in t.items():
            want = ref[k % 2][n]
            assert np.array_equal(a.cpu().numpy().view(np.uint8), want.view(np.uint8)), (k, n)
