"""Frames that cannot grow their lists (pr_render_async): records two or three
pixels wide and thousands high on a fresh context, whose 32 x 32 blocks would
outnumber the room for them, equal the synchronous frame."""
import ctypes as C

import numpy as np
import pytest

from helpers import Pair, assert_bitexact, options
from polyred_gb300 import _abi, native, render, scene as sc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("upright", [True, False])
@pytest.mark.parametrize("thick", [1.6, 2.7])
def test_thin_records(native_lib, device, upright, thick):
    import torch
    lib = native_lib
    long = 14000 if thick < 2 else 10900
    W, H = (64, 16384) if upright else (16384, 64)
    a, b = (10.2, 100.0), (10.2 + thick, 100.0 + long)  # pixels: across, along
    px = [(a[0], a[1]), (b[0], b[1]), (a[0], b[1])]
    if upright:
        px = px[::-1]
    pos = np.ones((2, 3, 4), np.float32)
    for k, (across, along) in enumerate(px):
        x, y = (across, along) if upright else (along, across)
        pos[:, k, :3] = (2 * x / W - 1, 2 * y / H - 1, 0)
    pos[1] = pos[1, ::-1]  # the other winding
    nor = np.tile(np.float32([0, 0, 1, 0]), (2, 3, 1))
    s = sc.Scene(sc.Geometry(sc.Mesh(pos, nor), sc.BlinnPhong()), sc.Ambient(intensity=0.5))
    cam = sc.Orthographic(position=(0, 0, 5), target=(0, 0, 0), up=(0, 1, 0), left=-1, right=1, bottom=-1, top=1, near=1, far=-20)
    opts = options(s, cam, W, H)
    gpu, cpu = Pair(device, opts, outputs=("rgba", "tri_id", "depth")).frame()
    assert_bitexact(gpu, cpu)
    assert (gpu["tri_id"] != 0xFFFFFFFF).sum() > long / 2
    flat = render.FlatScene(s)
    fd, desc = render.FrameDesc(opts, {}), flat.desc()
    d = render.Device(0)
    native.check(lib.pr_scene_upload(d.handle, C.byref(desc)))
    ids = torch.zeros((H, W), dtype=torch.int32, device="cuda")
    od = _abi.pr_outputs()
    od.size = C.sizeof(_abi.pr_outputs)
    od.flags = _abi.PR_OUT_DEVICE_PTRS
    od.tri_id = ids.data_ptr()
    torch.cuda.synchronize()
    native.check(lib.pr_render_async(d.handle, C.byref(fd.desc), C.byref(od)))
    native.check(lib.pr_sync(d.handle))
    assert np.array_equal(ids.cpu().numpy().view(np.uint32), gpu["tri_id"])
    d.close()
