"""A context whose first frame fails at any of its allocations keeps the NaN
bookkeeping's rest state: its next frame of a scene with NaN depths is an
undisturbed context's, bit for bit."""
import ctypes as C

import numpy as np
import pytest

from helpers import options
from polyred_gb300 import _abi, native, render, scene as sc
from test_gpu_parity import _basic_material, _degenerate_scene, _mesh, _ortho_cam

pytestmark = pytest.mark.gpu
W, H = 160, 128
OUTS = ("rgba", "tri_id", "depth")


def test_nan_depths_after_a_failed_allocation(native_lib):
    lib = native_lib
    m = _basic_material(ambient_occlusion=True, receive_shadow=True)
    s = sc.Scene(sc.Geometry(_mesh(_degenerate_scene(7)), m), sc.Point(position=(0, 0, 5), cast_shadow=True), sc.Ambient(0.1))
    cam = _ortho_cam()
    flat = render.FlatScene(s)
    desc = flat.desc()
    fd = render.FrameDesc(options(s, cam, W, H, shadow_map=True), {0: (cam.view_matrix(), cam.proj_matrix())})

    def frames(fail):
        d = render.Device(0)
        native.check(lib.pr_scene_upload(d.handle, C.byref(desc)))
        n0 = lib.pr_testing_alloc_count()
        native.check(lib.pr_testing_fail_alloc(fail))
        rcs, outs = [], []
        for _ in range(3):
            out = render.Outputs(W, H, OUTS)
            native.check(lib.pr_shadow_reset(d.handle))
            rcs.append(lib.pr_render(d.handle, C.byref(fd.desc), C.byref(out.desc)))
            outs.append(out.arrays)
            lib.pr_testing_fail_alloc(0)
        n = lib.pr_testing_alloc_count() - n0
        d.close()
        return rcs, outs, n

    rcs, outs, n = frames(0)
    want = outs[0]
    assert rcs == [_abi.PR_OK] * 3 and np.isnan(want["depth"]).any() and n >= 15
    for k in range(1, n + 1):
        rcs, outs, _ = frames(k)
        assert rcs[0] in (_abi.PR_OK, _abi.PR_ERR_OOM) and rcs[1:] == [_abi.PR_OK] * 2
        for got in outs[1:] if rcs[0] else outs:
            for name in OUTS:
                assert np.array_equal(got[name].view(np.uint8), want[name].view(np.uint8)), (k, name)
