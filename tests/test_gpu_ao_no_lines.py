"""Ambient occlusion without memory for the line maxima (16 bytes a pixel that
only speed the march up): the same images, of frames, of batches and of a
differentiable frame, and the allocation that fails may be theirs alone; one
that fails later takes their memory and succeeds. Host allocation results are
faked, nothing on the device fails."""
import ctypes as C

import numpy as np
import pytest

from helpers import options, shadow_cams
from polyred_gb300 import _abi, batch as pb, diff, native, procedural, render, scene as sc

pytestmark = pytest.mark.gpu
W, H = 420, 300  # pixels whose whole march lies inside the frame, and others
OUTS = ("rgba", "depth", "nor")


@pytest.fixture(autouse=True)
def _injection_off(native_lib):
    yield
    native_lib.pr_testing_fail_alloc(0)


def _scene(ao=True):
    s, cam = procedural.small_scene(W, H)
    for o, _ in s.iter_objects():
        if isinstance(o, sc.Geometry):
            for m in o.materials:
                m.ambient_occlusion = ao
    return s, options(s, cam, W, H)


def _frame(lib, h, opts):
    fd = render.FrameDesc(opts, shadow_cams(opts))
    out = render.Outputs(opts["width"], opts["height"], OUTS)
    return lib.pr_render(h, C.byref(fd.desc), C.byref(out.desc)), out.arrays


def _same(a, b):
    return all(np.array_equal(a[k].view(np.uint8), b[k].view(np.uint8)) for k in OUTS)


def test_frame(native_lib):
    lib = native_lib
    s, opts = _scene()
    flat = render.FlatScene(s)
    desc = flat.desc()
    small = dict(opts, width=W // 2, height=H // 2)
    dark = render.FlatScene(_scene(ao=False)[0])

    def device():
        d = render.Device(0)
        native.check(lib.pr_scene_upload(d.handle, C.byref(desc)))
        return d

    d = device()
    n0 = lib.pr_testing_alloc_count()
    rc, want = _frame(lib, d.handle, opts)
    native.check(rc)
    n = lib.pr_testing_alloc_count() - n0
    native.check(lib.pr_scene_upload(d.handle, C.byref(dark.desc())))
    assert not _same(_frame(lib, d.handle, opts)[1], want)  # AO shows
    d.close()
    went = []
    for k in range(1, n + 1):
        d = device()
        native.check(lib.pr_testing_fail_alloc(k))
        rc, got = _frame(lib, d.handle, opts)
        lib.pr_testing_fail_alloc(0)
        if rc == _abi.PR_OK:
            went.append(k)
            assert _same(got, want)
        else:
            assert rc == _abi.PR_ERR_OOM
        rc, got = _frame(lib, d.handle, opts)
        native.check(rc)
        assert _same(got, want)
        d.close()
    assert went  # the line maxima's own, and what is allocated after them
    # a context that holds them: any one allocation of a larger frame may fail
    d = device()
    native.check(_frame(lib, d.handle, small)[0])
    n0 = lib.pr_testing_alloc_count()
    native.check(_frame(lib, d.handle, opts)[0])
    n = lib.pr_testing_alloc_count() - n0
    d.close()
    for k in range(1, n + 1):
        d = device()
        native.check(_frame(lib, d.handle, small)[0])
        native.check(lib.pr_testing_fail_alloc(k))
        rc, got = _frame(lib, d.handle, opts)
        lib.pr_testing_fail_alloc(0)
        native.check(rc)
        assert _same(got, want)
        d.close()


def test_batch(native_lib):
    lib = native_lib
    scenes = [pb.sphere_scene(3_000, 0x5EED0004, n_lights=2), _scene(ao=True)[0]]

    def batch():
        b = pb.Batch(0)
        for s in scenes:
            b.add_scene(s)
        specs = []
        for cam in pb.ring_cameras(2, W, H, radius=6.0):
            for si, s in enumerate(scenes):
                o = pb.view_opts(s, cam, W, H, 128)
                specs.append((si, o, pb.shadow_cams(o)))
        return (b,) + tuple(b.views(specs, OUTS))

    def run(fail):
        b, arr, outs, keep = batch()
        n0 = lib.pr_testing_alloc_count()
        native.check(lib.pr_testing_fail_alloc(fail))
        rc = lib.pr_batch_render(b.handle, len(arr), arr)
        lib.pr_testing_fail_alloc(0)
        n = lib.pr_testing_alloc_count() - n0
        got = [{k: v.cpu().numpy() for k, v in o.items()} for o in outs]
        b.close()
        return rc, n, got

    rc, n, want = run(0)
    native.check(rc)
    went = 0
    for k in range(1, n + 1):
        rc, _, got = run(k)
        assert rc in (_abi.PR_OK, _abi.PR_ERR_OOM)
        if rc == _abi.PR_OK:
            went += 1
            assert all(_same(a, b) for a, b in zip(got, want))
    assert went


def test_differentiable_frame(native_lib):
    lib = native_lib
    s, opts = _scene()

    def gbuf(fail):
        r = diff.DiffRenderer(s, [diff.View(opts["camera"], W, H)], shadow_map=False)
        n0 = lib.pr_testing_alloc_count()
        native.check(lib.pr_testing_fail_alloc(fail))
        try:
            _, g = r.forward_raw(0, r.initial_params())
        except Exception:
            return None, 0
        finally:
            lib.pr_testing_fail_alloc(0)
            n = lib.pr_testing_alloc_count() - n0
            r.device.close()
        return g.cpu().numpy(), n

    want, n = gbuf(0)
    assert (want[..., 3] < 1).any()  # AO darkens some pixel's factor
    got = [g for g in (gbuf(k)[0] for k in range(1, n + 1)) if g is not None]
    assert got
    for g in got:
        # the factor float32(T^10000) is the same from either march
        assert np.array_equal(g.view(np.uint32), want.view(np.uint32))
