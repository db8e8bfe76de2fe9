"""The images' host memory: what stays idle is one frame's images at most, a
renderer that has none idle takes another's, and a pool that is gone leaves
nothing behind."""
import gc

import numpy as np
import pytest

from polyred_gb300 import render

FIELDS = ("rgba", "tri_id", "depth", "nor", "face_nor", "world_pos", "uvd", "vcol", "mat_id")


def idle(pool):
    return sum(n * len(q) for n, q in pool.free.items())


def frame(pool, w, h, want):
    return render.Outputs(w, h, want, spare=pool).arrays


@pytest.mark.parametrize("want", [("rgba",), ("rgba", "tri_id", "depth"), FIELDS])
def test_one_frame_stays(want):
    pool = render._Spare(len(FIELDS) + 1)
    held = [frame(pool, 64, 48, want) for _ in range(20)]
    size = sum(a.nbytes for a in held[0].values())
    addresses = {a.ctypes.data for f in held for a in f.values()}
    assert len(addresses) == 20 * len(want)
    del held
    assert 0 < idle(pool) <= size
    again = frame(pool, 64, 48, want)
    assert {a.ctypes.data for a in again.values()} <= addresses and idle(pool) == 0
    frame(pool, 32, 48, want)
    assert idle(pool) <= size // 2  # the other size is forgotten


def test_another_renderers_idle_memory():
    a, b = render._Spare(4), render._Spare(4)
    old = frame(a, 640, 480, ("rgba", "depth"))
    at = {v.ctypes.data for v in old.values()}
    kept = old.pop("depth")
    del old
    new = frame(b, 640, 480, ("rgba", "depth"))
    got = {v.ctypes.data for v in new.values()}
    assert len(got & at) == 1 and kept.ctypes.data not in got and idle(a) == 0
    del new
    assert idle(b) == 2 * 640 * 480 * 4 and idle(a) == 0


def test_gone_pools():
    gc.collect()
    n = len(render._Spare._live)
    pools = [render._Spare(3) for _ in range(5)]
    arrays = [frame(p, 16, 16, ("rgba",))["rgba"] for p in pools]
    arrays[0][...] = 7
    del pools
    gc.collect()
    assert len(render._Spare._live) <= n + 5
    del arrays
    gc.collect()
    assert len(render._Spare._live) == n
    assert np.all(frame(render._Spare(1), 16, 16, ("rgba",))["rgba"].shape == (16, 16, 4))
