"""The images' host memory: never shared by two arrays in use, also across a
view kept of a dropped array, used again afterwards, bounded, and dropped with
the sizes that are asked for no more."""
import threading

import numpy as np
import pytest

from polyred_gb300 import render


@pytest.mark.parametrize("shape", [(1, 1), (3, 5), (480, 640, 4)])
def test_in_use_is_not_shared(shape):
    n = int(np.prod(shape)) * 4
    s = render._Spare(3)
    s.only({n})
    first = s.array(shape, np.float32)
    assert first.flags.writeable and first.flags.c_contiguous and first.shape == shape
    at = first.ctypes.data
    view = first[..., :1]
    del first
    held = [s.array(shape, np.float32) for _ in range(5)]
    assert len({a.ctypes.data for a in held} | {at}) == 6  # the view keeps its memory
    del view
    assert s.array(shape, np.float32).ctypes.data == at
    del held
    assert len(s.free[n]) == 3  # bounded
    s.only({n + 4})
    assert n not in s.free
    s.only(())  # what Renderer.close does
    assert not s.free


def test_other_sizes_and_a_dropped_pool():
    s = render._Spare(2)
    a, z = s.array((2, 3), np.uint32), s.array((0, 4), np.uint8)  # sizes that were not announced
    assert z.shape == (0, 4)
    a[...] = 7
    del s
    assert (a == 7).all()


def test_threads():
    s, bad = render._Spare(4), []
    s.only({4096})

    def work(k):
        for _ in range(300):
            a = s.array((32, 32), np.uint32)
            a[...] = k
            b = s.array((32, 32), np.uint32)
            b[...] = k + 100
            if not ((a == k).all() and (b == k + 100).all()):
                bad.append(k)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad
