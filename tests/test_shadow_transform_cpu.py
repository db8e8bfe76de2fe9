"""The shadow lookup's single transform as the library computes it
(prh::shadow_composite): applied by float32 FMAs and divided by w as
shadow_hit_fast does it, a point stays within the bound it is given of the
reference's three Applies and Pos(); and the lookups that it is refused to."""
import numpy as np
import pytest

from polyred_gb300 import pmath
from test_shadow_composite_cpu import D, F, apply3, look


def composite(lib, v, p, w, h):
    v, p = (np.ascontiguousarray(m, F).reshape(16) for m in (v, p))
    smap, serr = np.empty(12, F), np.empty(12, F)
    rc = lib.pr_debug_shadow_composite(v.ctypes.data, p.ctypes.data, w, h, smap.ctypes.data, serr.ctypes.data)
    return rc, smap, serr


def pos(x):
    """Vec4.Pos (math/vec4.go): over w unless that is 1 or 0."""
    w = x[:, 3:]
    with np.errstate(all="ignore"):
        return np.where((w == 1) | (w == 0), x, x * (F(1) / w))[:, :3]


def rows(m, x):
    """Rows of a 3 x 4 matrix by single-rounding FMAs, as apply3 takes a 4 x 4 one."""
    return apply3(np.concatenate([m, F([0, 0, 0, 1])]), x)


@pytest.mark.parametrize("reach", [1e-2, 1.0, 30.0, 4e3])
@pytest.mark.parametrize("size", [(64, 64), (1000, 333), (16384, 5)])
def test_within_the_bound(native_lib, reach, size):
    g = np.random.default_rng(size[0])
    for _ in range(20):
        v = F(look(g.normal(0, reach, 3) + 0.1, g.normal(0, reach / 3, 3)).reshape(-1))
        n, f = -reach * g.uniform(0.1, 3), -reach * g.uniform(4, 9)
        w, h = reach * g.uniform(0.05, 5, 2)
        p = F(np.array([[1 / w, 0, 0, g.normal()], [0, 1 / h, 0, g.normal()], [0, 0, 2 / (n - f), (f + n) / (n - f)], [0, 0, 0, 1]]).reshape(-1))
        rc, smap, serr = composite(native_lib, v, p, *size)
        assert rc == 1
        # the matrix is the product (row order, transposition): against float64, to its own rounding
        s = np.array([[size[0] / 2, 0, 0, size[0] / 2], [0, size[1] / 2, 0, size[1] / 2], [0, 0, 1, 0], [0, 0, 0, 1]])
        full = s @ D(p).reshape(4, 4) @ D(v).reshape(4, 4)
        size_of = s @ np.abs(D(p)).reshape(4, 4) @ np.abs(D(v)).reshape(4, 4)
        assert (np.abs(D(smap).reshape(3, 4) - full[:3]) <= 1.01 * 2.0 ** -24 * size_of[:3]).all()
        assert (D(serr).reshape(3, 4) >= 17.02 * 2.0 ** -24 * size_of[:3]).all()
        x = F(np.concatenate([g.normal(0, reach, (3000, 3)) * g.choice([0, 1e-3, 1, 50], (3000, 1)),
                              g.choice([1.0, 0.0, 0.04, -0.3, 7.0], (3000, 1))], 1))
        ref = pos(apply3(F(s.reshape(-1)), apply3(p, apply3(v, x))))
        fast = pos(rows(smap, x))
        # shadow_hit_fast's bound, in float64 (its float32 evaluation rounds up)
        ww = D(x[:, 3])
        scale = np.where((ww == 1) | (ww == 0), 1.0, np.abs(D(F(1) / np.where(ww == 0, F(1), x[:, 3]))) * 1.0000002)
        bound = scale[:, None] * (np.abs(D(x)) @ D(serr).reshape(3, 4).T) + 2.4e-7 * np.abs(D(fast)) + 1e-30
        assert (np.abs(D(ref) - D(fast)) <= bound).all()


def test_a_perspective_light_is_refused(native_lib):
    v = pmath.view_matrix(F([3, 4, 5]), F([0, 0, 0]), F([0, 1, 0]))
    ortho = pmath.orthographic_matrix(-2, 2, -2, 2, 1, -20)
    persp = pmath.perspective_matrix(F(60), F(1), F(-0.1), F(-50))
    assert composite(native_lib, v, ortho, 64, 64)[0] == 1
    assert composite(native_lib, v, persp, 64, 64)[0] == 0
