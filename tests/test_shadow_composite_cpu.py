"""CPU check of the shadow test's composite transform (shadow_hit_fast in
pr_kernels.cu, LightK::smap and serr): the single matrix, rounded to float32
and applied by float32 FMAs, stays within its bound of the reference's three
Applies (each FMA through float64, math/math.go:265-267), on light cameras
near and far, wide and narrow, and points from the origin to far away."""
import numpy as np
import pytest

F, D = np.float32, np.float64


def fma(a, b, c):
    """float32(fma(float64(a), float64(b), float64(c))): the product of two float32 is exact in float64."""
    return F(D(a) * D(b) + D(c))


def apply3(m, x):
    """Vec4.Apply of (n, 4) points."""
    rows = [fma(m[4 * i], x[:, 0], fma(m[4 * i + 1], x[:, 1], fma(m[4 * i + 2], x[:, 2], F(m[4 * i + 3] * x[:, 3])))) for i in range(4)]
    return np.stack(rows, 1)


def look(eye, at):
    f = (at - eye) / np.linalg.norm(at - eye)
    s = np.cross(f, (0, 1, 0))
    s /= np.linalg.norm(s)
    u = np.cross(s, f)
    return np.array([[*s, -s @ eye], [*u, -u @ eye], [*-f, f @ eye], [0, 0, 0, 1]])


@pytest.mark.parametrize("reach", [1e-2, 1.0, 30.0, 4e3])
@pytest.mark.parametrize("size", [64, 1000, 16384])
def test_bound(reach, size):
    g = np.random.default_rng(size)
    for _ in range(20):
        v = look(g.normal(0, reach, 3) + 0.1, g.normal(0, reach / 3, 3))
        n, f = -reach * g.uniform(0.1, 3), -reach * g.uniform(4, 9)
        w, h = reach * g.uniform(0.05, 5, 2)
        p = np.array([[1 / w, 0, 0, g.normal()], [0, 1 / h, 0, g.normal()], [0, 0, 2 / (n - f), (f + n) / (n - f)], [0, 0, 0, 1]])
        s = np.array([[size / 2, 0, 0, size / 2], [0, size / 2, 0, size / 2], [0, 0, 1, 0], [0, 0, 0, 1]])
        v, p, s = (F(m.reshape(-1)) for m in (v, p, s))
        smap = F((D(s).reshape(4, 4) @ D(p).reshape(4, 4) @ D(v).reshape(4, 4)).reshape(-1))
        serr = F((np.abs(D(s)).reshape(4, 4) @ np.abs(D(p)).reshape(4, 4) @ np.abs(D(v)).reshape(4, 4)).reshape(-1) * (17.5 * 2.0 ** -24))
        x = F(np.concatenate([g.normal(0, reach, (3000, 3)) * g.choice([0, 1e-3, 1, 50], (3000, 1)),
                              g.choice([1.0, 0.04, -0.3, 7.0], (3000, 1))], 1))
        ref = apply3(s, apply3(p, apply3(v, x)))
        fast = apply3(smap, x)
        assert (ref[:, 3] == x[:, 3]).all()  # w passes through
        bound = np.abs(D(x)) @ D(serr).reshape(4, 4)[:3].T
        assert (np.abs(D(ref[:, :3]) - D(fast[:, :3])) <= bound).all()
