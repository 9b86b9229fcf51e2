"""The two-word direct sum of a system large enough that the scale of a body's
sum comes from one body in eight, where some of those stand very close to others:
a close body in the sample counts eight times and raises its neighbours' limit to
8 / 1024 of their sums.  64 units of 2^-48 of such terms, of either sign, are at
most 64 2^-48 sqrt(8 / 1024) = 2e-14 of A = sum |m_j| / r_j^2."""
import numpy as np
import pytest

from nbody_gb300.data import NBodyData

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("masses", ["equal", "drawn"])
def test_close_companions(make_engine, masses):
    n = 20011  # scales from the bodies 256 k .. 256 k + 31
    rng = np.random.default_rng(7)
    d = NBodyData.uniform_cube(n, side=2.0, seed=7)
    if masses == "drawn":
        d.mass = d.mass * rng.uniform(0.5, 1.5, n)
    rows = np.arange(40, n - 300, 311)
    rows = rows[rows % 256 >= 32]
    near = rows // 256 * 256 + rows % 32             # sampled, at half to most of the sum
    other = np.where(near + 64 == rows, near + 65, near + 64)  # not sampled, a hundredth of it
    unit = rng.normal(size=(2, len(rows), 3))
    unit /= np.linalg.norm(unit, axis=2, keepdims=True)
    r = 10.0 ** rng.uniform(-3.5, -2.0, len(rows))[:, None]
    d.vertices[near] = d.vertices[rows] + r * unit[0]
    d.vertices[other] = d.vertices[rows] + 10 * r * unit[1]
    e = make_engine(precision="fp64")
    assert e.init(d)
    f, a = e.create_buffer(8 * 6 * n), np.zeros(6 * n)
    e.fcompute(0.0, e.get_y(), f)
    e.read_buffer(a, f)
    a = a[3 * n:].reshape(3, n).T
    p, w = d.vertices.astype(np.longdouble), d.mass.astype(np.longdouble)
    for row in rows:
        v = p - p[row]
        r2 = np.maximum((v * v).sum(1), np.longdouble(1e-8))
        t = w / r2
        exact = (v * (t / np.sqrt(r2))[:, None]).sum(0)
        t[row] = 0
        assert np.all(np.abs(a[row] - exact) <= 2e-14 * t.sum())
