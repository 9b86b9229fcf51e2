"""The two FP64 direct-sum paths against extended precision.

Per body the error is measured against A = sum |m_j| / r_j^2, the scale its
rounding errors have.  A body's sum on the FP64 pipe carries a few 2^-53 of A.
In two-word FP32 arithmetic a term t is off by at most 64 units of 2^-48 t at
random, and no term of more than A / 1024 is taken that way, so the errors add
up to at most 64 2^-48 sqrt(A t_max) = 7e-15 A for the worst possible signs of
a normal distribution's 1 sigma at the bound of every term; a tenth of that is
measured.  Both stay below 7e-15 A.
"""
"""The two FP64 direct-sum paths against extended precision.

Per body the error is measured against A = sum |m_j| / r_j^2, the scale its
rounding errors have.  On the FP64 pipe a body's sum carries a few 2^-53 of A.
In two-word FP32 arithmetic a term t <= A / 1024 is off by at most some 64
units of 2^-48 t, of either sign; over all terms that is 64 2^-48 sqrt(sum t^2)
<= 64 2^-48 sqrt(A A / 1024) = 7e-15 A.
"""
import numpy as np
import pytest

from nbody_gb300.data import NBodyData

pytestmark = pytest.mark.gpu
BOUND = 7e-15


def _exact(v, m):
    """Accelerations and scales of (at most 256) bodies."""
    p, w = v.astype(np.longdouble), m.astype(np.longdouble)
    rows = np.unique(np.linspace(0, len(m) - 1, 256).astype(int))
    acc, scale = np.empty((len(rows), 3), np.longdouble), np.empty(len(rows), np.longdouble)
    for i, row in enumerate(rows):
        d = p - p[row]
        r2 = np.maximum((d * d).sum(1), np.longdouble(1e-8))
        acc[i] = (d * (w / (r2 * np.sqrt(r2)))[:, None]).sum(0)
        t = np.abs(w) / r2
        t[row] = 0
        scale[i] = t.sum()
    return rows, acc, scale


def _data(kind, n):
    rng = np.random.default_rng(n)
    d = NBodyData.uniform_cube(n, side=2.0, seed=n)
    if kind == "plummer":  # equal masses
        d = NBodyData.plummer(n, seed=n)
    elif kind == "far clusters":  # two tight groups at a large distance and offset
        d.vertices = 1e-3 * d.vertices + 1e3
        d.vertices[n // 2:] += [3e3, -5e3, 1e4]
    elif kind == "below the clamp":  # every pair closer than the clamp radius
        d.vertices *= 1e-6
    elif kind == "light bodies":  # masses over 60 binary orders, some negative
        d.mass = np.ldexp(rng.uniform(-1, 1, n), rng.integers(-60, 1, n))
    elif kind == "coincident":
        d.vertices[n // 3:2 * (n // 3)] = d.vertices[:2 * (n // 3) - n // 3]
    elif kind == "large numbers":
        d.vertices *= 2.0 ** 70
        d.mass *= 2.0 ** 90
    elif kind == "plane":
        d.vertices[:, 2] = 0.25
    return d


def _forces(make_engine, d, split=None):
    e = make_engine(precision="fp64")
    assert e.init(d)
    if split is not None:
        e.tune_set("direct.fp64_split", split)
    n = d.get_count()
    f = e.create_buffer(8 * 6 * n)
    e.fill_buffer(f, 1e10)
    e.fcompute(0.0, e.get_y(), f)
    out, again = np.zeros(6 * n), np.zeros(6 * n)
    e.read_buffer(out, f)
    e.fcompute(0.0, e.get_y(), f)
    e.read_buffer(again, f)
    assert np.array_equal(out, again, equal_nan=True)
    assert np.array_equal(out[:3 * n].reshape(3, n).T, d.velocities)
    return out[3 * n:].reshape(3, n).T


KINDS = ["cube", "plummer", "far clusters", "below the clamp", "light bodies", "coincident",
         "large numbers", "plane"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 257, 1535])
def test_fp64_pipe(make_engine, kind, n):
    d = _data(kind, n)
    rows, acc, scale = _exact(d.vertices, d.mass)
    a = _forces(make_engine, d, 0)
    assert np.all(np.abs(a[rows] - acc) <= BOUND * scale[:, None])


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [1, 65, 257, 1536, 1793, 3071])
def test_two_word(make_engine, kind, n):
    d = _data(kind, n)
    rows, acc, scale = _exact(d.vertices, d.mass)
    a = _forces(make_engine, d, 1)
    assert np.all(np.abs(a[rows] - acc) <= BOUND * scale[:, None])


@pytest.mark.parametrize("split", [0, 1])
def test_not_finite(make_engine, split):
    """A coordinate that is not finite reaches every body's sum, a massless
    body's own acceleration is 0 / 0, as in the reference."""
    d = _data("cube", 300)
    d.mass[7] = 0.0
    a = _forces(make_engine, d, split)
    assert np.all(np.isnan(a[7])) and np.all(np.isfinite(np.delete(a, 7, axis=0)))
    d.vertices[5] = np.nan
    assert np.all(np.isnan(_forces(make_engine, d, split)))
