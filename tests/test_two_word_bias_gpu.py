"""Values that every term of a two-word sum shares, masses and the softening,
whose second words are off by as much as they can be, 2^-49 of the value: the sums
are not off by that.

A sum's own errors: of a potential, some twenty roundings of the total at its end,
of either sign (the threads' sums before them are independent), in both kernels,
so 6 to 8 times 2^-53 between the two; of a body's acceleration, at most 7e-15 of
A = sum |m_j| / r_j^2 and independent of its neighbours', so that the mean over
1024 bodies with |a| > A / 4 of the error along a is within 7e-15 * 4 / 32 =
8.8e-16 of |a|."""
import numpy as np
import pytest

from nbody_gb300.data import NBodyData

pytestmark = pytest.mark.gpu

WORST = 0.5 + 2.0 ** -26 + 2.0 ** -50  # 0.5, 2^-26 and 2^-49 of itself left


def _left(x):
    """What two FP32 words leave of x, of x."""
    r = x - float(np.float32(x))
    return (r - float(np.float32(r))) / x


def _potentials(make_engine, d, soft):
    for split_min in (10 ** 7, 1):
        e = make_engine(precision="mixed", softening=soft)
        assert e.init(d)
        e.tune_set("statistics.split_min", split_min)
        yield e.statistics()[7]


@pytest.mark.parametrize("mass", [WORST, 2.0 - WORST, 1 / 20011])
@pytest.mark.parametrize("n,soft", [(4096, 0.0), (4096, 1e-3), (20011, 0.0)])
def test_potential_of_equal_masses(make_engine, mass, n, soft):
    d = NBodyData.uniform_cube(n, side=2.0, seed=5)
    d.mass = np.full(n, mass)
    a, b = _potentials(make_engine, d, soft)
    assert abs(a - b) <= 8 * 2.0 ** -53 * abs(a)


def test_potential_of_a_large_softening(make_engine):
    soft = next(s for s in 2.0 + np.arange(1, 100000) * 1e-6 if _left(s * s) > 1.7e-15)
    d = NBodyData.uniform_cube(9000, side=2.0, seed=5)
    d.mass = np.ones(9000)
    a, b = _potentials(make_engine, d, soft)
    assert abs(a - b) <= 6 * 2.0 ** -53 * abs(a)


def _forces(make_engine, d, algo, key, split):
    n = d.get_count()
    e = make_engine(algo=algo, precision="fp64")
    assert e.init(d)
    e.tune_set(key, split)
    f, a = e.create_buffer(8 * 6 * n), np.zeros(6 * n)
    e.fcompute(0.0, e.get_y(), f)
    e.read_buffer(a, f)
    return a[3 * n:].reshape(3, n).T


def _along(a, b, d):
    """Mean of the difference along a, of |a|, over 1024 bodies off the middle."""
    rows = np.nonzero((d.vertices ** 2).sum(1) > 0.8)[0][:1024]
    scale = np.array([(d.mass / np.maximum(((d.vertices - p) ** 2).sum(1), 1e-8)).sum() - d.mass[i] * 1e8
                      for i, p in zip(rows, d.vertices[rows])])
    size = np.sqrt((a[rows] ** 2).sum(1))
    keep = size > scale / 4
    assert keep.sum() > 512
    return (((b - a)[rows] * a[rows]).sum(1) / size ** 2)[keep].mean() * np.sqrt(keep.sum() / 1024)


@pytest.mark.parametrize("mass", [WORST, 2.0 - WORST])
def test_forces_of_one_mass(make_engine, mass):
    n = 4096
    d = NBodyData.uniform_cube(n, side=2.0, seed=6)
    d.mass = np.full(n, mass)
    a, b = (_forces(make_engine, d, "bh", "bh.fp64_split", split) for split in (0, 1))
    assert abs(_along(a, b, d)) <= 8.8e-16
    d.mass[0] = 1.0  # (else the direct sum leaves the mass out of the terms)
    a, b = (_forces(make_engine, d, "direct", "direct.fp64_split", split) for split in (0, 1))
    assert abs(_along(a, b, d)) <= 8.8e-16
