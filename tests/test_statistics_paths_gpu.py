"""The potential energy of one system on the FP64 pipe and in two-word FP32
arithmetic.  A term of at most 1/1024 of its body's sum is off by at most some
64 units of 2^-48 of itself, of either sign, so the sum is within 64 2^-48
sqrt(1/1024) = 7e-15 of sum |m_i m_j| / r; the FP64 reference here (pairwise
sums) is within a tenth of that."""
import numpy as np
import pytest

from nbody_gb300.data import NBodyData

pytestmark = pytest.mark.gpu


def _potential(d, soft):
    pe = mag = 0.0
    for i in range(1, d.get_count()):
        r2 = ((d.vertices[:i] - d.vertices[i]) ** 2).sum(1)
        inv = 1.0 / np.sqrt(r2 + soft * soft) if soft else \
            np.where(r2 < 1e-8, 0.0, 1.0 / np.sqrt(np.maximum(r2, 1e-300)))
        t = d.mass[:i] * (d.mass[i] * inv)
        pe -= t.sum()
        mag += np.abs(t).sum()
    return pe, mag


@pytest.mark.parametrize("soft", [0.0, 1e-3])
@pytest.mark.parametrize("split_min", [1, 10 ** 6], ids=["two-word", "fp64"])
@pytest.mark.parametrize("n", [1, 2, 3, 64, 255, 257, 512, 513, 1025, 3072])
@pytest.mark.parametrize("kind", ["cube", "plummer", "heavy pair", "coincident"])
def test_potential(make_engine, kind, n, split_min, soft):
    d = NBodyData.plummer(n, seed=n) if kind == "plummer" else \
        NBodyData.uniform_cube(n, side=2.0, seed=n)
    if kind == "heavy pair":  # one far pair is nearly all of the sum; a light body
        d.mass[:2] = 1e6
        d.mass[n // 2] = 1e-9
    elif kind == "coincident":
        d.vertices[n // 3:2 * (n // 3)] = d.vertices[:2 * (n // 3) - n // 3]
    e = make_engine(precision="mixed", softening=soft)
    assert e.init(d)
    e.tune_set("statistics.split_min", split_min)
    got = e.statistics()
    pe, mag = _potential(d, soft)
    assert abs(got[7] - pe) <= 7e-15 * mag
    assert np.array_equal(got, e.statistics())
    m = d.mass[:, None]
    assert np.allclose(got[0:3], (m * d.velocities).sum(0), rtol=0,
                       atol=1e-14 * (np.abs(m * d.velocities)).sum())
    assert np.allclose(got[8:11], (m * d.vertices).sum(0) / m.sum(), rtol=0,
                       atol=1e-14 * np.abs(m * d.vertices).sum() / m.sum())
    assert np.isclose(got[6], 0.5 * (m * d.velocities ** 2).sum(), rtol=1e-14)


@pytest.mark.parametrize("split_min", [1, 10 ** 6], ids=["two-word", "fp64"])
def test_not_finite(make_engine, split_min):
    d = NBodyData.uniform_cube(400, side=2.0, seed=3)
    d.vertices[5, 1] = np.nan
    e = make_engine(precision="fp64")
    assert e.init(d)
    e.tune_set("statistics.split_min", split_min)
    assert np.isnan(e.statistics()[7])
