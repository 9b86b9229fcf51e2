"""Masses at the ends of FP64's range in the sums that have a two-word FP32
path: the FP64 pipe's kernels and the two-word ones give the same."""
import numpy as np
import pytest

from nbody_gb300.data import NBodyData

pytestmark = pytest.mark.gpu

KEY = {"direct": "direct.fp64_split", "bh": "bh.fp64_split"}


def _forces(make_engine, d, algo, split):
    n = d.get_count()
    e = make_engine(algo=algo, precision="fp64")
    assert e.init(d)
    e.tune_set(KEY[algo], split)
    f, a = e.create_buffer(8 * 6 * n), np.zeros(6 * n)
    e.fcompute(0.0, e.get_y(), f)
    e.read_buffer(a, f)
    return a[3 * n:].reshape(3, n).T


def _potential(make_engine, d, split_min, soft):
    e = make_engine(precision="mixed", softening=soft)
    assert e.init(d)
    e.tune_set("statistics.split_min", split_min)
    return e.statistics()[7]


# bodies 5 and 7 are in the sample that sets a body's scale, 40 and 50 are not
@pytest.mark.parametrize("masses", [{5: np.inf}, {40: np.inf}, {5: -np.inf}, {40: -np.inf},
                                    {5: np.inf, 40: np.inf}, {7: np.inf, 50: -np.inf}, {5: np.nan},
                                    {40: np.nan}])
class TestNotFinite:
    def _data(self, masses):
        d = NBodyData.uniform_cube(2048, side=2.0, seed=1)
        for k, m in masses.items():
            d.mass[k] = m
        return d

    @pytest.mark.parametrize("algo", ["direct", "bh"])
    def test_forces(self, make_engine, masses, algo):
        d = self._data(masses)
        a, b = (_forces(make_engine, d, algo, split) for split in (0, 1))
        assert not np.any(np.isfinite(a))  # every body meets each of these masses
        assert np.array_equal(a, b, equal_nan=True)

    @pytest.mark.parametrize("soft", [0.0, 1e-3])
    def test_potential(self, make_engine, masses, soft):
        d = self._data(masses)
        a, b = (_potential(make_engine, d, split_min, soft) for split_min in (10 ** 6, 1))
        assert not np.isfinite(a)
        assert np.array_equal(a, b, equal_nan=True)


def _direct_sums(d):
    """Direct sums in FP64 (numpy) and sum |m_j| / r_j^2 of every body."""
    acc, scale = np.empty((d.get_count(), 3)), np.empty((d.get_count(), 1))
    for i, p in enumerate(d.vertices):
        v = d.vertices - p
        r2 = np.maximum((v * v).sum(1), 1e-8)
        acc[i] = (v * (d.mass / (r2 * np.sqrt(r2)))[:, None]).sum(0)
        scale[i] = (np.delete(d.mass, i) / np.delete(r2, i)).sum()
    return acc, scale


# (below 2^-1024 the reciprocal of the masses' power of two is not finite)
@pytest.mark.parametrize("exp", [-1022, -1026, -1029, 988])
@pytest.mark.parametrize("algo", ["direct", "bh"])
def test_largest_mass_at_the_ends_of_the_range(make_engine, algo, exp):
    """Masses times a power of two give that many times the forces.  (The walk's
    FP64 kernel is no measure here: it forms m_i m_j, which underflows.)  The
    two-word bound is that of tests/test_bh_fp64_gpu.py; a term's weight m r^-3,
    its product with d, |d| < 4, and their sum round to multiples of 2^-1074.  The
    walk's node centres round like that too, so that a node near a critical
    radius may change sides: its error against the direct sum stays."""
    n = 2048
    d = NBodyData.uniform_cube(n, side=2.0, seed=2)
    d.mass = np.random.default_rng(3).integers(1, 4, n).astype(float)
    acc, scale = _direct_sums(d)
    one = _forces(make_engine, d, algo, 1)
    d.mass = np.ldexp(d.mass, exp)
    a = np.ldexp(_forces(make_engine, d, algo, 1), -exp)
    grid = 2 * n * (4 + 2) * 2.0 ** (-1074 - exp)
    if algo == "direct":
        assert np.all(np.abs(a - acc) <= (7e-15 + 2 * n * 2.0 ** -53) * scale + grid)
    else:
        error = [np.sqrt(((x - acc) ** 2).sum() / (acc ** 2).sum()) for x in (one, a)]
        assert 0 < error[0] < 0.1 and abs(error[1] / error[0] - 1) < 1e-2


@pytest.mark.parametrize("split", [0, 1])
@pytest.mark.parametrize("algo", ["direct", "bh"])
@pytest.mark.parametrize("mass,want", [(np.inf, 0.0), (-np.inf, 0.0), (2.0, 0.0), (0.0, np.nan), (np.nan, np.nan)])
def test_lone_body(make_engine, algo, split, mass, want):
    """Its force is 0, which the reference divides by its mass."""
    d = NBodyData.uniform_cube(1, side=2.0, seed=1)
    d.mass[0] = mass
    assert np.array_equal(_forces(make_engine, d, algo, split), np.full((1, 3), want), equal_nan=True)
