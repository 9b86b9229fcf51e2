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
