"""A body of infinite mass in the mixed-precision sums that end in two FP32 words:
every other body's acceleration is infinite, towards it."""
import numpy as np
import pytest

from nbody_gb300.data import NBodyData
from nbody_gb300.ensemble import Ensemble

pytestmark = pytest.mark.gpu


def _data(n, heavy, sign):
    d = NBodyData.uniform_cube(n, side=2.0, seed=n)
    d.mass[heavy] = sign * np.inf
    return d


def _check(a, d, heavy, sign):
    want = np.copysign(np.inf, sign * (d.vertices[heavy] - d.vertices))
    rows = np.arange(d.get_count()) != heavy
    assert np.array_equal(a[rows], want[rows])


@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("heavy", [0, 700, 1499])
@pytest.mark.parametrize("g", [1, 2])
def test_ensemble(gpulib, g, heavy, sign):
    systems = [_data(1500, heavy, sign), NBodyData.plummer(300, seed=1)]
    ens = Ensemble(softening=1e-2)
    ens.tune_set("ensemble.pairs_per_lane", g)
    ens.init(systems)
    a = ens.fcompute().reshape(6, -1)[3:].T
    _check(a[:1500], systems[0], heavy, sign)
    assert np.all(np.isfinite(a[1500:]))
    ens.close()


@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("soft", [0.0, 1e-2])
@pytest.mark.parametrize("n,heavy", [(2, 0), (65, 64), (1500, 700), (5120, 5119)])
def test_small_direct_sum(make_engine, n, heavy, soft, sign):
    d = _data(n, heavy, sign)
    e = make_engine(precision="mixed", softening=soft)
    assert e.init(d)
    f, a = e.create_buffer(8 * 6 * n), np.zeros(6 * n)
    e.fcompute(0.0, e.get_y(), f)
    e.read_buffer(a, f)
    _check(a[3 * n:].reshape(3, n).T, d, heavy, sign)
