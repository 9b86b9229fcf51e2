"""Ensemble calls after, or during, something that fails on the host."""
import numpy as np
import pytest

from nbody_gb300._lib import NbgError
from nbody_gb300.data import NBodyData
from nbody_gb300.ensemble import Ensemble

pytestmark = pytest.mark.gpu


def _systems(*sizes):
    return [NBodyData.plummer(n, seed=n) for n in sizes]


def _empty():
    d = NBodyData.plummer(2, seed=1)
    d.vertices, d.velocities, d.mass = d.vertices[:0], d.velocities[:0], d.mass[:0]
    return d


@pytest.mark.parametrize("before", [0, 1], ids=["new", "loaded"])
def test_calls_after_a_failed_init(gpulib, before):
    """A batch that is refused leaves no batch behind: every call that needs
    one says so, and none runs on memory that is gone."""
    ens = Ensemble(softening=1e-2)
    if before:
        ens.init(_systems(200, 50))
        ens.step(1)
    with pytest.raises(NbgError):
        ens.init(_systems(100) + [_empty()])
    for call in (lambda: ens.step(1), ens.get_state, ens.fcompute, ens.status, ens.statistics,
                 ens.autotune):
        with pytest.raises(NbgError, match="not initialised"):
            call()
    ens.tune_set("ensemble.pairs_per_lane", 1)
    systems = _systems(300, 64)
    ens.init(systems)
    v, u = ens.get_state()
    assert np.array_equal(v, np.concatenate([d.vertices for d in systems]))
    assert np.array_equal(u, np.concatenate([d.velocities for d in systems]))
    ens.step(2)
    assert ens.status()[0].shape == (2,)
    ens.close()


def test_state_of_an_ensemble_without_a_batch(gpulib):
    ens = Ensemble()
    v, u = ens.get_state()
    assert v.shape == u.shape == (0, 3)
    ens.close()


@pytest.mark.parametrize("sizes", [(1,), (8192,), (8193,), (4096, 4096), (4096, 4096, 1)])
def test_state_laid_out_by_host_and_kernel(gpulib, sizes):
    systems = _systems(*sizes)
    ens = Ensemble()
    ens.init(systems)
    v, u = ens.get_state()
    assert np.array_equal(v, np.concatenate([d.vertices for d in systems]))
    assert np.array_equal(u, np.concatenate([d.velocities for d in systems]))
    ens.close()
