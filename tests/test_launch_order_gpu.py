"""Kernels are launched before their predecessors end and wait for them
themselves: chains in which every operation needs the whole result of the one
before give exact results (whole numbers below 2^53)."""
import numpy as np
import pytest

from nbody_gb300.data import NBodyData

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 257, 5003, 1 << 20])
def test_dependent_vector_operations(make_engine, n):
    e = make_engine(precision="mixed")
    assert e.init(NBodyData.plummer(64, seed=1))
    start = np.random.default_rng(n).integers(-3, 4, (2, n)).astype(np.float64)
    a, b, c = (e.create_buffer(8 * n) for _ in range(3))
    e.write_buffer(a, start[0])
    e.write_buffer(b, start[1])
    x, y = start
    for k in range(30):
        e.fmadd_inplace(a, b, 1.0)      # a += b
        e.fmadd(c, b, a, 1.0)           # c = b + a
        e.fmaddn_inplace(b, [a, c], [2.0, -1.0], 2)
        x = x + y
        y = y + 2.0 * x - (y + x)
        if k % 10 == 9:                 # a copy between the kernels
            e.copy_buffer(c, a)
            e.fill_buffer(a, 0.0)
            e.fmadd_inplace(a, c, 1.0)
    got = np.zeros((2, n))
    e.read_buffer(got[0], a)
    e.read_buffer(got[1], b)
    assert np.abs(x).max() < 2.0 ** 53
    assert np.array_equal(got, np.stack([x, y]))


BH = dict(algo="bh", distance_to_node_radius_ratio=2.0)


@pytest.mark.parametrize("n,param", [
    (n, dict(BH, **p)) for n in (64, 4096, 65536)
    for p in (dict(precision="mixed", softening=1e-3), dict(precision="fp64"))
] + [(64, dict(precision="fp64")), (4096, dict(precision="fp64"))])
def test_repeated_steps_are_equal(make_engine, param, n):
    d = NBodyData.plummer(n, seed=5)
    out = []
    for sync in (False, True):  # every kernel alone, then queued one after the other
        e = make_engine(**param)
        assert e.init(d)
        f = e.create_buffer(8 * 6 * n)
        for _ in range(5):
            e.fcompute(0.0, e.get_y(), f)
            if sync:
                e.synchronize()
            e.fmadd_inplace(e.get_y(), f, 1e-3)
            if sync:
                e.synchronize()
            e.advise_time(0.0)
        y = np.zeros(6 * n)
        e.read_buffer(y, e.get_y())
        out.append(y)
    assert np.array_equal(out[0], out[1])
