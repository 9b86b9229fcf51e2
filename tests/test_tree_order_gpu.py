"""Leaf orders of the GPU builds, leaf for leaf, at the sizes where the sort's
form changes (one cluster with 1, 2, 4 or 8 keys per thread up to 32768 keys,
several launches above) and the median splits move to one CTA per segment
(4096 bodies), with and without equal coordinates."""
import numpy as np
import pytest

from curve_order import leaf_order
from nbody_gb300.data import NBodyData

pytestmark = pytest.mark.gpu
SIZES = [1, 2, 64, 2048, 4096, 8192, 16384, 32768, 65536]


def _positions(n, ties):
    v = NBodyData.plummer(n, seed=n + 1).vertices
    return np.round(v, 1) if ties else v


def _leaves(make_engine, v, build):
    n = len(v)
    d = NBodyData(vertices=v, velocities=np.zeros((n, 3)), mass=np.full(n, 1.0 / n))
    e = make_engine(algo="bh", precision="mixed", softening=1e-3, distance_to_node_radius_ratio=1.2)
    e.tune_set("bh.build", build)
    assert e.init(d)
    f = e.create_buffer(8 * 6 * n)
    e.fcompute(0.0, e.get_y(), f)
    return e.tree_leaves()


@pytest.mark.parametrize("ties", [False, True])
@pytest.mark.parametrize("n", SIZES)
def test_curve(make_engine, n, ties):
    v = _positions(n, ties)
    assert np.array_equal(_leaves(make_engine, v, 2), leaf_order(v, True))


@pytest.mark.parametrize("ties", [False, True])
@pytest.mark.parametrize("n", SIZES)
def test_median(make_engine, n, ties):
    """Every segment's left half: its smallest bodies along the level's axis in
    the order of the FP64 keys (-0 before +0), ties by body index."""
    v = _positions(n, ties)
    bits = np.ascontiguousarray(v.T).view(np.uint64)
    keys = np.where(bits >> np.uint64(63), ~bits, bits | np.uint64(1 << 63))
    rank = [np.argsort(np.argsort(keys[c], kind="stable")) for c in range(3)]
    order, level = np.arange(n), 0
    while (n >> level) > 1:
        seg = order.reshape(1 << level, -1)
        by = np.argsort(rank[level % 3][seg], axis=1)
        order = np.take_along_axis(seg, by, axis=1).reshape(-1)
        level += 1
    assert np.array_equal(_leaves(make_engine, v, 0), order)
