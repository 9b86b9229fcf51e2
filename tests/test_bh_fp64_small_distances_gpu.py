"""The two FP64 Barnes-Hut walks on systems much smaller than their distance
from the origin, or than the distance of one far body: the two-word walk meets
the nodes of the reference's walk there too (equal visit and interaction
counts).  The forces' bound is that of tests/test_bh_fp64_gpu.py."""
import numpy as np
import pytest

from nbody_gb300.data import NBodyData

pytestmark = pytest.mark.gpu


def _data(kind, n):
    d = NBodyData.uniform_cube(n, side=2.0, seed=n)
    if kind.startswith("offset"):
        d.vertices = 1e-3 * d.vertices + float(kind.split()[1])
    elif kind == "far body":
        d = NBodyData.plummer(n, seed=n)
        d.vertices[n // 3] = 1e7
    elif kind == "tight clusters":  # 1e-9 to 1e-11 of the extent, near the origin
        rng = np.random.default_rng(n)
        d.vertices *= np.repeat([1e-5, 1e-6, 1e-7, 1e-7], n // 4)[:, None]
        d.vertices += np.repeat(rng.uniform(-1e-4, 1e-4, (n // 32, 3)), 32, axis=0)
        d.vertices[0] = 1e4
    return d


def _walks(make_engine, d, lam):
    n = d.get_count()
    for split in (0, 1):
        e = make_engine(algo="bh", precision="fp64", distance_to_node_radius_ratio=lam)
        assert e.init(d)
        e.tune_set("bh.fp64_split", split)
        f, a = e.create_buffer(8 * 6 * n), np.zeros(6 * n)
        e.fcompute(0.0, e.get_y(), f)
        e.read_buffer(a, f)
        yield a[3 * n:].reshape(3, n).T, e.bh_counters()


@pytest.mark.parametrize("kind", ["offset 1e5", "offset 1e6", "far body", "tight clusters"])
@pytest.mark.parametrize("n", [1024, 4096, 32768])
@pytest.mark.parametrize("lam", [1.11, 2.0])
def test_same_nodes(make_engine, kind, n, lam):
    d = _data(kind, n)
    (a, ca), (b, cb) = _walks(make_engine, d, lam)
    assert ca == cb
    rows = np.unique(np.linspace(0, n - 1, 1024).astype(int))
    scale = np.array([(d.mass / np.maximum(((d.vertices - p) ** 2).sum(1), 1e-8)).sum()
                      for p in d.vertices[rows]])
    assert np.all(np.abs(a - b)[rows] <= (7e-15 + 2 * n * 2.0 ** -53) * scale[:, None])
