"""The symmetric ensemble kernel's units of few and of many tiles: the tiles'
FP32 sums are the same, only where the two-word additions of up to 32 tiles and
8 ranges begin differs.  Each such addition keeps the rounding error of the
high word and rounds the low word, at most 2^-24 of the high one, to 24 bits:
40 of them differ by at most 40 2^-47 A, A the sum of the absolute terms
m / (r^2 + eps^2)."""
import numpy as np
import pytest

from nbody_gb300.data import NBodyData
from nbody_gb300.ensemble import Ensemble

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("g", [1, 2])
@pytest.mark.parametrize("masses", ["equal", "drawn"])
@pytest.mark.parametrize("edges", [[1, 2, 127, 128, 129], [255, 256, 257, 511, 512, 513], [2049]])
def test_unit_lengths_agree(gpulib, g, masses, edges):
    sizes = edges + [4096] * 30
    rng = np.random.default_rng(len(edges))
    systems = []
    for k, n in enumerate(sizes):
        d = NBodyData.plummer(n, seed=k + 1)
        if masses == "drawn":
            d.mass = d.mass * rng.uniform(0.5, 1.5, n)
        systems.append(d)
    out = []
    for blocks in (0, 1):  # 1: a quarter of the CTAs, units of several tiles
        ens = Ensemble(softening=1e-2)
        ens.tune_set("ensemble.pairs_per_lane", g)
        ens.tune_set("ensemble.blocks_per_sm", blocks)
        ens.init(systems)
        f = ens.fcompute()
        assert np.array_equal(f, ens.fcompute())
        out.append(f.reshape(6, -1))
        ens.close()
    assert np.array_equal(out[0][:3], out[1][:3])
    off = 0
    for d in systems[:len(edges) + 2]:
        n = d.get_count()
        rows = rng.choice(n, size=min(n, 64), replace=False)
        scale = np.array([(d.mass / (((d.vertices - p) ** 2).sum(1) + 1e-4)).sum()
                          for p in d.vertices[rows]])
        diff = np.abs(out[0] - out[1])[3:, off + rows].max(0)
        assert (diff / scale).max() <= 40 * 2.0 ** -47
        off += n
