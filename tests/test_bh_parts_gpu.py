"""The mixed-precision group walk with several warps per group ("bh.parts")
against one warp per group: the same accepted nodes (equal visit and
interaction counts, the same groups handed to the per-body walk), the same
FP32 terms, added in another order.

A list of at most 256 cells is summed in FP32 by four accumulators and then
folded with its rounding error kept, so an accumulator adds at most 64 terms
(cells with quadrupole terms: 128 in two accumulators, two additions each, so
128 additions) and two such sums differ by at most 2 (128 + 2) 2^-24 S with S
the sum of the absolute values of the terms.  Cells are accepted at d > 2 rho
(rho the cell's radius), so |M| / d^2 <= 2.25 times its bodies' sum of
m / r^2, and the quadrupole terms (3 m rho^2 / r^4 and 9 m rho^2 / r^4) add at
most three times the monopole's: S <= 9 A with A the body's sum of m / r^2."""
import numpy as np
import pytest

from nbody_gb300.data import NBodyData

pytestmark = pytest.mark.gpu

TOL = 2 * 130 * 2.0 ** -24 * 9


@pytest.mark.parametrize("n", [64, 128, 1024, 16384])
@pytest.mark.parametrize("order,npl", [(1, 2), (1, 1), (2, 1)])
@pytest.mark.parametrize("build", [0, 1])  # kd tree (no cap), Hilbert order (capped)
@pytest.mark.parametrize("cap", [0, 1, 700])
@pytest.mark.parametrize("softening", [0.0, 1e-2])
def test_parts_agree(make_engine, n, order, npl, build, cap, softening):
    d = NBodyData.plummer(n, seed=n)
    v = d.vertices
    rows = np.random.default_rng(n).choice(n, size=min(n, 256), replace=False)
    scale = np.array([(d.mass / np.maximum(((v - p) ** 2).sum(1) + softening ** 2, 1e-8)).sum()
                      for p in v[rows]])
    out = {}
    for parts in (1, 0, 2, 7, 16, 32, 16):  # (0: chosen, 7: rounded down)
        e = make_engine(algo="bh", precision="mixed", softening=softening,
                        distance_to_node_radius_ratio=2.0)
        e.tune_set("bh.order", order)
        e.tune_set("bh.walk_npl", npl)
        e.tune_set("bh.build", build)
        e.tune_set("bh.test_cap", cap)
        e.tune_set("bh.parts", parts)
        assert e.init(d)
        f = e.create_buffer(8 * 6 * n)
        e.fill_buffer(f, 1e10)
        e.fcompute(0.0, e.get_y(), f)
        a = np.zeros(6 * n)
        e.read_buffer(a, f)
        handed = e.bh_fallback_groups()  # (before bh_counters, which clears both)
        counts = (e.bh_counters(), handed)
        e.close()
        if parts in out:  # equal trees give equal forces
            assert np.array_equal(a, out[parts])
            continue
        out[parts] = a
        if parts == 1:
            want, want_counts = a, counts
            continue
        assert np.array_equal(a[:3 * n], want[:3 * n])
        err = np.abs(a - want).reshape(6, n)[3:, rows].max(0) / scale
        assert err.max() < TOL, (parts, err.max())
        assert counts[1] == want_counts[1]
        if counts[1] == 0:
            assert counts == want_counts
