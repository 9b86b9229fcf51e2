"""The mixed-precision direct sum's kernel for small systems ("direct.small")
against the symmetric kernel.

Both take the same FP32 positions, so their pair terms differ by the rounding
of at most four products each (8 units of 2^-24), and both fold their FP32
sums with the rounding error kept after at most 128 terms (and the symmetric
kernel adds at most 36 partial sums of a B body in FP32): per component the
results differ by at most (8 + 128 + 36) 2^-24 A, A the body's sum of
m / (r^2 + eps^2)."""
import numpy as np
import pytest

from nbody_gb300.data import NBodyData

pytestmark = pytest.mark.gpu

TOL = 172 * 2.0 ** -24


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 63, 64, 65, 129, 1000, 2049, 4099, 8191, 8192, 8193])
@pytest.mark.parametrize("masses", ["equal", "drawn", "both signs"])
@pytest.mark.parametrize("eps", [0.0, 1e-2])
def test_small_kernel(make_engine, n, masses, eps):
    d = NBodyData.plummer(n, seed=n)
    rng = np.random.default_rng(n)
    if masses != "equal":
        d.mass = d.mass * rng.uniform(0.5, 1.5, n)
    if masses == "both signs":
        d.mass = d.mass * rng.choice([-1.0, 1.0], n)
    if n > 4:
        d.vertices[3] = d.vertices[1]  # two bodies at one point
    rows = rng.choice(n, size=min(n, 300), replace=False)
    m = np.abs(d.mass)
    scale = np.array([(m / np.maximum(((d.vertices - p) ** 2).sum(1) + eps * eps, 1e-8)).sum()
                      for p in d.vertices[rows]])
    out = []
    for small in (1, 0):
        e = make_engine(precision="mixed", softening=eps)
        e.tune_set("direct.small", small)
        assert e.init(d)
        f = e.create_buffer(8 * 6 * n)
        for _ in range(2):  # (f is overwritten, not added to)
            e.fill_buffer(f, 1e10)
            e.fcompute(0.0, e.get_y(), f)
        a = np.zeros(6 * n)
        e.read_buffer(a, f)
        out.append(a)
    assert np.array_equal(out[0][:3 * n], out[1][:3 * n])
    err = np.abs(out[0] - out[1]).reshape(6, n)[3:, rows].max(0) / scale
    assert err.max() <= TOL
