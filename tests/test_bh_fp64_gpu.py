"""The two FP64 Barnes-Hut walks against each other: the same acceptance
decisions (the same visit and interaction counts) and, per body, forces
within rounding.  With A = sum |m_j| / r_j^2 over all bodies as the scale of a
body's sum, the FP64 pipe's serial sum of k terms is within k 2^-53 A of exact
and the two-word sum within 7e-15 A (tests/test_direct_fp64_gpu.py derives
it)."""
import numpy as np
import pytest

from nbody_gb300.data import NBodyData

pytestmark = pytest.mark.gpu


def _data(kind, n):
    rng = np.random.default_rng(n)
    d = NBodyData.uniform_cube(n, side=2.0, seed=n)
    if kind == "plummer":
        d = NBodyData.plummer(n, seed=n)
    elif kind == "far clusters":
        d.vertices = 1e-3 * d.vertices + 1e3
        d.vertices[n // 2:] += [3e3, -5e3, 1e4]
    elif kind == "below the clamp":
        d.vertices *= 1e-6
    elif kind == "both signs":  # mass centres far outside the bodies' extent
        d.mass *= rng.choice([-1.0, 1.0], n)
    elif kind == "coincident":
        d.vertices[n // 3:2 * (n // 3)] = d.vertices[:2 * (n // 3) - n // 3]
    elif kind == "not finite":
        d.vertices[n // 2, 0] = np.nan
    return d


def _scale(d):
    m, v = np.abs(d.mass), d.vertices
    return np.array([(m / np.maximum(((v - p) ** 2).sum(1), 1e-8)).sum() for p in v])


@pytest.mark.parametrize("kind", ["cube", "plummer", "far clusters", "below the clamp", "both signs",
                                  "coincident", "not finite"])
@pytest.mark.parametrize("n", [1, 2, 16, 32, 64, 128, 1024, 4096])
@pytest.mark.parametrize("lam", [1.11, 2.0, 1e8])
def test_walks_agree(make_engine, kind, n, lam):
    d = _data(kind, n)
    out = []
    for split in (0, 1):
        e = make_engine(algo="bh", precision="fp64", distance_to_node_radius_ratio=lam,
                        tree_build_rate=2)
        assert e.init(d)
        e.tune_set("bh.fp64_split", split)
        f = e.create_buffer(8 * 6 * n)
        got = []
        for _ in range(2):  # a build, then a refit at other positions
            e.fill_buffer(f, 1e10)
            e.fcompute(0.0, e.get_y(), f)
            a = np.zeros(6 * n)
            e.read_buffer(a, f)
            got.append((a, e.bh_counters()))
            e.fmadd_inplace(e.get_y(), e.get_y(), 0.25)
            e.advise_time(0.0)
        out.append(got)
    for step in range(2):
        (a, ca), (b, cb) = out[0][step], out[1][step]
        assert ca == cb
        assert np.array_equal(a[:3 * n], b[:3 * n], equal_nan=True)
        d2 = NBodyData(vertices=d.vertices * 1.25 ** step, mass=d.mass)
        # (a body that is not finite meets nothing and is met by none)
        bound = (7e-15 + 2 * n * 2.0 ** -53) * np.nan_to_num(_scale(d2), nan=np.inf)
        diff = np.abs(a - b)[3 * n:].reshape(3, n)
        assert np.array_equal(np.isnan(a), np.isnan(b))
        assert np.all(np.nan_to_num(diff) <= bound)


def test_repeats(make_engine):
    d = _data("plummer", 4096)
    e = make_engine(algo="bh", precision="fp64", distance_to_node_radius_ratio=2.0)
    assert e.init(d)
    f, a, b = e.create_buffer(8 * 6 * 4096), np.zeros(6 * 4096), np.zeros(6 * 4096)
    e.fcompute(0.0, e.get_y(), f)
    e.read_buffer(a, f)
    e.fcompute(0.0, e.get_y(), f)
    e.read_buffer(b, f)
    assert np.array_equal(a, b)
