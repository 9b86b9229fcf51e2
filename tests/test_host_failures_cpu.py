"""The library's host code when a CUDA call fails, in a process whose CUDA
runtime is tests/fakes/fake_cudart.c: no GPU, no kernel runs."""
import shutil
import subprocess
import sys
import textwrap

import pytest

from conftest import ROOT

PRELUDE = """
import ctypes as C, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from nbody_gb300 import _lib
from nbody_gb300._lib import NbgError
from nbody_gb300.data import NBodyData
from nbody_gb300.engine import create_engine
from nbody_gb300.ensemble import Ensemble
lib, fake = _lib.load(), C.CDLL(None)
fake.fake_launches.restype = C.c_char_p
fake.fake_used.restype = fake.fake_block.restype = C.c_size_t
fake.fake_block.argtypes = [C.c_void_p]

def put(name, value, kind=C.c_int):
    kind.in_dll(fake, "fake_" + name).value = value

def memory(value):
    put("memory", value, C.c_size_t)

def launched():
    return fake.fake_launches().decode().split()

def error_of(call):
    try:
        call()
    except NbgError as e:
        return str(e)
    return None
"""


@pytest.fixture(scope="module")
def run(gpulib, tmp_path_factory):
    cc = shutil.which("gcc")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = str((ROOT / nvcc).resolve().parent.parent / "include")
    if cc is None:
        pytest.skip("no host compiler")
    so = tmp_path_factory.mktemp("fake") / "fake_cudart.so"
    r = subprocess.run([cc, "-shared", "-fPIC", "-O1", "-Wall", "-Wextra", "-Werror", "-I", include,
                        str(ROOT / "tests" / "fakes" / "fake_cudart.c"), "-o", str(so)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def _run(code):
        r = subprocess.run([sys.executable, "-c", PRELUDE + textwrap.dedent(code), str(ROOT)],
                           capture_output=True, text=True, timeout=300,
                           env={"LD_PRELOAD": str(so), "PATH": "/usr/bin:/bin"})
        assert r.returncode == 0, r.stdout + r.stderr[-3000:]

    return _run


@pytest.mark.parametrize("n", [700, 9000])
@pytest.mark.parametrize("fails", ["sync", "copy"])
def test_state_arrays_keep_their_contents(run, fails, n):
    """A get_state that reports an error has written nothing to the caller's
    arrays."""
    run(f"""
    ens = Ensemble()
    ens.init([NBodyData.plummer({n}, seed=1)])
    v, u = (np.random.default_rng(k).normal(size=({n}, 3)) for k in (1, 2))
    want = v.copy(), u.copy()
    put("{fails}_error", 719)
    assert lib.nbg_ensemble_get_state(ens._h, v.ctypes.data, u.ctypes.data) != 0
    assert np.array_equal(v, want[0]) and np.array_equal(u, want[1])
    """)


@pytest.mark.parametrize("n,kernels", [(1, 0), (8192, 0), (8193, 1)])
def test_state_of_a_small_batch_needs_no_kernel(run, n, kernels):
    run(f"""
    ens = Ensemble()
    ens.init([NBodyData.uniform_cube({n}, seed=1)])
    launched()
    ens.get_state()
    assert len(launched()) == {kernels}
    """)


@pytest.mark.parametrize("spare,kernel", [
    (2 ** 40, "ens_sym_kernel"),    # segments of two tiles
    (10 << 20, "ens_sym_kernel"),   # 24 bytes a body: one segment a range
    (1 << 20, "ens_force_kernel"),  # the other partials fit, these do not
    (-20 << 20, "ens_force_kernel"),  # none do
])
def test_ensemble_with_little_memory(run, spare, kernel):
    """A batch whose state fits is accepted, whatever is left for the symmetric
    kernel's partials; `spare` bytes beyond the state and the B partials."""
    run(f"""
    systems = [NBodyData.uniform_cube(16384, seed=k) for k in range(4)]
    ens = Ensemble(use_graph=False)
    ens.tune_set("ensemble.symmetric", 0)
    ens.init(systems)
    state = fake.fake_used()
    partials = 4 * 16384 * (16384 // 512) * 12
    ens.tune_set("ensemble.symmetric", 1)   # with all the memory there is
    launched()
    ens.step(1)
    assert any("ens_sym_kernel" in k for k in launched())
    memory(state + partials + {spare})
    ens.init(systems)
    for call in (lambda: ens.step(1), lambda: ens.fcompute(), lambda: ens.autotune(1)):
        launched()
        call()
        assert any("{kernel}" in k for k in launched())
    assert fake.fake_used() <= state + partials + {spare}
    """)


def test_ensemble_without_a_configuration(run):
    """A tuning key whose shape cannot be had leaves a batch that says so and
    that another key makes whole again."""
    run("""
    ens = Ensemble()
    ens.init([NBodyData.uniform_cube(16384, seed=k) for k in range(4)])
    ens.step(1)
    memory(0)
    assert error_of(lambda: ens.tune_set("ensemble.symmetric", 0)) is not None
    launched()
    assert "not initialised" in error_of(lambda: ens.step(1))
    assert "not initialised" in error_of(lambda: ens.fcompute())
    assert launched() == []
    memory(2 ** 40)
    fake.cudaGetLastError()
    ens.tune_set("ensemble.symmetric", 0)
    ens.step(1)
    """)


@pytest.mark.parametrize("param", [dict(precision="fp64"), dict(precision="mixed")])
@pytest.mark.parametrize("clusters", [0, 1])
def test_tree_without_clusters(run, param, clusters):
    """A process whose SMs have no room for a cluster sorts in passes."""
    run(f"""
    put("clusters", {clusters})
    e = create_engine(dict({param}, engine="gb300", algo="bh"))
    assert e.init(NBodyData.uniform_cube(1024, seed=1))
    f = e.create_buffer(8 * 6 * 1024)
    for _ in range(2):
        e.fcompute(0.0, e.get_y(), f)
        names = launched()
        assert any("cluster_sort_kernel" in k for k in names) == bool({clusters})
        assert any("radix_scatter_kernel" in k for k in names) != bool({clusters})
        e.advise_time(0.0)
    """)


def test_scratch_of_captured_launches_is_kept(run):
    """A scratch block that captured launches read outlives its growth and is
    given back with the engine; one that none read is given back at once."""
    run("""
    def growth(captured):
        free = fake.fake_used()
        e = create_engine(dict(engine="gb300", precision="mixed", softening=1e-2))
        assert e.init(NBodyData.uniform_cube(20000, seed=1))
        f = e.create_buffer(8 * 6 * 20000)
        before = fake.fake_used()
        e.fcompute(0.0, e.get_y(), f)
        block = fake.fake_used() - before
        put("capturing", captured)
        e.fcompute(0.0, e.get_y(), f)
        put("capturing", 0)
        e.statistics()   # needs a larger block
        grown = fake.fake_used() - before
        e.close()
        assert fake.fake_used() == free
        return block, grown
    (b0, g0), (b1, g1) = growth(0), growth(1)
    assert b0 == b1 and b0 >= 20000 * 32 and g0 > b0
    assert g1 == g0 + b0
    """)
