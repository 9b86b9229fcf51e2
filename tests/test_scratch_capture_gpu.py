"""A caller may capture fcompute on the engine's stream and replay it at any
time in the engine's life, also after another call has outgrown the scratch
that the captured launches read: the block they read is kept."""
import numpy as np
import pytest

from nbody_gb300 import _lib
from nbody_gb300.data import NBodyData

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1000, 3000, 20000])
def test_replay_after_scratch_growth(make_engine, n):
    import torch
    d = NBodyData.plummer(n, seed=n)
    e = make_engine(precision="mixed", softening=1e-2)
    assert e.init(d)
    f = e.create_buffer(8 * 6 * n)

    def read():
        a = np.zeros(6 * n)
        e.read_buffer(a, f)
        return a

    e.fcompute(0.0, e.get_y(), f)
    want = read()
    stream = torch.cuda.ExternalStream(_lib.load().nbg_stream(e.handle))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        e.fcompute(0.0, e.get_y(), f)
    e.statistics()  # needs a larger block than the direct sum
    e.fill_buffer(f, 1e10)
    with torch.cuda.stream(stream):
        graph.replay()
    stream.synchronize()
    # (atomic adds of the mixed sum: equal but for the order of FP64 adds)
    np.testing.assert_allclose(read(), want, rtol=1e-12, atol=1e-12 * np.abs(want).max())
