"""The Shapiro filter at each length of its threads' chunks (1 to 8 rows, 1, 5 and 15 levels, by the number of fields and
the shell), over a random fluid floor that cuts every stencil, against the CPU oracle to the bit: one field through
the filter's own call, three through the linear iteration's filter pass."""
import numpy as np
import pytest

from atjup_b200.params import LIN_FIELDS, LIN_SHAPIRO
from helpers import gpu_from, oracle_from, synthetic_case

pytestmark = pytest.mark.gpu


def chunks(shape, n):
    """rows and levels per thread, as filters.cu chooses them"""
    im, jm, km = shape
    pairs = (km - 1) // 2 + 1
    th = min(256, -(-pairs // 32) * 32)
    warps = -(-pairs // th) * (th // 32) * jm * im * n
    return min(8, -(-warps // 12500)), 1 if warps <= 4000 else 5 if warps <= 100000 else 15


@pytest.mark.parametrize("shape, one, three", [
    ((9, 21, 33), (1, 1), (1, 1)), ((17, 40, 97), (1, 1), (1, 5)), ((41, 62, 385), (2, 5), (5, 5)),
    ((41, 121, 385), (3, 5), (8, 15)), ((46, 53, 321), (2, 5), (4, 5))], ids=lambda v: "x".join(map(str, v)))
def test_filter_chunks(shape, one, three):
    import torch
    assert (chunks(shape, 1), chunks(shape, 3)) == (one, three)
    p, g, f = synthetic_case(*shape)
    rng = np.random.default_rng(6)
    topo = rng.integers(0, shape[0], shape[1:]).astype(np.int32)
    topo[rng.uniform(size=topo.shape) < 0.6] = 0
    g = dict(g, topo=topo)
    o, m = oracle_from(p, g, f), gpu_from(p, g, f)
    pitch = m.field_ptr("t")[1]
    d = [torch.zeros((p.im, p.jm, pitch), dtype=torch.float64, device="cuda") for _ in LIN_FIELDS]
    try:
        for n in ("u", "v", "w"):
            x = d[LIN_FIELDS.index(n)]
            x[:, :, :p.km] = torch.from_numpy(np.ascontiguousarray(o.f[n])).cuda()
        for order in (4, 2):
            m.shapiro("t", order, 0.7, 1, True)
            o.shapiro("t", order, 0.7, 1, True)
            assert np.array_equal(m.download("t"), o.f["t"]), order
        m.iteration_tlm(d, 3, False, LIN_SHAPIRO)
        for n in ("u", "v", "w"):
            o.shapiro(n, 4, p.shapiro_strength, p.shapiro_inloop, True)
            assert np.array_equal(d[LIN_FIELDS.index(n)][:, :, :p.km].cpu().numpy(), o.f[n]), n
    finally:
        m.close()


def test_overlapped_launches_are_ordered():
    """Passes in a chain, each launch overlapping the tail of the one before: 40
    passes, the fields in turn."""
    p, g, f = synthetic_case(13, 37, 49)
    o, m = oracle_from(p, g, f), gpu_from(p, g, f)
    try:
        for it in range(10):
            for n in ("u", "v", "w", "v"):
                o.shapiro(n, 4, 0.7, 1, True)
                m.shapiro(n, 4, 0.7, 1, True)
        for n in ("u", "v", "w"):
            assert np.array_equal(m.download(n), o.f[n]), n
    finally:
        m.close()


def test_filters_are_captured():
    """The filters issued on a stream under capture, replayed twice: the oracle's three passes (one before, two replayed)"""
    import torch
    p, g, f = synthetic_case(13, 37, 49)
    o, m = oracle_from(p, g, f), gpu_from(p, g, f)
    st = torch.cuda.Stream()
    try:
        m.set_stream(st.cuda_stream)
        graph = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        for n in ("u", "w"):
            m.shapiro(n, 4, 0.7, 1, True)
        m.synchronize()
        with torch.cuda.graph(graph, stream=st):
            for n in ("u", "w"):
                m.shapiro(n, 4, 0.7, 1, True)
        graph.replay()
        graph.replay()
        torch.cuda.synchronize()
        for n in ("u", "w"):
            for _ in range(3):
                o.shapiro(n, 4, 0.7, 1, True)
            assert np.array_equal(m.download(n), o.f[n]), n
    finally:
        m.synchronize()
        m.set_stream(None)
        m.close()
