"""The Shapiro filters and the column balance at the edges of their tilings (pairs of meridians, chunks of
rows and levels, several blocks per row), over a random fluid floor that cuts every stencil, against
the CPU oracle. filters.cu is compiled without FMA contraction and keeps the reference's order of
operations, so the filters agree to the bit; the balance's row mean is summed in another order."""
import numpy as np
import pytest

from helpers import gpu_from, oracle_from, synthetic_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(6, 8, 9), (13, 16, 35), (17, 31, 259), (6, 9, 1027)],
                         ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("order, passes, use_topo", [(4, 1, True), (4, 2, False), (2, 1, True), (2, 2, False)])
def test_shapiro_shapes(shape, order, passes, use_topo):
    p, g, f = synthetic_case(*shape)
    rng = np.random.default_rng(5)
    topo = rng.integers(0, shape[0], shape[1:]).astype(np.int32)
    topo[rng.uniform(size=topo.shape) < 0.6] = 0
    g = dict(g, topo=topo)
    o, m = oracle_from(p, g, f), gpu_from(p, g, f)
    for n in ("u", "w"):
        o.shapiro(n, order, 0.7, passes, use_topo)
        m.shapiro(n, order, 0.7, passes, use_topo)
        assert np.array_equal(m.download(n), o.f[n]), n


@pytest.mark.parametrize("shape", [(6, 8, 9), (10, 16, 35), (9, 31, 387)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("zonal", [0, 1])
def test_balance_shapes(shape, zonal):
    p, g, f = synthetic_case(*shape)
    p.v_massbal_zonal = zonal
    o, m = oracle_from(p, g, f), gpu_from(p, g, f)
    o.call("ora_balance_column_v")
    m.balance_column_v()
    v = m.download("v")
    assert np.abs(v - o.f["v"]).max() <= 1e-14 * np.abs(o.f["v"]).max()
