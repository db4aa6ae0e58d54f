"""Shells of thousands of levels on a small ring, past the sizes at which three fields' levels exceed one launch's
blocks (21845 levels) and a level's weight for all of them exceeds a block's shared memory (6144): the filters
against the oracle bit for bit, and the filters' and the balance's transposes by the dot product
<A d, l> = <d, A' l>, to 1e-12 of the product of the norms."""
import numpy as np
import pytest

from atjup_b200.params import LIN_BALANCE, LIN_FIELDS, LIN_SHAPIRO
from helpers import gpu_from, oracle_from, synthetic_case

pytestmark = pytest.mark.gpu


def deep(im):
    """an (im, 8, 9) shell: the fields of a shallow one repeated upward, with a floor of its own"""
    p, g, f = synthetic_case(13, 8, 9, seed=3)
    p.im = im
    rep = lambda a: np.ascontiguousarray(np.resize(a, (im,) + a.shape[1:]))
    f = {n: rep(a) if getattr(a, "ndim", 0) == 3 else a for n, a in f.items()}
    rad = g["rad"][0] + p.dr * np.arange(im) / im
    topo = np.zeros_like(g["topo"])
    topo[3:5, 2:6] = 4
    solid = (np.arange(im)[:, None, None] < topo[None]).astype(np.uint8)
    g = dict(g, rad=rad, solid=solid, topo=topo,
             **{n: rep(g[n]) for n in ("cell_vbar0", "cell_ubar0") if g.get(n) is not None})
    return p, g, f


def test_filters_of_three_fields():
    from atjup_b200.gpu import GpuModel
    p, g, f = deep(22000)
    m = GpuModel(p, g)
    o = oracle_from(p, g, f)
    rng = np.random.default_rng(4)
    import torch
    x = {n: rng.standard_normal(m.shape) for n in ("u", "v", "w")}
    pitch = m.field_ptr("t")[1]
    d = [torch.zeros((p.im, p.jm, pitch), dtype=torch.float64, device="cuda") for _ in LIN_FIELDS]
    for n, a in x.items():
        d[LIN_FIELDS.index(n)][:, :, :p.km] = torch.from_numpy(a).cuda()
    try:
        m.iteration_tlm(d, 3, False, LIN_SHAPIRO)          # the filters are linear: their own passes
        for n, a in x.items():
            o.f[n][...] = a
            o.shapiro(n, 4, p.shapiro_strength, p.shapiro_inloop, True)
            assert np.array_equal(d[LIN_FIELDS.index(n)][:, :, :p.km].cpu().numpy(), o.f[n]), n
    finally:
        m.close()


@pytest.mark.parametrize("im", [127, 128, 129, 6200, 22000])
@pytest.mark.parametrize("zonal", [0, 1])
def test_transposes(im, zonal):
    import torch
    from atjup_b200.gpu import GpuModel
    p, g, f = deep(im)
    p.v_massbal_zonal = zonal
    m = GpuModel(p, g)
    pitch = m.field_ptr("t")[1]
    gen = torch.Generator(device="cuda").manual_seed(im)
    def fields():
        x = [torch.zeros((p.im, p.jm, pitch), dtype=torch.float64, device="cuda") for _ in LIN_FIELDS]
        for a in x:
            a[:, :, :p.km] = torch.randn((p.im, p.jm, p.km), generator=gen, dtype=torch.float64, device="cuda")
        return x
    dot = lambda a, b: sum(float((x * y).sum()) for x, y in zip(a, b))
    try:
        d, lam = fields(), fields()
        for parts in (LIN_SHAPIRO, LIN_BALANCE):
            ad, al = [x.clone() for x in d], [x.clone() for x in lam]
            m.iteration_tlm(ad, 3, False, parts)
            m.iteration_adjoint(al, 3, False, parts)
            lhs, rhs = dot(ad, lam), dot(d, al)
            size = float(np.sqrt(dot(ad, ad) * dot(lam, lam)))
            assert abs(lhs - rhs) <= 1e-12 * size
    finally:
        m.close()
