"""The residual solver on long rings, whose transform tables with the kernels' own shared memory pass a launch's
default 48 KB: both sides of that size, of the size where the tables alone pass it, and rings in common use
(quarter-degree: 1440); and two models whose rings need different amounts, in turn. The bar is
test_gpu_solver.py's: twice max(1e-10, 8 floor) on ||b - A p|| / ||b||. No obstacle (it would fill so few rows)."""
import numpy as np
import pytest

from atjup_b200 import synthetic
from atjup_b200.params import PREC_FP64, PREC_MIXED, SOLVE_RESIDUAL
from helpers import gpu_from, oracle_from, synthetic_case
from test_gpu_solver import _rel_residual

pytestmark = pytest.mark.gpu


def case(ring):
    shape = (9, 12, ring + 1)
    p, g, f = synthetic_case(*shape)
    g = dict(g, solid=np.zeros_like(g["solid"]), topo=np.zeros_like(g["topo"]))
    m = gpu_from(p, g, f)
    b = synthetic.poisson_rhs(*shape, seed=3)
    m.set_solve_rhs(b)
    return m, oracle_from(p, g, f), b


def solve(m, o, b, prec):
    st = m.pressure_solver(mode=SOLVE_RESIDUAL, rel_tol=1e-10, max_iter=3000, precision=prec, external_rhs=True)
    tol = max(1e-10, 8 * st.rel_floor)
    assert st.rel_residual <= tol
    assert _rel_residual(o, m.download("p_dyn"), b) <= 2 * tol


@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("ring", [952, 954, 960, 1000, 1440, 1442, 1444])
def test_residual_solve_rings(ring, prec):
    m, o, b = case(ring)
    try:
        solve(m, o, b, prec)
    finally:
        m.close()


def test_two_rings_in_turn():
    cases = [case(ring) for ring in (3000, 1500)]
    try:
        for _ in range(2):
            for m, o, b in cases:
                solve(m, o, b, PREC_FP64)
    finally:
        for m, _, _ in cases:
            m.close()
