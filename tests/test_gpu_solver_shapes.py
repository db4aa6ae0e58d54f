"""The residual solver's kernels at the edges of their tilings, against the CPU oracle's application of
the operator: one and several segments per radial line (ten levels each) and a line too long for
them, rings of an even and an odd half, a ring whose transform tables do not fit shared memory, and
few rows. The bar is test_gpu_solver.py's: twice max(1e-10, 8 floor) on ||b - A p|| / ||b||. The
extreme shapes have no obstacle: it would fill most of them, and the solve does not converge there."""
import numpy as np
import pytest

from atjup_b200 import synthetic
from atjup_b200.params import PREC_FP64, PREC_MIXED, SOLVE_RESIDUAL
from helpers import gpu_from, oracle_from, synthetic_case
from test_gpu_solver import _rel_residual

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("shape, cone", [((9, 8, 9), False), ((12, 21, 35), True), ((23, 34, 67), True),
                                         ((83, 12, 33), False), ((9, 21, 8193), False)],
                         ids=lambda s: "x".join(map(str, s)) if isinstance(s, tuple) else "")
def test_residual_solve_shapes(shape, cone, prec):
    p, g, f = synthetic_case(*shape)
    if not cone:
        g = dict(g, solid=np.zeros_like(g["solid"]), topo=np.zeros_like(g["topo"]))
    b = synthetic.poisson_rhs(*shape, seed=3)
    o = oracle_from(p, g, f)
    m = gpu_from(p, g, f)
    m.set_solve_rhs(b)
    st = m.pressure_solver(mode=SOLVE_RESIDUAL, rel_tol=1e-10, max_iter=3000, precision=prec,
                           external_rhs=True)
    tol = max(1e-10, 8 * st.rel_floor)
    assert st.rel_residual <= tol
    e = _rel_residual(o, m.download("p_dyn"), b)
    assert e <= 2 * tol, f"oracle residual {e:.3e} (solver {st.rel_residual:.3e}, {st.iterations} it)"
