"""The segments of the residual solver's radial lines (csrc/line_role.cuh, solver.cu): a block's warps in groups of
one warp per segment, where the segments need not divide the warps. On the CPU the role of every warp for every
number of segments; on the GPU solves at 3, 5, 6 and 7 segments against the oracle's application of the
operator, by test_gpu_solver.py's bar (twice max(1e-10, 8 floor) on ||b - A p|| / ||b||)."""
import subprocess

import pytest

from atjup_b200 import build, synthetic
from atjup_b200.params import PREC_FP64, PREC_MIXED, SOLVE_RESIDUAL
from helpers import gpu_from, oracle_from, synthetic_case

SRC = r"""
#include <cstdio>
#include "line_role.cuh"
using namespace atjup;
int main() {
    int bad = 0;
    for (int S = 1; S <= LWARPS; S++) {
        int with_role = 0;
        bool seen[LWARPS][LWARPS] = {};
        for (int w = 0; w < LWARPS; w++) {
            const LineRole r = line_role(w, S);
            // the warps whose maps and sums the kernel's loops read: w0 .. w0 + S - 1
            if (r.s < 0 || r.s >= r.S || r.w0 < 0 || r.w0 + r.S > LWARPS || w != r.w0 + r.s) bad++;
            if (!r.on) { bad += r.S != 1; continue; }
            with_role++;
            if (r.S != S || r.group >= LWARPS / S || seen[r.group][r.s]) bad++;
            else seen[r.group][r.s] = true;
        }
        bad += with_role != LWARPS / S * S;
    }
    printf("%d\n", bad);
}
"""


def test_roles_stay_in_the_block(tmp_path):
    src, exe = tmp_path / "r.cpp", tmp_path / "r"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-I", str(build.CSRC), "-o", str(exe), str(src)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.strip() == "0"


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("im, segments", [(27, 3), (47, 5), (57, 6), (67, 7)])
def test_residual_solve_segments(im, segments, prec):
    from test_gpu_solver import _rel_residual
    assert (im - 2 + 9) // 10 == segments
    shape = (im, 21, 67)
    p, g, f = synthetic_case(*shape)
    b = synthetic.poisson_rhs(*shape, seed=3)
    o = oracle_from(p, g, f)
    m = gpu_from(p, g, f)
    try:
        m.set_solve_rhs(b)
        st = m.pressure_solver(mode=SOLVE_RESIDUAL, rel_tol=1e-10, max_iter=3000, precision=prec,
                               external_rhs=True)
        assert st.rel_residual <= max(1e-10, 8 * st.rel_floor)
        assert _rel_residual(o, m.download("p_dyn"), b) <= 2 * max(1e-10, 8 * st.rel_floor)
    finally:
        m.close()
