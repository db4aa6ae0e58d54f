"""The projection's kernel forms over the boxes that choose between them, against the oracle bit for bit: a warp
per row (bands of 2 to 28 rows, at most 64 words a colour: odd and even widths, the widest, the fewest rows),
words over the block's warps (more rows, wider rows, bands of one row) and the box in HBM; two calls, the
second warm-started; with and without the divergence solve. The arithmetic is the reference's operation for
operation, so there is no tolerance."""
import numpy as np
import pytest

from helpers import gpu_from, oracle_from, synthetic_case

SHAPES = [
    # im, jm, km, margin, div
    (9, 37, 49, 40, 3),        # the whole shell's interior: 9 rows a block, 47 cells a row
    (9, 38, 51, 40, 1),
    (8, 10, 23, 40, 3),        # two rows a block
    (8, 33, 41, 4, 2),
    (9, 114, 49, 100, 3),      # 28 rows a block
    (7, 25, 127, 100, 3),      # 63 words a row
    (7, 25, 129, 100, 3),      # 65: words over the warps
    (7, 119, 33, 100, 3),      # 30 rows a block
    (8, 8, 33, 40, 3),         # bands of one and two rows
    (8, 33, 41, 40, 0),        # no divergence solve
    (6, 181, 361, 200, 2),     # a box that shared memory does not hold
]


@pytest.mark.gpu
@pytest.mark.parametrize("im,jm,km,margin,div", SHAPES)
def test_projection_equals_oracle(im, jm, km, margin, div):
    P, grid, fields = synthetic_case(im, jm, km, seed=im + jm + km)
    P.cone_proj_margin, P.cone_proj_div = margin, div
    o, m = oracle_from(P, grid, fields), gpu_from(P, grid, fields)
    rng = np.random.default_rng(3)
    try:
        for call in range(2):
            if call:
                for n in ("v", "w"):
                    a = (o.f[n] + 1e-3 * rng.standard_normal(o.f[n].shape)) * (o.g["solid"].reshape(o.f[n].shape) == 0)
                    o.f[n][...] = a
                    m.upload(n, a)
            want = o.cone_project()
            m.cone_project()
            levels, got = m.cone_stats()
            assert len(levels) > 0 and np.array_equal(got, want)
            for n in ("v", "w"):
                assert np.array_equal(m.download(n), o.f[n]), f"call {call}: {n}"
    finally:
        m.close()
