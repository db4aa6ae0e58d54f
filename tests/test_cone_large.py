"""A box whose bands take almost the shared memory a block can have, against the oracle bit for bit."""
import numpy as np
import pytest

from helpers import gpu_from, oracle_from, synthetic_case


@pytest.mark.gpu
def test_projection_of_a_large_box():
    im, jm, km = 6, 301, 181               # a box of 299 x 179: 206 KB a block
    P, grid, fields = synthetic_case(im, jm, km, seed=im + jm + km)
    P.cone_proj_margin, P.cone_proj_div = 200, 3
    o, m = oracle_from(P, grid, fields), gpu_from(P, grid, fields)
    try:
        want = o.cone_project()
        m.cone_project()
        assert np.array_equal(m.cone_stats()[1], want)
        for n in ("v", "w"):
            assert np.array_equal(m.download(n), o.f[n]), n
    finally:
        m.close()
