"""Models of different boxes in turn: each model's projection launches after another's was set up, whatever shared memory
their bands take, and equals the oracle's bit for bit."""
import numpy as np
import pytest

from helpers import gpu_from, oracle_from, synthetic_case

pytestmark = pytest.mark.gpu


# two of one form each: a warp per row (58 and 20 KB a block), words over the warps (156 and 24 KB)
@pytest.mark.parametrize("shapes", [((9, 114, 127), (9, 37, 49)), ((7, 119, 361), (7, 119, 33))], ids=["rows", "words"])
def test_models_in_turn(shapes):
    cases = []
    try:
        for im, jm, km in shapes:
            P, grid, fields = synthetic_case(im, jm, km, seed=im + jm + km)
            P.cone_proj_margin, P.cone_proj_div = 200, 3
            m = gpu_from(P, grid, fields)
            m.cone_stats()                       # sets the projection up
            cases.append((m, oracle_from(P, grid, fields)))
        for m, o in cases:
            want = o.cone_project()
            m.cone_project()
            assert np.array_equal(m.cone_stats()[1], want)
            for n in ("v", "w"):
                assert np.array_equal(m.download(n), o.f[n]), n
    finally:
        for m, _ in cases:
            m.close()
