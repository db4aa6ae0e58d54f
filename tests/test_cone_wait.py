"""A level's solve whose wait for a neighbour block's row gives up: the level's winds are NaN, nothing else changes,
the statistics say so with an error, and the next call is the one that would have followed, bit for bit. The
limit of the wait is set to 0 polls, so that every one of them runs out."""
import numpy as np
import pytest

from helpers import gpu_from, oracle_from, synthetic_case

pytestmark = pytest.mark.gpu


def box_cells(P, solid, level):
    """the fluid cells of the level's box"""
    j, k = np.nonzero(solid[level])
    M, (_, jm, km) = P.cone_proj_margin, solid.shape
    box = np.zeros(solid.shape, bool)
    box[level, max(1, j.min() - M):min(jm - 2, j.max() + M) + 1, max(1, k.min() - M):min(km - 2, k.max() + M) + 1] = True
    return box & (solid == 0)


@pytest.mark.parametrize("im,jm,km,margin,div", [(9, 37, 49, 40, 3), (8, 33, 41, 4, 2), (8, 33, 41, 40, 0), (9, 114, 49, 100, 3)])
def test_wait_that_gives_up(im, jm, km, margin, div):
    from atjup_b200.gpu import AtjupError
    P, grid, fields = synthetic_case(im, jm, km, seed=im + jm + km)
    P.cone_proj_margin, P.cone_proj_div = margin, div
    o, m = oracle_from(P, grid, fields), gpu_from(P, grid, fields)
    solid = np.asarray(grid["solid"]).reshape(im, jm, km)
    try:
        want = o.cone_project()
        m.cone_project()
        levels, got = m.cone_stats()
        assert np.array_equal(got, want)
        m.cone_wait_limit(0)
        m.cone_project()
        with pytest.raises(AtjupError, match="gave up on level") as e:
            m.cone_stats()
        assert e.value.code == 5
        lost = np.zeros(solid.shape, bool)
        for level in levels:
            lost |= box_cells(P, solid, level)
        lost[:, :, km - 1] = lost[:, :, 0]                # the seam copy
        for n in ("v", "w"):
            x, old = m.download(n), o.f[n].copy()
            old[:, :, km - 1] = old[:, :, 0]
            assert np.array_equal(np.isnan(x), lost), n
            assert np.array_equal(x[~lost], old[~lost]), n
        m.cone_wait_limit(65536)
        for n in ("v", "w"):
            m.upload(n, o.f[n])
        want = o.cone_project()
        m.cone_project()
        assert np.array_equal(m.cone_stats()[1], want)
        for n in ("v", "w"):
            assert np.array_equal(m.download(n), o.f[n]), n
    finally:
        m.close()
