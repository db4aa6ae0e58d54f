"""The census of the convective adjustment, whose bounds settle many pairs without solving them: every counter
against the oracle, which solves all of them, with the virtual-temperature options that change the bounds and
on shells that end in the middle of a block. The counters are equal but for pairs within rounding of the
1e-7 K threshold; the bar is the repository's for columns, 0.5 %."""
import numpy as np
import pytest

from atjup_b200.params import resolve_mca
from moist_cases import gpu_moist_model, synthetic_moist_case
from oracle_bridge import MCA_ENV, oracle_mca
import ref_dump as R

FIELDS = R.MCA_FIELDS


@pytest.mark.gpu
@pytest.mark.parametrize("ledoux,loading", [(1, 1), (1, 0), (0, 0)])
@pytest.mark.parametrize("shape,wet,unstable", [((41, 23, 37), 1.0, True), ((17, 19, 131), 1.0, False),
                                                ((12, 11, 29), 20.0, False), ((23, 13, 33), 0.0, True)])
def test_census_counts(shape, wet, unstable, ledoux, loading):
    P, PH, MC, g, f = synthetic_moist_case(*shape, seed=sum(shape))
    for n in FIELDS[1:]:
        f[n] = f[n] * wet
    if unstable:
        f = R.perturb_unstable(f, g["solid"], f["layer_heights"], seed=3)
    M = resolve_mca({**MCA_ENV, "ATJUP_MCA_LEDOUX": str(ledoux), "ATJUP_MCA_LOADING": str(loading)})
    want, wst = oracle_mca(P, MC, M, g, f)
    m = gpu_moist_model(P, PH, MC, g, f)
    m.set_mca(M)
    gst = m.mca()
    got = {n: m.download(n) for n in FIELDS}
    m.close()
    for n in ("columns", "unstable_t", "held", "skipped"):
        assert abs(gst[n] - wst[n]) <= 5e-3 * wst[n] + 1, (n, gst, wst)
    flipped = np.any([np.any(np.abs(got[n] - want[n]) > 1e-12 * max(np.abs(want[n]).max(), 1e-300), axis=0)
                      for n in FIELDS], axis=0)
    assert flipped.mean() <= 5e-3
