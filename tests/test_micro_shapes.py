"""The moist block's kernels at the ends of their ranges against the oracle, with the bars of test_micro.py: the
radiation at the most and the fewest levels and where its columns end in the middle of a block, the NH4SH
equilibrium from no NH4SH to far too much of it (the bracketed bisection makes the plain one's decisions, so it
has the plain one's bar)."""
import numpy as np
import pytest

from oracle_bridge import oracle_micro, rel_l2
from test_micro import MICRO_FIELDS, MICRO_TOL, SPECIES, gpu_micro, micro_case


def agree(got, want):
    for step in got:
        for n in MICRO_FIELDS + SPECIES:
            r = rel_l2(got[step][n], want[step][n])
            assert r <= MICRO_TOL, f"after {step}: {n} relative L2 {r:.3e}"


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(64, 9, 33), (6, 11, 97), (47, 8, 65), (48, 8, 31)])
@pytest.mark.parametrize("bottom,solar", [(0, 1), (1, 0)])
def test_radiation_levels(shape, bottom, solar):
    P, PH, MC, g, f = micro_case(*shape, seed=sum(shape))
    MC.rad_bottom, MC.solar_on = bottom, solar
    steps = ("radiation",)
    agree(gpu_micro(P, PH, MC, g, f, steps), oracle_micro(P, MC, g, f, steps))


@pytest.mark.gpu
@pytest.mark.parametrize("amount", [0.0, 1e-12, 1e-3, 1.0])
@pytest.mark.parametrize("cold", [0.0, 60.0])
def test_nh4sh_equilibrium(amount, cold):
    P, PH, MC, g, f = micro_case(12, 19, 45, seed=5)
    rng = np.random.default_rng(8)
    fluid = g["solid"].reshape(f["t"].shape) == 0
    f["nh4sh"] = np.where(fluid & (rng.random(f["t"].shape) < 0.7), amount * rng.random(f["t"].shape), 0.0)
    f["h2s"] = np.where(fluid, f["h2s"] * rng.choice([0.0, 1e-6, 1.0], f["t"].shape), 0.0)
    f["t"] = np.maximum(f["t"] - cold / P.t_ref, 40.0 / P.t_ref)
    steps = ("nh4sh_eq",)
    agree(gpu_micro(P, PH, MC, g, f, steps), oracle_micro(P, MC, g, f, steps))
