"""Plans with a fixed parameter, whose solves keep kernels of their own: one thread
per matrix and 2, 4 and 8 lanes in the full rounds, the lane-split rounds, and the
tail kernels.  Against the oracle by the bar of test_gpu_inversion.py: the share
of pixels that match it, and that reach 1.05 of its chi^2, beside the oracle's own
shares under a one-ulp change of the input."""
import numpy as np
import pytest

import me_b200
import me_maps
import oracle_bind as ob
from test_gpu_inversion import CHUNK, agreement, invert_chunks, ulp_perturb

pytestmark = pytest.mark.gpu
NAME = "fe15648_64x64"
FIXED = {"Damp_fixed": "YES"}

# (max_group, tail_slots, svd_lanes)
MODES = {"one_thread": (1, 0, 1), "two_lanes": (1, 0, 2), "four_lanes": (1, 0, 4),
         "eight_lanes": (1, 0, 8), "lane_split": (32, 0, 1), "tail": (1, -1, 1)}


@pytest.fixture(scope="module")
def fixed_map():
    lam = me_maps.wavelengths(NAME)
    ctl = me_maps.control_text(NAME, precision="FP64", extra=FIXED)
    orc = ob.Oracle(me_b200.parse_config_text(ctl), lam)
    npix = 4096
    prof = me_maps.add_noise(orc.synth_many(me_maps.draw_parameters(NAME, npix, 33)), 1e-3, 33)
    base = ob.oracle_invert_chunks(ctl, lam, prof, CHUNK)
    pert = ob.oracle_invert_chunks(ctl, lam, ulp_perturb(prof), CHUNK)
    return lam, prof, base, agreement(pert, base)


@pytest.mark.parametrize("mode", list(MODES))
@pytest.mark.parametrize("prec", ["FP64", "FP32"])
def test_against_the_oracle(fixed_map, prec, mode):
    lam, prof, base, (s_same, s_within, _) = fixed_map
    cfg = me_b200.parse_config_text(me_maps.control_text(NAME, precision=prec, extra=FIXED))
    with me_b200.Plan(cfg, lam) as plan:
        plan.max_group, plan.tail_slots, plan.svd_lanes = MODES[mode]
        res, stats = invert_chunks(plan, prof)
    same, within, med = agreement(res, base)
    print(f"{prec} {mode}: identical {same:.3f} (self {s_same:.3f}), chi2<=1.05x {within:.3f} "
          f"(self {s_within:.3f}), median ratio {med:.6f}")
    assert sum(st["valid"] - st["redo_pixels"] for st in stats) == np.sum(base[:, 9] > 0)
    assert abs(med - 1) < 1e-3
    assert within >= s_within - 0.02
    if prec == "FP64":
        assert same >= s_same - 0.03
    assert np.array_equal(res[:, 5], base[:, 5]) if prec == "FP64" else \
        np.allclose(res[:, 5], base[:, 5], rtol=1e-6)  # the fixed damping
