"""Fitted profiles of maps with skipped pixels (mean intensity below Icriteria):
zeros there, without a look at parameters that no inversion wrote, and elsewhere
what synthesize gives for the fitted parameters.  Without a filter, and with one
on both sides of the rule that gives a thread a sub-wavelength or a whole
wavelength; skipped pixels first, last and in a row, so that a block's pixels,
and a wavelength whose sub-wavelengths straddle two batches, are live, skipped
or both.  The bounds are those of test_synth_blocks.py."""
import numpy as np
import pytest

import me_b200
import me_maps

pytestmark = pytest.mark.gpu
NAME = "fe15648_64x64"


@pytest.mark.parametrize("prec,tol", [("FP64", 1e-12), ("FP32", 5e-6)])
@pytest.mark.parametrize("nl,points,count", [(11, 1, 70), (7, 21, 70), (6, 63, 61), (33, 5, 61),
                                             (16, 3, 9473)])
def test_skipped_pixels(nl, points, count, prec, tol):
    extra = {"num_iter": "2"}
    if points > 1:
        extra["filter"] = f"76, {points}"
    cfg = me_b200.parse_config_text(me_maps.control_text(NAME, precision=prec, extra=extra))
    lam = 15648.5 + 0.04 * 60 / nl * (np.arange(nl) - (nl - 1) / 2)
    par = me_maps.draw_parameters(NAME, count, nl + points)
    dark = np.zeros(count, bool)
    dark[[0, count - 1]] = True
    dark[2:4] = True
    dark[20:59] = True
    with me_b200.Plan(cfg, lam) as plan:
        prof = me_maps.add_noise(plan.synthesize(par), 1e-3, count)
        masked = prof.copy()
        masked[dark] *= 1e-5
        for first in (masked, prof, masked):  # on fresh memory, and after a map without any
            res, fit, st = plan.invert(first, want_fit=True)
            live = ~dark if first is masked else np.ones(count, bool)
            assert st["valid"] - st["redo_pixels"] == live.sum()
            assert np.all(fit[~live] == 0) and np.all(res[~live] == 0)
            got = np.where(live[:, None], res[:, :9], par)
            want = plan.synthesize(got)
            assert np.max(np.abs(fit[live] - want[live])) <= tol
