"""The FP32 tail kernel pixel by pixel.

In two orders of the pixels: a pixel's way through the tail kernel has nothing to
do with the slot, the CTA or the pixels before it there, so its result is the
same bits.  A stale factor, a buffer taken too early or a slot loaded wrongly
would change it.  (One schedule of starts, which depend on the profile alone:
random ones would depend on a pixel's number.)

And each pixel's chi^2 is that of its own result: the oracle's profiles for the
fitted parameters, in FP64, give it.  FP32 profiles are within 5e-6 of those and
residuals at least the noise of 1e-3 in root mean square, so chi^2 agrees to
2 x 5e-6 / 1e-3 = 1e-2."""
import numpy as np
import pytest

import me_b200
import me_maps
import oracle_bind as ob

pytestmark = pytest.mark.gpu
NAME = "fe15648_64x64"
CASES = [(11, 1), (31, 1), (33, 1), (97, 1), (6, 21), (11, 3), (12, 63), (33, 5)]


def _case(nl, points, fixed, count, **more):
    extra = {k: str(v) for k, v in more.items()}
    if points > 1:
        extra["filter"] = f"76, {points}"
    if fixed:
        extra["Damp_fixed"] = "YES"
    cfg = me_b200.parse_config_text(me_maps.control_text(NAME, widen_bounds=True, extra=extra))
    lam = 15648.5 + 0.04 * 60 / nl * (np.arange(nl) - (nl - 1) / 2)
    par = me_maps.draw_parameters(NAME, count, nl + points)
    prof = me_maps.add_noise(ob.Oracle(cfg, lam).synth_many(par), 1e-3, nl)
    return cfg, lam, prof


def _invert(plan, prof):
    plan.carry_chisq = np.inf  # (no pixel's regularisation depends on another's chi^2)
    res, st = plan.invert(prof)
    assert st["redo_pixels"] == 0
    return res, st["launches"] - 4 * st["rounds"]


@pytest.mark.parametrize("nl,points", CASES)
@pytest.mark.parametrize("fixed", [False, True])
@pytest.mark.parametrize("tail", [-1, 4096])
def test_order_of_pixels(nl, points, fixed, tail):
    cfg, lam, prof = _case(nl, points, fixed, 900, num_run=1)
    order = np.random.default_rng(nl).permutation(900)
    with me_b200.Plan(cfg, lam) as plan:
        plan.max_group, plan.tail_slots = 1, tail
        a, tails = _invert(plan, prof)
        assert tails == 1
        b, _ = _invert(plan, prof[order])
        np.testing.assert_array_equal(b, a[order])
    pick = np.arange(0, 900, 9)
    fit = ob.Oracle(cfg, lam).synth_many(a[pick, :9])
    imean = prof[pick, 0].mean(axis=1)
    weights = np.array([cfg.weights[k] for k in range(4)])
    rest = (fit - prof[pick]) * weights[None, :, None] / (1e-2 * imean)[:, None, None]
    sums = np.abs(prof[pick]).sum(axis=2)
    norm = 1 + (weights[1:] ** 2 * sums[:, 1:] ** 2).sum(axis=1) / prof[pick, 0].sum(axis=1) ** 2
    chi = (rest ** 2).sum(axis=(1, 2)) / (4 * lam.size) / norm
    assert np.max(np.abs(a[pick, 9] / chi - 1.0)) < 1e-2
