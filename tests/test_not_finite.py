"""Pixels whose parameters are not finite: a profile of one intensity at all
wavelengths has no velocity by its centre of gravity (0 / 0 in the initial
guess), and parameters given to the synthesis can be anything.  Such a pixel's
values are its own affair; the calls end, and every other pixel is what it is
without them."""
import numpy as np
import pytest

import me_b200
import me_maps

pytestmark = pytest.mark.gpu
NAME = "fe15648_64x64"


def _setup(prec, points, fixed=False):
    extra = {"num_iter": "4", "num_run": "2"}
    if points > 1:
        extra["filter"] = f"76, {points}"
    if fixed:
        extra["Damp_fixed"] = "YES"
    cfg = me_b200.parse_config_text(me_maps.control_text(NAME, precision=prec, extra=extra))
    nl = 11
    return cfg, 15648.5 + 0.24 * (np.arange(nl) - (nl - 1) / 2)


@pytest.mark.parametrize("prec", ["FP64", "FP32"])
@pytest.mark.parametrize("points", [1, 5])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_synthesis(prec, points, value):
    cfg, lam = _setup(prec, points)
    par = me_maps.draw_parameters(NAME, 36, 3)
    bad = par.copy()
    for k in range(9):
        bad[4 * k + 1, k] = value
    rest = np.ones(36, bool)
    rest[1::4] = False
    with me_b200.Plan(cfg, lam) as plan:
        if prec == "FP32":
            plan.faddeeva = 0  # the regions and Alg-916, as FP64 has them
        want, jac = plan.synthesize_jacobian(par, 0.1)
        got, gjac = plan.synthesize_jacobian(bad, 0.1)
        np.testing.assert_array_equal(got[rest], want[rest])
        np.testing.assert_array_equal(gjac[rest], jac[rest])
        np.testing.assert_array_equal(plan.synthesize(bad)[rest], plan.synthesize(par)[rest])


@pytest.mark.parametrize("prec", ["FP64", "FP32"])
@pytest.mark.parametrize("points,fixed", [(1, False), (1, True), (5, False)])
@pytest.mark.parametrize("group,tail", [(1, 0), (32, 0), (1, -1)])
def test_flat_profiles(prec, points, fixed, group, tail):
    cfg, lam = _setup(prec, points, fixed)
    par = me_maps.draw_parameters(NAME, 40, 5)
    with me_b200.Plan(cfg, lam) as plan:
        prof = me_maps.add_noise(plan.synthesize(par), 1e-3, 5)
        plan.max_group, plan.tail_slots = group, tail
        want, wfit, _ = plan.invert(prof, want_fit=True)
        more = np.concatenate([prof, np.zeros((3, 4, prof.shape[2]))])
        more[40:, 0] = 1.0           # (last: their chi^2 is carried to no other pixel)
        more[41, 1:] = 0.01
        more[42, 1, 2] = np.nan
        plan.carry_chisq = 0.0
        got, gfit, st = plan.invert(more, want_fit=True)
        plan.carry_chisq = 0.0
        want, wfit, _ = plan.invert(prof, want_fit=True)
        np.testing.assert_array_equal(got[:40], want)
        np.testing.assert_array_equal(gfit[:40], wfit)
