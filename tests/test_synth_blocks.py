"""The synthesis entry points at the edges of their split into blocks: a pixel
alone, counts around the block's pixels, grids shorter and longer than a
block's threads, and instrument filters on both sides of the rule that gives a
thread a sub-wavelength or a whole wavelength.  Against the oracle on a sample
of the pixels, within the bounds of test_gpu_kernels.py, and against the same
pixels one at a time: each pixel's arithmetic is its own, so those are equal."""
import numpy as np
import pytest

import me_b200
import me_maps
import oracle_bind as ob

pytestmark = pytest.mark.gpu


def _setup(nl, points, prec):
    name = "fe15648_64x64"
    extra = {"filter": f"76, {points}"} if points > 1 else {}
    cfg = me_b200.parse_config_text(me_maps.control_text(name, precision=prec, extra=extra))
    lam = 15648.5 + 0.04 * (np.arange(nl) - (nl - 1) / 2)
    return name, cfg, lam


@pytest.mark.parametrize("prec,tol", [("FP64", 1e-12), ("FP32", 5e-6)])
@pytest.mark.parametrize("nl,points,count", [(60, 1, 1), (60, 1, 33), (6, 1, 593), (129, 1, 1185),
                                             (7, 21, 1), (7, 21, 33), (6, 63, 40),
                                             (16, 3, 9471), (16, 3, 9473)])
def test_profiles_and_jacobians(nl, points, count, prec, tol):
    name, cfg, lam = _setup(nl, points, prec)
    par = me_maps.draw_parameters(name, count, nl + count)
    pick = np.unique(np.linspace(0, count - 1, 7).astype(int))
    with me_b200.Plan(cfg, lam) as plan:
        prof = plan.synthesize(par)
        small = par[:1200]
        pj, jac = plan.synthesize_jacobian(small, 0.1)
        np.testing.assert_array_equal(
            plan.synthesize_jacobian(par[pick[:3]], 0.1)[1][0], jac[pick[0]])
        one = np.concatenate([plan.synthesize(par[i:i + 1]) for i in pick])
    want = ob.Oracle(cfg, lam).synth_many(par[pick])
    assert np.max(np.abs(prof[pick] - want)) < tol
    assert np.max(np.abs(one - want)) < tol
    # with and without the Jacobian two compiled kernels: rounding apart
    assert np.max(np.abs(pj - prof[:1200])) < tol
    assert np.all(np.isfinite(jac)) and jac.shape == (small.shape[0], 4, 9, nl)
    if points == 1 or points == 21:
        np.testing.assert_array_equal(one, prof[pick])
