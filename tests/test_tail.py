"""The FP32 tail kernel at the edges of its batches of points: grids that fill
a batch of 32 wavelengths exactly, leave a remainder or fall short of one, and
instrument filters whose sub-wavelengths straddle its batches of 96.  A map small
enough that every LM step after the first batch of rounds runs in the tail
kernel is inverted with it and with one-thread-per-pixel rounds throughout,
which the oracle pins (test_gpu_inversion.py).  The two forms sum in the same
order and differ by the compiler's contraction alone, FP32 rounding (1e-7 of
the normal matrix), which twelve iterations amplify on the pixels that the
LM's last-bit sensitivity catches (a quarter of a map) and leave alone
elsewhere: at least half the pixels agree to 1e-3 in chi^2, and the median
ratio is 1 to 1e-3."""
import numpy as np
import pytest

import me_b200
import me_maps
import oracle_bind as ob

pytestmark = pytest.mark.gpu
NAME = "fe15648_64x64"


def _invert(cfg, lam, prof, tail):
    with me_b200.Plan(cfg, lam) as plan:
        plan.max_group = 1
        plan.tail_slots = prof.shape[0] if tail else 0
        res, st = plan.invert(prof)
        runs = plan.last_counters(prof.shape[0])
    assert st["launches"] - 4 * st["rounds"] == (1 if tail else 0)
    return res, runs


@pytest.mark.parametrize("nl,points", [(11, 1), (31, 1), (32, 1), (33, 1), (64, 1), (97, 1),
                                       (6, 21), (11, 3), (12, 63), (33, 5)])
@pytest.mark.parametrize("fixed", [False, True])
def test_tail_matches_rounds(nl, points, fixed):
    extra = {"num_iter": "12"}
    if points > 1:
        extra["filter"] = f"76, {points}"
    if fixed:
        extra["Damp_fixed"] = "YES"
    cfg = me_b200.parse_config_text(me_maps.control_text(NAME, widen_bounds=True, extra=extra))
    lam = 15648.5 + 0.04 * 60 / nl * (np.arange(nl) - (nl - 1) / 2)
    par = me_maps.draw_parameters(NAME, 96, nl + points)
    prof = me_maps.add_noise(ob.Oracle(cfg, lam).synth_many(par), 1e-3, nl)
    a, ca = _invert(cfg, lam, prof, True)
    b, cb = _invert(cfg, lam, prof, False)
    assert np.all(np.isfinite(a)) and np.all(a[:, 9] > 0)
    assert np.all(ca[:, 0] > 0) and np.all(cb[:, 0] > 0)
    ratio = a[:, 9] / b[:, 9]
    assert abs(np.median(ratio) - 1.0) < 1e-3
    assert np.mean(np.abs(ratio - 1.0) < 1e-3) >= 0.5
