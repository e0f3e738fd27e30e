"""The FP32 tail kernel with num_iter = 0: every run of the restart schedule ends
without a trial step, so a pixel goes from one synthesis to the next through the
run's end alone, where the kernel's warps have only the barriers of the step
loop between them.  Against one-thread-per-pixel rounds: chi^2 at the same
starting parameters, apart by FP32 profiles (5e-6 of the continuum, over noise
of 1e-3 and misfits above it) -- 1e-3 of chi^2 at most, in every pixel."""
import numpy as np
import pytest

import me_b200
import me_maps
import oracle_bind as ob

pytestmark = pytest.mark.gpu
NAME = "fe15648_64x64"


@pytest.mark.parametrize("nl,points", [(33, 1), (6, 21), (33, 5)])
def test_runs_without_trials(nl, points):
    extra = {"num_iter": "0", "num_run": "10"}
    if points > 1:
        extra["filter"] = f"76, {points}"
    cfg = me_b200.parse_config_text(me_maps.control_text(NAME, widen_bounds=True, extra=extra))
    lam = 15648.5 + 0.04 * 60 / nl * (np.arange(nl) - (nl - 1) / 2)
    par = me_maps.draw_parameters(NAME, 400, nl + points)
    prof = me_maps.add_noise(ob.Oracle(cfg, lam).synth_many(par), 1e-3, nl)
    out = {}
    for tail in (0, 400):
        with me_b200.Plan(cfg, lam) as plan:
            plan.max_group = 1
            plan.tail_slots = tail
            res, st = plan.invert(prof)
            runs = plan.last_counters(400)[:, 0]
        assert st["trials"] == 0
        # (one more per pass over pixels whose carried chi^2 changed)
        assert (st["launches"] - 4 * st["rounds"] > 0) == (tail > 0)
        out[tail] = res, runs
    (a, ra), (b, rb) = out.values()
    np.testing.assert_array_equal(ra, rb)
    assert np.all(a[:, 9] > 0)
    assert np.max(np.abs(a[:, 9] / b[:, 9] - 1.0)) < 1e-3
