"""me_plan_autotune leaves svd_lanes alone with all nine parameters free: the
solves then run one thread per matrix whatever it says, so a choice between its
values would be made on noise, and it selects the rounding that the LM amplifies."""
import numpy as np
import pytest

import me_b200
import me_maps

pytestmark = pytest.mark.gpu
NAME = "fe15648_64x64"


@pytest.mark.parametrize("lanes", [1, 2, 4])
def test_nine_free_parameters(lanes):
    torch = pytest.importorskip("torch")
    cfg = me_b200.parse_config_text(me_maps.control_text(NAME, precision="FP32"))
    with me_b200.Plan(cfg, me_maps.wavelengths(NAME)) as plan:
        par = me_maps.draw_parameters(NAME, 512, 7)
        prof = torch.from_numpy(me_maps.add_noise(plan.synthesize(par), 1e-3, 7)).cuda()
        plan.svd_lanes = lanes
        for _ in range(3):
            r = plan.autotune(prof.data_ptr(), 512)
            assert r["svd_lanes"] == lanes and plan.svd_lanes == lanes
