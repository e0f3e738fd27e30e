"""Round batches as CUDA graphs: a queue long enough to reach them (few slots, so
hundreds of batches) and one that ends before, against direct launches: the
same kernels in the same order, so equal bit for bit."""
import numpy as np
import pytest

import me_b200
import me_maps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window,count", [(32, 1024), (0, 1024)])
def test_graphs_equal_direct_launches(window, count):
    name = "fe15648_64x64"
    cfg = me_b200.parse_config_text(me_maps.control_text(name, precision="FP32", seed=7))
    par = me_maps.draw_parameters(name, count, 7)
    res = {}
    for on in (0, 1):
        with me_b200.Plan(cfg, me_maps.wavelengths(name)) as plan:
            prof = me_maps.add_noise(plan.synthesize(par), 1e-3, 7)
            if window:
                me_b200.lib().me_plan_set_window(plan.handle, window)
            # rounds only: which pixels the tail takes depends on the poll
            me_b200.lib().me_plan_set_tail_slots(plan.handle, 0)
            me_b200.lib().me_plan_set_graphs(plan.handle, on)
            res[on], stats = plan.invert(prof)
            if window:
                assert stats["rounds"] > 8 * 64
    np.testing.assert_array_equal(res[1], res[0])
