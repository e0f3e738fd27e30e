"""A filtered profile does not depend on how many pixels the call has: the two
forms of the filtered synthesis, a thread per sub-wavelength on small maps and
per wavelength on large ones, sum the same terms in the same order with the same
roundings, so both give the same bits, in both precisions, and so do Jacobians."""
import numpy as np
import pytest

import me_b200
import me_maps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["FP64", "FP32"])
@pytest.mark.parametrize("nl,points", [(6, 21), (16, 3), (33, 5), (7, 63)])
def test_both_forms_of_the_filter(nl, points, prec):
    torch = pytest.importorskip("torch")
    name = "fe15648_64x64"
    cfg = me_b200.parse_config_text(me_maps.control_text(name, precision=prec,
                                                         extra={"filter": f"76, {points}"}))
    lam = 15648.5 + 0.04 * 60 / nl * (np.arange(nl) - (nl - 1) / 2)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    line = -(-sms * 1024 // nl)  # pixels from which a thread takes a wavelength
    line_jac = -(-sms * 512 // nl)
    par = me_maps.draw_parameters(name, line, nl)
    with me_b200.Plan(cfg, lam) as plan:
        large = plan.synthesize(par)
        np.testing.assert_array_equal(plan.synthesize(par[:line - 1]), large[:line - 1])
        np.testing.assert_array_equal(plan.synthesize(par[:100]), large[:100])
        prof, jac = plan.synthesize_jacobian(par[:line_jac], 0.1)
        small = plan.synthesize_jacobian(par[:100], 0.1)
        np.testing.assert_array_equal(small[0], prof[:100])
        np.testing.assert_array_equal(small[1], jac[:100])
