"""What the build reports of kernels whose residency a neighbour's code once cost:
svd_grp_kernel, the lane-split solves of plans with a fixed parameter, holds four
CTAs of 128 threads per SM, so at most 128 registers a thread, in every lane
count (32 lanes stood at 255 while the nine-parameter form was inlined there)."""
import os
import re

import pytest

BUILD = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                     "milne-eddington_b200", "_build")


@pytest.mark.parametrize("unit", ["f32", "f32f", "f64", "f64f"])
def test_svd_grp_registers(unit):
    path = os.path.join(BUILD, f"me_invert_{unit}.o.ptxas.txt")
    if not os.path.exists(path):
        pytest.skip("no build log here")
    log = open(path).read()
    used = re.findall(r"Compiling entry function '\w*svd_grp_kernelILi(\d+)E\w*'.*?Used (\d+) reg",
                      log, re.S)
    assert {int(g) for g, _ in used} == {2, 4, 8, 16, 32}
    for g, regs in used:
        assert int(regs) <= 128, (g, regs)
