"""A training step in two kernels (the tcgen05 path) against the oracle of
test_mlp.py, at the edges of its split: feature rows that end within a block of
64, fill one, and take a second and a third piece of 256; the smallest batch,
one whose shares of the weight gradient are uneven in size to others, and a
large one.  The gradients within the bounds there: the oracle rounds at the same
places, so FP32 against FP64 sums and the few BF16 roundings that these turn.
The loss against the separate kernels' (the mma.sync path), which sum in FP32
too: apart by the order of 320 squares at most in FP32 and of the GEMMs' sums,
1e-6.  (A turned rounding weighs more in few rows of many features: at 256 rows
of 600 both paths' losses lie 2.6e-5 from the oracle's, side by side.)"""
import numpy as np
import pytest

import me_b200
import me_maps
from oracle import mlp_oracle as mo
from test_mlp import random_batch, random_params

pytestmark = pytest.mark.gpu

NAME = "fe15648_64x64"


def _plan(nl):
    cfg = me_b200.parse_config_text(me_maps.control_text(NAME, precision="FP32"))
    return me_b200.Plan(cfg, 15648.5 + 0.04 * (np.arange(nl) - (nl - 1) / 2))


@pytest.mark.parametrize("nl,rows", [(6, 256), (16, 768), (60, 4352), (65, 512), (150, 256)])
def test_loss_and_gradients(nl, rows):
    with _plan(nl) as plan:
        init = me_b200.Initializer.train(plan, samples=256, batch=256, epochs=0)
    nip = init.shape()[1]
    p = random_params(nip, 4 * nl, nl)
    init.set_params(p)
    x, t = random_batch(rows, nip, 4 * nl, rows)
    _, want = mo.loss_grad(p.astype(np.float64), x, t, nip, bf16=True)
    got = {}
    for path in ("tcgen05", "mma_sync", "tcgen05"):
        init.set_gemm(path)
        got[path] = init.loss_grad(x, t)  # the second call of a path starts from clean sums
    ends = np.cumsum([0] + [o * i + o for o, i in mo.shapes(nip)])
    assert abs(got["tcgen05"][0] - got["mma_sync"][0]) <= 1e-6 * got["mma_sync"][0]
    for _, g in got.values():
        assert np.linalg.norm(g - want) < 2e-3 * np.linalg.norm(want)
        for l0, l1 in zip(ends[:-1], ends[1:]):
            assert np.linalg.norm(g[l0:l1] - want[l0:l1]) <= \
                5e-3 * np.linalg.norm(want[l0:l1]) + 1e-12
    init.close()


@pytest.mark.parametrize("samples,batch", [(256, 256), (1000, 256), (4096, 4096), (9000, 512)])
def test_first_epoch_of_both_paths(samples, batch):
    """Whole trainings with the step's buffers in the training set's memory and
    (a batch as large as the set) beside it.  The first epoch's mean loss of the
    two paths: the same samples in the same order, parameters apart by what
    rounding does to Adam's steps."""
    loss = {}
    for path in (0, 1):  # tcgen05, mma.sync
        with _plan(7) as plan:
            with me_b200.Initializer.train(plan, samples=samples, batch=batch, epochs=1, seed=3,
                                           gemm=path) as init:
                loss[path] = init.final_loss
                assert np.all(np.isfinite(init.get_params()))
    a, b = loss.values()
    assert abs(a - b) <= 1e-3 * b
