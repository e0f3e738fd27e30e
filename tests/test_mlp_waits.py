"""The bounded waits of the fused inference and training kernels: with one
kind of event unannounced (loads of weights, completion of MMAs, release of
stages) a wait for it runs out, all other waits end with it and the barriers stay
in step: the call fails with the wait's error and within seconds, and the next
call on the same initialiser gives what the first one gave.  Limits of one try to
thousands, CTAs with one tile and with several, feature rows in one piece and in
two."""
import time

import numpy as np
import pytest

import me_b200
import me_maps
from test_mlp import random_batch

pytestmark = pytest.mark.gpu
NAME = "fe15648_64x64"
ME_ERR_CUDA = next(k for k, v in me_b200.STATUS.items() if v == "ME_ERR_CUDA")


def _initialiser(nl):
    cfg = me_b200.parse_config_text(me_maps.control_text(NAME, precision="FP32"))
    lam = 15648.5 + 0.04 * (np.arange(nl) - (nl - 1) / 2)
    with me_b200.Plan(cfg, lam) as plan:
        init = me_b200.Initializer.train(plan, samples=1024, batch=1024, epochs=1, seed=5)
        prof = me_maps.add_noise(plan.synthesize(me_maps.draw_parameters(NAME, 300, nl)), 1e-3, nl)
    return init, prof


def _fails(call):
    t0 = time.monotonic()
    with pytest.raises(me_b200.MeError) as e:
        call()
    assert e.value.status == ME_ERR_CUDA and "timed out" in str(e.value)
    assert time.monotonic() - t0 < 5.0


@pytest.mark.parametrize("drop", [1, 2, 3])
@pytest.mark.parametrize("nl,count", [(60, 1), (60, 300), (112, 300), (60, 40000)])
def test_inference(nl, count, drop):
    torch = pytest.importorskip("torch")
    init, prof = _initialiser(nl)
    d = torch.from_numpy(np.resize(prof, (count, 4, nl))).cuda()
    out = torch.zeros(count, 9, dtype=torch.float64, device="cuda")

    def predict():
        out.zero_()
        init.predict_device(d.data_ptr(), count, out.data_ptr())
        torch.cuda.synchronize()
        return out.cpu().numpy()

    first = predict()
    for tries in (1, 64, 1 << 14):
        init.set_waits(tries, drop)
        _fails(predict)
        init.set_waits()
        np.testing.assert_array_equal(predict(), first)
    init.close()


@pytest.mark.parametrize("drop", [1, 2, 3])
@pytest.mark.parametrize("nl,rows", [(60, 256), (112, 4096)])
def test_gradients(nl, rows, drop):
    init, _ = _initialiser(nl)
    nip = init.shape()[1]
    x, t = random_batch(rows, nip, 4 * nl, rows)
    loss, grad = init.loss_grad(x, t)
    for tries in (1, 64, 1 << 14):
        init.set_waits(tries, drop)
        _fails(lambda: init.loss_grad(x, t))
        init.set_waits()
        again = init.loss_grad(x, t)
        # (sums of FP32 atomics, in another order each time)
        assert abs(again[0] - loss) <= 1e-6 * loss
        assert np.linalg.norm(again[1] - grad) <= 1e-5 * np.linalg.norm(grad)
    init.close()


def test_bad_arguments():
    init, _ = _initialiser(6)
    for drop in (-1, 4):
        with pytest.raises(me_b200.MeError):
            init.set_waits(0, drop)
    init.close()
