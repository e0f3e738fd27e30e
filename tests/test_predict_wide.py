"""Inference of wide grids at the edges of the rule that sends few profiles of
many features through the separate kernels: counts on both sides of its two
lines, feature rows on both sides of its widths.  A profile's arithmetic is the
same on both ways, so its result is, bit for bit.  Under capture, where the
separate kernels could not allocate their buffers, and on two streams at once,
which share those buffers, the results are the same again."""
import numpy as np
import pytest

import me_b200
import me_maps

pytestmark = pytest.mark.gpu
NAME = "fe15648_64x64"


def _initialiser(nl):
    cfg = me_b200.parse_config_text(me_maps.control_text(NAME, precision="FP32"))
    lam = 15648.5 + 0.04 * (np.arange(nl) - (nl - 1) / 2)
    with me_b200.Plan(cfg, lam) as plan:
        init = me_b200.Initializer.train(plan, samples=1024, batch=512, epochs=2, seed=5)
        par = me_maps.draw_parameters(NAME, 300, nl)
        prof = me_maps.add_noise(plan.synthesize(par), 1e-3, nl)
    return init, prof


@pytest.mark.parametrize("nl,edge", [(96, 64), (97, 64), (128, 64), (192, 64), (193, 3072),
                                     (300, 3072), (512, 3072)])
def test_both_sides_of_the_rule(nl, edge):
    torch = pytest.importorskip("torch")
    init, prof = _initialiser(nl)
    rows = torch.from_numpy(prof).cuda()

    def predict(count):
        d = rows.repeat((count + 299) // 300, 1, 1)[:count].contiguous()
        out = torch.full((count + 1, 9), 7.0, dtype=torch.float64, device="cuda")
        init.predict_device(d.data_ptr(), count, out.data_ptr())
        torch.cuda.synchronize()
        assert torch.all(out[count] == 7.0)
        return out[:count].cpu().numpy()

    want = predict(max(edge, 300) + 100)[:300]  # one kernel
    for count in (1, 15, edge, edge + 1):
        got = predict(count)
        np.testing.assert_array_equal(got, np.resize(want, got.shape))
    init.close()


def test_first_call_under_capture():
    torch = pytest.importorskip("torch")
    init, prof = _initialiser(193)
    d = torch.from_numpy(prof).cuda()
    out = torch.zeros(300, 9, dtype=torch.float64, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        init.predict_device(d.data_ptr(), 300, out.data_ptr(),
                            torch.cuda.current_stream().cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy(), init.predict(prof))
    init.close()


def test_two_streams():
    torch = pytest.importorskip("torch")
    init, prof = _initialiser(256)
    maps = [torch.from_numpy(prof).cuda(), torch.from_numpy(prof[::-1].copy()).cuda()]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    out = [torch.zeros(300, 9, dtype=torch.float64, device="cuda") for _ in range(40)]
    torch.cuda.synchronize()
    for k, o in enumerate(out):
        init.predict_device(maps[k % 2].data_ptr(), 300, o.data_ptr(), streams[k % 2].cuda_stream)
    torch.cuda.synchronize()
    want = init.predict(prof)
    for k, o in enumerate(out):
        np.testing.assert_array_equal(o.cpu().numpy(), want[::-1] if k % 2 else want)
    init.close()
