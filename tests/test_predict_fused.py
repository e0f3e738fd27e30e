"""Map inference in one kernel (the tcgen05 path) against the separate kernels
(the mma.sync path) at the edges of its split: one profile, counts around its
tiles of 128, a second tile and a third for a CTA, feature rows that end within
a block of 64, fill one, and take a second and a third piece of 256, profiles on
and off 16 bytes.

Both round the same activations to BF16 after FP32 sums in another order; a sum
on a rounding boundary falls to either side, one unit of 2^-8 relative at most
per activation and in few of them, so the standardised outputs agree to 2^-8 in
norm; a row, column or piece out of place changes them by their own size."""
import numpy as np
import pytest

import me_b200
import me_maps

pytestmark = pytest.mark.gpu

NAME = "fe15648_64x64"
BOUND = 2.0 ** -8


def _angles(par):
    # bounded functions of the two angles, free of their wraps
    return np.stack([np.cos(par[:, 1]), np.cos(2 * par[:, 2]), np.sin(2 * par[:, 2])], 1)


@pytest.mark.parametrize("nl", [6, 16, 33, 60, 64, 65, 112, 150])
def test_against_the_separate_kernels(nl):
    torch = pytest.importorskip("torch")
    cfg = me_b200.parse_config_text(me_maps.control_text(NAME, precision="FP32"))
    lam = 15648.5 + 0.04 * (np.arange(nl) - (nl - 1) / 2)
    counts = [1, 15, 17, 127, 128, 129, 300]
    if nl in (6, 60, 150):
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        counts += [sms * 128 + 1, 2 * sms * 128 + 130]
    with me_b200.Plan(cfg, lam) as plan:
        init = me_b200.Initializer.train(plan, samples=2048, batch=1024, epochs=2, seed=5)
        par = me_maps.draw_parameters(NAME, 300, nl)
        one = torch.from_numpy(me_maps.add_noise(plan.synthesize(par), 1e-3, nl)).cuda().ravel()
        for count in counts:
            for off in (0, 1):
                rows = one.reshape(300, -1).repeat((count + 299) // 300, 1)[:count]
                prof = torch.zeros(count * 4 * nl + 1, dtype=torch.float64, device="cuda")
                prof[off:off + count * 4 * nl] = rows.ravel()
                out = {}
                for path in ("tcgen05", "mma_sync"):
                    init.set_gemm(path)
                    got = torch.full((count + 1, 9), 7.0, dtype=torch.float64, device="cuda")
                    before = init.gemm_launches()
                    init.predict_device(prof.data_ptr() + 8 * off, count, got.data_ptr())
                    torch.cuda.synchronize()
                    assert init.gemm_launches()[path] > before[path]
                    assert torch.all(got[count] == 7.0)  # nothing past the last profile
                    out[path] = got[:count].cpu().numpy()
                a, b = out["tcgen05"], out["mma_sync"]
                assert np.all(np.isfinite(a))
                # every profile by itself, wherever it lies: copies are equal
                tiled = np.tile(a[:300], ((count + 299) // 300, 1))[:count]
                np.testing.assert_array_equal(a, tiled)
                for k in (0, 3, 4, 5, 6, 7, 8):
                    size = np.linalg.norm(b[:, k])
                    assert np.linalg.norm(a[:, k] - b[:, k]) <= BOUND * size + 1e-6, k
                if count >= 127:
                    assert np.median(np.abs(_angles(a) - _angles(b))) <= BOUND
        init.close()
