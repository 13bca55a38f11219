"""The fused Farneback iteration at the edges of its tiles (64 x 32 outputs, half windows up to
16, any row pitch), against the CPU oracle's blur, flow and matrices bit for bit."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def pitched(a, pad):
    import torch
    t = torch.zeros(a.shape[0], a.shape[1] + pad, device="cuda")
    t[:, : a.shape[1]] = torch.from_numpy(a).cuda()
    return t[:, : a.shape[1]]


@pytest.mark.parametrize("kh", [0, 1, 10, 15, 16, 17])
@pytest.mark.parametrize("h,w,pad", [(17, 17, 0), (16, 40, 0), (32, 64, 0), (33, 65, 3), (63, 96, 0), (49, 81, 1),
                                     (96, 192, 0), (100, 203, 1)])
def test_fb_iteration_tiles(cuda_ok, h, w, pad, kh):
    from ofb200 import ops
    rng = np.random.default_rng(h * w + kh)
    M, R0, R1 = (rng.normal(0, 1, (5 * h, w)).astype(np.float32) for _ in range(3))
    M[: h] += 3  # a well-conditioned system at most pixels
    M[2 * h: 3 * h] += 3
    hk = np.exp(-0.5 * (np.arange(kh + 1) / (0.4 * kh + 0.5)) ** 2).astype(np.float32)
    hk /= hk[0] + 2 * hk[1:].sum()
    fx, fy = (pitched(np.zeros((h, w), np.float32), pad) for _ in range(2))
    Mo = pitched(np.zeros((5 * h, w), np.float32), pad)
    ops.fb_iteration(pitched(M, pad), Mo, pitched(R0, pad), pitched(R1, pad), fx, fy, hk, True)
    fxo, fyo = O.fb_update_flow(O.fb_blur(M, hk, 5) if kh else M * hk[0] * hk[0], h, w)
    assert np.array_equal(fx.cpu().numpy(), fxo) and np.array_equal(fy.cpu().numpy(), fyo)
    assert np.array_equal(Mo.cpu().numpy(), O.fb_update_matrices(fxo, fyo, R0, R1))
