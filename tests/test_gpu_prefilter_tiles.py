"""The 3- and 5-tap prefilters at the edges of their 64 x 32 tiles, with rows that can and cannot take
8-byte stores, from float32 and uint8, against the CPU oracle bit for bit."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("taps", [3, 5])
@pytest.mark.parametrize("h,w,pad", [(2, 2, 0), (3, 65, 1), (31, 63, 1), (32, 64, 0), (33, 66, 0), (35, 67, 2), (66, 130, 1),
                                     (100, 197, 0)])
@pytest.mark.parametrize("u8", [False, True])
def test_prefilter_tiles(cuda_ok, h, w, pad, taps, u8):
    import torch
    from gaussian_filter import prepareGaussianKernel
    from ofb200 import ops
    rng = np.random.default_rng(h * w)
    k = prepareGaussianKernel(1.3, taps)
    a = rng.integers(0, 256, (h, w)).astype(np.uint8) if u8 else rng.normal(0, 50, (h, w)).astype(np.float32)
    src = torch.zeros(h, w + pad, dtype=torch.uint8 if u8 else torch.float32, device="cuda")
    src[:, :w] = torch.from_numpy(a).cuda()
    dst = torch.full((h, w + pad), 7.0, device="cuda")
    ops.prefilter(src[:, :w], k, out=dst[:, :w])
    assert bool((dst[:, w:] == 7.0).all())
    assert np.array_equal(dst[:, :w].cpu().numpy(), O.prefilter(a.astype(np.float32), 1.3, taps))
