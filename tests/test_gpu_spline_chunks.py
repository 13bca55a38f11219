"""The spline's serial solve runs in chunks of 24 steps, loaded two chunks ahead, with pivots that are
constant from step 48 on: line lengths on both sides of every seam, bit for bit against the oracle."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(4, 4), (5, 33), (6, 5), (27, 28), (28, 27), (29, 52), (51, 53), (52, 29), (53, 51), (75, 76),
                                 (76, 77), (77, 75), (99, 100), (101, 148), (149, 150), (196, 197)])
def test_spline_chunk_seams(cuda_ok, h, w):
    import torch
    from ofb200 import ops
    a = np.random.default_rng(h * 1000 + w).normal(0, 3, (h, w)).astype(np.float32)
    if h % 2:
        a[h // 2, w // 2] = np.nan  # reaches its whole row and column, as in the oracle
    H, W = 2 * h - 1, 2 * w + 1
    out = ops.spline_upsample(torch.from_numpy(a).cuda(), H, W).cpu().numpy()
    with np.errstate(all="ignore"):
        ref = O.spline_upsample(a, H, W)
    assert np.array_equal(out, ref, equal_nan=True)
