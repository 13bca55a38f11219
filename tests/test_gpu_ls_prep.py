"""Liu-Shen's set-up takes four rows per thread on large images and one on small ones, and divides by
refinement with a fallback: both forms at the edges of their tiles, frames that are mostly black and
frames outside the refinement's range, against the CPU oracle bit for bit."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w,pad", [(1, 1, 0), (8, 32, 0), (9, 33, 1), (31, 65, 0), (32 * 17 + 1, 32 * 17 + 31, 0),
                                     (32 * 18 - 1, 32 * 17 - 31, 3), (9473, 1, 0), (5, 9473, 0)])
@pytest.mark.parametrize("scale", [1.0, 1e-25, 1e25])
def test_ls_setup(cuda_ok, h, w, pad, scale):
    import torch
    from ofb200 import ops
    rng = np.random.default_rng(h + w)
    a, b = (np.round(rng.uniform(0, 255, (h, w))).astype(np.float32) * np.float32(scale) for _ in range(2))
    a[rng.random((h, w)) < 0.5] = 0  # particles on black
    b[rng.random((h, w)) < 0.5] = 0
    a[0, 0] = b[0, 0] = 255 * np.float32(scale)
    u, v = (rng.normal(0, 1, (h, w)).astype(np.float32) for _ in range(2))
    buf = [torch.zeros(h, w + pad, device="cuda") for _ in range(4)]
    for t, x in zip(buf, (a, b, u, v)):
        t[:, :w] = torch.from_numpy(x).cuda()
    U, V, _, _ = ops.ls_solve(*(t[:, :w] for t in buf), 10.0, 1, 0.0, arithmetic="exact")
    with np.errstate(all="ignore"):
        Uo, Vo = O.ls_solve(a, b, u, v, 10.0, 1, 0.0)[:2]
    assert np.array_equal(U.cpu().numpy(), Uo, equal_nan=True) and np.array_equal(V.cpu().numpy(), Vo, equal_nan=True)
