"""Horn-Schunck's register-blocked sweep at the edges of its regions and of its quotient's
range, against the CPU oracle bit for bit (same values, the sign of zero included)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def same(a, b):
    return np.array_equal(a, b, equal_nan=True) and np.array_equal(np.signbit(a[~np.isnan(a)]), np.signbit(b[~np.isnan(b)]))


def solve(a, b, u, v, alpha, niter, pad, persistent):
    import torch
    from ofb200 import ops
    h, w = a.shape
    buf = [torch.zeros(h, w + pad, device="cuda") for _ in range(4)]  # row pitch w + pad
    for t, x in zip(buf, (a, b, u, v)):
        t[:, :w] = torch.from_numpy(x).cuda()
    I0, I1, U, V = (t[:, :w] for t in buf)
    U, V, _ = ops.hs_solve(I0, I1, U, V, alpha, niter, persistent=persistent)
    return U.cpu().numpy(), V.cpu().numpy()


def frames(h, w, seed, scale):
    rng = np.random.default_rng(seed)
    a, b = (np.round(rng.uniform(0, 255, (h, w))).astype(np.float32) * np.float32(scale) for _ in range(2))
    a[: h // 3], b[: h // 3] = 0, 0  # a flat part: numerators of exactly zero
    u, v = (rng.normal(0, 1, (h, w)).astype(np.float32) for _ in range(2))
    u[: h // 2] = 0
    return a, b, u, v


@pytest.mark.parametrize("persistent", [False, True])
@pytest.mark.parametrize("niter", [1, 4, 7])
@pytest.mark.parametrize("h,w,pad", [(16, 16, 0), (24, 56, 0), (25, 57, 0), (23, 55, 3), (32, 64, 1), (49, 113, 2),
                                     (72, 168, 0)])
def test_hs_region_edges(cuda_ok, h, w, pad, niter, persistent):
    a, b, u, v = frames(h, w, h * w, 1.0)
    U, V = solve(a, b, u, v, 21.0, niter, pad, persistent)
    Uo, Vo, _ = O.hs_solve(a, b, u, v, 21.0, niter)
    assert same(U, Uo) and same(V, Vo)


@pytest.mark.parametrize("persistent", [False, True])
@pytest.mark.parametrize("alpha,scale", [(21.0, 1e-18), (21.0, 1e-30), (1e-7, 1.0), (1e-7, 1e-9), (0.0, 1.0),
                                         (1e8, 1.0), (1e15, 1e12), (21.0, 1e30), (21.0, np.inf)])
def test_hs_quotient_range(cuda_ok, alpha, scale, persistent):
    """Numerators and denominators outside the range of the refined quotient (tiny, huge, zero
    and infinite ones): the pass is repeated with the divide."""
    a, b, u, v = frames(40, 70, 3, 1.0)
    if np.isinf(scale):
        a[20, 30], b[5, 5] = np.inf, np.nan
    else:
        a, b = a * np.float32(scale), b * np.float32(scale)
        a[30:, 40:], b[30:, 40:] = 17, 19  # and ordinary ones beside them
    U, V = solve(a, b, u, v, alpha, 9, 0, persistent)
    with np.errstate(all="ignore"):
        Uo, Vo, _ = O.hs_solve(a, b, u, v, alpha, 9)
    assert same(U, Uo) and same(V, Vo)
