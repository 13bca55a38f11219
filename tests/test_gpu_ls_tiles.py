"""The float32 Liu-Shen pass at the edges of its tiles (56 x 23 pixels, several per CTA on large
images) and of its stop rule, against the float64-sum arithmetic."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solve(a, b, u, v, sweeps, tol, arithmetic, pad):
    import torch
    from ofb200 import ops
    h, w = a.shape
    buf = [torch.zeros(h, w + pad, device="cuda") for _ in range(4)]
    for t, x in zip(buf, (a, b, u, v)):
        t[:, :w] = torch.from_numpy(x).cuda()
    I0, I1, U, V = (t[:, :w] for t in buf)
    U, V, it, err = ops.ls_solve(I0, I1, U, V, 10.0, sweeps, tol, arithmetic=arithmetic)
    return U.cpu().numpy(), V.cpu().numpy(), int(it.item()), float(err.item())


def inputs(h, w):
    rng = np.random.default_rng(h * w)
    a, b = (rng.uniform(1, 255, (h, w)).astype(np.float32) for _ in range(2))
    u, v = (rng.uniform(-4, 4, (h, w)).astype(np.float32) for _ in range(2))
    return a, b, u, v


@pytest.mark.parametrize("sweeps", [1, 4, 6, 11])
@pytest.mark.parametrize("h,w,pad", [(1, 1, 0), (2, 3, 1), (22, 55, 0), (23, 56, 0), (24, 57, 3), (46, 113, 0),
                                     (70, 168, 2), (461, 897, 0)])
def test_ls_fast_tile_edges(cuda_ok, h, w, pad, sweeps):
    """A sweep rounds each of its about 16 operations on values of the field's size once, and
    (a smoothing step) does not amplify what earlier sweeps left: sweeps * 16 * 2^-24 of it.
    The equations add their own conditioning at the few pixels of small determinants: 4 times."""
    x = inputs(h, w)
    Ue, Ve, ie, ee = solve(*x, sweeps, 0.0, "exact", pad)
    Uf, Vf, itf, ef = solve(*x, sweeps, 0.0, "fast", pad)
    assert ie == itf  # fewer than `sweeps` where a sweep changes nothing (one pixel)
    tol = 4 * sweeps * 16 * 2.0 ** -24 * max(np.abs(Ue).max(), np.abs(Ve).max(), 4.0)
    assert np.abs(Uf - Ue).max() <= tol and np.abs(Vf - Ve).max() <= tol
    assert ef == pytest.approx(ee, rel=1e-3)


@pytest.mark.parametrize("h,w", [(40, 120), (461, 897)])
def test_ls_fast_stops_inside_a_pass(cuda_ok, h, w):
    """The stop rule ends a solve at any sweep of a pass: the field is that of as many sweeps."""
    x = inputs(h, w)
    errs = [solve(*x, n, 0.0, "fast", 0)[3] for n in range(1, 10)]
    for n in (1, 2, 4, 5, 7):
        tol = 0.5 * (errs[n - 1] + errs[n])  # reached by sweep n + 1
        U, V, it, _ = solve(*x, 60, tol, "fast", 0)
        Un, Vn, _, _ = solve(*x, n + 1, 0.0, "fast", 0)
        assert it == n + 1 and np.array_equal(U, Un) and np.array_equal(V, Vn)
