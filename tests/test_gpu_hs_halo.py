"""The single-pair persistent Horn-Schunck solve: its three region shapes and the pass-per-launch
form beyond them, at the sizes where one hands over to the next, with sides that are and are not
multiples of a block, against the pass-per-launch solve bit for bit (which the CPU oracle pins)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def same(a, b):
    return np.array_equal(a, b, equal_nan=True) and np.array_equal(np.signbit(a[~np.isnan(a)]), np.signbit(b[~np.isnan(b)]))


def solve(x, pad, alpha, niter, persistent):
    import torch
    from ofb200 import ops
    h, w = x[0].shape
    buf = [torch.zeros(h, w + pad, device="cuda") for _ in range(4)]
    for t, y in zip(buf, x):
        t[:, :w] = torch.from_numpy(y).cuda()
    U, V, err = ops.hs_solve(*(t[:, :w] for t in buf), alpha, niter, persistent=persistent)
    return U.cpu().numpy(), V.cpu().numpy(), float(err)


def frames(h, w, seed):
    rng = np.random.default_rng(seed)
    x = [np.round(rng.uniform(0, 255, (h, w))).astype(np.float32) for _ in range(2)]
    return x + [rng.normal(0, 1, (h, w)).astype(np.float32) for _ in range(2)]


@pytest.mark.parametrize("h,w", [(16, 16), (17, 33), (592, 128), (593, 128), (591, 129), (592, 192), (593, 191),
                                 (1184, 192), (1183, 191), (1185, 192), (255, 257), (40, 1100)])
@pytest.mark.parametrize("niter", [9, 16, 29])
def test_shapes_hand_over(cuda_ok, h, w, niter):
    x = frames(h, w, h + w + niter)
    if niter == 29:
        x[0][h // 2, w // 2] = np.nan  # spreads by a cell per sweep; the quotient's range fails where it is
    a, b = solve(x, 0, 21.0, niter, True), solve(x, 0, 21.0, niter, False)
    assert same(a[0], b[0]) and same(a[1], b[1])
    assert a[2] == pytest.approx(b[2], rel=1e-12, nan_ok=True)  # float64 sums by atomics, in any order


@pytest.mark.parametrize("h,w,pad", [(16, 16, 0), (33, 49, 1), (48, 32, 3), (50, 95, 0), (31, 98, 2)])
@pytest.mark.parametrize("alpha", [21.0, 0.0])
def test_persistent_against_oracle(cuda_ok, h, w, pad, alpha):
    x = frames(h, w, h * w)
    U, V, _ = solve(x, pad, alpha, 19, True)
    with np.errstate(all="ignore"):
        Uo, Vo, _ = O.hs_solve(*x, alpha, 19)
    assert same(U, Uo) and same(V, Vo)


@pytest.mark.parametrize("h,w", [(256, 256), (300, 290), (401, 389)])
def test_beside_other_work(cuda_ok, h, w):
    """Another kernel holds all but 20 SMs for a few milliseconds when the solve starts: its CTAs do not
    all run, so they take the work queue (or, if the holder is gone by then, their resident stages);
    the result is the same."""
    import torch
    from ofb200 import ops
    from test_gpu_hs_batch import _occupy
    x = [torch.from_numpy(y).cuda() for y in frames(h, w, h)]
    ref = ops.hs_solve(x[0], x[1], x[2].clone(), x[3].clone(), 21.0, 41, persistent=False)
    side, main = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(main):  # sizes the stream's scratch
        ops.hs_solve(x[0], x[1], x[2].clone(), x[3].clone(), 21.0, 41, persistent=True)
        uv = x[2].clone(), x[3].clone()
    torch.cuda.synchronize()
    held = _occupy(torch, side, torch.cuda.get_device_properties(0).multi_processor_count - 20, 200 * 1024, 5_000_000)
    with torch.cuda.stream(main):
        U, V, err = ops.hs_solve(x[0], x[1], *uv, 21.0, 41, persistent=True)
    torch.cuda.synchronize()
    del held
    assert torch.equal(U, ref[0]) and torch.equal(V, ref[1])
    assert float(err) == pytest.approx(float(ref[2]), rel=1e-12)
