"""Horn-Schunck pairs whose one half is the same texture in both frames: the flow that diffuses into it
falls through all magnitudes to the subnormal numbers.  The results are the oracle's, bit for bit, and
such a pair takes about as long as one that moves everywhere."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def frames(h, w, seed, static):
    rng = np.random.default_rng(seed)
    a = np.round(rng.uniform(20, 230, (h, w)))
    b = np.clip(np.roll(a, 1, 1) + np.round(rng.normal(0, 2, (h, w))), 0, 255)
    if static:
        b[:, w // 2:] = a[:, w // 2:]
    return a.astype(np.float32), b.astype(np.float32)


def solver(a, b, niter, persistent):
    import torch
    from ofb200 import ops
    I0, I1 = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    U, V = torch.zeros_like(I0), torch.zeros_like(I0)

    def run():
        U.zero_()
        V.zero_()
        ops.hs_solve(I0, I1, U, V, 21.0, niter, persistent=persistent)
        return U, V
    return run


@pytest.mark.parametrize("persistent", [False, True])
@pytest.mark.parametrize("h,w", [(40, 200), (97, 251), (300, 290), (401, 389)])
def test_static_half_against_oracle(cuda_ok, h, w, persistent):
    a, b = frames(h, w, h, True)
    U, V = (t.cpu().numpy() for t in solver(a, b, 120, persistent)())
    z = np.zeros((h, w), np.float32)
    Uo, Vo, _ = O.hs_solve(a, b, z, z, 21.0, 120)
    tiny = (np.abs(Uo) < 2.0 ** -126) & (Uo != 0)
    assert tiny.sum() > h and np.array_equal(U.view(np.uint32), Uo.view(np.uint32))
    assert np.array_equal(V.view(np.uint32), Vo.view(np.uint32))


@pytest.mark.parametrize("persistent,s", [(True, 256), (False, 512)])
def test_static_half_is_not_slow(cuda_ok, persistent, s):
    """At most twice the time (1.1 and 1.5 times as measured; 3.7 when every pass with a tiny numerator
    ran again with the divide)."""
    import torch
    best = []
    for static in (False, True):
        run = solver(*frames(s, s, 1, static), 600, persistent)
        run()
        t = []
        for _ in range(7):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            run()
            e1.record()
            e1.synchronize()
            t.append(e0.elapsed_time(e1))
        best.append(min(t))
    assert best[1] < 2 * best[0], best


def particles(s):
    """Moving particles on black beside the same texture in both frames."""
    a = np.round(np.random.default_rng(0).uniform(20, 230, (s, s)))
    b = a.copy()
    rng = np.random.default_rng(1)
    p = np.zeros((s, s), np.float32)
    yy, xx = np.mgrid[-3:4, -3:4]
    for _ in range(s * s // 60):
        y, x = rng.uniform(4, s - 5, 2)
        i, j = int(y), int(x)
        p[i - 3:i + 4, j - 3:j + 4] += 200 * np.exp(-((yy + i - y) ** 2 + (xx + j - x) ** 2) / 2)
    p = np.clip(np.round(p), 0, 255)
    a[:, :s // 2], b[:, :s // 2] = p[:, :s // 2], np.roll(p, 1, 1)[:, :s // 2]
    return a.astype(np.float32), b.astype(np.float32)


@pytest.mark.parametrize("schedule,shape", [("queue", 0), ("queue", 1), ("queue", 3), ("resident", 3), ("resident", 1),
                                            ("cluster", 0)])
def test_batch_schedules_against_oracle(cuda_ok, schedule, shape):
    """Subnormal quotients that lie on rounding midpoints, in the kernels that divide by a float64 reciprocal."""
    import torch
    from ofb200 import ops
    a, b = particles(256)
    I0, I1 = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    U, V = torch.zeros_like(I0), torch.zeros_like(I0)
    st = ops.hs_batch([(I0, I1, U, V, 21.0, 200)], tile_shape=shape, schedule=schedule)
    z = np.zeros_like(a)
    Uo, Vo, _ = O.hs_solve(a, b, z, z, 21.0, 200)
    assert int(st.item()) == 0
    assert np.array_equal(U.cpu().numpy().view(np.uint32), Uo.view(np.uint32))
    assert np.array_equal(V.cpu().numpy().view(np.uint32), Vo.view(np.uint32))
