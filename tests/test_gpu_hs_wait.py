"""The one-launch Horn-Schunck solve: its waits that run out, its work queue when not all of its CTAs
start at once, and the scratch of the sizes it hands over."""
import ctypes

import numpy as np
import pytest

import oracle as O
from test_gpu_hs_halo import frames, same


def solve(x, niter, wait_limit=1 << 20):
    """(U, V, error, schedule) of of_hs_solve_persistent_limit."""
    import torch
    from ofb200 import ops
    from ofb200._lib import call, lib
    h, w = x[0].shape
    t = [torch.from_numpy(y).cuda() if isinstance(y, np.ndarray) else y for y in x]
    err = torch.zeros((), dtype=torch.float64, device="cuda")
    sched = torch.full((1,), 9, dtype=torch.int32, device="cuda")
    n = lib().of_hs_workspace_size(h, w, w)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    p = lambda a: ctypes.c_void_p(a.data_ptr())  # noqa: E731
    call("of_hs_solve_persistent_limit", *(p(a) for a in t), h, w, w, 21.0, niter, p(err), wait_limit, p(sched), p(ws), n,
         ops.stream_ptr())
    return t[2], t[3], err, sched


@pytest.mark.gpu
@pytest.mark.parametrize("h,w", [(256, 256), (300, 290), (401, 389)])
def test_a_wait_that_runs_out_ends_the_solve(cuda_ok, h, w):
    """A limit of one poll: no neighbour has published by then.  The launch ends, the error is NaN, and the
    next solve on the same stream is right again."""
    x = frames(h, w, 3)
    _, _, err, sched = solve(x, 41, wait_limit=1)
    assert np.isnan(float(err)) and int(sched) == 2
    U, V, err, _ = solve(x, 41)
    Uo, Vo, _ = O.hs_solve(*x, 21.0, 41)
    assert same(U.cpu().numpy(), Uo) and same(V.cpu().numpy(), Vo) and np.isfinite(float(err))


@pytest.mark.gpu
@pytest.mark.parametrize("h,w", [(256, 256), (300, 290), (401, 389)])
def test_queue_when_sms_are_taken(cuda_ok, h, w):
    """Another kernel holds all but 20 SMs for 30 ms when the solve starts."""
    import torch
    from test_gpu_hs_batch import _occupy
    x = frames(h, w, h)
    main, side = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(main):
        assert int(solve(x, 41)[3]) == 2  # alone: resident (and its kernel is loaded)
        t = [torch.from_numpy(y).cuda() for y in x]
    torch.cuda.synchronize()
    held = _occupy(torch, side, torch.cuda.get_device_properties(0).multi_processor_count - 20, 200 * 1024, 30_000_000)
    with torch.cuda.stream(main):
        U, V, err, sched = solve(t, 41)
    torch.cuda.synchronize()
    del held
    Uo, Vo, _ = O.hs_solve(*x, 21.0, 41)
    assert int(sched) == 1 and np.isfinite(float(err))
    assert same(U.cpu().numpy(), Uo) and same(V.cpu().numpy(), Vo)


@pytest.mark.gpu
@pytest.mark.parametrize("h,w", [(1185, 192), (500, 452)])
def test_beyond_one_launch_against_oracle(cuda_ok, h, w):
    x = frames(h, w, 4)
    U, V, _, sched = solve(x, 9)
    Uo, Vo, _ = O.hs_solve(*x, 21.0, 9)
    assert int(sched) == 0 and same(U.cpu().numpy(), Uo) and same(V.cpu().numpy(), Vo)


def test_scratch_beyond_one_launch_is_the_pass_form_s():
    """Seven planes (derivatives, the two ping-pong fields, the initial one) and two sums."""
    from ofb200._lib import lib
    for h, w in ((2048, 2048), (1185, 192), (512, 512)):
        assert lib().of_hs_workspace_size(h, w, w) <= 7 * 4 * h * w + 4096
