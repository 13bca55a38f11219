"""The training kernels that take 8 channels per thread, the ReLU masks fused into the passes that
produce a gradient, the input packing over one cluster and the weight packing of all layers.

Everything is bit-exact against the oracle or the unfused kernels, except the bias gradient: float32
sums of P bfloat16 values against float64, at most P * 2^-24 of the sum of magnitudes."""
import ctypes
import os
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "oracle"))


@pytest.fixture(scope="module")
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _P(t):
    return ctypes.c_void_p(t.data_ptr())


def _sp():
    from ofb200 import ops
    return ops.stream_ptr()


def _bf(torch, rng, *shape):
    return torch.from_numpy(rng.normal(0, 1, shape).astype(np.float32)).cuda().to(torch.bfloat16)


def _f(t):
    return t.float().cpu().numpy()


@pytest.mark.parametrize("P,C,ctot,coff", [(1, 8, 8, 0), (3, 2, 16, 0), (257, 24, 40, 8), (5000, 96, 96, 0),
                                           (1023, 256, 264, 8), (70, 1000, 1008, 0), (4096, 20, 28, 4), (999, 7, 7, 0)])
def test_bias_gradient_layouts(torch, P, C, ctot, coff):
    from ofb200._lib import call
    dy = _bf(torch, np.random.default_rng(P), P, ctot)
    db = torch.ones(C, dtype=torch.float32, device="cuda")
    call("of_cnn_bias_grad", _P(dy), ctot, coff, P, C, _P(db), _sp())
    torch.cuda.synchronize()
    x = _f(dy)[:, coff:coff + C].astype(np.float64)
    bound = (P + 1) * 2.0 ** -24 * (1 + np.abs(x).sum(0))
    assert (np.abs(db.cpu().numpy() - (1 + x.sum(0))) <= bound).all()


@pytest.mark.parametrize("n,h,w,C,ctot,coff", [(1, 1, 1, 8, 8, 0), (2, 3, 37, 24, 40, 16), (3, 5, 4, 128, 128, 0),
                                               (2, 3, 5, 12, 24, 4)])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_pool_and_upsample_backward_with_mask(torch, n, h, w, C, ctot, coff, accumulate):
    import cnn_oracle as O
    from ofb200._lib import call
    rng = np.random.default_rng(C + n)
    small, act = _bf(torch, rng, n, h, w, ctot), _bf(torch, rng, n, 2 * h, 2 * w, ctot)
    act[:, ::2, 0, coff] = 0.0  # a value that is not > 0
    acc = _bf(torch, rng, n, 2 * h, 2 * w, ctot)
    dx = acc.clone()
    call("of_cnn_avgpool2_relu_bwd", _P(small), ctot, coff, n, 2 * h, 2 * w, C, _P(dx), ctot, coff, accumulate, _P(act),
         ctot, coff, _sp())
    torch.cuda.synchronize()
    sl = slice(coff, coff + C)
    want = _f(acc)
    g = O.bf16(O.avgpool2_bwd(_f(small)[..., sl]) + (want[..., sl] if accumulate else 0))
    want[..., sl] = np.where(_f(act)[..., sl] > 0, g, 0)
    assert np.array_equal(_f(dx), want)
    big, act = acc, _bf(torch, rng, n, h, w, ctot)
    dx = small.clone()
    call("of_cnn_upsample2_relu_bwd", _P(big), ctot, coff, n, h, w, C, _P(dx), ctot, coff, _P(act), ctot, coff, _sp())
    torch.cuda.synchronize()
    want = _f(small)
    want[..., sl] = np.where(_f(act)[..., sl] > 0, O.bf16(O.upsample2_bwd(_f(big)[..., sl])), 0)
    assert np.array_equal(_f(dx), want)


@pytest.mark.parametrize("n,H,W,cin,cout,store", [(1, 16, 16, 16, 32, 32), (2, 8, 16, 64, 96, 96), (1, 16, 16, 32, 32, 20),
                                                  (2, 8, 8, 256, 384, 384)])
def test_input_gradient_with_mask(torch, n, H, W, cin, cout, store):
    from ofb200._lib import call
    rng = np.random.default_rng(cin + cout)
    dy, w, act = _bf(torch, rng, n, H, W, cin), _bf(torch, rng, 9, cout, cin), _bf(torch, rng, n, H, W, cout + 16)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    plain = torch.zeros((n, H, W, cout + 8), dtype=torch.bfloat16, device="cuda")
    fused = torch.zeros_like(plain)
    call("of_cnn_conv3x3", _P(dy), n, H, W, cin, cin, 0, _P(w), cout, None, 0, _P(plain), cout + 8, 8, store, _P(err), _sp())
    call("of_cnn_relu_bwd", _P(plain), cout + 8, 8, _P(act), cout + 16, 16, n * H * W, store, _sp())
    call("of_cnn_conv3x3_relu_bwd", _P(dy), n, H, W, cin, cin, 0, _P(w), cout, _P(act), cout + 16, 16, _P(fused), cout + 8,
         8, store, _P(err), _sp())
    torch.cuda.synchronize()
    assert int(err.item()) == 0 and torch.equal(plain, fused) and int((fused == 0).sum()) > 0


@pytest.mark.parametrize("H,W,pad", [(1, 1, 0), (3, 5, 3), (1, 4097, 0), (127, 131, 5), (256, 256, 0), (257, 256, 0)])
@pytest.mark.parametrize("cpad", [2, 16])
def test_pack_pair_sizes(torch, H, W, pad, cpad):
    import cnn_oracle as O
    from ofb200._lib import call
    rng = np.random.default_rng(H)
    a, b = (rng.uniform(0, 200, (H, W + pad)).astype(np.float32) for _ in range(2))
    if H == 3:
        b[:, :W] = 0.0  # a black frame packs as 0
    at, bt = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    a, b = a[:, :W], b[:, :W]
    mx = torch.full((2,), 7, dtype=torch.int32, device="cuda")
    out = torch.full((H, W, cpad), 3.0, dtype=torch.bfloat16, device="cuda")
    call("of_cnn_pack_pair", _P(at), _P(bt), H, W, W + pad, _P(mx), _P(out), cpad, _sp())
    torch.cuda.synchronize()
    o = _f(out)
    assert np.array_equal(o[..., 0], O.bf16(a / a.max()))
    assert np.array_equal(o[..., 1], O.bf16(b / b.max()) if b.any() else b)
    assert not o[..., 2:].any()
    assert np.array_equal(mx.cpu().numpy().view(np.float32), np.float32([a.max(), b.max()]))


def test_pack_weights_of_all_layers(torch):
    from ofb200._lib import call
    rng = np.random.default_rng(4)
    shapes = [(2, 32, 16, 32, 0), (32, 2, 32, 16, 1), (96, 64, 96, 64, 1), (256, 384, 256, 384, 0), (1, 1, 16, 16, 1)]
    ws, many, one = [], [], []
    for co, ci, cp, ip, flip in shapes:
        ws.append(torch.from_numpy(rng.normal(0, 1, (9, co, ci)).astype(np.float32)).cuda())
        many.append(torch.full((9, cp, ip), 5.0, dtype=torch.bfloat16, device="cuda"))
        one.append(torch.full((9, cp, ip), 6.0, dtype=torch.bfloat16, device="cuda"))
        call("of_cnn_pack_weights", _P(ws[-1]), co, ci, cp, ip, flip, _P(one[-1]), _sp())
    n = len(shapes)
    call("of_cnn_pack_weights_many", n, (ctypes.c_void_p * n)(*[w.data_ptr() for w in ws]),
         (ctypes.c_int * (5 * n))(*[d for s in shapes for d in s]), (ctypes.c_void_p * n)(*[o.data_ptr() for o in many]), _sp())
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(many, one))


@pytest.mark.parametrize("n,H,W,cin,cout,coff", [(10, 64, 64, 32, 2, 0), (10, 64, 64, 2, 32, 0), (10, 64, 64, 96, 32, 8),
                                                 (10, 64, 64, 20, 30, 4), (4, 64, 64, 64, 64, 0), (2, 64, 64, 192, 64, 0),
                                                 (4, 64, 64, 40, 128, 0), (64, 16, 16, 128, 144, 0), (5, 64, 64, 48, 48, 0)])
def test_weight_gradient_taps_per_cta(torch, n, H, W, cin, cout, coff):
    """Sizes with work enough for nine or three taps per CTA.  Sums of n H W products of two bfloat16
    values of unit variance, accumulated in float32 in any order: 1e-4 of the largest, as for one tap."""
    import cnn_oracle as O
    from ofb200._lib import call
    rng = np.random.default_rng(cin + cout)
    xct, dct = (max(16, cin + coff) + 7) // 8 * 8, max(16, (cout + 7) // 8 * 8)
    coff = coff // 8 * 8
    x, dy = _bf(torch, rng, n, H, W, xct), _bf(torch, rng, n, H, W, dct)
    dw = torch.zeros((9, cout, cin), dtype=torch.float32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    call("of_cnn_conv3x3_wgrad_tc", _P(x), xct, coff, _P(dy), dct, 0, n, H, W, cin, cout, _P(dw), _P(err), _sp())
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    want = O.conv3x3_wgrad(_f(x)[..., coff:coff + cin], _f(dy)[..., :cout])
    assert np.max(np.abs(dw.cpu().numpy() - want)) <= 1e-4 * np.max(np.abs(want))


@pytest.mark.parametrize("n,H,W,cin,cout", [(10, 64, 64, 8, 40), (10, 64, 64, 6, 41), (10, 64, 64, 40, 8), (2, 64, 64, 72, 137),
                                            (8, 16, 16, 129, 24), (2, 8, 8, 33, 33)])
def test_weight_gradient_sides_ending_inside_a_warp(torch, n, H, W, cin, cout):
    """Wider sides that no multiple of 32 channels makes: some lanes of a warp have no channel to add while
    the warp goes on reading accumulators together.  Nothing outside dw is written; the tolerance is the
    one above."""
    import cnn_oracle as O
    from ofb200._lib import call
    rng = np.random.default_rng(cin + cout)
    xct, dct = max(16, (cin + 7) // 8 * 8), max(16, (cout + 7) // 8 * 8)
    x, dy = _bf(torch, rng, n, H, W, xct), _bf(torch, rng, n, H, W, dct)
    size = 9 * cout * cin
    buf = torch.zeros(size + 64, dtype=torch.float32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    call("of_cnn_conv3x3_wgrad_tc", _P(x), xct, 0, _P(dy), dct, 0, n, H, W, cin, cout, _P(buf), _P(err), _sp())
    torch.cuda.synchronize()
    assert int(err.item()) == 0 and not buf[size:].any()
    want = O.conv3x3_wgrad(_f(x)[..., :cin], _f(dy)[..., :cout])
    got = buf[:size].cpu().numpy().reshape(9, cout, cin)
    assert np.max(np.abs(got - want)) <= 1e-4 * np.max(np.abs(want))
