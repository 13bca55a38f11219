"""Polynomial expansion into rows that are 16-byte aligned (vector stores) and into rows that are not
(stores through shared memory): bit-identical, at the edges of the 240 x 8 tile."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("poly", [5, 7])
@pytest.mark.parametrize("h,w", [(3, 3), (7, 239), (8, 240), (9, 241), (16, 247), (17, 480), (25, 485)])
def test_polyexp_row_alignment(cuda_ok, h, w, poly):
    import ctypes
    import torch
    import Farneback_PyCL as F
    from ofb200 import ops
    from ofb200._lib import call
    consts = F.Farneback_PyCL(polyN=poly)._poly
    gk = np.array([0.6, 0.2], np.float32)
    x = np.random.default_rng(h * w).uniform(0, 255, (h, w)).astype(np.float32)
    out = []
    for pitch in ((w + 3) // 4 * 4, (w + 3) // 4 * 4 + 1):
        src = torch.zeros(h, pitch, device="cuda")
        src[:, :w] = torch.from_numpy(x).cuda()
        for blurred in (False, True):
            dst = torch.full((5 * h, pitch), 7.0, device="cuda")
            s, d = ctypes.c_void_p(src.data_ptr()), ctypes.c_void_p(dst.data_ptr())
            if blurred:
                call("of_fb_polyexp_blurred", s, d, h, w, pitch, gk.ctypes.data, ctypes.byref(consts), ops.stream_ptr())
            else:
                call("of_fb_polyexp", s, d, h, w, pitch, ctypes.byref(consts), ops.stream_ptr())
            assert bool((dst[:, w:] == 7.0).all())  # nothing beyond the image
            out.append(dst[:, :w].clone())
    assert torch.equal(out[0], out[2]) and torch.equal(out[1], out[3])
