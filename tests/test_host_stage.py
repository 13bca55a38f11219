"""of_host_stage, the copy into upload buffers: byte-exact at every alignment of the destination and
the source and on both sides of the thread pool's threshold, nothing written outside, overlap refused."""
import numpy as np
import pytest


@pytest.mark.parametrize("n", [0, 1, 15, 64, 255, 256, 333, 4096, (1 << 20) - 1, 1 << 20, (1 << 20) + 77, 5 * (1 << 20) + 4099])
@pytest.mark.parametrize("dst_off,src_off", [(0, 0), (1, 0), (15, 3), (8, 8)])
def test_host_stage(n, dst_off, src_off):
    from ofb200 import _lib
    rng = np.random.default_rng(n + dst_off)
    src = rng.integers(0, 256, n + 32, dtype=np.uint8)
    dst = np.full(n + 64, 7, np.uint8)
    want = dst.copy()
    want[dst_off:dst_off + n] = src[src_off:src_off + n]
    assert _lib.lib().of_host_stage(dst.ctypes.data + dst_off, src.ctypes.data + src_off, n) == 0
    assert np.array_equal(dst, want)


def test_host_stage_refuses_overlap_and_converts_through_numpy():
    from ofb200 import _lib, stage_copyto
    buf = np.zeros(1 << 21, np.uint8)
    assert _lib.lib().of_host_stage(buf.ctypes.data + 16, buf.ctypes.data, 1 << 20) == -1
    a = np.random.default_rng(1).random((300, 1024), dtype=np.float32)
    for src in (a, a[::-1], a.T.copy().T, a.astype(np.float64)):
        out = np.zeros_like(a)
        stage_copyto(out, src)
        assert np.array_equal(out, src.astype(np.float32))


def test_batch_staging_takes_what_copy_takes():
    """HostBatch's staging copy: plain memory, strided and negated views, other types."""
    import torch
    from ofb200.batch import _stage
    a = torch.from_numpy(np.random.default_rng(2).random((300, 1030), dtype=np.float32))
    neg = torch.conj(torch.complex(a, a)).imag  # a lazily negated view: it has no numpy form
    assert neg.is_neg()
    for t in (a[:, :1024].contiguous(), a[:, 3:1027], a[:, :1024].double(), neg[:, :1024], a[:, :1024].clone().requires_grad_()):
        p = torch.zeros(300, 1024)
        _stage(p, t)
        assert torch.equal(p, t.detach().float()) and not p.requires_grad
