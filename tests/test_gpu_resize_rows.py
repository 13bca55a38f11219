"""Resizes sum four rows at a time: heights that leave 1, 2 and 3 rows over, widths at the edge of a
CTA's 128 columns, few and many taps (kept weight tables), bit for bit against the oracle."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("src,dst", [((1, 9), (1, 4)), ((5, 129), (5, 64)), ((18, 258), (9, 129)), ((35, 300), (7, 127)),
                                     ((66, 1040), (9, 130)), ((67, 2100), (8, 128)), ((9, 7000), (3, 100)), ((7, 64), (15, 129))])
@pytest.mark.parametrize("bicubic", [False, True])
def test_resize_rows(cuda_ok, src, dst, bicubic):
    import torch
    from ofb200 import ops
    a = np.random.default_rng(src[0] * src[1]).normal(100, 50, src).astype(np.float32)
    out = ops.resize(torch.from_numpy(a).cuda(), (dst[1], dst[0]), bicubic)
    assert np.array_equal(out.cpu().numpy(), O.resize(a, (dst[1], dst[0]), 1 if bicubic else 0))
