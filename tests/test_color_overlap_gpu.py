"""A ColorField convolved into its own bytes, and into bytes that overlap them, gives
what it gives into others."""
import numpy as np
import pytest
import torch

import oracle as O
from cctconv import _lib

pytestmark = pytest.mark.gpu


# one kernel (5x5 and 1x1; the largest in several waves of CTAs), three launches (9x9), outputs smaller and larger than the
# image; the output `shift` pixels after the image's start
@pytest.mark.parametrize("rows,cols,R,border,shift", [
    (1200, 1600, 5, O.CLAMP, 0), (1200, 1601, 5, O.CYCLIC, 1), (1200, 1600, 5, O.ZERO, -800), (64, 64, 1, O.CLAMP, 1),
    (301, 403, 7, O.VALID, 0), (301, 403, 3, O.FULL, 0), (200, 300, 9, O.CLAMP, 0)])
def test_overlap(rows, cols, R, border, shift):
    rng = np.random.default_rng(rows)
    x = rng.integers(0, 256, (rows, cols, 4), dtype=np.uint8)
    f = rng.random((R, R)).astype(np.float32)
    f /= f.sum()
    want = O.color_conv(O.make_desc(rows, cols, R, R, border=border), x, f)
    plan = _lib.ColorPlan(_lib.new_desc(image_rows=rows, image_cols=cols, filter_rows=R, filter_cols=R, border=border,
                                        algo=_lib.ALGO_DIRECT))
    fd = torch.from_numpy(f).cuda()
    st = torch.cuda.current_stream().cuda_stream
    before, after = max(0, -shift), max(shift, 0)
    for _ in range(3):
        buf = torch.zeros(4 * (before + after + max(x.size, want.size) // 4), device="cuda", dtype=torch.uint8)
        image = buf[4 * before:4 * before + x.size]
        image.copy_(torch.from_numpy(x).flatten())
        out = buf[4 * after:4 * after + want.size]
        plan.run(image.data_ptr(), fd.data_ptr(), out.data_ptr(), st)
        assert np.array_equal(out.cpu().numpy().reshape(want.shape), want)
    plan.close()
