"""FP32 filter banks under DownsampleOutput(2), in blocks of 16 planes (large grids whose
blocks are nearly full) and of 4, bit for bit against the FP32 oracle."""
import numpy as np
import pytest
import torch

import oracle as O
from cctconv import _lib
from helpers import bitwise_equal

pytestmark = pytest.mark.gpu


# 32 x 16 outputs a tile: 132, 128, 126 (small blocks), 144 blocks of 16 planes, of which
# the last is partly filled; 1x1 from 40 blocks on
@pytest.mark.parametrize("mode", [O.PROJECT_REDUCE, O.BACKPROJECT_REDUCE])
@pytest.mark.parametrize("B,N,K,rows,cols,R,border", [
    (33, 3, 30, 34, 66, 5, O.CLAMP), (16, 2, 61, 10, 130, 7, O.CYCLIC), (21, 4, 29, 66, 8, 5, O.ZERO),
    (48, 2, 47, 16, 34, 9, O.ZERO), (10, 5, 62, 30, 10, 1, O.CLAMP), (9, 4, 60, 30, 10, 1, O.CYCLIC)])
def test_down2(mode, B, N, K, rows, cols, R, border):
    rng = np.random.default_rng(K)
    x = rng.standard_normal((B * N, rows, cols)).astype(np.float32)
    f = rng.standard_normal((K * N, R, R)).astype(np.float32)
    orient = O.XCORR if mode == O.PROJECT_REDUCE else O.CONV
    od = O.make_desc(rows, cols, R, R, planes=B * N, f_planes=K * N, batch=B, border=border, orient=orient,
                     sampling=O.DOWN, step=2, mode=mode)
    ref = O.conv(od, x, f)
    for flags, want in ((0, ref), (_lib.FLAG_RELU, np.maximum(ref, 0))):
        plan = _lib.Plan(_lib.new_desc(image_rows=rows, image_cols=cols, image_planes=B * N, filter_rows=R,
                                       filter_cols=R, filter_planes=K * N, batch_size=B, border=border,
                                       orientation=orient, sampling=O.DOWN, step=2, vector_mode=mode, flags=flags))
        assert plan.algo == _lib.PLAN_FRAME_F32
        y = torch.full(ref.shape, float("nan"), device="cuda")
        xd, fd = torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda()
        plan.run(xd.data_ptr(), fd.data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert bitwise_equal(y.cpu().numpy(), want)
        plan.close()
