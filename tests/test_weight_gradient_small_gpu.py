"""Weight gradients of small gradient fields: the FP32 kernels on both sides of the sizes
from which four planes share a lane, bit for bit; the split-BF16 sum with 1, 4 and 16
threads per output, within the path's 1e-5 of FP64 and the same bits every run."""
import numpy as np
import pytest
import torch

import oracle as O
from cctconv import _lib
from helpers import bitwise_equal

pytestmark = pytest.mark.gpu


def _run(B, C, L, Hg, Wg, OH, OW, mode, prec):
    rng = np.random.default_rng(Hg * 100 + OW)
    H, W = Hg + OH - 1, Wg + OW - 1
    x = rng.standard_normal((B * C, H, W)).astype(np.float32)
    g = rng.standard_normal((B * L, Hg, Wg)).astype(np.float32)
    od = O.make_desc(H, W, Hg, Wg, planes=B * C, f_planes=B * L, batch=B, border=O.VALID, orient=O.XCORR, mode=mode)
    plan = _lib.Plan(_lib.new_desc(image_rows=H, image_cols=W, image_planes=B * C, filter_rows=Hg, filter_cols=Wg,
                                   filter_planes=B * L, batch_size=B, border=_lib.BORDER_VALID,
                                   orientation=_lib.CROSS_CORRELATION, vector_mode=mode, precision=prec))
    rows, cols, planes = plan.shape
    xd, gd = torch.from_numpy(x).cuda(), torch.from_numpy(g).cuda()
    runs = []
    for _ in range(2):
        y = torch.full((planes, rows, cols), float("nan"), device="cuda")
        plan.run(xd.data_ptr(), gd.data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream)
        runs.append(y.cpu().numpy())
    algo = plan.algo
    plan.close()
    assert bitwise_equal(runs[0], runs[1])
    return od, x, g, runs[0], algo


# few and many (plane, row) groups of 1 to 4 gradient rows
@pytest.mark.parametrize("mode", [O.FILTER_ADJOINT, O.FILTER_ADJOINT_REDUCE])
@pytest.mark.parametrize("B,C,L", [(1, 3, 5), (8, 38, 26)])
@pytest.mark.parametrize("Hg,Wg,OH,OW", [(1, 1, 1, 1), (1, 4, 3, 3), (2, 2, 3, 3), (3, 3, 2, 2), (1, 16, 5, 5),
                                         (2, 5, 5, 4), (3, 2, 5, 5), (4, 4, 3, 3), (2, 2, 8, 8)])
def test_fp32(B, C, L, Hg, Wg, OH, OW, mode):
    od, x, g, got, algo = _run(B, C, L, Hg, Wg, OH, OW, mode, _lib.PREC_FP32)
    assert algo == _lib.PLAN_FILTER_ADJOINT and bitwise_equal(got, O.conv(od, x, g))


@pytest.mark.parametrize("B,C,L,Hg,Wg,OH,OW", [(1, 12, 7, 1, 1, 30, 30), (2, 38, 20, 8, 8, 5, 7), (1, 64, 64, 24, 24, 8, 7),
                                               (2, 24, 20, 30, 31, 7, 7), (4, 16, 16, 20, 19, 3, 3)])
def test_split_bf16(B, C, L, Hg, Wg, OH, OW):
    od, x, g, got, algo = _run(B, C, L, Hg, Wg, OH, OW, O.FILTER_ADJOINT_REDUCE, _lib.PREC_BF16X3)
    if algo != _lib.PLAN_FILTER_ADJOINT_BF16X3:
        pytest.skip("not a tensor-core weight gradient")
    assert O.rel_errors(got, O.conv(od, x, g, np.float64))[0] <= 1e-5
