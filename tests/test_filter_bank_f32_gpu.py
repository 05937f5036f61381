"""The FP32 filter bank and its weight gradient at the edges of their tiles,
staging rings and splits, bit for bit against the FP32 oracle."""
import numpy as np
import pytest
import torch

import oracle as O
from cctconv import _lib
from helpers import bitwise_equal

pytestmark = pytest.mark.gpu


def _run(od, x, f, shift=0, flags=0):
    d = _lib.new_desc(image_rows=od.rows, image_cols=od.cols, image_planes=od.planes, filter_rows=od.f_rows,
                      filter_cols=od.f_cols, filter_planes=od.f_planes, batch_size=od.batch, border=od.border,
                      orientation=od.orient, sampling=od.sampling, step=od.step, vector_mode=od.mode, flags=flags)
    plan = _lib.Plan(d)
    rows, cols, planes = plan.shape
    xd = torch.zeros(x.size + shift, device="cuda")
    xd[shift:] = torch.from_numpy(x.reshape(-1)).cuda()
    fd = torch.from_numpy(f).cuda()
    y = torch.full((planes, rows, cols), float("nan"), device="cuda")
    plan.run(xd.data_ptr() + 4 * shift, fd.data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    plan.close()
    return y.cpu().numpy()


# input planes fewer than, equal to and past the three staging buffers; output
# planes that do not fill a block of 4 or 16; one large grid of 16-plane blocks
@pytest.mark.parametrize("mode", [O.PROJECT_REDUCE, O.BACKPROJECT_REDUCE])
@pytest.mark.parametrize("B,N,K,rows,cols,R,border,sampling,step", [
    (1, 1, 1, 16, 32, 3, O.ZERO, O.NOSAMPLE, 1), (2, 2, 5, 17, 33, 5, O.CLAMP, O.NOSAMPLE, 1),
    (1, 3, 16, 9, 7, 7, O.CYCLIC, O.NOSAMPLE, 1), (1, 4, 18, 33, 65, 9, O.FULL, O.NOSAMPLE, 1),
    (3, 7, 3, 24, 40, 5, O.VALID, O.NOSAMPLE, 1), (2, 5, 6, 34, 66, 9, O.ZERO, O.DOWN, 2),
    (64, 5, 32, 20, 40, 3, O.ZERO, O.NOSAMPLE, 1), (130, 2, 14, 10, 12, 1, O.CLAMP, O.NOSAMPLE, 1),
    (40, 3, 33, 34, 34, 3, O.CYCLIC, O.DOWN, 2)])
def test_bank(mode, B, N, K, rows, cols, R, border, sampling, step):
    rng = np.random.default_rng(rows * 100 + K)
    x = rng.standard_normal((B * N, rows, cols)).astype(np.float32)
    f = rng.standard_normal((K * N, R, R)).astype(np.float32)
    od = O.make_desc(rows, cols, R, R, planes=B * N, f_planes=K * N, batch=B, border=border,
                     orient=O.XCORR if mode == O.PROJECT_REDUCE else O.CONV, sampling=sampling, step=step, mode=mode)
    ref = O.conv(od, x, f)
    assert bitwise_equal(_run(od, x, f), ref)
    assert bitwise_equal(_run(od, x, f, flags=_lib.FLAG_RELU), np.maximum(ref, 0))


# gradient rows that end inside a step of 4, 8 or 16; gradient columns that end
# inside a float4; (plane, row) pairs and gradient planes that do not fill a
# warp or a group; 4- and 16-byte staging
@pytest.mark.parametrize("orient", [O.XCORR, O.CONV])
@pytest.mark.parametrize("B,C,L,Hg,Wg,OH,OW", [
    (1, 1, 1, 1, 1, 1, 1), (2, 3, 5, 3, 7, 3, 3), (1, 7, 4, 17, 16, 5, 5), (2, 9, 6, 16, 13, 7, 7),
    (1, 33, 2, 5, 9, 1, 1), (3, 4, 9, 33, 30, 2, 8), (1, 5, 3, 9, 21, 8, 6), (1, 2, 2, 6, 18, 6, 4),
    (30, 16, 24, 9, 12, 5, 5), (26, 32, 12, 6, 10, 3, 3), (1, 12, 8, 20, 100, 3, 3), (1, 9, 4, 40, 130, 5, 5),
    (1, 8, 4, 12, 390, 7, 7), (2, 8, 4, 10, 700, 3, 2)])
def test_weight_gradient(orient, B, C, L, Hg, Wg, OH, OW):
    rng = np.random.default_rng(Hg * 1000 + Wg)
    H, W = Hg + OH - 1, Wg + OW - 1
    x = rng.standard_normal((B * C, H, W)).astype(np.float32)
    g = rng.standard_normal((B * L, Hg, Wg)).astype(np.float32)
    for mode in (O.FILTER_ADJOINT, O.FILTER_ADJOINT_REDUCE):
        od = O.make_desc(H, W, Hg, Wg, planes=B * C, f_planes=B * L, batch=B, border=O.VALID, orient=orient, mode=mode)
        assert bitwise_equal(_run(od, x, g), O.conv(od, x, g))
    assert bitwise_equal(_run(od, x, g, shift=1), O.conv(od, x, g))
