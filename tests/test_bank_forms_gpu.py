"""The filter-bank kernel's block forms (128 filters a block; 64 filters x two
taps) at their edges: filter counts around a block, odd tap counts, ragged plane
counts, every border, both samplings, both directions, reductions long enough to
be promoted.  Bounds: each precision's own, 1e-5 (two terms) and 3e-6 (three
terms: 2^-24 per term of a few thousand) normwise against FP64."""
import numpy as np
import pytest
import torch

import oracle as O
from cctconv import _lib

pytestmark = pytest.mark.gpu

BOUND = {_lib.PREC_BF16X3: 1e-5, _lib.PREC_BF16X6: 3e-6}
N_, D_, U_ = O.NOSAMPLE, O.DOWN, O.UP


@pytest.mark.parametrize("prec", [_lib.PREC_BF16X3, _lib.PREC_BF16X6])
@pytest.mark.parametrize("mode", [O.PROJECT_REDUCE, O.BACKPROJECT_REDUCE])
@pytest.mark.parametrize("batch,C,K,rows,cols,R,border,sampling,step", [
    (1, 16, 65, 9, 11, 3, O.ZERO, N_, 1), (2, 20, 96, 17, 30, 5, O.CLAMP, N_, 1), (1, 33, 128, 40, 44, 3, O.CYCLIC, N_, 1),
    (1, 40, 129, 12, 70, 3, O.FULL, N_, 1), (2, 70, 200, 14, 15, 3, O.VALID, N_, 1), (3, 8, 130, 20, 24, 3, O.ZERO, D_, 2),
    (1, 24, 80, 11, 13, 5, O.ZERO, U_, 2), (1, 300, 140, 10, 12, 5, O.ZERO, N_, 1), (2, 16, 64, 30, 31, 7, O.CLAMP, N_, 1),
    (1, 9, 40, 25, 64, 5, O.ZERO, N_, 1), (4, 64, 32, 33, 20, 5, O.CYCLIC, N_, 1), (1, 5, 3, 50, 52, 7, O.VALID, N_, 1),
    (1, 160, 60, 16, 16, 7, O.ZERO, N_, 1), (1, 32, 33, 13, 9, 5, O.CYCLIC, U_, 2), (24, 32, 128, 28, 28, 1, O.ZERO, N_, 1)])
def test_forms(batch, C, K, rows, cols, R, border, sampling, step, mode, prec):
    rng = np.random.default_rng(C * 1000 + K)
    x = rng.standard_normal((batch * C, rows, cols)).astype(np.float32)
    f = (rng.standard_normal((K * C, R, R)) * np.sqrt(2.0 / (C * R * R))).astype(np.float32)
    orient = O.XCORR if mode == O.PROJECT_REDUCE else O.CONV
    od = O.make_desc(rows, cols, R, R, planes=batch * C, f_planes=K * C, batch=batch, border=border, orient=orient,
                     sampling=sampling, step=step, mode=mode)
    ref = O.conv(od, x, f, np.float64)
    plan = _lib.Plan(_lib.new_desc(image_rows=rows, image_cols=cols, image_planes=batch * C, filter_rows=R,
                                   filter_cols=R, filter_planes=K * C, batch_size=batch, border=border,
                                   orientation=orient, sampling=sampling, step=step, vector_mode=mode, precision=prec,
                                   flags=_lib.FLAG_RELU))
    assert plan.algo == _lib.PLAN_FRAME_BF16X3
    xd, fd = torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda()
    runs = []
    for static in (False, False, True):
        if static:
            plan.set_static_filter(f.ctypes.data)
        y = torch.full(ref.shape, float("nan"), device="cuda")
        plan.run(xd.data_ptr(), 0 if static else fd.data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream)
        runs.append(y.cpu().numpy())
    plan.close()
    assert _lib.LIB.cct_device_status() == _lib.OK
    assert np.array_equal(runs[0], runs[1]) and np.array_equal(runs[0], runs[2])
    scale = np.abs(ref).max()
    assert np.abs(runs[0] - np.maximum(ref, 0)).max() <= BOUND[prec] * scale


# DownsampleOutput(2) in three terms with one input phase per halo block, and
# two-term layers whose stages the plan lengthens
@pytest.mark.parametrize("prec", [_lib.PREC_BF16X3, _lib.PREC_BF16X6])
@pytest.mark.parametrize("batch,C,K,rows,cols,R,border", [
    (1, 64, 64, 64, 224, 3, O.ZERO), (2, 32, 32, 40, 44, 7, O.CYCLIC), (1, 40, 50, 32, 120, 5, O.CLAMP),
    (3, 17, 64, 18, 226, 3, O.CLAMP), (1, 128, 60, 20, 160, 5, O.ZERO), (1, 20, 20, 16, 16, 9, O.ZERO)])
def test_down2(batch, C, K, rows, cols, R, border, prec):
    test_forms(batch, C, K, rows, cols, R, border, O.DOWN, 2, O.PROJECT_REDUCE, prec)
    test_forms(batch, C, K, rows, cols, R, border, O.DOWN, 2, O.BACKPROJECT_REDUCE, prec)


# filter operands of one to three rows per packing thread of a CTA on each SM
@pytest.mark.parametrize("prec", [_lib.PREC_BF16X3, _lib.PREC_BF16X6])
@pytest.mark.parametrize("C,K,R", [(84, 32, 7), (96, 32, 7), (160, 32, 7), (176, 32, 7), (96, 64, 5), (200, 64, 5)])
def test_pack_rows(C, K, R, prec):
    test_forms(1, C, K, 12, 19, R, O.FULL, O.NOSAMPLE, 1, O.PROJECT_REDUCE, prec)
