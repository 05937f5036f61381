"""The filter-bank kernel's forms where their parts differ: each shape asserts the form
and the halo split that the plan gives it.  Filters that do not fill a block, every
border, both directions, both samplings, reductions long enough to be promoted.  Bounds:
each precision's own, 1e-5 (two terms) and 3e-6 (three terms) normwise against FP64."""
import numpy as np
import pytest
import torch

import oracle as O
from cctconv import _lib

pytestmark = pytest.mark.gpu

X3, X6 = _lib.PREC_BF16X3, _lib.PREC_BF16X6
BOUND = {X3: 1e-5, X6: 3e-6}
PLAIN, PAIR, WIDE, WIDE_PAIR = _lib.BANK_PLAIN, _lib.BANK_PAIR, _lib.BANK_WIDE, _lib.BANK_WIDE_PAIR
P, Q = O.PROJECT_REDUCE, O.BACKPROJECT_REDUCE
N_, D_, U_ = O.NOSAMPLE, O.DOWN, O.UP
Z, C, Y, V, F = O.ZERO, O.CLAMP, O.CYCLIC, O.VALID, O.FULL

CASES = [
    # 128 filters a block, two terms
    (X3, WIDE, 1, (1, 3, 260, 40, 70, 3, 3, Z, N_, 1, P)), (X3, WIDE, 1, (8, 3, 65, 95, 37, 3, 1, Z, N_, 1, Q)),
    (X3, WIDE, 1, (2, 3, 65, 31, 113, 3, 3, C, N_, 1, P)), (X3, WIDE, 1, (16, 3, 65, 7, 65, 3, 3, Y, N_, 1, Q)),
    (X3, WIDE, 1, (2, 3, 200, 25, 86, 3, 3, V, N_, 1, Q)), (X3, WIDE, 1, (8, 3, 65, 20, 40, 3, 3, F, N_, 1, P)),
    (X3, WIDE, 1, (8, 8, 260, 70, 16, 3, 3, F, D_, 2, P)), (X3, WIDE, 1, (2, 3, 100, 46, 19, 3, 3, Z, U_, 2, P)),
    (X3, WIDE, 1, (4, 3, 100, 15, 70, 3, 3, Y, U_, 2, Q)), (X3, WIDE, 1, (8, 3, 65, 11, 23, 3, 3, V, U_, 3, Q)),
    # 128 filters a block, three terms; promoted; one input phase per halo block
    (X6, WIDE, 1, (1, 3, 96, 66, 113, 7, 1, Z, N_, 1, P)), (X6, WIDE, 1, (16, 3, 65, 9, 58, 3, 3, C, N_, 1, P)),
    (X6, WIDE, 1, (1, 3, 200, 49, 74, 7, 1, Y, N_, 1, Q)), (X6, WIDE, 1, (4, 8, 65, 107, 21, 3, 1, V, N_, 1, Q)),
    (X6, WIDE, 1, (2, 3, 80, 84, 40, 3, 3, F, N_, 1, P)), (X6, WIDE, 1, (1, 17, 100, 26, 120, 7, 7, Z, D_, 2, P)),
    (X6, WIDE, 1, (1, 17, 80, 34, 56, 7, 7, Z, D_, 2, Q)), (X6, WIDE, 1, (1, 3, 130, 102, 62, 7, 3, C, D_, 2, P)),
    (X6, WIDE, 4, (16, 3, 130, 16, 102, 5, 5, Z, D_, 2, P)), (X6, WIDE, 4, (8, 3, 260, 14, 108, 7, 7, C, D_, 2, Q)),
    (X6, WIDE, 4, (16, 3, 100, 38, 82, 7, 3, Y, D_, 2, Q)), (X6, WIDE, 4, (8, 3, 65, 44, 116, 7, 3, F, D_, 2, Q)),
    (X6, WIDE, 1, (1, 3, 100, 42, 44, 3, 3, Z, U_, 2, Q)), (X6, WIDE, 1, (1, 3, 96, 96, 15, 3, 3, Y, U_, 3, P)),
    (X6, WIDE, 1, (1, 3, 100, 123, 15, 7, 3, V, U_, 2, P)), (X6, WIDE, 1, (2, 3, 80, 68, 13, 3, 3, F, U_, 3, P)),
    # 64 filters a block, one input phase per halo block
    (X6, PLAIN, 4, (2, 3, 16, 16, 36, 5, 5, F, D_, 2, P)), (X6, PLAIN, 4, (1, 64, 16, 10, 24, 7, 7, F, D_, 2, P)),
    # 64 filters x two taps, three terms; promoted; small sums promoted
    (X6, WIDE_PAIR, 1, (1, 3, 16, 15, 36, 5, 5, Z, N_, 1, P)), (X6, WIDE_PAIR, 1, (1, 96, 64, 9, 11, 5, 5, Z, N_, 1, Q)),
    (X6, WIDE_PAIR, 1, (1, 96, 16, 28, 18, 7, 7, C, N_, 1, P)), (X6, WIDE_PAIR, 1, (2, 3, 33, 31, 6, 7, 7, Y, N_, 1, P)),
    (X6, WIDE_PAIR, 1, (1, 64, 33, 32, 10, 7, 7, Y, N_, 1, Q)), (X6, WIDE_PAIR, 1, (1, 16, 33, 44, 11, 5, 5, V, N_, 1, P)),
    (X6, WIDE_PAIR, 1, (1, 16, 16, 22, 52, 5, 5, F, N_, 1, Q)), (X6, WIDE_PAIR, 1, (1, 17, 16, 9, 83, 7, 7, Z, U_, 2, Q)),
    (X6, WIDE_PAIR, 1, (1, 17, 33, 7, 10, 7, 7, Y, U_, 2, Q)), (X6, WIDE_PAIR, 1, (1, 40, 60, 8, 12, 5, 5, F, U_, 2, P)),
    (X6, WIDE_PAIR, 1, (1, 640, 32, 20, 20, 7, 7, Z, N_, 1, P)),
    # 32 filters x two taps
    (X3, PAIR, 1, (1, 9, 20, 25, 31, 5, 5, C, N_, 1, P)), (X3, PAIR, 1, (1, 9, 20, 12, 17, 5, 3, Z, U_, 2, Q)),
]


@pytest.mark.parametrize("prec,form,halo_blocks,shape", CASES)
def test_plan_and_result(prec, form, halo_blocks, shape):
    batch, c, k, rows, cols, R, S, border, sampling, step, mode = shape
    rng = np.random.default_rng(rows * 1000 + cols)
    x = rng.standard_normal((batch * c, rows, cols)).astype(np.float32)
    f = (rng.standard_normal((k * c, R, S)) * np.sqrt(2.0 / (c * R * S))).astype(np.float32)
    orient = O.XCORR if mode == P else O.CONV
    od = O.make_desc(rows, cols, R, S, planes=batch * c, f_planes=k * c, batch=batch, border=border, orient=orient,
                     sampling=sampling, step=step, mode=mode)
    ref = O.conv(od, x, f, np.float64)
    plan = _lib.Plan(_lib.new_desc(image_rows=rows, image_cols=cols, image_planes=batch * c, filter_rows=R,
                                   filter_cols=S, filter_planes=k * c, batch_size=batch, border=border,
                                   orientation=orient, sampling=sampling, step=step, vector_mode=mode, precision=prec))
    assert plan.bank()[:2] == (form, halo_blocks)
    xd, fd = torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda()
    runs = []
    for static in (False, True):
        if static:
            plan.set_static_filter(f.ctypes.data)
        y = torch.full(ref.shape, float("nan"), device="cuda")
        plan.run(xd.data_ptr(), 0 if static else fd.data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream)
        runs.append(y.cpu().numpy())
    plan.close()
    assert _lib.LIB.cct_device_status() == _lib.OK
    assert np.array_equal(runs[0], runs[1])
    assert np.abs(runs[0] - ref).max() <= BOUND[prec] * np.abs(ref).max()


def test_other_plans_have_no_form():
    plan = _lib.Plan(_lib.new_desc(image_rows=20, image_cols=20, filter_rows=3, filter_cols=3))
    assert plan.bank() == (-1, 0, 0)
    plan.close()
