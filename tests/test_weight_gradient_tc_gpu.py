"""Split-BF16 weight gradient: the sum over the reduction's splits, with outputs
that do not fill a CTA and few or many splits, within the path's normwise 1e-5
of FP64 and the same bits every run."""
import numpy as np
import pytest
import torch

import oracle as O
from cctconv import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,C,L,Hg,Wg,R", [(1, 1, 1, 6, 7, 1), (2, 3, 5, 9, 11, 3), (1, 16, 16, 57, 43, 3),
                                           (4, 24, 48, 30, 30, 7), (8, 33, 65, 12, 10, 3), (3, 10, 7, 40, 33, 5)])
def test_split_sums(B, C, L, Hg, Wg, R):
    rng = np.random.default_rng(Hg * Wg)
    x = rng.standard_normal((B * C, Hg + R - 1, Wg + R - 1)).astype(np.float32)
    g = rng.standard_normal((B * L, Hg, Wg)).astype(np.float32)
    od = O.make_desc(Hg + R - 1, Wg + R - 1, Hg, Wg, planes=B * C, f_planes=B * L, batch=B, border=O.VALID,
                     orient=O.XCORR, mode=O.FILTER_ADJOINT_REDUCE)
    ref = O.conv(od, x, g, np.float64)
    plan = _lib.Plan(_lib.new_desc(image_rows=Hg + R - 1, image_cols=Wg + R - 1, image_planes=B * C, filter_rows=Hg,
                                   filter_cols=Wg, filter_planes=B * L, batch_size=B, border=_lib.BORDER_VALID,
                                   orientation=_lib.CROSS_CORRELATION, precision=_lib.PREC_BF16X3,
                                   vector_mode=_lib.FILTER_ADJOINT_BLOCK_REDUCE_SUM))
    assert plan.algo == _lib.PLAN_FILTER_ADJOINT_BF16X3
    xd, gd = torch.from_numpy(x).cuda(), torch.from_numpy(g).cuda()
    runs = []
    for _ in range(2):
        y = torch.full((L * C, R, R), float("nan"), device="cuda")
        plan.run(xd.data_ptr(), gd.data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream)
        runs.append(y.cpu().numpy())
    plan.close()
    assert O.rel_errors(runs[0], ref)[0] <= 1e-5
    assert np.array_equal(runs[0], runs[1])
