"""Squares over zero-inserted grids: steps and borders past the phase form's, one and
several terms, at the edges of the 64 x 64 tiles and on both sides of the grid size from
which they are taken, bit for bit against the FP32 oracle."""
import numpy as np
import pytest
import torch

import oracle as O
from cctconv import _lib
from helpers import bitwise_equal

pytestmark = pytest.mark.gpu


def _run(od, x, f, flags=0):
    plan = _lib.Plan(_lib.new_desc(image_rows=od.rows, image_cols=od.cols, image_planes=od.planes, filter_rows=od.f_rows,
                                   filter_cols=od.f_cols, filter_planes=od.f_planes, batch_size=od.batch,
                                   border=od.border, orientation=od.orient, sampling=od.sampling, step=od.step,
                                   vector_mode=od.mode, algo=_lib.ALGO_DIRECT, flags=flags))
    rows, cols, planes = plan.shape
    xd, fd = torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda()
    y = torch.full((planes, rows, cols), float("nan"), device="cuda")
    plan.run(xd.data_ptr(), fd.data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    plan.close()
    return y.cpu().numpy()


@pytest.mark.parametrize("border,step", [(O.ZERO, 4), (O.CYCLIC, 5), (O.FULL, 2), (O.FULL, 3), (O.VALID, 2), (O.VALID, 4)])
@pytest.mark.parametrize("R", [1, 3, 5, 7])
@pytest.mark.parametrize("planes,fplanes,rows,cols", [(0, 0, 33, 65), (3, 0, 8, 7), (0, 5, 16, 16), (2, 2, 21, 40),
                                                      (910, 0, 9, 10), (105, 105, 17, 16)])
def test_planes(planes, fplanes, rows, cols, R, border, step):
    rng = np.random.default_rng(rows + R)
    x = rng.uniform(-1, 1, (max(planes, 1), rows, cols)).astype(np.float32)
    f = rng.uniform(-1, 1, (max(fplanes, 1), R, R)).astype(np.float32)
    od = O.make_desc(rows, cols, R, R, planes=planes, f_planes=fplanes, border=border,
                     orient=O.CONV if rows % 2 else O.XCORR, sampling=O.UP, step=step)
    assert bitwise_equal(_run(od, x, f), O.conv(od, x, f))


@pytest.mark.parametrize("mode", [O.PROJECT_REDUCE, O.BACKPROJECT_REDUCE, O.PROJECT])
@pytest.mark.parametrize("border,step,R", [(O.ZERO, 4, 3), (O.FULL, 2, 5), (O.VALID, 3, 7), (O.CYCLIC, 2, 1)])
def test_several_terms(mode, border, step, R):
    rng = np.random.default_rng(R)
    B, N, K, rows, cols = 2, 5, 3, 13, 24
    x = rng.standard_normal((B * N, rows, cols)).astype(np.float32)
    f = rng.standard_normal((N * K, R, R)).astype(np.float32)
    od = O.make_desc(rows, cols, R, R, planes=B * N, f_planes=N * K, batch=B, border=border,
                     orient=O.CONV if mode == O.BACKPROJECT_REDUCE else O.XCORR, sampling=O.UP, step=step, mode=mode)
    ref = O.conv(od, x, f)
    assert bitwise_equal(_run(od, x, f), ref)
    assert bitwise_equal(_run(od, x, f, _lib.FLAG_RELU), np.maximum(ref, 0))
