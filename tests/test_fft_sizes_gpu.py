"""Every transform length of the FFT path (rows 2^4..2^12, columns 2^4..2^12
points), with the grid rows past the field's border left out, a filter's rows
in the image's launch, and results stored from the last pass: within the FFT
path's normwise 1e-5 of the FP64 direct oracle."""
import numpy as np
import pytest
import torch

import oracle as O
from cctconv import _lib

pytestmark = pytest.mark.gpu

TOL = 1e-5
BORDERS = {"zero": O.ZERO, "clamp": O.CLAMP, "cyclic": O.CYCLIC}


def _run(plan, x, f):
    rows, cols, planes = plan.shape
    y = torch.full((planes, rows, cols), float("nan"), device="cuda")
    plan.run(x.data_ptr(), 0 if f is None else f.data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return y.cpu().numpy()


@pytest.mark.parametrize("border", list(BORDERS))
@pytest.mark.parametrize("rows,cols,R,S,planes,fplanes", [
    (9, 20, 3, 5, 0, 0), (16, 32, 5, 5, 2, 0), (17, 41, 7, 7, 0, 3), (33, 100, 9, 3, 2, 2), (64, 64, 15, 15, 5, 0),
    (70, 141, 31, 31, 0, 0), (130, 300, 41, 25, 3, 0), (260, 515, 63, 63, 0, 0), (512, 256, 47, 47, 2, 2),
    (515, 1030, 9, 9, 0, 0), (1030, 2046, 5, 7, 0, 0), (2050, 513, 7, 5, 0, 0), (40, 4100, 5, 5, 0, 0),
    (1024, 1024, 5, 5, 0, 0)])
def test_lengths(rows, cols, R, S, planes, fplanes, border):
    rng = np.random.default_rng(rows + cols)
    x = rng.uniform(-1, 1, (max(planes, 1), rows, cols)).astype(np.float32)
    f, f2 = (rng.uniform(-1, 1, (max(fplanes, 1), R, S)).astype(np.float32) for _ in range(2))
    orient = O.CONV if rows % 2 else O.XCORR
    od = O.make_desc(rows, cols, R, S, planes=planes, f_planes=fplanes, border=BORDERS[border], orient=orient)
    ref, ref2 = (O.conv(od, x, k, np.float64) for k in (f, f2))
    plan = _lib.Plan(_lib.new_desc(image_rows=rows, image_cols=cols, image_planes=planes, filter_rows=R, filter_cols=S,
                                   filter_planes=fplanes, border=BORDERS[border], orientation=orient,
                                   algo=_lib.ALGO_FFT))
    if plan.algo != _lib.PLAN_FFT:
        pytest.skip("FFT grid does not hold the extension")
    xd = torch.from_numpy(x).cuda()
    for k, want in ((f, ref), (f2, ref2), (f, ref)):  # a filter that changes from run to run
        assert O.rel_errors(_run(plan, xd, torch.from_numpy(k).cuda()), want)[0] <= TOL
    plan.set_static_filter(f2.ctypes.data)
    assert O.rel_errors(_run(plan, xd, None), ref2)[0] <= TOL
    plan.close()
