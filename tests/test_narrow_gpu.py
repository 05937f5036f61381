"""Fields narrower than the stencils' 64-column tiles, whose tiles are staged as far as
the field's own columns: bit for bit against the FP32 oracle."""
import numpy as np
import pytest
import torch

import cctconv as C
import oracle as O
from cctconv import _lib
from helpers import bitwise_equal

pytestmark = pytest.mark.gpu

BORDERS = {"clamp": (O.CLAMP, C.BorderClamp), "cyclic": (O.CYCLIC, C.BorderCyclic), "zero": (O.ZERO, C.BorderZero)}


# 16-byte staging (widths 4, 16, 36, 68: the last one with a second, narrow tile) and
# 4-byte staging; small, shared-weight and phase kernels
@pytest.mark.parametrize("border", list(BORDERS))
@pytest.mark.parametrize("cols", [1, 2, 4, 9, 16, 31, 36, 66, 68])
@pytest.mark.parametrize("R,sampling,step", [(3, O.NOSAMPLE, 1), (5, O.DOWN, 2), (7, O.DOWN, 2), (9, O.NOSAMPLE, 1),
                                             (21, O.NOSAMPLE, 1), (5, O.UP, 2), (7, O.UP, 3)])
def test_planes(R, sampling, step, cols, border):
    if (sampling == O.UP and border == "clamp") or (sampling == O.DOWN and cols % 2):
        pytest.skip("not a legal combination")
    rng = np.random.default_rng(cols * 100 + R)
    rows, planes = 34, 3
    x = rng.uniform(-1, 1, (planes, rows, cols)).astype(np.float32)
    f = rng.uniform(-1, 1, (R, R)).astype(np.float32)
    od = O.make_desc(rows, cols, R, R, planes=planes, border=BORDERS[border][0], orient=O.CONV, sampling=sampling, step=step)
    plan = _lib.Plan(_lib.new_desc(image_rows=rows, image_cols=cols, image_planes=planes, filter_rows=R, filter_cols=R,
                                   border=BORDERS[border][0], orientation=_lib.CONVOLUTION, sampling=sampling, step=step,
                                   algo=_lib.ALGO_DIRECT))
    xd, fd = torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda()
    y = torch.full((planes, plan.shape[0], plan.shape[1]), float("nan"), device="cuda")
    for _ in range(2):  # the second time over what the first left in shared memory
        plan.run(xd.data_ptr(), fd.data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert bitwise_equal(y.cpu().numpy(), O.conv(od, x, f))
    plan.close()


@pytest.mark.parametrize("border", list(BORDERS))
@pytest.mark.parametrize("cols", [1, 6, 16, 33, 65])
@pytest.mark.parametrize("rl,cl", [(1, 1), (5, 5), (15, 31)])
def test_separable(rl, cl, cols, border):
    rng = np.random.default_rng(cols)
    x = rng.uniform(-1, 1, (4, 40, cols)).astype(np.float32)
    rf, cf = rng.uniform(-1, 1, rl).astype(np.float32), rng.uniform(-1, 1, cl).astype(np.float32)
    y = C.convolveSeparable(torch.from_numpy(x).cuda(), torch.from_numpy(rf).cuda(), torch.from_numpy(cf).cuda(),
                            BORDERS[border][1])
    assert bitwise_equal(y.cpu().numpy(), O.separable(x, rf, cf, BORDERS[border][0], O.CONV))
