"""The direct stencils' tile edges, remainders and staging forms, bit for bit
against the FP32 oracle (the kernels keep its summation order, so the
tolerance is none)."""
import numpy as np
import pytest
import torch

import oracle as O
from cctconv import _lib
from helpers import bitwise_equal

pytestmark = pytest.mark.gpu

_BORDERS = {"zero": O.ZERO, "clamp": O.CLAMP, "cyclic": O.CYCLIC, "valid": O.VALID, "full": O.FULL}


def _offset(a, shift):
    """A device copy of `a` that starts `shift` floats past an aligned address."""
    t = torch.full((a.size + shift,), float("nan"), device="cuda")
    t[shift:] = torch.from_numpy(a.reshape(-1)).cuda()
    return t, t.data_ptr() + 4 * shift


def _run(od, x, f, shift=0, flags=0):
    d = _lib.new_desc(image_rows=od.rows, image_cols=od.cols, image_planes=od.planes, filter_rows=od.f_rows,
                      filter_cols=od.f_cols, filter_planes=od.f_planes, batch_size=od.batch, border=od.border,
                      orientation=od.orient, sampling=od.sampling, step=od.step, vector_mode=od.mode,
                      algo=_lib.ALGO_DIRECT, flags=flags)
    plan = _lib.Plan(d)
    rows, cols, planes = plan.shape
    xt, xp = _offset(x, shift)
    ft, fp = _offset(f, shift)
    yt, yp = _offset(np.full((planes, rows, cols), np.nan, np.float32), shift)
    plan.run(xp, fp, yp, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    plan.close()
    assert shift == 0 or bool(torch.isnan(yt[:shift]).all())
    return yt[shift:].cpu().numpy().reshape(planes, rows, cols)


def _check(rows, cols, fr, fc, border, orient, planes=0, fplanes=0, sampling=O.NOSAMPLE, step=1, shift=0, bad=False):
    rng = np.random.default_rng(rows * 7919 + cols * 31 + fr)
    x = rng.uniform(-1, 1, (max(planes, 1), rows, cols)).astype(np.float32)
    f = rng.uniform(-1, 1, (max(fplanes, 1), fr, fc)).astype(np.float32)
    if bad:
        x[0, rows // 2, cols // 2] = np.inf
        x[0, 0, 0] = np.nan
        x[0, -1, -1] = np.finfo(np.float32).min
    od = O.make_desc(rows, cols, fr, fc, planes=planes, f_planes=fplanes, border=_BORDERS[border], orient=orient,
                     sampling=sampling, step=step)
    assert bitwise_equal(_run(od, x, f, shift), O.conv(od, x, f))


# 16-byte staging (width a multiple of 4) and 4-byte staging, tall and short
# tiles (64 x 64 and 64 x 16; 64 x 32 and 64 x 16 down-sampling), a last tile of
# one row or column, fields smaller than a tile and than the filter
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("border", ["zero", "clamp", "cyclic", "valid", "full"])
@pytest.mark.parametrize("R", [1, 3, 5, 7])
@pytest.mark.parametrize("planes,rows,cols", [(1, 65, 64), (40, 129, 68), (1, 8, 260), (37, 65, 193), (1, 7, 7)])
def test_small(planes, rows, cols, R, border, shift):
    _check(rows, cols, R, R, border, O.CONV, planes=planes, shift=shift)


@pytest.mark.parametrize("border", ["zero", "clamp", "cyclic"])
@pytest.mark.parametrize("R", [1, 3, 5, 7])
@pytest.mark.parametrize("planes,rows,cols,shift", [(1, 130, 132, 0), (40, 258, 136, 0), (3, 66, 70, 0), (2, 64, 128, 1),
                                                    (1, 2, 4, 0)])
def test_down2(planes, rows, cols, shift, R, border):
    _check(rows, cols, R, R, border, O.XCORR, planes=planes, sampling=O.DOWN, step=2, shift=shift)


# every width of the shared-weight stencil on tall (48 rows) and short (16)
# tiles; a filter taller and one shorter than wide
@pytest.mark.parametrize("S", list(range(3, 33, 2)))
@pytest.mark.parametrize("rows,cols,planes,R,border", [(49, 65, 160, 3, "clamp"), (17, 129, 1, 9, "cyclic"),
                                                       (5, 6, 1, 11, "cyclic"), (40, 67, 2, 64, "full"),
                                                       (33, 66, 1, 2, "full"), (70, 40, 0, 7, "zero")])
def test_wide(S, rows, cols, planes, R, border):
    _check(rows, cols, R, S, border, O.XCORR if S % 4 == 1 else O.CONV, planes=planes)


def test_wide_bank_and_offsets():
    _check(100, 130, 11, 11, "clamp", O.XCORR, planes=0, fplanes=16)
    _check(100, 132, 9, 9, "zero", O.CONV, planes=3, fplanes=3, shift=3)


@pytest.mark.parametrize("border", ["zero", "cyclic"])
@pytest.mark.parametrize("R", [3, 5, 7])
@pytest.mark.parametrize("step", [2, 3])
@pytest.mark.parametrize("planes,rows,cols,shift", [(1, 17, 65, 0), (80, 33, 64, 0), (2, 9, 6, 1), (1, 1, 1, 0),
                                                    (90, 17, 67, 0)])
def test_up(planes, rows, cols, shift, step, R, border):
    _check(rows, cols, R, R, border, O.CONV, planes=planes, sampling=O.UP, step=step, shift=shift)


@pytest.mark.parametrize("rows,cols,R,border,sampling,step", [
    (40, 68, 5, "clamp", O.NOSAMPLE, 1), (40, 67, 7, "zero", O.NOSAMPLE, 1), (33, 61, 15, "cyclic", O.NOSAMPLE, 1),
    (40, 68, 3, "zero", O.DOWN, 2), (20, 33, 5, "cyclic", O.UP, 2), (20, 33, 7, "zero", O.UP, 3)])
def test_not_finite(rows, cols, R, border, sampling, step):
    with np.errstate(invalid="ignore", over="ignore"):
        _check(rows, cols, R, R, border, O.XCORR, planes=2, sampling=sampling, step=step, bad=True)


# several terms per output: the fused filter bank under UpsampleInput, with ReLU
@pytest.mark.parametrize("mode,rows,cols,R,step", [(O.PROJECT_REDUCE, 19, 35, 5, 2), (O.BACKPROJECT_REDUCE, 8, 70, 3, 2),
                                                   (O.PROJECT_REDUCE, 9, 9, 7, 3)])
def test_up_bank(mode, rows, cols, R, step):
    rng = np.random.default_rng(rows)
    B, N, K = 2, 5, 6
    x = rng.standard_normal((B * N, rows, cols)).astype(np.float32)
    f = rng.standard_normal((N * K, R, R)).astype(np.float32)
    orient = O.XCORR if mode == O.PROJECT_REDUCE else O.CONV
    od = O.make_desc(rows, cols, R, R, planes=B * N, f_planes=N * K, batch=B, border=O.ZERO, orient=orient,
                     sampling=O.UP, step=step, mode=mode)
    ref = O.conv(od, x, f)
    assert bitwise_equal(_run(od, x, f), ref)
    assert bitwise_equal(_run(od, x, f, flags=_lib.FLAG_RELU), np.maximum(ref, 0))


# the widths past 31, which take the short tile only
@pytest.mark.parametrize("S", list(range(33, 65, 2)))
@pytest.mark.parametrize("rows,cols,planes,R,border", [(17, 66, 2, 33, "clamp"), (40, 70, 1, 63, "cyclic"),
                                                       (16, 64, 0, 1, "zero")])
def test_widest(S, rows, cols, planes, R, border):
    _check(rows, cols, R, S, border, O.CONV if S % 4 == 1 else O.XCORR, planes=planes)


# the TMA stencils' two tile forms (64 x 128 and 128 x 64), with last tiles of one
# row or 4 columns and more tiles than the persistent grid's two stages hold
@pytest.mark.parametrize("border", ["zero", "valid", "full"])
@pytest.mark.parametrize("R", [1, 3, 5, 7])
@pytest.mark.parametrize("planes,rows,cols", [(400, 129, 64), (1300, 65, 132), (330, 64, 128), (700, 128, 68)])
def test_tma_tiles(planes, rows, cols, R, border):
    _check(rows, cols, R, R, border, O.CONV, planes=planes)


@pytest.mark.parametrize("rl,cl", [(1, 9), (3, 5), (5, 3), (7, 7), (9, 1)])
@pytest.mark.parametrize("planes,rows,cols", [(400, 129, 64), (1300, 65, 132), (5, 30, 20)])
def test_separable_tma_tiles(planes, rows, cols, rl, cl):
    rng = np.random.default_rng(rows + rl)
    x = rng.uniform(-1, 1, (planes, rows, cols)).astype(np.float32)
    rf, cf = rng.uniform(-1, 1, rl).astype(np.float32), rng.uniform(-1, 1, cl).astype(np.float32)
    import cctconv as C
    y = C.crossCorrelateSeparable(torch.from_numpy(x).cuda(), torch.from_numpy(rf).cuda(), torch.from_numpy(cf).cuda(),
                                  C.BorderZero)
    assert bitwise_equal(y.cpu().numpy(), O.separable(x, rf, cf, O.ZERO, O.XCORR))


# the separable tile form: tall and short tiles, every compiled row length, column
# lengths up to its limit and past it, 16- and 4-byte stores, fields smaller than
# the filters
@pytest.mark.parametrize("border", ["zero", "clamp", "cyclic"])
@pytest.mark.parametrize("rl,cl", [(1, 31), (3, 1), (5, 9), (7, 7), (9, 15), (11, 3), (13, 13), (15, 31), (15, 33), (17, 5)])
@pytest.mark.parametrize("planes,rows,cols", [(160, 65, 130), (2, 17, 65), (1, 6, 5), (3, 64, 72)])
def test_separable_tiles(planes, rows, cols, rl, cl, border):
    import cctconv as C
    rng = np.random.default_rng(rows * 40 + rl)
    x = rng.uniform(-1, 1, (planes, rows, cols)).astype(np.float32)
    rf, cf = rng.uniform(-1, 1, rl).astype(np.float32), rng.uniform(-1, 1, cl).astype(np.float32)
    b = {"zero": C.BorderZero, "clamp": C.BorderClamp, "cyclic": C.BorderCyclic}[border]
    y = C.convolveSeparable(torch.from_numpy(x).cuda(), torch.from_numpy(rf).cuda(), torch.from_numpy(cf).cuda(), b)
    assert bitwise_equal(y.cpu().numpy(), O.separable(x, rf, cf, _BORDERS[border], O.CONV))


@pytest.mark.parametrize("border", ["zero", "cyclic"])
@pytest.mark.parametrize("planes,rows,cols,shift", [(1, 17, 65, 0), (3, 33, 64, 0), (2, 9, 6, 1), (1, 3, 1, 0)])
def test_up2_9x9(planes, rows, cols, shift, border):
    _check(rows, cols, 9, 9, border, O.CONV, planes=planes, sampling=O.UP, step=2, shift=shift)


# narrow or flat fields of many planes, which fill less than half of a 64 x 128 or
# 128 x 64 tile
@pytest.mark.parametrize("border", ["zero", "valid", "full"])
@pytest.mark.parametrize("R", [1, 3, 5, 7])
@pytest.mark.parametrize("planes,rows,cols", [(60, 257, 32), (100, 130, 24), (100, 32, 132), (100, 68, 68), (100, 60, 64)])
def test_narrow(planes, rows, cols, R, border):
    _check(rows, cols, R, R, border, O.CONV, planes=planes)
