"""Repeated operator calls: every argument that decides a result is part of
what a remembered call is looked up by."""
import itertools

import numpy as np
import pytest
import torch

import cctconv as C
import oracle as O
from cctconv import _lib
from helpers import bitwise_equal

pytestmark = pytest.mark.gpu

_BORDERS = {C.BorderZero: O.ZERO, C.BorderClamp: O.CLAMP, C.BorderValid: O.VALID}


def _plain(op, x, f, border):
    orient = O.CONV if op is C.convolve else O.XCORR
    xn, fn = x.cpu().numpy(), f.cpu().numpy()
    planes = xn.shape[0] if xn.ndim == 3 else 0
    od = O.make_desc(xn.shape[-2], xn.shape[-1], *fn.shape, planes=planes, border=_BORDERS[border], orient=orient)
    y = O.conv(od, xn, fn)
    return y if planes else y[0]


def test_interleaved_calls():
    gen = torch.Generator(device="cuda").manual_seed(3)
    fields = [torch.rand(s, device="cuda", generator=gen) for s in ((33, 40), (40, 33), (1, 33, 40), (3, 33, 40))]
    fields.append(torch.rand((40, 33), device="cuda", generator=gen).t())  # not contiguous
    filters = [torch.rand(s, device="cuda", generator=gen) for s in ((3, 3), (5, 5))]
    for _ in range(2):
        for x, f, border, op in itertools.product(fields, filters, _BORDERS, (C.convolve, C.crossCorrelate)):
            y = op(x, f, border)
            ref = _plain(op, x, f, border)
            assert tuple(y.shape) == ref.shape and bitwise_equal(y.cpu().numpy(), ref)


def test_options_are_not_mixed():
    gen = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn((4, 16, 16), device="cuda", generator=gen)
    f = torch.randn((8, 3, 3), device="cuda", generator=gen)
    for _ in range(2):
        y = C.projectFrameBlockReduceSum(x, f, C.BorderZero, batchSize=2)
        z = C.projectFrameBlockReduceSum(x, f, C.BorderZero, batchSize=2, relu=True)
        t = C.projectFrameBlockReduceSum(x, f, C.BorderZero, batchSize=2, precision=_lib.PREC_BF16X3)
        b = C.backProjectFrameBlockReduceSum(x, f, C.BorderZero, batchSize=2)
        one = C.projectFrameBlockReduceSum(x, f, C.BorderZero, batchSize=1)
        assert torch.equal(z, y.clamp_min(0)) and not torch.equal(t, y) and torch.allclose(t, y, atol=1e-4)
        assert y.shape == (8, 16, 16) and one.shape == (2, 16, 16) and b.shape == y.shape and not torch.equal(b, y)


def test_refusals_after_a_good_call():
    x, f = torch.rand((20, 20), device="cuda"), torch.rand((3, 3), device="cuda")
    C.convolve(x, f, C.BorderZero)
    for bad in (x.double(), x.cpu(), x.reshape(2, 2, 10, 10), x.cpu().numpy()):
        with pytest.raises((TypeError, ValueError, AttributeError)):
            C.convolve(bad, f, C.BorderZero)
    with pytest.raises(ValueError):
        C.convolve(x, f[:2, :2], C.BorderZero)


def test_closed_plan_is_refused():
    x, f = torch.rand((21, 23), device="cuda"), torch.rand((3, 3), device="cuda")
    C.convolve(x, f, C.BorderZero)
    plan = C.plan_for(C.make_desc((21, 23, 0), (3, 3, 0), C.BorderZero, _lib.CONVOLUTION, C.NoSamplingConvolution,
                                  _lib.PLANE_BY_PLANE))
    handle, plan.handle = plan.handle, None
    try:
        with pytest.raises(C.CctError):
            C.convolve(x, f, C.BorderZero)
    finally:
        plan.handle = handle


@pytest.mark.parametrize("border", [C.BorderClamp, C.BorderZero])
def test_color_calls(border):
    rng = np.random.default_rng(5)
    for rows, cols, R in ((20, 24, 3), (24, 20, 5), (20, 24, 3)):
        x = rng.integers(0, 256, (rows, cols, 4), dtype=np.uint8)
        f = rng.uniform(0, 0.2, (R, R)).astype(np.float32)
        od = O.make_desc(rows, cols, R, R, border=_BORDERS[border])
        got = C.convolve(torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda(), border)
        assert np.array_equal(got.cpu().numpy(), O.color_conv(od, x, f))


# tall and short tiles, a last tile of one row or column, 16- and 4-byte stores,
# fields smaller than the filter
@pytest.mark.parametrize("border", [O.ZERO, O.CLAMP, O.CYCLIC, O.VALID, O.FULL])
@pytest.mark.parametrize("R", [1, 3, 5, 7])
@pytest.mark.parametrize("rows,cols", [(33, 65), (8, 64), (9, 7), (330, 961), (321, 960)])
def test_color_stencil(rows, cols, R, border):
    rng = np.random.default_rng(rows * cols + R)
    x = rng.integers(0, 256, (rows, cols, 4), dtype=np.uint8)
    f = rng.uniform(-0.1, 1.0 / R, (R, R)).astype(np.float32)
    od = O.make_desc(rows, cols, R, R, border=border, orient=O.XCORR)
    d = _lib.new_desc(image_rows=rows, image_cols=cols, filter_rows=R, filter_cols=R, border=border,
                      orientation=_lib.CROSS_CORRELATION, algo=_lib.ALGO_DIRECT)
    plan = _lib.ColorPlan(d)
    xd, fd = torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda()
    for static in (False, True):
        if static:
            plan.set_static_filter(f.ctypes.data)
        y = torch.zeros((plan.shape[0], plan.shape[1], 4), device="cuda", dtype=torch.uint8)
        plan.run(xd.data_ptr(), 0 if static else fd.data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert np.array_equal(y.cpu().numpy(), O.color_conv(od, x, f))
    plan.close()
