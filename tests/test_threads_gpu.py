"""Host threads that launch one kernel with different amounts of shared memory at the
same time, a stream each: every call succeeds and gives the bits it gives alone."""
import threading

import pytest
import torch

from cctconv import _lib

pytestmark = pytest.mark.gpu
LIB = _lib.LIB
CALLS = 6000


def _plan(x, f, y, **desc):
    plan = _lib.Plan(_lib.new_desc(**desc))
    handle, xp, fp, yp = plan.handle, x.data_ptr(), f.data_ptr(), y.data_ptr()
    return (lambda st: LIB.cct_conv_run(handle, xp, fp, yp, st)), y, (x, f, plan)


def _weight_gradient(n):  # 3x3 results: a ring of image rows n wide
    x, g = torch.randn((16, n + 2, n + 2), device="cuda"), torch.randn((16, n, n), device="cuda")
    return _plan(x, g, torch.empty((256, 3, 3), device="cuda"), image_rows=n + 2, image_cols=n + 2, image_planes=16,
                 filter_rows=n, filter_cols=n, filter_planes=16, border=_lib.BORDER_VALID, vector_mode=_lib.FILTER_ADJOINT)


def _wide(rows):  # rows x 63 filters: the tile and the filter in shared memory
    x, f = torch.randn((2, 40, 70), device="cuda"), torch.randn((rows, 63), device="cuda")
    return _plan(x, f, torch.empty_like(x), image_rows=40, image_cols=70, image_planes=2, filter_rows=rows,
                 filter_cols=63, algo=_lib.ALGO_DIRECT)


def _generic(rows):  # down-sampled, even widths: the general stencil
    x, f = torch.randn((2, 120, 240), device="cuda"), torch.randn((rows, 10), device="cuda")
    orows = (120 + rows - 1 + 2) // 3
    return _plan(x, f, torch.empty((2, orows, 83), device="cuda"), image_rows=120, image_cols=240, image_planes=2,
                 filter_rows=rows, filter_cols=10, border=_lib.BORDER_FULL, sampling=_lib.SAMPLE_DOWN, step=3)


def _separable(taps):
    x, y, tmp = (torch.randn((160, 65, 65), device="cuda") for _ in range(3))
    rf, cf = torch.randn(15, device="cuda"), torch.randn(taps, device="cuda")
    ptrs = (x.data_ptr(), rf.data_ptr(), 15, cf.data_ptr(), taps, _lib.BORDER_CLAMP, _lib.CONVOLUTION, tmp.data_ptr(),
            y.data_ptr())
    return (lambda st: LIB.cct_conv_separable(65, 65, 160, *ptrs, st)), y, (x, rf, cf, tmp)


@pytest.mark.parametrize("make,sizes", [(_weight_gradient, (64, 32)), (_wide, (63, 55)), (_generic, (31, 61)),
                                        (_separable, (19, 31))])
def test_shared_memory_sizes(make, sizes):
    jobs = [make(n) for n in sizes * 2]
    alone, errors = [], []
    for call, y, _ in jobs:
        assert call(torch.cuda.current_stream().cuda_stream) == _lib.OK, LIB.cct_last_error_string()
        alone.append(y.clone())
    torch.cuda.synchronize()
    for _, y, _ in jobs:
        y.fill_(float("nan"))
    torch.cuda.synchronize()
    start = threading.Barrier(len(jobs))

    def run(call, stream):
        start.wait()
        for _ in range(CALLS):
            if call(stream.cuda_stream):
                errors.append(LIB.cct_last_error_string())
                return

    streams = [torch.cuda.Stream() for _ in jobs]
    threads = [threading.Thread(target=run, args=(job[0], st)) for job, st in zip(jobs, streams)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors
    for (_, y, _), want in zip(jobs, alone):
        assert torch.equal(y, want)
