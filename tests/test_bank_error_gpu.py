"""Three-term filter banks: the error does not grow with the reduction.

Sums are promoted into an FP32 running sum at least every 64 k-steps of 16 planes, so
the RMS error of a long reduction is that of one of 64 k-steps, times
sqrt(1 + 0.003 + 0.02) for the small sums, promoted every 1280 MMAs, and the roundings of
up to 200 promotions; 1.05 leaves 4 % for the sample of 3136 outputs."""
import numpy as np
import pytest
import torch

import oracle as O
from cctconv import _lib

pytestmark = pytest.mark.gpu


def _rms_error(B, N, K, size, R, form, checked=4):
    gen = torch.Generator(device="cuda").manual_seed(N + R)
    x = torch.randn((B * N, size, size), device="cuda", generator=gen)
    f = torch.randn((K * N, R, R), device="cuda", generator=gen) * (2.0 / (N * R * R)) ** 0.5
    plan = _lib.Plan(_lib.new_desc(image_rows=size, image_cols=size, image_planes=B * N, filter_rows=R, filter_cols=R,
                                   filter_planes=K * N, batch_size=B, orientation=_lib.CROSS_CORRELATION,
                                   vector_mode=_lib.PROJECT_FRAME_BLOCK_REDUCE_SUM, precision=_lib.PREC_BF16X6))
    assert plan.bank()[0] == form
    y = torch.full((B * K, size, size), float("nan"), device="cuda")
    plan.run(x.data_ptr(), f.data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream)
    y = y[:checked].cpu().numpy()
    plan.close()
    od = O.make_desc(size, size, R, R, planes=N, f_planes=checked * N, batch=1, border=O.ZERO, orient=O.XCORR,
                     mode=O.PROJECT_REDUCE)
    ref = O.conv(od, x[:N].cpu().numpy(), f[:checked * N].cpu().numpy(), np.float64)
    return np.sqrt(np.mean((y - ref) ** 2) / np.mean(ref ** 2))


# 128 filters a block; 64 filters x two taps; the plain form; segments that the stages
# do not divide (144 k-steps)
@pytest.mark.parametrize("B,N,K,size,R,form", [
    (8, 8192, 512, 14, 3, _lib.BANK_WIDE), (8, 8192, 64, 28, 5, _lib.BANK_WIDE_PAIR),
    (1, 2048, 40, 28, 1, _lib.BANK_PLAIN), (8, 256, 192, 52, 3, _lib.BANK_PLAIN)])
def test_long_reductions(B, N, K, size, R, form):
    assert _rms_error(B, N, K, size, R, form) <= 1.05 * _rms_error(8, 1024, 64, 28, 1, _lib.BANK_PLAIN)
