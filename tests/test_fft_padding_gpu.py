"""FFT path: the spectrum of a filter that changes from run to run is made by the
same operations whether its rows fill the grid or only its ends, so rows of zeros
around a filter change no bit of the field."""
import numpy as np
import pytest
import torch

from cctconv import _lib

pytestmark = pytest.mark.gpu


def _run(rows, cols, border, x, f):
    plan = _lib.Plan(_lib.new_desc(image_rows=rows, image_cols=cols, filter_rows=f.shape[0], filter_cols=f.shape[1],
                                   border=border, orientation=_lib.CONVOLUTION, algo=_lib.ALGO_FFT))
    assert plan.algo == _lib.PLAN_FFT
    y = torch.full((rows, cols), float("nan"), device="cuda")
    plan.run(x.data_ptr(), f.data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    plan.close()
    return y.cpu().numpy()


# R rows fit the first and last sixteenth of the grid's Fr rows ((R - 1) / 2 < Fr / 16);
# padded rows do not
@pytest.mark.parametrize("rows,cols,R,padded,border", [
    (28, 60, 3, 5, _lib.BORDER_ZERO), (50, 60, 7, 9, _lib.BORDER_ZERO), (100, 130, 15, 17, _lib.BORDER_ZERO),
    (256, 256, 31, 33, _lib.BORDER_CYCLIC), (470, 300, 63, 65, _lib.BORDER_ZERO), (1024, 64, 127, 129, _lib.BORDER_CYCLIC),
    (2048, 64, 63, 257, _lib.BORDER_CYCLIC)])
def test_zero_rows_change_no_bit(rows, cols, R, padded, border):
    rng = np.random.default_rng(rows)
    x = torch.from_numpy(rng.uniform(-1, 1, (rows, cols)).astype(np.float32)).cuda()
    f = torch.from_numpy(rng.uniform(-1, 1, (R, 7)).astype(np.float32)).cuda()
    e = (padded - R) // 2
    wide = torch.nn.functional.pad(f, (0, 0, e, e))
    assert np.array_equal(_run(rows, cols, border, x, f), _run(rows, cols, border, x, wide))
