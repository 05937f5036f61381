"""Filter-bank plans of layers whose tiles take their epilogue longer than their few
matrix instructions: small tiles on more SMs, and 64 filters a block."""
import pytest

import oracle as O
from cctconv import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,shape,form,tile", [
    (_lib.PREC_BF16X6, (1, 7, 9, 20, 9, 1, O.ZERO, O.NOSAMPLE, 1, O.PROJECT_REDUCE), _lib.BANK_PLAIN, 64),
    (_lib.PREC_BF16X3, (2, 6, 26, 20, 37, 2, O.VALID, O.NOSAMPLE, 1, O.BACKPROJECT_REDUCE), _lib.BANK_PAIR, 64),
    (_lib.PREC_BF16X3, (1, 8, 5, 12, 17, 3, O.ZERO, O.UP, 2, O.PROJECT_REDUCE), _lib.BANK_PAIR, 64),
    (_lib.PREC_BF16X6, (2, 18, 145, 104, 36, 5, O.FULL, O.UP, 4, O.BACKPROJECT_REDUCE), _lib.BANK_PLAIN, 224),
    # the multiply-adds of these take longer: the long stages and wide blocks stay
    (_lib.PREC_BF16X3, (8, 64, 64, 224, 224, 3, O.ZERO, O.DOWN, 2, O.PROJECT_REDUCE), _lib.BANK_PLAIN, 256),
    (_lib.PREC_BF16X6, (8, 256, 512, 28, 28, 3, O.ZERO, O.NOSAMPLE, 1, O.PROJECT_REDUCE), _lib.BANK_WIDE, 96)])
def test_tiles(prec, shape, form, tile):
    batch, c, k, rows, cols, R, border, sampling, step, mode = shape
    plan = _lib.Plan(_lib.new_desc(image_rows=rows, image_cols=cols, image_planes=batch * c, filter_rows=R,
                                   filter_cols=R, filter_planes=k * c, batch_size=batch, border=border,
                                   orientation=O.XCORR if mode == O.PROJECT_REDUCE else O.CONV, sampling=sampling,
                                   step=step, vector_mode=mode, precision=prec))
    got = plan.bank()
    plan.close()
    assert (got[0], got[2]) == (form, tile)
