"""What an operator refuses it refuses whatever was called before: an option equal to a
good one but of another type is no good one."""
import numpy as np
import pytest
import torch

import cctconv as C
from cctconv import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [{"batchSize": 2 + 0j}, {"precision": _lib.PREC_BF16X3 + 0j}, {"batchSize": 2.0},
                                 {"batchSize": np.complex64(2)}, {"batchSize": None}, {"precision": "bf16"}])
def test_frame_options(bad):
    x, f = torch.randn((4, 12, 14), device="cuda"), torch.randn((6, 3, 3), device="cuda")
    good = {"batchSize": 2, "precision": _lib.PREC_BF16X3}

    def outcome(**options):
        try:
            return C.projectFrameBlockReduceSum(x, f, C.BorderZero, **options)
        except Exception as e:
            return type(e)

    before = outcome(**(good | bad))
    y = outcome(**good)
    after = outcome(**(good | bad))
    assert torch.is_tensor(y)
    assert torch.equal(before, after) if torch.is_tensor(before) else before is after
