"""ColorField convolution through the FFT: the bytes of fixed inputs.  They are rounded
from FP32 transforms, so they show any change of the transforms' operations; the digests
are those of the transform of the whole expanded grid."""
import hashlib

import numpy as np
import pytest
import torch

import oracle as O
from cctconv import _lib

pytestmark = pytest.mark.gpu

# by border: a filter given at the run, a static one
DIGESTS = {O.CLAMP: ["48eabbff6228d1e6", "eb7a877e87b7afbc"], O.CYCLIC: ["242d54a1d3ecb9e5", "b38e4a446df85a02"],
           O.ZERO: ["d10b6a7d7d7b668a", "2c02cbd296cbc254"]}


@pytest.mark.parametrize("rows,cols,R,border", [(600, 700, 31, O.CLAMP), (700, 500, 25, O.CYCLIC),
                                                (900, 500, 31, O.ZERO)])
def test_bytes(rows, cols, R, border):
    rng = np.random.default_rng(rows + cols)
    x = rng.integers(0, 256, (rows, cols, 4), dtype=np.uint8)
    f = rng.random((R, R)).astype(np.float32)
    f /= f.sum()
    d = _lib.new_desc(image_rows=rows, image_cols=cols, filter_rows=R, filter_cols=R, border=border,
                      orientation=_lib.CONVOLUTION, algo=_lib.ALGO_FFT)
    plan = _lib.ColorPlan(d)
    xd, fd = torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda()
    got = []
    for static in (False, True):
        if static:
            plan.set_static_filter(f.ctypes.data)
        y = torch.zeros((rows, cols, 4), device="cuda", dtype=torch.uint8)
        plan.run(xd.data_ptr(), 0 if static else fd.data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream)
        got.append(hashlib.sha256(y.cpu().numpy().tobytes()).hexdigest()[:16])
    plan.close()
    assert got == DIGESTS[border]
