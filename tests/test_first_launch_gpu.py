"""Kernels with static and dynamic shared memory, launched first with sizes around what
a kernel may use without asking (48 KB in all): each size in a process of its own, since
a limit once raised stays."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import sys, numpy as np, torch
sys.path[:0] = {paths!r}
import oracle as O
from cctconv import _lib
rows, cols, B, C, K, R, sampling, step, prec = {case!r}
rng = np.random.default_rng(rows)
x = rng.standard_normal((B * C, rows, cols)).astype(np.float32)
f = rng.standard_normal((K * C, R, R)).astype(np.float32)
ref = O.conv(O.make_desc(rows, cols, R, R, planes=B * C, f_planes=K * C, batch=B, border=O.VALID, orient=O.XCORR,
                         sampling=sampling, step=step, mode=O.PROJECT_REDUCE), x, f, np.float64)
plan = _lib.Plan(_lib.new_desc(image_rows=rows, image_cols=cols, image_planes=B * C, filter_rows=R, filter_cols=R,
                               filter_planes=K * C, batch_size=B, border=_lib.BORDER_VALID,
                               orientation=_lib.CROSS_CORRELATION, sampling=sampling, step=step,
                               vector_mode=_lib.PROJECT_FRAME_BLOCK_REDUCE_SUM, precision=prec))
y = torch.full(ref.shape, float("nan"), device="cuda")
xd, fd = torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda()
plan.run(xd.data_ptr(), fd.data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream)
assert np.abs(y.cpu().numpy() - ref).max() <= 1e-5 * np.abs(ref).max()
"""


@pytest.mark.parametrize("case", [(74, 5, 2, 1, 1, 1, 2, 2, 1), (20, 9, 1, 7, 9, 1, 0, 1, 1), (20, 9, 1, 7, 9, 1, 0, 1, 2),
                                  (30, 40, 2, 3, 5, 1, 0, 1, 1), (12, 17, 1, 8, 5, 3, 0, 1, 1)])
def test_first_launch(case):
    root = Path(__file__).resolve().parent.parent
    paths = [str(root / "cct-core_b200"), str(root / "oracle")]
    done = subprocess.run([sys.executable, "-c", PROGRAM.format(paths=paths, case=case)], capture_output=True, text=True,
                          timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
