"""The adjoint on images whose coarse levels have only a few rows or columns, where
a pixel of a pyramid step's window can reflect onto a level twice: the transposed
step gathers those taps one by one.  Against the FP64 gradient, branch-matched,
with the bound of the other adjoint comparisons; and the backward of a long thin
image takes no longer than that of a taller one."""
import numpy as np
import pytest
import torch

from bimp_b200 import api
from test_gpu_adjoint import GRAD_TOL, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,lam", [
    (96, 16, [32.0]),             # rows 16, 8, 4, 2
    (16, 300, [32.0]),            # the same in columns
    (128, 20, [16.0, 32.0]),      # rows 20, 10, 5, 3: both reflections on one pixel
    (130, 24, [32.0]),            # rows 24, 12, 6, 3
    (36, 300, [32.0]),            # columns 36, 18, 9, 5
    (200, 17, [4.0, 16.0, 32.0]),  # rows 17, 9, 5, 3
    (24, 200, [4.0, 32.0]),       # columns 24, 12, 6, 3
    (23, 97, [16.0, 32.0]),       # columns 23, 12, 6, 3
])
def test_gradient_through_small_levels(w, h, lam):
    imgs = np.random.default_rng(w * 1009 + h).random((2, h, w)).astype(np.float32)
    _, g, gp, ref = _run(w, h, 2, lam, seed=19, imgs=imgs)
    want = np.stack(ref["g"])
    assert np.linalg.norm(want) > 0
    assert np.linalg.norm(g - want) <= GRAD_TOL * np.linalg.norm(want)
    assert np.all(np.abs(gp - ref["p"]) <= GRAD_TOL * np.abs(ref["p"]) + 1e-6), (gp, ref["p"])


def test_backward_of_a_thin_image_takes_no_longer_than_of_a_taller_one():
    """4096 x 16 (rows 16, 8, 4, 2) against 4096 x 64: a quarter of the work, at
    most one and a half times the time (where every pixel of a small level looked
    at the whole coarser level: forty times)."""
    us = []
    for h in (16, 64):
        a = api.Adjoint(4096, h, 1, [32.0])
        x = torch.rand((1, h, 4096), generator=torch.Generator().manual_seed(1)).cuda()
        a.forward(x, torch.ones(a.mask_stride, device="cuda"))
        t = []
        for _ in range(9):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            a.backward()
            e1.record()
            e1.synchronize()
            t.append(1e3 * e0.elapsed_time(e1))
        us.append(float(np.median(t)))
        a.close()
    print("backward us", us)
    assert us[0] <= 1.5 * us[1]
