"""The adjoint's tile kernels with items of several orientations and CTAs of
several items, from kept responses and recomputing them: what large images run,
here also at the ragged sizes (one-row tiles, warps without rows, window edges
at 16-byte chunks) that otherwise give every CTA one orientation of one tile.

Against the default plan: all sum the same floats, an item's orientations in the
frequency domain and the items' gradients by atomics, in other groups, which
moves a pixel by less than 1e-5 of the largest gradient; the loss and the
parameter gradients are FP64 sums of the same values in another order.  And
against the FP64 gradient, branch-matched, with the bound of the other adjoint
comparisons."""
import numpy as np
import pytest
import torch

from bimp_b200 import api, synth
from test_gpu_adjoint import GRAD_TOL, _run

pytestmark = pytest.mark.gpu


def _step(monkeypatch, w, h, n, lam, keep, grid):
    monkeypatch.setenv("BIMP_ADJOINT_KEEP", keep)
    if grid:
        monkeypatch.setenv("BIMP_ADJOINT_GRID", str(grid))
    else:
        monkeypatch.delenv("BIMP_ADJOINT_GRID", raising=False)
    x = torch.rand((n, h, w), generator=torch.Generator().manual_seed(w * 31 + h)).cuda()
    a = api.Adjoint(w, h, n, lam)
    m = torch.randn(n * a.mask_stride, generator=torch.Generator().manual_seed(h)).cuda()
    for _ in range(2):   # the second step on what the first left behind
        loss = float(a.forward(x, m))
        g, gp = a.backward()
    out = loss, g.cpu().numpy(), gp.cpu().numpy().copy()
    a.close()
    return out


def _same(got, want):
    (l0, g0, p0), (l1, g1, p1) = got, want
    assert abs(l0 - l1) <= 1e-9 * max(1.0, abs(l1))
    assert np.abs(g0 - g1).max() <= 1e-5 * np.abs(g1).max()
    assert np.abs(p0 - p1).max() <= 1e-9 * np.abs(p1).max()


@pytest.mark.parametrize("w,h,n,lam,chunk", [
    (16, 18, 1, [4.0], 0),               # one tile
    (99, 99, 1, [4.0], 0),               # a second tile row with one row
    (113, 60, 1, [4.0], 0),              # window ends one value before the data does
    (229, 70, 1, [4.0, 5.656854], 0),    # ragged chunk at the right edge, both tile sizes
    (64, 64, 2, [4.0, 8.0], 0),          # fftW == dataW, the window wraps the torus
    (131, 103, 1, [4.0, 11.0], 0),       # offsets outside the built-in sets
    (300, 220, 1, [2.0, 7.4], 0),        # the smallest and a large kernel
    (131, 77, 5, [4.0, 22.0], 2),        # chunks of two, the last of one
])
def test_small_grids_equal_the_default_plan(monkeypatch, w, h, n, lam, chunk):
    if chunk:
        monkeypatch.setenv("BIMP_ADJOINT_CHUNK", str(chunk))
    want = _step(monkeypatch, w, h, n, lam, "1", 0)
    for grid in (1, 2, 5):
        for keep in ("1", "0"):
            _same(_step(monkeypatch, w, h, n, lam, keep, grid), want)


@pytest.mark.parametrize("w,h,n,scales", [(512, 512, 2, 6), (1333, 1001, 1, 6)])
def test_recomputed_equals_kept_over_many_items(monkeypatch, w, h, n, scales):
    """196 and 451 tiles: up to four items a CTA on 148 CTAs."""
    lam = synth.bank(scales)
    _same(_step(monkeypatch, w, h, n, lam, "0", 0), _step(monkeypatch, w, h, n, lam, "1", 0))


@pytest.mark.parametrize("keep", ["1", "0"])
@pytest.mark.parametrize("w,h,n,lam,grid", [
    (96, 80, 2, [4.0, 5.656854, 8.0], 3),     # padded torus, two levels
    (128, 128, 1, [4.0, 8.0], 2),             # fftW == dataW at both levels
    (229, 70, 1, [4.0, 5.656854], 2),
])
def test_small_grids_match_the_fp64_gradient(monkeypatch, keep, w, h, n, lam, grid):
    monkeypatch.setenv("BIMP_ADJOINT_KEEP", keep)
    monkeypatch.setenv("BIMP_ADJOINT_GRID", str(grid))
    _, g, gp, ref = _run(w, h, n, lam, seed=17)
    want = np.stack(ref["g"])
    assert np.linalg.norm(g - want) <= GRAD_TOL * np.linalg.norm(want)
    assert np.all(np.abs(gp - ref["p"]) <= GRAD_TOL * np.abs(ref["p"]) + 1e-6), (gp, ref["p"])
