"""The adjoint's backward from the forward's kept responses against the one that
recomputes them (what an adjoint does whose responses find no memory), over the
sizes where the kept layout changes: one tile, a last tile row or column of one
line, rows that end inside a block of four, tiles cut between CTAs, tori as wide
as the data, several chunks.

Both sum the same floats, the gradient's atomics in any order: a pixel's sum of
at most a few hundred terms moves by less than 1e-5 of the largest gradient;
the parameter gradients are FP64 sums of the same values in another order."""
import numpy as np
import pytest
import torch

from bimp_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,n,lam,chunk", [
    (16, 18, 1, [4.0], 0),                      # one tile, 20 rows
    (99, 99, 2, [4.0], 0),                      # a second tile row with one row (V = 100)
    (100, 131, 1, [4.0, 11.0], 0),              # a second tile column with one column
    (230, 67, 3, [5.656854, 4.0], 0),           # V = 90: blocks of two rows at a tile's end
    (300, 220, 1, [2.0, 7.4], 0),               # the smallest and a large kernel
    (256, 256, 1, [4.0, 8.0], 0),               # fftW == dataW
    (131, 77, 5, [4.0, 22.0], 2),               # chunks of two, the last of one
])
def test_kept_equals_recomputed(monkeypatch, w, h, n, lam, chunk):
    if chunk:
        monkeypatch.setenv("BIMP_ADJOINT_CHUNK", str(chunk))
    g = torch.Generator().manual_seed(w * 31 + h)
    x = torch.rand((n, h, w), generator=g).cuda()
    out, bytes_ = [], []
    for keep in ("1", "0"):
        monkeypatch.setenv("BIMP_ADJOINT_KEEP", keep)
        a = api.Adjoint(w, h, n, lam)
        m = torch.randn(n * a.mask_stride, generator=torch.Generator().manual_seed(h)).cuda()
        loss = float(a.forward(x, m))
        for _ in range(2):   # a second backward of the same forward
            grad, gp = a.backward()
        out.append((loss, grad.cpu().numpy().copy(), gp.cpu().numpy().copy()))
        bytes_.append(a.device_bytes())
        a.close()
    assert bytes_[0] > bytes_[1]
    (l0, g0, p0), (l1, g1, p1) = out
    assert abs(l0 - l1) <= 1e-9 * max(1.0, abs(l1))
    assert np.abs(g0 - g1).max() <= 1e-5 * np.abs(g1).max()
    assert np.abs(p0 - p1).max() <= 1e-9 * np.abs(p1).max()
