"""The caller's limit on the memory that the adjoint's forward keeps its responses
in: nothing below what they take, all from there on, the same gradients."""
import numpy as np
import pytest
import torch

from bimp_b200 import api

pytestmark = pytest.mark.gpu


def test_keep_bytes_limits_what_is_kept(monkeypatch):
    w, h, n, lam = 131, 77, 2, [4.0, 5.656854]
    x = torch.rand((n, h, w), generator=torch.Generator().manual_seed(3)).cuda()

    def step(**kw):
        a = api.Adjoint(w, h, n, lam, **kw)
        m = torch.randn(n * a.mask_stride, generator=torch.Generator().manual_seed(4)).cuda()
        loss = float(a.forward(x, m))
        g, gp = a.backward()
        out = a.kept_bytes(), a.device_bytes(), loss, g.cpu().numpy(), gp.cpu().numpy().copy()
        a.close()
        return out

    kept, held, loss, g, gp = step()
    assert kept > 0
    monkeypatch.setenv("BIMP_ADJOINT_KEEP", "0")   # decides only where the caller does not
    assert step()[0] == 0
    for limit, want in ((0, 0), (kept - 1, 0), (kept, kept), (1 << 40, kept)):
        k, b, l2, g2, gp2 = step(keep_bytes=limit)
        assert (k, b) == (want, held - kept + want)
        assert abs(l2 - loss) <= 1e-9 * max(1.0, abs(loss))
        assert np.abs(g2 - g).max() <= 1e-5 * np.abs(g).max()
        assert np.abs(gp2 - gp).max() <= 1e-9 * np.abs(gp).max()
