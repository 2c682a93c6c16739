"""An expired device wait of the adjoint reaches the caller: the status query
fails once, also through further calls, and torch.autograd raises; the calls
after it work.  The expiry is marked by the host (bimp_adjoint_inject_fault): no
device wait runs out here."""
import pytest
import torch

from bimp_b200 import _lib as L
from bimp_b200 import api
from bimp_b200.autograd import summed_map_loss, summed_map_theta

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("keep", ["1", "0"])
def test_expired_wait_is_reported_once(monkeypatch, keep):
    monkeypatch.setenv("BIMP_ADJOINT_KEEP", keep)
    x = torch.rand((2, 80, 96), generator=torch.Generator().manual_seed(1)).cuda()
    a = api.Adjoint(96, 80, 2, [4.0, 8.0])
    m = torch.ones(2 * a.mask_stride, device="cuda")
    want = float(a.forward(x, m))
    a.backward()
    a.check()
    stream = api._stream_ptr()
    for calls in ((), (lambda: a.forward(x, m),), (lambda: a.forward(x, m), a.backward)):
        assert L.lib().bimp_adjoint_inject_fault(a._h, stream) == L.BIMP_OK
        for c in calls:
            c()
        with pytest.raises(L.BimpError, match="wait expired"):
            a.check()
        a.check()
    loss = summed_map_loss(x.clone().requires_grad_(True), summed_map_theta(a), m, a)
    assert L.lib().bimp_adjoint_inject_fault(a._h, stream) == L.BIMP_OK
    with pytest.raises(L.BimpError, match="wait expired"):
        loss.backward()
    assert float(a.forward(x, m)) == pytest.approx(want, rel=1e-12)
    a.check()
    a.close()
