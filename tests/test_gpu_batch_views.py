"""Batch.keypoints() and input_tensor(): an expired device wait of the run reaches
the caller (it is marked by the host: no device wait runs out here), and the
views that calls return share the library's memory but nothing of torch's state."""
import numpy as np
import pytest
import torch

from bimp_b200 import _lib as L
from bimp_b200 import api, synth

pytestmark = pytest.mark.gpu


def _batch(sizes, lam=(4.0, 8.0), kp_capacity=8192):
    b = api.Batch(sizes, list(lam), kp_capacity=kp_capacity)
    b.load([synth.synth_image(w, h, 4, seed=w + h) for w, h in sizes])
    return b


def test_keypoints_report_an_expired_wait():
    sizes = [(160, 120), (99, 131), (64, 64)]
    b = _batch(sizes)
    b.run()
    want = [b.keypoints(i).cpu().numpy().copy() for i in range(len(sizes))]
    assert [k.shape[1] for k in want] == b.counts().tolist()
    assert L.lib().bimp_batch_inject_fault(b._h, api._stream_ptr()) == L.BIMP_OK
    for i in range(len(sizes)):
        with pytest.raises(L.BimpError, match="wait expired"):
            b.keypoints(i)
    b.run()   # the next run starts without it
    for i in range(len(sizes)):
        assert np.array_equal(b.keypoints(i).cpu().numpy().view(np.int32), want[i].view(np.int32)), i
    b.close()


def test_batch_made_in_inference_mode_works_outside():
    sizes = [(96, 80)]
    with torch.inference_mode():
        b = _batch(sizes)
    b.load([synth.synth_image(96, 80, 4, seed=5)])   # writes into the input's alias
    b.run()
    kp = b.keypoints(0)
    assert not kp.is_inference() and not b.input_tensor(0).is_inference()
    w = torch.ones((), device="cuda", requires_grad=True)
    (w * kp).sum().backward()                        # saves the view for its backward
    assert torch.isfinite(w.grad)
    with torch.inference_mode():
        b.load([synth.synth_image(96, 80, 4, seed=6)])
        b.run()
        assert b.keypoints(0).shape[1] == int(b.counts()[0])
    b.close()


def test_views_of_two_calls_share_memory_but_no_autograd_state():
    b = _batch([(96, 80)])
    b.run()
    first = b.keypoints(0)
    w = torch.full((), 2.0, device="cuda", requires_grad=True)
    out = (w * first).sum()            # saves `first`
    b.keypoints(0).mul_(w)             # an in-place operation with a gradient on another view
    second = b.keypoints(0)
    assert second.data_ptr() == first.data_ptr()
    assert not second.requires_grad and second.grad_fn is None
    out.backward()                     # the other view's change of the memory is not this one's version
    x = b.input_tensor(0)
    assert x.data_ptr() == b.input_tensor(0).data_ptr()
    emb = (w * x).sum()
    b.load([synth.synth_image(96, 80, 4, seed=7)])
    emb.backward()
    b.close()
