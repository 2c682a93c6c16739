"""Batch.keypoints(): an expired device wait of the run reaches the caller (it is
marked by the host: no device wait runs out here)."""
import numpy as np
import pytest

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
