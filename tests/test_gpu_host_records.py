"""Host records belong to the caller: an array of exactly what was found, apart
from the library's staging and from the next call's, at counts of none, some and
more than the capacity, and for frames in flight."""
import ctypes as C

import numpy as np
import pytest

from bimp_b200 import _lib as L
from bimp_b200 import api, synth

pytestmark = pytest.mark.gpu
LAM = [4.0, 8.0]


def _owned(rec, n):
    assert len(rec) == n and rec.nbytes == 28 * n
    assert rec.flags.owndata and rec.base is None and rec.flags.writeable


def test_detect_host_returns_owned_arrays():
    cs = api.CudaStuff(333, 277, LAM)
    imgs = [synth.synth_image(333, 277, 6, seed=s) for s in (1, 2)]
    first, n, rc = api.detect_host(cs, imgs[0], capacity=100000)
    assert rc == L.BIMP_OK and n > 256
    _owned(first, n)
    kept = first.copy()
    second, n2, _ = api.detect_host(cs, imgs[1], capacity=100000)
    _owned(second, n2)
    assert np.array_equal(first, kept) and not np.array_equal(first[:64], second[:64])
    few, n3, rc = api.detect_host(cs, imgs[0], capacity=37)
    assert rc == L.BIMP_ERR_CAPACITY and n3 == n
    _owned(few, 37)
    assert np.array_equal(few, kept[:37])
    none, n4, _ = api.detect_host(cs, np.full((277, 333), 128, np.uint8), capacity=100000)
    _owned(none, n4)
    empty, n5, rc = api.detect_host(cs, imgs[0], capacity=0)
    assert rc == L.BIMP_ERR_CAPACITY and n5 == n
    _owned(empty, 0)
    # the C entry point that fills the caller's array gives the same
    out = (L.KeyPointC * 100000)()
    m = C.c_int(0)
    assert L.lib().bimp_detect_host(cs.handle, C.c_void_p(imgs[0].ctypes.data), 333, 333, 277, out, 100000,
                                    C.byref(m), api._stream_ptr()) == L.BIMP_OK
    assert m.value == n and bytes(out)[:28 * n] == kept.tobytes()
    with pytest.raises(L.BimpError):
        api.detect_host(cs, imgs[0], capacity=-1)
    cs.close()


def test_pipeline_returns_owned_arrays():
    frames = [synth.synth_image(200, 150, 5, seed=s) for s in range(5)]
    cs = api.CudaStuff(200, 150, LAM)
    want = [api.detect_host(cs, f, capacity=20000)[0] for f in frames]
    cs.close()
    p = api.Pipeline(200, 150, LAM, depth=2, capacity=20000)
    got = []
    for f in frames:
        if p.in_flight() == 2:
            got.append(p.pop()[0])
        p.push(f)
    got.append(p.pop()[0])
    few, n, rc = p.pop(capacity=5)
    p.close()
    for g, w in zip(got, want):
        _owned(g, len(w))
        assert np.array_equal(g, w)
    _owned(few, 5)
    assert rc == L.BIMP_ERR_CAPACITY and n == len(want[4]) and np.array_equal(few, want[4][:5])
