"""The pipelined tile kernel (set_tile_plan(kernel=1), BIMP_TILE_KERNEL=pipelined)
against the phased one: the same maps bit for bit where its window staging
changes (16-byte chunks and columns outside the data, tori smaller than a
window), on byte and float levels, and a detection that takes at most 18%
longer.  It is a plan that a program may choose, and was 25-28% behind while it
read the stored spectra and its window value by value, 10-14% with 16-byte loads;
runs of one plan differ by 1%."""
import numpy as np
import pytest
import torch

from bimp_b200 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,lam", [
    (128 - 15, 60, [4.0]),        # one column short of a window's data
    (229, 101, [4.0]),            # a 9th chunk, a second tile row
    (241, 202, [4.0]),            # chunks past the data inside the row
    (16, 16, [4.0]),              # torus 16: the window wraps it many times
    (256, 256, [4.0]),            # fftW == dataW
    (230, 67, [5.656854, 11.0]),  # V = 90; offsets outside the built-in sets
])
def test_pipelined_maps_equal_phased(monkeypatch, w, h, lam):
    img = synth.synth_image(w, h, 4, seed=3 * w + h)
    b = api.Batch([(w, h)], lam)
    b.load([img])
    maps = []
    for kernel in (0, 1):
        b.set_tile_plan(0, 0, 0, kernel)
        b.run()
        maps.append([b.dense_map(0, s).cpu().numpy() for s in range(len(lam))])
    b.close()
    for s in range(len(lam)):
        assert np.array_equal(maps[0][s], maps[1][s]), s
    x = torch.from_numpy(img.astype(np.float32) / 255.0).cuda().reshape(1, h, w)
    maps = []
    for kernel in ("phased", "pipelined"):
        monkeypatch.setenv("BIMP_TILE_KERNEL", kernel)
        a = api.Adjoint(w, h, 1, lam)
        a.forward(x, torch.ones(a.mask_stride, device="cuda"))
        maps.append([a.dense_map(0, s).cpu().numpy() for s in range(len(lam))])
        a.close()
    for s in range(len(lam)):
        assert np.array_equal(maps[0][s], maps[1][s]), s


@pytest.mark.parametrize("sizes,scales,plan,bound", [
    ([(1280, 720), (1920, 1080), (640, 480), (1600, 900)], 8, (0, 0, 0), 1.18),
    # the split plan, with cost weights of this kernel's own: 1.05 (1.12 with the phased kernel's)
    ([(58, 444), (680, 636), (45, 839), (55, 119)], 6, (0, 1, 296), 1.09),
])
def test_pipelined_kernel_keeps_its_speed(sizes, scales, plan, bound):
    rng = np.random.default_rng(3)
    b = api.Batch(sizes, synth.bank(scales), kp_capacity=1 << 18)
    b.load([rng.integers(0, 256, (h, w), dtype=np.uint8) for w, h in sizes])
    ms = {0: [], 1: []}
    for _ in range(7):
        for kernel in (0, 1):
            b.set_tile_plan(*plan, kernel)
            b.run()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            for _ in range(4):
                b.run()
            e1.record()
            e1.synchronize()
            ms[kernel].append(e0.elapsed_time(e1))
    b.close()
    phased, pipelined = np.median(ms[0]), np.median(ms[1])
    print("phased", phased / 4, "pipelined", pipelined / 4, "ms, ratio", pipelined / phased)
    assert pipelined <= bound * phased
