"""The tile kernel's window staging, row blocks and plans at the sizes where
they change: windows inside and outside the data (16-byte chunks and a ragged
lead, a 9th chunk, columns past either edge, tori smaller than a window), tiles
with one row to a full block of rows, the smallest and largest kernel half
sizes, and items cut at any orientation.

Complex cells against the FP64 oracle, within the peak-relative bound of the
other map comparisons (float transforms of 128 x 128 tiles are within about
1e-6 of the peak); plans bit for bit against each other."""
import numpy as np
import pytest

from bimp_b200 import api, synth
from oracle import bimp_oracle as O
from parity import MAP_TOL, peak_rel_error

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,lam", [
    (128 - 15, 60, [4.0]),        # one column short of a window's data, one tile row
    (99, 99, [4.0]),              # 100 columns, 101 rows of cells: a second tile row with one row
    (228, 130, [4.0]),            # window origin 86, data to its last column: aligned end, no 9th chunk
    (229, 101, [4.0]),            # the same with a 9th chunk
    (241, 202, [4.0]),            # pitch 256: chunks past the data inside the row
    (16, 16, [4.0]),              # torus 16: the window wraps it many times
    (300, 220, [2.0]),            # kX = 7: V = 114, 29 row blocks
    (300, 220, [7.4]),            # kX = 26: V = 76, 19 row blocks
    (256, 256, [4.0]),            # fftW == dataW, fftH == dataH
    (230, 67, [5.656854]),        # V = 90, tile rows of 90 (23 blocks) inside a 69-row map
])
def test_complex_cells_at_window_edges(w, h, lam):
    img = synth.synth_image(w, h, 4, seed=3 * w + h)
    res = O.run(img, lam)
    cs = api.CudaStuff(w, h, lam)
    api.getKeypoints(img, cs, capacity=50000)
    for i, r in enumerate(res):
        for o in range(8):
            assert peak_rel_error(cs.complex_map(i, o).cpu().numpy(), r["Cw"][o]) <= MAP_TOL, (i, o)
    cs.close()


@pytest.mark.parametrize("grid", [1, 2, 5, 37, 148, 296])
def test_plans_of_any_grid_are_bitwise_equal(grid):
    """Items of every orientation range, CTAs with many items and with one."""
    sizes = [(333, 277), (128, 128), (500, 90)]
    lam = [4.0, 5.656854, 11.0]
    imgs = [synth.synth_image(w, h, 5, seed=w + h) for w, h in sizes]
    b = api.Batch(sizes, lam, kp_capacity=1 << 15)
    b.load(imgs)
    b.set_tile_plan(0, 0, 0, 0)      # one CTA per tile
    b.run()
    ref = [[b.dense_map(i, s).cpu().numpy() for s in range(len(lam))] for i in range(len(sizes))]
    b.set_tile_plan(0, 1, grid, 0)
    b.run()
    for i in range(len(sizes)):
        for s in range(len(lam)):
            assert np.array_equal(ref[i][s], b.dense_map(i, s).cpu().numpy()), (i, s)
    b.close()
