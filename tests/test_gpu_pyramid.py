"""The pyramid kernels at the sizes where their passes change: one to three
levels in a launch and launches behind it, owned tiles of one pixel to a full
tile, odd and even sides, regions inside a level and partly outside it, levels
smaller than a region's reflection.

The levels are whole numbers, so a wrong one shows as an error of at least one
grey level: with noise of the full range the peak response is some tens of grey
levels and the largest filter weight above 1e-2, some 1e-4 .. 1e-3 of the peak
for a single wrong pixel at a scale's own level.  The maps are held to the
peak-relative bound of the other map comparisons."""
import numpy as np
import pytest

from bimp_b200 import api
from oracle import bimp_oracle as O
from parity import MAP_TOL, peak_rel_error

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,lam", [
    (64, 64, [8.0]),                       # one level: one full tile of 32
    (66, 129, [8.0]),                      # one level: a second tile of one column and of 33 rows
    (131, 67, [8.0, 16.0]),                # two levels, odd sides: 66 x 34, 33 x 17
    (64, 128, [16.0]),                     # two levels, tiles of 16 exactly full
    (250, 131, [8.0, 16.0, 32.0]),         # three levels: 125 x 66, 63 x 33, 32 x 17
    (64, 192, [32.0]),                     # three levels, tiles of 8 exactly full: 8 x 24
    (257, 263, [32.0, 64.0]),              # a launch behind the first: 17 x 17
    (520, 310, [64.0, 128.0]),             # the same with two levels: 33 x 20, 17 x 10
    (40, 33, [8.0, 16.0]),                 # levels smaller than a tile's region: 20 x 17, 10 x 9
])
def test_levels_at_tile_edges(w, h, lam):
    img = np.random.default_rng(w * 1009 + h).integers(0, 256, (h, w), dtype=np.uint8)
    img[: h // 3, : w // 3] = 255          # the largest sum of a packed lane
    res = O.run(img, lam)
    cs = api.CudaStuff(w, h, lam)
    api.getKeypoints(img, cs, capacity=50000)
    for i, r in enumerate(res):
        for o in range(8):
            assert peak_rel_error(cs.complex_map(i, o).cpu().numpy(), r["Cw"][o]) <= MAP_TOL, (i, o)
    cs.close()
