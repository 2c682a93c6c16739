"""Tile plans of grids far above the SM count fit the work list's buffer and give
the maps of the default plan.  (A split plan's padded list holds the CTAs times
the most items of one: at these grids some CTA gets a second item, or does not,
by the weights of the cost model.)"""
import numpy as np
import pytest

from bimp_b200 import api, synth

pytestmark = pytest.mark.gpu

BANK = [4.0, 5.656854, 8.0, 11.313708]


@pytest.mark.parametrize("w,h,scales,grid,policy,order", [
    (1448, 711, 4, 941, 0, 1),
    (1567, 640, 3, 816, 0, 0),
    (910, 910, 4, 811, 0, 1),
    (1350, 1086, 2, 1063, 0, 0),
    (908, 1096, 4, 946, 0, 1),
    (460, 993, 4, 1233, 1, 0),
])
def test_large_grids_are_taken(w, h, scales, grid, policy, order):
    lam = BANK[:scales]
    b = api.Batch([(w, h)], lam)
    b.load([synth.synth_image(w, h, 6, seed=w + h)])
    b.run()
    want = [b.dense_map(0, s).cpu().numpy() for s in range(scales)]
    b.set_tile_plan(policy, order, grid, 0)
    b.run()
    for s in range(scales):
        got = b.dense_map(0, s).cpu().numpy()
        if policy == 0:   # the same tiles: the same numbers
            assert np.array_equal(got, want[s]), s
        else:
            assert np.abs(got - want[s]).max() <= 1e-4 * np.abs(want[s]).max(), s
    b.close()
