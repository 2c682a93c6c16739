"""The adjoint at the sizes where its tile kernels change: float windows that
end one value before, at and past a 16-byte chunk, tiles with one row or column
inside the map, a torus of one tile (its wrapped column carries gradient), and
items that share a tile.  Branch-matched against the FP64 gradient with the
bound of the other adjoint comparisons (the loss, a sum of both signs that can
cancel to less than its rounding allows relatively, is the other files')."""
import numpy as np
import pytest

from test_gpu_adjoint import GRAD_TOL, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,n,lam", [
    (99, 99, 1, [4.0]),                # 101 rows of cells: a second tile row with one row
    (113, 60, 1, [4.0]),               # window ends one value before the data does
    (229, 70, 1, [4.0, 5.656854]),     # ragged chunk at the right edge, both tile sizes
    (64, 64, 2, [4.0, 8.0]),           # fftW == dataW, the window wraps the torus
    (131, 103, 1, [4.0, 11.0]),        # offsets outside the built-in sets
])
def test_adjoint_window_edges(w, h, n, lam):
    _, g, gp, ref = _run(w, h, n, lam, seed=17)
    want = np.stack(ref["g"])
    assert np.linalg.norm(g - want) <= GRAD_TOL * np.linalg.norm(want)
    assert np.all(np.abs(gp - ref["p"]) <= GRAD_TOL * np.abs(ref["p"]) + 1e-6), (gp, ref["p"])
