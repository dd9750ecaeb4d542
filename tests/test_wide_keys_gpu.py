"""Cell keys above 31 bits (clusters in a box of many cells) against the oracle:
keys of 33 to 48 bits, whose upper half holds part of or all of the first
coordinate, one and two cells per Eps, labels by lists and by scan.  Results are
exact integers, so no tolerance."""
import numpy as np
import pytest

import oracle as O
from rtdbstream_gb300 import Engine
from rtdbstream_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,box,bits", [(3, 900.0, 33), (3, 20_000.0, 45), (2, 100_000.0, 34)])
@pytest.mark.parametrize("cells", [1, 2])
@pytest.mark.parametrize("min_pts,precision", [(3, "fp64"), (40, "fp32")])
def test_matches_oracle(dim, box, bits, cells, min_pts, precision):
    O.build(ref=False)
    W, S, slides, eps = 21_000, 700, 3, 0.7
    pts = wl.gaussian_mixture(W + slides * S, dim=dim, k=30, box=box, sigma=3.0, seed=dim + cells)
    with Engine(dim, W, S, eps, min_pts, precision=precision, cell_mult=cells) as eng:
        eng.load_window(pts[:W])
        assert eng.stats()["key_bits"] >= bits
        win = pts[:W].copy()
        for k in range(slides):
            lab, cid = eng.slide(pts[W + k * S: W + (k + 1) * S])
            win[k * S: (k + 1) * S] = pts[W + k * S: W + (k + 1) * S]
        enn, elab, ecid, _ = O.window_grid(win, eps, min_pts, O.MODE_FP64 if precision == "fp64" else O.MODE_FP32)
        assert np.array_equal(eng.counts(), enn)
        assert np.array_equal(lab, elab)
        assert np.array_equal(cid[elab != 2], ecid[elab != 2])
