"""Slides of two chunks whose plan (chunk steps or one build from all slots)
changes with the window loaded, against the oracle.  Results are exact
integers, so no tolerance."""
import numpy as np
import pytest

import oracle as O
from rtdbstream_gb300 import Engine

pytestmark = pytest.mark.gpu

W, S = 68_000, 17_000


def prices(n, levels, seed):
    rng = np.random.default_rng(seed)
    return (rng.integers(0, levels, (n, 1)) * 0.01).astype(np.float32)


@pytest.mark.parametrize("min_pts,cells", [(4, 1), (40, 2)])
def test_plan_follows_the_window_loaded(min_pts, cells):
    O.build(ref=False)
    with Engine(1, W, S, 0.015, min_pts, cell_mult=cells) as eng:
        for levels, chunks in ((100_000, 1), (60, 2), (100_000, 1)):  # sparse, dense, sparse
            pts = prices(W + 3 * S, levels, levels)
            eng.load_window(pts[:W])
            assert eng.stats()["chunks_per_slide"] == chunks
            win = pts[:W].copy()
            for k in range(3):
                new = pts[W + k * S: W + (k + 1) * S]
                lab, cid = eng.slide(new)
                win[k * S: (k + 1) * S] = new
                enn, elab, ecid, _ = O.window_grid(win, 0.015, min_pts, O.MODE_FP64)
                assert np.array_equal(eng.counts(), enn)
                assert np.array_equal(lab, elab)
                assert np.array_equal(cid[elab != 2], ecid[elab != 2])
