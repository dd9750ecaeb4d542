"""Two cells per Eps in 3-D (13 and 25 stencil rows of five cells) against the
oracle: windows around the union's and the label pass's blocks of 8 and 16
positions and around the switches between them, sparse and dense cells, labels
by neighbour lists and by grid scan, and a cell table half full, whose probes
run on past the first slot.  Results are exact integers, so no tolerance."""
import numpy as np
import pytest

import oracle as O
from rtdbstream_gb300 import Engine
from rtdbstream_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    O.build(ref=False)
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no GPU")


SMALL = [(W, W, 3.0, 0.4) for W in (1, 7, 8, 9, 15, 16, 17, 33)]
LARGE = [(65_535, 4_369, 60.0, 0.6), (65_536, 4_096, 60.0, 0.6), (131_000, 6_550, 60.0, 0.3), (32_767, 1_057, 60.0, 0.6),
         (32_768, 2_048, 60.0, 0.6), (400_000, 8_000, 60.0, 0.2), (16_384, 1_024, 60.0, 1.2),
         (16_385, 565, 60.0, 1.2)]


@pytest.mark.parametrize("W,S,box,eps", SMALL + LARGE)
@pytest.mark.parametrize("mp", [2, 8, 40])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_matches_oracle(W, S, box, eps, mp, precision):
    slides = 2
    pts = wl.gaussian_mixture(W + slides * S, dim=3, k=40 if W > 1_000 else 2, box=box, seed=W)
    with Engine(3, W, S, eps, mp, precision=precision, cell_mult=2) as eng:
        eng.load_window(pts[:W])
        win = pts[:W].copy()
        for k in range(slides):
            lab, cid = eng.slide(pts[W + k * S: W + (k + 1) * S])
            at = (k * S) % W
            win[at: at + S] = pts[W + k * S: W + (k + 1) * S]
        enn, elab, ecid, _ = O.window_grid(win, eps, mp, O.MODE_FP64 if precision == "fp64" else O.MODE_FP32)
        assert np.array_equal(eng.counts(), enn)
        assert np.array_equal(lab, elab)
        keep = elab != 2
        assert np.array_equal(cid[keep], ecid[keep])
        assert np.array_equal(cid[~keep], np.flatnonzero(~keep))
