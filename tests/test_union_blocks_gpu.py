"""Clustering by blocks of sorted positions (link pass and union) against the
FP64/FP32 oracle, at the edges of its blocks: windows around 16 and 32
positions, around the block-size switch at 32,768 points, cells spanning many
blocks, keys above 31 bits (64-bit lookups), and slides in which components
are kept, cut and joined.  Results are exact integers, so no tolerance."""
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


def _chain(n, dim, step, seed):
    """Points of a line, `step` apart, in a shuffled order: one long component."""
    p = np.zeros((n, dim), np.float32)
    p[:, -1] = np.arange(n, dtype=np.float32) * np.float32(step)
    return p[np.random.default_rng(seed).permutation(n)]


CASES = [(f"W{W}_{dim}d", lambda W=W, dim=dim: wl.gaussian_mixture(3 * W, dim=dim, k=2, box=3.0, seed=W), W, W, 0.4, 3)
         for W in (1, 15, 16, 17, 31, 32, 33, 97) for dim in (1, 2, 3)]
CASES += [
    ("W32767_3d", lambda: wl.random_walkers(32_767 + 2 * 31, n_walkers=65, seed=3), 32_767, 31, 5e-3, 6),
    ("W32768_3d", lambda: wl.random_walkers(32_768 + 2 * 512, n_walkers=65, seed=4), 32_768, 512, 5e-3, 6),
    ("one_cell", lambda: np.random.default_rng(5).normal(0, 0.02, (3_000, 2)).astype(np.float32), 1_000, 500, 0.5, 4),
    ("chain", lambda: _chain(4_000, 2, 0.4, 6), 2_000, 400, 0.5, 2),
    ("wide_keys", lambda: wl.gaussian_mixture(3_000, dim=3, k=6, box=4_000.0, sigma=0.02, noise_frac=0.3, seed=7),
     2_000, 250, 0.02, 3),
]


@pytest.mark.parametrize("name,gen,W,S,eps,mp", CASES, ids=[c[0] for c in CASES])
@pytest.mark.parametrize("precision,cell_mult", [("fp64", 1), ("fp32", 2)])
def test_blocks_match_oracle(name, gen, W, S, eps, mp, precision, cell_mult):
    pts = gen()
    slides = min(5, (len(pts) - W) // S)
    mode = O.MODE_FP64 if precision == "fp64" else O.MODE_FP32
    enn, elab, ecid = O.stream(pts, W, S, eps, mp, mode, first_slide=1, n_out=slides)
    with Engine(pts.shape[1], W, S, eps, mp, precision=precision, cell_mult=cell_mult) as eng:
        eng.load_window(pts[:W])
        if name == "wide_keys":
            assert eng.stats()["key_bits"] > 31
        for k in range(slides):
            lab, cid = eng.slide(pts[W + k * S: W + (k + 1) * S])
            assert np.array_equal(eng.counts(), enn[k])
            assert np.array_equal(lab, elab[k])
            keep = elab[k] != 2
            assert np.array_equal(cid[keep], ecid[k][keep])
            assert np.array_equal(cid[~keep], np.flatnonzero(~keep))
