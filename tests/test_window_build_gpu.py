"""The grid built from all slots at once (first windows, slides of two chunks
or more) against the oracle: sizes around one chunk, the radix sort's tiles
and the switch to its separate scan, both cell multipliers, list and scan
labels, device and host points, non-finite points, keys too wide for one sort
word (chunk steps), and a pool's stream slid on its own between rounds.
Results are exact integers, so no tolerance."""
import ctypes

import numpy as np
import pytest

import oracle as O
from rtdbstream_gb300 import Engine, Pool, make_params
from rtdbstream_gb300 import workloads as wl
from rtdbstream_gb300.engine import load_library

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    O.build(ref=False)
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no GPU")


def mix(n, dim, box, seed):
    return wl.gaussian_mixture(n, dim=dim, k=12, box=box, seed=seed)


def check(eng, lab, cid, win, eps, mp, precision):
    mode = O.MODE_FP64 if precision == "fp64" else O.MODE_FP32
    enn, elab, ecid, _ = O.window_grid(win, eps, mp, mode)
    assert np.array_equal(eng.counts(), enn)
    assert np.array_equal(lab, elab)
    keep = elab != 2
    assert np.array_equal(cid[keep], ecid[keep])
    assert np.array_equal(cid[~keep], np.flatnonzero(~keep))


FIRST = [(W, 1 + W % 3, 5 if W % 2 else 40) for W in (1, 33, 1_023, 1_024, 1_025, 4_097, 16_383, 16_384, 16_385)]
FIRST += [(20_480, 3, 6), (20_481, 2, 2), (262_144, 3, 8), (262_145, 2, 12)]


@pytest.mark.parametrize("W,dim,mp", FIRST)
@pytest.mark.parametrize("precision,cells,device", [("fp64", 1, False), ("fp32", 2, True)])
def test_first_window(W, dim, mp, precision, cells, device):
    import torch

    pts = mix(W, dim, 60.0, W)
    eps = 0.02 if dim == 1 else (0.3 if dim == 2 else 0.8)
    if W > 1_000:
        pts[::997] = np.nan  # cell 0, no neighbours
    with Engine(dim, W, W, eps, mp, precision=precision, cell_mult=cells) as eng:
        eng.load_window(torch.from_numpy(pts).cuda() if device else pts)
        lab, cid = eng.cluster()
        check(eng, lab, cid, pts, eps, mp, precision)


SLIDES = [("S_is_W", 20_000, 20_000, 2), ("half", 40_000, 20_000, 2), ("fifth", 100_000, 20_000, 3),
          ("one_chunk", 32_768, 16_384, 2), ("two_chunks", 32_770, 16_385, 2), ("steps", 378_000, 18_000, 2)]


@pytest.mark.parametrize("name,W,S,dim", SLIDES, ids=[s[0] for s in SLIDES])
@pytest.mark.parametrize("mp,precision,cells", [(5, "fp64", 1), (36, "fp32", 2)])
def test_slides(name, W, S, dim, mp, precision, cells):
    slides = 3
    pts = mix(W + slides * S, dim, 80.0, S)
    eps = 0.25 if dim == 2 else 0.6
    with Engine(dim, W, S, eps, mp, precision=precision, cell_mult=cells) as eng:
        eng.load_window(pts[:W])
        win = pts[:W].copy()
        for k in range(slides):
            new = pts[W + k * S: W + (k + 1) * S]
            lab, cid = eng.slide(new)
            at = (k * S) % W
            win[at: at + S] = new
        check(eng, lab, cid, win, eps, mp, precision)


def test_wide_keys_load_by_chunk_steps():
    W, S, eps = 17_000, 17_000, 1e-3
    rng = np.random.default_rng(8)
    pts = np.concatenate([rng.uniform(-60.0, 60.0, (200, 3)), rng.normal(0, 0.01, (2 * W - 200, 3))])
    pts = pts[rng.permutation(len(pts))].astype(np.float32)
    with Engine(3, W, S, eps, 3, bbox=([-64.0, -64.0, -32.0], [64.0, 64.0, 32.0])) as eng:
        assert eng.stats()["key_bits"] + 15 > 64
        eng.load_window(pts[:W])
        lab, cid = eng.cluster()
        check(eng, lab, cid, pts[:W], eps, 3, "fp64")
        lab, cid = eng.slide(pts[W:])
        check(eng, lab, cid, pts[W:], eps, 3, "fp64")


def test_pool_stream_slid_on_its_own():
    """A whole-window slide keeps no chunk order: later rounds sort."""
    import torch

    W, S, eps, mp = 40_000, 20_000, 0.25, 5
    pts = mix(W + 6 * S, 2, 80.0, 3)
    pool = Pool()
    sid = pool.add_stream(make_params(2, W, S, eps, mp))
    pool.load_window(sid, pts[:W])
    h = ctypes.c_void_p()
    L = load_library()
    assert L.rtdbs_pool_engine(pool._h, sid, ctypes.byref(h)) == 0
    lab, cid = np.empty(W, np.int32), np.empty(W, np.int32)
    for k in range(6):
        new = np.ascontiguousarray(pts[W + k * S: W + (k + 1) * S])
        if k == 2:
            assert L.rtdbs_slide(h, new.ctypes.data, lab.ctypes.data, cid.ctypes.data) == 0
        else:
            pool.slide([sid], torch.from_numpy(new).cuda())
            pool.sync()
        win = pts[k * S + S: k * S + S + W]
        win = np.roll(win, ((k + 1) * S) % W, axis=0)
        enn, elab, ecid, _ = O.window_grid(win, eps, mp, O.MODE_FP64)
        lab, cid = pool.outputs(sid)
        assert np.array_equal(pool.counts(sid), enn) and np.array_equal(lab, elab)
        assert np.array_equal(cid[elab != 2], ecid[elab != 2])
    pool.close()
