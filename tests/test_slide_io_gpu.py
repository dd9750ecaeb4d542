"""The arrays a slide exchanges with its caller: read and written by the
kernels where they are the device's own aligned memory (or the engine's pinned
buffers), copied otherwise.  Every form gives the oracle's labels and ids."""
import ctypes

import numpy as np
import pytest

import oracle as O
from rtdbstream_gb300 import Engine
from rtdbstream_gb300 import workloads as wl
from rtdbstream_gb300.engine import load_library

pytestmark = pytest.mark.gpu

W, S, EPS, MP, SLIDES = 2_400, 300, 0.5, 5, 10


@pytest.fixture(scope="module", autouse=True)
def _built():
    O.build(ref=False)
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no GPU")


@pytest.fixture(scope="module")
def stream():
    pts = wl.gaussian_mixture(W + SLIDES * S, dim=2, k=6, box=20.0, seed=91)
    return pts, O.stream(pts, W, S, EPS, MP, O.MODE_FP64, first_slide=1, n_out=SLIDES)


def equal(lab, cid, exp, k):
    keep = exp[1][k] != 2
    return (np.array_equal(lab, exp[1][k]) and np.array_equal(cid[keep], exp[2][k][keep])
            and np.array_equal(cid[~keep], np.flatnonzero(~keep)))


@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("mp", [MP, 40])  # label pass by lists and by grid scan
@pytest.mark.parametrize("form", ["aligned", "odd_bytes", "own", "joined", "changing"])
def test_device_arrays(stream, form, use_graph, mp):
    import torch

    pts, exp = stream
    if mp != MP:
        exp = O.stream(pts, W, S, EPS, mp, O.MODE_FP64, first_slide=1, n_out=SLIDES)
    L = load_library()
    with Engine(2, W, S, EPS, mp, use_graph=use_graph) as eng:
        eng.load_window(pts[:W])
        own = eng.device_outputs()
        raw = torch.zeros(2 * 4 * W + 64, dtype=torch.uint8, device="cuda")
        inp = torch.zeros(8 * S + 64, dtype=torch.uint8, device="cuda")
        for k in range(SLIDES):
            new = torch.from_numpy(np.ascontiguousarray(pts[W + k * S: W + (k + 1) * S])).cuda()
            src, lab, cid = new.data_ptr(), raw.data_ptr(), raw.data_ptr() + 4 * W
            if form == "odd_bytes":  # no alignment at all: copied
                inp[3: 3 + 8 * S].copy_(new.reshape(-1).view(torch.uint8))
                src, lab, cid = inp.data_ptr() + 3, raw.data_ptr() + 1, raw.data_ptr() + 4 * W + 5
            elif form == "own":
                lab, cid = own
            elif form == "joined":  # one array: the ids come last
                cid = lab
            elif form == "changing":  # other arrays, or none, from slide to slide
                lab, cid = (lab, None) if k % 3 == 1 else ((None, cid) if k % 3 == 2 else (cid, lab))
            torch.cuda.synchronize()
            assert L.rtdbs_slide_async(eng._h, ctypes.c_void_p(src), ctypes.c_void_p(lab), ctypes.c_void_p(cid)) == 0
            eng.sync()

            def ints(at):
                off = at - raw.data_ptr()
                return np.frombuffer(raw.cpu().numpy().tobytes()[off: off + 4 * W], np.int32)

            keep = exp[1][k] != 2
            if form == "own":
                glab, gcid = (torch.as_tensor(_Ints(p), device="cuda").cpu().numpy() for p in (lab, cid))
            elif form == "joined":
                glab, gcid = exp[1][k], ints(cid)
            else:
                glab = ints(lab) if lab is not None else exp[1][k]
                gcid = ints(cid) if cid is not None else np.where(keep, exp[2][k], np.arange(W))
            assert equal(glab, gcid, exp, k), f"{form}: slide {k + 1}"


class _Ints:
    def __init__(self, address):
        self.__cuda_array_interface__ = {"shape": (W,), "typestr": "<i4", "data": (int(address), False), "version": 3}


@pytest.mark.parametrize("n_w,n_s", [(131_072, 4_096), (135_168, 4_096)])  # pinned buffers, and copies above
def test_host_arrays_at_the_staging_limit(n_w, n_s):
    pts = wl.gaussian_mixture(n_w + 2 * n_s, dim=2, k=30, box=200.0, seed=7)
    with Engine(2, n_w, n_s, 0.4, 6) as eng:
        eng.load_window(pts[:n_w])
        lab0, cid0 = eng.cluster()
        _, elab, ecid, _ = O.window_grid(pts[:n_w], 0.4, 6, O.MODE_FP64)
        assert np.array_equal(lab0, elab) and np.array_equal(cid0[elab != 2], ecid[elab != 2])
        for k in range(2):
            lab, cid = eng.slide(pts[n_w + k * n_s: n_w + (k + 1) * n_s])
        win = pts[:n_w].copy()
        win[: 2 * n_s] = pts[n_w:]
        _, elab, ecid, _ = O.window_grid(win, 0.4, 6, O.MODE_FP64)
        assert np.array_equal(lab, elab) and np.array_equal(cid[elab != 2], ecid[elab != 2])


@pytest.mark.parametrize("bbox", [None, ([-5.0, -5.0], [25.0, 25.0])])
@pytest.mark.parametrize("odd", [0, 3])
def test_first_window_from_device_bytes(stream, bbox, odd):
    """Device points at any byte: read in place where aligned, copied otherwise."""
    import torch

    pts = stream[0][:W]
    raw = torch.zeros(8 * W + 64, dtype=torch.uint8, device="cuda")
    raw[odd: odd + 8 * W].copy_(torch.from_numpy(np.ascontiguousarray(pts)).cuda().reshape(-1).view(torch.uint8))
    torch.cuda.synchronize()
    with Engine(2, W, S, EPS, MP, bbox=bbox) as eng:
        assert load_library().rtdbs_load_window(eng._h, ctypes.c_void_p(raw.data_ptr() + odd), 1) == 0
        lab, cid = eng.cluster()
        _, elab, ecid, _ = O.window_grid(pts, EPS, MP, O.MODE_FP64)
        assert np.array_equal(lab, elab) and np.array_equal(cid[elab != 2], ecid[elab != 2])
