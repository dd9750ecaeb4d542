"""Host-buffer calls with every kind of host array: points that work queued on
the engine's stream is still writing (pinned and managed arrays, and plain
ones above the size that the driver takes at once) are read in the stream's
order, and results reach plain, pinned and managed arrays alike, at windows on
both sides of the engine's own pinned buffers.  Results are exact integers, so
no tolerance."""
import ctypes

import numpy as np
import pytest

import oracle as O
from rtdbstream_gb300 import Engine
from rtdbstream_gb300 import workloads as wl
from rtdbstream_gb300.engine import load_library

pytestmark = pytest.mark.gpu

EPS, MP = 0.3, 6
DELAY = 20_000_000  # clock cycles of queued work before the points arrive (about 10 ms)


@pytest.fixture(scope="module", autouse=True)
def _built():
    O.build(ref=False)
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no GPU")


class Managed:
    """A managed array, freed with the object."""

    def __init__(self, rt, a):
        self.rt, self.shape, self.dtype = rt, a.shape, a.dtype
        p = ctypes.c_void_p()
        assert rt.cudaMallocManaged(ctypes.byref(p), ctypes.c_size_t(a.nbytes), 1) == 0
        self.ptr = p.value
        ctypes.memmove(self.ptr, a.ctypes.data, a.nbytes)

    def get(self):
        n = int(np.prod(self.shape)) * np.dtype(self.dtype).itemsize
        return np.frombuffer(ctypes.string_at(self.ptr, n), self.dtype).reshape(self.shape).copy()

    def __del__(self):
        self.rt.cudaFree(ctypes.c_void_p(self.ptr))


class Plain:
    def __init__(self, rt, a):
        self.a = np.ascontiguousarray(a).copy()
        self.ptr = self.a.ctypes.data

    def get(self):
        return self.a


class Pinned(Plain):
    def __init__(self, rt, a):
        import torch

        self.t = torch.from_numpy(np.ascontiguousarray(a).copy()).pin_memory()
        self.a, self.ptr = self.t.numpy(), self.t.data_ptr()


KINDS = {"plain": Plain, "pinned": Pinned, "managed": Managed}


@pytest.fixture(scope="module")
def rt():
    for name in ("libcudart.so.13", "libcudart.so"):
        try:
            return ctypes.CDLL(name)
        except OSError:
            continue
    pytest.skip("no shared CUDA runtime to allocate managed memory with")


def expected(win, mp):
    _, lab, cid, _ = O.window_grid(win, EPS, mp, O.MODE_FP64)
    return lab, np.where(lab == 2, np.arange(len(lab)), cid)


def same(lab, cid, exp):
    return np.array_equal(lab, exp[0]) and np.array_equal(cid, exp[1])


# plain arrays of 96 kB: up to 64 kB the driver takes them when called, in no order
@pytest.mark.parametrize("kind,W,S", [("pinned", 2_400, 300), ("managed", 2_400, 300), ("plain", 48_000, 12_000),
                                      ("pinned", 140_000, 5_000), ("managed", 140_000, 5_000)])
def test_points_written_by_queued_work(rt, kind, W, S):
    import torch

    pts = wl.gaussian_mixture(W + S, dim=2, k=20, seed=3)
    new, stale = np.ascontiguousarray(pts[W:]), np.full((S, 2), 7.0, np.float32)
    exp = expected(np.concatenate([new, pts[S:W]]), MP)
    st = torch.cuda.Stream()
    with Engine(2, W, S, EPS, MP, stream=st.cuda_stream) as eng:
        eng.load_window(pts[:W])
        d = torch.from_numpy(new).cuda()
        torch.cuda.synchronize()
        arr = KINDS[kind](rt, stale)
        lab, cid = np.empty(W, np.int32), np.empty(W, np.int32)
        write = ctypes.CFUNCTYPE(None, ctypes.c_void_p)(lambda _: ctypes.memmove(arr.ptr, new.ctypes.data, new.nbytes))
        with torch.cuda.stream(st):
            torch.cuda._sleep(DELAY)
        s = ctypes.c_void_p(st.cuda_stream)
        if kind == "plain":
            assert rt.cudaLaunchHostFunc(s, write, None) == 0
        else:
            assert rt.cudaMemcpyAsync(ctypes.c_void_p(arr.ptr), ctypes.c_void_p(d.data_ptr()),
                                      ctypes.c_size_t(new.nbytes), 4, s) == 0
        assert load_library().rtdbs_slide(eng._h, ctypes.c_void_p(arr.ptr), ctypes.c_void_p(lab.ctypes.data),
                                          ctypes.c_void_p(cid.ctypes.data)) == 0
        torch.cuda.synchronize()
        assert same(lab, cid, exp)


@pytest.mark.parametrize("W,S", [(2_400, 300), (140_000, 5_000)])
@pytest.mark.parametrize("mp", [MP, 40])  # label pass by lists and by grid scan
@pytest.mark.parametrize("points,label,ids", [("plain", "plain", "plain"), ("pinned", "pinned", "pinned"),
                                              ("managed", "managed", "managed"), ("plain", "pinned", "plain"),
                                              ("pinned", "plain", "managed"), ("plain", None, "pinned"),
                                              ("managed", "plain", None), ("plain", None, None)])
def test_results_reach_every_kind_of_array(rt, W, S, mp, points, label, ids):
    L = load_library()
    pts = wl.gaussian_mixture(W + 2 * S, dim=2, k=20, seed=4)
    blank = np.full(W, -9, np.int32)
    with Engine(2, W, S, EPS, mp) as eng:
        eng.load_window(pts[:W])
        win = pts[:W].copy()
        for k in range(3):
            lab, cid = (None if x is None else KINDS[x](rt, blank) for x in (label, ids))
            out = [ctypes.c_void_p(None if x is None else x.ptr) for x in (lab, cid)]
            if k < 2:
                new = pts[W + k * S: W + (k + 1) * S]
                win[k * S: (k + 1) * S] = new
                assert L.rtdbs_slide(eng._h, ctypes.c_void_p(KINDS[points](rt, new).ptr), *out) == 0
            else:
                assert L.rtdbs_cluster(eng._h, *out, 0) == 0
            exp = expected(win, mp)
            assert lab is None or np.array_equal(lab.get(), exp[0])
            assert cid is None or np.array_equal(cid.get(), exp[1])


# lists off: the grid scan stores to the engine's pinned buffers up to 24,576
# points, copies follow it above
@pytest.mark.parametrize("W,S", [(24_576, 1_024), (24_577, 3_511), (131_072, 4_096)])
@pytest.mark.parametrize("mp", [1, 40])
def test_grid_scan_results_reach_plain_arrays(W, S, mp):
    pts = wl.gaussian_mixture(W + S, dim=2, k=20, seed=5)
    with Engine(2, W, S, EPS, mp) as eng:
        eng.load_window(pts[:W])
        assert same(*eng.cluster(), expected(pts[:W], mp))
        win = pts[:W].copy()
        win[:S] = pts[W:]
        assert same(*eng.slide(pts[W:]), expected(win, mp))
