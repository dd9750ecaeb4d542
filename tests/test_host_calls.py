"""The host side of the C ABI (rtdbs_engine.cpp) against a stand-in for the
CUDA runtime (cuda_stub/stub.cpp): which resources its calls make, and which
arrays of the caller the kernels are given."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from rtdbstream_gb300 import build as B
from rtdbstream_gb300 import engine as E

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++")
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(B.nvcc()))), "include")
    if not cxx or not os.path.exists(os.path.join(inc, "cuda_runtime.h")):
        pytest.skip("no host compiler or CUDA headers")
    out = str(tmp_path_factory.mktemp("stub") / "librtdbs_stub.so")
    subprocess.run([cxx, "-std=c++17", "-O1", "-ffp-contract=off", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I", inc, "-I", B.CSRC,
                    "-I", os.path.join(B.ROOT, "include"), os.path.join(B.CSRC, "rtdbs_engine.cpp"),
                    os.path.join(HERE, "cuda_stub", "stub.cpp"), "-o", out], check=True)
    L = ctypes.CDLL(out)
    vp = ctypes.c_void_p
    L.stub_memory.restype = vp
    L.stub_memory.argtypes = [ctypes.c_size_t, ctypes.c_int]
    L.stub_io.restype = vp
    L.stub_pinned_limit.argtypes = [ctypes.c_size_t]
    L.stub_calls.argtypes = [ctypes.c_char_p]
    L.rtdbs_create.argtypes = [ctypes.POINTER(E.Params), vp, ctypes.POINTER(vp)]
    for name in ("rtdbs_load_window", "rtdbs_pool_load_window", "rtdbs_slide_async", "rtdbs_slide", "rtdbs_destroy",
                 "rtdbs_pool_destroy", "rtdbs_get_stats"):
        getattr(L, name).argtypes = {"rtdbs_load_window": [vp, vp, ctypes.c_int],
                                     "rtdbs_pool_load_window": [vp, ctypes.c_int32, vp, ctypes.c_int],
                                     "rtdbs_slide_async": [vp, vp, vp, vp], "rtdbs_slide": [vp, vp, vp, vp],
                                     "rtdbs_get_stats": [vp, vp]}.get(name, [vp])
    return L


DEVICE = 2  # cudaMemoryTypeDevice


def params(W, S, dim=2, **kw):
    p = E.Params()
    p.dim, p.window, p.stride, p.min_pts, p.eps = dim, W, S, 5, 0.5
    for k, v in kw.items():
        setattr(p, k, v)
    return p


def test_pool_streams_loaded_from_the_device_make_no_cuda_streams(lib):
    """A first window from device points without a box needs one event for the
    order between the streams, not a slide's side streams."""
    pp, pool = E.PoolParams(), ctypes.c_void_p()
    assert lib.rtdbs_pool_params_init(ctypes.byref(pp)) == 0
    assert lib.rtdbs_pool_create(ctypes.byref(pp), None, ctypes.byref(pool)) == 0
    pts = lib.stub_memory(1_000 * 8, DEVICE)
    lib.stub_reset()
    for _ in range(5):
        sid, p = ctypes.c_int32(), params(1_000, 100)
        assert lib.rtdbs_pool_add_stream(pool, ctypes.byref(p), ctypes.byref(sid)) == 0
        for _ in range(2):
            assert lib.rtdbs_pool_load_window(pool, sid.value, pts, 1) == 0
    assert lib.stub_calls(b"launch_bbox") == 10
    assert lib.stub_calls(b"cudaStreamCreate") == 0
    assert lib.stub_calls(b"cudaEventCreate") == 5
    assert lib.rtdbs_pool_destroy(pool) == 0
    assert lib.stub_calls(b"cudaEventDestroy") >= 5


def test_device_arrays_shorter_than_the_call_are_refused(lib):
    """Kernels are given a caller's device array only where its allocation
    holds all of it; a shorter one goes to the copy, which refuses it."""
    W, S = 1_000, 100
    h, p = ctypes.c_void_p(), params(W, S)
    assert lib.rtdbs_create(ctypes.byref(p), None, ctypes.byref(h)) == 0
    full = lib.stub_memory(8 * W, DEVICE)
    assert lib.rtdbs_load_window(h, full, 1) == 0
    assert lib.stub_io(0) == full
    assert lib.rtdbs_load_window(h, lib.stub_memory(8 * W - 4, DEVICE), 1) == E.RTDBS_ERR_CUDA
    assert lib.rtdbs_load_window(h, full + 4, 1) == E.RTDBS_ERR_CUDA
    new, lab, cid = lib.stub_memory(8 * S, DEVICE), lib.stub_memory(8 * W, DEVICE), lib.stub_memory(4 * W, DEVICE)
    assert lib.rtdbs_slide_async(h, new, lab + 4 * W, cid) == 0  # the second half of lab
    assert (lib.stub_io(0), lib.stub_io(1), lib.stub_io(2)) == (new, lab + 4 * W, cid)
    launched = lib.stub_calls(b"launch")
    assert lib.rtdbs_slide_async(h, new + 4, lab, cid) == E.RTDBS_ERR_CUDA
    assert lib.stub_calls(b"launch") == launched  # nothing ran
    assert lib.rtdbs_slide_async(h, new, lab + 4 * W + 4, cid) == E.RTDBS_ERR_CUDA
    assert (lib.stub_io(1), lib.stub_io(2)) == (None, cid)  # the label pass was not given it
    assert lib.rtdbs_slide_async(h, new, lab, cid + 8) == E.RTDBS_ERR_CUDA
    assert (lib.stub_io(1), lib.stub_io(2)) == (lab, None)
    assert lib.rtdbs_destroy(h) == 0


def test_engine_without_pinned_staging_still_runs(lib):
    """Where the pinned buffers of host calls cannot be had, an engine keeps
    the control block's mirror alone, and host calls copy."""
    W, S = 1_000, 100
    h, p = ctypes.c_void_p(), params(W, S)
    lib.stub_pinned_limit(4_096)
    try:
        assert lib.rtdbs_create(ctypes.byref(p), None, ctypes.byref(h)) == 0
    finally:
        lib.stub_pinned_limit(1 << 62)
    pts = (ctypes.c_float * (2 * W))()
    out = [(ctypes.c_int32 * W)() for _ in range(2)]
    at = [ctypes.c_void_p(ctypes.addressof(x)) for x in (pts, *out)]
    assert lib.rtdbs_load_window(h, at[0], 0) == 0
    copies = lib.stub_calls(b"cudaMemcpyAsync")
    assert lib.rtdbs_slide(h, *at) == 0
    assert lib.stub_calls(b"cudaMemcpyAsync") == copies + 4  # points, label, ids, control block
    assert (lib.stub_io(1), lib.stub_io(2)) == (None, None)
    assert lib.rtdbs_destroy(h) == 0


@pytest.mark.parametrize("warps,S,cells,lanes,want", [(5_472, 5_472, 1, 0, 32), (5_472, 5_473, 1, 0, 16),
                                                      (4_752, 4_753, 1, 0, 16), (4_752, 4_752, 0, 0, 32),
                                                      (5_472, 9_000, 2, 0, 32), (5_472, 9_000, 1, 32, 32),
                                                      (5_472, 100, 1, 16, 16)])
def test_lanes_per_query_by_resident_warps(lib, warps, S, cells, lanes, want):
    """A whole warp per query while the device holds the warps of a stride at once."""
    lib.stub_warps(warps)
    h, p = ctypes.c_void_p(), params(2 * S, S, cell_mult=cells, query_lanes=lanes)
    assert lib.rtdbs_create(ctypes.byref(p), None, ctypes.byref(h)) == 0
    assert lib.rtdbs_load_window(h, lib.stub_memory(16 * S, DEVICE), 1) == 0
    assert lib.stub_lanes() == want
    assert lib.rtdbs_destroy(h) == 0
    lib.stub_warps(5_472)


@pytest.mark.parametrize("cells", [1, 2])
@pytest.mark.parametrize("lo,hi,eps", [(0.0, 100.0, 0.5), (-0.25, 1.25, 3.3e-3), (39.5, 40.5, 1e-3), (116.0, 117.0, 1e-3),
                                       (-1e4, 1e4, 0.37), (0.0, 4.0e6, 1.0), (1e6, 1e6 + 10, 0.02), (0.0, 1e-3, 1e-9),
                                       (-3e38, 3e38, 1e30), (0.0, 1e-36, 1e-38)])
def test_cells_as_compiled_are_the_double_ones(lib, lo, hi, eps, cells):
    """The cell coordinate (its single-precision shortcut and the geometry that
    bounds it, as the library compiles them) against floor((x - lo) / side) in
    double, clamped: on, next to, between and outside cell edges."""
    lo, hi = float(np.float32(lo)), float(np.float32(hi))
    ext, side, err = ctypes.c_longlong(), ctypes.c_double(), ctypes.c_float()

    def run(x):
        out = np.empty(len(x), np.int64)
        assert lib.stub_cells(ctypes.c_double(eps), cells, ctypes.c_float(lo), ctypes.c_float(hi),
                              x.ctypes.data_as(ctypes.c_void_p), ctypes.c_longlong(len(x)),
                              out.ctypes.data_as(ctypes.c_void_p), ctypes.byref(ext), ctypes.byref(side),
                              ctypes.byref(err)) == 0
        return out

    run(np.zeros(1, np.float32))
    rng = np.random.default_rng(int(abs(lo) % 1e9) + cells)
    with np.errstate(over="ignore"):
        edges = (lo + rng.integers(-3, ext.value + 3, 200_000) * side.value).astype(np.float32)
        span = hi - lo
        x = np.concatenate([rng.uniform(lo - 0.1 * span, hi + 0.1 * span, 400_000).astype(np.float32), edges,
                            np.nextafter(edges, np.float32(np.inf)), np.nextafter(edges, np.float32(-np.inf)),
                            np.array([hi, lo, 3e38, -3e38, np.inf, -np.inf, np.nan], np.float32)])
    with np.errstate(invalid="ignore", over="ignore"):
        t = np.floor((x.astype(np.float64) - lo) * (1.0 / side.value))
    want = np.clip(np.where(t >= 0, t, 0), 0, ext.value - 1).astype(np.int64)
    assert np.array_equal(run(x), want)
    assert err.value > 0


# W, S, dim, cells per Eps, cell runs and distance tests of the first window, and
# the slide's measured us by chunk steps and by a whole build
PLANS = [(1_000_000, 50_000, 1, 1, 32_217, 13_389_424_178, 17_473, 73_530),  # many equal prices
         (200_000, 40_000, 1, 2, 8_005, 472_327_967, 1_259, 3_539),
         (1_000_000, 50_000, 3, 2, 998_791, 522_560, 733, 2_308),            # near-empty cells
         (400_000, 20_000, 3, 2, 384_839, 6_766_817, 366, 925),
         (100_000, 100_000, 3, 2, 99_987, 5_868, 689, 324),
         (400_000, 80_000, 3, 1, 398_056, 124_137, 424, 252),
         (100_000, 50_000, 2, 1, 27_762, 8_132_314, 292, 137),
         (40_000, 40_000, 3, 1, 9_710, 2_947_298, 232, 127),
         (1_000_000, 200_000, 1, 2, 78_762, 102_659_006, 1_496, 327),
         (1_000_000, 500_000, 3, 1, 358_049, 173_499_013, 3_807, 850)]


def test_slides_build_the_window_where_that_is_cheaper(lib):
    """The plan of a slide of two chunks or more follows the window that was
    loaded last; one chunk, or less than a twentieth, is always stepped."""
    for W, S, dim, cells, runs, tests, steps, build in PLANS:
        h, p, s = ctypes.c_void_p(), params(W, S, dim, cell_mult=cells), E.Stats()
        assert lib.rtdbs_create(ctypes.byref(p), None, ctypes.byref(h)) == 0
        pts, new = (lib.stub_memory(4 * dim * n, DEVICE) for n in (W, S))
        chunks = -(-S // 16_384)
        for r, t, want in ((runs, tests, 1 if build < steps else chunks), (100, 0, 1)):
            lib.stub_window(r, ctypes.c_ulonglong(t))
            assert lib.rtdbs_load_window(h, pts, 1) == 0
            lib.stub_reset()
            assert lib.rtdbs_slide_async(h, new, None, None) == 0
            assert lib.stub_calls(b"launch_window_build") == (1 if want == 1 else 0), (W, S, dim, cells, r, t)
            assert lib.rtdbs_get_stats(h, ctypes.byref(s)) == 0 and s.chunks_per_slide == want
        assert lib.rtdbs_destroy(h) == 0
    for W, S in ((1_000, 1_000), (16_384, 16_384), (357_000, 17_000)):
        h, p = ctypes.c_void_p(), params(W, S)
        lib.stub_window(100, ctypes.c_ulonglong(0))
        assert lib.rtdbs_create(ctypes.byref(p), None, ctypes.byref(h)) == 0
        assert lib.rtdbs_load_window(h, lib.stub_memory(8 * W, DEVICE), 1) == 0
        lib.stub_reset()
        assert lib.rtdbs_slide_async(h, lib.stub_memory(8 * S, DEVICE), None, None) == 0
        assert lib.stub_calls(b"launch_window_build") == 0
        assert lib.rtdbs_destroy(h) == 0
