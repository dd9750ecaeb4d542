"""Performance cases of the streaming DBSCAN engine, through its public entry points.

Every case is one call (or the pair of calls) that a user's program makes per
window: a slide of one stream with host buffers, with device buffers or
pipelined; a round of a pool; the first window of a stream (load and cluster);
one window through the allocation-free entry point.  Window, stride, Eps and
MinPts are those of the reference's four data sets at its script's defaults
(STK 1-D, RBF 2-D, TAO 3-D, GeoLife 3-D) and of this repository's benchmark
(2-D mixture, 1M-point walkers, offset precision stream, mixed pools); the
points are synthetic, seeded and made on the GPU.

A sliding state holds one turn of the window and a few strides more, and slides
through them in a ring, so a window never holds a point twice.  All engines and
pools run on one CUDA stream, as in a program whose other kernels feed them.
Labels and ids are whole numbers, so there is no 64-bit reference to give here:
the engine's results are exact in both predicates.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from rtdbstream_gb300 import Engine, Pool, make_params
from rtdbstream_gb300.engine import load_library

_DEV = "cuda"
_stream = None


def _cuda_stream() -> torch.cuda.Stream:
    """The program's own stream (made on the first call)."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


# ------------------------------------------------------------------ the cases

def _case(name, **kw):
    c = {"name": name, "call": "slide", "data": "mixture", "dim": 2, "window": 10_000, "stride": 1_000,
         "eps": 0.5, "min_pts": 5, "precision": "fp64", "cells": 1, "clusters": 20, "box": 100.0,
         "sigma": 1.0, "neighbours": 20.0}
    c.update(kw)
    return c


def listed() -> list:
    return [
        # the smallest window the reference's scripts sweep (RBF, 2-D): one
        # blocking host call per slide, nearly all launches and latency
        _case("rbf2d-2500-host", window=2_500, stride=125, eps=0.035, min_pts=4, clusters=50, box=1.0, sigma=0.05,
              neighbours=7.0),
        # the reference's own CPU-checkable configuration: 2-D mixture, FP32
        # predicate, host buffers
        _case("mixture2d-10k-host-fp32", precision="fp32", neighbours=45.0),
        # TAO (3-D buoy measurements), device buffers: a sensor pipeline on the GPU
        _case("tao3d-10k-device", call="device", dim=3, window=10_000, stride=500, eps=1.3, min_pts=6, clusters=70,
              box=40.0, neighbours=27.0),
        # STK (1-D trade prices in cents, many equal), MinPts 2, host buffers
        _case("stk1d-100k-host", data="prices", dim=1, window=100_000, stride=5_000, eps=0.07, min_pts=2,
              clusters=500, neighbours=60.0),
        # GeoLife (3-D trajectories, dense trails), pinned host buffers with one
        # slide in flight: the steady ingest loop
        _case("geolife3d-200k-pipelined", call="pipelined", data="walkers", dim=3, window=200_000, stride=10_000,
              eps=0.01, min_pts=6, neighbours=90.0),
        # the benchmark's headline: 1M-point walker window, device buffers
        _case("walkers3d-1M-device", call="device", data="walkers", dim=3, window=1_000_000, stride=10_000,
              eps=3.3328e-3, min_pts=10),
        # the benchmark's precision stream: large offsets, many pairs within
        # rounding of Eps, near-empty cells; MinPts 2 (as in the band fixtures),
        # so that those pairs decide labels
        _case("offset3d-500k-device", call="device", data="offset", dim=3, window=500_000, stride=5_000, eps=1e-3,
              min_pts=2, neighbours=1.1),
        # tumbling window: every slide replaces the whole window (several grid
        # chunks), MinPts above the neighbour-list limit, two cells per Eps
        _case("tumbling2d-48k-device-fp32", call="device", window=48_000, stride=48_000, eps=0.4, min_pts=40,
              precision="fp32", cells=2, neighbours=130.0),
        # a pool round: 32 uneven streams (2-D and 3-D, W 1k to 200k) slide together
        _case("pool-32-mixed", call="pool", dim=0, window=200_000, stride=0, eps=0.0, min_pts=0, clusters=32),
        # first window of a small stream from host memory (a stream admitted by
        # the serving loop), at an odd size
        _case("first2d-20011-host-fp32", call="first", window=20_011, stride=20_011, eps=0.3, precision="fp32",
              neighbours=32.0),
        # first window of the 1M walker stream, points already on the device
        _case("first3d-1M-device", call="first-device", data="walkers", dim=3, window=1_000_000, stride=10_000,
              eps=3.3328e-3, min_pts=10),
        # one window through the allocation-free call (a host that owns the GPU's memory)
        _case("noalloc3d-12345", call="noalloc", dim=3, window=12_345, stride=12_345, eps=0.8, min_pts=8, box=60.0,
              neighbours=27.0),
    ]


def _log(rng, lo, hi) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng) -> dict:
    call = rng.choice(["slide", "device", "device", "pipelined", "pool", "first", "first-device", "noalloc"])
    if call == "pool":
        c = _case("", call="pool", dim=0, window=int(_log(rng, 20_000, 200_000)), stride=0, eps=0.0, min_pts=0,
                  clusters=rng.randint(4, 32))
        del c["name"]
        return c
    data = rng.choice(["mixture", "mixture", "walkers", "prices", "offset"])
    if call == "noalloc":
        W = int(_log(rng, 100, 16_384))
        S = W
    else:
        units = int(_log(rng, 1.0, 120.0))
        S = max(1, int(_log(rng, 1_000, 400_000)) // units)
        W = S * units
    precision, cells = rng.choice(["fp64", "fp64", "fp32"]), 1
    dim, k, box, sigma = rng.choice([2, 3]), 20, 100.0, 1.0
    min_pts = rng.choice([2, 4, 5, 6, 8, 10, 16, 33, 40])
    nb = _log(rng, 5.0, 60.0)
    if data == "mixture":
        n_c = 0.9 * W / k
        vol = nb / (n_c / (4.0 * math.pi) ** (dim / 2.0))
        eps = math.sqrt(vol / math.pi) if dim == 2 else (vol * 0.75 / math.pi) ** (1.0 / 3.0)
        if call not in ("noalloc", "pool"):
            cells = rng.choice([1, 1, 1, 2])
    elif data == "walkers":
        dim, eps, nb = 3, _log(rng, 2e-3, 1e-2), 40.0
    elif data == "prices":
        dim, k, eps, nb = 1, max(4, W // 200), 0.07, 60.0
    else:
        dim, eps, nb, min_pts = 3, 1e-3, 1.5, 2
    c = _case("", call=call, data=data, dim=dim, window=W, stride=S, eps=eps, min_pts=min_pts, precision=precision,
              cells=cells, clusters=k, box=box, sigma=sigma, neighbours=nb)
    del c["name"]
    return c


# ------------------------------------------------------------------ the points

def _generator(seed: int) -> torch.Generator:
    g = torch.Generator(device=_DEV)
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFF)
    return g


def _mixture(n, dim, k, box, sigma, g):
    """k Gaussians with centres uniform in the box, 10% uniform noise."""
    centres = torch.rand((k, dim), generator=g, device=_DEV, dtype=torch.float64) * box
    pts = centres[torch.randint(k, (n,), generator=g, device=_DEV)]
    pts = pts + torch.randn((n, dim), generator=g, device=_DEV, dtype=torch.float64) * sigma
    noise = torch.rand((n, dim), generator=g, device=_DEV, dtype=torch.float64) * box
    return torch.where(torch.rand((n, 1), generator=g, device=_DEV) < 0.10, noise, pts).float()


def _walkers(n, window, g):
    """Random walkers with 500 points each in a window, steps N(0, 1e-3), started
    uniformly in a 1 x 1 x 0.1 box, interleaved in time order."""
    m = max(1, round(window / 500))
    steps = -(-n // m)
    start = torch.rand((m, 3), generator=g, device=_DEV, dtype=torch.float64)
    start = start * torch.tensor([1.0, 1.0, 0.1], device=_DEV, dtype=torch.float64)
    walk = torch.randn((steps, m, 3), generator=g, device=_DEV, dtype=torch.float64).mul_(1e-3).cumsum_(0)
    return (walk + start).reshape(-1, 3)[:n].float()


def _prices(n, k, g):
    """Trades of k symbols: price levels log-uniform in 5..500, 0.2% spread, in cents."""
    level = torch.exp(torch.rand((k,), generator=g, device=_DEV, dtype=torch.float64) * math.log(100.0)) * 5.0
    p = level[torch.randint(k, (n,), generator=g, device=_DEV)]
    p = p * (1.0 + 0.002 * torch.randn((n,), generator=g, device=_DEV, dtype=torch.float64))
    return (torch.round(p * 100.0) / 100.0).float().reshape(-1, 1)


def _offset(n, eps, g):
    """Map-like offsets; 5% of the points at distance Eps (1 +- 1e-6) from another."""
    lo = torch.tensor([39.5, 116.0, 0.0], device=_DEV, dtype=torch.float64)
    size = torch.tensor([1.0, 1.0, 0.05], device=_DEV, dtype=torch.float64)
    pts = (torch.rand((n, 3), generator=g, device=_DEV, dtype=torch.float64) * size + lo).float()
    m = n // 20
    at = torch.randint(n, (2, m), generator=g, device=_DEV)
    a = pts[at[0]].double()
    d = torch.randn((m, 3), generator=g, device=_DEV, dtype=torch.float64)
    d = d / d.norm(dim=1, keepdim=True) * (0.9 * eps)
    d2 = (eps * (1.0 + 2e-6 * (torch.rand((m,), generator=g, device=_DEV, dtype=torch.float64) - 0.5))) ** 2
    near = (a + d).float()  # x and y on the float grid; z makes up the distance in doubles
    off = near[:, :2].double() - a[:, :2]
    dz = torch.sqrt(torch.clamp(d2 - off.square().sum(1), min=0.0)) * torch.sign(d[:, 2])
    near[:, 2] = (a[:, 2] + dz).float()
    keep = torch.arange(m, device=_DEV) * 20 % max(n, 1)  # places of their own, so the result is the seed's alone
    pts[keep] = near
    return pts


def _points(case, n, g):
    if case["data"] == "walkers":
        return _walkers(n, case["window"], g)
    if case["data"] == "prices":
        return _prices(n, case["clusters"], g)
    if case["data"] == "offset":
        return _offset(n, case["eps"], g)
    return _mixture(n, case["dim"], case["clusters"], case["box"], case["sigma"], g)


# ------------------------------------------------------------------ the states

class _DeviceInts:
    """int32 device memory of the library, as torch sees it; keeps its owner alive."""

    def __init__(self, owner, address, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (int(address), False), "version": 3}


def _pool_specs(case):
    """Uneven streams: 2-D and 3-D, W log-uniform in 1k..window, S 1-10% of W,
    20 neighbours, MinPts 4-16; the same for every seed."""
    r = np.random.default_rng([case["clusters"], case["window"]])
    specs = []
    for _ in range(case["clusters"]):
        dim = 2 + int(r.integers(2))
        W = int(np.exp(r.uniform(np.log(1_000), np.log(case["window"]))))
        units = int(r.integers(10, 101))
        S = max(1, W // units)
        W = S * units
        vol = float(r.uniform(10.0, 30.0)) / (0.9 * W / 20 / (4.0 * math.pi) ** (dim / 2.0))
        eps = math.sqrt(vol / math.pi) if dim == 2 else (vol * 0.75 / math.pi) ** (1.0 / 3.0)
        specs.append((dim, W, S, eps, int(r.integers(4, 17)), float(r.uniform(40.0, 160.0))))
    return specs


def _prepare_pool(case, g):
    specs = _pool_specs(case)
    rounds = max(W // S for _, W, S, _, _, _ in specs) + 2
    pool = Pool(stream=_cuda_stream().cuda_stream)
    ids, rows, outs = [], [], []
    for dim, W, S, eps, mp, box in specs:
        pts = _mixture(W + rounds * S, dim, 20, box, 1.0, g)
        torch.cuda.synchronize()
        sid = pool.add_stream(make_params(dim, W, S, eps, mp))
        pool.load_window(sid, pts[:W].contiguous())
        ids.append(sid)
        rows.append(pts[W:].reshape(rounds, S * dim))
        lab, cid = ctypes.c_void_p(), ctypes.c_void_p()
        load_library().rtdbs_pool_outputs(pool._h, sid, ctypes.byref(lab), ctypes.byref(cid))
        outs += [torch.as_tensor(_DeviceInts(pool, p.value, W), device=_DEV) for p in (lab, cid)]
    return {"call": "pool", "pool": pool, "ids": ids, "rounds": torch.cat(rows, 1).contiguous(), "outs": outs, "k": 0}


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def prepare(case, seed) -> dict:
    g = _generator(seed)
    if case["call"] == "pool":
        st = _prepare_pool(case, g)
        torch.cuda.synchronize()
        return st
    W, S, dim, call = case["window"], case["stride"], case["dim"], case["call"]
    st = {"call": call, "k": 0}
    if call == "noalloc":
        st["points"] = _points(case, W, g)
        lo, hi = st["points"].min(0).values.cpu().numpy(), st["points"].max(0).values.cpu().numpy()
        st["box"] = (np.ascontiguousarray(lo), np.ascontiguousarray(hi))
        st["args"] = (W, dim, case["eps"], case["min_pts"], 1 if case["precision"] == "fp32" else 0)
        st["out"] = tuple(torch.empty(n, dtype=torch.int32, device=_DEV) for n in (W, W, 1))
        torch.cuda.synchronize()
        return st
    st["engine"] = eng = Engine(dim, W, S, case["eps"], case["min_pts"], precision=case["precision"],
                                cell_mult=case["cells"], stream=_cuda_stream().cuda_stream)
    if call in ("first", "first-device"):
        pts = _points(case, W, g)
        st["points"] = pts if call == "first-device" else pts.cpu().numpy()
        torch.cuda.synchronize()
        return st
    m = W // S + 8  # strides in the ring
    pts = _points(case, m * S, g)
    st["ring"], st["k"] = m, W // S
    torch.cuda.synchronize()
    eng.load_window(pts[:W].contiguous())
    if call == "device":
        st["strides"] = pts.reshape(m, S, dim)
        st["out"] = tuple(torch.empty(W, dtype=torch.int32, device=_DEV) for _ in range(2))
    elif call == "pipelined":
        h = _pinned((m, S, dim), torch.float32)
        h[...] = pts.cpu().numpy().reshape(m, S, dim)
        st["strides"] = h
        st["out"] = [tuple(_pinned((W,), torch.int32) for _ in range(2)) for _ in range(2)]
    else:
        st["strides"] = pts.cpu().numpy().reshape(m, S, dim)
    torch.cuda.synchronize()
    return st


def run(st):
    call = st["call"]
    if call == "pool":
        k = st["k"]
        st["pool"].slide(st["ids"], st["rounds"][k])
        st["k"] = (k + 1) % len(st["rounds"])
        return st["outs"]
    if call == "noalloc":
        n, dim, eps, mp, prec = st["args"]
        lab, cid, status = st["out"]
        rc = load_library().rtdbs_cluster_window_noalloc_async(
            ctypes.c_void_p(st["points"].data_ptr()), n, dim, ctypes.c_double(eps), mp, prec,
            ctypes.c_void_p(st["box"][0].ctypes.data), ctypes.c_void_p(st["box"][1].ctypes.data),
            ctypes.c_void_p(lab.data_ptr()), ctypes.c_void_p(cid.data_ptr()), ctypes.c_void_p(status.data_ptr()),
            ctypes.c_void_p(_cuda_stream().cuda_stream))
        if rc != 0:
            raise RuntimeError(f"noalloc status {rc}")
        return [lab, cid, status]
    eng = st["engine"]
    if call in ("first", "first-device"):
        eng.load_window(st["points"])
        return list(eng.cluster())
    k = st["k"]
    st["k"] = (k + 1) % st["ring"]
    new = st["strides"][k]
    if call == "device":
        eng.slide_async(new, *st["out"])
        return list(st["out"])
    if call == "pipelined":
        out = st["out"][k % 2]
        eng.slide_pipelined(new, *out)
        return list(out)
    return list(eng.slide(new))


def work(case) -> dict:
    """The new points in, the window's points read once, label and id of every
    slot out; the distances of the new and expired points' neighbours, and each
    neighbour pair of the window once for the clustering."""
    if case["call"] == "pool":
        specs = _pool_specs(case)
    else:
        specs = [(case["dim"], case["window"], case["stride"], 0.0, 0, 0.0)]
    b = f = 0.0
    for dim, W, S, _, _, _ in specs:
        first = case["call"] in ("first", "first-device", "noalloc")
        b += (0 if first else 4.0 * dim * S) + 4.0 * dim * W + 8.0 * W
        pairs = W * case["neighbours"] / 2 + (0 if first else 2.0 * S * case["neighbours"])
        f += pairs * (3 * dim)
    return {"bytes": b, "flops": f}
