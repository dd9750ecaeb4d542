"""The single-precision shortcut of the cell coordinates (rtdbs_kernels.cu,
cell_coord) restated in numpy against the double-precision coordinate: the
same cell wherever the shortcut is taken, over offsets, cell sides and points
on, next to and outside cell edges."""
import numpy as np
import pytest


def geometry(lo, hi, L):
    ext = int(np.floor((hi - lo) / L)) + 1
    err = 2.0 * 2.0 ** -24 * (abs(lo) / L + 4.0 * (ext + 2.0))
    err = np.nextafter(np.float32(err), np.float32(1.0)) if err < 0.4 else np.float32(2.0)
    return ext, np.float32(lo), np.float32(1.0 / L), err


def exact(x, lo, L, ext):
    t = np.floor((x.astype(np.float64) - lo) * (1.0 / L))
    return np.clip(np.where(t >= 0, t, 0), 0, ext - 1).astype(np.int64)


@pytest.mark.parametrize("lo,hi,L", [(0.0, 100.0, 0.5), (-0.25, 1.25, 3.3e-3), (39.5, 40.5, 1e-3), (116.0, 117.0, 1e-3),
                                     (-1e4, 1e4, 0.37), (0.0, 4.0e6, 1.0), (1e6, 1e6 + 10, 0.02), (0.0, 1e-3, 1e-9)])
def test_shortcut_gives_the_double_cell(lo, hi, L):
    rng = np.random.default_rng(int(abs(lo) + 7))
    ext, lo32, inv32, err = geometry(lo, hi, L)
    k = rng.integers(-3, ext + 3, 200_000)
    edges = (lo + k * L).astype(np.float32)
    x = [rng.uniform(lo - 0.1 * (hi - lo), hi + 0.1 * (hi - lo), 400_000).astype(np.float32), edges,
         np.nextafter(edges, np.float32(np.inf)), np.nextafter(edges, np.float32(-np.inf)),
         np.array([hi * 1e6, -hi * 1e6, 3e38, -3e38], np.float32)]
    x = np.concatenate(x)
    with np.errstate(over="ignore", invalid="ignore"):
        t = (x - lo32) * inv32
        f = np.floor(t)
        frac = t - f
        taken = (t >= 0) & (t < np.float32(4194304.0)) & (frac >= err) & (frac <= np.float32(1.0) - err)
    got = np.minimum(f[taken].astype(np.int64), ext - 1)
    assert np.array_equal(got, exact(x[taken], lo, L, ext))
    if err < 0.01:
        assert taken[:400_000].mean() > 0.8
