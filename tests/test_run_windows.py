"""CPU check of the run kernel's shared-memory windows: for every 32 x 32 tile and
angle the window starts at the lowest corner's bin minus one, rounded down, and
holds Wrun elements; every pixel's bin and the four elements after it must lie
inside, and the window inside the stored row, so that the kernel's clamp never
changes a result.  The plan's row layout comes from the library (raft_plan_window),
the tile's width and rule are restated (backproject.cu plan_window, angle_param)."""
import numpy as np
import pytest

TILE = 32
f32 = np.float32


def _plan(pf, pi, geometry, store):
    from sscRaft.rafttypes import _ptr, check_error, libraft
    out = np.zeros(4, np.int32)
    if libraft.raft_plan_window(_ptr(pf), _ptr(pi), geometry, store, _ptr(out)):
        check_error("plan_window")
    wlo, Wg, _, align = [int(v) for v in out]
    return wlo, Wg, int(np.ceil(np.hypot(31.0, 31.0))) + 8 + align, align


def _tiles(a):
    n = a.shape[0] // TILE
    return a.reshape(n, TILE, n, TILE).transpose(0, 2, 1, 3)


@pytest.mark.parametrize("N,pad,pixel,geometry", [(33, 0, 1.0, 0), (64, 2, 1.0, 0), (130, 1, 0.7, 0), (257, 2, 2.5, 0),
                                                  (1000, 2, 1.0, 0), (48, 0, 1.0, 2), (129, 0, 1.0, 2), (700, 0, 1.0, 2),
                                                  (50, 1, 1.0, 1), (513, 2, 1.0, 1)])
def test_run_windows_in_bounds(N, pad, pixel, geometry):
    rng = np.random.default_rng(N)
    angles = np.concatenate([[0, np.pi / 4, np.pi / 2, np.pi, 1.5 * np.pi], rng.uniform(0, 2 * np.pi, 20)])
    ext = -(-N // TILE) * TILE
    i = np.arange(ext)
    for store in ((1, 2) if geometry == 1 else (0,)):
        pf = np.array([0, 0, 1, 0, pixel, pixel, 0], np.float32)
        pi = np.array([N, 20, 1, N, pad, 0, 0, 1 if geometry == 2 else 7, 1, 0], np.int32)
        wlo, Wg, W, align = _plan(pf, pi, geometry, store)
        Np, off = N * (1 + pad), (pad * N) // 2
        for th in angles.astype(np.float32):
            c, s = np.cos(th, dtype=f32), np.sin(th, dtype=f32)
            if geometry == 1:
                c64, s64 = np.cos(float(th)), np.sin(float(th))
                x = i + off - 0.5 * Np
                v = x[None, :] * c64 - x[:, None] * s64 + 0.5 * Np - wlo - 0.5
                k = _tiles(np.rint(v).astype(np.int64))
                lo = np.floor(_tiles(v).min((2, 3))).astype(np.int64) - 1
            else:
                if geometry == 0:
                    d, lo0 = f32(pixel), f32(-f32(pixel) * f32(Np) / f32(2))
                    x, sgn = (lo0 + (i + off).astype(f32) * d).astype(f32), f32(-1)
                else:
                    d, lo0 = f32(2.0 / (N - 1)), f32(-1)
                    x, sgn = (lo0 + i.astype(f32) * d).astype(f32), f32(1)
                t = (x[None, :] * c + sgn * (x[:, None] * s)).astype(f32)
                k = _tiles(np.trunc(((t - lo0) / d).astype(f32)).astype(np.int64)) - wlo
                lo = np.minimum.reduce([k[:, :, 0, 0], k[:, :, 0, -1], k[:, :, -1, 0], k[:, :, -1, -1]]) - 1
            # plain rows of four-byte elements (one slice): start and width in whole 16-byte granules
            for b, w in ((lo - lo % align, W), (lo - lo % 4, (W + 3) // 4 * 4)):
                assert b.min() >= 0 and b.max() <= Wg - w, (th, int(b.min()), int(b.max()), Wg, w)
                e = k - b[:, :, None, None]
                assert e.min() >= 0 and e.max() + 4 < w, (th, int(e.min()), int(e.max()), w)
