"""The backprojector's run kernel (pixels in runs along the image axis on which
the detector coordinate moves slowest; one, four, eight or sixteen slices per CTA) against
the single-pixel kernel: both compute every pixel's bin with the same
single-precision expressions and add the angles in the same order, so images are
equal bit for bit.  RAFT_BP_TUNE="2,16" selects the single-pixel kernel on plain
rows.  The list has sizes around the 32-pixel tile, angle counts around the 16-
and 32-angle stages, slices that leave one, two and three groups of four (sixteen
or eight slices per CTA need 296 CTAs: 704^2 and 1100^2), bins narrower and wider than 1,
detectors without padding (negative bins at the corners), scans over 2 pi,
backwards and with the slopes where the slope classes meet, and a scan that
changes the run axis too often for the run kernel."""
import ctypes
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.fixture
def restore_env():
    old = os.environ.pop("RAFT_BP_TUNE", None)
    yield
    os.environ.pop("RAFT_BP_TUNE", None)
    if old is not None:
        os.environ["RAFT_BP_TUNE"] = old


def _angles(kind, A):
    k = np.arange(A)
    if kind == "edges":      # slopes 0, 1/3, 1/2, 2/3, 1/sqrt(2) and around them, in every octant
        s = np.array([0, 1 / 3, 0.5, 2 / 3, np.sqrt(0.5)])
        s = np.concatenate([np.arcsin(np.clip(s + d, 0, 1)) for d in (-2e-3, -1e-4, 0, 1e-4, 2e-3)])
        a = np.concatenate([s, np.pi / 2 - s])
        return np.sort(np.concatenate([a, np.pi - a])).astype(np.float32)
    return {"pi": k * np.pi / A, "2pi": k * 2 * np.pi / A, "back": 1 - k * np.pi / A,
            "golden": (k * 2.3999632) % np.pi}[kind].astype(np.float32)


def _fbp(sino, ang, N, pad, pixel, offset, ftype, geometry, store):
    import torch
    from sscRaft.rafttypes import _ptr, libraft
    n, A = sino.shape[0], len(ang)
    pf = np.array([0, 0, 1, 0, pixel, pixel, offset], np.float32)
    pi = np.array([N, A, n, N, pad, 0, 0, ftype, 0, 0], np.int32)
    out = torch.full((n, N, N), 7.0, device="cuda")
    assert libraft.raft_fbp_device(0, _p(out), _p(sino), _ptr(ang), _ptr(pf), _ptr(pi), geometry, store, None) == 0
    return out


@pytest.mark.parametrize("N,A,n,pad,offset,pixel,kind", [
    (31, 15, 1, 2, 0.5, 1.0, "pi"), (32, 16, 2, 1, 0.0, 1.0, "pi"), (33, 17, 5, 0, 0.3, 1.0, "pi"),
    (64, 32, 4, 2, 0.0, 0.5, "2pi"), (97, 33, 1, 0, 0.0, 2.0, "back"), (129, 100, 9, 0, -1.5, 1.0, "edges"),
    (257, 100, 1, 1, 1.25, 0.7, "edges"), (300, 61, 6, 2, 1.25, 1.0, "back"), (704, 48, 8, 2, 3.5, 1.0, "pi"),
    (1100, 40, 13, 1, -2.0, 1.0, "2pi"), (601, 37, 29, 0, 0.0, 1.0, "pi"), (100, 64, 4, 2, 0.0, 1.0, "golden")])
def test_runs_equal_single_pixels(restore_env, N, A, n, pad, offset, pixel, kind):
    import torch
    ang = _angles(kind, A)
    g = torch.Generator(device="cuda").manual_seed(N)
    sino = torch.randn((n, len(ang), N), generator=g, device="cuda")
    for geometry, store in ((0, 0), (1, 1), (1, 2)):
        os.environ["RAFT_BP_TUNE"] = "2,16"
        ref = _fbp(sino, ang, N, pad, pixel, offset, 5, geometry, store)
        del os.environ["RAFT_BP_TUNE"]
        assert torch.equal(_fbp(sino, ang, N, pad, pixel, offset, 5, geometry, store), ref), (geometry, store)


@pytest.mark.parametrize("n", [1, 4, 8, 16])
def test_non_finite_bins_stay_where_they_are(restore_env, n):
    """Without a filter a bin's infinity or NaN reaches the pixels that sample it, and no other."""
    import torch
    N = 720
    ang = _angles("pi", 24)
    g = torch.Generator(device="cuda").manual_seed(3)
    sino = torch.rand((n, 24, N), generator=g, device="cuda")
    sino[:, 3, 100] = float("inf")
    sino[:, 9, 640] = float("nan")
    os.environ["RAFT_BP_TUNE"] = "2,16"
    ref = _fbp(sino, ang, N, 1, 1.0, 0.0, 0, 0, 0)
    del os.environ["RAFT_BP_TUNE"]
    out = _fbp(sino, ang, N, 1, 1.0, 0.0, 0, 0, 0)
    assert not torch.isfinite(ref).all() and torch.isfinite(ref).float().mean() > 0.9
    assert torch.equal(torch.nan_to_num(out, 123.0, 456.0, -456.0), torch.nan_to_num(ref, 123.0, 456.0, -456.0))


@pytest.mark.parametrize("kind", [0, 1])
def test_em_slices_alone_equal_the_batch(kind):
    """EM on one slice (plain rows, planar projector), on three (one group of four,
    interleaved projector) and on nine slices of 600^2 (eight slices per CTA and a
    last one): a slice's result does not depend on its batch."""
    import torch
    from sscRaft.rafttypes import _ptr, libraft
    N, A, n, iters = 600, 40, 9, 2
    ang = _angles("pi", A)
    g = torch.Generator(device="cuda").manual_seed(5)
    data = (0.2 + 0.8 * torch.rand((n, A, N), generator=g, device="cuda")).contiguous()
    flat = torch.ones((n, N), device="cuda")

    def run(k0, k1):
        obj = torch.ones((k1 - k0, N, N), device="cuda")
        d, f = data[k0:k1].contiguous(), flat[k0:k1].contiguous()
        assert libraft.raft_em_device(kind, 0, _p(obj), _p(d), _p(f) if kind == 0 else None, _ptr(ang), N, A,
                                      k1 - k0, iters, None, 1, None) == 0
        return obj

    whole = run(0, n)
    for k0, k1 in ((0, 1), (2, 5), (8, 9)):
        assert torch.equal(run(k0, k1), whole[k0:k1]), (k0, k1)
