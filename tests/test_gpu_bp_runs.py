"""The backprojector's run kernel (pixels in runs along the image axis on which
the detector coordinate moves slowest; one, four, eight or sixteen slices per thread) against
the single-pixel kernel: both compute every pixel's bin with the same
single-precision expressions and add the angles in the same order, so images are
equal bit for bit.  RAFT_BP_TUNE="2,16" selects the single-pixel kernel on plain rows,
"4,16" on interleaved ones, "run,K" the run kernel with K slices per thread;
raft_bp_split says which kernel a call takes, and is asked before each comparison.  The
list has sizes around the 32-pixel tile, angle counts around the 16- and 32-angle
stages, slices that leave one, two and three groups of four behind the wider forms,
bins narrower and wider than 1, detectors without padding (negative bins at the
corners), scans over 2 pi, backwards and with the slopes where the slope classes
meet, and a scan that changes the run axis too often for the rule to take the run
kernel."""
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


def _split(N, ang, n, pixel, geometry, store):
    """(groups by 16, by 8, by 4, single-pixel groups, one slice on plain rows)"""
    from sscRaft.rafttypes import _ptr, libraft
    pf = np.array([0, 0, 1, 0, pixel, pixel, 0], np.float32)
    pi = np.array([N, len(ang), n, N, 0, 0, 0, 1 if geometry == 2 else 5, 1 if geometry == 2 else 0, 0], np.int32)
    out = np.zeros(5, np.int32)
    assert libraft.raft_bp_split(_ptr(pf), _ptr(pi), _ptr(ang), geometry, store, n, _ptr(out)) == 0
    return tuple(int(v) for v in out)


def _forms(n, geometry, store):
    """Slices per thread that n slices can take, and the split each must give."""
    g = -(-n // 4)
    forms = {4: (0, 0, g, 0, 0), 8: (0, g // 2 * 2, g % 2, 0, 0)}
    if geometry != 1:
        forms[16] = (g // 4 * 4, g % 4 // 2 * 2, g % 2, 0, 0)
    if n == 1 and (geometry, store) != (1, 1):
        forms[1] = (0, 0, 0, 0, 1)
    return {k: v for k, v in forms.items() if k <= 4 or v[0] or v[1]}


@pytest.mark.parametrize("N,A,n,pad,offset,pixel,kind", [
    (31, 15, 1, 2, 0.5, 1.0, "pi"), (32, 16, 2, 1, 0.0, 1.0, "pi"), (33, 17, 5, 0, 0.3, 1.0, "pi"),
    (64, 32, 4, 2, 0.0, 0.5, "2pi"), (97, 33, 1, 0, 0.0, 2.0, "back"), (129, 100, 9, 0, -1.5, 1.0, "edges"),
    (257, 100, 1, 1, 1.25, 0.7, "edges"), (300, 61, 6, 2, 1.25, 1.0, "back"), (704, 48, 8, 2, 3.5, 1.0, "pi"),
    (1100, 40, 13, 1, -2.0, 1.0, "2pi"), (601, 37, 29, 0, 0.0, 1.0, "pi"), (129, 143, 17, 0, 0.0, 1.0, "edges"),
    (257, 161, 30, 1, 0.5, 0.7, "2pi")])
def test_runs_equal_single_pixels(restore_env, N, A, n, pad, offset, pixel, kind):
    import torch
    ang = _angles(kind, A)
    g = torch.Generator(device="cuda").manual_seed(N)
    sino = torch.randn((n, len(ang), N), generator=g, device="cuda")
    for geometry, store in ((0, 0), (1, 1), (1, 2)):
        os.environ["RAFT_BP_TUNE"] = "2,16"
        assert _split(N, ang, n, pixel, geometry, store) == (0, 0, 0, -(-n // 4), 0)
        ref = _fbp(sino, ang, N, pad, pixel, offset, 5, geometry, store)
        for k, split in _forms(n, geometry, store).items():
            os.environ["RAFT_BP_TUNE"] = "run,%d" % k
            assert _split(N, ang, n, pixel, geometry, store) == split
            assert torch.equal(_fbp(sino, ang, N, pad, pixel, offset, 5, geometry, store), ref), (geometry, store, k)
        del os.environ["RAFT_BP_TUNE"]
        assert torch.equal(_fbp(sino, ang, N, pad, pixel, offset, 5, geometry, store), ref), (geometry, store)


@pytest.mark.parametrize("N,A,n,kind,want", [
    (512, 360, 1, "pi", "one"), (300, 128, 4, "pi", "g4"), (512, 256, 16, "pi", "g16"), (512, 256, 28, "pi", "mixed"),
    (512, 720, 12, "pi", "mixed"), (300, 47, 4, "pi", "single"), (300, 300, 4, "golden", "single")])
def test_the_rules_choice_equals_single_pixels(restore_env, N, A, n, kind, want):
    """Without forcing, one call of every kind that the rule makes (nearest sample)."""
    import torch
    ang = _angles(kind, A)
    got = _split(N, ang, n, 1.0, 0, 0)
    assert {"one": got[4], "g4": got[2], "g16": got[0], "mixed": got[0] + got[1] > 0 and got[2] + got[3] > 0,
            "single": got == (0, 0, 0, -(-n // 4), 0)}[want], got
    g = torch.Generator(device="cuda").manual_seed(N + n)
    sino = torch.randn((n, len(ang), N), generator=g, device="cuda")
    out = _fbp(sino, ang, N, 1, 1.0, 0.25, 5, 0, 0)
    os.environ["RAFT_BP_TUNE"] = "2,16"
    assert torch.equal(_fbp(sino, ang, N, 1, 1.0, 0.25, 5, 0, 0), out)


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
    assert not torch.isfinite(ref).all() and torch.isfinite(ref).float().mean() > 0.9
    for k, split in _forms(n, 0, 0).items():
        os.environ["RAFT_BP_TUNE"] = "run,%d" % k
        assert _split(N, ang, n, 1.0, 0, 0) == split
        out = _fbp(sino, ang, N, 1, 1.0, 0.0, 0, 0, 0)
        assert torch.equal(torch.nan_to_num(out, 123.0, 456.0, -456.0), torch.nan_to_num(ref, 123.0, 456.0, -456.0)), k


def _em(kind, data, flat, ang, N, iters):
    import torch
    from sscRaft.rafttypes import _ptr, libraft
    obj = torch.ones((data.shape[0], N, N), device="cuda")
    assert libraft.raft_em_device(kind, 0, _p(obj), _p(data), _p(flat) if kind == 0 else None, _ptr(ang), N, len(ang),
                                  data.shape[0], iters, None, 1, None) == 0
    return obj


@pytest.mark.parametrize("N,A,n,kind", [(97, 33, 1, 0), (161, 100, 6, 1), (300, 143, 18, 0), (129, 64, 29, 1)])
def test_em_runs_equal_single_pixels(restore_env, N, A, n, kind):
    """EM with every form of the run kernel, with the rule's choice and on an angle
    list in golden-ratio order, against the single-pixel kernel."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(N)
    data = (0.2 + 0.8 * torch.rand((n, A, N), generator=g, device="cuda")).contiguous()
    flat = torch.ones((n, N), device="cuda")

    def same(a, b):          # steps between angles out of order are negative weights: EM overflows there
        return torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.nan_to_num(a), torch.nan_to_num(b))

    for order in ("pi", "golden"):
        ang = _angles(order, A)
        os.environ["RAFT_BP_TUNE"] = "4,16"
        assert _split(N, ang, n, 1.0, 2, 0) == (0, 0, 0, -(-n // 4), 0)
        ref = _em(kind, data, flat, ang, N, 2)
        for k, split in _forms(n, 2, 0).items():
            os.environ["RAFT_BP_TUNE"] = "run,%d" % k
            assert _split(N, ang, n, 1.0, 2, 0) == split
            assert same(_em(kind, data, flat, ang, N, 2), ref), (order, k)
        del os.environ["RAFT_BP_TUNE"]
        assert same(_em(kind, data, flat, ang, N, 2), ref), order


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
