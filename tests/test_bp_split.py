"""CPU check of the rule that shares a launch's slices out between the backprojector's
kernels (raft_bp_split)."""
import os

import numpy as np
import pytest

F32 = (1, 1)     # linear interpolation, FP32


@pytest.fixture(autouse=True)
def unforced():
    old = os.environ.pop("RAFT_BP_TUNE", None)
    yield
    os.environ.pop("RAFT_BP_TUNE", None)
    if old is not None:
        os.environ["RAFT_BP_TUNE"] = old


def _split(N, A, n, geometry=0, store=0, pixel=(1.0, 1.0), angles=None):
    from sscRaft.rafttypes import _ptr, libraft
    ang = (np.arange(A) * (np.pi / A)).astype(np.float32) if angles is None else angles.astype(np.float32)
    pf = np.array([0, 0, 1, 0, pixel[0], pixel[1], 0], np.float32)
    pi = np.array([N, A, n, N, 0, 0, 0, 1 if geometry == 2 else 7, 1 if geometry == 2 else 0, 0], np.int32)
    out = np.zeros(5, np.int32)
    assert libraft.raft_bp_split(_ptr(pf), _ptr(pi), _ptr(ang), geometry, store, n, _ptr(out)) == 0
    return [int(v) for v in out]


@pytest.mark.parametrize("geometry,store", [(0, 0), F32, (1, 2), (2, 0)])
def test_every_slice_is_taken_once_and_by_a_form_that_exists(geometry, store):
    seen = set()
    for N in (64, 200, 301, 512, 700, 1024, 2048):
        for A in (30, 47, 48, 100, 360, 1800):
            for n in (1, 2, 3, 4, 5, 8, 9, 11, 16, 17, 28, 32, 64):
                g16, g8, g4, single, one = s = _split(N, A, n, geometry, store)
                assert min(s) >= 0 and g16 % 4 == 0 and g8 % 2 == 0
                if one:
                    assert n == 1 and (geometry, store) != F32 and s[:4] == [0, 0, 0, 0]
                else:
                    assert g16 + g8 + g4 + single == -(-n // 4)
                if geometry == 1:
                    assert g16 == 0
                if (geometry, store) == F32:     # its interleaved single floats are the run kernel's alone
                    assert not (single and (g16 or g8 or g4))
                if A < 48:
                    assert s == [0, 0, 0, -(-n // 4), 0]
                seen |= {k for k, v in zip(("g16", "g8", "g4", "single", "one"), s) if v}
    assert seen >= {"g8", "g4", "single"} | (set() if (geometry, store) == F32 else {"one"}) | \
        ({"g16"} if geometry != 1 else set())


@pytest.mark.parametrize("geometry,store,N,A,n,single,run", [
    (0, 0, 700, 120, 8, 121, 148), (0, 0, 384, 60, 2, 37, 46), (0, 0, 200, 60, 8, 38, 46), (0, 0, 700, 60, 1, 50, 58),
    (1, 1, 200, 60, 1, 33, 49), (1, 1, 700, 60, 16, 187, 233), (1, 1, 1501, 60, 8, 435, 514)])
def test_scans_over_two_pi_count_their_turns(geometry, store, N, A, n, single, run):
    """Few angles over 2 pi (four changes of the run axis instead of two): whole passes
    measured with the single-pixel and the run kernel (us)."""
    assert single < run
    s = _split(N, A, n, geometry, store, angles=np.arange(A) * (2 * np.pi / A))
    assert s == [0, 0, 0, -(-n // 4), 0], s


def test_where_the_run_kernel_does_not_apply():
    k = np.arange(300)
    assert _split(512, 300, 8, angles=(k * 2.3999632) % np.pi) == [0, 0, 0, 2, 0]      # turns too often
    assert _split(512, 300, 8, pixel=(1.0, 0.5)) == [0, 0, 0, 2, 0]                    # pixels unlike bins
    assert _split(512, 300, 8)[3] == 0


@pytest.mark.parametrize("env,want", [("2,16", [0, 0, 0, 5, 0]), ("4,8", [0, 0, 0, 5, 0]), ("run,4", [0, 0, 5, 0, 0]),
                                      ("run,8", [0, 4, 1, 0, 0]), ("run,16", [4, 0, 1, 0, 0])])
def test_forced(env, want):
    os.environ["RAFT_BP_TUNE"] = env
    assert _split(100, 20, 18) == want


# Measured backprojector times on a B200 (us): single-pixel kernel, then the run kernel
# with 4, 8 and 16 slices per thread over all slices (None: no such form)
MEASURED = [
    # geometry, store, N, angles, slices, single, by 4, by 8, by 16, one slice
    (0, 0, 512, 96, 1, 33, 33, None, None, 25),
    (0, 0, 512, 360, 1, 105, 80, None, None, 52),
    (0, 0, 2048, 128, 1, 287, 383, None, None, 224),
    (0, 0, 2048, 360, 1, 783, 893, None, None, 512),
    (0, 0, 512, 128, 8, 54, 68, 54, None, None),
    (0, 0, 512, 720, 8, 257, 267, 201, None, None),
    (0, 0, 768, 128, 4, 54, 68, None, None, None),
    (0, 0, 768, 720, 4, 258, 267, None, None, None),
    (0, 0, 1024, 96, 4, 78, 91, None, None, None),
    (0, 0, 1024, 360, 4, 265, 240, None, None, None),
    (0, 0, 2048, 96, 4, 224, 322, None, None, None),
    (0, 0, 2048, 200, 8, 881, 1067, 873, None, None),
    (0, 0, 384, 128, 16, 54, 68, 54, 68, None),
    (0, 0, 384, 720, 16, 258, 269, 214, 248, None),
    (0, 0, 1024, 128, 16, 293, 383, 322, 318, None),
    (0, 0, 1024, 720, 16, 1557, 1661, 1326, 1301, None),
    (0, 0, 320, 256, 32, 127, None, 131, 158, None),
    (1, 1, 512, 96, 1, 43, 46, None, None, None),
    (1, 1, 512, 360, 1, 146, 121, None, None, None),
    (1, 1, 2048, 128, 1, 318, 584, None, None, None),
    (1, 1, 2048, 360, 1, 873, 1448, None, None, None),
    (1, 1, 512, 128, 8, 105, 95, 80, None, None),
    (1, 1, 512, 720, 8, 547, 424, 342, None, None),
    (1, 1, 768, 128, 4, 105, 97, None, None, None),
    (1, 1, 768, 720, 4, 545, 426, None, None, None),
    (1, 1, 1024, 96, 4, 132, 125, None, None, None),
    (1, 1, 1024, 360, 4, 465, 379, None, None, None),
    (1, 1, 2048, 96, 4, 480, 465, None, None, None),
    (1, 1, 2048, 200, 8, 1823, 1680, 1393, None, None),
    (1, 1, 384, 128, 16, 105, 97, 80, None, None),
    (1, 1, 384, 720, 16, 547, 425, 343, None, None),
    (1, 1, 1024, 128, 16, 601, 584, 490, None, None),
    (1, 1, 1024, 720, 16, 3287, 2790, 2258, None, None),
    (1, 1, 320, 256, 32, 262, None, 201, None, None),
    (1, 2, 512, 96, 1, 50, 43, None, None, 29),
    (1, 2, 512, 360, 1, 168, 119, None, None, 64),
    (1, 2, 2048, 128, 1, 461, 574, None, None, 306),
    (1, 2, 2048, 360, 1, 1285, 1415, None, None, 689),
    (1, 2, 512, 128, 8, 80, 95, 78, None, None),
    (1, 2, 512, 720, 8, 422, 414, 330, None, None),
    (1, 2, 768, 128, 4, 82, 95, None, None, None),
    (1, 2, 768, 720, 4, 422, 414, None, None, None),
    (1, 2, 1024, 96, 4, 117, 123, None, None, None),
    (1, 2, 1024, 360, 4, 414, 369, None, None, None),
    (1, 2, 2048, 96, 4, 353, 457, None, None, None),
    (1, 2, 2048, 200, 8, 1412, 1653, 1362, None, None),
    (1, 2, 384, 128, 16, 82, 95, 78, None, None),
    (1, 2, 384, 720, 16, 422, 414, 332, None, None),
    (1, 2, 1024, 128, 16, 465, 574, 486, None, None),
    (1, 2, 1024, 720, 16, 2560, 2725, 2182, None, None),
    (1, 2, 320, 256, 32, 218, None, 195, None, None),
    (2, 0, 512, 96, 1, 30, 35, None, None, 25),
    (2, 0, 512, 360, 1, 96, 84, None, None, 53),
    (2, 0, 2048, 128, 1, 282, 395, None, None, 227),
    (2, 0, 2048, 360, 1, 770, 940, None, None, 541),
    (2, 0, 512, 128, 8, 51, 68, 53, None, None),
    (2, 0, 512, 720, 8, 248, 279, 205, None, None),
    (2, 0, 768, 128, 4, 51, 70, None, None, None),
    (2, 0, 768, 720, 4, 250, 281, None, None, None),
    (2, 0, 1024, 96, 4, 76, 92, None, None, None),
    (2, 0, 1024, 360, 4, 255, 252, None, None, None),
    (2, 0, 2048, 96, 4, 220, 330, None, None, None),
    (2, 0, 2048, 200, 8, 868, 1116, 875, None, None),
    (2, 0, 384, 128, 16, 51, 70, 53, 66, None),
    (2, 0, 384, 720, 16, 248, 281, 209, 246, None),
    (2, 0, 1024, 128, 16, 287, 395, 319, 312, None),
    (2, 0, 1024, 720, 16, 1532, 1767, 1331, 1294, None),
    (2, 0, 320, 256, 32, 127, None, 131, 156, None),
]


@pytest.mark.parametrize("geometry,store,N,A,n,single,r4,r8,r16,r1", MEASURED)
def test_never_slower_than_the_single_pixel_kernel(geometry, store, N, A, n, single, r4, r8, r16, r1):
    """At measured points where the launch takes one form, the form chosen is within 8 % of
    the fastest one measured (the fit of the cost table is off by up to 4 % for 95 % of the
    launches, on either side)."""
    g16, g8, g4, s, one = _split(N, A, n, geometry, store)
    groups = -(-n // 4)
    t = r1 if one else single if s == groups else r4 if g4 == groups else r8 if g8 == groups else r16 if g16 == groups else None
    assert t is not None, "a mixed launch: not in the table"
    assert t <= 1.08 * min(x for x in (single, r4, r8, r16, r1) if x is not None), (t, single, r4, r8, r16, r1)
