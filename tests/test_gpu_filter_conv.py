"""Padded rows of up to 2048 bins whose length has a prime factor above 7: the
nearest-sample filter runs them as a circular convolution inside a compiled
transform of at least 2 Np - 1 points (1024 .. 4096); longer, unpadded or linear
ones keep Bluestein's algorithm.

Lengths on both sides of the compiled ones and of the rule, odd and even, against
the FP64 oracle: lowpass <= 3e-6 rel-L2 on uniform noise in [1, 2], whose filtered
rows keep a fixed share of the input's norm (two FP32 transforms of M points with
an error of about 1.2e-7 sqrt(log2 M) each, times three; measured <= 9.3e-7, with
Bluestein's algorithm <= 1.4e-6), and the kernels compiled for the transform length
against the generic one, bit for bit, on planar and interleaved rows (single floats: the
nearest-sample operator has no other row format)."""
import ctypes
import os

import numpy as np
import pytest

from conftest import rel_l2
from helpers import fbp_params

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


# Np = N (1 + pad): 2 Np - 1 just below and above 1024, 1536, 2048, 3072 and 4096, and unpadded
@pytest.mark.parametrize("N,pad", [(11, 1), (251, 1), (257, 1), (383, 1), (389, 1), (341, 2), (507, 1), (517, 1),
                                   (767, 1), (779, 1), (1001, 1), (1023, 1), (1031, 1), (509, 0), (2039, 0)])
@pytest.mark.parametrize("ftype", [5, 7])
def test_lowpass_vs_oracle(oracle, N, pad, ftype):
    from sscRaft.rafttypes import check_error, libraft
    A = 3                              # an odd count: the last row is filtered alone
    sino = (1 + np.random.default_rng(N).random((2, A, N))).astype(np.float32)
    pf, pi = fbp_params(N, A, 2, pad=pad, ftype=ftype)
    out = sino.copy()
    g = np.array([0], np.intc)
    libraft.getFilterLowPassMultiGPU(g.ctypes.data, 1, out.ctypes.data, pf.ctypes.data, pi.ctypes.data)
    check_error("lowpass")
    ref = oracle.lowpass(sino, oracle.MODE_REF, ftype, pad)
    assert rel_l2(out, ref) <= 3e-6, rel_l2(out, ref)


@pytest.mark.parametrize("N,pad", [(257, 1), (251, 1), (341, 2), (1023, 1)])
@pytest.mark.parametrize("tune", [None, "2,16"])     # interleaved rows, planar rows
def test_compiled_length_equals_generic(N, pad, tune):
    import torch
    from sscRaft.rafttypes import _ptr, libraft
    A, n = 37, 5
    ang = (np.arange(A) * (np.pi / A)).astype(np.float32)
    g = torch.Generator(device="cuda").manual_seed(N)
    sino = torch.randn((n, A, N), generator=g, device="cuda")
    pf, pi = fbp_params(N, A, n, pad=pad, ftype=6, offset=1.25)
    old = os.environ.pop("RAFT_BP_TUNE", None)
    outs = []
    try:
        if tune:
            os.environ["RAFT_BP_TUNE"] = tune
        for fixed in (1, 0):
            libraft.raft_filter_set_fixed(fixed)
            out = torch.empty((n, N, N), device="cuda")
            assert libraft.raft_fbp_device(0, _p(out), _p(sino), _ptr(ang), _ptr(pf), _ptr(pi), 0, 0, None) == 0
            outs.append(out)
    finally:
        libraft.raft_filter_set_fixed(1)
        os.environ.pop("RAFT_BP_TUNE", None)
        if old is not None:
            os.environ["RAFT_BP_TUNE"] = old
    assert torch.equal(outs[0], outs[1])
