"""BST and tEMFQ at the sizes where their real-data symmetries meet an edge: odd
grids (no row that is its own mirror image but the first), odd crop widths (a last
column alone), odd angle counts (a last projection alone), one angle, unpadded and
smallest grids.  FP64 oracle, tolerances as in test_gpu_bst.py (1e-5) and
test_gpu_temfq.py (5e-6; 2e-5 with Bluestein transforms)."""
import ctypes

import numpy as np
import pytest

from conftest import rel_l2
from helpers import fbp_params, sino_case, temfq_counts

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("N,A,pad,ftype", [(45, 31, 2, 7), (64, 33, 0, 5), (63, 20, 1, 0), (35, 9, 2, 6), (27, 2, 0, 7),
                                           (100, 45, 2, 7)])
def test_bst_sizes(oracle, N, A, pad, ftype):
    import torch
    from sscRaft.rafttypes import _ptr, libraft
    B = 9                              # one slice past the eight a regridding thread takes
    ang = np.linspace(0, np.pi, A, endpoint=False).astype(np.float32)
    sino, _ = sino_case(N, A, B, seed=N + A, angles=ang)
    pf, pi = fbp_params(N, A, B, pad=pad, ftype=ftype)
    d = torch.from_numpy(sino).cuda()
    out = torch.empty((B, N, N), device="cuda")
    assert libraft.raft_bst_device(0, _p(out), _p(d), _ptr(pf), _ptr(pi), None) == 0
    ref = oracle.bst(sino[:1], ftype, pad)
    assert rel_l2(out[:1].cpu().numpy(), ref) <= 1e-5, rel_l2(out[:1].cpu().numpy(), ref)
    one = torch.empty((1, N, N), device="cuda")
    pi[2] = 1
    assert libraft.raft_bst_device(0, _p(one), _p(d[8:].contiguous()), _ptr(pf), _ptr(pi), None) == 0
    assert torch.equal(one, out[8:])


@pytest.mark.parametrize("N,A,zpad,interp", [(64, 33, 1, 1), (48, 31, 2, 0), (32, 1, 1, 1), (30, 7, 3, 1), (44, 15, 1, 1)])
def test_temfq_sizes(oracle, N, A, zpad, interp):
    import torch
    from sscRaft.rafttypes import _ptr, libraft
    counts, flat, ang = temfq_counts(N, A, 2, 0.02, seed=N + A)
    pi = np.array([N, A, 2, N, zpad, 0, 0, 2, 2, interp, 0], np.int32)
    pf = np.array([0.02, 0.02, 0], np.float32)
    obj = torch.ones((2, N, N), device="cuda")
    c, f = torch.from_numpy(counts).cuda(), torch.from_numpy(flat).cuda()
    assert libraft.raft_temfq_device(0, _p(obj), _p(c), _p(f), _ptr(np.ascontiguousarray(ang, np.float32)), _ptr(pf),
                                     _ptr(pi), None) == 0
    ref = oracle.temfq(counts, flat, ang, zpad, interp, 2, dx=0.02)
    tol = 2e-5 if N == 44 else 5e-6
    got = obj.cpu().numpy()
    assert rel_l2(got, ref) <= tol, rel_l2(got, ref)
