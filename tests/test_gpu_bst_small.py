"""BST and tEMFQ on small grids: the interpolation and the row transforms run as one
kernel up to a number of grid points in all slices, as two above it.  A slice has the
same bits in a batch on either side of that number."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("N,pad,n", [(140, 1, 32), (200, 1, 16), (250, 2, 5), (300, 1, 7)])
def test_bst_slice_equals_batch(N, pad, n):
    import torch
    from sscRaft.rafttypes import _ptr, libraft
    A, S = 45, N * (1 + pad)
    assert n * S * S > 2.5e6 >= (n - 1) * S * S      # n slices take two kernels, n - 1 one
    g = torch.Generator(device="cuda").manual_seed(N)
    sino = torch.randn((n, A, N), generator=g, device="cuda")

    def run(k0, k1):
        x = sino[k0:k1].contiguous()
        out = torch.full((k1 - k0, N, N), 7.0, device="cuda")
        pi = np.array([N, A, k1 - k0, N, pad, 0, 0, 7, 0, k1 - k0], np.int32)
        pf = np.array([0, 0, 1, 0, 1, 1, 0], np.float32)
        assert libraft.raft_bst_device(0, _p(out), _p(x), _ptr(pf), _ptr(pi), None) == 0
        return out

    more, less = run(0, n), run(0, n - 1)
    assert torch.equal(more[:n - 1], less)
    for k in (0, n - 1):
        assert torch.equal(run(k, k + 1)[0], more[k])


@pytest.mark.parametrize("N,pad,n", [(250, 2, 5), (300, 1, 7), (300, 2, 4)])
def test_temfq_slice_equals_batch(N, pad, n):
    import torch
    from sscRaft.rafttypes import _ptr, libraft
    A = 40
    ang = (np.arange(A) * (np.pi / A)).astype(np.float32)
    g = torch.Generator(device="cuda").manual_seed(N)
    counts = 1e4 * (0.5 + 0.5 * torch.rand((n, A, N), generator=g, device="cuda"))
    flat = torch.full((n, N), 1e4, device="cuda")

    def run(k0, k1):
        m = k1 - k0
        obj = torch.full((m, N, N), 1e-3, device="cuda")
        c, f = counts[k0:k1].contiguous(), flat[k0:k1].contiguous()
        pi = np.array([N, A, m, N, pad, 0, 0, m, 2, 1, 0], np.int32)
        pf = np.array([2.0 / (N - 1), 2.0 / (N - 1), 0], np.float32)
        assert libraft.raft_temfq_device(0, _p(obj), _p(c), _p(f), _ptr(ang), _ptr(pf), _ptr(pi), None) == 0
        return obj

    batch = run(0, n)
    for k in (0, n - 1):
        one = run(k, k + 1)[0]
        assert torch.equal(torch.isnan(one), torch.isnan(batch[k]))
        assert torch.equal(torch.nan_to_num(one), torch.nan_to_num(batch[k]))
