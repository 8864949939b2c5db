"""The projector on few slices: interleaved or planar copies of the images by a rule on
slices, angles and width.  A slice's projection has the same bits alone and in any
batch, on both sides of every limit of the rule, through the device and the host call
(whose last chunk may take another layout than the first)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _angles(A):
    return (np.arange(A) * (np.pi / A)).astype(np.float32)


@pytest.mark.parametrize("nx,ny", [(64, 64), (68, 64), (67, 66), (61, 128)])
@pytest.mark.parametrize("A", [15, 16, 47, 48, 127, 128])
def test_slices_alone_equal_batches(nx, ny, A):
    import torch
    from sscRaft.rafttypes import _ptr, libraft
    n, rays, ang = 9, 70, _angles(A)
    g = torch.Generator(device="cuda").manual_seed(nx + A)
    img = torch.rand((n, ny, nx), generator=g, device="cuda")

    def run(k0, k1):
        x = img[k0:k1].contiguous()
        out = torch.full((k1 - k0, A, rays), 7.0, device="cuda")
        assert libraft.raft_radon_device(0, _p(out), _p(x), _ptr(ang), nx, ny, rays, A, k1 - k0, 1.0, 1.0, None) == 0
        return out

    alone = torch.cat([run(k, k + 1) for k in range(n)])
    for m in (2, 3, 4, 5, 7, 8, 9):
        assert torch.equal(run(n - m, n), alone[n - m:]), m


@pytest.mark.parametrize("n", [5, 7, 11, 19])
@pytest.mark.parametrize("nx,A", [(62, 48), (64, 16), (61, 128)])
def test_host_chunks_equal_slices(n, nx, A):
    from sscRaft.rafttypes import _ptr, check_error, libraft
    ang, g = _angles(A), np.array([0], np.intc)
    img = np.random.default_rng(n).random((n, nx, nx)).astype(np.float32)

    def run(x):
        x = np.ascontiguousarray(x)
        out = np.full((len(x), A, 70), 7, np.float32)
        libraft.getRadonRTMultiGPU(_ptr(g), 1, _ptr(out), _ptr(x), _ptr(ang), nx, nx, 70, A, len(x), 1.0, 1.0)
        check_error("radon")
        return out

    whole = run(img)
    for k in range(n):
        assert np.array_equal(run(img[k:k + 1])[0], whole[k]), k
