"""Halo tiles of the tcgen05 convolution with 64 and 96 output channels (from 32) and
32 from 64, against the FP64 oracle on BF16 inputs (rel-L2 <= 1e-2: BF16 outputs) and
the per-tap tiles (<= 2e-3), at heights that leave a part of a 2- or 4-row tile, widths
around its 128 pixels, several images, and the split output of the data gradient.
The weight gradient's reduction over splits, whose eight warps take them in turn: one
k-block (one split) and fewer splits than warps, against the oracle (<= 1e-4, as in
test_gpu_unet_tc.py)."""
import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_unet_tc import _bf, _conv, _f64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,H,W,Cin,Co,split", [(1, 1, 128, 32, 96, 0), (2, 5, 130, 32, 96, 64), (3, 6, 257, 32, 96, 64),
                                                (1, 3, 128, 32, 64, 0), (2, 9, 200, 32, 64, 32), (1, 7, 256, 64, 32, 0)])
def test_halo_tiles(oracle, N, H, W, Cin, Co, split):
    import torch
    from sscRaft.rafttypes import libraft
    torch.manual_seed(H + W + Co)
    x = _bf(torch.randn(N, H, W, Cin, device="cuda"))
    w = _bf(torch.randn(Co, 3, 3, Cin, device="cuda") * 0.1)
    b = None if split else torch.randn(Co, device="cuda")
    relu = 0 if split else 1
    y = _conv(x, None, w, b, N, H, W, Cin, 0, Co, relu=relu, split=split)
    libraft.raft_unet_set_conv_halo(0)
    try:
        tap = _conv(x, None, w, b, N, H, W, Cin, 0, Co, relu=relu, split=split)
    finally:
        libraft.raft_unet_set_conv_halo(1)
    ref = oracle.conv3x3(_f64(x), _f64(w), _f64(b) if b is not None else np.zeros(Co), relu=bool(relu))
    assert rel_l2(_f64(y), ref) <= 1e-2, rel_l2(_f64(y), ref)
    assert rel_l2(_f64(y), _f64(tap)) <= 2e-3, rel_l2(_f64(y), _f64(tap))


@pytest.mark.parametrize("N,H,W,Cin,Co", [
    (1, 1, 64, 32, 32), (1, 24, 64, 64, 64), (1, 40, 64, 96, 32), (1, 16, 128, 32, 256),
    (9, 1, 64, 32, 32),         # columns of one row: three ring slots per k-block
    (3, 13, 128, 64, 64),       # ranges that start and end inside a column and span several
    (1, 700, 64, 1024, 128),    # long columns: the ring goes round
    (40, 37, 64, 32, 32),
])
def test_wgrad_splits(oracle, N, H, W, Cin, Co):
    import torch
    from sscRaft import warmstart as ws
    from sscRaft.rafttypes import libraft
    torch.manual_seed(H + Cin + Co)
    x = _bf(torch.randn(N, H, W, Cin, device="cuda"))
    dy = _bf(torch.randn(N, H, W, Co, device="cuda"))
    dw = torch.ones(Co, 3, 3, Cin, device="cuda")
    db = torch.zeros(Co, device="cuda")
    assert libraft.raft_unet_conv_wgrad(ws._p(dy), ws._p(x), Cin, None, 0, ws._p(dw), ws._p(db), N, H, W, Co, None) == 0
    torch.cuda.synchronize()
    assert libraft.raft_unet_conv_error() == 0
    ref = 1.0 + oracle.conv3x3_wgrad(_f64(dy), _f64(x))      # added to what dw holds
    assert rel_l2(dw.double().cpu().numpy(), ref) <= 1e-4
    assert rel_l2(db.double().cpu().numpy(), _f64(dy).sum((0, 1, 2))) <= 1e-4
