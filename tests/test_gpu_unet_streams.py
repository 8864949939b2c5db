"""Gradients on several streams and host threads at a time: no call's partial sums may
be another call's.  Per layer (widths that are multiples of 64: sums in a fixed order)
the results are those of a call alone, bit for bit, with the caller's workspace and
with the call's own; for whole training steps at a width that is not (atomic sums: the
order varies) two networks' gradients agree with a lone one's to FP32 summation."""
import threading

import pytest

from conftest import rel_l2
from test_gpu_unet_tc import _bf

pytestmark = pytest.mark.gpu


def _layer(seed, N, H, W, Cin, Co):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    return dict(N=N, H=H, W=W, Cin=Cin, Co=Co, x=_bf(torch.randn(N, H, W, Cin, generator=g, device="cuda")),
                y=_bf(torch.randn(N, H, W, Co, generator=g, device="cuda")),
                dy=_bf(torch.randn(N, H, W, Co, generator=g, device="cuda")))


def _grads(c, own):
    """(dpre, dw, db) of layer c on the current stream."""
    import ctypes
    import torch
    from sscRaft import warmstart as ws
    from sscRaft.rafttypes import libraft
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    dpre = torch.empty_like(c["dy"])
    dw = torch.zeros(c["Co"], 3, 3, c["Cin"], device="cuda")
    db = torch.zeros(c["Co"], device="cuda")
    n = 0 if own else libraft.raft_unet_layer_grads_work(c["Cin"], c["Co"])
    work = None if own else torch.empty(n, device="cuda")
    assert libraft.raft_unet_layer_grads(ws._p(c["y"]), ws._p(c["dy"]), ws._p(dpre), ws._p(c["x"]), c["Cin"], None, 0,
                                         ws._p(dw), ws._p(db), c["N"], c["H"], c["W"], c["Co"],
                                         None if own else ws._p(work), n, st) == 0
    return dpre, dw, db


@pytest.mark.parametrize("own", [True, False])
def test_layers_on_two_streams(own):
    import torch
    # the second layer needs more partial sums than the first, so that a shared buffer would grow under it
    layers = [_layer(1, 2, 96, 64, 32, 32), _layer(2, 1, 64, 128, 256, 128)]
    alone = [_grads(c, own) for c in layers]
    torch.cuda.synchronize()
    bad, streams = [], [torch.cuda.Stream(), torch.cuda.Stream()]

    def run(k):
        with torch.cuda.stream(streams[k]):
            outs = [(j, _grads(layers[j], own)) for i in range(40) for j in ((i + k) % 2,)]
        streams[k].synchronize()
        bad.extend(j for j, o in outs if not all(torch.equal(a, b) for a, b in zip(o, alone[j])))

    ts = [threading.Thread(target=run, args=(k,)) for k in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    assert not bad, bad


def test_a_short_workspace_is_refused():
    import torch
    from sscRaft import warmstart as ws
    from sscRaft.rafttypes import libraft
    c = _layer(3, 1, 16, 64, 32, 32)
    dpre, dw, db = torch.empty_like(c["dy"]), torch.zeros(32, 3, 3, 32, device="cuda"), torch.zeros(32, device="cuda")
    work = torch.empty(16, device="cuda")
    assert libraft.raft_unet_layer_grads(ws._p(c["y"]), ws._p(c["dy"]), ws._p(dpre), ws._p(c["x"]), 32, None, 0,
                                         ws._p(dw), ws._p(db), 1, 16, 64, 32, ws._p(work), 16, None) != 0


def test_two_networks_train_at_a_time():
    import torch
    from sscRaft.warmstart import UNet, input_scale
    g = torch.Generator(device="cuda").manual_seed(7)
    img, tgt = torch.rand((2, 104, 104), generator=g, device="cuda"), torch.rand((2, 104, 104), generator=g, device="cuda")
    sc = input_scale(img)
    lone = UNet(torch.device("cuda"), seed=3)
    lone.train_step(img, tgt, sc, 0.0)
    torch.cuda.synchronize()
    nets, streams = [UNet(torch.device("cuda"), seed=3) for _ in range(2)], [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()

    def run(k):
        with torch.cuda.stream(streams[k]):
            for _ in range(5):
                nets[k].train_step(img, tgt, sc, 0.0)
        streams[k].synchronize()

    ts = [threading.Thread(target=run, args=(k,)) for k in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    for net in nets:
        for k in lone.gb:
            # 2 x 104^2 terms in another order: at most about sqrt(21632) * 2^-24 of the sum of magnitudes
            assert rel_l2(net.gb[k].double().cpu().numpy(), lone.gb[k].double().cpu().numpy()) <= 1e-4, k
            assert rel_l2(net.gw[k].double().cpu().numpy(), lone.gw[k].double().cpu().numpy()) <= 1e-4, k
