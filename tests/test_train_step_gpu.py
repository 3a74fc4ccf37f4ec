"""ssmd_mlp_train_step (rows read through their indices, sum, Adam and average in
two launches) against the separate calls on gathered rows: the same bits."""
import numpy as np
import pytest
import torch

from ssmdlbm_b200 import _lib, closure
from ssmdlbm_b200._lib import check, lib

pytestmark = pytest.mark.gpu


def _rows(n, seed, shift=0):
    """n rows of features, targets, weights; shift: floats the features start off a 16-byte boundary."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    flat = torch.randn(12 * n + shift, device="cuda", generator=g)
    return flat[shift:].view(n, 12), torch.randn(n, 2, device="cuda", generator=g), torch.rand(n, 2, device="cuda", generator=g)


# one row, around a tile of 128, one and two tiles per CTA of 148, a ragged last tile
@pytest.mark.parametrize("batch,shift", [(1, 0), (127, 0), (128, 1), (129, 0), (128 * 148, 0), (128 * 149 + 5, 2), (50000, 0)])
@pytest.mark.parametrize("weighted,average", [(True, True), (False, False)])
def test_train_step_matches_separate_calls(batch, shift, weighted, average):
    n = 4000
    feats, targets, weights = _rows(n, batch, shift)
    if not weighted:
        weights = None
    idx = torch.randint(0, n, (batch,), device="cuda")
    L, st = lib(), torch.cuda.current_stream().cuda_stream
    P = _lib.MLP_PARAMS
    a, b = closure.Network(3), closure.Network(3)
    for k in (a, b):
        k.net[P:] = torch.tensor([0.1] * 12 + [0.7] * 12 + [0.02, 2.0, 0.01, 1.0], device="cuda")
    avg = [a.net.clone(), b.net.clone()]
    fb, tb = feats[idx].contiguous(), targets[idx].contiguous()
    wb = weights[idx].contiguous() if weighted else None
    for t in (1, 2):
        a._grad(fb, tb, wb, batch, st)
        check(L.ssmd_mlp_adam(a.net.data_ptr(), a.grad.data_ptr(), a.m.data_ptr(), a.v.data_ptr(), t, 1e-3, 0.9, 0.999, 1e-8, st))
        if average:
            check(L.ssmd_mlp_average(avg[0].data_ptr(), a.net.data_ptr(), 0.99, st))
        check(L.ssmd_mlp_train_step(b.net.data_ptr(), feats.data_ptr(), targets.data_ptr(),
                                    weights.data_ptr() if weighted else None, n, idx.data_ptr(), batch, b.grad.data_ptr(),
                                    b.loss.data_ptr(), b.m.data_ptr(), b.v.data_ptr(), t, 1e-3, 0.9, 0.999, 1e-8,
                                    avg[1].data_ptr() if average else None, 0.99, b.ws.data_ptr(), b.ws.numel() * 4, st))
    torch.cuda.synchronize()
    for x, y in ((a.grad, b.grad), (a.loss, b.loss), (a.m, b.m), (a.v, b.v), (a.net, b.net), (avg[0], avg[1])):
        assert np.array_equal(x.cpu().numpy(), y.cpu().numpy())
    assert torch.isfinite(b.grad).all() and float(b.grad.abs().max()) > 0
    assert b.status() == 0


@pytest.mark.parametrize("form", ["strided", "double rows"])
def test_train_takes_rows_the_kernel_cannot_read_in_place(form):
    """Other layouts are gathered first, as before, with the same result."""
    feats, targets, weights = _rows(3000, 5)
    nets = [closure.Network(1), closure.Network(1)]
    nets[0].train(feats, targets, weights, steps=3, batch=700, seed=2, average=0.9)
    if form == "strided":
        feats = torch.cat((feats, feats), 1)[:, :12]
    else:
        targets = torch.stack((targets, targets), 1)[:, 0]
    nets[1].train(feats, targets, weights, steps=3, batch=700, seed=2, average=0.9)
    assert nets[0].t == nets[1].t == 3
    for k in ("net", "m", "v", "grad", "loss"):
        assert torch.equal(getattr(nets[0], k), getattr(nets[1], k)), k
    with pytest.raises((TypeError, AttributeError)):
        nets[0].train(feats, targets, None, steps=1)
