"""The training kernel over several tiles per CTA against the oracle, and a training
step with row indices out of range."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from ssmdlbm_b200 import closure
from ssmdlbm_b200._lib import check, lib
from oracle import closure_oracle as co
from test_closure_gpu import _dev, _net

pytestmark = pytest.mark.gpu


def _data(n, seed):
    rng = np.random.default_rng(seed)
    feat = rng.normal(0, 1.5, (n, co.IN)).astype(np.float32)
    tgt = np.stack([rng.uniform(0, 0.02, n), rng.uniform(0.5, 2, n)], 1).astype(np.float32)
    return feat, tgt, rng.uniform(0.1, 1.0, (n, 2)).astype(np.float32)


@pytest.mark.parametrize("how", ["gradient", "gradient with atomics", "training step"])
def test_gradient_over_several_tiles_matches_oracle(how):
    """Three tiles per CTA of 148 and a ragged fourth; the training step reads the rows
    through a permutation.  Tolerances of the one-tile test: a row's products carry bf16
    roundings of 2^-9, and both the sum and its error grow with the rows alike."""
    n = 128 * 148 * 3 + 5
    net = _net(6)
    feat, tgt, w = _data(n, 11)
    l_ref, g_ref = co.loss_and_grad(net, feat, tgt, w)
    k = closure.Network(0)
    k.net.copy_(_dev(net))
    perm = np.random.default_rng(3).permutation(n)
    st = torch.cuda.current_stream().cuda_stream
    if how == "training step":
        at = np.argsort(perm)  # row i of the batch is row perm[i] of the shuffled data
        df, dt, dw = _dev(feat[at]), _dev(tgt[at]), _dev(w[at])
        idx = _dev(perm, torch.int64)
        check(lib().ssmd_mlp_train_step(k.net.data_ptr(), df.data_ptr(), dt.data_ptr(), dw.data_ptr(), n, idx.data_ptr(), n,
                                        k.grad.data_ptr(), k.loss.data_ptr(), k.m.data_ptr(), k.v.data_ptr(), 1, 1e-3, 0.9,
                                        0.999, 1e-8, None, 0.0, k.ws.data_ptr(), k.ws.numel() * 4, st))
    else:
        df, dt, dw = _dev(feat), _dev(tgt), _dev(w)
        if how == "gradient":
            k._grad(df, dt, dw, n, st)
        else:
            check(lib().ssmd_mlp_grad(k.net.data_ptr(), df.data_ptr(), dt.data_ptr(), dw.data_ptr(), n, k.grad.data_ptr(),
                                      k.loss.data_ptr(), st))
    torch.cuda.synchronize()
    g = k.grad.cpu().numpy().astype(np.float64)
    assert abs(k.loss.item() - l_ref) <= 1e-3 * l_ref
    assert np.linalg.norm(g - g_ref) <= 1e-2 * np.linalg.norm(g_ref)
    for a, b in ((co.oW1, co.oB1), (co.oB1, co.oW2), (co.oW2, co.oB2), (co.oB2, co.oW3), (co.oW3, co.oB3), (co.oB3, co.PARAMS)):
        assert np.linalg.norm(g[a:b] - g_ref[a:b]) <= 2e-2 * np.linalg.norm(g_ref[a:b]), (a, b)
    if how == "training step":
        rn, rm, rv = co.adam(net, g, np.zeros(co.PARAMS), np.zeros(co.PARAMS), 1, 1e-3)
        assert np.allclose(k.net.cpu().numpy(), rn, rtol=1e-5, atol=1e-7)
        assert np.allclose(k.m.cpu().numpy(), rm, rtol=1e-5, atol=1e-9)


# (the status word is sticky: a process of its own)
_OUT_OF_RANGE = """
import sys
sys.path[:0] = [{root!r}, {tests!r}]
import numpy as np, torch
from ssmdlbm_b200 import closure
from ssmdlbm_b200._lib import check, lib
from test_closure_gpu import _dev, _net
from test_train_rows_gpu import _data
n, batch = 500, 128 * 3 + 40
feat, tgt, w = _data(n, 2)
idx = np.random.default_rng(4).integers(0, n, batch)
bad = np.zeros(batch, bool)
bad[[0, 5, 127, 128, 300, batch - 1]] = True
used = np.where(bad, 0, idx)
a, b = closure.Network(0), closure.Network(0)
for k in (a, b):
    k.net.copy_(_dev(_net(5)))
st = torch.cuda.current_stream().cuda_stream
wb = np.where(bad[:, None], np.float32(0), w[used])
fb, tb, wd = _dev(feat[used]), _dev(tgt[used]), _dev(wb)
a._grad(fb, tb, wd, batch, st)
check(lib().ssmd_mlp_adam(a.net.data_ptr(), a.grad.data_ptr(), a.m.data_ptr(), a.v.data_ptr(), 1, 1e-3, 0.9, 0.999, 1e-8, st))
torch.cuda.synchronize()
assert a.status() == 0
sent = np.where(bad, np.where(np.arange(batch) % 2 == 0, -1, n), idx)
df, dt, dw, di = _dev(feat), _dev(tgt), _dev(w), _dev(sent, torch.int64)
check(lib().ssmd_mlp_train_step(b.net.data_ptr(), df.data_ptr(), dt.data_ptr(), dw.data_ptr(), n, di.data_ptr(), batch,
                                b.grad.data_ptr(), b.loss.data_ptr(), b.m.data_ptr(), b.v.data_ptr(), 1, 1e-3, 0.9, 0.999, 1e-8,
                                None, 0.0, b.ws.data_ptr(), b.ws.numel() * 4, st))
torch.cuda.synchronize()
assert b.status() == 2, b.status()
for x in ("grad", "loss", "net", "m", "v"):
    assert torch.equal(getattr(a, x), getattr(b, x)), x
assert float(b.grad.abs().max()) > 0
print("as expected")
"""


def test_row_indices_out_of_range_contribute_nothing_and_set_the_status():
    tests = os.path.dirname(os.path.abspath(__file__))
    code = _OUT_OF_RANGE.format(root=os.path.dirname(tests), tests=tests)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "as expected" in r.stdout, r.stdout + r.stderr
