"""Features, filter and targets of the closure at the edges of their kernels,
against the numpy oracle: axes of 4 and 6 cells, wrapped and clamped; numbers of
cells around a block of 256; fields and outputs off 8- and 16-byte boundaries.
Tolerances are those of test_features_filter_targets_match_oracle."""
import ctypes

import numpy as np
import pytest
import torch

from ssmdlbm_b200 import _lib, closure, configs
from ssmdlbm_b200._lib import check, lib
from oracle import closure_oracle as co
from oracle.oracle import seeded_macros

pytestmark = pytest.mark.gpu

COPY, PER, JET = _lib.BC_PERIODIC_COPY, _lib.BC_PERIODIC, _lib.BC_JET


def _params(nx, ny, nz, faces):
    p = configs.reference_like(nx, ny, nz, 19, diam_water=3, diam_oil=3, reynolds_water=10, reynolds_oil=8, weber=4)
    p.bc_x, p.bc_y, p.bc_z = faces
    return p


def _fields(m, shift):
    """Device copies `shift` floats off an allocation's start, and their LBMFields."""
    f, keep = _lib.LBMFields(), []
    for k, v in zip(("rho", "ux", "uy", "uz", "phi"), m):
        t = torch.zeros(v.size + shift, device="cuda")[shift:]
        t.copy_(torch.as_tensor(np.ascontiguousarray(v, np.float32)).reshape(-1))
        setattr(f, k, t.data_ptr())
        keep.append(t)
    return f, keep


def _out(n, shift):
    return torch.full((n + shift,), float("nan"), device="cuda")[shift:]


@pytest.mark.parametrize("shift", [0, 1, 2])
@pytest.mark.parametrize("faces", [(PER, PER, PER), (PER, PER, JET), (COPY, JET, JET), (COPY, COPY, PER)],
                         ids=lambda k: "".join("cpj"[f] for f in k))
@pytest.mark.parametrize("shape", [(6, 6, 6), (8, 8, 8), (16, 16, 2 * 4), (18, 10, 14), (34, 6, 12)], ids=str)
def test_filter_targets_features(shape, faces, shift):
    nx, ny, nz = shape
    p = _params(nx, ny, nz, faces)
    per = tuple(b == PER for b in faces)
    m = [np.asarray(a, np.float32) for a in seeded_macros((nz, ny, nx), seed=5)]
    f, keep = _fields(m, shift)
    L = lib()
    n, nc = nx * ny * nz, nx * ny * nz // 8
    feat = _out(12 * n, shift)
    check(L.ssmd_closure_features(ctypes.byref(p), ctypes.byref(f), feat.data_ptr(), None))
    coarse, tau, area = _out(5 * nc, shift), _out(6 * nc, shift), _out(nc, shift)
    check(L.ssmd_closure_filter(ctypes.byref(p), ctypes.byref(f), coarse.data_ptr(), tau.data_ptr(), area.data_ptr(), None))
    torch.cuda.synchronize()
    ref = co.features(*m, per, float(p.nu_water), float(p.nu_oil))
    got = feat.cpu().numpy().reshape(n, 12)
    for k in range(12):
        assert np.abs(got[:, k] - ref[:, k]).max() <= 2e-5 * max(np.abs(ref[:, k]).max(), 1e-12), k
    rc, rt, ra = co.box_filter(*m, per)
    cshape = rc[0].shape
    got_c = coarse.cpu().numpy().reshape(5, *cshape)
    got_t = tau.cpu().numpy().reshape(6, *cshape)
    for q in range(5):
        assert np.allclose(got_c[q], rc[q], rtol=1e-6, atol=1e-7), q
    for q in range(6):
        assert np.allclose(got_t[q], rt[q], rtol=1e-4, atol=1e-10), q
    assert np.allclose(area.cpu().numpy().reshape(cshape), ra, rtol=1e-5, atol=1e-7)
    if min(shape) < 12:
        return  # (test_targets_on_every_face_kind has the small ones: a coarse axis with ghost layers needs 6 cells)
    cp = _params(nx // 2, ny // 2, nz // 2, faces)
    tg, wt = _out(2 * nc, shift), _out(2 * nc, shift)
    check(L.ssmd_closure_targets(ctypes.byref(cp), coarse.data_ptr(), tau.data_ptr(), area.data_ptr(), 0.05, tg.data_ptr(),
                                 wt.data_ptr(), None))
    torch.cuda.synchronize()
    rtg, rw = co.targets(list(got_c), list(got_t), area.cpu().numpy().reshape(cshape), per, 0.05)
    tg, wt = tg.cpu().numpy().reshape(nc, 2), wt.cpu().numpy().reshape(nc, 2)
    assert np.allclose(tg[:, 0], rtg[:, 0], rtol=1e-3, atol=1e-7)
    assert np.allclose(tg[:, 1], rtg[:, 1], rtol=1e-4, atol=1e-5)
    assert np.allclose(wt, rw, rtol=1e-5, atol=1e-6)


def test_targets_on_every_face_kind():
    for faces in ((PER, PER, PER), (COPY, JET, JET), (COPY, COPY, PER)):
        nx, ny, nz = 6, 7, 9
        cp = _params(nx, ny, nz, faces)
        per = tuple(b == PER for b in faces)
        m = [np.asarray(a, np.float32) for a in seeded_macros((nz, ny, nx), seed=6)]
        rng = np.random.default_rng(0)
        n = nx * ny * nz
        tau = [rng.normal(0, 1e-5, (nz, ny, nx)).astype(np.float32) for _ in range(6)]
        area = rng.uniform(0, 0.2, (nz, ny, nx)).astype(np.float32)
        dev = [torch.as_tensor(np.concatenate([v.ravel() for v in k]), device="cuda") for k in (m, tau, [area])]
        tg, wt = _out(2 * n, 0), _out(2 * n, 0)
        check(lib().ssmd_closure_targets(ctypes.byref(cp), *(d.data_ptr() for d in dev), 0.05, tg.data_ptr(), wt.data_ptr(), None))
        torch.cuda.synchronize()
        rtg, rw = co.targets(m, tau, area, per, 0.05)
        assert np.allclose(tg.cpu().numpy().reshape(n, 2)[:, 0], rtg[:, 0], rtol=1e-3, atol=1e-7)
        assert np.allclose(tg.cpu().numpy().reshape(n, 2)[:, 1], rtg[:, 1], rtol=1e-4, atol=1e-5)
        assert np.allclose(wt.cpu().numpy().reshape(n, 2), rw, rtol=1e-5, atol=1e-6)
