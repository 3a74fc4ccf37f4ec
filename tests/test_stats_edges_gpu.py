"""Statistics kernels at the edges of their work split, against numpy and the oracle.

Reductions march columns of 32 x by 16 z planes, the phase flux visits face
planes only, droplets take 2048 cells per block: sizes one below, at and one
above those, ghost layers and periodic wraps on every axis.  Tolerances: sums of
n FP64 terms in another order, n * 2^-53 of the sum of magnitudes; counts are
exact."""
import numpy as np
import pytest

from ssmdlbm_b200 import _lib, configs
from oracle.oracle import Oracle, seeded_macros
from helpers import interior_mask

pytestmark = pytest.mark.gpu

COPY, PER, JET = _lib.BC_PERIODIC_COPY, _lib.BC_PERIODIC, _lib.BC_JET
SHAPES = [(3, 3, 3), (6, 7, 18), (31, 6, 17), (32, 9, 16), (33, 8, 19), (65, 6, 34)]  # nx, ny, nz
FACES = [(PER, PER, PER), (COPY, JET, JET), (PER, PER, JET), (COPY, COPY, PER)]


def _case(shape, faces, storage=_lib.STORAGE_F32):
    p = configs.reference_like(*shape, 19, diam_water=3, diam_oil=3, reynolds_water=10, reynolds_oil=8, weber=4)
    p.bc_x, p.bc_y, p.bc_z = faces
    p.storage = storage
    return p


def _gathered_phi(g, p):
    """phi of the next step and the flux through the fluid region's faces, FP64, from pull populations [q][z][y][x]."""
    c = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1)]
    fl = interior_mask(p)
    phi = np.zeros(fl.shape)
    flow_in = flow_out = 0.0
    for q, (x, y, z) in enumerate(c):
        phi += np.roll(g[q], (z, y, x), (0, 1, 2))
        src, dst = np.roll(fl, (z, y, x), (0, 1, 2)), np.roll(fl, (-z, -y, -x), (0, 1, 2))
        flow_in += np.roll(g[q], (z, y, x), (0, 1, 2))[fl & ~src].sum()
        flow_out += g[q][fl & ~dst].sum()
    return phi[fl].sum(), flow_in, flow_out, fl


@pytest.mark.parametrize("storage", [_lib.STORAGE_F32, _lib.STORAGE_F16])
@pytest.mark.parametrize("faces", FACES, ids=["".join("cpj"[f] for f in k) for k in FACES])
@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
def test_reductions_and_flux(shape, faces, storage):
    from ssmdlbm_b200.lbm import Simulation
    if faces != FACES[0] and min(shape) < 6:
        pytest.skip("axes with ghost layers need 6 cells")
    p = _case(shape, faces, storage)
    sim = Simulation(p)
    m = seeded_macros((p.nz, p.ny, p.nx), seed=4)
    sim.init_from_macros(*m)
    g = sim.t["g"].cpu().numpy().astype(np.float64).reshape(7, p.nz, p.ny, p.nx)
    nxt, flow_in, flow_out, fl = _gathered_phi(g, p)
    rho, ux, uy, uz, phi = (np.asarray(a, np.float32).astype(np.float64)[fl] for a in m)
    u2 = ux * ux + uy * uy + uz * uz
    st = sim.reduce()
    n = fl.sum()
    eps = n * 2.0 ** -53

    def close(a, b, size):
        assert abs(a - b) <= 2 * eps * size + 1e-300, (a, b)

    assert st["cells"] == n and st["nonfinite"] == 0
    close(st["phi_sum"], phi.sum(), np.abs(phi).sum())
    close(st["phi_sum_next"], nxt, np.abs(g).sum())
    close(st["mass"], rho.sum(), rho.sum())
    for k, u in enumerate((ux, uy, uz)):
        close(st["momentum"][k], (rho * u).sum(), np.abs(rho * u).sum())
    close(st["kinetic"], (0.5 * rho * u2).sum(), (0.5 * rho * u2).sum())
    assert abs(st["u_max"] - np.sqrt(u2.max())) <= 4 * 2.0 ** -53 * st["u_max"]
    a, b = sim.phase_flux()
    close(a, flow_in, np.abs(g).sum())
    close(b, flow_out, np.abs(g).sum())


def test_reduction_counts_nonfinite_cells():
    from ssmdlbm_b200.lbm import Simulation
    p = _case((33, 8, 19), FACES[2])
    sim = Simulation(p)
    rho, ux, uy, uz, phi = (np.array(a) for a in seeded_macros((p.nz, p.ny, p.nx), seed=4))
    ux[5, 3, 32], uy[7, 0, 0], rho[18, 7, 5] = np.inf, np.nan, np.nan  # the last one a ghost cell
    sim.init_from_macros(rho, ux, uy, uz, phi)
    st = sim.reduce(raise_unstable=False)
    bad = 0
    g = sim.t["g"].cpu().numpy().astype(np.float64).reshape(7, p.nz, p.ny, p.nx)
    c = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1)]
    with np.errstate(invalid="ignore"):
        pn = sum(np.roll(g[q], (z, y, x), (0, 1, 2)) for q, (x, y, z) in enumerate(c))
        u2 = ux.astype(np.float64) ** 2 + uy.astype(np.float64) ** 2 + uz.astype(np.float64) ** 2
    fl = interior_mask(p)
    ok = np.isfinite(rho) & np.isfinite(u2) & np.isfinite(phi) & np.isfinite(pn)
    bad = int((fl & ~ok).sum())
    assert bad >= 2 and st["nonfinite"] == bad and st["status"] == _lib.SSMD_ERR_UNSTABLE
    assert abs(st["u_max"] - np.sqrt(u2[fl & ok].max())) <= 4 * 2.0 ** -53 * st["u_max"]


@pytest.mark.parametrize("fill", ["none", "all", "noise", "slabs"])
@pytest.mark.parametrize("shape", [(3, 3, 3), (16, 16, 8), (23, 10, 9), (33, 17, 12)], ids=str)
def test_droplets_of_any_filling(shape, fill):
    """No, one, many and warp-mixed components; 2048 cells exactly, and lists longer than one read."""
    from ssmdlbm_b200.lbm import Simulation
    p = configs.periodic_box(shape, 19)
    nz, ny, nx = shape[::-1]
    rng = np.random.default_rng(1)
    phi = {"none": np.zeros((nz, ny, nx)), "all": np.ones((nz, ny, nx)),
           "noise": (rng.random((nz, ny, nx)) < 0.2) * rng.uniform(0.6, 1.0, (nz, ny, nx)),
           "slabs": (np.arange(nz) % 3 == 0)[:, None, None] * rng.uniform(0.6, 1.0, (nz, ny, nx))}[fill].astype(np.float32)
    rho, ux, uy, uz, _ = seeded_macros((nz, ny, nx), seed=2)
    sim, o = Simulation(p), Oracle(p, 32)
    sim.init_from_macros(rho, ux, uy, uz, phi)
    o.init_macros(rho, ux, uy, uz, phi)
    got, want = sim.droplets(0.5), o.droplets(0.5)
    for k in ("root", "cells", "touches_inlet"):
        assert np.array_equal(got[k], want[k]), k
    assert np.allclose(got["volume"], want["volume"], rtol=1e-12, atol=0)
    if len(want) > 1:
        with pytest.raises(_lib.SSMDError):
            sim.droplets(0.5, max_droplets=len(want) - 1)
