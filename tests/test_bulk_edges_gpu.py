"""The bulk kernel's instantiations at the sizes where they can go wrong.

* Lattices with ghost layers in x or y (their near-ghost normals) against the
  FP32 oracle: single-cell interiors between two ghost layers' neighbours,
  tile remainders of one and two cells, every combination of face kinds.
  Tolerance as in test_parity_gpu.py (5e-6 after one step).
* Lattices periodic in x and y run an instantiation of their own: the same
  bits as the general one, which the TMA path runs.
"""
import numpy as np
import pytest
import torch

from ssmdlbm_b200 import _lib, configs
from oracle.oracle import Oracle, seeded_macros
from helpers import compare_fields, oracle_fields, sim_fields

pytestmark = pytest.mark.gpu

COPY, PER, JET = _lib.BC_PERIODIC_COPY, _lib.BC_PERIODIC, _lib.BC_JET
FACES = [(COPY, JET, JET), (COPY, COPY, JET), (COPY, PER, JET), (PER, JET, JET), (PER, COPY, PER), (COPY, JET, PER)]
SHAPES = [(6, 6, 6), (33, 9, 8), (34, 10, 7), (35, 7, 11), (66, 17, 9)]


def _params(shape, faces, vs):
    p = configs.reference_like(*shape, vs, diam_water=3, diam_oil=3, reynolds_water=10, reynolds_oil=8, weber=4)
    p.bc_x, p.bc_y, p.bc_z = faces
    return p


@pytest.mark.parametrize("vs", [19, 27])
@pytest.mark.parametrize("faces", FACES, ids=["".join("cpj"[f] for f in k) for k in FACES])
@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
def test_ghost_faces_match_oracle(shape, faces, vs):
    from ssmdlbm_b200.lbm import Simulation
    p = _params(shape, faces, vs)
    sim, o = Simulation(p), Oracle(p, 32)
    m = seeded_macros((p.nz, p.ny, p.nx), seed=7)
    sim.init_from_macros(*m)
    o.init_macros(*m)
    sim.step(1, store_macros=True)
    o.step(1)
    compare_fields(sim_fields(sim), oracle_fields(o), 5e-6)


@pytest.mark.parametrize("storage", [_lib.STORAGE_F32, _lib.STORAGE_F16, _lib.STORAGE_BF16, _lib.STORAGE_F16_G32])
@pytest.mark.parametrize("vs", [19, 27])
@pytest.mark.parametrize("shape,box", [((8, 3, 7), True), ((40, 9, 12), False), ((64, 24, 40), False), ((72, 17, 6), True)])
def test_periodic_xy_instantiation_gives_the_same_bits(shape, box, vs, storage):
    from ssmdlbm_b200.lbm import Simulation
    if box:
        p = configs.periodic_box(shape, vs, storage=storage)
    else:
        p = configs.oil_jet(*shape, vs, tau=0.56, sigma=5e-3, diam=6, noise=0.02, seed=5, storage=storage)
    m = seeded_macros((p.nz, p.ny, p.nx), seed=3)
    got = []
    for path in (_lib.PATH_GATHER, _lib.PATH_TMA):
        p.bulk_path = path
        sim = Simulation(p)
        sim.init_from_macros(*m)
        sim.step(6, store_macros=True)
        sim.sync()
        got.append({k: sim.t[k].cpu().numpy().copy() if sim.t[k].dtype.itemsize == 4 else
                    sim.t[k].view(torch.int16).cpu().numpy().copy() for k in ("f", "g", "rho", "ux", "uy", "uz", "phi")})
        assert sim.check_status() == 0
    for k in got[0]:
        assert np.array_equal(got[0][k], got[1][k]), k
