"""Batched steps against single-lattice steps, bit for bit, for every velocity set and
storage a batch takes: lists of lattices all periodic in x and y (16-bit storage: the
batched kernel's own instantiation) and lists with ghost layers among them."""
import pytest
import torch

from ssmdlbm_b200 import _lib, configs

pytestmark = pytest.mark.gpu

COPY, PER, JET = _lib.BC_PERIODIC_COPY, _lib.BC_PERIODIC, _lib.BC_JET


def _jet(shape, vs, storage, **kw):
    return configs.oil_jet(*shape, vs, tau=0.56, sigma=3e-3, mobility=0.1, w_in=0.05, storage=storage, **kw)


def _faces(shape, vs, storage, faces):
    p = configs.reference_like(*shape, vs, diam_water=6, diam_oil=6, reynolds_water=10, reynolds_oil=8, weber=5)
    p.bc_x, p.bc_y, p.bc_z = faces
    p.storage = storage
    return p


def _list(kind, vs, storage):
    periodic = [_jet((32, 32, 40), vs, storage, diam=6, noise=0.02, seed=1),
                _jet((40, 20, 33), vs, storage, diam=8, noise=0.0),
                configs.periodic_box((20, 9, 5), vs, storage=storage),  # narrower than a tile and its halo on every axis
                configs.periodic_box((67, 18, 21), vs, storage=storage)]
    if kind == "periodic":
        return periodic
    return [periodic[0], _faces((24, 40, 36), vs, storage, (COPY, JET, JET)), periodic[2],
            _faces((35, 11, 19), vs, storage, (PER, JET, PER)), _faces((34, 10, 18), vs, storage, (COPY, COPY, JET))]


def _bits(sim):
    return {k: sim.t[k].view(torch.int16 if sim.t[k].element_size() == 2 else torch.int32)
            for k in ("f", "g", "f_alt", "g_alt", "rho", "ux", "uy", "uz", "phi")}


@pytest.mark.parametrize("storage", [_lib.STORAGE_F32, _lib.STORAGE_F16, _lib.STORAGE_BF16])
@pytest.mark.parametrize("vs", [19, 27])
@pytest.mark.parametrize("kind", ["periodic", "mixed"])
def test_batched_steps_equal_single_lattice_steps(kind, vs, storage):
    from ssmdlbm_b200.batch import Sweep
    from ssmdlbm_b200.lbm import Simulation
    ps = _list(kind, vs, storage)
    sw = Sweep(ps)
    sw.init()
    sw.step(3)
    sw.run_graph(2, steps=2)
    sw.step(2, store_macros=True)
    sw.sync()
    for p, b in zip(ps, sw.sims):
        s = Simulation(p)
        s.init()
        s.step(9, store_macros=True)
        s.sync()
        one, many = _bits(s), _bits(b)
        for k in one:
            assert torch.equal(one[k], many[k]), (p.nx, p.ny, p.nz, k)
        assert b.check_status() == 0
    sw.close()


def test_batches_refuse_split_storage():
    from ssmdlbm_b200.batch import Sweep
    with pytest.raises(RuntimeError):
        Sweep([_jet((16, 16, 16), 19, _lib.STORAGE_F16_G32, diam=4)])
