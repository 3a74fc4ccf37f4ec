"""Running means in the step against the standalone update of the stored fields,
bit for bit: lattices without ghost layers, with them on one, two and three axes,
planes around a block of 256 cells, the gather and the TMA path, some arrays left out."""
import numpy as np
import pytest
import torch

from ssmdlbm_b200 import _lib, configs

pytestmark = pytest.mark.gpu

COPY, PER, JET = _lib.BC_PERIODIC_COPY, _lib.BC_PERIODIC, _lib.BC_JET


@pytest.mark.parametrize("path", [_lib.PATH_GATHER, _lib.PATH_TMA])
@pytest.mark.parametrize("faces", [(PER, PER, PER), (PER, PER, JET), (COPY, PER, PER), (COPY, JET, JET)],
                         ids=lambda k: "".join("cpj"[f] for f in k))
@pytest.mark.parametrize("shape,vs,storage", [((8, 7, 9), 19, _lib.STORAGE_F32), ((16, 17, 6), 27, _lib.STORAGE_F16),
                                              ((40, 9, 33), 27, _lib.STORAGE_F32)])
def test_fused_means_equal_standalone(shape, vs, storage, faces, path):
    from ssmdlbm_b200.lbm import Simulation
    p = configs.reference_like(*shape, vs, diam_water=3, diam_oil=3, reynolds_water=10, reynolds_oil=8, weber=4)
    p.bc_x, p.bc_y, p.bc_z = faces
    p.storage, p.bulk_path = storage, path
    names = ("avg_phi", "avg_ux", "avg_uz", "avg_uxux", "avg_uxuy", "avg_uyuz")
    sims = []
    for fused in (True, False):
        s = Simulation(p)
        s.enable_derived(names)
        s.init()
        for _ in range(5):
            s.step(1, store_macros=not fused, average=fused)
            if not fused:
                s.derived_update(_lib.DERIVED_AVERAGES)
        s.sync()
        sims.append(s)
    for k in names:
        assert torch.equal(sims[0].t[k], sims[1].t[k]), k
    if JET in faces:
        assert float(sims[0].t["avg_uz"].abs().max()) > 0
