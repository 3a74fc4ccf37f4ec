"""The boundary launches' values, bit for bit.

* The regularized ghost populations of an FP32 step, from the macroscopic fields the
  bulk kernel stored, against the same formulas with every rounding written out:
  each product and sum rounds once, and in a sum of two products the first one is
  fused unless its coefficient is negative and the other's positive (a compiler's
  canonical order, which turns -c p + d q into d q - c p).
* States after 20 steps against recorded digests: a last bit at the inlet grows
  along the jet, so any change of order in the step or the boundaries shows.
"""
import hashlib

import numpy as np
import pytest
import torch

from ssmdlbm_b200 import _lib, configs

pytestmark = pytest.mark.gpu

COPY, PER, JET = _lib.BC_PERIODIC_COPY, _lib.BC_PERIODIC, _lib.BC_JET
F, L = np.float32, np.longdouble
C = np.array([(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0),
              (1, 0, 1), (-1, 0, -1), (0, 1, 1), (0, -1, -1), (1, -1, 0), (-1, 1, 0), (1, 0, -1), (-1, 0, 1), (0, 1, -1),
              (0, -1, 1), (1, 1, 1), (-1, -1, -1), (1, 1, -1), (-1, -1, 1), (1, -1, 1), (-1, 1, -1), (-1, 1, 1), (1, -1, -1)])


def _fma(a, b, c):
    return (np.asarray(a, F).astype(L) * np.asarray(b, F).astype(L) + np.asarray(c, F).astype(L)).astype(F)


def _mul(a, b):
    return _fma(a, b, F(0))


def _add(a, b):
    return _fma(a, F(1), b)


def _two(a, x, b, y):
    return _fma(b, y, _mul(a, x)) if a < 0 < b else _fma(a, x, _mul(b, y))


def _weight(vs, q):
    order = int(np.abs(C[q]).sum())
    return F((1 / 3, 1 / 18, 1 / 36)[order] if vs == 19 else (8 / 27, 2 / 27, 1 / 54, 1 / 216)[order])


def _regularized(vs, q, rho, u, p, v, omco):
    """f_eq(rho, u) + omco f_neq(p, v), p = (pxx, pyy, pzz, pxy, pxz, pyz)."""
    c, w, cs2 = C[q].astype(F), _weight(vs, q), F(1.0 / 3.0)
    u2 = _fma(u[2], u[2], _fma(u[0], u[0], _mul(u[1], u[1])))
    uu = _mul(F(1.5), u2)
    cu = _mul(F(3), _fma(c[2], u[2], _fma(c[0], u[0], _mul(c[1], u[1]))))
    b = _add(F(1), -uu) if vs == 27 else _fma(F(-1.5), u2, F(1))
    b = _fma(_mul(F(0.5), cu), cu, _add(b, cu))
    if vs == 27:
        b = _add(b, _fma(_mul(_mul(cu, cu), cu), F(1.0 / 6.0), -_mul(uu, cu)))
    feq = _fma(_mul(w, rho), b, -w)
    k = [_add(_mul(i, i), -cs2) for i in c]
    h = _fma(k[2], p[2], _two(k[0], p[0], k[1], p[1]))
    h = _fma(F(2), _fma(c[1] * c[2], p[5], _fma(c[0] * c[2], p[4], _mul(c[0] * c[1], p[3]))), h)
    if vs == 27:
        def t(first, a, i, b, pij):  # first * v_a + 2 v_b pij, either product fused
            return lambda second: _fma(_mul(F(2), v[b]), pij, _mul(first, v[a])) if second else _fma(first, v[a], _mul(_mul(F(2), v[b]), pij))
        s = _two(k[0] * c[1], t(p[0], 1, 0, 0, p[3])(True), k[0] * c[2], t(p[0], 2, 0, 0, p[4])(True))
        s = _fma(k[1] * c[0], t(p[1], 0, 1, 1, p[3])(False), s)
        s = _fma(k[1] * c[2], t(p[1], 2, 1, 1, p[5])(True), s)
        s = _fma(k[2] * c[0], t(p[2], 0, 2, 2, p[4])(False), s)
        s = _fma(k[2] * c[1], t(p[2], 1, 2, 2, p[5])(False), s)
        c6 = F(6) * c[0] * c[1] * c[2]
        m = _fma(v[2], p[3], _fma(v[0], p[5], _mul(v[1], p[4])))
        h = _add(h, _fma(c6, m, _mul(F(3), s)) if c6 > 0 else _fma(F(3), s, _mul(c6, m)))
    return _fma(omco, _mul(_mul(w, F(4.5)), h), feq)


def _macros(shape, seed):
    r = np.random.default_rng(seed)
    return [np.asarray(a, F) for a in (1 + 0.02 * (r.random(shape) - 0.5), *(0.1 * (r.random(shape) - 0.5) for _ in range(3)),
                                       r.random(shape))]


def _params(shape, vs, faces, storage=_lib.STORAGE_F32, u_water=0.05, u_oil=0.05):
    p = configs.reference_like(*shape, vs, u_water=u_water, u_oil=u_oil, diam_water=15, diam_oil=16, reynolds_water=10,
                               reynolds_oil=8, weber=4)
    p.bc_x, p.bc_y, p.bc_z = faces
    p.storage, p.noise_amp, p.seed = storage, F(0.03), 9
    return p


def _run(p, steps):
    from ssmdlbm_b200.lbm import Simulation
    s = Simulation(p)
    s.init_from_macros(*_macros((p.nz, p.ny, p.nx), 3))
    s.step(steps, store_macros=True)
    s.sync()
    return s


@pytest.mark.parametrize("vs", [19, 27])
@pytest.mark.parametrize("faces", [(COPY, JET, JET), (PER, PER, JET), (COPY, JET, PER)], ids=lambda k: "".join("cpj"[f] for f in k))
@pytest.mark.parametrize("u_in", [0.05, 0.093])
def test_ghost_populations(vs, faces, u_in):
    p = _params((37, 26, 30), vs, faces, u_water=u_in, u_oil=0.7 * u_in)
    s = _run(p, 2)
    shape = (p.nz, p.ny, p.nx)
    f = s.t["f"].view(vs, *shape).cpu().numpy()  # (an even number of steps ends in f)
    m = {k: s.field(k) for k in ("rho", "ux", "uy", "uz", "pxx", "pyy", "pzz", "pxy", "pxz", "pyz")}
    compared = 0
    for axis, face in ((1, "y"), (0, "z")):  # numpy axis of [z][y][x]; velocity component 2 - axis
        if faces[2 - axis] != JET:
            continue
        n, comp, o = shape[axis], 2 - axis, 1 - axis  # o: the face's other axis, with x
        grid = np.meshgrid(np.arange(3, shape[o] - 3), np.arange(3, p.nx - 3), indexing="ij")
        io, ix = (g.reshape(-1) for g in grid)

        def at(name, plane, j=io, i=ix):
            return m[name].take(plane, axis)[j, i]
        for side in (1, -1):  # inflow at plane 0 (directions +), outflow at plane n - 1 (directions -)
            ghost, inner = (0, 1) if side > 0 else (n - 1, n - 2)
            if side > 0:  # the inflow disc, whose cells carry phi and u of the inlet
                a, b, r2 = (p.water_cx, p.water_cz, p.water_r2) if face == "y" else (p.oil_cx, p.oil_cy, p.oil_r2)
                keep = (ix - a) ** 2 + (io - b) ** 2 < 0.9 * r2
                assert keep.sum() > 50
            else:
                keep = np.ones(ix.shape, bool)
            j, i = io[keep], ix[keep]
            omco = F(p.omco_ref if side < 0 else (p.omco_water if face == "y" else p.omco_oil))
            rho = np.ones(j.shape, F) if side > 0 else at("rho", inner, j, i)
            u = [at(k, ghost if side > 0 else inner, j, i) for k in ("ux", "uy", "uz")]
            for q in np.flatnonzero(C[:vs, comp] == side):
                fj, fi = j + C[q][2 - o], i + C[q][0]
                P = [at(k, inner, fj, fi) for k in ("pxx", "pyy", "pzz", "pxy", "pxz", "pyz")]
                v = [at(k, inner, fj, fi) for k in ("ux", "uy", "uz")]
                want = _regularized(vs, q, rho, u, P, v, omco)
                got = f[q].take(ghost, axis)[j, i]
                assert np.array_equal(got, want), (face, side, q, int((got != want).sum()), got.size)
                compared += got.size
    assert compared > 3000


# sha256 over f, g, phi and u after 20 steps
RECORDED = {
    ("crossflow", 19, 0): "61a06a5264faec026a084fbb",
    ("crossflow", 19, 1): "878e891a5cb6bff664ef0ce1",
    ("crossflow", 19, 2): "17f2e2514b4495c299464fb0",
    ("crossflow", 19, 3): "cffc4517570b4d64c62edc46",
    ("crossflow", 27, 0): "2768e3cac9b81f2454989148",
    ("crossflow", 27, 1): "62c6a6abb80b6ae54326b298",
    ("crossflow", 27, 2): "15bdeeec6c1238c1c82addb0",
    ("crossflow", 27, 3): "17ead1fd4efae6742a5b69bb",
    ("jet", 19, 0): "5474f0d481172bcf76219473",
    ("jet", 19, 1): "ce408d8abf91eab763530024",
    ("jet", 19, 2): "12aad5646cbe68517c7541ed",
    ("jet", 19, 3): "c9a6cfd05e2c4d70b0d92840",
    ("jet", 27, 0): "a76d8c31af6a30e24ec21170",
    ("jet", 27, 1): "3a422161305d9931127072eb",
    ("jet", 27, 2): "a29562754a0d459bafbd1bda",
    ("jet", 27, 3): "22a80b3882eeb29ac7cd4e94",
    ("copy jet", 19, 0): "02b0c1b0c1cbc8422af5e27d",
    ("copy jet", 19, 1): "b237f66e68f2753215375a9f",
    ("copy jet", 19, 2): "1051c06f0d075b039a741ada",
    ("copy jet", 19, 3): "08f380db08b0b5a489f0cbc2",
    ("copy jet", 27, 0): "ef88e51108f2f5099b2f8db3",
    ("copy jet", 27, 1): "f476580066e60b6160641300",
    ("copy jet", 27, 2): "5c1f78fd57a8ab3414d96891",
    ("copy jet", 27, 3): "4f8da99a9afe74b496aaaad7",
}
CASES = {"crossflow": ((37, 26, 30), (COPY, JET, JET)), "jet": ((36, 32, 48), (PER, PER, JET)), "copy jet": ((35, 33, 40), (COPY, COPY, JET))}


def _digest(s):
    h = hashlib.sha256()
    for k in ("f", "g", "phi", "ux", "uy", "uz"):
        t = s.t[k]
        h.update((t.view(torch.int16) if t.element_size() == 2 else t.view(torch.int32)).cpu().numpy().tobytes())
    return h.hexdigest()[:24]


@pytest.mark.parametrize("storage", [_lib.STORAGE_F32, _lib.STORAGE_F16, _lib.STORAGE_BF16, _lib.STORAGE_F16_G32])
@pytest.mark.parametrize("vs", [19, 27])
@pytest.mark.parametrize("case", list(CASES))
def test_states_after_20_steps_are_the_recorded_ones(case, vs, storage):
    shape, faces = CASES[case]
    s = _run(_params(shape, vs, faces, storage), 20)
    assert s.check_status() == 0
    assert _digest(s) == RECORDED[case, vs, storage]
