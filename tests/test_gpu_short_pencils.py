"""Grids of few y points, down to the nine that the library takes: y kernels
whose pencil is one to three chunks, so that a block needs more modes to be a
whole warp, and scans with groups that hold no chunk.  Operators, one step in
every form and with every option, and the physical export, against the FP64
oracle.

Bars, those of the operator and step parity tests: operators <= 1e-12 (relative
L2), one RK3 step <= 1e-10 per field in FP64 and <= 1e-6 in the mixed forms
(3e-6 with the variable viscosity).  Some of these coarse meshes have operators
next to singular (11 points: the condition of the Poisson problem of one mode is
3e5, and psi moves by 6e7 times a relative change of the mesh), which amplify any
rounding, the oracle's own included.  Where the oracle's result moves by more
than the bar when its mesh and state are changed by 16 times the unit roundoff of
FP64, or its state by four times that of FP32, that is the bar; the mixed forms are
not held to anything at 11 points, where it would be 1e-3.
"""
import numpy as np
import pytest

from loma_phd_b200 import Lomacte
from tests.helpers import FIELDS, case, mixing_scalar, oracle_for, rel_l2

pytestmark = pytest.mark.gpu

PR = float(np.float32(0.7))
NY = [9, 10, 11, 13, 15, 16, 17, 18, 19]
# few modes; more than 2368, by sweeps and (LMC_YPATH=warp) by chunks
GRIDS = [(16, 16, ""), (64, 96, ""), (64, 96, "warp")]


def _moved(a, d, rng):
    return np.asarray(a) * (1.0 + d * rng.uniform(-1.0, 1.0, np.shape(a)))


def _amplification(run, y, st, d, mesh):
    """The largest relative change of a field of run(mesh, state) for a relative
    change d of the state (and of the mesh), over d."""
    rng = np.random.default_rng(1)
    a = run(y, st)
    b = run(_moved(y, d, rng) if mesh else y,
            {k: _moved(v, d, rng) if isinstance(v, np.ndarray) else v for k, v in st.items()})
    return max(rel_l2(b[k], a[k]) for k in a) / d


def _bar(run, y, st, prec, least):
    if prec == 0:
        return max(least, 16 * 2.0**-53 * _amplification(run, y, st, 1e-10, True))
    return max(least, 4 * 2.0**-24 * _amplification(run, y, st, 1e-7, False))


def _path(monkeypatch, path):
    if path:
        monkeypatch.setenv("LMC_YPATH", path)
    else:
        monkeypatch.delenv("LMC_YPATH", raising=False)


@pytest.mark.parametrize("nx,nz,path", GRIDS)
@pytest.mark.parametrize("ny", NY)
def test_operators(gpu, monkeypatch, nx, nz, path, ny):
    import torch
    _path(monkeypatch, path)
    p, y, st = case(nx=nx, nz=nz, ny=ny)
    g = Lomacte(p, y)
    o, d = oracle_for(p, y, st), 1e-10
    om = oracle_for(p, _moved(y, d, np.random.default_rng(1)), st)
    rng = np.random.default_rng(7)
    shp = p.shape
    f = rng.standard_normal(shp) + 1j * rng.standard_normal(shp)
    fin = torch.from_numpy(f.view(np.float64).copy()).cuda()
    out, out2 = torch.zeros_like(fin), torch.zeros_like(fin)
    kx = p.alp * np.arange(p.nplanes)
    kz = p.bet * np.array([k if k <= (p.mz - 1) // 2 else k - p.mz for k in range(p.mz)])
    modes = [(0, 0), (0, 1), (1, 0), (p.nplanes - 1, p.mz - 1), (3, 5), (p.nplanes // 2, 2)]
    for op in (1, 2, 3, 4):
        g.op_y(op, fin, out, out2 if op == 3 else None)
        torch.cuda.synchronize()
        a = out.cpu().numpy().view(np.complex128).reshape(shp)
        a2 = out2.cpu().numpy().view(np.complex128).reshape(shp)
        for i, k in modes:
            u, k2 = f[i, k], kx[i] ** 2 + kz[k] ** 2

            def run(q):
                if op == 1:
                    return (q.deryr(u.real) + 1j * q.deryr(u.imag),)
                if op == 2:
                    return (q.deryyr(u.real) + 1j * q.deryyr(u.imag),)
                return q.lapvdvhom(u, k2) if op == 3 else q.solvepsi(u, k2)[:1]

            for got, ref, mv in zip((a[i, k], a2[i, k]), run(o), run(om)):
                tol = max(1e-12, 16 * 2.0**-53 * rel_l2(mv, ref) / d)
                assert rel_l2(got, ref) < tol, (op, i, k, tol)
    g.close()


@pytest.mark.parametrize("full", [0, 1])
@pytest.mark.parametrize("nx,nz,path", GRIDS[:2])
@pytest.mark.parametrize("ny,prec", [(n, q) for n in NY for q in (0, 1, 2) if n != 11 or q == 0])
def test_one_step(gpu, monkeypatch, nx, nz, path, ny, prec, full):
    _path(monkeypatch, path)
    kw = dict(nx=nx, nz=nz, ny=ny, **(dict(scalar=1, visc=1, sigma=0.7) if full else {}))
    p, y, st = case(precision=prec, **kw)
    z = mixing_scalar(p, y)
    g = Lomacte(p, y)
    g.load_state(st)
    if full:
        g.load_scalar(z)
    g.step(1)
    sg, zg = g.get_state(), g.get_scalar() if full else None
    g.close()

    def run(ym, stm):
        o = oracle_for(case(**kw)[0], ym, stm)
        if full:
            o.set_scalar(z, PR)
            o.set_viscosity(0.7)
        o.step(1)
        so = o.get_state()
        return {k: so[k] for k in FIELDS + ("u00", "v00")} | ({"Z": o.get_scalar()} if full else {})

    tol = _bar(run, y, st, prec, 1e-10 if prec == 0 else 3e-6 if full else 1e-6)
    ref = run(y, st)
    for k in ref:
        got = zg if k == "Z" else sg[k]
        assert rel_l2(got, ref[k]) < tol, (k, rel_l2(got, ref[k]), tol)


@pytest.mark.parametrize("ny", [9, 11, 16])
def test_variant_2014(gpu, ny):
    p, y, st = case(nx=24, nz=24, ny=ny, variant=1)
    g = Lomacte(p, y)
    g.load_state(st)
    g.step(1)
    sg = g.get_state()
    g.close()

    def run(ym, stm):
        o = oracle_for(p, ym, stm)
        o.step(1)
        so = o.get_state()
        return {k: so[k] for k in FIELDS + ("u00", "v00")}

    tol, ref = _bar(run, y, st, 0, 1e-10), run(y, st)
    for k in ref:
        assert rel_l2(sg[k], ref[k]) < tol, (k, rel_l2(sg[k], ref[k]), tol)


@pytest.mark.parametrize("ny", [9, 12])
def test_physical_export(gpu, ny):
    p, y, st = case(nx=16, nz=16, ny=ny)
    g = Lomacte(p, y)
    g.load_state(st)
    planes = list(range(1, p.my + 1))
    dev = g.physical(planes)
    ref = oracle_for(p, y, g.get_state()).physical(planes)
    g.close()
    for q, k in enumerate(dev):
        assert rel_l2(dev[k], ref[:, q]) < 1e-10, (k, rel_l2(dev[k], ref[:, q]))
