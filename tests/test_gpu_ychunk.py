"""The chunked y kernels (lmc_ychunk.cuh) at every geometry of their dispatch
-- five or nine rows per chunk, 8, 16 or 32 modes per block -- with last
chunks of one row, of all rows and in between, and the sweeps of grids with
many modes with a last block that is not full, against the FP64 oracle.

Bars, those of the operator and step parity tests: operators <= 1e-12
(relative L2; above the 129 points those tests go to, times (ny/129)^2, as the
condition of the second-order operators grows), one RK3 step <= 1e-10 per
field (FP64) and <= 1e-6 (mixed; 3e-6 with the variable viscosity).
"""
import numpy as np
import pytest

from loma_phd_b200 import Lomacte
from tests.helpers import FIELDS, case, oracle_for, rel_l2

pytestmark = pytest.mark.gpu

# 401 rows: the operators' tables stay in global memory, in shared memory below
# (nx, nz, ny, LMC_YPATH): 5 rows x 8 modes; 9 x 32; 9 x 16; 9 x 8; sweeps (forced, short pencils)
GRIDS = [(16, 16, 31, "warp"), (16, 16, 36, "warp"), (16, 24, 65, "warp"),
         (64, 96, 64, "warp"), (64, 96, 72, "warp"), (64, 96, 73, "warp"), (64, 96, 145, "warp"),
         (64, 96, 289, "warp"), (16, 24, 401, "warp"), (16, 24, 40, "mode"), (64, 96, 28, "")]


def _path(monkeypatch, path):
    if path:
        monkeypatch.setenv("LMC_YPATH", path)
    else:  # the automatic choice: sweeps for short pencils
        monkeypatch.delenv("LMC_YPATH", raising=False)


@pytest.mark.parametrize("nx,nz,ny,path", GRIDS)
def test_operators(gpu, monkeypatch, nx, nz, ny, path):
    import torch
    _path(monkeypatch, path)
    p, y, st = case(nx=nx, nz=nz, ny=ny)
    g = Lomacte(p, y)
    o = oracle_for(p, y, st, nthreads=4)
    rng = np.random.default_rng(5)
    shp = p.shape
    f = (rng.standard_normal(shp) + 1j * rng.standard_normal(shp)) * np.exp(-(y / 6.0) ** 2)
    fin = torch.from_numpy(f.view(np.float64).copy()).cuda()
    out, out2 = torch.zeros_like(fin), torch.zeros_like(fin)
    kx = p.alp * np.arange(p.nplanes)
    kz = p.bet * np.array([k if k <= (p.mz - 1) // 2 else k - p.mz for k in range(p.mz)])
    tol = 1e-12 * max(1.0, (ny / 129.0) ** 2)
    modes = sorted({(0, 0), (0, 1), (1, 0), (p.nplanes - 1, p.mz - 1)}
                   | {(int(i), int(k)) for i, k in zip(rng.integers(0, p.nplanes, 40), rng.integers(0, p.mz, 40))})
    for op in (1, 2, 3, 4):
        g.op_y(op, fin, out, out2 if op == 3 else None)
        torch.cuda.synchronize()
        a = out.cpu().numpy().view(np.complex128).reshape(shp)
        a2 = out2.cpu().numpy().view(np.complex128).reshape(shp)
        got, ref, got2, ref2 = [], [], [], []
        for i, k in modes:
            u, k2 = f[i, k], kx[i] ** 2 + kz[k] ** 2
            got.append(a[i, k])
            if op == 1:
                ref.append(o.deryr(u.real) + 1j * o.deryr(u.imag))
            elif op == 2:
                ref.append(o.deryyr(u.real) + 1j * o.deryyr(u.imag))
            elif op == 3:
                v, dv = o.lapvdvhom(u, k2)
                ref.append(v)
                got2.append(a2[i, k])
                ref2.append(dv)
            else:
                ref.append(o.solvepsi(u, k2)[0])
        assert rel_l2(np.array(got), np.array(ref)) < tol, op
        if op == 3:
            assert rel_l2(np.array(got2), np.array(ref2)) < tol
    g.close()


@pytest.mark.parametrize("prec,tol", [(0, 1e-10), (1, 1e-6)])
@pytest.mark.parametrize("nx,nz,ny,path", [GRIDS[0], GRIDS[3], GRIDS[6], GRIDS[7], (24, 32, 300, "warp"), (64, 96, 129, "warp"),
                                          GRIDS[-2], GRIDS[-1]])
def test_one_step(gpu, monkeypatch, nx, nz, ny, path, prec, tol):
    _path(monkeypatch, path)
    p, y, st = case(nx=nx, nz=nz, ny=ny, precision=prec)
    g = Lomacte(p, y)
    g.load_state(st)
    g.step(1)
    sg = g.get_state()
    g.close()
    o = oracle_for(case(nx=nx, nz=nz, ny=ny)[0], y, st)
    o.step(1)
    so = o.get_state()
    for k in FIELDS + ("u00", "v00"):
        assert rel_l2(sg[k], so[k]) < tol, (k, rel_l2(sg[k], so[k]))


@pytest.mark.parametrize("prec,tol", [(0, 1e-10), (1, 3e-6)])
@pytest.mark.parametrize("nx,nz,ny", [(16, 16, 31), (64, 96, 129)])
def test_one_step_visc(gpu, monkeypatch, nx, nz, ny, prec, tol):
    """The strain-rate inputs from three blocks per group of modes, and from one."""
    _path(monkeypatch, "warp")
    kw = dict(nx=nx, nz=nz, ny=ny, visc=1, sigma=0.7)
    p, y, st = case(precision=prec, **kw)
    g = Lomacte(p, y)
    g.load_state(st)
    g.step(1)
    sg = g.get_state()
    g.close()
    o = oracle_for(case(**kw)[0], y, st)
    o.set_viscosity(0.7)
    o.step(1)
    so = o.get_state()
    for k in FIELDS + ("u00", "w00"):
        assert rel_l2(sg[k], so[k]) < tol, (k, rel_l2(sg[k], so[k]))
