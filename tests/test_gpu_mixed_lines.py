"""What the packed FP32 lines of the mixed form 1 carry, field by field,
against the FP64 oracle.

psi is solved from d(rho)/dt alone, which leaves the x stage as one half of a
packed line and vanishes with the density contrast.  Bar 3e-7: an FP32
transform of a white line rounds at 0.9e-7 of it (2^-24 over sqrt(3) times
sqrt(2 log2 N) to within 20 percent), d(rho)/dt sees two of them on the way in
and two on the way out and six roundings of stored values at 0.3e-7, together
2e-7, and the solve that follows smooths.  Beside a field that is larger by the
factor f its own line alone would add 0.9e-7 f.
"""
import os

import numpy as np
import pytest

from loma_phd_b200 import Lomacte
from tests.helpers import FIELDS, case, mixing_scalar, oracle_for, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s", [1.05, 1.2, 2.0, 4.0, 8.0])
@pytest.mark.parametrize("nx,nz", [(64, 64), (32, 96)])
def test_psi_at_low_density_contrast(gpu, nx, nz, s):
    p, y, st = case(nx, nz, 65, s=s, dt=0.005, Re=200.0, precision=1)
    g = Lomacte(p, y)
    g.load_state(st)
    g.step(2)
    psi = g.get_state()["psi"]
    g.close()
    o = oracle_for(case(nx, nz, 65, s=s, dt=0.005, Re=200.0)[0], y, st)
    o.step(2)
    e = rel_l2(psi, o.get_state()["psi"])
    assert e < 3e-7, e


@pytest.mark.parametrize("nx,nz", [(768, 16), (16, 768)])
def test_phi_where_the_rounding_is_largest(gpu, nx, nz):
    """The largest errors of phi in form 1 are not random: they are what the
    rounded twiddles let through from the energetic modes to those near the cut,
    times k^3, and depend on the factors of the transforms (1152 points here).
    tests/golden/mixed_rounding.npz has phi after one step at the 300 modes and
    rows with the largest ones, from the two-pass transforms (the library of
    commit b33f533, s = 4, Re = 400, Deltat = 0.005, ny = 33).  Other factors give
    errors that have nothing to do with these, a relative difference of 1 and
    more; the same factors leave only the random part: bar 1/2."""
    gold = np.load(os.path.join(os.path.dirname(__file__), "golden", "mixed_rounding.npz"))
    w, ref = gold[f"modes_{nx}x{nz}"], gold[f"phi_{nx}x{nz}"]
    phi = {}
    for prec in (0, 1):
        p, y, st = case(nx, nz, 33, s=4.0, Re=400.0, dt=0.005, precision=prec)
        g = Lomacte(p, y)
        g.load_state(st)
        g.step(1)
        phi[prec] = g.get_state()["phi"].ravel()[w]
        g.close()
    off = np.linalg.norm(phi[1] - ref) / np.linalg.norm(ref - phi[0])
    assert off < 0.5, off


@pytest.mark.parametrize("mask", ["1", "2", "4", "5", "7"])
def test_fft64_with_other_radices(gpu, monkeypatch, mask):
    """Stages with FP64 butterflies beside stages with FP32 ones at lengths whose
    radices differ between the two (72 and 288 points in x and z): nearer to the
    FP64 oracle or as near, within the one-step bar of the mixed forms."""
    p, y, st = case(48, 192, 17, precision=1)
    monkeypatch.setenv("LMC_FFT64", mask)
    g = Lomacte(p, y)
    g.load_state(st)
    g.step(1)
    sg = g.get_state()
    g.close()
    o = oracle_for(case(48, 192, 17)[0], y, st)
    o.step(1)
    so = o.get_state()
    for k in FIELDS:
        assert rel_l2(sg[k], so[k]) < 1e-6, (k, rel_l2(sg[k], so[k]))


@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("nx,nz,full", [(256, 16, 1), (384, 16, 1), (512, 16, 1), (768, 16, 1), (1024, 16, 0), (16, 256, 1),
                                        (16, 384, 1), (16, 512, 1), (16, 768, 1), (16, 1024, 1)])
def test_long_lines(gpu, nx, nz, full, prec):
    """Every transform length from 384 to 1536 points through one step, with the
    scalar and mu = T^0.7 where the x stage has room for them.  Bars: FP64 1e-10;
    the mixed forms those of the shorter lengths (up to 192 and 384 modes), 3e-6
    and 1e-6, times the growth of what weights the rounding: k^2 in Omega_y, k^3 in
    phi (one and a half times 1.1e-4 and 2.9e-5 at 1024 modes)."""
    kw = dict(nx=nx, nz=nz, ny=17, **(dict(scalar=1, visc=1, sigma=0.7) if full else {}))
    p, y, st = case(precision=prec, **kw)
    z = mixing_scalar(p, y)
    g = Lomacte(p, y)
    g.load_state(st)
    if full:
        g.load_scalar(z)
    g.step(1)
    got = g.get_state()
    if full:
        got["Z"] = g.get_scalar()
    g.close()
    o = oracle_for(case(**kw)[0], y, st)
    if full:
        o.set_scalar(z, float(np.float32(0.7)))
        o.set_viscosity(0.7)
    o.step(1)
    ref = o.get_state()
    if full:
        ref["Z"] = o.get_scalar()
    bar = (1e-10, 3e-6, 1e-6)[prec]
    n = max(nx, nz)
    grown = {"vor": bar * (n / (n, 192, 384)[prec]) ** 2, "phi": 1.5 * (0.0, 1.1e-4, 2.9e-5)[prec] * (n / 1024) ** 3}
    for k in FIELDS + (("Z",) if full else ()):
        e = rel_l2(got[k], ref[k])
        assert e < max(bar, grown.get(k, 0.0)), (k, e)
