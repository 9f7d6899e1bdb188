"""Every transform length in x and in z (the radices of FFT_RADIX and the block
shapes that go with them) through one RK3 step with the passive scalar and
mu = T^0.7, all inputs and outputs of the x stage, against the FP64 oracle.

Bars, those of the step parity tests of these options: FP64 <= 1e-10 per
field and for Z; mixed form 1 <= 3e-6 up to 192 modes and form 2 <= 1e-6 up to
384: above, the FP32 rounding that k^3 weights in phi is the forms' own error
(16 x 512 .. 16 x 1024 modes: 4.9e-6 .. 1.1e-4 in form 1, 1.1e-6 .. 2.9e-5 in form
2, whatever the transforms' passes).
"""
import numpy as np
import pytest

from loma_phd_b200 import Lomacte
from tests.helpers import FIELDS, case, mixing_scalar, oracle_for, rel_l2

pytestmark = pytest.mark.gpu

PR = float(np.float32(0.7))
XS = [(16, 24), (24, 16), (32, 16), (48, 16), (64, 16), (96, 16), (128, 16), (192, 16), (256, 16), (384, 16),
      (512, 16), (768, 16)]
ZS = [(16, 24), (16, 32), (16, 48), (16, 64), (16, 96), (16, 128), (16, 192), (16, 256), (16, 384), (16, 512),
      (16, 768), (16, 1024)]


@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("nx,nz", XS + ZS[1:])
def test_one_step_every_length(gpu, nx, nz, prec):
    if prec and max(nx, nz) > (192, 384)[prec - 1]:
        pytest.skip("the mixed forms' own error at these lengths")
    kw = dict(nx=nx, nz=nz, ny=17, scalar=1, visc=1, sigma=0.7)
    p, y, st = case(precision=prec, **kw)
    z = mixing_scalar(p, y)
    g = Lomacte(p, y)
    g.load_state(st)
    g.load_scalar(z)
    g.step(1)
    sg, zg = g.get_state(), g.get_scalar()
    g.close()
    o = oracle_for(case(**kw)[0], y, st)
    o.set_scalar(z, PR)
    o.set_viscosity(0.7)
    o.step(1)
    so, zo = o.get_state(), o.get_scalar()
    tol = (1e-10, 3e-6, 1e-6)[prec]
    for k in FIELDS:
        assert rel_l2(sg[k], so[k]) < tol, (k, rel_l2(sg[k], so[k]))
    assert rel_l2(zg, zo) < tol
