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
import pytest

from loma_phd_b200 import Lomacte
from tests.helpers import case, oracle_for, rel_l2

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
