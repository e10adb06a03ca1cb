"""MaxDivergence where 1/h is infinite (subnormal h) or a product overflows:
what is not a number counts for nothing, as in the reference's comparison."""
import numpy as np
import pytest

from aeroflux_gb300 import AF_PRECISION_MIXED, Config, New
from aeroflux_gb300.batch import Batch
from tests.helpers import oracle_kwargs
from oracle.oracle import OracleEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [1e-309, 5e-324, 1e-300, 1e300])
@pytest.mark.parametrize("face", [0.0, 1e-320, 1e10, 1e308, -1e308])
def test_max_divergence_at_extreme_spacings(h, face):
    cfg = Config(NX=5, NY=4, NZ=3, H=h, DT=0.004, Viscosity=0.0, GaussSeidelIters=2)
    gpu, orc = New(cfg), OracleEngine(**oracle_kwargs(cfg))
    u = np.zeros(gpu.Mesh.U.Count)
    u[gpu.Mesh.U.Index(3, 2, 2)] = face
    gpu.upload("U", u)
    orc.data(1)[:] = u
    want = orc.max_divergence()
    assert gpu.MaxDivergence() == want
    b = Batch(1)
    cfg.Precision, cfg.DivTol = AF_PRECISION_MIXED, 1e-10
    s = b.assign(cfg)
    b.upload(s, "U", u)
    assert b.max_divergence(s) == want
    b.close()
    gpu.Close()
    orc.close()
