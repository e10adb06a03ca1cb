"""A kernel launch that the device refuses while a Step is captured fails the
call (it ends the capture): no Step runs without it."""
import pytest

from aeroflux_gb300 import AerofluxError, Config
from aeroflux_gb300 import _lib as L
from tests.helpers import assert_bit_identical, make_pair

pytestmark = pytest.mark.gpu


def test_a_step_whose_launches_are_refused_is_an_error():
    # The FP64 sweeps take three grid layers a plane of faces, of which a
    # launch holds 65535: a column of 22000 cells is past that.  A Step either
    # is the oracle's or says that it failed.
    gpu, orc = make_pair(Config(NX=4, NY=3, NZ=22000, H=0.25, DT=0.004, Viscosity=1e-4, GaussSeidelIters=2))
    try:
        gpu.Step(1)
    except AerofluxError:
        # The call after a refused one may report what that one recorded.
        L.lib().af_apply_velocity_bc(gpu._h)
    else:
        orc.step(1)
        assert_bit_identical(gpu, orc, ["U", "V", "W", "P"], "column of 22000 cells")
    gpu.Close()
