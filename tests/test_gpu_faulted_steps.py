"""A call of many Steps whose first one faults: the state is that of the fault,
whatever number of Steps the call was for, and the call does not go on solving
for the rest of them."""
import time

import numpy as np
import pytest

from aeroflux_gb300 import Config, New
from aeroflux_gb300.engine import FaultError
from tests.helpers import FIELDS, same_bits

pytestmark = pytest.mark.gpu


def engine(n, gsi, poison):
    e = New(Config(NX=n, NY=n, NZ=n, H=1.0 / n, DT=0.25 / n, Viscosity=1e-5, GaussSeidelIters=gsi))
    e.SeedDevice(1.0, 0.01, 42, 0)
    e.applyVelocityBC()
    if poison:
        u = e.download("U")
        u[e.Mesh.U.Index(n // 2, n // 2, n // 2)] = np.nan
        e.upload("U", u)
    return e


# One launch a solve and a launch a colour; Steps within a chunk, a whole
# number of chunks of 8, and past one.
@pytest.mark.parametrize("n", [12, 40])
@pytest.mark.parametrize("steps", [2, 16, 25])
def test_the_state_is_that_of_the_first_fault(n, steps):
    got = []
    for count in (1, steps):
        e = engine(n, 6, True)
        with pytest.raises(FaultError) as x:
            e.Step(count)
        got.append([str(x.value)] + [e.download(name) for name in FIELDS])
        e.Close()
    assert got[0][0] == got[1][0]
    for name, a, b in zip(FIELDS, got[0][1:], got[1][1:]):
        assert same_bits(a, b).all(), name


@pytest.mark.parametrize("n", [12, 40])
@pytest.mark.parametrize("steps", [7, 8, 9, 16, 25])
def test_many_steps_in_one_call_and_in_many(n, steps):
    a, b = engine(n, 6, False), engine(n, 6, False)
    a.Step(steps)
    for _ in range(steps):
        b.Step(1)
    for name in FIELDS:
        assert same_bits(a.download(name), b.download(name)).all(), name
    a.Close()
    b.Close()


def test_a_faulted_call_does_not_solve_on():
    def ms(poison):
        e = engine(96, 60, poison)
        u = e.download("U")
        best = float("inf")
        for _ in range(3):
            e.upload("U", u)
            t = time.perf_counter()
            try:
                e.Step(60)
            except FaultError:
                pass
            best = min(best, time.perf_counter() - t)
        e.Close()
        return best

    assert ms(True) < 0.3 * ms(False)
