"""A bounded wait that runs out is an error of the call, not a wrong result.

AEROFLUX_MARCH_POLLS=0 lets every wait of the marching pair give up at once;
the kernel records it and runs to its end."""
import numpy as np
import pytest

from aeroflux_gb300 import AF_PRECISION_MIXED, AerofluxError, Config, New
from aeroflux_gb300.batch import Batch
from tests.helpers import same_bits

pytestmark = pytest.mark.gpu


def config(**kw):
    return Config(NX=64, NY=32, NZ=24, H=1.0 / 64, DT=0.004, Viscosity=1e-4, **kw)


MIXED = dict(Precision=AF_PRECISION_MIXED, DivTol=1e-10)


def mixed():
    return New(config(**MIXED))


def multigrid():
    e = New(config())
    e.EnableMultigridSolver()
    return e


@pytest.mark.parametrize("make", [mixed, multigrid])
@pytest.mark.parametrize("call", ["Step", "project"])
def test_a_marching_pair_that_gives_up_fails_the_call(make, call, monkeypatch):
    monkeypatch.setenv("AEROFLUX_PAIR_VARIANT", "3")
    monkeypatch.setenv("AEROFLUX_MARCH_POLLS", "0")
    e = make()
    e.SeedDevice(1.0, 0.05, 42, 0)
    e.applyVelocityBC()
    with pytest.raises(AerofluxError, match="gave up"):
        getattr(e, call)()
    e.applyVelocityBC()  # the record is that call's alone
    e.Close()
    # Later engines are not touched by it.
    monkeypatch.delenv("AEROFLUX_MARCH_POLLS")
    got = []
    for _ in range(2):
        e = make()
        e.SeedDevice(1.0, 0.05, 42, 0)
        e.applyVelocityBC()
        getattr(e, call)()
        got.append(e.download("U"))
        e.Close()
    assert np.isfinite(got[0]).all() and same_bits(got[0], got[1]).all()


def test_a_batch_whose_marching_pairs_give_up_reports_it(monkeypatch):
    monkeypatch.setenv("AEROFLUX_PAIR_VARIANT", "3")
    monkeypatch.setenv("AEROFLUX_MARCH_POLLS", "0")
    b = Batch(2)
    for k in range(2):
        b.seed(b.assign(config(**MIXED)), 1.0, 0.05, 42, k)
    b.apply_velocity_bc()
    with pytest.raises(AerofluxError, match="gave up"):
        b.step(2)
    b.close()
