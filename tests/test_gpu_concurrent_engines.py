"""Engines of different sizes on a thread each: a call's result and success do
not depend on what another engine does meanwhile (one engine is one thread's,
but the kernels and their attributes are the process's)."""
import threading

import numpy as np
import pytest

from aeroflux_gb300 import AF_PRECISION_MIXED, Config, New
from tests.helpers import same_bits

pytestmark = pytest.mark.gpu


def _in_threads(calls):
    """Runs every call on a thread of its own; the exceptions they raised."""
    gate, errors = threading.Barrier(len(calls)), []

    def body(call):
        try:
            gate.wait()
            call()
        except Exception as x:  # noqa: BLE001
            errors.append(x)

    threads = [threading.Thread(target=body, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return errors


# Pairs that run the same instantiation of the one-cluster solve (one or two
# cells a thread) with different amounts of shared memory.
@pytest.mark.parametrize("sizes", [((24, 24, 24), (6, 6, 6)), ((27, 27, 28), (26, 26, 26))])
def test_red_black_solves_of_two_sizes_at_once(sizes):
    engines, want = [], []
    for n in sizes:
        e = New(Config(NX=n[0], NY=n[1], NZ=n[2], H=1.0 / max(n), DT=0.004, Viscosity=1e-4, GaussSeidelIters=2))
        e.SeedDevice(1.0, 0.05, 42, 0)
        e.applyVelocityBC()
        e.computeDivergence()
        e.solvePressureRedBlack()
        engines.append(e)
        want.append(e.download("P"))
        assert np.abs(want[-1]).max() > 0.0

    def solves(e):
        for _ in range(10000):
            e.solvePressureRedBlack()

    assert not _in_threads([lambda e=e: solves(e) for e in engines])
    for e, p in zip(engines, want):
        assert same_bits(e.download("P"), p).all()
        e.Close()


def test_mixed_projections_of_two_sizes_at_once():
    # Each projection is captured anew; the two tails of the V-cycle take 64
    # and 2 KiB of shared memory.
    def engine(n):
        e = New(Config(NX=n, NY=n, NZ=n, H=1.0 / n, DT=0.004, Viscosity=1e-4, Precision=AF_PRECISION_MIXED, DivTol=1e-10))
        e.SeedDevice(1.0, 0.05, 42, 0)
        e.applyVelocityBC()
        return e

    def project(e):
        for _ in range(400):
            e.project()

    def fields(e):
        return np.concatenate([e.download(name) for name in ("P", "U", "V", "W")])

    want = []
    for n in (16, 4):
        e = engine(n)
        project(e)
        want.append(fields(e))
        e.Close()
    engines = [engine(n) for n in (16, 4)]
    assert not _in_threads([lambda e=e: project(e) for e in engines])
    for e, w in zip(engines, want):
        assert same_bits(fields(e), w).all()
        e.Close()
