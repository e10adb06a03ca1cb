"""Projections that need no refinement pass: a fluid at rest, a tolerance the
field meets already.  Same bits as the oracle, no pass counted, and none of a
pass's launches walked."""
import time

import pytest

from aeroflux_gb300 import AF_PRECISION_MIXED, Config, New
from aeroflux_gb300.batch import Batch
from tests.helpers import FIELDS
from tests.test_gpu_mixed_bits import assert_same, make_mixed_pair, mixed_cfg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(16, 16, 16), (33, 17, 20), (48, 32, 64)])
@pytest.mark.parametrize("rest", [True, False])
def test_no_pass_is_needed(n, rest):
    e, o = make_mixed_pair(n, amp=0.0 if rest else 1.0, noise=0.0 if rest else 0.01, DivTol=1e-10 if rest else 1e4)
    for k in range(2):
        e.Step(1)
        o.step(1)
        assert e.LastProjectionStats()[0] == o.passes == 0
        assert_same(e.download, o, FIELDS, f"{n} step {k}")
    e.project()
    o.project()
    assert e.LastProjectionStats()[0] == o.passes == 0
    assert_same(e.download, o, FIELDS, f"{n} projection")
    e.Close()


def test_a_slot_at_rest_beside_one_that_needs_passes():
    b = Batch(2)
    e, o = make_mixed_pair((32, 24, 40))
    e.Close()
    s0, s1 = b.assign(mixed_cfg((48, 32, 64))), b.assign(mixed_cfg((32, 24, 40)))
    for i, name in enumerate(("U", "V", "W"), start=1):
        b.upload(s1, name, o.data(i))
    b.step(2)
    o.step(2)
    assert b.projection_stats(s0)[0] == 0 and b.projection_stats(s1)[0] == o.passes > 0
    assert_same(lambda name: b.download(s1, name), o, FIELDS, "the slot beside")
    assert all((b.download(s0, name) == 0.0).all() for name in FIELDS)
    b.close()


def test_a_step_at_rest_walks_no_pass(monkeypatch):
    # Against an engine whose projections always run two passes (of V-cycles
    # that return at once, the slot having converged): about 0.4 of its time.
    def ms(e):
        e.Step(20)
        best = float("inf")
        for _ in range(5):
            t = time.perf_counter()
            e.Step(50)
            best = min(best, time.perf_counter() - t)
        e.Close()
        return best

    cfg = Config(NX=48, NY=32, NZ=64, H=1.0 / 64, DT=0.004, Viscosity=1e-5, Precision=AF_PRECISION_MIXED, DivTol=1e-10)
    none = ms(New(cfg))
    monkeypatch.setenv("AEROFLUX_FIXED_REFINEMENT_PASSES", "2")
    assert none < 0.7 * ms(New(cfg))
