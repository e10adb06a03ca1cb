"""Bit-level parity with the CPU oracles at the edges of the kernels' tiles.

Grids whose sizes sit on or next to a limit of a kernel's split: rows of an
odd number of cell pairs and rows longer than a warp's lanes in the
restriction and prolongation, tile columns and z chunks of the marching pair,
backtraces of exactly one cell and results next to zero in the staged sweep,
and the largest grids whose red-black solve runs in one cluster launch.  The
comparison is on bit patterns, so there is no tolerance.
"""
import numpy as np
import pytest

from aeroflux_gb300 import Config
from tests.helpers import assert_bit_identical, make_pair
from tests.test_gpu_mixed_bits import assert_same, make_mixed_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(18, 20, 24), (22, 18, 26), (66, 34, 18), (130, 10, 12), (132, 20, 10), (260, 18, 8),
                               (516, 6, 10), (1028, 4, 6), (20, 300, 4), (16, 12, 70), (28, 257, 3)])
@pytest.mark.parametrize("march", [False, True])
def test_one_vcycle_at_tile_edges(n, march):
    kw = {"AEROFLUX_FIXED_REFINEMENT_PASSES": 1, "AEROFLUX_MG_VCYCLES": 1}
    if march:
        kw["AEROFLUX_PAIR_VARIANT"] = 3
    e, o = make_mixed_pair(n, env_kw=kw,
                           orc_kw={"fixed_passes": 1, "vcycles": 1}, DT=0.256 / max(n))
    e.project()
    o.project()
    assert_same(e.download, o, ("P", "U", "V", "W", "Div"), f"{n} one V-cycle")
    e.Close()


@pytest.mark.parametrize("n,ghost", [((27, 27, 28), 1), ((32, 32, 20), 1), ((32, 32, 21), 1), ((2, 3, 3), 1),
                                     ((33, 5, 17), 2), ((2000, 1, 1), 1), ((1, 150, 130), 1), ((5, 1, 4000), 1)])
def test_red_black_solve_at_cluster_edges(n, ghost):
    nx, ny, nz = n
    cfg = Config(NX=nx, NY=ny, NZ=nz, H=1.0 / max(n), DT=0.256 / max(n), Viscosity=1e-4, Ghost=ghost, GaussSeidelIters=5)
    gpu, orc = make_pair(cfg, "tg", 1.0)
    gpu.applyVelocityBC()
    orc.apply_velocity_bc()
    gpu.project()
    orc.project()
    assert_bit_identical(gpu, orc, ["P", "U", "V", "W", "Div"], f"{n} projection")


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("nu", [0.0, 1e-4])
def test_sweep_at_backtrace_edges(axis, nu):
    # Velocities whose backtrace is 0 of either sign, exactly one cell, or its
    # neighbouring floats (dt / h = 0.5), among values whose interpolation is
    # subnormal; n is odd against the sweep's 32 x 8 x 6 tile.
    n = (37, 11, 13)
    e, o = make_mixed_pair(n, apply_bc=False, H=0.0625, Viscosity=nu)
    two = np.float32(2.0)
    values = np.array([0.0, -0.0, 2.0, -2.0, np.nextafter(two, np.float32(0)), -np.nextafter(two, np.float32(3)),
                       np.nextafter(two, np.float32(3)), 1.2e-38, -1.2e-38, 1e-40, 0.75, -1.5], np.float64)
    rng = np.random.default_rng(11 + axis)
    for i, name in enumerate(("U", "V", "W"), start=1):
        a = rng.choice(values, o.data(i).size)
        e.upload(name, a)
        o.data(i)[:] = a
    e.sweep(axis, 0.03125)
    o.sweep(axis, 0.03125)
    assert_same(e.download, o, ("U", "V", "W", "Tmp0", "Tmp1", "Tmp2"), f"axis {axis}")
    e.Close()
