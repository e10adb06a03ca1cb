"""Every launch shape of the marching pair, and every tile variant of the fused
pair, against the restatement bit for bit: the shapes are chosen by size or by
timing, so small grids are made to run those of large ones.

Columns of tiles: rows of 64, 128 and 256 cells and past them (16, 32 and 64 quads
a column).  Chunks of 4 to 32 planes: extents along z on both sides of 16 and 32.
Tiles of 12 to 30 rows: extents along y that leave a ragged last one."""
import pytest

from tests.test_gpu_mixed_bits import FIELDS, assert_same, make_mixed_pair

pytestmark = pytest.mark.gpu

SIZES = [(64, 45, 16), (68, 14, 33), (132, 29, 18), (260, 17, 34), (264, 31, 15), (516, 15, 17), (36, 70, 70), (8, 26, 66)]


def one_vcycle(n, monkeypatch, **env):
    for k, v in env.items():
        monkeypatch.setenv(k, str(v))
    kw = {"AEROFLUX_FIXED_REFINEMENT_PASSES": 1, "AEROFLUX_MG_VCYCLES": 1, "AEROFLUX_PAIR_VARIANT": env["AEROFLUX_PAIR_VARIANT"]}
    e, o = make_mixed_pair(n, env_kw=kw, orc_kw={"fixed_passes": 1, "vcycles": 1}, DT=0.256 / max(n))
    e.project()
    o.project()
    assert_same(e.download, o, ("P", "U", "V", "W", "Div"), f"{n} {env}")
    e.Close()


@pytest.mark.parametrize("shape", range(8))
@pytest.mark.parametrize("n", SIZES)
def test_march_shapes_bit_exact(n, shape, monkeypatch):
    one_vcycle(n, monkeypatch, AEROFLUX_PAIR_VARIANT=3, AEROFLUX_MARCH_SHAPE=shape)


@pytest.mark.parametrize("var", [0, 1, 2, 4])
@pytest.mark.parametrize("n", SIZES + [(66, 34, 18), (130, 10, 12), (22, 18, 26)])
def test_tile_variants_bit_exact(n, var, monkeypatch):
    one_vcycle(n, monkeypatch, AEROFLUX_PAIR_VARIANT=var)


@pytest.mark.parametrize("shape", [1, 4, 7])
def test_march_shapes_over_steps(shape, monkeypatch):
    monkeypatch.setenv("AEROFLUX_MARCH_SHAPE", str(shape))
    e, o = make_mixed_pair((132, 30, 36), env_kw={"AEROFLUX_PAIR_VARIANT": 3}, DT=0.001)
    for k in range(2):
        e.Step(1)
        o.step(1)
        assert e.LastProjectionStats()[0] == o.passes
        assert_same(e.download, o, FIELDS, f"shape {shape} step {k}")
    e.Close()
