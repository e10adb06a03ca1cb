"""KineticEnergy over every shape of rows: the value, its repeatability and
its time on short rows."""
import time

import numpy as np
import pytest

from aeroflux_gb300 import Config, New

pytestmark = pytest.mark.gpu


def engine(n, ghost=1):
    e = New(Config(NX=n[0], NY=n[1], NZ=n[2], Ghost=ghost, H=1.0 / max(n), DT=0.1 / max(n), GaussSeidelIters=1))
    e.SeedDevice(1.0, 0.3, 42, 0)
    e.applyVelocityBC()
    return e


def reference(e):
    g, cfg = e.Cfg.Ghost, e.Cfg
    u, v, w = (e.download(k).reshape(getattr(e.Mesh, k).NZ, getattr(e.Mesh, k).NY, getattr(e.Mesh, k).NX) for k in "UVW")
    z, y, x = slice(g, g + cfg.NZ), slice(g, g + cfg.NY), slice(g, g + cfg.NX)
    z1, y1, x1 = slice(g + 1, g + cfg.NZ + 1), slice(g + 1, g + cfg.NY + 1), slice(g + 1, g + cfg.NX + 1)
    cells = (0.5 * (u[z, y, x] + u[z, y, x1])) ** 2 + (0.5 * (v[z, y, x] + v[z, y1, x])) ** 2 + \
        (0.5 * (w[z, y, x] + w[z1, y, x])) ** 2
    return 0.5 * float(np.sum(cells.astype(np.longdouble))) * cfg.H ** 3


# Rows of 1, of a warp and next to it; planes of 1, 3 and 4 rows; blocks of less
# than a plane, of one and of more rows than it has; more planes than partial
# sums allow blocks of 8 rows.
@pytest.mark.parametrize("n,ghost", [((1, 1, 1), 1), ((1, 2000, 3), 1), ((7, 139, 20), 2), ((31, 40, 9), 1), ((32, 40, 9), 1),
                                     ((33, 40, 9), 1), ((5, 1, 700), 1), ((100, 1, 50), 1), ((100, 3, 50), 1), ((100, 4, 50), 2),
                                     ((1000, 2, 5), 1), ((3, 400, 300), 1), ((2, 6, 16384), 1), ((40, 20, 5000), 1)])
def test_value_and_repeatability(n, ghost):
    e = engine(n, ghost)
    ke, want = e.KineticEnergy(), reference(e)
    # At most a rounding per term of sums of up to 10^6 cells, in any order.
    assert abs(ke - want) <= 1e-12 * want
    assert all(e.KineticEnergy() == ke for _ in range(3))
    e.Close()


def test_short_rows_take_no_longer_than_long_ones():
    def us(n):
        e = engine(n)
        best = float("inf")
        for _ in range(50):
            t = time.perf_counter()
            e.KineticEnergy()
            best = min(best, time.perf_counter() - t)
        e.Close()
        return best

    # A million cells each (a row a warp: 8 and 2.5 times as long).
    long_rows = us((1000, 1000, 1))
    assert us((1, 1000, 1000)) < 2.0 * long_rows
    assert us((4, 512, 512)) < 2.0 * long_rows
