"""Boundaries that remap cells (mirroring walls, one-sided walls, periods that
are not whole bricks) against the oracle, bit for bit, with one and two
materials: the schemes that take their box normals once per cell, and forward
Euler runs that cross bricks between two maintenances."""
import numpy as np
import pytest

from parity_cases import compare, params, run_gpu, run_oracle
from viennals_b200 import BoundaryConditionEnum as BC, Grid
from viennals_b200.geometry import make_circle, sdf_levelset
from viennals_b200.velocity import FunctorVelocity

pytestmark = pytest.mark.gpu

INF, PER, REF = BC.INFINITE_BOUNDARY, BC.PERIODIC_BOUNDARY, BC.REFLECTIVE_BOUNDARY
POS, NEG = BC.POS_INFINITE_BOUNDARY, BC.NEG_INFINITE_BOUNDARY
D = 0.25


def _same(g, lss, v, p):
    ols, ro = run_oracle(g, lss, v, p)
    ctx, rg = run_gpu(g, lss, v, p)
    assert rg.number_of_time_steps == ro.number_of_time_steps
    assert rg.advected_time == ro.advected_time
    assert rg.current_time_step == ro.current_time_step
    assert rg.point_updates == ro.point_updates
    if g.dim == 3:
        compare(ols, ctx)
    else:
        oi, ov = ols[0].points(0)
        gi, gv, _ = ctx.download(0)
        assert np.array_equal(oi, gi) and np.array_equal(ov.view(np.int64), gv.view(np.int64))
    ctx.close()
    return rg


def _velocity(n):
    v = FunctorVelocity(n)
    v.set_rate(0, -0.4 if n > 1 else -1.0)
    if n > 1:
        v.set_rate(1, -1.0)
    v.set_linear(n - 1, 2, -0.3)
    v.set_square(n - 1, 0, 0.2, 0.1)
    return v


def _hills(bcx, nx, bcy, ny, levels):
    """A wavy surface (bottom to top: a part of it, then all of it)."""
    g = Grid(None, [bcx, bcy, INF], D, index_min=[0, 0, -40], index_max=[nx, ny, 40])
    kx, ky = [(2 if b == PER else 1) * np.pi / (n * D) for b, n in ((bcx, nx), (bcy, ny))]

    def surface(x, y, z):
        return z - 0.031 - 0.45 * np.cos(kx * x) - 0.3 * np.cos(ky * y)

    def block(x, y, z):
        return np.maximum(surface(x, y, z), 0.2 - z)

    hi = [n - (1 if b == PER else 0) for b, n in ((bcx, nx), (bcy, ny))] + [9]
    return g, [sdf_levelset(g, f, [0, 0, -9], hi, lipschitz=1.5)
               for f in ((surface,), (block, surface))[levels - 1]]


WALLS = {"reflective": (REF, 21, REF, 18), "ragged": (PER, 21, PER, 13), "mixed": (REF, 16, PER, 11)}


@pytest.mark.parametrize("levels", [1, 2])
@pytest.mark.parametrize("spatial", [7, 8])
@pytest.mark.parametrize("walls", sorted(WALLS))
def test_box_normals_at_walls(walls, spatial, levels):
    g, lss = _hills(*WALLS[walls], levels)
    r = _same(g, lss, _velocity(levels), params(spatial, 1, 0.5, cfl=0.4, max_steps=60))
    assert r.number_of_time_steps > 2


@pytest.mark.parametrize("spatial", [0, 1, 5, 7, 10])
@pytest.mark.parametrize("levels", [1, 2])
@pytest.mark.parametrize("walls", sorted(WALLS))
def test_forward_euler_across_bricks_at_walls(walls, levels, spatial):
    g, lss = _hills(*WALLS[walls], levels)
    r = _same(g, lss, _velocity(levels), params(spatial, 0, 2.2, cfl=0.45, max_steps=120))
    assert r.number_of_time_steps > 10


@pytest.mark.parametrize("bc", [REF, INF])
@pytest.mark.parametrize("spatial", [0, 1, 2, 10])
def test_forward_euler_across_bricks_2d(spatial, bc):
    g = Grid([-20, 20, -20, 20], [bc, bc], 0.5, dim=2)
    v = FunctorVelocity(1)
    v.set_rate(0, 1.0)
    v.set_linear(0, 1, 0.3)
    r = _same(g, [make_circle(g, [3.0, 0.0], 5.3)], v, params(spatial, 0, 5.0, cfl=0.45))
    assert r.number_of_time_steps > 10


@pytest.mark.parametrize("spatial,temporal", [(0, 0), (1, 1), (7, 1), (8, 0), (11, 2)])
@pytest.mark.parametrize("bcs,centre", [((POS, INF, INF), (0.6, 0.0, 0.0)),
                                        ((INF, NEG, INF), (0.0, -0.6, 0.0)),
                                        ((POS, NEG, POS), (0.6, -0.6, 0.7))])
def test_one_sided_walls(bcs, centre, spatial, temporal):
    """A sphere cut by walls at index 3 (nothing below) or -3 (nothing above)."""
    lo = [3 if b == POS else -40 for b in bcs]
    hi = [-3 if b == NEG else 40 for b in bcs]
    g = Grid(None, list(bcs), D, index_min=lo, index_max=hi)
    dom = sdf_levelset(g, lambda x, y, z: np.sqrt((x - centre[0]) ** 2 + (y - centre[1]) ** 2 +
                                                  (z - centre[2]) ** 2) - 2.37,
                       [max(v, -15) for v in lo], [min(v, 15) for v in hi])
    v = FunctorVelocity(1)
    v.set_rate(0, 1.0)
    v.set_square(0, 0, 0.4, 0.1)
    _same(g, [dom], v, params(spatial, temporal, 0.8, cfl=0.4, max_steps=60))
