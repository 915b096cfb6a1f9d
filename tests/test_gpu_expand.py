"""vlsg_prepare_ls (Expand of the top level set) against the oracle's Expand,
bit for bit: two cycles run as one pass, in place, and are repeated exactly
where a value defined by the first decides the second.  Bands with exact zeros
(0, 1, 2 within two cycles), bands that miss cells within their stated width,
and noisy ones reach that path; smooth bands do not.  The start widths and
the schemes' widths give every split into passes."""
import numpy as np
import pytest

from parity_cases import compare
from viennals_b200 import BoundaryConditionEnum as BC, Domain, Grid
from viennals_b200.advect import Context
from viennals_b200.domain import make_runs
from viennals_b200.geometry import sdf_levelset, sdf_levelset_2d

pytestmark = pytest.mark.gpu

INF, PER, REF = BC.INFINITE_BOUNDARY, BC.PERIODIC_BOUNDARY, BC.REFLECTIVE_BOUNDARY


def _plane(bc, n):
    """A plane through grid points: every surface value is exactly 0."""
    g = Grid(None, [bc, bc, INF], 0.5, index_min=[0, 0, -8], index_max=[n, n + 3, 8])
    hi = [g.max[d] - (1 if bc == PER else 0) for d in range(2)] + [4]
    return g, sdf_levelset(g, lambda x, y, z: z + 0 * x, [0, 0, -4], hi)


def _sphere_sdf(shift):
    return lambda x, y, z: np.sqrt((x - shift) ** 2 + y * y + z * z) - 2.5


def _sphere(half=1.0, shift=0.0):
    g = Grid(None, [INF] * 3, 0.25)
    return g, sdf_levelset(g, _sphere_sdf(shift), [-16] * 3, [16] * 3, half_width=half)


def _thinned_sphere(seed):
    """A sphere's band of width 4 without two thirds of the cells that no sign
    change needs (the runs rebuilt for the points that are left)."""
    shift = 0.07
    g, dom = _sphere(2.0, shift)
    rng = np.random.default_rng(seed)
    keep = (np.abs(dom.values) <= 0.9) | (rng.random(dom.n_points) < 1 / 3)
    sdf = _sphere_sdf(shift)
    rs, sg = make_runs(dom.idx[keep], lambda x, y, z: np.where(
        sdf(x * 0.25, y * 0.25, z * 0.25) < 0, -1, 1), [-17] * 3, [17] * 3)
    return g, Domain(g, dom.idx[keep], dom.values[keep], rs, sg, dom.width)


def _noisy(g, dom, seed):
    """Magnitudes scaled at random, some exactly 0, signs kept."""
    rng = np.random.default_rng(seed)
    v = dom.values * rng.uniform(0.2, 1.0, dom.n_points)
    v[rng.random(dom.n_points) < 0.1] = 0.0
    return g, Domain(g, dom.idx, v, dom.run_start, dom.run_sign, dom.width)


CASES = {
    "plane_periodic_16": lambda: _plane(PER, 16),
    "plane_periodic_ragged": lambda: _plane(PER, 13),
    "plane_reflective": lambda: _plane(REF, 17),
    "sphere": lambda: _sphere(1.0, 0.11),
    "sphere_centred": lambda: _sphere(1.0),
    "sphere_width_4": lambda: _sphere(2.0, 0.07),
    "sphere_thinned": lambda: _thinned_sphere(3),
    "sphere_noisy": lambda: _noisy(*_sphere(1.0), 4),
    "plane_noisy": lambda: _noisy(*_plane(PER, 16), 5),
    "circle": lambda: _circle(0.0),
    "circle_shifted": lambda: _circle(0.13),
}


def _circle(shift):
    g = Grid(None, [INF] * 2, 0.25, dim=2, index_min=[0, 0], index_max=[0, 0])
    return g, sdf_levelset_2d(g, lambda x, y: np.sqrt((x - shift) ** 2 + y * y) - 2.5, [-16] * 2,
                              [16] * 2)


@pytest.mark.parametrize("scheme,width", [(0, 3), (1, 5), (11, 7), (9, 8), (8, 9)])
@pytest.mark.parametrize("name", sorted(CASES))
def test_expand_equals_oracle(name, scheme, width):
    from oracle import oracle as O

    g, dom = CASES[name]()
    ols = O.OracleLS(g, dom)
    ols.expand(width)
    ctx = Context(0, 0)
    ctx.set_grid(g)
    ctx.set_level_set_count(1)
    ctx.upload(0, dom)
    ctx.prepare_ls(scheme)
    if g.dim == 3:
        compare([ols], ctx)
    else:
        oi, ov = ols.points(0)
        gi, gv, _ = ctx.download(0)
        assert np.array_equal(oi, gi)
        assert np.array_equal(ov.view(np.int64), gv.view(np.int64))
    ctx.close()
