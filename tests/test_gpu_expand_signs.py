"""vlsg_prepare_ls (Expand of the top level set) on bands in which undefined
cells of opposite sign lie side by side, or next to a value of the other sign
of magnitude 1 or more: cells change sign within an Expand.  Reference: every
cycle evaluates the undefined cells next to a defined one, and all undefined
cells of the 8^3 bricks at walls that remap cells, from the values before it
(lsExpand.hpp:104-157), written out densely here.  Points, values
and the signs of the undefined cells next to a defined one are equal bit for
bit, in every run."""
import numpy as np
import pytest

from viennals_b200 import BoundaryConditionEnum as BC, Domain, Grid
from viennals_b200.advect import Context
from viennals_b200.domain import make_runs

pytestmark = pytest.mark.gpu

INF, PER, REF = BC.INFINITE_BOUNDARY, BC.PERIODIC_BOUNDARY, BC.REFLECTIVE_BOUNDARY
Z0, NZ = -16, 32  # dense box in z


def _grid(bcx, nx, bcy, ny):
    return Grid(None, [bcx, bcy, INF], 0.5, index_min=[0, 0, Z0], index_max=[nx, ny, Z0 + NZ])


def _extent(g, d):
    return g.max[d] - g.min[d] + (0 if g.bc[d] == PER else 1)


def _shift(a, axis, step, bc):
    """The neighbour of every cell in direction `step` of `axis`."""
    r = np.roll(a, -step, axis)
    if bc == PER:
        return r
    edge = [slice(None)] * 3
    edge[axis] = -1 if step > 0 else 0
    inner = list(edge)
    inner[axis] = (-2 if step > 0 else 1) if bc == REF else edge[axis]
    r[tuple(edge)] = a[tuple(inner)]
    return r


def _wall_cells(g, shape):
    """Cells of the bricks at a wall that remaps cells."""
    m = np.zeros(shape, bool)
    for d in range(2):
        c = np.arange(shape[d]) // 8
        if g.bc[d] == REF or shape[d] % 8:
            m |= ((c == 0) | (c == c[-1])).reshape([-1 if k == d else 1 for k in range(3)])
    return m


def _expand(phi, g, start, width):
    """phi: dense values, +-max where undefined."""
    walls = _wall_cells(g, phi.shape)
    top = np.finfo(phi.dtype).max
    bcs = [g.bc[0], g.bc[1], None]
    moves = [(0, 1), (1, 1), (2, 1), (0, -1), (1, -1), (2, -1)]
    one = phi.dtype.type(1)
    for w in range(start + 1, width + 1):
        limit = phi.dtype.type(w) * phi.dtype.type(0.5)
        star = [_shift(phi, a, s, bcs[a]) for a, s in moves]
        defined = np.abs(phi) < top
        cand = ~defined & (walls | np.any([np.abs(n) < top for n in star], axis=0))
        up = np.min([np.minimum(n + one, top) for n in star], axis=0)
        down = np.max([np.maximum(n - one, -top) for n in star], axis=0)
        new = np.where(phi > 0, np.where(up <= limit, up, top), np.where(down >= -limit, down, -top))
        phi = np.where(cand, new, phi).astype(phi.dtype)
    return phi


def _plane(g, dtype, offset=0.5):
    """Values z + offset next to the plane, undefined elsewhere (dense)."""
    nx, ny = _extent(g, 0), _extent(g, 1)
    z = (np.arange(NZ) + Z0 + offset).astype(dtype)
    top = np.finfo(dtype).max
    line = np.where(np.abs(z) <= 0.5, z, np.where(z > 0, top, -top)).astype(dtype)
    return np.broadcast_to(line, (nx, ny, NZ)).copy()


def _undefine(phi, cells):
    top = np.finfo(phi.dtype).max
    for c in cells:
        phi[c] = np.copysign(top, phi[c])


def _pairs(xy):
    k = -Z0  # cell z = 0 (value +0.5) and z = -1 (value -0.5)
    return [(x, y, z) for x, y in xy for z in (k, k - 1)]


def _one_pair(g, dtype):
    phi = _plane(g, dtype)
    _undefine(phi, _pairs([(3, 4)]))
    return phi


def _pairs_at_faces(g, dtype):
    """Pairs on both sides of the brick faces in x, in y, and at the walls."""
    nx, ny = _extent(g, 0), _extent(g, 1)
    phi = _plane(g, dtype)
    _undefine(phi, _pairs([(7, 3), (8, 3), (2, 7), (2, 8), (0, 5), (nx - 1, 6), (5, 0), (5, ny - 1),
                           (nx - 1, ny - 1)]))
    return phi


def _patch(g, dtype):
    """A hole of 6 x 5 pairs: candidates of more than one warp's share."""
    phi = _plane(g, dtype)
    _undefine(phi, _pairs([(x, y) for x in range(4, 10) for y in range(3, 8)]))
    return phi


def _wall_patch(g, dtype):
    """Holes at a corner of the walls and across brick faces: pairs away from any
    defined cell."""
    nx, ny = _extent(g, 0), _extent(g, 1)
    phi = _plane(g, dtype)
    _undefine(phi, _pairs([(x, y) for x in range(6) for y in range(5)]))
    _undefine(phi, _pairs([(x, y) for x in range(5, 12) for y in range(6, 11)]))
    _undefine(phi, _pairs([(nx - 1 - x, ny - 1 - y) for x in range(2) for y in range(3)]))
    return phi


def _scattered(g, dtype):
    nx, ny = _extent(g, 0), _extent(g, 1)
    rng = np.random.default_rng(7)
    phi = _plane(g, dtype)
    _undefine(phi, _pairs([(x, y) for x in range(nx) for y in range(ny) if rng.random() < 0.3]))
    half = [(x, y, -Z0 - (rng.random() < 0.5)) for x in range(nx) for y in range(ny)
            if rng.random() < 0.1]
    _undefine(phi, half)
    return phi


def _far_values(g, dtype):
    """Values of magnitude 1 and above next to undefined cells of the other
    sign (0, and a sign change, come out)."""
    phi = _plane(g, dtype)
    k = -Z0
    for i, v in enumerate((1.0, 1.0, 0.9375)):
        phi[2 + 3 * i, 4, k] = v
        phi[2 + 3 * i, 9, k - 1] = -v
        _undefine(phi, [(2 + 3 * i, 4, k - 1), (2 + 3 * i, 9, k)])
    return phi


def _levels(g, dtype):
    """The plane moved by one brick in z (pairs across faces in z), with holes."""
    phi = np.roll(_plane(g, dtype), 8, 2)
    nx, ny = _extent(g, 0), _extent(g, 1)
    k = -Z0 + 8
    _undefine(phi, [(x, y, z) for x, y in ((1, 1), (9, 9), (nx - 1, 2)) for z in (k, k - 1)])
    return phi


BANDS = dict(pair=_one_pair, faces=_pairs_at_faces, patch=_patch, wall_patch=_wall_patch, scattered=_scattered,
             far=_far_values, levels=_levels)
GRIDS = {"periodic": (PER, 16, PER, 24), "ragged": (PER, 13, PER, 18), "reflective": (REF, 17, REF, 14),
         "mixed": (REF, 14, PER, 16)}


LO = np.array([0, 0, Z0])


def _cells(mask):
    i = np.argwhere(mask) + LO
    return i[np.lexsort((i[:, 0], i[:, 1], i[:, 2]))].astype(np.int32)


def _at(a, i):
    return a[tuple((i - LO).T)]


def _domain(g, phi):
    idx = _cells(np.abs(phi) < np.finfo(phi.dtype).max)

    def sign(x, y, z):
        c = [np.clip(v, 0, n - 1) for v, n in zip((x, y, z - Z0), phi.shape)]
        return np.where(phi[tuple(c)] < 0, -1, 1)

    rs, sg = make_runs(idx, sign, LO, LO + np.array(phi.shape) - 1)
    return Domain(g, idx, _at(phi, idx).astype(np.float64), rs, sg, 2)


def _context(g, phi, precision):
    ctx = Context(0, precision)
    ctx.set_grid(g)
    ctx.set_level_set_count(1)
    ctx.upload(0, _domain(g, phi))
    return ctx


def _same(ctx, g, want, scheme):
    top = np.finfo(want.dtype).max
    defined = np.abs(want) < top
    near = ~defined & np.any([np.abs(_shift(want, a, s, (g.bc[0], g.bc[1], None)[a])) < top
                              for a in range(3) for s in (1, -1)], axis=0)
    wi, ni = _cells(defined), _cells(near)
    gi, gv, _ = ctx.download(0)
    assert np.array_equal(gi, wi), (scheme, len(gi), len(wi))
    assert np.array_equal(gv.astype(want.dtype).view(np.uint8), _at(want, wi).view(np.uint8)), scheme
    assert np.array_equal(ctx.values_at(0, ni) < 0, _at(want, ni) < 0), scheme


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("walls", sorted(GRIDS))
@pytest.mark.parametrize("band", sorted(BANDS))
def test_cells_that_change_sign(band, walls, precision):
    g = _grid(*GRIDS[walls])
    phi = BANDS[band](g, np.float32 if precision else np.float64)
    dom = _domain(g, phi)
    ctx = _context(g, phi, precision)
    for scheme, width in [(0, 3), (1, 5), (11, 7), (9, 8), (8, 9)]:
        want = _expand(phi, g, 2, width)
        for _ in range(3):
            ctx.upload(0, dom)
            ctx.prepare_ls(scheme)
            _same(ctx, g, want, scheme)
    ctx.close()


@pytest.mark.parametrize("walls", sorted(GRIDS))
@pytest.mark.parametrize("band", ["patch", "scattered"])
def test_expands_after_one_that_changed_signs(band, walls):
    """Further Expands of the same band, without an upload in between."""
    g = _grid(*GRIDS[walls])
    phi = BANDS[band](g, np.float64)
    ctx, at = _context(g, phi, 0), 2
    for scheme, width in [(0, 3), (1, 5), (11, 7), (8, 9)]:
        phi, at = _expand(phi, g, at, width), width
        ctx.prepare_ls(scheme)
        _same(ctx, g, phi, scheme)
    ctx.close()
