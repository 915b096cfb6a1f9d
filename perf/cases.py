"""Timed workloads: level sets advanced through the public entry points.

A pass is what one call costs a simulation: its level sets, held in host memory
as points and undefined runs, go to the GPU, are advanced, and come back as
points and runs (batch: every domain of a batch, several steps).  Inputs are
seeded analytic shapes -- spheres with a smooth perturbation, circles, square
trenches, hole arrays -- whose place on the grid changes with the seed.

`exact` advances the same inputs with dense arrays and plain torch in 64 bits.
"""
import math

import numpy as np
import torch

from viennals_b200 import BoundaryConditionEnum as BC
from viennals_b200 import Domain, Grid
from viennals_b200 import SpatialSchemeEnum as S
from viennals_b200 import TemporalSchemeEnum as TS
from viennals_b200.advect import Advect, BatchContext, Context
from viennals_b200._abi import AdvectParams, Precision
from viennals_b200.domain import INF_INDEX
from viennals_b200.velocity import FunctorVelocity, VelocityField

DEV = "cuda"


def _case(name, shape, via, cells, scheme, temporal, bits, steps, delta, **more):
    return dict(name=name, shape=shape, via=via, cells=cells, scheme=scheme, temporal=temporal,
                bits=bits, steps=steps, delta=delta, **more)


def listed():
    return [
        # the smallest call: one step of a sphere of radius 8 cells
        _case("sphere_8_eo1_step", "sphere", "apply", 8, "EO1", "FE", 64, 1, 0.25),
        # the plain method's workload: radius 5 at 0.25, EO1, FE, up to t = 2
        _case("sphere_20_eo1", "sphere", "apply", 20, "EO1", "FE", 64, 16, 0.25),
        # a 2D cross-section simulation
        _case("circle_150_weno3_rk3", "circle", "apply", 150, "WENO3", "RK3", 64, 3, 0.1),
        # reflective side walls, odd extents: a quarter of a symmetric trench
        _case("mirror_trench_llf1_rk2", "trench", "apply", 40, "LLF1", "RK2", 64, 3, 0.1, nx=101,
              ny=75, mirror=True),
        # the square-trench etch at 128 x 128 x 64 cells, mask and substrate
        _case("trench_128_llf2_rk3", "trench", "context", 40, "LLF2", "RK3", 64, 3, 0.1, nx=128,
              ny=128, mirror=False),
        # a host velocity field (numpy, asked in batches), as process models have
        _case("callback_40_eo1", "sphere", "context", 40, "EO1", "FE", 64, 3, 0.1, callback=True),
        # perturbed spheres, the accuracy study's shape: ordinary sizes of both
        # precisions
        _case("sphere_160_weno5_rk3", "sphere", "context", 160, "WENO5", "RK3", 32, 4, 0.05),
        _case("sphere_293_weno5_rk3_fp64", "sphere", "context", 293, "WENO5", "RK3", 64, 2, 0.05),
        # stacked layers over a periodic hole array (deposition, three materials)
        _case("holes_384_weno5_rk3", "holes", "context", 32, "WENO5", "RK3", 32, 2, 0.02, nx=384,
              ny=384),
        # many independent domains in one context
        _case("batch_24_llf1_rk2", "batch", "batch", 24, "LLF1", "RK2", 32, 6, 0.1),
        # the largest: radius 40 at 0.05, 16.8M band points
        _case("sphere_800_weno5_rk3", "sphere", "context", 800, "WENO5", "RK3", 32, 3, 0.05),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["apply", "sphere", "sphere", "circle", "trench", "trench", "holes", "batch",
                       "callback"])
    if kind == "apply":
        c = _case("", "sphere", "apply", log(8, 60), rng.choice(["EO1", "EO2", "LLLF1", "LF1"]),
                  rng.choice(["FE", "RK2"]), 64, rng.randint(1, 12), 0.25)
    elif kind == "sphere":
        bits = rng.choice([32, 32, 64])
        c = _case("", "sphere", "context", log(40, 500 if bits == 32 else 300),
                  rng.choice(["WENO5", "WENO5", "WENO3", "EO2", "LLF1"]),
                  rng.choice(["RK3", "RK3", "RK2", "FE"]), bits, rng.randint(1, 3), 0.05)
    elif kind == "circle":
        c = _case("", "circle", "apply", log(20, 400), rng.choice(["EO1", "WENO3", "LF1"]),
                  rng.choice(["FE", "RK2", "RK3"]), 64, rng.randint(1, 6), 0.1)
    elif kind == "trench":
        c = _case("", "trench", rng.choice(["apply", "context"]), log(12, 60),
                  rng.choice(["LLF1", "LLF2", "WENO5", "EO1"]), rng.choice(["FE", "RK2", "RK3"]),
                  64, rng.randint(1, 4), 0.1, nx=rng.randint(80, 280), ny=rng.randint(80, 280),
                  mirror=rng.random() < 0.4)
    elif kind == "holes":
        n = 64 * rng.randint(2, 8)
        c = _case("", "holes", "context", 32, "WENO5", "RK3", rng.choice([32, 64]),
                  rng.randint(1, 2), 0.02, nx=n, ny=n)
    elif kind == "batch":
        c = _case("", "batch", "batch", rng.randint(2, 40), rng.choice(["LLF1", "WENO5"]),
                  rng.choice(["FE", "RK2", "RK3"]), 32, rng.randint(2, 8), 0.1)
    else:
        c = _case("", "sphere", "context", log(16, 60), "EO1", rng.choice(["FE", "RK2"]), 64,
                  rng.randint(1, 4), 0.1, callback=True)
    del c["name"]
    return c


SCHEMES = dict(EO1=S.ENGQUIST_OSHER_1ST_ORDER, EO2=S.ENGQUIST_OSHER_2ND_ORDER,
               LF1=S.LAX_FRIEDRICHS_1ST_ORDER, LLLF1=S.LOCAL_LOCAL_LAX_FRIEDRICHS_1ST_ORDER,
               LLF1=S.LOCAL_LAX_FRIEDRICHS_1ST_ORDER, LLF2=S.LOCAL_LAX_FRIEDRICHS_2ND_ORDER,
               WENO3=S.WENO_3RD_ORDER, WENO5=S.WENO_5TH_ORDER)
TEMPORAL = dict(FE=TS.FORWARD_EULER, RK2=TS.RUNGE_KUTTA_2ND_ORDER, RK3=TS.RUNGE_KUTTA_3RD_ORDER)
STAGES = dict(FE=1, RK2=2, RK3=3)
CFL = 0.4


# ------------------------------------------------------------------ inputs
def _shape(case, rng):
    """Grid, signed distance functions (bottom to top) and velocity of a case."""
    d = case["delta"]
    if case["shape"] == "sphere":
        return _sphere(case["cells"] * d, d, rng) + (_sphere_velocity(case),)
    if case["shape"] == "trench":
        return _trench(case, rng)
    return _holes(case, rng)


def _sphere(radius, d, rng):
    """A sphere whose radius is modulated by six smooth waves of 1% each."""
    cx, cy, cz = (float(v) * d for v in rng.uniform(-0.5, 0.5, 3))
    waves = [(rng.normal(0, 2.0, 3), float(rng.uniform(0, 6.28))) for _ in range(6)]

    def sdf(x, y, z):
        x, y, z = x - cx, y - cy, z - cz
        rho = torch.sqrt(x * x + y * y + z * z).clamp(min=0.5 * d)
        n = (x / rho, y / rho, z / rho)
        r = torch.full_like(rho, radius)
        g = [torch.zeros_like(rho) for _ in range(3)]
        for w, p in waves:
            a = n[0] * w[0] + n[1] * w[1] + n[2] * w[2] + p
            r = r + 0.01 * radius * torch.cos(a)
            s = -0.01 * radius * torch.sin(a)
            for k in range(3):
                g[k] = g[k] + s * w[k]
        dot = g[0] * n[0] + g[1] * n[1] + g[2] * n[2]
        tang = sum((g[k] - dot * n[k]) ** 2 for k in range(3)) / (rho * rho)
        return (rho - r) / torch.sqrt(1 + tang)

    m = int(radius / d * 1.07) + 4
    grid = Grid(None, [BC.INFINITE_BOUNDARY] * 3, d)
    return grid, [sdf], [-m] * 3, [m] * 3


class _HostField(VelocityField):
    """A process model on the host: a flux that falls off with height."""

    def batch(self, coords, materials, normals, point_ids, scalar_out, vector_out):
        scalar_out[:] = _host_speed(coords[:, 2], normals[:, 2])
        vector_out[:] = 0.0


def _host_speed(z, nz):
    return 1.0 + 0.05 * z + 0.2 * nz * nz


def _sphere_velocity(case):
    if case.get("callback"):
        return _HostField()
    v = FunctorVelocity(1)
    v.set_rate(0, 1.0)
    v.set_linear(0, 2, 0.3)
    return v


def _trench(case, rng):
    d, nx, ny = case["delta"], case["nx"], case["ny"]
    half = 0.5 * case["cells"] * d
    sx, sy, sz = (float(v) * d for v in rng.uniform(-0.4, 0.4, 3))
    top = 0.5 + 0.3 * sz
    bc = BC.REFLECTIVE_BOUNDARY if case["mirror"] else BC.PERIODIC_BOUNDARY
    x0, y0 = (0, 0) if case["mirror"] else (-(nx // 2), -(ny // 2))
    grid = Grid(None, [bc, bc, BC.INFINITE_BOUNDARY], d, index_min=[x0, y0, -32],
                index_max=[x0 + nx, y0 + ny, 32])

    def mask(x, y, z):
        z = z - sz
        qx, qy = torch.abs(x - sx) - half, torch.abs(y - sy) - half
        hole = torch.sqrt(qx.clamp(min=0) ** 2 + qy.clamp(min=0) ** 2) + \
            torch.maximum(qx, qy).clamp(max=0)
        return torch.maximum(torch.maximum(-z, z - top), -hole)

    def surface(x, y, z):
        return torch.minimum(z - sz, mask(x, y, z))

    v = FunctorVelocity(2)
    v.set_rate(1, -1.0)
    v.set_linear(1, 2, -0.3)
    last = 0 if case["mirror"] else 1
    return (grid, [mask, surface], [x0, y0, -12], [x0 + nx - last, y0 + ny - last, 14], v)


def _holes(case, rng):
    d, n = case["delta"], case["nx"]
    pitch, radius, depth = 64 * d, 0.39 * 64 * d, 2.0
    sx, sy, sz = (float(v) * d for v in rng.uniform(-0.4, 0.4, 3))
    lo = [-(n // 2), -(n // 2), -int(depth / d) - 8]
    hi = [n - n // 2 - 1, n - n // 2 - 1, int(0.3 / d) + 8]
    grid = Grid(None, [BC.PERIODIC_BOUNDARY, BC.PERIODIC_BOUNDARY, BC.INFINITE_BOUNDARY], d,
                index_min=lo, index_max=[lo[0] + n, lo[1] + n, hi[2]])

    def rho(x, y):
        px = torch.remainder(x - sx, pitch) - pitch / 2
        py = torch.remainder(y - sy, pitch) - pitch / 2
        return torch.sqrt(px * px + py * py)

    def substrate(x, y, z):
        z = z - sz
        return torch.maximum(z, -torch.maximum(rho(x, y) - radius, -z - depth))

    def slab(h):
        def f(x, y, z):
            s = torch.maximum(torch.maximum(z - sz - h, sz - z), radius - rho(x, y))
            return torch.minimum(substrate(x, y, z), s)
        return f

    v = FunctorVelocity(3)
    for m, rate in enumerate((1.0, 0.6, 0.0)):
        v.set_rate(m, rate)
        v.set_abs(m, 2, 0.2)
    return grid, [substrate, slab(0.1), slab(0.3)], lo, hi, v


def _batch_sizes(case):
    """Extent in cells, spacing, width (of the extent), depth in cells and kind
    of the domains of a batch, the same for every seed."""
    rng = np.random.default_rng(case["cells"])
    return [(8 * int(round(math.exp(rng.uniform(math.log(7), math.log(40))))),
             float(math.exp(rng.uniform(math.log(0.05), math.log(0.2)))),
             float(rng.uniform(0.1, 0.4)), float(rng.uniform(6, 60)), bool(rng.integers(2)))
            for _ in range(case["cells"])]


def _batch_items(case, rng):
    """Planes with a trench or a hole, periodic, bands of 1e4 to 3e5 points."""
    items = []
    for n, d, width, depth, round_hole in _batch_sizes(case):
        half = width * n * d * (1 + float(rng.uniform(-0.02, 0.02))) / 2
        depth = depth * d
        rate = float(rng.uniform(0.2, 1.5))
        sz = float(rng.uniform(-0.4, 0.4)) * d
        c2 = n // 2
        lo, hi = [-c2, -c2, -int(depth / d) - 6], [c2 - 1, c2 - 1, 6]

        def sdf(x, y, z, half=half, depth=depth, round_hole=round_hole, sz=sz):
            z = z - sz
            q = (torch.sqrt(x * x + y * y) if round_hole else torch.abs(x)) - half
            return torch.maximum(z, -torch.maximum(q, -z - depth))

        grid = Grid(None, [BC.PERIODIC_BOUNDARY, BC.PERIODIC_BOUNDARY, BC.INFINITE_BOUNDARY], d,
                    index_min=lo, index_max=[c2, c2, hi[2]])
        v = FunctorVelocity(1)
        v.set_rate(0, -rate)
        items.append((grid, _band(grid, sdf, lo, hi), v))
    return items


def _key(x, y, z):
    o = 1 << 20
    return ((z + o) << 42) + ((y + o) << 21) + (x + o)


def _band(grid, sdf, lo, hi):
    """The width-2 band of a signed distance over the index box [lo, hi], in
    HRLE order, and its undefined runs (row heads, gaps, tails, empty rows and
    the space around the box), as host arrays."""
    d, B = grid.delta, 8
    nb = [(hi[k] - lo[k]) // B + 1 for k in range(3)]
    reach = (math.sqrt(3.0) * 4.2 + 2.0) * d
    off = torch.arange(B, device=DEV)
    oz, oy, ox = (t.reshape(-1) for t in torch.meshgrid(off, off, off, indexing="ij"))
    by, bx = (t.reshape(-1) for t in torch.meshgrid(torch.arange(nb[1], device=DEV),
                                                    torch.arange(nb[0], device=DEV), indexing="ij"))
    corners = []
    for z0 in range(0, nb[2], 16):
        bz = torch.arange(z0, min(z0 + 16, nb[2]), device=DEV)
        c = torch.stack([(lo[0] + bx * B).repeat(len(bz)), (lo[1] + by * B).repeat(len(bz)),
                         (lo[2] + bz * B).repeat_interleave(len(bx))], 1)
        m = c.double() + 3.5
        corners.append(c[torch.abs(sdf(m[:, 0] * d, m[:, 1] * d, m[:, 2] * d)) <= reach])
    corners = torch.cat(corners)
    points, vals = [], []
    for s in range(0, len(corners), 1 << 15):
        c = corners[s:s + (1 << 15), None, :]
        x, y, z = ((c[:, :, 0] + ox).reshape(-1), (c[:, :, 1] + oy).reshape(-1),
                   (c[:, :, 2] + oz).reshape(-1))
        v = sdf(x.double() * d, y.double() * d, z.double() * d) / d
        keep = (torch.abs(v) <= 1.0) & (x <= hi[0]) & (y <= hi[1]) & (z <= hi[2])
        points.append(_key(x[keep], y[keep], z[keep]))
        vals.append(v[keep])
    key, order = torch.sort(torch.cat(points))
    vals = torch.cat(vals)[order]
    o, m21 = 1 << 20, (1 << 21) - 1
    px, py, pz = (key & m21) - o, ((key >> 21) & m21) - o, (key >> 42) - o
    rs, sg = _runs(sdf, d, key, px, py, pz, [v - 1 for v in lo], [v + 1 for v in hi])
    idx = torch.stack([px, py, pz], 1).to(torch.int32)
    return Domain(grid, idx.cpu().numpy(), vals.cpu().numpy(), rs, sg, width=2)


def _runs(sdf, d, key, px, py, pz, lo, hi):
    ny, nz = hi[1] - lo[1] + 1, hi[2] - lo[2] + 1
    zs = torch.arange(lo[2], hi[2] + 1, device=DEV)
    one = torch.ones(1, dtype=torch.int64, device=DEV)
    cx, cy, ni = (lo[0] + hi[0]) // 2, (lo[1] + hi[1]) // 2, -INF_INDEX
    row = (pz - lo[2]) * ny + (py - lo[1])
    has = torch.zeros(ny * nz, dtype=torch.bool, device=DEV)
    has[row] = True
    empty = torch.nonzero(~has).reshape(-1)
    ey, ez = lo[1] + empty % ny, lo[2] + torch.div(empty, ny, rounding_mode="floor")
    new_row = row[1:] != row[:-1]
    t = torch.ones(1, dtype=torch.bool, device=DEV)
    first, last = torch.cat([t, new_row]), torch.cat([new_row, t])
    gap = last.clone()
    gap[:-1] |= px[1:] > px[:-1] + 1
    starts = [(one * ni, one * ni, one * ni), (one * ni, one * ni, one * (hi[2] + 1)),
              (torch.full_like(zs, ni), torch.full_like(zs, ni), zs),
              (torch.full_like(zs, ni), torch.full_like(zs, hi[1] + 1), zs),
              (torch.full_like(ey, ni), ey, ez),
              (torch.full_like(px[first], ni), py[first], pz[first]),
              (px[gap] + 1, py[gap], pz[gap])]
    inside = [(one * cx, one * cy, one * (lo[2] - 1)), (one * cx, one * cy, one * (hi[2] + 1)),
              (torch.full_like(zs, cx), torch.full_like(zs, lo[1] - 1), zs),
              (torch.full_like(zs, cx), torch.full_like(zs, hi[1] + 1), zs),
              (torch.full_like(ey, lo[0]), ey, ez),
              (px[first] - 1, py[first], pz[first]), (px[gap] + 1, py[gap], pz[gap])]
    x, y, z = (torch.cat([s[k] for s in starts]) for k in range(3))
    ex, ey, ez = (torch.cat([s[k] for s in inside]).double() * d for k in range(3))
    sign = torch.cat([torch.where(sdf(ex[s:s + (1 << 23)], ey[s:s + (1 << 23)], ez[s:s + (1 << 23)])
                                  < 0, -1, 1) for s in range(0, len(ex), 1 << 23)]).to(torch.int8)
    rkey, order = torch.sort(_key(x, y, z))
    x, y, z, sign = x[order], y[order], z[order], sign[order]
    before = torch.searchsorted(key, rkey)
    keep = torch.ones(len(x), dtype=torch.bool, device=DEV)
    keep[1:] = (sign[1:] != sign[:-1]) | (before[1:] != before[:-1])
    start = torch.stack([x, y, z], 1)[keep].to(torch.int32)
    return start.cpu().numpy(), sign[keep].cpu().numpy()


def _circle(case, rng):
    from viennals_b200.geometry import make_circle

    d, r = case["delta"], case["cells"]
    grid = Grid(None, [BC.INFINITE_BOUNDARY] * 2, d, dim=2, index_min=[0, 0], index_max=[0, 0])
    v = FunctorVelocity(1)
    v.set_rate(0, 1.0)
    v.set_linear(0, 1, 0.3)
    origin = [float(v) * d for v in rng.uniform(-0.4, 0.4, 2)]
    return grid, [make_circle(grid, origin, r * d)], v


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    if case["shape"] == "circle":
        return _circle(case, rng)
    grid, sdfs, lo, hi, vel = _shape(case, rng)
    return grid, [_band(grid, f, lo, hi) for f in sdfs], vel


def _speed(case):
    """The largest speed of the case's velocity field."""
    if case.get("callback"):
        return 1.2 + 0.05 * case["cells"] * case["delta"]
    return 1.2 if case["shape"] == "holes" else 1.3


def _params(case):
    p = AdvectParams.defaults()
    p.spatial_scheme = int(SCHEMES[case["scheme"]])
    p.temporal_scheme = int(TEMPORAL[case["temporal"]])
    p.time_step_ratio = CFL
    if case["via"] != "batch":
        p.advection_time = case["steps"] * CFL * case["delta"] / _speed(case)
    return p


def _pinned(shape, dtype):
    return torch.zeros(shape, dtype=dtype, pin_memory=True).numpy()


def _pin(a):
    t = torch.from_numpy(a)
    return (t.pin_memory() if t.numel() else t).numpy()


def prepare(case, seed):
    precision = Precision.FP32 if case["bits"] == 32 else Precision.FP64
    if case["via"] == "batch":
        n = _room(case)[0]
        return dict(case=case, items=_batch_items(case, np.random.default_rng(seed)),
                    ctx=BatchContext(0, precision), params=_params(case),
                    idx=np.zeros((n, 3), np.int32), values=np.zeros(n))
    grid, doms, vel = _inputs(case, seed)
    st = dict(case=case, grid=grid, doms=doms, vel=vel)
    if case["via"] == "apply":
        a = Advect(precision=precision)
        a.setVelocityField(vel)
        a.setSpatialScheme(SCHEMES[case["scheme"]])
        a.setTemporalScheme(TEMPORAL[case["temporal"]])
        a.setTimeStepRatio(CFL)
        a.setAdvectionTime(_params(case).advection_time)
        st["advect"] = a
        return st
    # a program on the C ABI: one context, page-locked host arrays, room for
    # the band to grow
    ctx = Context(0, precision)
    ctx.set_grid(grid)
    ctx.set_level_set_count(len(doms))
    if vel.descriptor() is not None:
        ctx.set_velocity(vel.descriptor())
    else:
        ctx.set_velocity_callback(vel)
    out, (n, m) = [], _room(case)
    for d in doms:
        b = Domain(grid)
        b.idx, b.values = _pinned((n, 3), torch.int32), _pinned((n,), torch.float64)
        b.run_start, b.run_sign = _pinned((m, 3), torch.int32), _pinned((m,), torch.int8)
        out.append(b)
        d.idx, d.values, d.run_start, d.run_sign = (
            _pin(d.idx), _pin(d.values), _pin(d.run_start), _pin(d.run_sign))
    st.update(ctx=ctx, out=out, params=_params(case))
    return st


# -------------------------------------------------------------------- a pass
def _room(case):
    """Points and runs a level set of the case (batch: all domains) may have:
    output arrays have this size for every seed, zeros after the last entry."""
    a = _area(case)
    return int(2.8 * a) + 20000, int(a) + 20000


def _padded(a, n):
    assert len(a) <= n, (len(a), n)
    return np.concatenate([a, np.zeros((n - len(a),) + a.shape[1:], a.dtype)])


def _outputs(case, doms, r):
    n, m = _room(case)
    got = dict(points=np.array([d.n_points for d in doms]),
               runs=np.array([len(d.run_sign) for d in doms]),
               time=r.advected_time, step=r.current_time_step, updates=int(r.point_updates))
    for k, size in (("idx", n), ("values", n), ("run_start", m), ("run_sign", m)):
        got[k] = [_padded(getattr(d, k), size) for d in doms]
    return got


def run(state):
    case = state["case"]
    if case["via"] == "batch":
        ctx = state["ctx"]
        ctx.set_domains(state["items"])
        res = [ctx.advect(state["params"]) for _ in range(case["steps"])]
        got = [ctx.download(k) for k in range(len(state["items"]))]
        idx, values, at = state["idx"], state["values"], 0
        for i, v, _ in got:
            idx[at:at + len(v)], values[at:at + len(v)] = i, v
            at += len(v)
        return dict(points=np.array([len(g[1]) for g in got]), idx=idx, values=values,
                    time=np.array([[r.advected_time for r in step] for step in res]),
                    updates=int(sum(r.point_updates for step in res for r in step)))
    if case["via"] == "apply":
        a = state["advect"]
        a.clearLevelSets()
        doms = []
        for d in state["doms"]:  # apply() replaces the arrays of the objects it is given
            doms.append(Domain(d.grid, d.idx, d.values, d.run_start, d.run_sign, d.width))
            a.insertNextLevelSet(doms[-1])
        r = a.apply()
        return _outputs(case, doms, r)
    ctx = state["ctx"]
    for k, d in enumerate(state["doms"]):
        ctx.upload(k, d)
    r = ctx.advect(state["params"])
    out = state["out"]
    doms = [ctx.download_domain(k, state["grid"], out=b) for k, b in enumerate(out)]
    got = dict(points=np.array([d.n_points for d in doms]),
               runs=np.array([len(d.run_sign) for d in doms]),
               time=r.advected_time, step=r.current_time_step, updates=int(r.point_updates))
    for k in ("idx", "values", "run_start", "run_sign"):
        got[k] = [getattr(b, k) for b in out]
    return got


# ------------------------------------------------------------ what it needs
def _area(case):
    """Surface cells of a level set (batch: of all domains); a band of width w
    holds about w times as many points."""
    c, n = case["cells"], case.get("nx", 0) * case.get("ny", 0)
    if case["shape"] == "sphere":
        return 4 * math.pi * c * c
    if case["shape"] == "circle":
        return 2 * math.pi * c
    if case["shape"] == "trench":
        return 2 * n + 4 * c * 6
    if case["shape"] == "holes":
        return n + n / 4096 * 2 * math.pi * 25 * 105
    return sum(m * m + (math.pi * w if hole else 2) * m * depth
               for m, _, w, depth, hole in _batch_sizes(case))


LEVELS = dict(trench=2, holes=3)
FLOPS = dict(EO1=40, EO2=90, LF1=60, LLLF1=70, LLF1=900, LLF2=950, WENO3=200, WENO5=450)


def work(case):
    """Points and runs in and out once; per stage the width-2 band read and
    written once (and the saved band read by each stage combination)."""
    a, size = _area(case), case["bits"] // 8
    stages = STAGES[case["temporal"]]
    combos = stages - 1
    state = case["steps"] * size * 2 * a * (2 * stages + 3 * combos)
    exchange = LEVELS.get(case["shape"], 1) * 2 * (2 * a * 20 + 0.5 * a * 13)
    return dict(bytes=state + exchange, flops=case["steps"] * stages * a * FLOPS[case["scheme"]])


# --------------------------------------------------------- 64-bit dense form
MAXV = torch.finfo(torch.float64).max
EPS = torch.finfo(torch.float64).eps
WIDTH = dict(EO1=3, EO2=5, LF1=3, LLLF1=3, LLF1=7, LLF2=9, WENO3=5, WENO5=7)


def _far(negative):
    """The sentinels of undefined cells, by sign."""
    return torch.where(negative, -MAXV, torch.tensor(MAXV, dtype=torch.float64, device=DEV))


class _Dense:
    """Level sets on a dense box, undefined cells +-MAXV."""

    def __init__(self, grid, doms, case, speed):
        self.dim, self.delta, self.case, self.speed = grid.dim, grid.delta, case, speed
        pad = WIDTH[case["scheme"]] // 2 + 4 + case["steps"]
        self.lo, self.n, self.near = [], [], []
        for d in range(3):
            if d >= self.dim:
                lo, n = 0, 1
            elif grid.bc[d] == BC.INFINITE_BOUNDARY:
                lo = min(int(x.idx[:, d].min()) for x in doms) - pad
                n = max(int(x.idx[:, d].max()) for x in doms) + pad - lo + 1
            else:
                lo = grid.min[d]
                n = grid.max[d] - lo + (0 if grid.is_periodic(d) else 1)
            at = torch.arange(-5, n + 5, device=DEV)
            if d >= self.dim:
                at = torch.zeros_like(at)
            elif grid.bc[d] == BC.PERIODIC_BOUNDARY:
                at = at % n
            elif grid.bc[d] == BC.REFLECTIVE_BOUNDARY:
                at = (n - 1) - torch.abs((n - 1) - torch.abs(at))
            else:
                at = at.clamp(0, n - 1)
            self.lo.append(lo), self.n.append(n), self.near.append(at)

    def cells(self):
        return self.n[0] * self.n[1] * self.n[2]

    def fill(self, dom, sign):
        """The dense array of a level set; sign(x, y, z) of the undefined."""
        z, y, x = torch.meshgrid(*[(torch.arange(self.n[d], device=DEV) + self.lo[d]).double()
                                   * self.delta for d in (2, 1, 0)], indexing="ij")
        a = _far(sign(x, y, z) < 0)
        i = torch.from_numpy(dom.idx).to(DEV).long()
        zi = i[:, 2] - self.lo[2] if self.dim == 3 else torch.zeros_like(i[:, 0])
        a[zi, i[:, 1] - self.lo[1], i[:, 0] - self.lo[0]] = torch.from_numpy(dom.values).to(DEV)
        return a

    def star(self, a):
        for k in (1, -1):  # +x, +y, +z, -x, -y, -z
            for d in range(self.dim):
                yield a.index_select(2 - d, self.near[d][5 + k:5 + k + self.n[d]])

    def expand(self, a, w0, w):
        for c in range(w0, w):
            limit = 0.5 * (c + 1)
            low = torch.full_like(a, MAXV)
            high = torch.full_like(a, -MAXV)
            for b in self.star(a):
                low, high = torch.minimum(low, b + 1), torch.maximum(high, b - 1)
            up = torch.where(low <= limit, low, MAXV)
            down = torch.where(high >= -limit, high, -MAXV)
            a = torch.where(torch.abs(a) <= 0.5 * w, a, torch.where(a > -EPS, up, down))
        return a

    def prune(self, a):
        for stray in (True, False):
            neg = a <= -EPS
            keep = a == 0
            nb = list(self.star(a))
            for b in nb:
                keep |= (b <= -EPS) != neg
                if stray:
                    keep |= b == 0
            out = torch.where(keep & (torch.abs(a) < MAXV), a, _far(neg))
            if stray:
                done = torch.zeros_like(keep)
                for p, q in zip(nb[:self.dim], nb[self.dim:]):
                    mono = (p == 0) | (q == 0) | ((p <= -EPS) != (q <= -EPS))
                    hit = (a == 0) & ~mono & ~done
                    out = torch.where(hit, torch.where(torch.abs(p) < torch.abs(q), p, q), out)
                    done |= hit
            a = out
        return a

    def rebuild(self, a):
        side = torch.signbit(a + 1e-7)
        crossing = torch.zeros_like(side)
        above, below = torch.zeros_like(side), torch.zeros_like(side)
        low, high = torch.full_like(a, MAXV), torch.full_like(a, -MAXV)
        for b in self.star(a):
            crossing |= torch.signbit(b - 1e-7) != side
            near = torch.abs(b) <= 1.0
            below |= near & (b < -0.5)
            above |= near & (b > 0.5)
            low = torch.where(near & (b < 0), torch.minimum(low, b + 1), low)
            high = torch.where(near & (b > 0), torch.maximum(high, b - 1), high)
        kept = torch.where((a > 0.5) & below, 0.5, torch.where((a < -0.5) & above, -0.5, a))
        inner = torch.where(crossing, kept, _far(a < 0))
        outer = torch.where(a >= 0, torch.where(low <= 1, low, MAXV),
                            torch.where(high >= -1, high, -MAXV))
        return torch.where(torch.abs(a) <= 1.0, inner, outer)

    # ------------------------------------------------------------- one stage
    def stage(self, ls, cap):
        """Rates of the top level set's active points, the step and the update."""
        top = ls[-1] = self.expand(ls[-1], 2, WIDTH[self.case["scheme"]])
        at = torch.nonzero(torch.abs(top) <= 0.5)
        zi, yi, xi = at[:, 0], at[:, 1], at[:, 2]

        def value(dx, dy, dz):
            return top[self.near[2][zi + dz + 5], self.near[1][yi + dy + 5], self.near[0][xi + dx + 5]]

        coord = [(i + lo).double() * self.delta for i, lo in zip((xi, yi, zi), self.lo)]
        phi = value(0, 0, 0)
        below = [b[zi, yi, xi] for b in ls[:-1]] + [phi]
        made = [self.rate(value, coord, m) for m in range(len(ls))]
        v, cfl = phi.clone(), torch.full_like(phi, CFL)
        most, going = torch.zeros_like(phi), torch.ones_like(phi, dtype=torch.bool)
        legs, alpha = [], [torch.zeros((), device=DEV, dtype=torch.float64)] * 3
        for cur in range(len(ls) - 1, -1, -1):
            g, d = torch.zeros_like(phi), torch.zeros_like(phi)
            free = going.clone()
            for m in range(len(ls)):
                pick = free & (below[m] <= v + 1e-4)
                g, d = torch.where(pick, made[m][0], g), torch.where(pick, made[m][1], d)
                if made[m][2] is not None:
                    alpha = [torch.maximum(p, torch.where(pick, q, 0.0).max())
                             for p, q in zip(alpha, made[m][2])]
                free &= ~pick
            vel = g - d
            use = torch.where(((g < 0) & (vel > 0)) | ((g > 0) & (vel < 0)), 0.0, vel)
            under = below[cur - 1] if cur > 0 else torch.full_like(phi, MAXV)
            gap = torch.abs(under - v)
            far = gap >= cfl
            step = torch.where(vel > 0, cfl / vel, torch.where(far, -cfl / vel, -gap / vel))
            most = torch.where(going, torch.where(vel == 0, MAXV, most + step), most)
            stop = torch.where(vel > 0, -MAXV, torch.where((vel == 0) | far, MAXV, under))
            legs.append((use, stop))
            on = going & (vel < 0) & ~far
            cfl, v = torch.where(on, cfl - gap, cfl), torch.where(on, under, v)
            going = on
        dt = cap
        if len(phi):
            dt = min(dt, float(torch.where(most >= 0, most, MAXV).min()))
        if made[0][2] is not None:
            total = sum(float(x) / self.delta for x in alpha)
            dt = min(dt, 1.0 / total if total else math.inf)
        new, time = phi.clone(), torch.full_like(phi, dt)
        walking = torch.ones_like(phi, dtype=torch.bool)
        for vel, stop in legs:
            rate = time * vel
            on = walking & (torch.abs(stop - new) < torch.abs(rate))
            new = torch.where(walking & ~on, new - rate, new)
            time = torch.where(on, time - torch.abs((stop - new) / vel), time)
            new = torch.where(on, stop, new)
            walking = on
        out = _far(top < 0)
        out[zi, yi, xi] = new
        ls[-1] = self.rebuild(out)
        return dt

    def rate(self, value, coord, m):
        s, h = self.case["scheme"], self.delta
        c = value(0, 0, 0)
        axis = lambda i, k: value(*[k if j == i else 0 for j in range(3)])  # noqa: E731
        zero = torch.zeros_like(c)
        if s.startswith("LLF") or s == "LLLF1" or s == "LF1":
            return None if s in ("LLLF1", "LF1") else self.llf(value, axis, c, coord, m)
        gp, gn, n2, normal = zero, zero, zero, []
        for i in range(3):
            if s in ("WENO3", "WENO5"):
                r = 3 if s == "WENO5" else 2
                x = [axis(i, k) for k in range(-r, r + 1)]
                f = _weno5 if r == 3 else _weno3
                minus, plus = f(x, h), f(x[::-1], -h)
            else:
                plus, minus = (axis(i, 1) - c) / h, (c - axis(i, -1)) / h
                if s == "EO2":
                    minus, plus = self.second(axis, c, i, minus, plus)
            gp = gp + minus.clamp(min=0) ** 2 + plus.clamp(max=0) ** 2
            gn = gn + minus.clamp(max=0) ** 2 + plus.clamp(min=0) ** 2
            normal.append(axis(i, 1) - axis(i, -1))
            n2 = n2 + normal[-1] ** 2
        normal = [n / torch.sqrt(n2) for n in normal]
        speed = self.speed(coord, m, normal)
        return torch.where(speed > 0, torch.sqrt(gp), torch.sqrt(gn)) * speed, zero, None

    def second(self, axis, c, i, minus, plus):
        h = self.delta
        mid = (axis(i, 1) - 2 * c + axis(i, -1)) / (2 * h * h)
        out = []
        for sgn, first in ((-1, minus), (1, plus)):
            far = (axis(i, 2 * sgn) - 2 * axis(i, sgn) + c) / (2 * h * h)
            pick = torch.where(torch.abs(far) < torch.abs(mid), far, mid)
            same = torch.signbit(far) == torch.signbit(mid)
            out.append(first - sgn * h * torch.where(same, pick, 0.0))
        return out

    def llf(self, value, axis, c, coord, m):
        h = self.delta
        g2, n2, centre, back, fwd = 0, 0, [], [], []
        for i in range(3):
            plus, minus = (axis(i, 1) - c) / h, (c - axis(i, -1)) / h
            if self.case["scheme"] == "LLF2":
                minus, plus = self.second(axis, c, i, minus, plus)
            back.append(minus), fwd.append(plus), centre.append((minus + plus) / 2)
            g2 = g2 + centre[-1] ** 2
        speed = self.speed(coord, m, [n / torch.sqrt(g2) for n in centre])
        ham = speed * torch.sqrt(g2)
        alpha = [torch.zeros_like(c) for _ in range(3)]
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    n = [(value(dx + (i == 0), dy + (i == 1), dz + (i == 2))
                          - value(dx - (i == 0), dy - (i == 1), dz - (i == 2))) / (2 * h)
                         for i in range(3)]
                    n2 = torch.sqrt(n[0] ** 2 + n[1] ** 2 + n[2] ** 2)
                    n = [v / n2 for v in n]
                    s = self.speed(coord, m, n)
                    for i in range(3):
                        t = torch.abs(s * n[i])
                        alpha[i] = torch.where(t > alpha[i], t, alpha[i])
        diss = sum(alpha[i] * (fwd[i] - back[i]) / 2 for i in range(3))
        on = ham != 0
        return ham, torch.where(on, diss, 0.0), [torch.where(on, a, 0.0) for a in alpha]

    # -------------------------------------------------------------- the steps
    def lower(self, ls):
        for k in range(len(ls) - 1):
            ls[k] = self.prune(torch.maximum(ls[k], ls[-1]))

    def combine(self, ls, first, source, target, stages):
        w = math.ceil(2 * stages * CFL + 1)
        a, b = self.expand(ls[-1], 2, w), self.expand(first, 2, w)
        both = (torch.abs(a) < MAXV) & (torch.abs(b) < MAXV)
        mix = torch.where(both, source * torch.where(both, a, 0.0) + target * torch.where(both, b, 0.0),
                          torch.where(torch.abs(a) < MAXV, b, a))
        moved = bool((both & (mix > b)).any())
        ls[-1] = self.rebuild(self.prune(mix))
        return moved

    def step(self, ls, cap):
        t = self.case["temporal"]
        first = list(ls)
        dt1 = self.stage(ls, cap)
        if t == "FE":
            self.lower(ls)
            return dt1
        dt2 = self.stage(ls, dt1)
        if t == "RK2":
            self.combine(ls, first[-1], 0.5, 0.5, 2)
            self.lower(ls)
            return 0.5 * dt1 + 0.5 * dt2
        self.combine(ls, first[-1], 0.25, 0.75, 3)
        self.lower(ls)
        dt3 = self.stage(ls, dt1)
        if self.combine(ls, first[-1], 2.0 / 3.0, 1.0 / 3.0, 3):
            ls[:-1] = first[:-1]
        self.lower(ls)
        return (dt1 + dt2 + 4 * dt3) / 6

    def points(self, a):
        """Values of the defined points in HRLE order."""
        return a[torch.abs(a) < MAXV].cpu().numpy()


def _weno3(x, h):
    d = [x[k + 1] - x[k] for k in range(3)]
    n, m = 1e-6 + (d[1] - d[0]) ** 2, 1e-6 + (d[2] - d[1]) ** 2
    w = m * m / (m * m + 2 * n * n)
    return (d[1] + d[2] - w * (d[0] - 2 * d[1] + d[2])) / (2 * h)


def _weno5(x, h):
    d = [x[k + 1] - x[k] for k in range(5)]
    s = [13 / 12 * (d[k] - 2 * d[k + 1] + d[k + 2]) ** 2 for k in range(3)]
    s[0] = s[0] + (d[0] - 4 * d[1] + 3 * d[2]) ** 2 / 4
    s[1] = s[1] + (d[1] - d[3]) ** 2 / 4
    s[2] = s[2] + (3 * d[2] - 4 * d[3] + d[4]) ** 2 / 4
    w = [g / (1e-6 * h * h + q) for g, q in zip((0.1, 0.6, 0.3), s)]
    p = [(2 * d[0] - 7 * d[1] + 11 * d[2]) / 6, (-d[1] + 5 * d[2] + 2 * d[3]) / 6,
         (2 * d[2] + 5 * d[3] - d[4]) / 6]
    return (w[0] * p[0] + w[1] * p[1] + w[2] * p[2]) / ((w[0] + w[1] + w[2]) * h)


def _speeds(case, vel):
    """vel as torch arithmetic: speed(coordinates, material, normal)."""
    if case.get("callback"):
        return lambda x, m, n: _host_speed(x[2], n[2])

    def speed(x, m, n):
        s = torch.full_like(n[0], vel.rate[m])
        for k in range(3):
            s = s + vel.lin_pos[m][k] * n[k] + vel.abs_pos[m][k] * torch.abs(n[k])
        return s
    return speed


def _advance(case, grid, doms, sdfs, vel):
    dense = _Dense(grid, doms, case, _speeds(case, vel))
    if dense.cells() * case["steps"] * STAGES[case["temporal"]] > 5e8:
        return None
    ls = [dense.fill(d, f) for d, f in zip(doms, sdfs)]
    if case["via"] == "batch":
        time = np.array([dense.step(ls, math.inf) for _ in range(case["steps"])])
        return [dense.points(a) for a in ls], time
    t, end = 0.0, _params(case).advection_time
    while t < end:
        t += dense.step(ls, end - t)
    return [dense.points(a) for a in ls], t


def exact(case, seed):
    """`run`'s values and times on a dense grid in 64 bits (indices, runs and
    counts are whole numbers; None for boxes too large for a few seconds)."""
    if case["scheme"] in ("LF1", "LLLF1"):
        return None
    rng = np.random.default_rng(seed)
    if case["via"] == "batch":
        got = []
        for grid, dom, vel in _batch_items(case, rng):
            got.append(_advance(case, grid, [dom], [_sign_of(grid, dom)], vel))
            if got[-1] is None:
                return None
        values = _padded(np.concatenate([v[0] for v, _ in got]), _room(case)[0])
        return dict(values=values, time=np.stack([t for _, t in got], 1))
    if case["shape"] == "circle":
        grid, doms, vel = _circle(case, rng)
        sdfs = [_sign_of(grid, doms[0])]
    else:
        grid, sdfs, lo, hi, vel = _shape(case, rng)
        if (hi[0] - lo[0]) * (hi[1] - lo[1]) * (hi[2] - lo[2]) > 1e8:
            return None
        doms = [_band(grid, f, lo, hi) for f in sdfs]
    got = _advance(case, grid, doms, sdfs, vel)
    if got is None:
        return None
    return dict(values=[_padded(v, _room(case)[0]) for v in got[0]], time=float(got[1]))


def _sign_of(grid, dom):
    """Sign of the undefined cells from the domain's runs: sign(x, y, z)."""
    start = torch.from_numpy(np.ascontiguousarray(dom.run_start)).to(DEV).long()
    if grid.dim == 2:
        start = torch.cat([start, torch.zeros_like(start[:, :1])], 1)
    keys = _key(start[:, 0], start[:, 1], start[:, 2])
    signs = torch.from_numpy(dom.run_sign).to(DEV)

    def sign(x, y, z):
        i = [torch.round(v / grid.delta).long() for v in (x, y, z)]
        at = torch.searchsorted(keys, _key(*i), right=True) - 1
        return signs[at.clamp(min=0)].double()

    return sign
