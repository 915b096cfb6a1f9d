"""Routes that small inputs do not take: replays of the batching form's captured
step, and the 64-entry tiles of large level sets, each against the same work done
another way, bit for bit."""
import numpy as np
import pytest

from parity_cases import params
from test_gpu_batch import _same
from viennals_b200 import BoundaryConditionEnum as BC, Domain, Grid
from viennals_b200.advect import Context
from viennals_b200.domain import make_runs
from viennals_b200.geometry import sdf_levelset
from viennals_b200.synth import batch_domains
from viennals_b200.velocity import FunctorVelocity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("spatial,temporal", [(0, 0), (7, 1), (11, 2)])
def test_batch_steps_after_the_captured_one(spatial, temporal, precision):
    items = batch_domains(6, seed=17, points_range=(1e3, 8e3))
    _same(items, params(spatial, temporal, 0.0, cfl=0.4), precision, steps=5)


N, K, D = 48, 44, 0.25  # cells of a period, periods per direction, grid spacing


def _surface(x, y, z):
    k = 2 * np.pi / (N * D)
    return z - 0.031 - 0.5 * np.cos(k * x) - 0.4 * np.sin(k * y)


def _advected(g, dom, p):
    v = FunctorVelocity(1)
    v.set_rate(0, -1.0)
    v.set_square(0, 0, 0.3, 0.1)
    ctx = Context(0, 1)
    ctx.set_grid(g)
    ctx.set_level_set_count(1)
    ctx.upload(0, dom)
    ctx.set_velocity(v.descriptor())
    r = ctx.advect(p)
    idx, val, _ = ctx.download(0)
    ctx.close()
    return r, idx, val


def _grid(n):
    return Grid(None, [BC.PERIODIC_BOUNDARY, BC.PERIODIC_BOUNDARY, BC.INFINITE_BOUNDARY], D,
                index_min=[0, 0, -24], index_max=[n, n, 24])


@pytest.mark.parametrize("spatial,temporal", [(11, 2), (1, 0)])
def test_tiles_of_large_level_sets(spatial, temporal):
    """44 x 44 copies of a periodic surface (about 280,000 bricks, over 256 list
    entries per block of a pass) advance as the one copy does."""
    g = _grid(N)
    one = sdf_levelset(g, _surface, [0, 0, -10], [N - 1, N - 1, 10], lipschitz=1.5)
    off = np.stack(np.meshgrid(np.arange(K), np.arange(K), indexing="ij"), -1).reshape(-1, 2) * N
    idx = np.repeat(one.idx[None], len(off), 0)
    idx[:, :, :2] += off[:, None, :].astype(np.int32)
    idx = idx.reshape(-1, 3)
    val = np.tile(one.values, len(off))
    order = np.lexsort((idx[:, 0], idx[:, 1], idx[:, 2]))
    idx, val = np.ascontiguousarray(idx[order]), val[order]
    rs, sg = make_runs(idx, lambda x, y, z: np.where(_surface(x * D, y * D, z * D) < 0, -1, 1),
                       [0, 0, -11], [N * K - 1, N * K - 1, 11])
    big = Domain(_grid(N * K), idx, val, rs, sg, one.width)
    p = params(spatial, temporal, 0.3, cfl=0.4)
    r1, i1, v1 = _advected(g, one, p)
    r2, i2, v2 = _advected(big.grid, big, p)
    assert r2.number_of_time_steps == r1.number_of_time_steps
    assert r2.advected_time == r1.advected_time
    assert r2.point_updates == K * K * r1.point_updates
    assert len(v2) == K * K * len(v1)
    dense = np.full((N, N, 64), np.nan)
    dense[i1[:, 0], i1[:, 1], i1[:, 2] + 32] = v1
    assert np.array_equal(dense[i2[:, 0] % N, i2[:, 1] % N, i2[:, 2] + 32].view(np.int64),
                          v2.view(np.int64))


@pytest.mark.parametrize("spatial,temporal,cfl", [(7, 1, 0.4), (11, 2, 0.4), (8, 2, 0.4)])
def test_point_data_on_grid_faces(spatial, temporal, cfl):
    """Faces on grid planes (values of exactly 0, equal neighbours everywhere):
    the source of every point's data against the oracle."""
    from parity_cases import compare, run_gpu, run_oracle

    g = Grid(None, [BC.PERIODIC_BOUNDARY, BC.PERIODIC_BOUNDARY, BC.INFINITE_BOUNDARY], D,
             index_min=[0, 0, -24], index_max=[24, 21, 24])

    def steps(x, y, z):
        q = np.maximum(np.maximum(np.abs(x - 3.0) - 1.5, np.abs(y - 2.5) - 1.25), z - 1.0)
        return np.minimum(z, q)

    dom = sdf_levelset(g, steps, [0, 0, -8], [23, 20, 10], lipschitz=1.8)
    v = FunctorVelocity(1)
    v.set_rate(0, -1.0)
    p = params(spatial, temporal, 0.4, cfl=cfl, save_advection_velocities=1, max_steps=40)
    ols, ro = run_oracle(g, [dom], v, p)
    for _ in range(3):
        ctx, rg = run_gpu(g, [dom], v, p)
        assert rg.number_of_time_steps == ro.number_of_time_steps
        compare(ols, ctx)
        for got, want in zip(ctx.download_point_data(0), ols[-1].point_data()):
            assert np.array_equal(got, want)
        ctx.close()
