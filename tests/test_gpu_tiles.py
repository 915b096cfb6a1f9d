"""The tiled rate and update kernels and the deferred brick maintenance against
the oracle, bit for bit: forward Euler runs long enough for the surface to cross
bricks between two maintenances (every 10 - width steps)."""
import pytest

from parity_cases import compare, egg_velocity, params, run_gpu, run_oracle, sphere_case

pytestmark = pytest.mark.gpu


def _parity(g, lss, v, p):
    ols, ro = run_oracle(g, lss, v, p)
    ctx, rg = run_gpu(g, lss, v, p)
    assert rg.number_of_time_steps == ro.number_of_time_steps
    assert rg.advected_time == ro.advected_time
    assert rg.current_time_step == ro.current_time_step
    assert rg.point_updates == ro.point_updates
    compare(ols, ctx)
    return rg


@pytest.mark.parametrize("spatial", [0, 1, 2, 5, 7, 8, 10, 11])
def test_forward_euler_between_maintenances(spatial):
    g, lss = sphere_case(1.4, 0.2)
    r = _parity(g, lss, egg_velocity(), params(spatial, 0, 1.2, cfl=0.45))
    assert r.number_of_time_steps > 9
