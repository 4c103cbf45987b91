"""FP64 stochastic steps on neighbour lists against the oracle on the same
normals: sizes around the launches' 256 threads and the scan's tile, systems
sparse enough that particles without a neighbour keep a torque of zero, and
the trigger's accumulated displacement.

Tolerance: that of the trajectory tests, 1e-11 relative for a handful of
steps, 1e-12 for the accumulated displacement; rebuild flags are equal."""
import numpy as np
import pytest

from helpers import gpu_context, initial, oracle_system, params, per_component_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,stepper", [(1, 1), (1, 2), (2, 1), (2, 2)])
@pytest.mark.parametrize("variant", [2, 4])
@pytest.mark.parametrize("n,density", [(1, 0.1), (255, 0.2), (257, 2.0), (3000, 0.2), (9001, 2.0)])
def test_steps_match_the_oracle(n, density, variant, model, stepper):
    L = max(4.0, np.sqrt(n / density))
    p = params(model, n)
    p.update(rho=1.0 / L, v0=0.5 / L)
    if variant == 4:
        r = 1.25 / L
        p.update(r_max=r, nc_verlet=max(3, int(1.0 / r)))
    x0 = initial(model, n, n)
    dt = 0.05
    with gpu_context(p, variant=variant, seed=11) as ctx:
        orc = oracle_system(p)
        ctx.set_state(x0)
        x = x0.copy()
        t = 0.0
        for k in range(6):
            t += dt
            normals = ctx.noise(stepper, k)
            if k < 3:
                ctx.step(stepper, t, dt)
            else:
                ctx.steps(stepper, t - dt, dt, 1)
            orc.step(stepper, variant, x, t, dt, normals)
            if variant == 4:
                acc, flag, _ = ctx.verlet_state()
                assert flag == orc.should_update_lists
                assert abs(acc - orc.accumulated_displacement) <= 1e-12
        per_component_close(ctx.get_state(), x, 4 if model == 1 else 6, 1e-11, "state")
