"""Steps interrupted by trial steps whose snapshot is put back: the next step
bins anew from the positions instead of going on with the cell ids and counts the
last one left, and gives the same bits and counters; on Verlet lists, whose
lists are rebuilt then, the state itself is what it was."""
import numpy as np
import pytest

from helpers import gpu_context, initial, params
from test_gpu_cell_lists import clustered

pytestmark = pytest.mark.gpu

F32 = 1


@pytest.mark.parametrize("model", [1, 2])
@pytest.mark.parametrize("stepper", [1, 2])
@pytest.mark.parametrize("n,dense", [(257, False), (20000, True)])
def test_cell_steps_binned_anew_give_the_same_bits(model, stepper, n, dense):
    x = clustered(model, n, 3) if dense else initial(model, n, 3)
    out = []
    for trial in (False, True):
        with gpu_context(params(model, n), precision=F32, variant=2, seed=2) as ctx:
            ctx.set_state(x)
            for k in range(3):
                ctx.steps(stepper, 0.0, 0.005, 3)
                if trial:
                    ctx.autotune(stepper, 0.005, steps=2)
            ctx.step(stepper, 0.0, 0.005)
            out.append((ctx.get_state(), ctx.step_counter, ctx.rebuild_count))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    assert out[0][1:] == out[1][1:]


@pytest.mark.parametrize("model", [1, 2])
def test_trial_steps_leave_a_verlet_state_as_it_was(model):
    n = 20000
    p = params(model, n)
    r = 1.3 * p["rho"]
    with gpu_context(p, precision=F32, variant=4, seed=2, r_max=r, nc_verlet=int(1.0 / r)) as ctx:
        ctx.set_state(clustered(model, n, 3))
        ctx.steps(2, 0.0, 0.005, 4)
        before = (ctx.get_state(), ctx.step_counter, ctx.verlet_state()[0])
        ctx.autotune(2, 0.005, steps=3)
        after = (ctx.get_state(), ctx.step_counter, ctx.verlet_state()[0])
    np.testing.assert_array_equal(before[0], after[0])
    assert before[1:] == after[1:]
