"""The list flag cleared before any list was built: the reference's Verlet lists
are empty then, so no particle has a neighbour; its cell list is made by every
evaluation whatever the flag says.  And a state that was never given."""
import numpy as np
import pytest

from helpers import gpu_context, initial, params

pytestmark = pytest.mark.gpu


def context(model, n, precision, variant, **kw):
    p = params(model, n, D=0.0)
    if model == 2:
        p["D_r"] = 0.0
    r = 1.3 * p["rho"]
    return gpu_context(p, precision=precision, variant=variant, r_max=r, nc_verlet=max(1, int(1.0 / r)), seed=3, **kw)


@pytest.mark.parametrize("model", [1, 2])
@pytest.mark.parametrize("variant", [3, 4])
def test_fp64_verlet_lists_are_empty(model, variant):
    n = 4000
    x = initial(model, n, 1)
    with context(model, n, 0, variant) as ctx:
        ctx.set_should_update_lists(0)
        k = ctx.evaluate_rhs(variant, x, np.zeros_like(x), np.full_like(x, 7.0), 0.0, 0.01)
    s = 4 if model == 1 else 6
    np.testing.assert_array_equal(k.reshape(n, s)[:, -1], 7.0)  # untouched without a neighbour


@pytest.mark.parametrize("model", [1, 2])
@pytest.mark.parametrize("graph", [False, True])
def test_fp32_verlet_lists_are_empty(model, graph):
    n = 4000
    x = initial(model, n, 1)
    with context(model, n, 1, 4) as ctx:
        ctx.set_state(x)
        ctx.set_should_update_lists(0)
        if graph:
            ctx.steps(1, 0.0, 0.005, 1)
        else:
            ctx.step(1, 0.0, 0.005)
        got = ctx.get_state()
    s = 4 if model == 1 else 6
    np.testing.assert_array_equal(got.reshape(n, s)[:, -1], x.reshape(n, s)[:, -1].astype(np.float32))


@pytest.mark.parametrize("model", [1, 2])
def test_fp32_cells_are_binned_all_the_same(model):
    n = 4000
    x = initial(model, n, 1)
    out = []
    for keep in (False, True):
        with context(model, n, 1, 2) as ctx:
            ctx.set_state(x)
            if keep:
                ctx.set_should_update_lists(0)
            ctx.step(1, 0.0, 0.005)
            out.append((ctx.get_state(), ctx.rebuild_count, ctx.step_counter))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    assert out[0][1:] == out[1][1:]


@pytest.mark.parametrize("precision", [0, 1])
def test_a_state_never_given_can_be_read(precision):
    with context(2, 1000, precision, 4) as ctx:
        assert ctx.get_state().shape == (6000,)
