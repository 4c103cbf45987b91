"""Cell-list steps where their binning, ranks and runs can go wrong: grids of a
few cells a side, dense clusters (runs far longer than a group, cells of more
than 64 members), more cells than one scan tile, block edges, and steps on an
earlier binning, against the FP64 oracle on the GPU's normals (one-step tolerance
of test_gpu_fast_parity.py) and against the same steps run another way."""
import numpy as np
import pytest

from helpers import gpu_context, initial, oracle_system, params
from test_gpu_fast_parity import state_err

pytestmark = pytest.mark.gpu

F32, CELLS = 1, 2


def clustered(model, n, seed):
    """Half of the particles in five clusters about a cell wide."""
    rng = np.random.default_rng(seed)
    x = initial(model, n, seed).reshape(n, -1)
    rho = params(model, n)["rho"]
    half = n // 2
    centre = rng.random((5, 2))[rng.integers(0, 5, half)]
    x[:half, :2] = centre + rng.normal(0.0, 0.5 * rho, (half, 2))
    x[:half, :2] -= np.floor(x[:half, :2])
    return x.reshape(-1)


@pytest.mark.parametrize("model", [1, 2])
@pytest.mark.parametrize("stepper", [1, 2])
@pytest.mark.parametrize("n,rho,dense", [(1, 0.3, False), (127, 0.45, False), (129, 0.3, True), (500, 0.21, True),
                                         (3000, None, True), (9001, None, False), (20000, None, True)])
def test_steps_match_oracle(model, stepper, n, rho, dense):
    p = params(model, n)
    if rho is not None:
        p["rho"] = rho
    x = clustered(model, n, n) if dense else initial(model, n, n, v=p["v0"])
    orc = oracle_system(p)
    with gpu_context(p, precision=F32, variant=CELLS, seed=9) as ctx:
        ctx.set_state(x)
        for k in range(2):
            normals = ctx.noise(stepper, k)
            ctx.step(stepper, 0.0, 0.005)
            orc.step(stepper, CELLS, x, 0.0, 0.005, normals)
        assert state_err(ctx.get_state(), x, 4 if model == 1 else 6).max() <= 1e-5


@pytest.mark.parametrize("model", [1, 2])
def test_graph_single_and_interrupted_steps_agree(model):
    """Graph steps, single steps, and single steps with the state taken out and
    put back in between (which bins anew) give the same bits."""
    n = 20000
    x = clustered(model, n, 3)
    out = []
    for how in range(3):
        with gpu_context(params(model, n), precision=F32, variant=CELLS, seed=2) as ctx:
            ctx.set_state(x)
            if how == 0:
                ctx.steps(1, 0.0, 0.005, 6)
            else:
                for k in range(6):
                    ctx.step(1, 0.0, 0.005)
                    if how == 2 and k == 2:
                        ctx.order_parameters()
                        ctx.set_tiling(48)
            out.append((ctx.get_state(), ctx.step_counter, ctx.rebuild_count))
    for got, steps, builds in out[1:]:
        np.testing.assert_array_equal(got, out[0][0])
        assert (steps, builds) == out[0][1:]


def test_state_put_back_between_steps_continues():
    n = 5000
    p = params(2, n)
    x = initial(2, n, 4, v=p["v0"])
    orc = oracle_system(p)
    with gpu_context(p, precision=F32, variant=CELLS, seed=5) as ctx:
        ctx.set_state(x)
        ctx.steps(1, 0.0, 0.005, 3)
        y = ctx.get_state()
        ctx.set_state(y)
        normals = ctx.noise(1, 3)
        ctx.steps(1, 0.0, 0.005, 1)
        orc.step(1, CELLS, y, 0.0, 0.005, normals)
        assert state_err(ctx.get_state(), y, 6).max() <= 1e-5


def test_step_on_the_last_binning():
    """With the list flag cleared a single step uses the lists of the last binning;
    particles have moved by far less than a cell, so only pairs between cells that
    stopped or started being neighbours can differ: the step agrees with a
    re-binned one to that."""
    n = 5000
    p = params(2, n)
    x = initial(2, n, 6, v=p["v0"])
    out = []
    for keep in (False, True):
        with gpu_context(p, precision=F32, variant=CELLS, seed=5) as ctx:
            ctx.set_state(x)
            ctx.steps(1, 0.0, 0.005, 2)
            if keep:
                ctx.set_should_update_lists(0)
            ctx.step(1, 0.0, 0.005)
            ctx.step(1, 0.0, 0.005)
            assert ctx.step_counter == 4
            out.append(ctx.get_state())
    err = state_err(out[1], out[0], 6).max(axis=1)
    assert np.quantile(err, 0.99) <= 1e-6
