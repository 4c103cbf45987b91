"""Verlet lists longer than the capacity: the dense states of the list tests do
overflow it (counted here on the host), and every step of such a run equals the
FP64 oracle's from the same state, before and after the capacity has grown.

Tolerance: one step's, 1e-5 (test_gpu_fast_parity.py)."""
import math

import numpy as np
import pytest

from helpers import gpu_context, oracle_system, params
from test_gpu_cell_lists import clustered
from test_gpu_fast_parity import state_err

F32, VERLET = 1, 4


def capacity(n, r_max):
    """Entries a list is given at first: the mean, six standard deviations and room."""
    mean = math.pi * r_max * r_max * n
    return max(16, (math.ceil(mean + 6.0 * math.sqrt(mean) + 8.0) + 3) & ~3)


def longest(x, s, r_max):
    tree = pytest.importorskip("scipy.spatial").cKDTree(x.reshape(-1, s)[:, :2], boxsize=1.0)
    return tree.query_ball_point(tree.data, r_max, return_length=True).max() - 1


@pytest.mark.parametrize("model", [1, 2])
@pytest.mark.parametrize("n,seed", [(600, 600), (5000, 5000), (3000, 5), (40000, 5)])
def test_the_dense_states_overflow(model, n, seed):
    r_max = 1.3 * params(model, n)["rho"]
    assert longest(clustered(model, n, seed), 4 if model == 1 else 6, r_max) > capacity(n, r_max)


@pytest.mark.gpu
@pytest.mark.parametrize("model,stepper", [(1, 1), (1, 2), (2, 1), (2, 2)])
@pytest.mark.parametrize("n", [600, 5000, 40000])
def test_each_step_equals_the_oracle_from_the_same_state(model, stepper, n):
    p = params(model, n)
    r_max = 1.3 * p["rho"]
    s = 4 if model == 1 else 6
    orc = oracle_system(p, r_max=r_max, nc_verlet=int(1 / r_max))
    with gpu_context(p, precision=F32, variant=VERLET, seed=3, r_max=r_max, nc_verlet=int(1 / r_max)) as ctx:
        ctx.set_state(clustered(model, n, n))
        for k in range(4):
            x = ctx.get_state()
            normals = ctx.noise(stepper, k)
            ctx.set_should_update_lists(1)  # the grown lists are filled by the next build
            ctx.steps(stepper, 0.0, 0.005, 1)
            orc.should_update_lists = 1
            orc.step(stepper, VERLET, x, 0.0, 0.005, normals)
            assert state_err(ctx.get_state(), x, s).max() <= 1e-5
