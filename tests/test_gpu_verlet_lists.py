"""Verlet lists by slot where they can go wrong: lists longer than the capacity
(the step scans the stencil, and the capacity grows between calls), slot
offsets that wrap around a system of more than 32,767 particles, one-CTA
rebuilds of small systems in a batch (sizes around its limits), against the FP64
oracle on the GPU's normals and against the same systems run alone."""
import numpy as np
import pytest

from helpers import gpu_context, initial, oracle_system, params
from test_gpu_cell_lists import clustered
from test_gpu_fast_parity import state_err

pytestmark = pytest.mark.gpu

F32, VERLET = 1, 4


def context(p, **kw):
    r_max = 1.3 * p["rho"]
    return gpu_context(p, precision=F32, variant=VERLET, r_max=r_max, nc_verlet=int(1 / r_max), **kw)


@pytest.mark.parametrize("model,stepper", [(1, 1), (1, 2), (2, 1), (2, 2)])
@pytest.mark.parametrize("n,dense", [(33, False), (600, True), (5000, True), (40000, False), (70000, False)])
def test_steps_match_oracle(model, stepper, n, dense):
    """Three calls, so the second and third run with the capacity grown."""
    p = params(model, n)
    x = clustered(model, n, n) if dense else initial(model, n, n, v=p["v0"])
    r_max = 1.3 * p["rho"]
    orc = oracle_system(p, r_max=r_max, nc_verlet=int(1 / r_max))
    with context(p, seed=3) as ctx:
        ctx.set_state(x)
        for k in range(3):
            normals = ctx.noise(stepper, k)
            ctx.steps(stepper, 0.0, 0.005, 1)
            orc.step(stepper, VERLET, x, 0.0, 0.005, normals)
            # compare step by step from the GPU's state, so that a pair at the cutoff does not add up
            assert state_err(ctx.get_state(), x, 4 if model == 1 else 6).max() <= 2e-5


@pytest.mark.parametrize("n", [3000, 40000])
def test_results_do_not_depend_on_when_the_capacity_grows(n):
    p = params(2, n)
    x = clustered(2, n, 5)
    out = []
    for chunks in ((60,), (1,) * 60, (7, 20, 33)):
        with context(p, seed=4) as ctx:
            ctx.set_state(x)
            for c in chunks:
                ctx.steps(2, 0.0, 0.005, c)
            out.append((ctx.get_state(), ctx.verlet_state()))
    for got in out[1:]:
        np.testing.assert_array_equal(got[0], out[0][0])
        assert got[1] == out[0][1]


@pytest.mark.parametrize("sizes", [(1, 31, 1024, 1025), (4096, 700, 2000), (4097, 1024, 300)])
@pytest.mark.parametrize("stepper", [1, 2])
def test_batches_of_small_systems_equal_single_contexts(sizes, stepper):
    """The last set holds a system beyond the one-CTA rebuild, so all take the
    general one.  Speeds differ, so the systems rebuild at different steps."""
    from spsslangevinintegration_gb300 import Batch, Context

    systems, xs = [], []
    for r, n in enumerate(sizes):
        p = params(2, n, v0=0.3 + 0.4 * r)
        r_max = 1.3 * p["rho"]
        kw = {k: p[k] for k in ("v0", "xi_r", "xi_phi", "D_r", "D_phi", "sigma")}
        systems.append(dict(model=2, n=n, rho=p["rho"], precision=F32, variant=VERLET, r_max=r_max,
                            nc_verlet=max(1, int(1 / r_max)), seed=6, replica=r, **kw))
        xs.append(clustered(2, n, r) if n > 900 else initial(2, n, r, v=p["v0"]))
    with Batch(systems) as b:
        b.set_state(np.concatenate(xs))
        for c in (1, 3, 80):
            b.run(stepper, 0.0, 0.005, c)
        out = b.get_state()
        assert b.rebuild_count > 2
        for r, s in enumerate(systems):
            kw = dict(s)
            with Context(kw.pop("model"), kw.pop("n"), kw.pop("rho"), **kw) as ctx:
                ctx.set_state(xs[r])
                ctx.steps(stepper, 0.0, 0.005, 84)
                np.testing.assert_array_equal(ctx.get_state(), b.system_rows(out, r))
