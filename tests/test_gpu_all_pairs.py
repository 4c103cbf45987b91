"""The sliced all-pairs scan of the GPU path at the edges of its blocks (32
particles) and slices (sixteenths of a system), against the FP64 oracle on the
GPU's normals (one-step tolerance of test_gpu_fast_parity.py), and batches
whose systems share blocks."""
import numpy as np
import pytest

from helpers import gpu_context, initial, oracle_system, params
from test_gpu_fast_parity import state_err

pytestmark = pytest.mark.gpu

F32 = 1


@pytest.mark.parametrize("model", [1, 2])
@pytest.mark.parametrize("stepper", [1, 2])
@pytest.mark.parametrize("n", [1, 15, 32, 33, 500, 1025])
def test_all_pairs_slices_match_oracle(model, stepper, n):
    p = params(model, n)
    p["rho"] = 0.31
    x0 = initial(model, n, n, v=p["v0"])
    orc = oracle_system(p)
    with gpu_context(p, precision=F32, variant=1, seed=4) as ctx:
        ctx.set_state(x0)
        x = x0.copy()
        for k in range(2):
            normals = ctx.noise(stepper, k)
            ctx.step(stepper, 0.0, 0.005)
            orc.step(stepper, 1, x, 0.0, 0.005, normals)
        assert state_err(ctx.get_state(), x, 4 if model == 1 else 6).max() <= 1e-5


@pytest.mark.parametrize("stepper", [1, 2])
def test_all_pairs_batch_equals_single_contexts(stepper):
    """Systems that share a block of 32 particles with their neighbours in the batch."""
    from spsslangevinintegration_gb300 import Batch, Context

    sizes = (1, 7, 40, 300, 2, 129)
    systems, xs = [], []
    for r, n in enumerate(sizes):
        systems.append(dict(model=2, n=n, rho=0.3, precision=F32, variant=1, v0=0.1, xi_r=1.0, xi_phi=1.0,
                            D_phi=0.1 * r, sigma=1.0 + r, seed=6, replica=r))
        xs.append(initial(2, n, r))
    with Batch(systems) as b:
        b.set_state(np.concatenate(xs))
        b.run(stepper, 0.0, 0.005, 5)
        out = b.get_state()
        for r, s in enumerate(systems):
            kw = dict(s)
            with Context(kw.pop("model"), kw.pop("n"), kw.pop("rho"), **kw) as ctx:
                ctx.set_state(xs[r])
                ctx.steps(stepper, 0.0, 0.005, 5)
                np.testing.assert_array_equal(ctx.get_state(), b.system_rows(out, r))
