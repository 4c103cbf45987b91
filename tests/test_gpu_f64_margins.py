"""The range pre-test of the FP64 path at and around its margin (1e-6 of the box
either side of the cutoff, two of them added to it), and for particles many boxes
away, against the oracle: the same neighbours (a term too few or too many shows
in the derivative at 1e-3) and the FP64 path's tolerance, 1e-12."""
import numpy as np
import pytest

from helpers import gpu_context, initial, oracle_system, params, per_component_close

pytestmark = pytest.mark.gpu

EPS = np.array([3e-8, 1e-7, 3e-7, 1e-6, 1.5e-6, 2e-6, 2.5e-6, 4e-6, 8e-6])


def edge_state(model, n, cut, boxes, seed):
    """Every other particle beside another one at the cutoff +- EPS, some of both
    `boxes` boxes away."""
    rng = np.random.default_rng(seed)
    x = initial(model, n, seed).reshape(n, -1)
    a = rng.uniform(0.0, 2.0 * np.pi, n // 2)
    a[::5] = np.round(a[::5] / (0.5 * np.pi)) * (0.5 * np.pi)  # along an axis too
    r = cut + rng.choice(np.concatenate([EPS, -EPS, [0.0]]), n // 2)
    x[1::2, 0] = x[0:2 * (n // 2):2, 0] + r * np.cos(a)
    x[1::2, 1] = x[0:2 * (n // 2):2, 1] + r * np.sin(a)
    x[:, :2] -= np.floor(x[:, :2])
    far = rng.random((n, 2)) < 0.3
    x[:, :2] += np.where(far, np.round(rng.uniform(-boxes, boxes, (n, 2))), 0.0)
    return x.reshape(-1)


def compare(model, variant, n, rho, r_max, x):
    s = 4 if model == 1 else 6
    p = dict(params(model, n), rho=rho)
    zero = np.zeros_like(x)
    orc = oracle_system(p, r_max=r_max, nc_verlet=int(1.0 / r_max))
    with gpu_context(p, precision=0, variant=variant, r_max=r_max, nc_verlet=int(1.0 / r_max)) as ctx:
        got = ctx.evaluate_rhs(variant, x, zero, zero, 0.0, 0.01)
    ref = orc.evaluate(variant, x, zero, zero.copy(), 0.0, 0.01)
    per_component_close(got, ref, s, 1e-12, "k_next")
    np.testing.assert_array_equal(got == 0.0, ref == 0.0)


@pytest.mark.parametrize("model", [1, 2])
@pytest.mark.parametrize("variant", [1, 2, 4])
@pytest.mark.parametrize("edge", ["rho", "r_max"])
@pytest.mark.parametrize("n,rho", [(1500, 0.02), (4000, 0.004)])
@pytest.mark.parametrize("boxes", [0, 10000])
def test_neighbours_at_the_margin(boxes, n, rho, edge, variant, model):
    if variant == 1 and (model == 2 and boxes or edge == "r_max"):
        pytest.skip("not a case of this routine")
    r_max = 1.3 * rho
    compare(model, variant, n, rho, r_max, edge_state(model, n, rho if edge == "rho" else r_max, boxes, n + variant))


@pytest.mark.parametrize("model", [1, 2])
@pytest.mark.parametrize("variant", [1, 2, 4])
@pytest.mark.parametrize("boxes", [2.0 ** 19, 2.0 ** 21, 1e11])
def test_neighbours_far_from_the_box(boxes, variant, model):
    if variant == 1 and model == 2:
        pytest.skip("this routine takes the positions as they are")
    n, rho = 6000, 0.01
    compare(model, variant, n, rho, 1.3 * rho, edge_state(model, n, rho, boxes, 7))
