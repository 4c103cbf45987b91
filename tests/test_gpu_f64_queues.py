"""FP64 neighbour sums: many neighbours, particle numbers around the warp and
block sizes, pairs within the pre-test's margin of the cutoff (decided in
FP64), and coordinates several boxes away, against the oracle (the FP64 path's
tolerance, 1e-12)."""
import numpy as np
import pytest

from helpers import gpu_context, initial, oracle_system, params, per_component_close

pytestmark = pytest.mark.gpu


def edge_state(model, n, rho, seed):
    """Random positions, a quarter of them moved to a neighbour of another
    particle at rho (1 + eps), eps from -4e-5 to 4e-5 of the box, and every
    fifth particle whole boxes away."""
    rng = np.random.default_rng(seed)
    x = initial(model, n, seed).reshape(n, -1)
    for i in range(0, n - 1, 4):
        a = rng.uniform(0.0, 2.0 * np.pi)
        r = rho + rng.choice([-4e-5, -1e-5, -1e-9, 0.0, 1e-9, 1e-5, 4e-5])
        x[i + 1, 0] = x[i, 0] + r * np.cos(a)
        x[i + 1, 1] = x[i, 1] + r * np.sin(a)
    x[:, :2] -= np.floor(x[:, :2])
    x[::5, 0] += rng.integers(-3, 4, len(x[::5]))
    return x.reshape(-1)


@pytest.mark.parametrize("model", [1, 2])
@pytest.mark.parametrize("variant", [1, 2, 3, 4])
@pytest.mark.parametrize("n,rho,alpha", [(1, 0.1, 0.0), (31, 0.24, 0.0), (65, 0.2, 0.3), (700, 0.2, 0.0), (3001, 0.02, 0.2)])
def test_derivative_and_complementary_force(model, variant, n, rho, alpha):
    p = dict(params(model, n), rho=rho, alpha=alpha)
    x = edge_state(model, n, rho, n)
    if model == 2 and variant == 1:
        x = x.reshape(n, 6)
        x[:, :2] -= np.floor(x[:, :2])  # this routine takes the positions as they are
        x = x.reshape(-1)
    r_max = rho + 0.01
    zero = np.zeros_like(x)
    s = 4 if model == 1 else 6
    orc = oracle_system(p, r_max=r_max, nc_verlet=int(1.0 / r_max))
    orc.set_higher_order(True)
    with gpu_context(p, precision=0, variant=variant, r_max=r_max, nc_verlet=int(1.0 / r_max)) as ctx:
        ctx.set_higher_order(True)
        got = ctx.evaluate_rhs(variant, x, zero, zero, 0.0, 0.01)
        caf = ctx.complementary_force()
    ref = orc.evaluate(variant, x, zero, zero.copy(), 0.0, 0.01)
    per_component_close(got, ref, s, 1e-12, "k_next")
    np.testing.assert_array_equal(got == 0.0, ref == 0.0)  # the same particles have neighbours
    np.testing.assert_allclose(caf, orc.complementary_force(), rtol=1e-11, atol=1e-11)
