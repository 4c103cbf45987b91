"""FP64 torques from sums of directions: more neighbours than the integer sums
hold before they are emptied (511 a thread; all pairs spreads a particle over
64 threads), the complementary force, a nonzero alpha, and phases that are not
numbers, against the pair sums in extended precision for some particles.

Tolerance: a direction carries 3e-16 (the sine and cosine) and 2^-55; the mean
over the neighbours no more than that, times at most four such terms: 2e-15 of
sigma, and of the largest |omega_j - omega_i| (below 10 here) for the
complementary force."""
import numpy as np
import pytest

from helpers import gpu_context, params

pytestmark = pytest.mark.gpu


def wrapped(d):
    return d - np.rint(d)


def expected(x, model, rho, alpha, some):
    phi = x[:, -2].astype(np.longdouble)
    torque, force = [], []
    for i in some:
        dx, dy = wrapped(x[:, 0] - x[i, 0]), wrapped(x[:, 1] - x[i, 1])
        near = dx * dx + dy * dy <= rho * rho
        near[i] = False
        d = phi[near] - phi[i] - np.longdouble(alpha)
        dw = x[near, -1] - x[i, -1]
        torque.append(float(np.sin(d).mean()) if near.any() else 0.0)
        force.append(float((dw * np.cos(d)).mean()) if near.any() else 0.0)
    return np.array(torque), np.array(force)


@pytest.mark.parametrize("model", [1, 2])
@pytest.mark.parametrize("variant,n,rho", [(1, 33, 0.2), (1, 70000, 0.48), (2, 4000, 0.3), (2, 30000, 0.02), (3, 2500, 0.32),
                                           (4, 5000, 0.25)])
@pytest.mark.parametrize("alpha", [0.0, 0.4])
def test_torque_and_complementary_force(model, variant, n, rho, alpha):
    if np.finfo(np.longdouble).precision <= 15:
        pytest.skip("no extended precision here")
    rng = np.random.default_rng(n)
    s = 4 if model == 1 else 6
    x = np.zeros((n, s))
    x[:, 0], x[:, 1] = rng.random(n), rng.random(n)
    x[:, -2], x[:, -1] = rng.uniform(-30.0, 30.0, n), rng.normal(0.0, 1.0, n)
    p = dict(params(model, n), rho=rho, alpha=alpha, sigma=1.0)
    p["xi" if model == 1 else "xi_phi"] = 0.0
    r_max = rho + 0.01
    zero = np.zeros(n * s)
    with gpu_context(p, precision=0, variant=variant, r_max=r_max, nc_verlet=int(1.0 / r_max)) as ctx:
        ctx.set_higher_order(True)
        k = ctx.evaluate_rhs(variant, x.reshape(-1), zero, zero, 0.0, 0.01).reshape(n, s)
        force = ctx.complementary_force()
    some = rng.choice(n, min(n, 40), replace=False)
    torque, want = expected(x, model, rho, alpha, some)
    np.testing.assert_allclose(k[some, -1], torque, rtol=0.0, atol=2e-15)
    np.testing.assert_allclose(force[some], want, rtol=0.0, atol=2e-14)


@pytest.mark.parametrize("variant", [1, 2, 4])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_a_phase_that_is_no_number_reaches_its_neighbours(variant, value):
    n, rho = 500, 0.1
    rng = np.random.default_rng(3)
    x = np.zeros((n, 4))
    x[:, 0], x[:, 1], x[:, 2] = rng.random(n), rng.random(n), rng.uniform(-3.0, 3.0, n)
    x[7, 2] = value
    zero = np.zeros(4 * n)
    p = dict(params(1, n), rho=rho)
    with gpu_context(p, precision=0, variant=variant, r_max=0.11, nc_verlet=9) as ctx:
        k = ctx.evaluate_rhs(variant, x.reshape(-1), zero, zero, 0.0, 0.01).reshape(n, 4)
    dx, dy = wrapped(x[:, 0] - x[7, 0]), wrapped(x[:, 1] - x[7, 1])
    near = dx * dx + dy * dy <= rho * rho
    np.testing.assert_array_equal(np.isnan(k[:, 3]), near)
