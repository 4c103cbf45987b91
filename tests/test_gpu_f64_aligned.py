"""FP64 torques where the neighbours' phases are nearly or exactly the particle's
own, or opposite to it: every term is then far smaller than a cosine and a sine,
and has to be right to the last bits of itself, as sin(phi_j - phi_i - alpha) of
each pair is.  Against extended precision of the phases as given.

Tolerance, alpha = 0: a term is right to 4 units of 2^-53 of itself (a sine to 2,
or a direction to 2^-57 where the mean term is at least 1/32), the mean to as
many of the mean magnitude, and the last products round four times more: 8 units
of 2^-53 of the mean |sin|.  With alpha the sums of sines and cosines are rotated
in FP64: 8 units of 2^-53 of the mean |sin| + |cos| |sin alpha|.  The
complementary force: 8 units of the mean |(omega_j - omega_i)|."""
import numpy as np
import pytest

from helpers import gpu_context, params

pytestmark = pytest.mark.gpu

UNIT = 2.0 ** -53


def wrapped(d):
    return d - np.rint(d)


def phases(kind, spread, centre, n, rng):
    phi = centre + rng.uniform(-spread, spread, n)
    if kind == "opposite":
        phi[::2] += np.pi
    elif kind == "clusters":  # of the size of the particles' neighbourhoods, and a few phases anywhere
        phi += rng.integers(-3, 4, n) * (2.0 * np.pi)
        phi[::97] = rng.uniform(-30.0, 30.0, phi[::97].size)
    return phi


def run(variant, n, rho, model, alpha, phi, higher_order, seed=1):
    rng = np.random.default_rng(seed)
    s = 4 if model == 1 else 6
    x = np.zeros((n, s))
    x[:, 0], x[:, 1] = rng.random(n), rng.random(n)
    x[:, -2], x[:, -1] = phi, rng.normal(0.0, 1.0, n)
    p = dict(params(model, n), rho=rho, alpha=alpha, sigma=1.0)
    p["xi" if model == 1 else "xi_phi"] = 0.0
    r_max = rho + 0.01
    zero = np.zeros(n * s)
    with gpu_context(p, precision=0, variant=variant, r_max=r_max, nc_verlet=int(1.0 / r_max)) as ctx:
        ctx.set_higher_order(higher_order)
        k = ctx.evaluate_rhs(variant, x.reshape(-1), zero, zero, 0.0, 0.01).reshape(n, s)
        force = ctx.complementary_force() if higher_order else None
    return x, k[:, -1], force


def check(x, model, rho, alpha, some, torque, force):
    phi = x[:, -2].astype(np.longdouble)
    for i in some:
        dx, dy = wrapped(x[:, 0] - x[i, 0]), wrapped(x[:, 1] - x[i, 1])
        near = dx * dx + dy * dy <= rho * rho
        near[i] = False
        if not near.any():
            assert torque[i] == 0.0
            continue
        d = phi[near] - phi[i]
        want = np.sin(d - np.longdouble(alpha))
        size = np.abs(want).mean() + np.abs(np.cos(d)).mean() * abs(np.sin(alpha))
        assert abs(torque[i] - want.mean()) <= 8 * UNIT * size, (i, torque[i], want.mean())
        if force is not None:
            dw = x[near, -1] - x[i, -1]
            ref = (dw * np.cos(d - np.longdouble(alpha))).mean()
            assert abs(force[i] - ref) <= 8 * UNIT * np.abs(dw).mean()


@pytest.mark.parametrize("model", [1, 2])
@pytest.mark.parametrize("variant,n,rho", [(1, 700, 0.2), (1, 9, 0.4), (2, 4000, 0.05), (3, 500, 0.3), (4, 3001, 0.04)])
@pytest.mark.parametrize("kind", ["aligned", "opposite", "clusters"])
@pytest.mark.parametrize("spread", [0.3, 0.03, 1e-3, 1e-6, 1e-9, 1e-13])
def test_small_terms_are_right_to_their_last_bits(spread, kind, variant, n, rho, model):
    if np.finfo(np.longdouble).precision <= 18:
        pytest.skip("no quadruple precision here")
    rng = np.random.default_rng(n)
    for centre, alpha in ((0.0, 0.0), (2.0, 0.0), (-417.3, 0.0), (0.7, 0.4)):
        phi = phases(kind, spread, centre, n, rng)
        x, torque, force = run(variant, n, rho, model, alpha, phi, True)
        check(x, model, rho, alpha, rng.choice(n, min(n, 60), replace=False), torque, force)


@pytest.mark.parametrize("model", [1, 2])
@pytest.mark.parametrize("variant", [1, 2, 3, 4])
@pytest.mark.parametrize("centre", [0.0, 0.3, -2.7, 1e3, 3e7])
def test_equal_phases_give_no_torque(centre, variant, model):
    n = 600
    _, torque, _ = run(variant, n, 0.1, model, 0.0, np.full(n, centre), False)
    assert (torque == 0.0).all()


@pytest.mark.parametrize("variant", [1, 2, 4])
def test_phases_beyond_the_reduction(variant):
    """Neighbours above 2^20 have no fixed-point direction."""
    if np.finfo(np.longdouble).precision <= 18:
        pytest.skip("no quadruple precision here")
    n, rho = 1500, 0.06
    rng = np.random.default_rng(5)
    phi = rng.uniform(-3.0, 3.0, n)
    phi[::3] += 2.0 ** 21
    x, torque, force = run(variant, n, rho, 1, 0.0, phi, True)
    check(x, 1, rho, 0.0, rng.choice(n, 100, replace=False), torque, force)


@pytest.mark.parametrize("variant", [1, 2, 4])
def test_an_infinite_frequency_meets_its_own_cosine(variant):
    n, rho = 500, 0.1
    rng = np.random.default_rng(6)
    x = np.zeros((n, 4))
    x[:, 0], x[:, 1] = rng.random(n), rng.random(n)
    x[:, 2], x[:, 3] = rng.uniform(-3.0, 3.0, n), rng.normal(0.0, 1.0, n)
    x[7, 3] = np.inf
    zero = np.zeros(4 * n)
    with gpu_context(dict(params(1, n), rho=rho, sigma=1.0), precision=0, variant=variant, r_max=0.11, nc_verlet=9) as ctx:
        ctx.set_higher_order(True)
        ctx.evaluate_rhs(variant, x.reshape(-1), zero, zero, 0.0, 0.01)
        force = ctx.complementary_force()
    dx, dy = wrapped(x[:, 0] - x[7, 0]), wrapped(x[:, 1] - x[7, 1])
    near = dx * dx + dy * dy <= rho * rho
    near[7] = False
    np.testing.assert_array_equal(force[near], np.inf * np.cos(x[7, 2] - x[near, 2]))
    near[7] = True
    assert np.isfinite(force[~near]).all()


@pytest.mark.parametrize("model", [1, 2])
@pytest.mark.parametrize("kind", ["aligned", "clusters"])
@pytest.mark.parametrize("spread", [0.3, 1e-6])
@pytest.mark.parametrize("n,rho", [(4097, 0.06), (9001, 0.03), (9001, 0.2)])
def test_all_pairs_in_several_stretches(n, rho, spread, kind, model):
    """More candidates a warp than a lane remembers the hits of (2,048)."""
    if np.finfo(np.longdouble).precision <= 18:
        pytest.skip("no quadruple precision here")
    rng = np.random.default_rng(n)
    phi = phases(kind, spread, 0.4, n, rng)
    x, torque, force = run(1, n, rho, model, 0.0, phi, True)
    check(x, model, rho, 0.0, rng.choice(n, 60, replace=False), torque, force)
