"""The global-field step against its equations in FP64 from the downloaded
state: the first step on the field of an uploaded state, the second on the
field the first one left, a third on a new upload; sizes around the launch's
304 blocks of 256 threads.

Tolerance: the new angular velocity is rounded once to FP32 (2^-24 of it); its
increment is at most 5 dt = 0.025 with some twenty FP32 roundings, another
3e-8; the downloaded positions of the phases are exact to 1e-9.  So 2^-22 of
the largest angular velocity (at least 1)."""
import numpy as np
import pytest

from helpers import gpu_context, params

pytestmark = pytest.mark.gpu


def expected_omega(x, nu, sigma, alpha, xi, dt, srk):
    phi, w = x[:, 2], x[:, 3]
    Z, W = np.exp(1j * phi).mean(), (w * np.exp(1j * phi)).mean()
    SZ, KZ = np.abs(Z) * np.sin(np.angle(Z) - phi), np.abs(Z) * np.cos(np.angle(Z) - phi)
    ca, sa = np.cos(alpha), np.sin(alpha)
    f = -xi * w + nu + sigma * (ca * SZ - sa * KZ)
    out = w + f * dt
    if srk:
        sW, KW = np.sin(np.angle(W) - phi), np.abs(W) * np.cos(np.angle(W) - phi)
        C = sigma * (ca * KW + sa * np.abs(W) * sW - w * (ca * KZ + sa * np.abs(Z) * sW))
        out = out + 0.5 * dt * dt * (C - xi * f)
    return out


@pytest.mark.parametrize("stepper", [1, 2])
@pytest.mark.parametrize("n", [1, 255, 257, 77823, 77825, 200001])
def test_steps_follow_the_field_of_the_state(n, stepper):
    sigma, alpha, xi, dt = 1.5, 0.3, 0.4, 0.005
    rng = np.random.default_rng(n)
    x0 = np.column_stack([rng.random(n), rng.random(n), rng.normal(0.3, 0.8, n), rng.normal(0.5, 1.0, n)])
    nu = rng.normal(0.0, 0.5, n)
    p = dict(params(1, n, sigma=sigma, alpha=alpha, D=0.0), xi=xi)
    with gpu_context(p, precision=1, variant=5, seed=3) as ctx:
        ctx.set_natural_frequencies(nu)
        for start in (x0, x0[::-1]):
            ctx.set_state(np.ascontiguousarray(start).reshape(-1))
            x = ctx.get_state().reshape(n, 4)
            for k in range(2):
                if k == 0:
                    ctx.step(stepper, 0.0, dt)
                else:
                    ctx.steps(stepper, 0.0, dt, 1)
                y = ctx.get_state().reshape(n, 4)
                want = expected_omega(x, nu, sigma, alpha, xi, dt, stepper == 2)
                np.testing.assert_allclose(y[:, 3], want, rtol=0.0, atol=2.0 ** -22 * max(1.0, np.abs(want).max()))
                x = y
