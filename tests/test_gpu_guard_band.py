"""The GPU path's neighbour decision inside, at and outside its FP32 guard band
around r = rho, for radii from 2^-12 to 0.06 of the box and positions with random
low words: isolated pairs whose separation lies up to two band widths on either
side.  The decision is the FP64 one of the 64-bit positions; without noise and
friction a particle's omega changes if and only if its pair interacts, so every
decision is read off the state exactly."""
import numpy as np
import pytest

from helpers import gpu_context

pytestmark = pytest.mark.gpu

WORD = 2.0 ** -32


def pairs(rho, seed):
    """Pairs on a grid of cells too far apart to meet; AoS positions [2 m, 2]."""
    rng = np.random.default_rng(seed)
    g = min(64, int(1.0 / (4.5 * rho)))
    m = g * g
    base = (np.stack(np.meshgrid(np.arange(g), np.arange(g)), -1).reshape(-1, 2) + rng.random((m, 2)) * 0.01) / g
    width = 4.0 * WORD + 5.0 * rho * 2.0 ** -24  # of the band, as a distance
    off = rng.choice([-2.0, -1.5, -1.0, -0.75, -0.5, -0.25, -0.02, 0.02, 0.25, 0.5, 0.75, 1.0, 1.5, 2.0], m) * width
    a = rng.uniform(0.0, 2.0 * np.pi, m)
    a[::7] = np.round(a[::7] / (0.5 * np.pi)) * 0.5 * np.pi
    other = base + ((rho + off) * np.stack([np.cos(a), np.sin(a)])).T
    x = np.empty((2 * m, 2))
    x[0::2], x[1::2] = base, other
    x -= np.floor(x)
    return x[rng.permutation(m).repeat(2) * 2 + np.tile([0, 1], m)]


def inside(x, rho):
    """The FP64 decision from the fixed-point positions (2^-64 of the box)."""
    fixed = np.array([[int(v * 2.0 ** 64) for v in p] for p in x], dtype=object)
    d = (fixed[1::2] - fixed[0::2]) % 2 ** 64
    d = np.where(d >= 2 ** 63, d - 2 ** 64, d)
    e = np.array([[float(np.float64(int(v))) for v in p] for p in d]) * 2.0 ** -64
    return e[:, 0] * e[:, 0] + e[:, 1] * e[:, 1] <= rho * rho


@pytest.mark.parametrize("model,stepper", [(1, 1), (1, 2), (2, 1), (2, 2)])
@pytest.mark.parametrize("variant", [1, 2, 4])
@pytest.mark.parametrize("rho", [2.0 ** -12, 4.4e-4, 2.0 ** -9 * 1.1, 2.0 ** -6, 0.06])
def test_decisions_around_the_band(rho, variant, model, stepper):
    x2 = pairs(rho, int(1e6 * rho) + variant)
    n, s = len(x2), 4 if model == 1 else 6
    x = np.zeros((n, s))
    x[:, :2] = x2
    x[0::2, -2], x[1::2, -2] = 0.3, 1.5
    x[:, -1] = 0.25
    want = inside(x2, rho).repeat(2)
    assert 0.2 < want.mean() < 0.8
    r_max = 1.3 * rho
    p = dict(model=model, n=n, rho=rho, v0=0.0, sigma=1.0, xi=0.0, xi_r=0.0, xi_phi=0.0, D_r=0.0, D_phi=0.0)
    with gpu_context(p, precision=1, variant=variant, seed=2, r_max=r_max, nc_verlet=int(1.0 / r_max)) as ctx:
        ctx.set_state(x.reshape(-1))
        ctx.step(stepper, 0.0, 0.01)
        got = ctx.get_state().reshape(n, s)[:, -1]
    np.testing.assert_array_equal(got != 0.25, want)
