"""Sine and cosine of the FP64 path next to multiples of a quarter turn, where
one of them is as small as the remainder of the phase: v0 cos phi and v0 sin phi
of the derivative against extended precision.

Tolerance: a remainder rounded once, its polynomial and a product by +-1, at
most 2 ulp: 4.5e-16 of the small component; the other one 3e-16, as elsewhere."""
import numpy as np
import pytest

from helpers import gpu_context, params

pytestmark = pytest.mark.gpu


def phases():
    rng = np.random.default_rng(0)
    k = np.concatenate([np.arange(-2700, 2701), rng.integers(-600000, 600001, 3000)])
    k = k[k != 0].astype(np.float64)
    at = k * (0.5 * np.pi)  # within an ulp or two of the multiple itself
    out = [at, np.nextafter(at, np.inf), np.nextafter(at, -np.inf)]
    out += [at + rng.choice([-1.0, 1.0], at.size) * 10.0 ** rng.uniform(-15.0, -3.0, at.size) for _ in range(3)]
    return np.concatenate(out)


def test_the_small_component_is_right_to_an_ulp_of_itself():
    if np.finfo(np.longdouble).precision <= 18:
        pytest.skip("no quadruple precision here")
    phi = phases()
    n = phi.size
    x = np.zeros((n, 4))
    rng = np.random.default_rng(1)
    x[:, 0], x[:, 1], x[:, 2] = rng.random(n), rng.random(n), phi
    x = x.reshape(-1)
    with gpu_context(dict(params(1, n), v0=1.0), precision=0, variant=2) as ctx:
        k = ctx.evaluate_rhs(2, x, np.zeros_like(x), np.zeros_like(x), 0.0, 0.01).reshape(n, 4)
    wide = phi.astype(np.longdouble)
    for got, ref in ((k[:, 0], np.cos(wide)), (k[:, 1], np.sin(wide))):
        small = np.abs(ref) < 0.01
        err = np.abs(got - ref)
        assert (err[small] <= 4.5e-16 * np.abs(ref[small])).all()
        assert (err[~small] <= 3e-16).all()
