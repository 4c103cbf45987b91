"""Velocity directions of the order parameters: zero, subnormal, huge and
missing (NaN) components, against FP64 sums of the same velocities.

Tolerance: a direction carries a few units of 2^-53 (1e-15)."""
import numpy as np
import pytest

from helpers import gpu_context, initial, params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [7, 300, 60001])
def test_directions_of_unusual_velocities(n):
    x = initial(2, n, n).reshape(n, 6)
    unusual = [(0.0, 0.0), (0.0, -2.0), (3.0e38, -1.0e38), (1.0e-41, 0.0), (np.nan, 1.0), (1.0, 1.0e-40), (-0.0, 5.0)]
    for k, v in enumerate(unusual):
        x[k::max(7, n // 40), 2:4] = v
    with gpu_context(params(2, n), precision=1, variant=2) as ctx:
        ctx.set_state(x.reshape(-1))
        got = [ctx.order_parameters(), ctx.system_order_parameters()[0]]
    v = x[:, 2:4].astype(np.float32).astype(np.float64)
    size = np.hypot(v[:, 0], v[:, 1])
    ok = size > 0.0
    z = (v[ok] / size[ok, None]).sum(axis=0) / n
    for g in got:
        np.testing.assert_allclose([g[2] * np.cos(g[3]), g[2] * np.sin(g[3])], z, rtol=0.0, atol=1e-14)


def test_an_infinite_velocity_has_no_direction():
    n = 100
    x = initial(2, n, 1).reshape(n, 6)
    x[5, 2] = np.inf
    with gpu_context(params(2, n), precision=1, variant=2) as ctx:
        ctx.set_state(x.reshape(-1))
        for g in (ctx.order_parameters(), ctx.system_order_parameters()[0]):
            assert np.isnan(g[2])
