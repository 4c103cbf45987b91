"""Velocity directions with a subnormal component beside a large one, against
FP64 (the FP32 components are exact in it; a direction carries a few units of
2^-53 of each component: 2e-15)."""
import numpy as np
import pytest

from helpers import gpu_context, initial, params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 40])
@pytest.mark.parametrize("v", [(1.0, 1e-40), (-1.5, 3e-45), (2.0, -1.1e-38), (1e30, 1e-9), (3.0, 1.17549435e-38)])
def test_the_small_component_is_kept(v, n):
    x = initial(2, n, n).reshape(n, 6)
    x[:, 2:4] = v
    with gpu_context(params(2, n), precision=1, variant=2) as ctx:
        ctx.set_state(x.reshape(-1))
        got = [ctx.order_parameters(), ctx.system_order_parameters()[0]]
    vx, vy = (float(np.float32(c)) for c in v)
    want = np.arctan2(vy, vx)
    for g in got:
        assert abs(g[2] - 1.0) <= 2e-15
        assert abs(g[3] - want) <= 2e-15 * abs(want)
        assert (np.sin(g[3]) == 0.0) == (vy == 0.0)
