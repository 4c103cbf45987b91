"""Order parameters whose terms are small: sines of phases a few quanta from a
multiple of a quarter turn, whose last bit is 2^-53.

Tolerance: the phase is a 32-bit integer on the device, its FP32 sine is right to
2^-23 of itself there, and everything after it is FP64: 2^-22 of the argument."""
import numpy as np
import pytest

from helpers import gpu_context, initial, params

pytestmark = pytest.mark.gpu

QUANTUM = 2.0 * np.pi / 2.0 ** 32


@pytest.mark.parametrize("k", [1, 2, 3, 5, 9, 100, 12345])
def test_arguments_of_a_few_quanta(k):
    x = initial(1, 1, 0).reshape(1, 4)
    for sign in (1, -1):
        x[0, 2] = QUANTUM * (sign * k + 0.25)  # uploads as the k-th quantum
        with gpu_context(params(1, 1), precision=1, variant=2) as ctx:
            ctx.set_state(x.reshape(-1))
            got = ctx.system_order_parameters()[0]
        assert abs(got[1] - sign * k * QUANTUM) <= 2.0 ** -22 * k * QUANTUM


@pytest.mark.parametrize("n", [2, 300, 5000])
def test_opposite_phases_cancel_exactly(n):
    """Half the particles at one phase, half opposite: no order is left but the FP32 sines' own last bits."""
    x = initial(1, n, 1).reshape(n, 4)
    x[:, 2] = 0.0
    x[::2, 2] = QUANTUM * 7.25
    x[1::2, 2] = -QUANTUM * 6.75
    with gpu_context(params(1, n), precision=1, variant=2) as ctx:
        ctx.set_state(x.reshape(-1))
        got = ctx.system_order_parameters()[0]
    assert got[1] == 0.0
