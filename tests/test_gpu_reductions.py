"""The GPU path's order parameters (tables and direct evaluation) against
extended-precision sums of the downloaded state, and frames into page-locked
and pageable memory.

Tolerance of the order parameters: a term carries at most a few units of
2^-53 (the phase is a 32-bit integer on the device; the downloaded phase
rounds to about 1e-15 at |phi| <= 10), so the means agree within 1e-14, and
the arguments within 1e-14 / |R|."""
import numpy as np
import pytest

from helpers import gpu_context, initial, params

pytestmark = pytest.mark.gpu

F32 = 1


def aligned(model, n, seed):
    rng = np.random.default_rng(seed)
    x = initial(model, n, seed).reshape(n, -1)
    phi = rng.normal(0.4, 0.7, n)
    x[:, -2] = phi
    if model == 2:
        speed = 10.0 ** rng.uniform(-25.0, 8.0, n)  # float range, squares far outside it
        speed[1:: max(2, n // 7)] = 0.0
        x[:, 2], x[:, 3] = speed * np.cos(phi), speed * np.sin(phi)
    return x.reshape(-1)


def expected(x, model):
    x = x.reshape(-1, 4 if model == 1 else 6).astype(np.longdouble)
    z = [np.cos(x[:, -2]).mean(), np.sin(x[:, -2]).mean()]
    if model == 2:
        v = np.sqrt(x[:, 2] ** 2 + x[:, 3] ** 2)
        ok = v > 0
        z += [(x[ok, 2] / v[ok]).sum() / len(v), (x[ok, 3] / v[ok]).sum() / len(v)]
    else:
        z += z
    return np.array([np.hypot(z[0], z[1]), np.arctan2(z[1], z[0]), np.hypot(z[2], z[3]), np.arctan2(z[3], z[2])],
                    dtype=np.float64)


@pytest.mark.parametrize("model", [1, 2])
@pytest.mark.parametrize("n", [1, 255, 257, 20011, 49999, 50000, 400001])
def test_order_parameters_match_extended_sums(model, n):
    x = aligned(model, n, n)
    with gpu_context(params(model, n), precision=F32, variant=2) as ctx:
        ctx.set_state(x)
        got, state = ctx.order_parameters(), ctx.get_state()
        per_system = ctx.system_order_parameters()[0]
    ref = expected(state, model)
    smallest = max(min(ref[0], ref[2]), 1e-300)
    np.testing.assert_allclose(got, ref, rtol=0.0, atol=1e-14 / smallest)
    # the sampling kernel normalises the velocities the same way (its phases are the FP32 records)
    if model == 2:
        np.testing.assert_allclose(per_system[2:], ref[2:], rtol=0.0, atol=1e-14 / smallest)


@pytest.mark.parametrize("model", [1, 2])
@pytest.mark.parametrize("wrapped", [False, True])
@pytest.mark.parametrize("n", [1, 257, 1003])
def test_frame_into_pinned_memory_equals_pageable(model, wrapped, n):
    from spsslangevinintegration_gb300 import PinnedArray, _native as N
    from spsslangevinintegration_gb300 import observers

    with gpu_context(params(model, n), precision=F32, variant=2) as ctx:
        ctx.set_state(aligned(model, n, n + 1))
        ref = observers.frame(ctx, wrapped=wrapped)
        with PinnedArray(ctx.length + 1, np.float32) as buf:
            for shift in (0, 1):  # 16-byte aligned rows, and not
                a = buf.array[shift:shift + ctx.length]
                a[:] = np.nan
                N.check(ctx.L.spss_frame_async(ctx.h, int(wrapped), N.fptr(a), a.size), "spss_frame_async")
                ctx.synchronize()
                np.testing.assert_array_equal(a, ref)
