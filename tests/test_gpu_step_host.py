"""One step of a page-locked host array against upload, step and download: the
same bits and step counter, for every kind of neighbour search; and a
step that fails leaves the array as it was."""
import numpy as np
import pytest

import spsslangevinintegration_gb300 as spss
from helpers import gpu_context, initial, params

pytestmark = pytest.mark.gpu

F32 = 1


def context(model, n, variant):
    p = params(model, n)
    if variant == 4:
        r = 1.3 * p["rho"]
        p.update(r_max=r, nc_verlet=max(3, int(1.0 / r)))
    return gpu_context(p, precision=F32, variant=variant, seed=7)


@pytest.mark.parametrize("model,variant", [(1, 1), (2, 1), (1, 2), (2, 2), (1, 4), (2, 4), (1, 5)])
@pytest.mark.parametrize("n", [64, 257, 3000])
def test_bits_of_upload_step_download(n, model, variant):
    x0 = initial(model, n, 5)
    with context(model, n, variant) as a, context(model, n, variant) as b:
        host = spss.PinnedArray(a.length)
        host.array[:] = x0.reshape(-1)
        want = x0.reshape(-1).copy()
        for k in range(12):
            stepper = 1 + k % 2
            a.step_host(stepper, host.array, 0.0, 0.02)
            b.set_state(want)
            b.step(stepper, 0.0, 0.02)
            want = b.get_state().reshape(-1)
            np.testing.assert_array_equal(host.array, want)
            assert a.step_counter == b.step_counter


@pytest.mark.parametrize("variant", [1, 2, 4])
def test_a_failed_step_leaves_the_array(variant):
    n = 1000
    with context(2, n, variant) as ctx:
        host = spss.PinnedArray(ctx.length)
        host.array[:] = initial(2, n, 6).reshape(-1)
        host.array[2::6] = 1.0e6  # a displacement no fixed-point increment holds
        before = host.array.copy()
        with pytest.raises(Exception):
            ctx.step_host(1, host.array, 0.0, 0.02)
        np.testing.assert_array_equal(host.array, before)
