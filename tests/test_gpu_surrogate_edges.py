"""The fused training kernel and the tiled forward kernel at the edges of their
tiles (128 rows) and grids (304 CTAs), with the tolerances of
test_gpu_surrogate.py (BF16 operands, FP32 accumulation)."""
import numpy as np
import pytest

from oracle import mlp_oracle as mo
from test_gpu_surrogate import data, tensors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 129, 304 * 128, 304 * 128 + 1, 70001])
def test_forward_rows_do_not_depend_on_their_tile(n):
    """Every row's output equals that row evaluated among the first rows of a smaller call."""
    from spsslangevinintegration_gb300.surrogate import Network

    x, _ = data(n, seed=n)[:2]
    with Network(seed=3) as net:
        y = net.forward(x)
        take = np.unique(np.r_[0, n - 1, np.random.default_rng(0).integers(0, n, 200)])
        np.testing.assert_array_equal(y[take], net.forward(x[take]))
        ref, _ = mo.forward(net.params.astype(np.float64), x[take], bf16=True)
    assert np.all(np.abs(y[take] - ref) <= 5e-3 * (1.0 + np.abs(ref)))


@pytest.mark.parametrize("n", [1, 127, 129, 304 * 128 + 200])
def test_gradient_at_tile_edges(n):
    """The last size gives some CTAs a second tile to accumulate."""
    from spsslangevinintegration_gb300.surrogate import Network

    x, t = data(n, seed=n)[:2]
    w = [1.0, 0.5, 2.0, 0.25]
    with Network(seed=4) as net:
        loss, grad = net.gradient(x, t, w)
        grad = grad.astype(np.float64)
        ref_loss, ref = mo.loss_and_gradient(net.params.astype(np.float64), x, t, np.array(w), bf16=True)
    assert abs(loss - ref_loss) <= 5e-3 * abs(ref_loss)
    for name, g in tensors(grad).items():
        r = tensors(ref)[name]
        assert np.linalg.norm(g - r) <= 0.03 * np.linalg.norm(r), name
