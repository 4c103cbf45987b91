"""The table-driven FP64 sine, cosine, logarithm and square root of the FP64
path, through what the library returns: the derivative's v0 cos phi and v0 sin
phi, and the FP64 normals, against extended-precision evaluation.

Tolerances: sine and cosine carry the roundings of a table entry, of the
correction and of their sum, at most 1.5 units of 2^-53 of a result near 1
(3e-16 absolute), and 4e-16 relative for a small angle, whose table entry is
exact.  A normal is r cos or r sin with r <= 6.7: a few units of 2^-53 of r
(5e-15 absolute)."""
import numpy as np
import pytest

from helpers import gpu_context, params

pytestmark = pytest.mark.gpu


def angles():
    rng = np.random.default_rng(0)
    k = np.arange(-600, 601)
    near = np.concatenate([k * np.pi / 128.0 + d for d in (0.0, 1e-9, -1e-9, np.pi / 256.0, -np.pi / 256.0)])
    return np.concatenate([near, rng.uniform(-10.0, 10.0, 20000), rng.uniform(-4096.0, 4096.0, 20000),
                           rng.uniform(-1e6, 1e6, 2000), [4096.0, -4096.0, 4096.1, -4096.1, 0.0],
                           10.0 ** rng.uniform(-300.0, -2.0, 2000)])


def test_sine_and_cosine_match_extended_precision():
    if np.finfo(np.longdouble).precision <= 15:
        pytest.skip("no extended precision here")
    phi = angles()
    n = phi.size
    x = np.zeros((n, 4))
    rng = np.random.default_rng(1)
    x[:, 0], x[:, 1], x[:, 2] = rng.random(n), rng.random(n), phi
    x = x.reshape(-1)
    with gpu_context(dict(params(1, n), v0=1.0), precision=0, variant=2) as ctx:
        k = ctx.evaluate_rhs(2, x, np.zeros_like(x), np.zeros_like(x), 0.0, 0.01).reshape(n, 4)
    ref_c, ref_s = np.cos(phi.astype(np.longdouble)), np.sin(phi.astype(np.longdouble))
    assert np.abs(k[:, 0] - ref_c).max() <= 3e-16
    assert np.abs(k[:, 1] - ref_s).max() <= 3e-16
    small = (np.abs(phi) < 0.01) & (phi != 0.0)
    assert (np.abs(k[small, 1] - ref_s[small]) <= 4e-16 * np.abs(ref_s[small])).all()


@pytest.mark.parametrize("model,stepper", [(1, 1), (1, 2), (2, 1), (2, 2)])
def test_normals_match_extended_precision(model, stepper):
    if np.finfo(np.longdouble).precision <= 15:
        pytest.skip("no extended precision here")
    n, seed, step = 60000, 77, 5
    with gpu_context(params(model, n), precision=0, variant=2, seed=seed) as ctx:
        z = ctx.noise(stepper, step).reshape(n, -1)
    c = [np.arange(n, dtype=np.uint64), np.full(n, step, np.uint64), np.zeros(n, np.uint64), np.zeros(n, np.uint64)]
    pairs = []
    for block in range(2):
        w = philox([c[0], c[1], c[2], np.full(n, block, np.uint64)], seed)
        pairs += [(w[0], w[1]), (w[2], w[3])]
    out = []
    two_pi = np.longdouble(2.0) * np.arccos(np.longdouble(-1.0))
    for a, b in pairs:
        u1 = (a.astype(np.longdouble) + 0.5) / np.longdouble(2.0) ** 32
        th = two_pi * (b.astype(np.longdouble) + 0.5) / np.longdouble(2.0) ** 32
        r = np.sqrt(-2.0 * np.log(u1))
        out += [r * np.cos(th), r * np.sin(th)]
    ref = np.stack(out, axis=1)[:, :z.shape[1]]
    assert np.abs(z - ref).max() <= 5e-15


def philox(c, seed):
    """Philox4x32-10 (Salmon et al., SC'11) on arrays of 32-bit words."""
    mask = np.uint64(0xFFFFFFFF)
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & mask, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & mask]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c
