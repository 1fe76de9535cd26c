"""Products, reductions and tensor products at the splits of a limb row among blocks and threads: rows shorter than a warp and than a
block, one block per row and several; against Python integers."""
import numpy as np
import pytest

from gpu_util import rand_rows

pytestmark = pytest.mark.gpu

BITS = [60, 59, 50, 40]  # near 2^60, integer, FP64


@pytest.mark.parametrize("logn", [4, 8, 9, 10, 12, 16])
@pytest.mark.parametrize("batch", [1, 3, 37])
def test_products_by_rows(oracle_mod, logn, batch):
    from lancelot_b200 import cabi

    n = 1 << logn
    mods = oracle_mod.coeff_modulus_create(n, BITS) if logn > 4 else oracle_mod.coeff_modulus_create(32, BITS)
    L, rng = len(mods), np.random.default_rng(10 * logn + batch)
    ctx = cabi.Context(logn, mods, 0)
    a, b = (np.stack([np.stack([rand_rows(rng, mods, n) for _ in range(2)]) for _ in range(batch)]) for _ in range(2))
    words = rng.integers(0, 2 ** 64, (batch, L, n), dtype=np.uint64)
    at = sorted({0, 1, n // 2 - 1, n // 2, n - 1, *(int(x) for x in rng.integers(0, n, 12))})
    q = np.array(mods, dtype=object)[:, None]
    A, B, W = (x[..., at].astype(object) for x in (a, b, words))
    got = cabi.to_host(ctx.multiply_poly(L, cabi.to_device(a), cabi.to_device(b))).reshape(a.shape)[..., at]
    assert np.array_equal(got.astype(object), A * B % q)
    got = cabi.to_host(ctx.reduce_mod(L, cabi.to_device(words))).reshape(words.shape)[..., at]
    assert np.array_equal(got.astype(object), W % q)
    got = cabi.to_host(ctx.multiply(L, cabi.to_device(a), cabi.to_device(b), batch=batch)).reshape(batch, 3, L, n)[..., at].astype(object)
    a0, a1, b0, b1 = A[:, 0], A[:, 1], B[:, 0], B[:, 1]
    for k, want in enumerate((a0 * b0, a0 * b1 + a1 * b0, a1 * b1)):
        assert np.array_equal(got[:, k], want % q), k
