"""The transforms at every ring degree their schedules differ at, for each prime class and for batches that do and do not
fill the blocks that several polynomials share: forward against the CPU checker and back, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# 60 bits next to 2^60, 59 bits (the integer class without the cheap reduction), lazy integers, and the FP64 classes at both ends
BITS = [60, 59, 57, 50, 47, 46, 43, 41, 30]


@pytest.mark.parametrize("logn", [11, 12, 13, 14, 15, 16])
@pytest.mark.parametrize("batch", [1, 2, 5, 8])
def test_forward_and_inverse_against_the_checker(oracle_mod, logn, batch):
    import torch

    from lancelot_b200 import cabi

    n = 1 << logn
    mods = oracle_mod.coeff_modulus_create(n, BITS)
    o = oracle_mod.Oracle(logn, mods, 0)
    ctx = cabi.Context(logn, mods, 0)
    rng = np.random.default_rng(100 * logn + batch)
    x = np.empty((batch, len(mods), n), dtype=np.uint64)
    for r, q in enumerate(mods):
        x[:, r] = rng.integers(0, q, (batch, n), dtype=np.uint64)
        x[:, r, :4] = [0, 1, q - 1, q // 2]
    x[-1] = np.array(mods, dtype=np.uint64)[:, None] - 1  # every value at the top of its range
    d = cabi.to_device(x)
    ctx.ntt_forward(d, batch, len(mods), 0)
    assert np.array_equal(cabi.to_host(d), o.ntt_rows(x.copy(), batch, len(mods), 0).reshape(x.shape))
    ctx.ntt_inverse(d, batch, len(mods), 0)
    assert torch.equal(d, cabi.to_device(x))
