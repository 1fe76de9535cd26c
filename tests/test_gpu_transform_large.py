"""The ring of 131072 points, the one whose transforms are a cluster of sixteen blocks per limb: every prime class against the CPU
checker and back, and a rescale and an encryption for the fused ends."""
import numpy as np
import pytest

from gpu_util import rand_rows, seeds

pytestmark = pytest.mark.gpu

LOGN, N = 17, 1 << 17


def test_forward_and_inverse_against_the_checker(oracle_mod):
    import torch

    from lancelot_b200 import cabi

    mods = oracle_mod.coeff_modulus_create(N, [60, 59, 57, 50, 46, 43, 30])
    o, ctx = oracle_mod.Oracle(LOGN, mods, 0), cabi.Context(LOGN, mods, 0)
    rng = np.random.default_rng(LOGN)
    x = np.stack([rand_rows(rng, mods, N) for _ in range(2)])
    x[-1, :, : N // 2] = np.array(mods, dtype=np.uint64)[:, None] - 1
    d = cabi.to_device(x)
    ctx.ntt_forward(d, 2, len(mods), 0)
    assert np.array_equal(cabi.to_host(d), o.ntt_rows(x.copy(), 2, len(mods), 0).reshape(x.shape))
    ctx.ntt_inverse(d, 2, len(mods), 0)
    assert torch.equal(d, cabi.to_device(x))


def test_rescale_and_encryption(oracle_mod):
    from lancelot_b200 import cabi

    mods = oracle_mod.coeff_modulus_create(N, [60, 40, 50, 60])
    o, ctx = oracle_mod.Oracle(LOGN, mods, 1), cabi.Context(LOGN, mods, 1)
    rng = np.random.default_rng(LOGN)
    ct = np.stack([rand_rows(rng, mods[:3], N) for _ in range(2)])
    assert np.array_equal(cabi.to_host(ctx.rescale(3, cabi.to_device(ct))).reshape(2, 2, N), o.rescale(3, ct))
    pk = o.gen_pk(o.gen_sk(seeds(rng, 1)), seeds(rng, 1), seeds(rng, 1))
    pt, s = rand_rows(rng, mods[:3], N), seeds(rng, 2)
    got = cabi.to_host(ctx.encrypt_asymmetric(cabi.to_device(pk), cabi.to_device(pt), s)).reshape(2, 3, N)
    assert np.array_equal(got, o.encrypt_asym(pk, pt, s[:64], s[64:]))
