"""Encoding and decoding at every split of their transforms: the fused encode + encrypt (two-kernel inverse FFT from 4096 slots on)
against the two single calls word for word, decoding against the CPU checker."""
import numpy as np
import pytest

from gpu_util import rand_rows, seeds

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("logn,slots", [(13, 4096), (14, 8192), (15, 16384), (16, 32768), (14, 4096), (16, 8192), (12, 2048)])
@pytest.mark.parametrize("dtype", ["float32", "float64", "complex128"])
def test_fused_encoding(oracle_mod, logn, slots, dtype):
    import torch

    from lancelot_b200 import cabi

    n = 1 << logn
    mods = oracle_mod.coeff_modulus_create(n, [60, 40, 50, 51, 59, 33, 60])
    ctx = cabi.Context(logn, mods, 1)
    rng = np.random.default_rng(logn + slots)
    pk = ctx.gen_public_key(ctx.gen_secret_key(seeds(rng, 1)), seeds(rng, 1), seeds(rng, 1))
    batch, s, Q = 3, seeds(rng, 6), len(mods) - 1
    # small values, values whose coefficients pass 2^51 and 2^64, and fewer values than slots
    for scale, n_values in [(2.0 ** 40, slots), (2.0 ** 55, slots - 3), (2.0 ** 70, slots // 2 + 1)]:
        v = rng.uniform(-1, 1, (batch, n_values))
        v = torch.from_numpy(v + 1j * rng.uniform(-1, 1, v.shape) if dtype == "complex128" else v.astype(dtype)).cuda()
        two = ctx.encrypt_asymmetric(pk, ctx.encode(Q, v, scale, sparse_slots=slots, batch=batch), s, batch)
        one = ctx.encode_encrypt(pk, v, scale, s, slots, batch)
        ctx.check_status()
        assert torch.equal(one.reshape(-1), two.reshape(-1)), scale


@pytest.mark.parametrize("logn,slots", [(5, 2), (5, 4), (6, 8), (10, 16), (10, 32), (12, 1024), (13, 4096), (14, 512), (15, 16384), (16, 32768)])
@pytest.mark.parametrize("limbs", [1, 2, 3, 4, 5])
def test_decoding(oracle_mod, logn, slots, limbs):
    from lancelot_b200 import cabi

    n = 1 << logn
    mods = oracle_mod.coeff_modulus_create(n, [60, 40, 50, 59, 45])
    o, ctx = oracle_mod.Oracle(logn, mods, 0), cabi.Context(logn, mods, 0)
    rng = np.random.default_rng(logn + slots + limbs)
    pts = np.stack([rand_rows(rng, mods[:limbs], n) for _ in range(2)])  # centred values of the whole range, both signs
    got = ctx.decode_batch(limbs, cabi.to_device(pts), 2.0 ** 40, slots, 2).cpu().numpy()
    for b in range(2):
        want = np.asarray(o.decode(limbs, pts[b], 2.0 ** 40, slots)).reshape(-1)
        # 15 stages of rounding at 2^-53 each and the word-wise sums of the composition: a few 1e-15 of the largest value
        assert np.max(np.abs(got[b].reshape(-1) - want)) <= 1e-13 * np.max(np.abs(want))
