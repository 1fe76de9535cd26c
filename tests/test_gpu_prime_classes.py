"""Products, sums of products and base conversions for every class of primes (near 2^60, the integer rest, FP64 at both ends
of its range, too small for FP64), with residues at the top of their range: bit for bit against the CPU checker."""
import numpy as np
import pytest

from gpu_util import seeds

pytestmark = pytest.mark.gpu

# the class limits of the reductions: 2^34, 2^50 and 2^60 - 2^28; of the transforms: 2^47, 2^50, 2^58
BITS = [60, 59, 57, 51, 50, 48, 47, 35, 34, 28]


def _rows(rng, mods, shape, n):
    x = np.empty(shape + (len(mods), n), dtype=np.uint64)
    for r, q in enumerate(mods):
        x[..., r, :] = rng.integers(0, q, shape + (n,), dtype=np.uint64)
        x[..., r, :5] = [q - 1, q - 1, 0, 1, q // 2]
    return x


@pytest.mark.parametrize("logn", [10, 12])
def test_products_and_powers(oracle_mod, logn):
    from lancelot_b200 import cabi

    n = 1 << logn
    mods = oracle_mod.coeff_modulus_create(n, BITS)
    L = len(mods)
    o, ctx = oracle_mod.Oracle(logn, mods, 0), cabi.Context(logn, mods, 0)
    rng = np.random.default_rng(logn)
    a, b = _rows(rng, mods, (2,), n), _rows(rng, mods, (2,), n)
    assert np.array_equal(cabi.to_host(ctx.multiply(L, cabi.to_device(a), cabi.to_device(b))).reshape(3, L, n), o.tensor(L, a, b))
    got = cabi.to_host(ctx.multiply_poly(L, cabi.to_device(a[0]), cabi.to_device(b[0])))
    want = [[int(x) * int(y) % q for x, y in zip(a[0, r, :64], b[0, r, :64])] for r, q in enumerate(mods)]
    assert np.array_equal(got.reshape(L, n)[:, :64], np.array(want, dtype=np.uint64))
    # decryption adds products up before it reduces them: one, two and more polynomials than a window takes
    for polys in (1, 2, 3, 40):
        ct, sk = _rows(rng, mods, (polys,), n), _rows(rng, mods, (), n)
        got = cabi.to_host(ctx.decrypt(L, cabi.to_device(ct), cabi.to_device(sk))).reshape(L, n)
        want = [[sum(int(ct[p, r, k]) * int(sk[r, k]) ** p for p in range(polys)) % q for k in range(16)] for r, q in enumerate(mods)]
        assert np.array_equal(got[:, :16], np.array(want, dtype=np.uint64)), polys


@pytest.mark.parametrize("clients,chunks", [(1, 1), (3, 2), (33, 5), (64, 9)])
def test_mask_sums(oracle_mod, clients, chunks):
    from lancelot_b200 import cabi

    logn, n = 10, 1 << 10
    mods = oracle_mod.coeff_modulus_create(n, [60, 59, 50, 40, 34])
    L = len(mods)
    ctx = cabi.Context(logn, mods, 0)
    rng = np.random.default_rng(clients)
    cts, masks = _rows(rng, mods, (clients, chunks, 2), n), _rows(rng, mods, (clients, 2), n)
    d = cabi.to_device(cts)
    got = cabi.to_host(ctx.mask_accumulate(L, [d[k] for k in range(clients)], cabi.to_device(masks), chunks)).reshape(chunks, 3, L, n)
    for c in range(chunks):
        for r, q in enumerate(mods):
            for k in (0, 1, 2, 5, n - 1):
                x = [(int(cts[i, c, 0, r, k]), int(cts[i, c, 1, r, k]), int(masks[i, 0, r, k]), int(masks[i, 1, r, k])) for i in range(clients)]
                want = [sum(a0 * b0 for a0, _, b0, _ in x) % q, sum(a0 * b1 + a1 * b0 for a0, a1, b0, b1 in x) % q, sum(a1 * b1 for _, a1, _, b1 in x) % q]
                assert [int(v) for v in got[c, :, r, k]] == want, (c, r, k)


# data primes, special primes: every class as a target of a conversion from one row, of few rows, and of more than eight
CHAINS = [(BITS, [60]), ([60, 50, 47, 35, 34, 59], [60, 51]), ([60, 59, 50, 50, 48, 47, 35, 34, 57], [60, 60, 60, 60, 60, 60, 59, 59, 50])]


@pytest.mark.parametrize("logn", [11, 12, 13, 15])
@pytest.mark.parametrize("chain", range(len(CHAINS)))
def test_key_switch_rescale_and_encryption(oracle_mod, logn, chain):
    import torch

    from lancelot_b200 import cabi

    data, special = CHAINS[chain]
    n, Q, P = 1 << logn, len(data), len(special)
    mods = oracle_mod.coeff_modulus_create(n, data + special)
    o, ctx = oracle_mod.Oracle(logn, mods, P), cabi.Context(logn, mods, P)
    rng = np.random.default_rng(10 * logn + chain)
    sk = o.gen_sk(seeds(rng, 1))
    rlk = o.gen_ksk(sk, o.sk_square(sk), seeds(rng, 2 * (Q // P)))
    for L in {Q, max(2, Q - 2)}:
        ct3 = _rows(rng, mods[:L], (3,), n)
        want = o.relinearize(L, ct3.copy(), rlk)
        got = ctx.relinearize(L, cabi.to_device(ct3), cabi.to_device(rlk)).contiguous()
        assert np.array_equal(cabi.to_host(got).reshape(2, L, n), want)
        assert np.array_equal(cabi.to_host(ctx.rescale(L, got)).reshape(2, L - 1, n), o.rescale(L, want))
    pk = o.gen_pk(sk, seeds(rng, 1), seeds(rng, 1))
    batch, s = 3, seeds(rng, 6)
    pts = _rows(rng, mods[:Q], (batch,), n)
    got = cabi.to_host(ctx.encrypt_asymmetric(cabi.to_device(pk), cabi.to_device(pts), s, batch)).reshape(batch, 2, Q, n)
    for b in range(batch):
        assert np.array_equal(got[b], o.encrypt_asym(pk, pts[b], s[128 * b:128 * b + 64], s[128 * b + 64:128 * b + 128]))
    # the plaintext folded into the closing transform
    vals = torch.from_numpy(rng.uniform(-1, 1, (batch, n // 2))).cuda()
    two = ctx.encrypt_asymmetric(cabi.to_device(pk), ctx.encode(Q, vals, 2.0 ** 40, sparse_slots=n // 2, batch=batch), s, batch)
    one = ctx.encode_encrypt(cabi.to_device(pk), vals, 2.0 ** 40, s, n // 2, batch)
    assert np.array_equal(cabi.to_host(one).ravel(), cabi.to_host(two).ravel())
