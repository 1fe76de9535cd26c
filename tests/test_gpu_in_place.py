"""Calls whose result shares memory with an operand, on rings of either kind of transform (one kernel, two kernels): word for
word what the same calls give on separate buffers, and what the CPU checker gives."""
import ctypes as C

import numpy as np
import pytest

from gpu_util import rand_rows, seeds

pytestmark = pytest.mark.gpu

CHAINS = [([60, 40, 40], [60]), ([60, 50, 47, 59], [60, 55])]


def _setup(oracle_mod, logn, chain):
    from lancelot_b200 import cabi

    data, special = chain
    mods = oracle_mod.coeff_modulus_create(1 << logn, data + special)
    return oracle_mod.Oracle(logn, mods, len(special)), cabi.Context(logn, mods, len(special)), mods, len(data), len(special)


@pytest.mark.parametrize("logn", [11, 12, 13, 16])
@pytest.mark.parametrize("chain", CHAINS)
def test_mod_down(oracle_mod, logn, chain):
    from lancelot_b200 import cabi
    from lancelot_b200._lib import check, lib

    o, ctx, mods, Q, P = _setup(oracle_mod, logn, chain)
    n, rng = 1 << logn, np.random.default_rng(logn)
    for L in (Q, 2):
        cx = rand_rows(rng, mods[:L] + mods[Q:], n)
        d = cabi.to_device(cx)
        want = cabi.to_host(ctx.moddown(L, d)).reshape(L, n)
        assert np.array_equal(want, o.moddown(L, cx).reshape(L, n))
        p = C.c_void_p(d.data_ptr())
        check(lib.lb_moddown(ctx.h, L, p, p, ctx._stream()))
        got = cabi.to_host(d).reshape(L + P, n)
        assert np.array_equal(got[:L], want) and np.array_equal(got[L:], cx[L:])


@pytest.mark.parametrize("logn", [11, 12, 13, 15, 16])
@pytest.mark.parametrize("chain", CHAINS)
@pytest.mark.parametrize("entry", ["lb_rescale", "lb_rescale_no_alloc"])
def test_rescale_of_one_polynomial(oracle_mod, logn, chain, entry):
    from lancelot_b200 import cabi
    from lancelot_b200._lib import check, lib

    o, ctx, mods, Q, _ = _setup(oracle_mod, logn, chain)
    n, rng = 1 << logn, np.random.default_rng(logn)
    for L in (Q, 2):
        x = rand_rows(rng, mods[:L], n)
        d = cabi.to_device(x[None])
        p = C.c_void_p(d.data_ptr())
        check(getattr(lib, entry)(ctx.h, L, 1, p, p, ctx._stream()))
        assert np.array_equal(cabi.to_host(d).reshape(L, n)[:L - 1], o.rescale(L, x[None]).reshape(L - 1, n))


@pytest.mark.parametrize("logn", [11, 12, 13])
@pytest.mark.parametrize("chain", CHAINS)
def test_encryption_of_a_plaintext_in_its_result(oracle_mod, logn, chain):
    from lancelot_b200 import cabi

    o, ctx, mods, Q, _ = _setup(oracle_mod, logn, chain)
    n, rng = 1 << logn, np.random.default_rng(logn)
    pk = o.gen_pk(o.gen_sk(seeds(rng, 1)), seeds(rng, 1), seeds(rng, 1))
    pt, s = rand_rows(rng, mods[:Q], n), seeds(rng, 2)
    ct = ctx.empty(1, 2, Q, n)
    ct[0, 0] = cabi.to_device(pt)
    ctx.encrypt_asymmetric(cabi.to_device(pk), ct[0, 0], s, 1, out=ct)
    assert np.array_equal(cabi.to_host(ct).reshape(2, Q, n), o.encrypt_asym(pk, pt, s[:64], s[64:]))
