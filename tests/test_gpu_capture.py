"""The allocation-free rescale and a key switch recorded into a CUDA graph: their transforms are launched with programmatic stream
serialisation, which the graph has to keep.  Replayed on fresh operands, against the CPU checker."""
import ctypes as C

import numpy as np
import pytest

from gpu_util import rand_rows, seeds

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("logn", [11, 13, 16])
def test_captured_rescale_and_relinearization(oracle_mod, logn):
    import torch

    from lancelot_b200 import cabi
    from lancelot_b200._lib import check, lib

    n, L = 1 << logn, 3
    mods = oracle_mod.coeff_modulus_create(n, [60, 40, 40, 60])
    o, ctx = oracle_mod.Oracle(logn, mods, 1), cabi.Context(logn, mods, 1)
    rng = np.random.default_rng(logn)
    sk = o.gen_sk(seeds(rng, 1))
    rlk = o.gen_ksk(sk, o.sk_square(sk), seeds(rng, 2 * L))
    d_rlk, ct3, out, one = cabi.to_device(rlk), ctx.empty(3, L, n), ctx.empty(2, L - 1, n), ctx.empty(L, n)
    ct3.zero_()
    one.zero_()

    def work():
        ctx.relinearize(L, ct3, d_rlk)
        check(lib.lb_rescale_no_alloc(ctx.h, L, 2, C.c_void_p(ct3.data_ptr()), C.c_void_p(out.data_ptr()), ctx._stream()))
        p = C.c_void_p(one.data_ptr())
        check(lib.lb_rescale_no_alloc(ctx.h, L, 1, p, p, ctx._stream()))  # in place

    work()  # grows the workspace and resolves the static array outside the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        work()
    for _ in range(2):
        x, y = np.stack([rand_rows(rng, mods[:L], n) for _ in range(3)]), rand_rows(rng, mods[:L], n)
        ct3.copy_(cabi.to_device(x))
        one.copy_(cabi.to_device(y))
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(cabi.to_host(out), o.rescale(L, o.relinearize(L, x.copy(), rlk)))
        assert np.array_equal(cabi.to_host(one)[: L - 1], o.rescale(L, y[None]).reshape(L - 1, n))
