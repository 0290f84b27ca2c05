"""The tensor-core conversion's two reductions: a Montgomery step for output primes
from 2^50 up, a Barrett step below; ModUp and ModDown with primes on both sides,
against the oracle and the CUDA-core kernel, on uniform and all-(q - 1) inputs."""
import numpy as np
import pytest

from oracle import Oracle
from tests.ckks_inputs import uniform_residues
from tests.gpu_util import require_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(50, 51), (51, 50), (60, 45), (62, 52)])
@pytest.mark.parametrize("top", [False, True])
def test_conversion_on_both_sides_of_the_montgomery_bound(sizes, top):
    require_gpu()
    import aoa_b200 as aoa
    from aoa_b200 import capi, params
    log_n, k, kl = 12, 5, 6
    mod = 2 << log_n
    Q = params.ntt_primes(sizes[0], mod, k - 1) + params.ntt_primes(51 if sizes[0] != 51 else 60, mod, 1)
    B = params.ntt_primes(sizes[1] + 1, mod, 2)[1:] + params.ntt_primes(sizes[1], mod, kl - 1)
    B = [b for b in B if b not in Q]
    B = B + [p for p in params.ntt_primes(49, mod, kl) if p not in Q + B][: kl - len(B)]
    E = aoa.Engine(log_n, Q, B)
    ctx, o, lib = aoa.Context(E), Oracle(E.N, Q, B), capi.load()
    x = uniform_residues(np.random.default_rng(1), Q + B, E.N)
    if top:
        x[:] = np.array(Q + B, dtype=np.uint64)[:, None] - np.uint64(1)
    d = ctx.upload(x)
    for level in (0, 2, k - 1):
        res = []
        for tc in (1, 0):
            E.tune("conv_tensor_cores", tc)
            up, down = ctx.alloc((kl, E.N)), ctx.alloc((k, E.N))
            capi.check(lib.aoa_modup(ctx.handle, d.ptr, up.ptr, level))
            capi.check(lib.aoa_moddown(ctx.handle, d.ptr, down.ptr, level))
            res.append((up.numpy(), down.numpy()[: level + 1]))
        for a, b in zip(*res):
            assert np.array_equal(a, b)
        assert np.array_equal(res[0][0], np.asarray(o.modup(x[:k], level))[-kl:])
        assert np.array_equal(res[0][1], np.asarray(o.moddown(x, level))[: level + 1])
