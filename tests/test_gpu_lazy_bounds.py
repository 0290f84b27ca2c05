"""Limb transforms at the edges of the lazy butterflies' primes: the largest below
2^60, the first bit lengths on either side of 2^34 (below it the butterflies are
canonical), bit-exact with the oracle on uniform and all-(q - 1) inputs."""
import numpy as np
import pytest

from oracle import Oracle
from tests.ckks_inputs import uniform_residues
from tests.gpu_util import require_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n", [11, 12, 16])
@pytest.mark.parametrize("top", [False, True])
def test_transforms_at_the_lazy_prime_bounds(log_n, top):
    require_gpu()
    import aoa_b200 as aoa
    from aoa_b200 import params
    ps = (params.ntt_primes(60, 2 << log_n, 1) + params.ntt_primes(35, 2 << log_n, 1)
          + params.ntt_primes(34, 2 << log_n, 1) + params.ntt_primes(60, 1 << 32, 1))
    E = aoa.Engine(log_n, ps[:3], ps[3:])
    E.tune("ntt_whole", 0)                       # the two-pass kernels
    ctx, o = aoa.Context(E), Oracle(E.N, ps[:3], ps[3:])
    x = uniform_residues(np.random.default_rng(log_n), ps, E.N)
    if top:
        x[:] = np.array(ps, dtype=np.uint64)[:, None] - np.uint64(1)
    d = ctx.upload(x)
    ctx.ntt_fwd(d, 1, 0, len(ps))
    assert np.array_equal(d.numpy(), o.ntt_fwd(x))
    ctx.ntt_inv(d, 1, 0, len(ps))
    assert np.array_equal(d.numpy(), x)
    ctx.dgt_fwd(d, 1, 0, len(ps))                # its twist hands lazy words to lazy limbs only
    ctx.dgt_inv(d, 1, 0, len(ps))
    assert np.array_equal(d.numpy(), x)


@pytest.mark.parametrize("whole_limb", [False, True])
@pytest.mark.parametrize("log_n", [10, 13, 15, 16])
def test_inverse_sums_at_the_lazy_prime_bounds(log_n, whole_limb):
    """The inverse's sums reach their bounds on all-(q - 1) and on blocks of q - 1 and 0 of each
    butterfly span, on odd and even stage counts of both passes."""
    require_gpu()
    import aoa_b200 as aoa
    from aoa_b200 import params
    ps = (params.ntt_primes(60, 2 << log_n, 1) + params.ntt_primes(60, 1 << 32, 1)
          + params.ntt_primes(35, 2 << log_n, 1) + params.ntt_primes(62, 2 << log_n, 1))
    E = aoa.Engine(log_n, ps[:2], ps[2:])
    if not whole_limb:
        E.tune("ntt_whole", 0)                   # the two-pass kernels
    ctx, o = aoa.Context(E), Oracle(E.N, ps[:2], ps[2:])
    top = np.array(ps, dtype=np.uint64)[:, None] - np.uint64(1)
    for span in [0, 1, 2, 8, 64, E.N // 4, E.N // 2]:
        on = np.ones(E.N, bool) if span == 0 else (np.arange(E.N) // span) % 2 == 0
        x = np.where(on[None, :], top, np.uint64(0))
        d = ctx.upload(x)
        ctx.ntt_inv(d, 1, 0, len(ps))
        assert np.array_equal(d.numpy(), o.ntt_inv(x)), span
