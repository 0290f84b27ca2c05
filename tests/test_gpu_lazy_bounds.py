"""Limb transforms at the edges of the lazy butterflies' primes: the largest below
2^60, primes around 2^32 and far below it, where 2^32 is no longer small beside q,
bit-exact with the oracle on uniform and all-(q - 1) inputs."""
import numpy as np
import pytest

from oracle import Oracle
from tests.ckks_inputs import uniform_residues
from tests.gpu_util import require_gpu
from tests.pymodel import bitrev

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


@pytest.mark.parametrize("log_n,whole_limb", [(11, False), (11, True), (14, False), (14, True), (15, False)])
def test_primes_below_34_bits_are_lazy(log_n, whole_limb):
    """They share the launches of 55-bit primes (a pass runs the limbs of one butterfly kind), and their
    transforms are the oracle's; below 2^31, where the reference's Barrett step is no longer exact, they are
    the polynomial's values."""
    require_gpu()
    import aoa_b200 as aoa
    from aoa_b200 import params
    n = 2 << log_n
    ps = [params.ntt_primes(b, n, 1)[0] for b in (34, 33, 55, 32, 26, 22)]
    E = aoa.Engine(log_n, ps, [])
    E.tune("ntt_whole", 2 if whole_limb else 0)
    ctx, o = aoa.Context(E), Oracle(E.N, ps, [])
    x = np.stack([uniform_residues(np.random.default_rng(log_n), ps, E.N)] * 2)
    x[1] = np.array(ps, dtype=np.uint64)[:, None] - np.uint64(1)
    d = ctx.upload(x)
    n0 = aoa.kernel_launches()
    ctx.ntt_fwd(d, 2, 0, len(ps))
    assert aoa.kernel_launches() - n0 == (1 if whole_limb else 2)
    got = d.numpy()
    for l, q in enumerate(ps):
        if q > 1 << 31:
            want = [o.ntt_fwd(x[p, l:l + 1], first=l)[0] for p in range(2)]
            assert np.array_equal(got[:, l], want), q
            continue
        psi = pow(params.primitive_root(q), (q - 1) // n, q)
        for pos in (0, 1, E.N // 2, E.N - 1):
            at, value = pow(psi, 2 * bitrev(pos, log_n) + 1, q), 0
            for c in x[0, l][::-1].tolist():
                value = (value * at + c) % q
            assert got[0, l, pos] == value, (q, pos)
    ctx.ntt_inv(d, 2, 0, len(ps))
    assert np.array_equal(d.numpy(), x)
