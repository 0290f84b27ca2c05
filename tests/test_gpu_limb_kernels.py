"""Whole-limb transforms (rings up to 2^15, small calls) against the oracle, and the
HMult and rotations built on them against the two-pass kernels, around the sizes
at which the engine changes from one to the other."""
import numpy as np
import pytest

from oracle import Oracle
from tests.ckks_inputs import uniform_residues
from tests.gpu_util import require_gpu

pytestmark = pytest.mark.gpu


def _primes(log_n, k, kl):
    """Canonical (63 bits), both lazy kinds and 55-bit primes side by side."""
    from aoa_b200 import params
    n = 2 << log_n
    ps = params.ntt_primes(63, n, 1) + params.ntt_primes(60, 1 << 32, 2) + params.ntt_primes(60, n, 1)
    ps += params.ntt_primes(55, n, max(0, k + kl - len(ps)))
    return ps[:k], ps[k:k + kl]


@pytest.mark.parametrize("log_n", [10, 11, 12, 13, 14, 15])
@pytest.mark.parametrize("npolys", [1, 3])
def test_transforms_equal_the_oracle(log_n, npolys):
    """Strided polys (a gap limb after each), a run of primes that starts in the middle."""
    require_gpu()
    import aoa_b200 as aoa
    Q, B = _primes(log_n, 4, 2)
    ps = (Q + B)[:5]
    E = aoa.Engine(log_n, Q, B)
    ctx, o = aoa.Context(E), Oracle(E.N, Q, B)
    rng = np.random.default_rng(log_n)
    x = np.stack([uniform_residues(rng, ps + [1 << 40], E.N) for _ in range(npolys)])
    x[0, :5, :] = np.array(ps, dtype=np.uint64)[:, None] - np.uint64(1)
    d = ctx.upload(x)
    ctx.ntt_fwd(d, npolys, 0, 5, poly_stride=6)
    got = d.numpy()
    for p in range(npolys):
        assert np.array_equal(got[p, :5], o.ntt_fwd(x[p, :5])) and np.array_equal(got[p, 5], x[p, 5])
    ctx.ntt_inv(d, npolys, 0, 5, poly_stride=6)
    assert np.array_equal(d.numpy(), x)
    y = uniform_residues(rng, ps[2:4], E.N)
    dy = ctx.upload(y)
    ctx.ntt_inv(dy, 1, 2, 2)
    assert np.array_equal(dy.numpy(), o.ntt_inv(y, first=2))
    ctx.dgt_fwd(d, npolys, 0, 5, poly_stride=6)
    ctx.dgt_inv(d, npolys, 0, 5, poly_stride=6)
    assert np.array_equal(d.numpy(), x)


@pytest.mark.parametrize("log_n,k,n", [(10, 2, 1), (11, 5, 2), (12, 4, 1), (12, 12, 12), (13, 4, 9), (13, 6, 1),
                                       (14, 3, 6), (14, 12, 2), (15, 3, 2), (15, 4, 2)])
@pytest.mark.parametrize("rescale", [True, False])
def test_hmult_and_rotations_equal_the_two_pass_kernels(log_n, k, n, rescale):
    """Calls below, at and above the change; outputs apart and in place; a step and key per operation."""
    require_gpu()
    import aoa_b200 as aoa
    Q, B = _primes(log_n, k, k + 1)
    E = aoa.Engine(log_n, Q, B)
    ctx = aoa.Context(E)
    rng = np.random.default_rng(k)
    key = [aoa.SwitchKey(ctx, uniform_residues(rng, Q + B, E.N), uniform_residues(rng, Q + B, E.N)) for _ in range(2)]
    host = [(uniform_residues(rng, Q, E.N), uniform_residues(rng, Q, E.N)) for _ in range(2 * n)]
    scale = 1 << 40

    def run(in_place):
        cts = [aoa.Ciphertext.from_residues(ctx, *h, slots=8, scale=scale, domain=aoa.AOA_NTT) for h in host]
        a, b = cts[:n], cts[n:]
        out = a if in_place else [aoa.Ciphertext(ctx) for _ in range(n)]
        aoa.ckks_mul_batch(ctx, out, a, b, key[0], rescale=rescale)
        res = [x.download(domain=aoa.AOA_NTT) for x in out]
        rot = b if in_place else [aoa.Ciphertext(ctx) for _ in range(n)]
        aoa.ckks_rotate_batch_steps(ctx, rot, b, [3 + i for i in range(n)], [key[i % 2] for i in range(n)])
        return res + [x.download(domain=aoa.AOA_NTT) for x in rot]

    whole = run(False) + run(True)
    E.tune("ntt_whole", 0)                       # the two-pass kernels
    passes = run(False)
    for i, w in enumerate(whole):
        p = passes[i % len(passes)]
        assert np.array_equal(w[0], p[0]) and np.array_equal(w[1], p[1])


def test_expired_waits_are_reported_and_the_context_recovers():
    require_gpu()
    import aoa_b200 as aoa
    Q, B = _primes(12, 4, 2)
    E = aoa.Engine(12, Q, B)
    ctx, o = aoa.Context(E), Oracle(E.N, Q, B)
    x = uniform_residues(np.random.default_rng(0), Q + B, E.N)
    d = ctx.upload(x)
    E.tune("spin_limit", 0)
    ctx.ntt_fwd(d, 1, 0, 6)
    with pytest.raises(aoa.AoaError) as e:
        ctx.sync()
    assert e.value.name == "AOA_ERR_TIMEOUT"
    E.tune("spin_limit", 1 << 20)
    d = ctx.upload(x)
    ctx.ntt_fwd(d, 1, 0, 6)
    assert np.array_equal(d.numpy(), o.ntt_fwd(x))


def test_launch_shapes_choose_between_the_kernels():
    """A shape knob moves every call to the two passes while it differs from its default and no longer;
    "ntt_whole" overrides either way; the tuner times the two passes, leaves the small calls as they were, and
    its reported choice set on another engine gives the same launches."""
    require_gpu()
    import aoa_b200 as aoa
    Q, B = _primes(12, 4, 5)
    E = aoa.Engine(12, Q, B)

    def launches(E):
        ctx = aoa.Context(E)
        d = ctx.upload(np.zeros((4, E.N), dtype=np.uint64))
        n0 = aoa.kernel_launches()
        ctx.ntt_fwd(d, 1, 0, 4)
        ctx.ntt_inv(d, 1, 0, 4)
        n = aoa.kernel_launches() - n0
        ctx.sync()
        return n

    assert launches(E) == 2
    shapes = {"ntt_split": 1, "dgt_split": 0, "ntt_cols_div": 1, "ntt_rows_div": 0, "ntt_cols_kind": 1,
              "ntt_cols_tma": 0, "ntt_waves": 2, "ntt_waves_large": 2, "ntt_chunk_bytes": 1 << 30}
    two = {}
    for knob, value in shapes.items():
        default = E.tune_get(knob)
        E.tune(knob, default)
        assert launches(E) == 2, knob            # the default value chooses nothing
        E.tune(knob, value)
        two[knob] = launches(E)
        E.tune("ntt_whole", 2)
        assert launches(E) == 2, knob
        E.tune("ntt_whole", 1)
        E.tune(knob, default)
        assert two[knob] >= 4 and launches(E) == 2, knob
    E.tune("ntt_whole", 0)
    assert launches(E) >= 4
    E.tune("ntt_whole", 1)
    n0 = aoa.kernel_launches()
    rep = E.autotune(limbs=64)
    # every figure: three runs of two forward + inverse pairs and of four on each of two streams
    assert aoa.kernel_launches() - n0 >= (len(rep["trials"]) + 1) * 3 * (2 * 2 + 4 * 4) * 2
    assert launches(E) == 2
    E2 = aoa.Engine(12, Q, B)
    for knob, value in rep["choice"].items():
        E2.tune(knob, value)
    assert launches(E2) == 2 and E2.transform_shapes() == E.transform_shapes()
