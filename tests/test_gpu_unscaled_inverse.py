"""HMult and rotations whose inverse transforms leave N^-1 to the basis conversions:
both conversion kernels, every fusing mode, transforms of one call on whole-limb
and two-pass kernels at once, all-(q - 1) operands, against the oracle; and the
rescaled limb inside and outside the special limbs' inverse, also in front of the
conversion of more than 32 primes, which takes the limb and the rest in two launches."""
import numpy as np
import pytest

from oracle import ST_NTT, Oracle
from tests.ckks_inputs import make_keys, uniform_residues
from tests.gpu_util import require_gpu

pytestmark = pytest.mark.gpu
SCALE = 1 << 40


def _primes(bits, log_n, count):
    from aoa_b200 import params
    if bits == "q1":
        return params.ntt_primes(60, 1 << 32, count)
    if bits == "mixed":
        return params.ntt_primes(63, 2 << log_n, 1) + params.ntt_primes(55, 2 << log_n, count - 1)
    return params.ntt_primes(bits, 2 << log_n, count)


# 4 limbs of 2^15 are whole-limb transforms, the 22 key-product limbs two passes
@pytest.mark.parametrize("log_n,k,kl", [(12, 3, 4), (15, 4, 11)])
@pytest.mark.parametrize("bits", ["q1", "mixed", 60, 62, 34])
@pytest.mark.parametrize("fuse,tensor_cores", [(1, 1), (1, 0), (0, 1), (7, 1)])
def test_hmult_and_rotation(log_n, k, kl, bits, fuse, tensor_cores):
    require_gpu()
    import aoa_b200 as aoa
    ps = _primes(bits, log_n, k + kl)
    E = aoa.Engine(log_n, ps[:k], ps[k:])
    E.tune("fuse", fuse)
    E.tune("conv_tensor_cores", tensor_cores)
    ctx, o = aoa.Context(E), Oracle(E.N, ps[:k], ps[k:])
    keys = make_keys(o, seed=3, rotations=(5,))
    rng = np.random.default_rng(k)
    top = np.repeat(np.array(ps[:k], dtype=np.uint64)[:, None] - np.uint64(1), E.N, axis=1)
    host = [(top, top), (uniform_residues(rng, ps[:k], E.N), uniform_residues(rng, ps[:k], E.N))]
    a, b = [aoa.Ciphertext.from_residues(ctx, *h, slots=8, scale=SCALE, domain=aoa.AOA_NTT) for h in host]
    out = aoa.Ciphertext(ctx)
    aoa.ckks_mul(ctx, out, a, b, aoa.SwitchKey(ctx, *keys["evk"]))
    w0, w1, _ = o.hmult(host[0], host[1], keys["evk"], k - 1, SCALE, SCALE, rescale=True, a_state=ST_NTT,
                        b_state=ST_NTT)
    g0, g1 = out.download(nlimbs=k - 1, domain=aoa.AOA_COEF)
    assert np.array_equal(g0, w0[: k - 1]) and np.array_equal(g1, w1[: k - 1])
    E2 = aoa.Engine(log_n, ps[:k], ps[k:])       # rotations: against the reference's op sequence
    ctx2 = aoa.Context(E2)
    for c in host:
        got, want = aoa.Ciphertext(ctx), aoa.Ciphertext(ctx2)
        x, y = [aoa.Ciphertext.from_residues(t, *c, slots=8, scale=SCALE, domain=aoa.AOA_NTT) for t in (ctx, ctx2)]
        aoa.ckks_rotate_left(ctx, got, x, 5, aoa.SwitchKey(ctx, *keys["rtk"][5]))
        aoa.ckks_rotate_plain(ctx2, want, y, 5, aoa.SwitchKey(ctx2, *keys["rtk"][5]))
        for u, v in zip(got.download(nlimbs=k, domain=aoa.AOA_COEF), want.download(nlimbs=k, domain=aoa.AOA_COEF)):
            assert np.array_equal(u, v)


@pytest.mark.parametrize("n", [55, 56])
@pytest.mark.parametrize("m", [2, 4])
def test_rescaled_limb_joins_the_special_limbs_up_to_one_wave(n, m):
    """Batches at 2^14 on both sides of the rule (2 n N <= 3 x 148 x 4096) equal single products."""
    require_gpu()
    import aoa_b200 as aoa
    ps = _primes("mixed", 14, 9)
    E = aoa.Engine(14, ps[:4], ps[4:])
    E.tune("batch_streams", 1)
    E.tune("ntt_whole", 0)                       # the two-pass kernels
    ctx = aoa.Context(E)
    rng = np.random.default_rng(n)
    evk = aoa.SwitchKey(ctx, uniform_residues(rng, ps, E.N), uniform_residues(rng, ps, E.N))
    cts = []
    for _ in range(3):
        h = (uniform_residues(rng, ps[:4], E.N), uniform_residues(rng, ps[:4], E.N))
        cts.append(aoa.Ciphertext.from_residues(ctx, *h, slots=8, scale=SCALE, domain=aoa.AOA_NTT))
        cts[-1].set(m - 1, 8, SCALE, aoa.AOA_NTT)
    a, b = [cts[i % 3] for i in range(n)], [cts[i % 2] for i in range(n)]
    outs = [aoa.Ciphertext(ctx) for _ in range(n)]
    aoa.ckks_mul_batch(ctx, outs, a, b, evk)
    one = aoa.Ciphertext(ctx)
    for i in (0, 1, 5, n - 1):
        aoa.ckks_mul(ctx, one, a[i], b[i], evk)
        want, got = one.download(nlimbs=m - 1, domain=aoa.AOA_COEF), outs[i].download(nlimbs=m - 1, domain=aoa.AOA_COEF)
        assert np.array_equal(want[0], got[0]) and np.array_equal(want[1], got[1])


@pytest.mark.parametrize("m", [32, 33, 34])
@pytest.mark.parametrize("whole", [False, True])
def test_more_than_32_primes(m, whole):
    """34 + 35 primes, levels on both sides of the two-launch form."""
    require_gpu()
    import aoa_b200 as aoa
    k = 34
    ps = _primes("mixed", 11, 2 * k + 1)
    E = aoa.Engine(11, ps[:k], ps[k:])
    E.tune("ntt_whole", 2 if whole else 0)
    ctx, o = aoa.Context(E), Oracle(E.N, ps[:k], ps[k:])
    keys = make_keys(o, seed=3, rotations=(5,))
    rng = np.random.default_rng(m)
    top = np.repeat(np.array(ps[:k], dtype=np.uint64)[:, None] - np.uint64(1), E.N, axis=1)
    host = [(top, top), (uniform_residues(rng, ps[:k], E.N), uniform_residues(rng, ps[:k], E.N))]
    a, b = [aoa.Ciphertext.from_residues(ctx, *h, slots=8, scale=SCALE, domain=aoa.AOA_NTT) for h in host]
    for c in (a, b):
        c.set(m - 1, 8, SCALE, aoa.AOA_NTT)
    evk, rtk = aoa.SwitchKey(ctx, *keys["evk"]), aoa.SwitchKey(ctx, *keys["rtk"][5])
    for rescale in (True, False):
        out = aoa.Ciphertext(ctx)
        (aoa.ckks_mul if rescale else aoa.ckks_mul_without_rescale)(ctx, out, a, b, evk)
        w0, w1, _ = o.hmult(host[0], host[1], keys["evk"], m - 1, SCALE, SCALE, rescale=rescale, a_state=ST_NTT,
                            b_state=ST_NTT)
        n = m - 1 if rescale else m
        g0, g1 = out.download(nlimbs=n, domain=aoa.AOA_COEF)
        assert np.array_equal(g0, w0[:n]) and np.array_equal(g1, w1[:n])
    out = aoa.Ciphertext(ctx)
    aoa.ckks_rotate_left(ctx, out, b, 5, rtk)
    r0, r1 = o.rotate_left(host[1], 5, keys["rtk"][5], m - 1, state=ST_NTT)
    g0, g1 = out.download(nlimbs=m, domain=aoa.AOA_COEF)
    assert np.array_equal(g0, r0[:m]) and np.array_equal(g1, r1[:m])


@pytest.mark.parametrize("n", [27, 28])
def test_more_than_32_primes_on_both_sides_of_the_joined_limb(n):
    """2 n N <= 3 x 148 x 4096 or not, at 2^15: the batch equals single products."""
    require_gpu()
    import aoa_b200 as aoa
    k, m = 34, 33
    ps = _primes("mixed", 15, 2 * k + 1)
    E = aoa.Engine(15, ps[:k], ps[k:])
    E.tune("batch_streams", 1)
    ctx = aoa.Context(E)
    rng = np.random.default_rng(n)
    evk = aoa.SwitchKey(ctx, uniform_residues(rng, ps, E.N), uniform_residues(rng, ps, E.N))
    cts = []
    for _ in range(2):
        h = (uniform_residues(rng, ps[:k], E.N), uniform_residues(rng, ps[:k], E.N))
        cts.append(aoa.Ciphertext.from_residues(ctx, *h, slots=8, scale=SCALE, domain=aoa.AOA_NTT))
        cts[-1].set(m - 1, 8, SCALE, aoa.AOA_NTT)
    a, b = [cts[i % 2] for i in range(n)], [cts[i % 3 // 2] for i in range(n)]
    outs = [aoa.Ciphertext(ctx) for _ in range(n)]
    aoa.ckks_mul_batch(ctx, outs, a, b, evk)
    one = aoa.Ciphertext(ctx)
    for i in (0, 1, 2, n - 1):
        aoa.ckks_mul(ctx, one, a[i], b[i], evk)
        want, got = one.download(nlimbs=m - 1, domain=aoa.AOA_COEF), outs[i].download(nlimbs=m - 1, domain=aoa.AOA_COEF)
        assert np.array_equal(want[0], got[0]) and np.array_equal(want[1], got[1])
