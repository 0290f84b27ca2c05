"""The Q limbs of HMult and rotations in one last pass over the operands: outputs
that are operands (of the same product, of another one in the batch), squares,
primes too wide for the three-product sum (61 to 63 bits), the lowest level,
with and without rescale, on the two-pass kernels and the whole-limb ones, against
the oracle."""
import numpy as np
import pytest

from oracle import ST_NTT, Oracle
from tests.ckks_inputs import make_keys, uniform_residues
from tests.gpu_util import require_gpu

pytestmark = pytest.mark.gpu
SCALE = 1 << 40


def _setup(bits, whole, log_n=15, k=4):
    import aoa_b200 as aoa
    from aoa_b200 import params
    ps = []
    for b in bits:
        ps += [p for p in params.ntt_primes(b, 2 << log_n, 2 * k + 1) if p not in ps][: 2 * k + 1 - len(ps)
                                                                                   if b == bits[-1] else 1]
    E = aoa.Engine(log_n, ps[:k], ps[k:])
    E.tune("ntt_whole", 2 if whole else 0)
    o = Oracle(E.N, ps[:k], ps[k:])
    return aoa, E, aoa.Context(E), o, make_keys(o, seed=3, rotations=(5, 9))


def _ct(aoa, ctx, rng, m):
    E = ctx.engine
    c = (uniform_residues(rng, E.q_primes, E.N), uniform_residues(rng, E.q_primes, E.N))
    ct = aoa.Ciphertext.from_residues(ctx, *c, slots=8, scale=SCALE, domain=aoa.AOA_NTT)
    ct.set(m - 1, 8, SCALE, aoa.AOA_NTT)
    return c, ct


@pytest.mark.parametrize("whole", [False, True])
@pytest.mark.parametrize("bits", [(60,), (61,), (63, 62, 55)])
@pytest.mark.parametrize("m", [2, 4])
@pytest.mark.parametrize("rescale", [True, False])
@pytest.mark.parametrize("alias", ["none", "a", "b", "square"])
def test_hmult_last_pass(whole, bits, m, rescale, alias):
    require_gpu()
    aoa, E, ctx, o, keys = _setup(bits, whole)
    evk = aoa.SwitchKey(ctx, *keys["evk"])
    rng = np.random.default_rng(m)
    ha, a = _ct(aoa, ctx, rng, m)
    hb, b = _ct(aoa, ctx, rng, m)
    if alias == "square":
        hb, b = ha, a
    out = {"a": a, "b": b}.get(alias) or aoa.Ciphertext(ctx)
    (aoa.ckks_mul if rescale else aoa.ckks_mul_without_rescale)(ctx, out, a, b, evk)
    w0, w1, _ = o.hmult(ha, hb, keys["evk"], m - 1, SCALE, SCALE, rescale=rescale, a_state=ST_NTT, b_state=ST_NTT)
    n = m - 1 if rescale else m
    g0, g1 = out.download(nlimbs=n, domain=aoa.AOA_COEF)
    assert out.level == n - 1
    assert np.array_equal(g0, w0[:n]) and np.array_equal(g1, w1[:n])


@pytest.mark.parametrize("whole", [False, True])
@pytest.mark.parametrize("n", [1, 3, 9])
def test_batch_whose_outputs_are_operands_of_other_products(whole, n):
    """Products whose output is the next product's operand read every operand before any output is written."""
    require_gpu()
    aoa, E, ctx, o, keys = _setup((60,), whole, log_n=12)
    evk = aoa.SwitchKey(ctx, *keys["evk"])
    rng = np.random.default_rng(n)
    cts = [_ct(aoa, ctx, rng, 3) for _ in range(n + 1)]
    outs = [cts[i + 1][1] for i in range(n)]
    aoa.ckks_mul_batch(ctx, outs, [c[1] for c in cts[:n]], [cts[0][1]] * n, evk)
    for i in range(n):
        w0, w1, _ = o.hmult(cts[i][0], cts[0][0], keys["evk"], 2, SCALE, SCALE, rescale=True, a_state=ST_NTT,
                            b_state=ST_NTT)
        g0, g1 = outs[i].download(nlimbs=2, domain=aoa.AOA_COEF)
        assert np.array_equal(g0, w0[:2]) and np.array_equal(g1, w1[:2])


@pytest.mark.parametrize("whole", [False, True])
@pytest.mark.parametrize("bits", [(60,), (61,), (63, 62, 55)])
@pytest.mark.parametrize("in_place", [False, True])
@pytest.mark.parametrize("steps", [(5, 5, 9, 5), (5, 9, 9, 9)])   # two keys in the group of two, or one
def test_rotation_last_pass(whole, bits, in_place, steps):
    require_gpu()
    aoa, E, ctx, o, keys = _setup(bits, whole)
    rtk = {s: aoa.SwitchKey(ctx, *keys["rtk"][s]) for s in (5, 9)}
    rng = np.random.default_rng(7)
    cts = [_ct(aoa, ctx, rng, m) for m in (1, 3, 3, 4)]
    outs = [c[1] if in_place else aoa.Ciphertext(ctx) for c in cts]
    aoa.ckks_rotate_left(ctx, outs[0], cts[0][1], steps[0], rtk[steps[0]])
    aoa.ckks_rotate_batch_steps(ctx, outs[1:], [c[1] for c in cts[1:]], steps[1:], [rtk[s] for s in steps[1:]])
    for (h, _), out, m, s in zip(cts, outs, (1, 3, 3, 4), steps):
        r0, r1 = o.rotate_left(h, s, keys["rtk"][s], m - 1, state=ST_NTT)
        g0, g1 = out.download(nlimbs=m, domain=aoa.AOA_COEF)
        assert np.array_equal(g0, r0[:m]) and np.array_equal(g1, r1[:m])
