"""DGT contexts' HMult with its Q limbs in one last pass: against the separate
kernels (a batch in which one output is another product's operand), against the
oracle's residues, with squares, outputs in place, primes too wide for the summed
products, the lowest level, with and without rescale."""
import numpy as np
import pytest

from oracle import ST_COEF, Oracle
from tests.ckks_inputs import make_keys, uniform_residues
from tests.gpu_util import require_gpu

pytestmark = pytest.mark.gpu
SCALE = 1 << 40


@pytest.mark.parametrize("bits", [60, 61])
@pytest.mark.parametrize("m", [2, 4])
@pytest.mark.parametrize("rescale", [True, False])
@pytest.mark.parametrize("alias", ["none", "a", "square", "chain"])
def test_dgt_hmult_last_pass(bits, m, rescale, alias):
    require_gpu()
    import aoa_b200 as aoa
    from aoa_b200 import params
    log_n, k = 12, 4
    ps = params.ntt_primes(bits, 2 << log_n, 2 * k + 1)
    E = aoa.Engine(log_n, ps[:k], ps[k:])
    ctx, o = aoa.Context(E), Oracle(E.N, ps[:k], ps[k:])
    ctx.set_transform(aoa.AOA_DGT)
    keys = make_keys(o, seed=3)
    b_, a_ = ctx.upload(keys["evk"][0]), ctx.upload(keys["evk"][1])
    for d in (b_, a_):                           # the oracle's keys are in the NTT domain
        ctx.ntt_inv(d, 1, 0, len(ps))
        ctx.dgt_fwd(d, 1, 0, len(ps))
    evk = aoa.SwitchKey(ctx, b_.numpy(), a_.numpy(), domain=aoa.AOA_DGT)
    rng = np.random.default_rng(m)
    host = [(uniform_residues(rng, ps[:k], E.N), uniform_residues(rng, ps[:k], E.N)) for _ in range(3)]
    cts = []
    for h in host:
        ct = aoa.Ciphertext.from_residues(ctx, *h, slots=8, scale=SCALE, domain=aoa.AOA_COEF)
        ct.set(m - 1, 8, SCALE, aoa.AOA_COEF)
        cts.append(ct)
    pairs = {"square": [(0, 0), (1, 1)]}.get(alias, [(0, 2), (1, 2)])
    outs = {"a": [cts[0], cts[1]], "chain": [cts[1], aoa.Ciphertext(ctx)]}.get(
        alias, [aoa.Ciphertext(ctx), aoa.Ciphertext(ctx)])
    aoa.ckks_mul_batch(ctx, outs, [cts[x] for x, _ in pairs], [cts[y] for _, y in pairs], evk, rescale=rescale)
    n = m - 1 if rescale else m
    for (x, y), out in zip(pairs, outs):
        w0, w1, _ = o.hmult(host[x], host[y], keys["evk"], m - 1, SCALE, SCALE, rescale=rescale, a_state=ST_COEF,
                            b_state=ST_COEF)
        g0, g1 = out.download(nlimbs=n, domain=aoa.AOA_COEF)
        assert np.array_equal(g0, w0[:n]) and np.array_equal(g1, w1[:n])
