"""Slot sums add each rotation in its last pass: equal to rotations and additions
apart, on small (whole-limb) and large rings, in place and out of place, on DGT
contexts (through a temporary) too."""
import numpy as np
import pytest

from tests.ckks_inputs import uniform_residues
from tests.gpu_util import require_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n", [11, 13, 16])
@pytest.mark.parametrize("in_place", [False, True])
@pytest.mark.parametrize("dgt", [False, True])
def test_slot_sum_equals_rotations_and_additions(log_n, in_place, dgt):
    require_gpu()
    import aoa_b200 as aoa
    from aoa_b200 import params
    ps = params.ntt_primes(60, 1 << 32, 7)
    E = aoa.Engine(log_n, ps[:3], ps[3:])
    ctx = aoa.Context(E)
    dom = aoa.AOA_DGT if dgt else aoa.AOA_NTT
    if dgt:
        ctx.set_transform(dom)
    rng = np.random.default_rng(log_n)
    keys = {1 << j: aoa.SwitchKey(ctx, uniform_residues(rng, ps, E.N), uniform_residues(rng, ps, E.N), domain=dom)
            for j in range(3)}
    c = [uniform_residues(rng, ps[:3], E.N) for _ in range(2)]

    def ct():
        x = aoa.Ciphertext.from_residues(ctx, *c, slots=8, scale=1 << 40, domain=dom)
        x.set(1, 8, 1 << 40, dom)                # a limb below the top is stale
        return x
    a = ct()
    out = a if in_place else aoa.Ciphertext(ctx)
    aoa.ckks_sumslots(ctx, out, a, keys)
    want, rot = ct(), aoa.Ciphertext(ctx)
    for step in (4, 2, 1):
        aoa.ckks_rotate_left(ctx, rot, want, step, keys[step])
        aoa.ckks_add(ctx, want, want, rot)
    g, w = out.download(domain=aoa.AOA_COEF), want.download(domain=aoa.AOA_COEF)
    assert out.level == want.level == 1 and np.array_equal(g[0], w[0]) and np.array_equal(g[1], w[1])
