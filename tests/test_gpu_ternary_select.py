"""The cluster-wide radix select of the ternary sampler against the host
restatement: odd lengths, shares that do not fill every CTA, the first length
whose keys are drawn again in every pass, and the extreme weights."""
import numpy as np
import pytest

from tests import philox_ref
from tests.gpu_util import require_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,hw", [(1, 0), (1, 1), (7, 3), (1024, 64), (4099, 4099), (16384, 8192), (16385, 1),
                                  (131072, 65536), (131073, 131072), (200001, 77)])
def test_ternary_equals_the_host_draws(n, hw):
    require_gpu()
    import aoa_b200 as aoa
    from aoa_b200 import params
    ps = params.ntt_primes(60, 1 << 17, 2)
    ctx = aoa.Context(aoa.Engine(10, ps[:1], ps[1:]))
    for seed, stream in ((1, 0), (0xFFFFFFFF12345678, 5)):
        got = aoa.sample_ternary(ctx, n, hw, seed, stream).numpy()
        want = philox_ref.ternary(n, hw, seed, stream)
        assert np.array_equal(got, want) and np.count_nonzero(got) == hw
