"""Past one cluster, job counts on both sides of the lines between 2^16-word
sub-blocks on 4-CTA clusters and 2^14-word ones on single CTAs (counts for 152
SMs), both modulus classes below 2^62: every word of transforms, products,
products with NTT(b) given and lifts against the oracle."""
import numpy as np
import pytest

from vkhel_gb300 import workloads

pytestmark = pytest.mark.gpu

LIFT = [("elemmod", 65537, 0)]
PERIOD = 3     # distinct jobs; a batch repeats them


@pytest.mark.parametrize("bits", [60, 62])
@pytest.mark.parametrize("log_n, jobs", [(18, 9), (18, 10), (18, 18), (18, 19), (18, 20), (18, 37), (18, 46), (19, 13),
                                         (19, 14), (19, 23), (20, 7), (20, 8), (21, 1), (21, 4)])
def test_rounds(vk, ctx, oracle, log_n, jobs, bits):
    n = 1 << log_n
    q = workloads.ntt_primes(n, 1, bound=1 << bits)[0]
    w = workloads.root_for(n, q)
    t = vk.NttTables(n, q, w)
    rng = np.random.default_rng(100 * log_n + jobs + bits)
    period = min(PERIOD, jobs)
    a_h = [workloads.uniform(rng, q, n) for _ in range(period)]
    b_h = [workloads.uniform(rng, q, n) for _ in range(period)]
    prod = [oracle.polymul(x, y, n, q, w)[0] for x, y in zip(a_h, b_h)]
    fa, fb = ([oracle.forward(x, n, q, w)[0] for x in h] for h in (a_h, b_h))
    lifted = lambda xs: [oracle.elemmod(x, 65537, q) for x in xs]
    every = lambda xs: np.concatenate([xs[j % period] for j in range(jobs)])
    a, b, f, g = (vk.Vector(ctx, every(x)) for x in (a_h, b_h, fa, fb))
    c = vk.Vector(ctx, jobs * n)
    ts = [t] * jobs
    for name, want, add in (
            ("product", prod, lambda bt: bt.add_polymul(ts, a, b, c)),
            ("product with a lift", lifted(prod), lambda bt: bt.add_polymul(ts, a, b, c, lift=LIFT)),
            ("product with NTT(b)", prod, lambda bt: bt.add_polymul(ts, a, g, c, b_ntt=True)),
            ("forward", fa, lambda bt: bt.add_transform(ts, a, c)),
            ("inverse", a_h, lambda bt: bt.add_transform(ts, f, c, inverse=True)),
            ("inverse with a lift", lifted(a_h), lambda bt: bt.add_transform(ts, f, c, inverse=True, lift=LIFT))):
        bt = vk.Batch(ctx)
        add(bt)
        bt.commit(graph=True)
        bt.run()
        bt.close()
        np.testing.assert_array_equal(c.download(), every(want), err_msg=name)
    for v in (a, b, f, g, c):
        v.close()
