"""The splits of few jobs over 2, 4 and 8 CTAs and of the jobs past whole rounds
in both modulus classes below 2^62 (q < 2^60 and above), with two primes in the
batch and with a lift after the products: every word of every job against the
oracle.  The counts lie on both sides of each line, by the GPU's SMs."""
import numpy as np
import pytest

from vkhel_gb300 import workloads

pytestmark = pytest.mark.gpu

LIFT = [("elemmod", 65537, 0)]
PERIOD = 13     # distinct jobs; prime to the counts of a round, so that no shift goes unseen


def _counts(sms):
    s = sms
    lines = {12: [s // 8], 13: [s // 5, s // 2, s], 14: [s // 5, 2 * s // 5, s // 2, s, s + s // 5, s + s * 7 // 10],
             15: [s // 3, s // 2, s // 2 + s * 3 // 10], 16: [s // 8]}
    return [(log_n, c + more) for log_n, cs in lines.items() for c in cs for more in (0, 1)]


# 152 SMs unless the GPU says otherwise: the index picks the count at run time
@pytest.mark.parametrize("bits", [60, 62])
@pytest.mark.parametrize("case", range(len(_counts(152))))
def test_splits_and_tails(vk, ctx, oracle, case, bits):
    log_n, jobs = _counts(ctx.sm_count)[case]
    n = 1 << log_n
    qs = workloads.ntt_primes(n, 2, bound=1 << bits)
    ws = [workloads.root_for(n, q) for q in qs]
    tabs = [vk.NttTables(n, q, w) for q, w in zip(qs, ws)]
    rng = np.random.default_rng(1000 * log_n + jobs + bits)
    a_h = [workloads.uniform(rng, qs[k % 2], n) for k in range(PERIOD)]
    b_h = [workloads.uniform(rng, qs[k % 2], n) for k in range(PERIOD)]
    prod = [oracle.polymul(a_h[k], b_h[k], n, qs[k % 2], ws[k % 2])[0] for k in range(PERIOD)]
    fa = [oracle.forward(a_h[k], n, qs[k % 2], ws[k % 2])[0] for k in range(PERIOD)]
    fb = [oracle.forward(b_h[k], n, qs[k % 2], ws[k % 2])[0] for k in range(PERIOD)]
    lifted = lambda x: [oracle.elemmod(x[k], 65537, qs[k % 2]) for k in range(PERIOD)]
    every = lambda x: np.concatenate([x[j % PERIOD] for j in range(jobs)])
    ts = [tabs[j % PERIOD % 2] for j in range(jobs)]
    a, b, f, g = (vk.Vector(ctx, every(x)) for x in (a_h, b_h, fa, fb))
    c = vk.Vector(ctx, jobs * n)
    for name, want, add in (
            ("product", prod, lambda bt: bt.add_polymul(ts, a, b, c)),
            ("product with a lift", lifted(prod), lambda bt: bt.add_polymul(ts, a, b, c, lift=LIFT)),
            ("product with NTT(b)", prod, lambda bt: bt.add_polymul(ts, a, g, c, b_ntt=True)),
            ("forward", fa, lambda bt: bt.add_transform(ts, a, c)),
            ("inverse", a_h, lambda bt: bt.add_transform(ts, f, c, inverse=True)),
            ("inverse with a lift", lifted(a_h), lambda bt: bt.add_transform(ts, f, c, inverse=True, lift=LIFT))):
        bt = vk.Batch(ctx)
        add(bt)
        bt.commit(graph=False)
        bt.run()
        bt.close()
        np.testing.assert_array_equal(c.download(), every(want), err_msg=name)
    for v in (a, b, f, g, c):
        v.close()
