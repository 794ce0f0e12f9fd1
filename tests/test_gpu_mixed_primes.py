"""Primes on both sides of 2^60 in one batch or server: few jobs of a degree run
as one launch, many as one per modulus class; every word against the oracle, on
both sides of the line between the two."""
import numpy as np
import pytest

from vkhel_gb300 import workloads

pytestmark = pytest.mark.gpu

LIFT = [("elemmod", 65537, 0)]
PERIOD = 8      # distinct jobs; a batch repeats them


def _jobs(oracle, n, above, seed):
    """PERIOD jobs, `above` of them with a prime in [2^60, 2^62), in mixed order."""
    lo, hi = workloads.ntt_primes(n, 2), workloads.ntt_primes(n, 1, bound=1 << 62)
    rng = np.random.default_rng(seed)
    out = []
    for k in range(PERIOD):
        q = hi[0] if (3 * k) % PERIOD < above else lo[k % 2]
        w = workloads.root_for(n, q)
        a, b = workloads.uniform(rng, q, n), workloads.uniform(rng, q, n)
        out.append((q, w, a, b, oracle.polymul(a, b, n, q, w)[0], oracle.forward(a, n, q, w)[0],
                    oracle.forward(b, n, q, w)[0]))
    return out


# words with q < 2^60 on both sides of 2^18 (n < 2^8), 3 2^20 (2^13 .. 2^15) and 3 2^18
@pytest.mark.parametrize("above", [1, 4])
@pytest.mark.parametrize("log_n, below", [(5, 8184), (5, 8192), (8, 3064), (8, 3072), (10, 760), (10, 768), (12, 184),
                                          (12, 192), (13, 376), (13, 384), (14, 184), (14, 192), (15, 88), (15, 96),
                                          (16, 4), (16, 12), (17, 4), (17, 8), (18, 4)])
def test_one_launch_or_two(vk, ctx, oracle, log_n, below, above):
    n = 1 << log_n
    jobs = max(below * PERIOD // (PERIOD - above), 2)   # `below` of them with q < 2^60, about
    kinds = _jobs(oracle, n, above, log_n + above)
    small = sum(kinds[j % PERIOD][0] < 1 << 60 for j in range(jobs))
    line = (1 << 18) * (1 if log_n < 8 else 12 if 13 <= log_n <= 15 else 3)
    tabs = {q: vk.NttTables(n, q, w) for q, w, *_ in kinds}
    ts = [tabs[kinds[j % PERIOD][0]] for j in range(jobs)]
    every = lambda f: np.concatenate([f(kinds[j % PERIOD]) for j in range(jobs)])
    lifted = lambda i: lambda k: oracle.elemmod(k[i], 65537, k[0])
    a, b, fa, fb = (vk.Vector(ctx, every(lambda k, i=i: k[i])) for i in (2, 3, 5, 6))
    c = vk.Vector(ctx, jobs * n)
    for name, want, add in (
            ("product", lambda k: k[4], lambda bt: bt.add_polymul(ts, a, b, c)),
            ("product with a lift", lifted(4), lambda bt: bt.add_polymul(ts, a, b, c, lift=LIFT)),
            ("product with NTT(b)", lambda k: k[4], lambda bt: bt.add_polymul(ts, a, fb, c, b_ntt=True)),
            ("forward", lambda k: k[5], lambda bt: bt.add_transform(ts, a, c)),
            ("inverse with a lift", lifted(2), lambda bt: bt.add_transform(ts, fa, c, inverse=True, lift=LIFT))):
        bt = vk.Batch(ctx)
        add(bt)
        bt.commit(graph=True)
        bt.run()
        if name == "forward" and log_n < 13:       # one kernel a launch there (no tails, no global passes)
            assert bt.kernels == (1 if small * n < line else 2)
        bt.close()
        np.testing.assert_array_equal(c.download(), every(want), err_msg=name)
    for v in (a, b, fa, fb, c):
        v.close()


@pytest.mark.parametrize("log_n", [5, 12, 14])
def test_server_requests_of_both_classes(vk, oracle, log_n):
    """Limbs of three modulus classes in one request, with and without a
    resident operand, several requests in a micro-batch."""
    n = 1 << log_n
    qs = workloads.ntt_primes(n, 2) + workloads.ntt_primes(n, 2, bound=1 << 62) + workloads.ntt_primes(n, 1, bound=1 << 63)
    qs = [qs[i] for i in (2, 0, 4, 3, 1)]
    ws = [workloads.root_for(n, q) for q in qs]
    tabs = [vk.NttTables(n, q, w) for q, w in zip(qs, ws)]
    rng = np.random.default_rng(log_n)
    new = lambda: np.concatenate([workloads.uniform(rng, q, n) for q in qs])
    key = new()
    with vk.Server() as srv:
        op = srv.add_operand(tabs, key)
        reqs = []
        for k in range(6):
            a, b, c = new(), new() if k % 2 else key, np.zeros(len(qs) * n, np.uint64)
            rid = srv.submit(tabs, a, b, c) if k % 2 else srv.submit_operand(tabs, a, op, c)
            reqs.append((rid, a, b, c))
        for rid, a, b, c in reqs:
            assert srv.wait(rid) == 0
            for i, (q, w) in enumerate(zip(qs, ws)):
                s = slice(i * n, (i + 1) * n)
                np.testing.assert_array_equal(c[s], oracle.polymul(a[s], b[s], n, q, w)[0])
