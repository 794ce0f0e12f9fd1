"""Job counts on both sides of each line of the split of few jobs over several
CTAs (n = 2^12 .. 2^16), and of the split of the jobs past a launch's whole
rounds: products, transforms and inverse transforms with a lift of that many
jobs, every word against the oracle (the forward transforms through the inverse,
which gives the inputs back)."""
import numpy as np
import pytest

from vkhel_gb300 import workloads

pytestmark = pytest.mark.gpu

LIFT = [("elemmod", 65537, 0)]
# on 152 SMs: the last count of each choice and the first of the next, then
# counts past one or two rounds of one job per SM (2^14, 2^13) or SM pair (2^15)
COUNTS = [(12, 19), (12, 20), (13, 30), (13, 31), (13, 76), (13, 77), (13, 160),
          (14, 30), (14, 31), (14, 60), (14, 61), (14, 76), (14, 77), (14, 153), (14, 182), (14, 212), (14, 228),
          (14, 256), (14, 259), (14, 304), (15, 50), (15, 51), (15, 77), (15, 121), (15, 122), (15, 153),
          (16, 19), (16, 20)]


@pytest.mark.parametrize("log_n, jobs", COUNTS)
def test_job_counts(vk, ctx, oracle, log_n, jobs):
    n = 1 << log_n
    q = workloads.ntt_primes(n, 1)[0]
    w = workloads.root_for(n, q)
    t = vk.NttTables(n, q, w)
    rng = np.random.default_rng(1000 * log_n + jobs)
    a_h, b_h = workloads.uniform(rng, q, jobs * n), workloads.uniform(rng, q, jobs * n)
    a, b = vk.Vector(ctx, a_h), vk.Vector(ctx, b_h)
    p, f, g = (vk.Vector(ctx, jobs * n) for _ in range(3))

    def run(add):
        bt = vk.Batch(ctx)
        add(bt)
        bt.commit(graph=False)
        bt.run()
        bt.close()

    run(lambda bt: bt.add_polymul([t] * jobs, a, b, p))
    got = p.download().reshape(jobs, n)
    for k in range(jobs):
        ref = oracle.polymul(a_h[k * n:(k + 1) * n], b_h[k * n:(k + 1) * n], n, q, w)[0]
        np.testing.assert_array_equal(got[k], ref, err_msg=f"product {k} of {jobs}")
    run(lambda bt: bt.add_transform([t] * jobs, a, f))
    last = slice((jobs - 1) * n, jobs * n)
    np.testing.assert_array_equal(f.download()[last], oracle.forward(a_h[last], n, q, w)[0])
    run(lambda bt: bt.add_transform([t] * jobs, f, g, inverse=True))
    np.testing.assert_array_equal(g.download(), a_h, err_msg="inverse(forward(a))")
    run(lambda bt: bt.add_transform([t] * jobs, f, g, inverse=True, lift=LIFT))
    np.testing.assert_array_equal(g.download(), oracle.elemmod(a_h, 65537, q), err_msg="with a lift")
    run(lambda bt: bt.add_transform([t] * jobs, b, g))
    run(lambda bt: bt.add_polymul([t] * jobs, a, g, p, b_ntt=True))
    np.testing.assert_array_equal(p.download().reshape(jobs, n), got, err_msg="with NTT(b) given")
