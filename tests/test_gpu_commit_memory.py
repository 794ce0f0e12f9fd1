"""Few products of 2^17 as a batch in a context whose memory would hold the
global passes' scratch but not the job table beside it: the commit succeeds,
the fused kernel computes the oracle's words and the budget's rest stays free."""
import numpy as np
import pytest

from vkhel_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jobs", [1, 9])
@pytest.mark.parametrize("spare", [0, 4096])
def test_commit_within_a_budget(vk, oracle, jobs, spare):
    n = 1 << 17
    q = workloads.ntt_primes(n, 1)[0]
    w = workloads.root_for(n, q)
    t = vk.NttTables(n, q, w)
    rng = np.random.default_rng(jobs)
    a_h, b_h = workloads.uniform(rng, q, jobs * n), workloads.uniform(rng, q, jobs * n)
    with vk.Context() as own:
        a, b, c = vk.Vector(own, a_h), vk.Vector(own, b_h), vk.Vector(own, jobs * n)
        bt = vk.Batch(own)
        bt.add_polymul([t] * jobs, a, b, c)     # the tables are resident from here on
        own.set_budget(own.bytes_in_use + jobs * n * 8 + spare)
        bt.commit(graph=True)
        if spare:
            vk.Vector(own, jobs * n).close()
        bt.run()
        for k in range(jobs):
            s = slice(k * n, (k + 1) * n)
            np.testing.assert_array_equal(c.download()[s], oracle.polymul(a_h[s], b_h[s], n, q, w)[0])
        bt.close()
