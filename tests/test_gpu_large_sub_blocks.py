"""Degrees past one cluster: global passes around 2^16-word sub-blocks on 4
CTAs, or 2^14-word ones on 8 where the jobs are few, and products whose
sub-blocks run forward, product and inverse in one launch.  Job counts on both
sides of the line between the two (16 and 20 sub-blocks of 2^16 words), both
modulus classes, NTT(b) given, and the epilogue in the last global pass; every
word against the oracle."""
import numpy as np
import pytest

from vkhel_gb300 import workloads

pytestmark = pytest.mark.gpu

LIFT = [("elemmod", 65537, 0), ("elemgtadd", 32768, 3)]


def _lift(oracle, x, q):
    return oracle.elemgtadd(oracle.elemmod(x, 65537, q), 32768, 3)


@pytest.mark.parametrize("bits", [60, 62])
@pytest.mark.parametrize("log_n, jobs", [(18, 1), (18, 4), (18, 5), (19, 2), (19, 3), (20, 1), (20, 2), (22, 1)])
def test_products_and_transforms(vk, ctx, oracle, log_n, jobs, bits):
    n = 1 << log_n
    q = workloads.ntt_primes(n, 1, bound=1 << bits)[0]
    w = workloads.root_for(n, q)
    t = vk.NttTables(n, q, w)
    rng = np.random.default_rng(100 * log_n + jobs)
    a_h, b_h = workloads.uniform(rng, q, jobs * n), workloads.uniform(rng, q, jobs * n)
    part = [slice(k * n, (k + 1) * n) for k in range(jobs)]
    want_f = [oracle.forward(a_h[s], n, q, w)[0] for s in part]
    want_p = [oracle.polymul(a_h[s], b_h[s], n, q, w)[0] for s in part]
    a, b = vk.Vector(ctx, a_h), vk.Vector(ctx, b_h)
    tabs = [t] * jobs

    def batch(add):
        out = vk.Vector(ctx, jobs * n)
        bt = vk.Batch(ctx)
        add(bt, out)
        bt.commit(graph=True)
        bt.run()
        bt.close()
        return out, out.download()

    _, got = batch(lambda bt, o: bt.add_polymul(tabs, a, b, o))
    for s, ref in zip(part, want_p):
        np.testing.assert_array_equal(got[s], ref, err_msg="product")
    _, got = batch(lambda bt, o: bt.add_polymul(tabs, a, b, o, lift=LIFT))
    for s, ref in zip(part, want_p):
        np.testing.assert_array_equal(got[s], _lift(oracle, ref, q), err_msg="product with a lift")
    fa, got = batch(lambda bt, o: bt.add_transform(tabs, a, o))
    for s, ref in zip(part, want_f):
        np.testing.assert_array_equal(got[s], ref, err_msg="forward")
    fb, _ = batch(lambda bt, o: bt.add_transform(tabs, b, o))
    _, got = batch(lambda bt, o: bt.add_polymul(tabs, a, fb, o, b_ntt=True))
    for s, ref in zip(part, want_p):
        np.testing.assert_array_equal(got[s], ref, err_msg="product with NTT(b)")
    _, got = batch(lambda bt, o: bt.add_transform(tabs, fa, o, inverse=True))
    np.testing.assert_array_equal(got, a_h, err_msg="inverse")
    _, got = batch(lambda bt, o: bt.add_transform(tabs, fa, o, inverse=True, lift=LIFT))
    np.testing.assert_array_equal(got, _lift(oracle, a_h, q), err_msg="inverse with a lift")


@pytest.mark.parametrize("log_n", [18, 20])
def test_single_calls_in_place(vk, ctx, oracle, log_n):
    """A product over its own operand a, then b, as single calls."""
    n = 1 << log_n
    q = workloads.ntt_primes(n, 1)[0]
    w = workloads.root_for(n, q)
    t = vk.NttTables(n, q, w)
    rng = np.random.default_rng(log_n)
    a_h, b_h = workloads.uniform(rng, q, n), workloads.uniform(rng, q, n)
    ref = oracle.polymul(a_h, b_h, n, q, w)[0]
    a, b = vk.Vector(ctx, a_h), vk.Vector(ctx, b_h)
    vk.polymul(a, b, a, t)
    np.testing.assert_array_equal(a.download(), ref)
    a = vk.Vector(ctx, a_h)
    vk.polymul(a, b, b, t)
    np.testing.assert_array_equal(b.download(), ref)


@pytest.mark.parametrize("bits", [60, 62])
@pytest.mark.parametrize("jobs", [1, 9, 10])
def test_few_of_the_largest_cluster_degree(vk, ctx, oracle, jobs, bits):
    """2^17: few jobs in global passes and sub-blocks, more on 8-CTA clusters;
    and where the context's budget leaves no room for the passes' scratch."""
    n = 1 << 17
    q = workloads.ntt_primes(n, 1, bound=1 << bits)[0]
    w = workloads.root_for(n, q)
    t = vk.NttTables(n, q, w)
    rng = np.random.default_rng(jobs)
    a_h, b_h = workloads.uniform(rng, q, jobs * n), workloads.uniform(rng, q, jobs * n)
    part = [slice(k * n, (k + 1) * n) for k in range(jobs)]
    want = np.concatenate([oracle.polymul(a_h[s], b_h[s], n, q, w)[0] for s in part])
    own = vk.Context()
    a, b, c, f = vk.Vector(own, a_h), vk.Vector(own, b_h), vk.Vector(own, jobs * n), vk.Vector(own, jobs * n)

    def run(add):
        bt = vk.Batch(own)
        add(bt)
        bt.commit(graph=True)
        bt.run()
        bt.close()

    run(lambda bt: bt.add_transform([t] * jobs, b, f))
    np.testing.assert_array_equal(f.download(n), oracle.forward(b_h[:n], n, q, w)[0])
    run(lambda bt: bt.add_polymul([t] * jobs, a, f, c, b_ntt=True))
    np.testing.assert_array_equal(c.download(), want, err_msg="NTT(b) given")
    run(lambda bt: bt.add_transform([t] * jobs, f, f, inverse=True, lift=LIFT))
    np.testing.assert_array_equal(f.download(), _lift(oracle, b_h, q))
    for budget in (0, own.bytes_in_use + 4096 * jobs):  # room for the job table alone
        own.set_budget(budget)
        run(lambda bt: bt.add_polymul([t] * jobs, a, b, c, lift=LIFT))
        np.testing.assert_array_equal(c.download(), _lift(oracle, want, q), err_msg=f"budget {budget}")
        if jobs == 1:
            vk.polymul(a, b, c, t)
            np.testing.assert_array_equal(c.download(), want, err_msg=f"one call, budget {budget}")
            vk.forward_transform(b, f, t)
            vk.polymul_ntt(a, f, c, t)
            np.testing.assert_array_equal(c.download(), want, err_msg="one call, NTT(b) given")
    own.close()
