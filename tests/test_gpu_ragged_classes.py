"""The single-launch ragged batch (tuning entry (3, 2) = 1) with primes in
[2^60, 2^62), alone and beside primes below 2^60: one kernel, the oracle's words."""
import numpy as np
import pytest

from vkhel_gb300 import workloads

pytestmark = pytest.mark.gpu

# odd numbers of 2^15 and of 2^12 products, each degree twice
SHAPES = [(16, 2), (15, 3), (14, 2), (13, 1), (12, 3), (15, 4), (16, 1), (12, 2), (13, 3), (14, 1)]


@pytest.fixture
def single_launch(vk):
    L = vk.lib()
    saved = L.vkhel_tune_get(3, 2)
    L.vkhel_tune_set(3, 2, 1)
    yield
    L.vkhel_tune_set(3, 2, saved)


@pytest.mark.parametrize("mixed", [False, True])
def test_one_launch(vk, ctx, oracle, single_launch, mixed):
    rng = np.random.default_rng(11 + mixed)
    tabs, inst = {}, []
    bt = vk.Batch(ctx)
    for k, (log_n, limbs) in enumerate(SHAPES):
        n = 1 << log_n
        qs = workloads.ntt_primes(n, limbs, bound=1 << (60 if mixed and k % 2 else 62))
        if mixed and limbs > 1:
            qs[0] = workloads.ntt_primes(n, 1)[0]
        ws = [workloads.root_for(n, q) for q in qs]
        for q, w in zip(qs, ws):
            tabs.setdefault((n, q), vk.NttTables(n, q, w))
        a, b = (np.concatenate([workloads.uniform(rng, q, n) for q in qs]) for _ in range(2))
        va, vb, vc = vk.Vector(ctx, a), vk.Vector(ctx, b), vk.Vector(ctx, limbs * n)
        bt.add_polymul([tabs[n, q] for q in qs], va, vb, vc)
        inst.append((n, qs, ws, a, b, vc))
    bt.commit(graph=True)
    assert bt.kernels == 1
    bt.run()
    bt.close()
    for n, qs, ws, a, b, vc in inst:
        got = vc.download()
        for i, (q, w) in enumerate(zip(qs, ws)):
            s = slice(i * n, (i + 1) * n)
            np.testing.assert_array_equal(got[s], oracle.polymul(a[s], b[s], n, q, w)[0], err_msg=f"n={n} limb {i}")
