"""The edges of the modulus classes' lazy bounds.

Odd q < 2^60 run butterflies whose words grow to 12q (ntt_core.cuh, Mod60),
other q < 2^62 to 4q (Mod62).  The largest and smallest moduli of the first
class, the first prime past it, and words at the top of the range a stage may
meet -- q - 1 everywhere, q - 1 against 0, words around the first stage's
fast-path bound 3q, and arbitrary 64-bit words -- for one degree per pass
schedule (first passes of 1 .. 4 stages, clusters, passes over HBM).  Every
word equals the oracle's.
"""
import numpy as np
import pytest

from vkhel_gb300 import workloads

pytestmark = pytest.mark.gpu


def _prime_from(n, start):
    q = (start // (2 * n)) * (2 * n) + 1
    while q < start or not workloads.is_prime(q):
        q += 2 * n
    return q


def _modulus(n, which):
    if which == "top60":  # the largest of the class
        return workloads.ntt_primes(n, 1, bound=1 << 60)[0]
    if which == "past60":  # the first prime past it
        return _prime_from(n, 1 << 60)
    if which == "bits31":
        return workloads.ntt_primes(n, 1, bound=1 << 31)[0]
    return _prime_from(n, 2 * n)  # "least": the smallest NTT prime of the degree


def _inputs(n, q, rng):
    """(name, words below q)."""
    yield "top", np.full(n, q - 1, np.uint64)
    x = np.zeros(n, np.uint64)
    x[: n // 2] = q - 1
    yield "half", x
    y = np.full(n, q - 1, np.uint64)
    y[::2] = 0
    yield "alternating", y
    yield "uniform", workloads.uniform(rng, q, n)


@pytest.mark.parametrize("which", ["top60", "past60", "bits31", "least"])
@pytest.mark.parametrize("log_n", [3, 8, 9, 11, 12, 13, 14, 16, 17, 19])
def test_words_at_the_bounds(vk, ctx, oracle, log_n, which):
    n = 1 << log_n
    q = _modulus(n, which)
    w = workloads.root_for(n, q)
    t = vk.NttTables(n, q, w)
    rng = np.random.default_rng(log_n)
    r = vk.Vector(ctx, n)
    b_h = np.full(n, q - 1, np.uint64)
    b = vk.Vector(ctx, b_h)
    for name, a_h in _inputs(n, q, rng):
        a = vk.Vector(ctx, a_h)
        vk.forward_transform(a, r, t)
        np.testing.assert_array_equal(r.download(), oracle.forward(a_h, n, q, w)[0], err_msg=f"forward {name} q={q}")
        vk.inverse_transform(a, r, t)
        np.testing.assert_array_equal(r.download(), oracle.inverse(a_h, n, q, w)[0], err_msg=f"inverse {name} q={q}")
        vk.polymul(a, b, r, t)
        np.testing.assert_array_equal(r.download(), oracle.polymul(a_h, b_h, n, q, w)[0],
                                      err_msg=f"polymul {name} q={q}")


@pytest.mark.parametrize("which", ["top60", "past60"])
@pytest.mark.parametrize("log_n", [8, 11, 14, 16, 18])
def test_words_around_the_fast_path_bound(vk, ctx, oracle, log_n, which):
    n = 1 << log_n
    q = _modulus(n, which)
    w = workloads.root_for(n, q)
    t = vk.NttTables(n, q, w)
    rng = np.random.default_rng(60 + log_n)
    edges = np.array([0, q - 1, q, 2 * q - 1, 2 * q, 3 * q - 1, 3 * q], np.uint64)
    a_h = rng.choice(edges, n)
    a, r = vk.Vector(ctx, a_h), vk.Vector(ctx, n)
    vk.forward_transform(a, r, t)
    np.testing.assert_array_equal(r.download(), oracle.forward(a_h, n, q, w)[0])
    vk.inverse_transform(a, r, t)
    np.testing.assert_array_equal(r.download(), oracle.inverse(a_h, n, q, w)[0])
    a_h = rng.integers(0, 1 << 64, n, dtype=np.uint64)
    a_h[: n // 8] = (1 << 64) - 1
    a = vk.Vector(ctx, a_h)
    vk.forward_transform(a, r, t)
    np.testing.assert_array_equal(r.download(), oracle.forward(a_h, n, q, w)[0])


@pytest.mark.parametrize("log_n", [5, 10, 14, 15, 18])
def test_batch_of_both_classes_and_an_even_modulus(vk, ctx, oracle, log_n):
    """Limbs on both sides of 2^60 share a batch; an even modulus (accepted,
    though it has no inverse transform) keeps its forward words."""
    n = 1 << log_n
    qs = [_modulus(n, "top60"), _modulus(n, "past60"), workloads.ntt_primes(n, 2, bound=1 << 60)[1]]
    ws = [workloads.root_for(n, q) for q in qs]
    tabs = [vk.NttTables(n, q, w) for q, w in zip(qs, ws)]
    rng = np.random.default_rng(log_n)
    a_h = np.concatenate([workloads.uniform(rng, q, n) for q in qs])
    b_h = np.concatenate([workloads.uniform(rng, q, n) for q in qs])
    a, b, c, f = vk.Vector(ctx, a_h), vk.Vector(ctx, b_h), vk.Vector(ctx, 3 * n), vk.Vector(ctx, 3 * n)
    bt = vk.Batch(ctx)
    bt.add_polymul(tabs, a, b, c)
    bt.add_transform(tabs, a, f)
    bt.commit(graph=True)
    bt.run()
    for k, (q, w) in enumerate(zip(qs, ws)):
        s = slice(k * n, (k + 1) * n)
        np.testing.assert_array_equal(c.download()[s], oracle.polymul(a_h[s], b_h[s], n, q, w)[0])
        np.testing.assert_array_equal(f.download()[s], oracle.forward(a_h[s], n, q, w)[0])
    q = (1 << 40) + 6
    t = vk.NttTables(n, q, 5)
    x_h = workloads.uniform(rng, q, n)
    x, y = vk.Vector(ctx, x_h), vk.Vector(ctx, n)
    vk.forward_transform(x, y, t)
    np.testing.assert_array_equal(y.download(), oracle.forward(x_h, n, q, 5)[0])


@pytest.mark.parametrize("which", ["top60", "past60", "bits31", "least"])
@pytest.mark.parametrize("log_n", [3, 9, 10, 12, 14, 15, 17, 18])
def test_single_words_past_the_inverse_group_check(vk, ctx, oracle, log_n, which):
    """The inverse's first sub-stage checks its group's words against 2^bits(q)
    together: words on both sides of that and of 2q, one in 97 among words below
    q.  (2^64 - 1 only where the butterfly subtracts from it: the reference's
    subtraction loop wraps past 2^64 before it reaches it as the other operand.)"""
    n = 1 << log_n
    q = _modulus(n, which)
    w = workloads.root_for(n, q)
    t = vk.NttTables(n, q, w)
    rng = np.random.default_rng(97 + log_n)
    top = 1 << q.bit_length()
    edges = np.array([q, top - 1, top, 2 * q - 1, 2 * q, 3 * q, (1 << 64) - 1], np.uint64)
    a_h = workloads.uniform(rng, q, n)
    a_h[::97] = rng.choice(edges, len(a_h[::97]))
    a_h[1::2] = np.minimum(a_h[1::2], np.uint64(3 * q))
    a, r = vk.Vector(ctx, a_h), vk.Vector(ctx, n)
    vk.inverse_transform(a, r, t)
    np.testing.assert_array_equal(r.download(), oracle.inverse(a_h, n, q, w)[0])
