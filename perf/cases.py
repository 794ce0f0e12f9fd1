"""Performance cases: what programs have this library do, through its public
Python entry points (one ctypes call per C entry point).

Every case is a dict of plain values; `kind` says which entry points it goes
through:

  calls     the plain call pattern of the reference's users: forward(a),
            forward(b), elemmul, inverse, one blocking call each
  polymul   one blocking vkhel_vector_polymul per pass
  batch     a committed batch of RNS products (limbs x products limb
            products), replayed from its CUDA graph; `operand`: "plain", "ntt"
            (b kept as NTT(b): a key or a plaintext used many times) or
            "lift" (plain with the centred reduction mod 65537 at the end)
  transform a committed batch of forward or inverse transforms, the inverse
            with or without the centred reduction mod 65537
  ragged    a batch whose instances differ in degree and limb count
  elem      element-wise jobs of ragged lengths in one launch
  serve     a burst of requests with host operands through the server

Sizes follow this repository's configurations (vkhel_gb300/workloads.py) and
tests: degrees 2^10 .. 2^20, 1 .. 24 limbs, primes of 30 .. 62 bits (the first
q = 1 mod 2n below 2^bits), operands uniform below their prime.
"""
import functools
import random

import numpy as np
import torch

import vkhel_gb300 as vk
from vkhel_gb300 import workloads

LIFT_MOD = 65537


def listed():
    return [
        # the reference's own call pattern at its usual small degree: launch latency
        dict(name="calls_4096", kind="calls", log_n=12, bits=60),
        # one fused product per call, as an interactive program multiplies
        dict(name="polymul_16384", kind="polymul", log_n=14, bits=60),
        # ciphertext multiplication: an RNS batch of 32 pairs of 8 limbs
        dict(name="rns_16384", kind="batch", log_n=14, limbs=8, products=32, bits=60, operand="plain"),
        # a batch of independent single-limb products of a larger degree
        dict(name="single_limb_65536", kind="batch", log_n=16, limbs=1, products=64, bits=60, operand="plain"),
        # many products of a small degree (packed plaintext arithmetic)
        dict(name="small_1024", kind="batch", log_n=10, limbs=3, products=1001, bits=50, operand="plain"),
        # products with stored keys: b stays in the transform domain
        dict(name="keys_8192", kind="batch", log_n=13, limbs=13, products=37, bits=55, operand="ntt"),
        # the largest degree of the batch, above what one cluster holds
        dict(name="large_1048576", kind="batch", log_n=20, limbs=5, products=3, bits=60, operand="plain"),
        # encoding: forward transforms of many limbs
        dict(name="forward_16384", kind="transform", log_n=14, count=1000, bits=60, inverse=False, lift=False),
        # decryption: inverse transforms ending in the centred reduction
        dict(name="inverse_lift_32768", kind="transform", log_n=15, count=150, bits=60, inverse=True, lift=True),
        # requests of several parameter sets collected into one batch
        dict(name="ragged_512", kind="ragged", instances=512, log_lo=12, log_hi=16, max_limbs=16, bits=60, shape_seed=3),
        # element-wise arithmetic on ragged vectors
        dict(name="elem_2048", kind="elem", jobs=2048, max_len=1 << 17, bits=60, shape_seed=5),
        # a burst of requests with host operands
        dict(name="serve_12", kind="serve", requests=12, log_lo=12, log_hi=16, max_limbs=24, bits=60, shape_seed=4),
    ]


# Total words of one operand of a drawn batch: at most the ragged batch's.
_MAX_WORDS = 1 << 25


def draw(rng):
    kind = rng.choice(["calls", "polymul", "batch", "batch", "batch", "transform", "transform", "ragged", "elem", "serve"])
    bits = rng.choice([30, 45, 50, 55, 60, 60, 60, 62])
    if kind in ("calls", "polymul"):
        return dict(kind=kind, log_n=rng.randint(10, 20), bits=bits)
    if kind in ("batch", "transform"):
        log_n = rng.randint(10, 20)
        units = max(1, int(2 ** rng.uniform(0, 24.5 - log_n)))  # limb jobs
        if kind == "transform":
            inverse = rng.random() < 0.5
            return dict(kind=kind, log_n=log_n, count=units, bits=bits, inverse=inverse,
                        lift=inverse and rng.random() < 0.5)
        limbs = min(units, rng.randint(1, 24))
        return dict(kind=kind, log_n=log_n, limbs=limbs, products=max(1, units // limbs), bits=bits,
                    operand=rng.choice(["plain", "plain", "ntt", "lift"]))
    if kind == "ragged":
        lo = rng.randint(10, 14)
        return dict(kind=kind, instances=int(2 ** rng.uniform(2, 8)), log_lo=lo, log_hi=rng.randint(lo + 1, 17),
                    max_limbs=rng.randint(1, 16), bits=bits, shape_seed=rng.randrange(1 << 20))
    if kind == "elem":
        return dict(kind=kind, jobs=int(2 ** rng.uniform(0, 11)), max_len=int(2 ** rng.uniform(8, 17)), bits=bits,
                    shape_seed=rng.randrange(1 << 20))
    return dict(kind=kind, requests=rng.randint(1, 12), log_lo=12, log_hi=rng.randint(12, 16),
                max_limbs=rng.randint(1, 24), bits=bits, shape_seed=rng.randrange(1 << 20))


# ---------------------------------------------------------------------------
# what a program keeps: one context, one server, the primes and their tables


@functools.lru_cache(maxsize=None)
def _primes(log_n, bits):
    """(q, w) of the first 24 primes of the size, fewer where there are fewer."""
    n = 1 << log_n
    return [(q, workloads.root_for(n, q)) for q in workloads.ntt_primes(n, 24, bound=1 << bits)]


@functools.lru_cache(maxsize=None)
def _tables(log_n, bits):
    return [vk.NttTables(1 << log_n, q, w) for q, w in _primes(log_n, bits)]


@functools.lru_cache(maxsize=None)
def _context():
    return vk.Context()


@functools.lru_cache(maxsize=None)
def _server():
    return vk.Server()


def _limb_tables(log_n, bits, limbs):
    t = _tables(log_n, bits)
    return [t[k % len(t)] for k in range(limbs)]


class _Words:
    """A vector's device words as __cuda_array_interface__ (no copy)."""

    def __init__(self, vec):
        self.vec = vec
        self.__cuda_array_interface__ = dict(shape=(vec.length,), typestr="<i8", data=(vec.device_ptr, False), version=3)


def _view(vec):
    return torch.as_tensor(_Words(vec), device="cuda")


def _vector(ctx, words):
    """A vector holding the words of an int64 CUDA tensor."""
    v = vk.Vector(ctx, words.numel(), zero=False)
    ctx.sync()
    _view(v).copy_(words)
    return v


def _generator(seed, salt, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed((seed * 1000003 + salt) % (1 << 62))
    return g


def _uniform(gen, qs, n, device="cuda", pin=False):
    """Words uniform below q for each q of qs, n each, one after another."""
    out = torch.empty(len(qs) * n, dtype=torch.int64, device=device, pin_memory=pin)
    same = {}
    for k, q in enumerate(qs):
        same.setdefault(q, []).append(k)
    rows = out.view(len(qs), n)
    for q, ks in same.items():
        words = torch.randint(0, q, (len(ks), n), dtype=torch.int64, device=device, generator=gen)
        if len(same) == 1:
            rows.copy_(words)
        else:
            rows[torch.tensor(ks, device=device)] = words
    return out


def _shapes(case):
    """(log_n, limbs) of each instance of a ragged batch or of each request."""
    rng = random.Random(case["shape_seed"])
    count = case["instances"] if case["kind"] == "ragged" else case["requests"]
    got, words = [], 0
    for _ in range(count):
        log_n, limbs = rng.randint(case["log_lo"], case["log_hi"]), rng.randint(1, case["max_limbs"])
        if words + (limbs << log_n) > 4 * _MAX_WORDS:
            break
        words += limbs << log_n
        got.append((log_n, limbs))
    return got


def _jobs(case):
    """(op, length) of each element-wise job."""
    rng = random.Random(case["shape_seed"])
    top = np.log2(case["max_len"])
    return [(rng.choice(["elemfma", "elemmul", "elemmod", "elemgtadd", "elemgtsub"]), int(2 ** rng.uniform(0, top)))
            for _ in range(case["jobs"])]


# ---------------------------------------------------------------------------


def _operands(case, seed):
    """The host-made or device-made operands of a case: {name: tensor}."""
    kind = case["kind"]
    if kind in ("calls", "polymul"):
        q = _primes(case["log_n"], case["bits"])[0][0]
        return {k: _uniform(_generator(seed, i), [q], 1 << case["log_n"]) for i, k in enumerate("ab")}
    if kind in ("batch", "transform"):
        p = _primes(case["log_n"], case["bits"])
        if kind == "batch":
            qs = [p[k % len(p)][0] for _ in range(case["products"]) for k in range(case["limbs"])]
        else:
            qs = [p[k % len(p)][0] for k in range(case["count"])]
        names = "ab" if kind == "batch" else "a"
        return {k: _uniform(_generator(seed, i), qs, 1 << case["log_n"]) for i, k in enumerate(names)}
    raise ValueError(kind)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        return _prepare_serve(case, seed)
    ctx = _context()
    st = {"case": case, "ctx": ctx}
    if kind in ("calls", "polymul"):
        ops = _operands(case, seed)
        n = 1 << case["log_n"]
        st["tables"] = _tables(case["log_n"], case["bits"])[0]
        st["a"], st["b"] = _vector(ctx, ops["a"]), _vector(ctx, ops["b"])
        st["out"] = [vk.Vector(ctx, n) for _ in range(4 if kind == "calls" else 1)]
        st["views"] = [_view(v) for v in st["out"]]
    elif kind == "batch":
        ops = _operands(case, seed)
        n = 1 << case["log_n"]
        a, b = _vector(ctx, ops["a"]), _vector(ctx, ops["b"])
        c = vk.Vector(ctx, a.length)
        tabs = _limb_tables(case["log_n"], case["bits"], case["limbs"])
        bt = vk.Batch(ctx)
        if case["operand"] == "lift":  # one job list over all limbs: the epilogue form takes vectors
            bt.add_polymul(tabs * case["products"], a, b, c, lift=[("elemmod", LIFT_MOD, 0)])
        else:
            for i in range(case["products"]):
                off = 8 * i * case["limbs"] * n
                bt.add_polymul(tabs, a.device_ptr + off, b.device_ptr + off, c.device_ptr + off,
                               b_ntt=case["operand"] == "ntt")
        bt.commit(graph=True)
        st.update(batch=bt, keep=(a, b, c), views=[_view(c)])
    elif kind == "transform":
        ops = _operands(case, seed)
        a = _vector(ctx, ops["a"])
        c = vk.Vector(ctx, a.length)
        bt = vk.Batch(ctx)
        bt.add_transform(_limb_tables(case["log_n"], case["bits"], case["count"]), a, c, inverse=case["inverse"],
                         lift=[("elemmod", LIFT_MOD, 0)] if case["lift"] else None)
        bt.commit(graph=True)
        st.update(batch=bt, keep=(a, c), views=[_view(c)])
    elif kind == "ragged":
        shapes = _shapes(case)
        total = sum(l << k for k, l in shapes)
        ab = []
        for i in range(2):
            v = vk.Vector(ctx, total, zero=False)
            ctx.sync()
            out, gen, off = _view(v), _generator(seed, i), 0
            for log_n, limbs in shapes:
                # one draw per instance, below its smallest prime
                p = _primes(log_n, case["bits"])
                out[off:off + (limbs << log_n)] = torch.randint(0, min(q for q, _ in p), (limbs << log_n,),
                                                                dtype=torch.int64, device="cuda", generator=gen)
                off += limbs << log_n
            ab.append(v)
        c = vk.Vector(ctx, total)
        bt = vk.Batch(ctx)
        off = 0
        for log_n, limbs in shapes:
            bt.add_polymul(_limb_tables(log_n, case["bits"], limbs), *[v.device_ptr + 8 * off for v in (*ab, c)])
            off += limbs << log_n
        bt.commit(graph=True)
        st.update(batch=bt, keep=(ab, c), views=[_view(c)])
    elif kind == "elem":
        jobs = _jobs(case)
        q = _primes(14, case["bits"])[0][0]
        total = sum(-(-n // 4) * 4 for _, n in jobs)
        words = [_uniform(_generator(seed, i), [q], total) for i in range(2)]
        a, b = _vector(ctx, words[0]), _vector(ctx, words[1])
        c = vk.Vector(ctx, total)
        eb = vk.ElemBatch(ctx)
        off = 0
        for op, n in jobs:
            pa, pb, pc = (v.device_ptr + 8 * off for v in (a, b, c))
            params = {"elemfma": (123456789, q), "elemmul": (q,), "elemmod": (LIFT_MOD, q),
                      "elemgtadd": (q // 2, 12345), "elemgtsub": (q // 2, q, LIFT_MOD)}[op]
            eb.add(op, pa, pb if op in ("elemfma", "elemmul") else None, (pc, n), *params)
            off += -(-n // 4) * 4
        eb.commit(graph=True)
        st.update(batch=eb, keep=(a, b, c), views=[_view(c)])
    ctx.sync()
    return st


def _prepare_serve(case, seed):
    reqs = []
    for i, (log_n, limbs) in enumerate(_shapes(case)):
        p = _primes(log_n, case["bits"])
        tabs = _limb_tables(log_n, case["bits"], limbs)
        qs = [p[k % len(p)][0] for k in range(limbs)]
        host = []
        for j in range(2):  # made on the GPU (quick), held in pinned host memory
            h = torch.empty(limbs << log_n, dtype=torch.int64, pin_memory=True)
            h.copy_(_uniform(_generator(seed, 2 * i + j), qs, 1 << log_n))
            host.append(h)
        reqs.append((tabs, *host, torch.zeros(limbs << log_n, dtype=torch.int64, pin_memory=True)))
    return {"case": case, "server": _server(), "reqs": reqs}


def run(state):
    kind = state["case"]["kind"]
    if kind == "calls":
        t, a, b = state["tables"], state["a"], state["b"]
        fa, fb, prod, res = state["out"]
        vk.forward_transform(a, fa, t)
        vk.forward_transform(b, fb, t)
        vk.elemmul(fa, fb, prod, t.q)
        vk.inverse_transform(prod, res, t)
        return state["views"]
    if kind == "polymul":
        vk.polymul(state["a"], state["b"], state["out"][0], state["tables"])
        return state["views"]
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit(t, a, b, c) for t, a, b, c in state["reqs"]]
        for rid in ids:
            if srv.wait(rid):
                raise RuntimeError("a request failed")
        return [c for _, _, _, c in state["reqs"]]
    state["batch"].launch()
    return state["views"]


# ---------------------------------------------------------------------------


def _product_work(log_n, transforms, vectors):
    """Bytes and integer operations of one limb job: each vector moved once,
    log2(n) n/2 butterflies (one modular product, one sum, one difference)
    per transform; a product adds n modular products."""
    n = 1 << log_n
    return 8 * n * vectors, transforms * (n // 2) * log_n * 3 + (n if vectors == 3 else 0)


def work(case):
    kind = case["kind"]
    if kind == "calls":  # a, b in; NTT(a), NTT(b), their product and the result out
        b, f = _product_work(case["log_n"], 3, 3)
        return {"bytes": 2 * b, "flops": f}
    if kind == "polymul":
        b, f = _product_work(case["log_n"], 3, 3)
        return {"bytes": b, "flops": f}
    if kind == "batch":
        b, f = _product_work(case["log_n"], 2 if case["operand"] == "ntt" else 3, 3)
        k = case["limbs"] * case["products"]
        return {"bytes": b * k, "flops": f * k}
    if kind == "transform":
        b, f = _product_work(case["log_n"], 1, 2)
        return {"bytes": b * case["count"], "flops": f * case["count"]}
    if kind in ("ragged", "serve"):
        got = [(limbs, _product_work(log_n, 3, 3)) for log_n, limbs in _shapes(case)]
        return {"bytes": sum(k * b for k, (b, _) in got), "flops": sum(k * f for k, (_, f) in got)}
    jobs = _jobs(case)
    return {"bytes": sum(8 * n * (3 if op in ("elemfma", "elemmul") else 2) for op, n in jobs),
            "flops": sum(2 * n for _, n in jobs)}


# ---------------------------------------------------------------------------
# The same results from Python integers (small cases only).


def _bitrev(n):
    bits = n.bit_length() - 1
    r = np.zeros(n, dtype=np.int64)
    for i in range(bits):
        r |= ((np.arange(n) >> i) & 1) << (bits - 1 - i)
    return r


def _roots(n, q, w):
    """Powers of w at bit-reversed places, as Python integers."""
    p = [1] * n
    for i in range(1, n):
        p[i] = p[i - 1] * w % q
    return np.array(p, dtype=object)[_bitrev(n)]


def _forward(x, q, roots):
    n, m = len(x), 1
    x = x.copy()
    while m < n:
        v = x.reshape(m, 2, n // (2 * m))
        t = v[:, 1] * roots[m:2 * m, None] % q
        x = np.stack([(v[:, 0] + t) % q, (v[:, 0] - t) % q], axis=1).reshape(n)
        m *= 2
    return x


def _inverse(x, q, roots):
    n, m = len(x), len(x) // 2
    inv = np.array([pow(int(r), -1, q) for r in roots], dtype=object)
    x = x.copy()
    while m >= 1:
        v = x.reshape(m, 2, n // (2 * m))
        x = np.stack([(v[:, 0] + v[:, 1]) % q, (v[:, 0] - v[:, 1]) * inv[m:2 * m, None] % q], axis=1).reshape(n)
        m //= 2
    return x * pow(n, -1, q) % q


def _centred(x, q):
    """x mod 65537 of the representative of x in (-q/2, q/2]."""
    return np.array([(v - q if v > q // 2 else v) % LIFT_MOD for v in x], dtype=object)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("ragged", "elem", "serve") or work(case)["flops"] > 6_000_000:
        return None
    log_n = case["log_n"]
    n, p = 1 << log_n, _primes(case["log_n"], case["bits"])
    ops = {k: v.cpu().numpy().astype(object) for k, v in _operands(case, seed).items()}
    jobs = {"calls": 1, "polymul": 1, "transform": case.get("count")}.get(kind) or case["limbs"] * case["products"]
    out = []
    for j in range(jobs):
        q, w = p[(j % case["limbs"] if kind == "batch" else j) % len(p)]
        r = _roots(n, q, w)
        a = ops["a"][j * n:(j + 1) * n]
        if kind == "transform":
            y = _inverse(a, q, r) if case["inverse"] else _forward(a, q, r)
            out.append(_centred(y, q) if case["lift"] else y)
            continue
        b = ops["b"][j * n:(j + 1) * n]
        fa = _forward(a, q, r)
        fb = b if case.get("operand") == "ntt" else _forward(b, q, r)
        prod = fa * fb % q
        res = _inverse(prod, q, r)
        if kind == "calls":
            return [x.astype(np.int64) for x in (fa, fb, prod, res)]
        out.append(_centred(res, q) if case.get("operand") == "lift" else res)
    return [np.concatenate(out).astype(np.int64)]
