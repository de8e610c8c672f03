"""The work that users of this package have it do, as cases that can be timed.

Three kinds, each through the package's public entry points:

  one    one Fermat PRP test as genefer drives its transform: a squareDup call
         per exponent bit, and (``gl``) the Gerbicz-Li update of d(t) that ends
         a block (copy, mul, copy, copy)
  prime  the deterministic test's loop: a squareMul call per exponent bit
         (base a on the set bits, 1 on the others)
  batch  many tests of one size: Gerbicz-Li blocks (B squarings with each
         test's own exponent bits, then the d(t) update) replayed from a CUDA
         graph

A pass runs a stretch of an exponentiation from a dense residue and reads the
registers back, as a program does at a checkpoint or at the end of a test.
Bases are even, log-uniform in [b_lo, b_hi] (or uniform, where the case says so).  The digits the engine returns
stand for a residue but are not unique (balanced, a unit of carry may stay
unreduced), so a pass returns them in the one canonical form, digits in [0, b).
"""
import math

import numpy as np
import torch

from genefer22_b200.transform import Batch, Transform

# Largest base per size that genefer tests (n >= 19: its CPU limits, as the
# serving and uneven workloads of this package use).
B_MAX = {15: 2_000_000_000, 16: 1_500_000_000, 17: 1_000_000_000, 18: 1_000_000_000, 19: 70_000_000, 20: 55_000_000,
         21: 45_000_000, 22: 35_000_000, 23: 25_000_000}
BLOCK = 1000            # Gerbicz-Li block of the batched workloads
# no drawn case does more digit-squarings than the largest listed one
MOST_DIGIT_SQUARINGS = 400 << 23


def b_max(n):
    return 2_000_000_000 if n <= 15 else B_MAX[n]


def listed():
    return [
        # the smallest call: a lone n = 12 test, latency and launches
        {"name": "one n12", "kind": "one", "n": 12, "b_lo": 1024, "b_hi": 2_000_000, "steps": 512, "gl": False},
        # the primality proof of a small find
        {"name": "prime n13", "kind": "prime", "n": 13, "b_lo": 1024, "b_hi": 2_000_000, "steps": 512, "gl": False},
        # a lone test whose base needs the widest number of primes
        {"name": "one n15 large base", "kind": "one", "n": 15, "b_lo": 500_000_000, "b_hi": 2_000_000_000, "steps": 512, "gl": False},
        # an ordinary lone test
        {"name": "one n17", "kind": "one", "n": 17, "b_lo": 1_000_000, "b_hi": 100_000_000, "steps": 512, "gl": False},
        # the verified large test: a block ends with its Gerbicz-Li update
        {"name": "one n20", "kind": "one", "n": 20, "b_lo": 1_000_000, "b_hi": 50_000_000, "steps": 1000, "gl": True},
        # a large size at the small bases where its search begins
        {"name": "one n21 small base", "kind": "one", "n": 21, "b_lo": 50_000, "b_hi": 1_000_000, "steps": 600, "gl": False},
        # the two largest sizes
        {"name": "one n22", "kind": "one", "n": 22, "b_lo": 2_000_000, "b_hi": 35_000_000, "steps": 600, "gl": False},
        {"name": "one n23", "kind": "one", "n": 23, "b_lo": 20_000_000, "b_hi": 25_000_000, "steps": 400, "gl": False},
        # the size class that holds most of an uneven batch, bases of every width
        {"name": "batch n12 x 102", "kind": "batch", "n": 12, "count": 102, "b_lo": 1024, "b_hi": 2_000_000_000, "blocks": 2},
        {"name": "batch n14 x 38", "kind": "batch", "n": 14, "count": 38, "b_lo": 1024, "b_hi": 2_000_000_000, "blocks": 2},
        # the batched search at the headline size
        {"name": "batch n16 x 64", "kind": "batch", "n": 16, "count": 64, "b_lo": 1_000_000, "b_hi": 100_000_000, "blocks": 2, "uniform": True},
        # a serving pool, bases up to the size's limit
        {"name": "batch n18 x 8", "kind": "batch", "n": 18, "count": 8, "b_lo": 50_000_000, "b_hi": 1_000_000_000, "blocks": 2},
    ]


def _bases_range(rng, n):
    """The bases of a search at size n: small, ordinary, or up to the limit."""
    top = b_max(n)
    edges = [1024, 1_000_000, min(100_000_000, top), top]
    lo, hi = rng.choice([(0, 1), (1, 2), (1, 2), (0, 3), (2, 3)])
    if edges[lo] >= edges[hi]:
        lo, hi = 1, 3
    return edges[lo], edges[hi]


def draw(rng):
    kind = rng.choice(["one", "one", "one", "batch", "batch", "prime"])
    if kind == "batch":
        n = rng.randint(12, 20)
        lo, hi = _bases_range(rng, n)
        most = min(130 if n <= 13 else 64, MOST_DIGIT_SQUARINGS // (BLOCK << n))
        count = max(1, int(math.exp(rng.uniform(0.0, math.log(most + 1)))))
        blocks = max(1, min(2, MOST_DIGIT_SQUARINGS // (count * BLOCK << n)))
        return {"kind": kind, "n": n, "count": count, "b_lo": lo, "b_hi": hi, "blocks": blocks, "uniform": rng.random() < 0.5}
    n = rng.randint(12, 16) if kind == "prime" else rng.randint(12, 23)
    lo, hi = _bases_range(rng, n)
    steps = min(int(math.exp(rng.uniform(math.log(200), math.log(1000)))), MOST_DIGIT_SQUARINGS >> n)
    return {"kind": kind, "n": n, "b_lo": lo, "b_hi": hi, "steps": steps, "gl": kind == "one" and rng.random() < 0.5}


def _bases(case, rng, count):
    lo, hi = case["b_lo"], case["b_hi"]
    b = rng.uniform(lo, hi, count) if case.get("uniform") else np.exp(rng.uniform(math.log(lo), math.log(hi), count))
    return [max(lo, int(x)) & ~1 for x in b]


def _inputs(case, seed):
    """Bases, canonical digits of register 0 per test, exponent bits (first squaring first)."""
    rng = np.random.default_rng(seed)
    count = case.get("count", 1)
    bases = _bases(case, rng, count)
    digits = [rng.integers(0, b, 1 << case["n"], dtype=np.int32) for b in bases]
    steps = case["blocks"] * BLOCK if case["kind"] == "batch" else case["steps"]
    bits = rng.integers(0, 2, (count, steps), dtype=np.uint8)
    return bases, digits, bits


def prepare(case, seed):
    bases, digits, bits = _inputs(case, seed)
    n = case["n"]
    if case["kind"] != "batch":
        t = Transform(bases[0], n, 3)
        t.setInt(digits[0])
        if case["kind"] == "one" and case["gl"]:
            t.copy(1, 0)
        return {"case": case, "t": t, "b": bases[0], "bits": [bool(x) for x in bits[0]], "a": 3}
    bt = Batch(bases, n, 3)
    bal = np.stack([np.where(d > b // 2, d - b, d) for d, b in zip(digits, bases)]).astype(np.int32)
    bt.put_all(bal, 0)
    bt.put_all(bal, 1)
    steps = bits.shape[1]
    words = (steps + 31) // 32
    for i in range(len(bases)):
        w = np.packbits(bits[i][::-1], bitorder="little")      # the first squaring takes the top bit
        w = np.concatenate([w, np.zeros(4 * words - w.size, np.uint8)]).view("<u4")
        bt.set_exponent(i, w, steps)
    graph = bt.capture(lambda: (bt.square_exp(BLOCK), bt.gl_step()))
    return {"case": case, "bt": bt, "graph": graph, "bases": np.array(bases, np.int32)[:, None],
            "pos": np.full(len(bases), steps - 1, np.int64), "out": [np.empty((len(bases), 1 << n), np.int32) for _ in range(2)]}


def _unbalanced(d, b):
    """Digits in [0, b) of the residues modulo b^N + 1 that the balanced digits d (a row per test, |d| <= b/2 + 1)
    stand for; in place."""
    x, b = torch.from_numpy(d), torch.from_numpy(b)
    sign = x >> 31                                              # -1 where the digit is negative
    x[:, 1:] += sign[:, :-1]                                    # it takes b from the next digit
    x[:, 0] -= sign[:, -1]                                      # b^N = -1
    x += sign.bitwise_and_(b)
    while x.amin() < 0 or (x - b).amax() >= 0:                # a digit 0 lent, or one reached b: rare
        for i, j in ((x < 0) | (x >= b)).nonzero().tolist():
            q = int(x[i, j]) // int(b[i, 0])                    # -1 below zero, 1 from b
            x[i, j] -= q * int(b[i, 0])
            if j + 1 < x.shape[1]:
                x[i, j + 1] += q
            else:
                x[i, 0] -= q
    return d


def run(s):
    case = s["case"]
    if case["kind"] == "batch":
        bt = s["bt"]
        bt.set_pos(s["pos"])
        for _ in range(case["blocks"]):
            s["graph"].launch()
        return {"residues": _unbalanced(bt.get_all(0, s["out"][0]), s["bases"]),
                "check": _unbalanced(bt.get_all(1, s["out"][1]), s["bases"])}
    t, b = s["t"], np.array([[s["b"]]], np.int32)
    if case["kind"] == "prime":
        a = s["a"]
        for bit in s["bits"]:
            t.squareMul(a if bit else 1)
    else:
        for bit in s["bits"]:
            t.squareDup(bit)
        if case["gl"]:                                          # the end of a block, as genefer's prp loop has it
            t.copy(2, 0)
            t.mul(1)
            t.copy(1, 0)
            t.copy(0, 2)
    out = {"residue": _unbalanced(t.getInt()[None, :], b)}
    if case["gl"]:
        out["check"] = _unbalanced(t.batch.get(0, 1)[None, :], b)
    return out


def work(case):
    """Per squaring: each digit of the register read once and written once; the
    additions, subtractions and products of a forward and an inverse transform
    over the two words that a coefficient of the product needs at least."""
    count = case.get("count", 1)
    steps = case["blocks"] * (BLOCK + 1) if case["kind"] == "batch" else case["steps"]
    N = 1 << case["n"]
    return {"bytes": 8 * N * count * steps, "flops": 2 * (3 * N * case["n"] + N) * count * steps}


def tolerance(case):
    return "exact"


# ---- plain integers

def _to_int(d, b):
    v = [int(x) for x in d]
    p = b
    while len(v) > 1:
        v = [v[i] + v[i + 1] * p for i in range(0, len(v), 2)]
        p = p * p
    return v[0]


def _to_digits(x, b, n):
    pw = [b]
    for _ in range(n - 1):
        pw.append(pw[-1] * pw[-1])
    v = [x]
    for p in reversed(pw):
        v = [y for z in v for y in (z % p, z // p)]
    return v


def exact(case, seed):
    if case["kind"] == "batch" or case["n"] > 13:
        return None                                             # minutes of big-integer products
    bases, digits, bits = _inputs(case, seed)
    b, n = bases[0], case["n"]
    if (b.bit_length() << n) * case["steps"] > 80_000_000:
        return None
    top = b ** (1 << n)
    mod = top + 1
    x = _to_int(digits[0], b) % mod
    r1 = x
    for bit in bits[0]:
        hi, lo = divmod(x * x * (1 if not bit else 3 if case["kind"] == "prime" else 2), top)
        x = lo - hi                                             # b^N = -1
        while x < 0:
            x += mod
    def row(v):
        if v == top:                                            # -1 has the digits -1, 0, 0, ...
            return np.array([[-1] + [0] * ((1 << n) - 1)], np.int32)
        return np.array([_to_digits(v, b, n)], np.int32)

    out = {"residue": row(x)}
    if case["gl"]:
        out["check"] = row(x * r1 % mod)
    return out
