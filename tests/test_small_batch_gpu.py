"""Batches at n = 10..14: every mix of prime sets in one single-CTA launch, and
the default plans by number of tests."""
import math
import time

import numpy as np
import pytest

from genefer22_b200 import Batch, gint

pytestmark = pytest.mark.gpu

B2, B3 = 1_000_002, 1_999_999_998          # two and three primes


def _squared(bases, n, plan, steps=3):
    """Canonical residues of every test after a few squarings and a product from seeded digits."""
    bt = Batch(bases, n)
    if plan is not None:
        bt.set_plan(plan)
    rng = np.random.default_rng(n)
    for i, b in enumerate(bases):
        bt.put(i, rng.integers(-(b // 2), b // 2 + 1, 1 << n).astype(np.int32))
    bt.copy(1, 0)
    bt.square(True, steps)
    bt.init_multiplicand(1)
    bt.mul_into(0)
    out = [gint.unbalance(bt.get(i), b) for i, b in enumerate(bases)]
    bt.close()
    return out


def _base(n, prime_set):
    """A base of prime set 3 (two 31-bit primes), 0 (two 32-bit primes) or 1 (three primes) at size n."""
    m3 = (127 * 2**24 + 1) * (63 * 2**25 + 1)
    return {3: 1_026, 0: 2 * math.isqrt((m3 // 2) >> n), 1: B3}[prime_set]


# 160 tests: more than SMs, the CTAs without plane-split passes
@pytest.mark.parametrize("sets", [(3,), (0,), (1,), (3, 0), (0, 1), (3, 1), (3, 0, 1)])
@pytest.mark.parametrize("n,count", [(10, 4), (10, 160), (11, 4), (11, 160), (12, 4), (12, 160), (13, 4), (14, 4)])
@pytest.mark.parametrize("made", ["at once", "by assign"])
def test_both_sets_in_one_launch(oracle, n, count, sets, made):
    """One single-CTA launch over tests of any prime sets; tests moved from set 3
    leave a batch whose kernels hold its body beside theirs."""
    bases = [_base(n, sets[i % len(sets)]) for i in range(count)]
    if made == "at once":
        bt = Batch(bases, n)
    else:
        bt = Batch([_base(n, 3)] * count, n)
        for i, b in enumerate(bases):
            bt.assign(i, b)
    bt.set_plan(0)
    rng = np.random.default_rng(n)
    digits = {b: rng.integers(-(b // 2), b // 2 + 1, 1 << n).astype(np.int32) for b in bases}
    bt.put_all(np.stack([digits[b] for b in bases]))
    bt.copy(1, 0)
    bt.square(True, 2)
    g = bt.capture(lambda: bt.square(False, 2))
    g.launch()
    bt.init_multiplicand(1)
    bt.mul_into(0)
    got = bt.get_all(0)
    g.close()
    bt.close()
    for b, d in digits.items():
        o = oracle.OracleTransform(b, n)
        o.setInt(d)
        o.copy(1, 0)
        for dup in (True, True, False, False):
            o.squareDup(dup)
        o.initMultiplicand(1)
        o.mul()
        ref = gint.unbalance(o.getInt(), b)
        for i in range(count):
            assert bases[i] != b or np.array_equal(gint.unbalance(got[i], b), ref), i


@pytest.mark.parametrize("n,bases,plan", [
    (12, [B2] * 48, 1), (12, [B2, B3] * 25, 0), (13, [B2, B3] * 6, 1), (13, [B2] * 13, 3), (13, [B3] * 64, 0),
    (13, [B2, B3] * 40, 3), (14, [B3] * 7, 1), (14, [B2] * 8, 3), (14, [B2, B3] * 40, 3), (14, [B3] * 64, 0)])
def test_default_small_plans(n, bases, plan):
    bt = Batch(bases, n, num_regs=2)
    assert bt.plan() == plan
    bt.close()
    if len(bases) <= 13:
        got, ref = _squared(bases, n, None), _squared(bases, n, 0)
        assert all(np.array_equal(g, r) for g, r in zip(got, ref))


@pytest.mark.parametrize("n", [12, 13, 14])
def test_cluster_default_while_every_cluster_runs_at_once(oracle, n):
    """The last number of tests on the cluster plan and the first one past it square
    right, of every prime set, and the last takes no second wave of clusters."""
    plans = {}
    for count in range(1, 64):
        bt = Batch([B2] * count, n, num_regs=1)
        plans[count] = bt.plan()
        bt.close()
    last = max(c for c, p in plans.items() if p == 1)
    assert all(plans[c] == 1 for c in range(1, last + 1))
    d = {}
    for count in (last, last + 1):
        bases = [_base(n, (3, 0, 1)[i % 3]) for i in range(count)]
        bt = Batch(bases, n)
        rng = np.random.default_rng(n)
        for i, b in enumerate(bases):
            d.setdefault(b, rng.integers(-(b // 2), b // 2 + 1, 1 << n).astype(np.int32))
            bt.put(i, d[b])
        bt.square(True, 2)
        got = bt.get_all(0)
        bt.close()
        for b in d:
            o = oracle.OracleTransform(b, n)
            o.setInt(d[b])
            o.squareDup(True)
            o.squareDup(True)
            ref = gint.unbalance(o.getInt(), b)
            assert all(bases[i] != b or np.array_equal(gint.unbalance(got[i], b), ref) for i in range(count))

    def us(count):
        bt = Batch([B2] * count, n)
        bt.set_plan(1)
        g = bt.capture(lambda: bt.square(False, 400))
        best = 1e9
        for _ in range(5):
            bt.sync()
            t0 = time.perf_counter()
            g.launch()
            bt.sync()
            best = min(best, time.perf_counter() - t0)
        g.close()
        bt.close()
        return best

    one, full = us(1), us(last)
    assert full < 1.8 * one, (one, full)      # a second wave takes twice the time
