"""Batches at n = 10..14: both prime sets in one single-CTA launch, and the
default plans by number of tests."""
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


# 150 tests: more than SMs, the CTAs without plane-split passes
@pytest.mark.parametrize("n,count", [(10, 3), (11, 4), (12, 3), (12, 150), (13, 2), (14, 2)])
def test_both_sets_in_one_launch(n, count):
    bases = [(B3, B2)[i % 2] for i in range(count)]
    got, ref = _squared(bases, n, 0), _squared(bases, n, 3 if n > 10 else 0)
    for i, b in enumerate(bases):
        assert np.array_equal(got[i], ref[i]), i
    one = {b: _squared([b], n, 0)[0] for b in (B2, B3)} if n == 10 else {}
    if one:                                 # n = 10 has no other plan: a lone test is its own reference
        assert np.array_equal(got[0], one[B3])


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
