"""The two-prime set of 31-bit primes at the edges of its range: the largest
base it holds, the next one (32-bit primes) and batches that mix the sets,
against the oracle, on every shape of plan."""
import numpy as np
import pytest

from genefer22_b200 import Batch, Transform, gint

pytestmark = pytest.mark.gpu

M3 = (127 * 2**24 + 1) * (63 * 2**25 + 1)


def top_base(n):
    """Largest even b with 2^n (b/2 + 1)^2 < M3 / 2."""
    b = 2
    for k in range(30, 0, -1):
        if (1 << n) * ((b + (1 << k)) // 2 + 1) ** 2 < M3 // 2:
            b += 1 << k
    return b


@pytest.mark.parametrize("n,plan", [(10, 0), (11, 3), (12, 0), (12, 1), (13, 1), (14, 1), (13, 3), (14, 4), (14, 6), (15, 1),
                                    (16, 4), (18, 10), (17, 103), (18, 104), (19, 105), (20, 106), (21, 107)])
@pytest.mark.parametrize("step", [0, 2])
def test_edge_of_the_range(oracle, n, plan, step):
    b = top_base(n) + step
    t = Transform(b, n)
    t.batch.set_plan(plan)
    assert t.width() == 2
    o = oracle.OracleTransform(b, n)
    d = np.full(1 << n, b // 2, dtype=np.int64)              # every product coefficient at its largest
    d[np.random.default_rng(n).integers(0, 1 << n, 9)] -= 1
    t.setInt(d)
    o.setInt(d)
    for dup in (False, True):
        t.squareDup(dup)
        o.squareDup(dup)
    t.copy(1, 0); o.copy(1, 0)
    t.mul(1); o.mul(1)
    assert np.array_equal(gint.unbalance(t.getInt(), b), gint.unbalance(o.getInt(), b))


@pytest.mark.parametrize("n,plan", [(12, 0), (12, 1), (13, 3), (14, 5), (16, 103)])
def test_mixed_sets(oracle, n, plan):
    bases = [top_base(n), 1_999_999_998 if n <= 15 else 1_400_000_000, top_base(n) + 2, 1026]
    bt = Batch(bases, n)
    bt.set_plan(plan)
    rng = np.random.default_rng(n + plan)
    digs = [rng.integers(-(b // 2), b // 2 + 1, 1 << n).astype(np.int32) for b in bases]
    for i, d in enumerate(digs):
        bt.put(i, d)
    bt.square(True, 3)
    for i, b in enumerate(bases):
        o = oracle.OracleTransform(b, n)
        o.setInt(digs[i])
        for _ in range(3):
            o.squareDup(True)
        assert np.array_equal(gint.unbalance(bt.get(i), b), gint.unbalance(o.getInt(), b)), i
    bt.close()
