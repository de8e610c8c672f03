"""The two-prime set of 31-bit primes at the edges of its range: the largest
base it holds, the next one (32-bit primes) and batches that mix the sets,
against the oracle, on every shape of plan."""
import numpy as np
import pytest

from genefer22_b200 import Batch, GfcError, Transform, gint

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
    assert t.width() == 2 and list(t.batch.prime_sets()) == [0 if step else 3]
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


# Set 0 twists its middle pass from n = 22 (8 B of row roots per point, 32 MB), set 3 from n = 21.
@pytest.mark.parametrize("n,plan", [(21, 104), (22, 105), (22, 106), (23, 107)])
@pytest.mark.parametrize("step", [0, 2])
def test_largest_sizes_on_both_two_prime_sets(oracle, n, plan, step):
    b = top_base(n) + step
    t, o = Transform(b, n), oracle.OracleTransform(b, n)
    t.batch.set_plan(plan)
    assert list(t.batch.prime_sets()) == [0 if step else 3]
    d = np.random.default_rng(n + plan).integers(-(b // 2), b // 2 + 1, 1 << n)
    t.setInt(d); o.setInt(d)
    t.copy(1, 0); o.copy(1, 0)
    t.squareDup(True); o.squareDup(True)
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


def _load(oracle, bt, seed):
    """Seeded digits in register 0 of every test, and oracles that hold the same."""
    rng = np.random.default_rng(seed)
    oracles = []
    for i, b in enumerate(int(x) for x in bt.bases):
        d = rng.integers(-(b // 2), b // 2 + 1, 1 << bt.n).astype(np.int32)
        bt.put(i, d)
        oracles.append(oracle.OracleTransform(b, bt.n))
        oracles[-1].setInt(d)
    return oracles


def _squared(bt, oracles, run, times):
    """run() squares register 0 of every test `times` times with dup."""
    run()
    for i, (o, b) in enumerate(zip(oracles, bt.bases)):
        for _ in range(times):
            o.squareDup(True)
        assert np.array_equal(gint.unbalance(bt.get(i), int(b)), gint.unbalance(o.getInt(), int(b))), i


@pytest.mark.parametrize("n,plan", [(10, 0), (11, 0), (12, 0), (12, 1), (13, 0), (13, 1), (14, 0), (14, 1)])
def test_graph_outlives_a_move_between_the_two_prime_sets(oracle, n, plan):
    """A graph recorded with every test on one two-prime set serves a test that
    moves to the other one; a change of width is refused until a new capture."""
    low, high, wide = 1026, top_base(n) + 2, 1_999_999_998
    bt = Batch([low, low + 2], n)
    bt.set_plan(plan)
    g = bt.capture(lambda: bt.square(True, 2))
    for slot, b in ((0, high), (1, high + 2), (0, low)):
        bt.assign(slot, b)
        assert list(bt.widths()) == [2, 2]
        _squared(bt, _load(oracle, bt, b % 97), g.launch, 2)
        _squared(bt, _load(oracle, bt, b % 89), lambda: bt.square(True, 2), 2)
    bt.assign(1, wide)
    with pytest.raises(GfcError):
        g.launch()
    g.close()
    g = bt.capture(lambda: bt.square(True, 2))
    _squared(bt, _load(oracle, bt, 5), g.launch, 2)
    _squared(bt, _load(oracle, bt, 6), lambda: bt.square(True, 2), 2)
    g.close()
    bt.close()


@pytest.mark.parametrize("n,plan", [(12, 0), (12, 1), (13, 3), (14, 5), (15, 1), (16, 4), (18, 103)])
@pytest.mark.parametrize("width", [2, 3])
def test_small_base_in_a_batch_made_without_one(oracle, n, plan, width):
    """A batch made without a base of set 3's range has kernels without its body:
    a small base that comes later (assign, admit) stays on the 32-bit primes."""
    b0 = top_base(n) + 2 if width == 2 else 1_999_999_998 if n <= 15 else 999_999_998
    bt = Batch([b0, b0 + 2], n)
    bt.set_plan(plan)
    assert list(bt.widths()) == [width] * 2
    g = bt.capture(lambda: bt.square(True, 2)) if plan > 1 or width == 2 else None
    bt.assign(0, 1026)
    _squared(bt, _load(oracle, bt, n), lambda: bt.square(True, 2), 2)
    if g is not None:
        _squared(bt, _load(oracle, bt, n + 1), g.launch, 2)
        g.close()
    bt.reserve(64)
    bt.admit(1, 2050, np.array([0b1011], np.uint32), 4)
    bt.assign(0, b0)
    bt.square_exp(4)
    o = oracle.OracleTransform(2050, n)
    o.set(1)
    for bit in (True, False, True, True):
        o.squareDup(bit)
    assert np.array_equal(gint.unbalance(bt.get(1), 2050), gint.unbalance(o.getInt(), 2050))
    bt.close()


@pytest.mark.parametrize("n,plan", [(11, 0), (12, 0), (12, 1), (13, 3), (14, 1), (16, 4), (18, 103)])
def test_admissions_across_the_sets(oracle, n, plan):
    """A reserved batch on set 3 whose slots take tests of every set, and of set 3 again."""
    wide = 1_999_999_998 if n <= 15 else 999_999_998
    bt = Batch([1026, 2050, 4098], n)
    bt.set_plan(plan)
    bt.reserve(64)
    bits = (True, False, True, True)
    for bases, sets in (([top_base(n) + 2, wide, 1028], [0, 1, 3]), ([2052, top_base(n) + 4, wide - 2], [3, 0, 1]),
                        ([1030, 2054, 4100], [3, 3, 3])):
        for i, b in enumerate(bases):
            bt.admit(i, b, np.array([0b1011], np.uint32), 4)
        assert list(bt.prime_sets()) == sets
        bt.square_exp(4)
        for i, b in enumerate(bases):
            o = oracle.OracleTransform(b, n)
            o.set(1)
            for bit in bits:
                o.squareDup(bit)
            assert np.array_equal(gint.unbalance(bt.get(i), b), gint.unbalance(o.getInt(), b)), (sets, i)
        # dense digits through the same slots
        _squared(bt, _load(oracle, bt, n), lambda: bt.square(True, 2), 2)
    bt.close()
