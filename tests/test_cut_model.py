"""Arithmetic that the kernels do for themselves from lengths the host does not know, restated on the CPU: the cut of few-row calls with a cost for every sequence
(csrc/decode_splitk.cu: every unit is done once, by the columns that count themselves among its sequence's parts), and tile pairs with the heads of a group in a tile
(csrc/prefill_tcgen05.cu: the closed form by which a CTA finds its pair counts what an enumeration counts, and shares of a cluster cover every tile)."""
import random

import pytest


def _columns(units, columns, seq_cost, forced=0):
    """What each column does: [(sequence, first unit, one past the last)], as the kernel walks; and (total, share, more)."""
    total_units = sum(units)
    cost = 0 if forced or total_units <= columns + columns // 8 else seq_cost
    span = [u + cost if u else 0 for u in units]
    total = sum(span)
    columns = min(columns, max(total, 1))
    share, more = divmod(total, columns)
    if share < forced or (share == forced and more == 0):
        share, more = forced, 0
    first = lambda c: share * c + min(c, more)
    begins = [sum(span[:i]) for i in range(len(span))]
    work = []
    for c in range(columns):
        b, e = first(c), min(total, first(c + 1))
        mine = []
        for s, (at, u) in enumerate(zip(begins, units)):
            lo, hi = max(b, at), min(e, at + u)
            if u and lo < hi:
                mine.append((s, lo - at, hi - at))
        work.append(mine)

    def column_of(unit):
        split = more * (share + 1)
        return unit // (share + 1) if unit < split else more + (unit - split) // share
    return work, begins, column_of


@pytest.mark.parametrize("forced", [0, 3])
def test_every_unit_is_done_once_and_every_part_counted(forced):
    rng = random.Random(forced)
    for _ in range(250):
        n = rng.choice([1, 2, 3, 9, 40, 150])
        units = [rng.choice([0, 1, 1, rng.randint(1, 6), rng.randint(1, 200)]) for _ in range(n)]
        if not any(units):
            continue
        columns = rng.choice([1, 2, 9, 37, 55, 148, 222])
        if forced:
            columns = -(-sum(units) // forced)
        work, begins, column_of = _columns(units, columns, rng.choice([3, 5]), forced)
        done = [[0] * u for u in units]
        for mine in work:
            assert sum(1 for s, lo, hi in mine if lo > 0) <= 1 and sum(1 for s, lo, hi in mine if hi < units[s]) <= 1     # one slot each for a part
            for s, lo, hi in mine:
                for u in range(lo, hi):
                    done[s][u] += 1
        assert all(x == 1 for d in done for x in d)
        for s, u in enumerate(units):
            if u:
                parts = column_of(begins[s] + u - 1) - column_of(begins[s]) + 1
                assert parts == sum(1 for mine in work if any(x[0] == s for x in mine))


def _pack_log2(group):
    return min(group & -group, 32).bit_length() - 1


def _tile(idx, packs, pl, q_len, kv_len):
    """K/V tiles of 128 keys that tile `idx` sees."""
    mb = idx // packs
    last = (min(mb * 128 + 128, q_len << pl) - 1) >> pl
    key = min(kv_len - 1, kv_len - q_len + last)
    return key // 128 + 1 if key >= 0 else 0


def test_pairs_of_shared_tiles_by_the_closed_form():
    rng = random.Random(1)
    for _ in range(2500):
        group = rng.choice([1, 2, 3, 4, 6, 8, 12, 16, 32, 64, 5])
        pl = _pack_log2(group)
        packs = group >> pl
        q_len = rng.choice([1, 2, 31, 32, 33, 64, 127, 128, 129, rng.randint(1, 700)])
        kv_len = rng.choice([q_len, rng.randint(0, 3000), q_len + rng.randint(0, 2000)])
        blocks = (q_len + (128 >> pl) - 1) >> (7 - pl)
        assert blocks == -(-(q_len << pl) // 128)
        tiles = packs * blocks
        pairs = (tiles + 1) // 2
        longest = [max(_tile(i, packs, pl, q_len, kv_len) for i in (2 * p, 2 * p + 1) if i < tiles) for p in range(pairs)]
        assert longest == sorted(longest)
        for w in range(0, 26):
            if w <= 0:
                want, got = pairs, pairs
            else:
                key = (w - 1) * 128
                token = key - (kv_len - q_len)
                got = 0 if key >= kv_len or token >= q_len else pairs - (max(token, 0) << pl) // 128 * packs // 2
                want = sum(1 for x in longest if x >= w)
            assert got == want if packs == 1 else abs(got - want) <= packs // 2 + 1     # (heads of one row block in several pairs: an order, not a count, hangs on it)


def test_shares_of_a_cluster_cover_every_tile():
    for parts in (2, 4, 8):
        for n0 in range(0, 70):
            for n1 in (0, max(0, n0 - 1), n0):
                per = -(-max(n0, n1) // parts)
                for n in (n0, n1):
                    shares = [max(0, min(per, n - r * per)) for r in range(parts)]
                    assert sum(shares) == n and all(x == per or not any(shares[i + 1:]) for i, x in enumerate(shares))
