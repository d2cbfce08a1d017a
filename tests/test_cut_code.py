"""The arithmetic by which CTAs share work, from lengths that the host does not know (csrc/shares.cuh), compiled for the host and compared with enumerations: the cut of few-row
calls with a cost for every sequence (csrc/decode_splitk.cu: every unit is done once, by the columns that count themselves among its sequence's parts), and tile pairs with the heads
of a group in a tile (csrc/prefill_tcgen05.cu: every row of every head in one tile, the keys that a tile sees, the closed form by which a CTA finds its pair, shares of a cluster)."""
import ctypes
import random
import subprocess
from pathlib import Path

import pytest

from luma_b200.build import find_nvcc


@pytest.fixture(scope="module")
def code(tmp_path_factory):
    out = tmp_path_factory.mktemp("shares") / "shares.so"
    subprocess.run([find_nvcc(), "-std=c++17", "-O2", "-shared", "-Xcompiler", "-fPIC", "-gencode", "arch=compute_100a,code=sm_100a", str(Path(__file__).parent / "cpp" / "shares.cu"), "-o", str(out)],
                   check=True)
    lib = ctypes.CDLL(str(out))
    lib.cut_span.restype = lib.cut_column_of.restype = ctypes.c_uint
    lib.pair_count.restype = ctypes.c_longlong
    lib.pair_count.argtypes = [ctypes.c_int, ctypes.c_longlong]
    lib.f32_pair_parts.argtypes = [ctypes.c_longlong, ctypes.c_longlong, ctypes.c_int]
    lib.pair_band.argtypes = [ctypes.c_int, ctypes.c_longlong, ctypes.c_int, ctypes.c_int]
    lib.pair_parts.argtypes = [ctypes.c_longlong, ctypes.c_longlong, ctypes.c_int, ctypes.c_longlong, ctypes.c_int]
    return lib


def _columns(code, units, columns, seq_cost, forced=0):
    """What each column does: [(sequence, first unit, one past the last)], where the sequences begin, and the column of a unit."""
    cost = 0 if forced else code.cut_cost(sum(units), columns, seq_cost)
    span = [code.cut_span(u, cost) for u in units]
    total = sum(span)
    columns = min(columns, max(total, 1))
    first = (ctypes.c_uint * (columns + 1))()
    code.cut_firsts(total, columns, forced, first)
    begins = [sum(span[:i]) for i in range(len(span))]
    work = []
    for c in range(columns):
        b, e = first[c], min(total, first[c + 1])
        work.append([(s, max(b, at) - at, min(e, at + u) - at) for s, (at, u) in enumerate(zip(begins, units)) if u and max(b, at) < min(e, at + u)])
    return work, begins, lambda unit: code.cut_column_of(total, columns, forced, unit)


@pytest.mark.parametrize("forced", [0, 3])
def test_every_unit_is_done_once_and_every_part_counted(code, forced):
    rng = random.Random(forced)
    for _ in range(250):
        n = rng.choice([1, 2, 3, 9, 40, 150])
        units = [rng.choice([0, 1, 1, rng.randint(1, 6), rng.randint(1, 200)]) for _ in range(n)]
        if not any(units):
            continue
        columns = rng.choice([1, 2, 9, 37, 55, 148, 222])
        if forced:
            columns = -(-sum(units) // forced)
        work, begins, column_of = _columns(code, units, columns, rng.choice([3, 5]), forced)
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


def test_columns_end_within_a_unit_of_one_another(code):
    rng = random.Random(5)
    for _ in range(300):
        units = [rng.randint(1, 300) for _ in range(rng.randint(1, 60))]
        columns, cost = rng.choice([37, 55, 148]), rng.choice([0, 3, 5])
        total = sum(code.cut_span(u, cost) for u in units)
        first = (ctypes.c_uint * (columns + 1))()
        code.cut_firsts(total, columns, 0, first)
        shares = [first[c + 1] - first[c] for c in range(columns)]
        assert first[0] == 0 and first[columns] == total and max(shares) - min(shares) <= 1


def test_division_by_an_inverse(code):
    rng = random.Random(2)
    for _ in range(20000):
        d = rng.choice([1, 2, 3, 5, 7, 8, 12, 64, 127, rng.randint(1, 1 << 20), rng.randint(1, (1 << 31) - 1)])
        n = rng.choice([0, 1, d - 1, d, min(d * rng.randint(1, 9), (1 << 31) - 1), rng.randint(0, (1 << 31) - 1), (1 << 31) - 1])
        assert code.divided(n, d) == n // d


def _tiles(code, q_len, kv_len, pos_off, group, mask=0, kv_head=0):
    """Tiles of a sequence and KV head by pair, tile 1 (the earlier) first: (valid, head, row0, K/V tiles)."""
    pl = code.pair_pack(group).bit_length() - 1
    got = []
    for pair in range(code.pair_count(group, q_len)):
        for t in (1, 0):
            out = (ctypes.c_int * 4)()
            code.pair_tile(q_len, kv_len, pos_off, pair, t, kv_head, group >> pl, pl, mask, out)
            got.append(tuple(out))
    return got, pl


GROUPS = [1, 2, 3, 4, 5, 6, 8, 12, 16, 32, 64, 96]


def test_every_row_is_in_one_tile_and_sees_its_keys(code):
    rng = random.Random(1)
    for _ in range(300):
        group, kv_head = rng.choice(GROUPS), rng.randint(0, 3)
        q_len = rng.choice([1, 2, 31, 32, 33, 64, 127, 128, 129, rng.randint(1, 500)])
        kv_len = rng.choice([q_len, rng.randint(0, 3000), q_len + rng.randint(0, 2000)])
        pos_off = rng.choice([0, kv_len - q_len, rng.randint(0, 2500)])
        tiles, pl = _tiles(code, q_len, kv_len, pos_off, group, kv_head=kv_head)
        rows = set()
        for i, (valid, head, row0, n_kv) in enumerate(tiles):
            assert valid or i == len(tiles) - 1                  # the last pair may have one tile
            if not valid:
                assert n_kv == 0
                continue
            mine = [(row >> pl, head + (row & ((1 << pl) - 1))) for row in range(row0, row0 + 128) if row >> pl < q_len]
            assert mine and not rows & set(mine)
            rows |= set(mine)
            seen = [min(kv_len, pos_off + token + 1) for token, _ in mine]
            assert n_kv == max(0, -(-max(seen) // 128))
            assert code.pair_token_end(q_len, i, group >> pl, pl) == max(token for token, _ in mine) + 1
        assert rows == {(token, kv_head * group + h) for token in range(q_len) for h in range(group)}


def test_a_tile_whose_rows_are_all_padding_sees_nothing(code):
    for group in GROUPS:
        for q_len, kv_len in ((300, 200), (300, 300), (64, 1), (400, 127), (129, 128)):
            for (valid, _, row0, n_kv), (_, _, _, plain) in zip(_tiles(code, q_len, kv_len, 0, group, 1)[0], _tiles(code, q_len, kv_len, 0, group)[0]):
                pl = code.pair_pack(group).bit_length() - 1
                assert n_kv == (0 if row0 >> pl >= kv_len else plain)


def test_pairs_by_the_closed_form(code):
    """A CTA finds its pair by counting the pairs of at least w K/V tiles per sequence."""
    rng = random.Random(3)
    for _ in range(1500):
        group = rng.choice(GROUPS)
        pl = code.pair_pack(group).bit_length() - 1
        packs = group >> pl
        q_len = rng.choice([1, 2, 31, 32, 33, 64, 127, 128, 129, rng.randint(1, 700)])
        kv_len = rng.choice([q_len, rng.randint(0, 3000), q_len + rng.randint(0, 2000)])
        tiles, _ = _tiles(code, q_len, kv_len, kv_len - q_len, group)
        longest = [max(tiles[2 * p][3], tiles[2 * p + 1][3]) for p in range(len(tiles) // 2)]
        assert longest == sorted(longest)
        for w in range(0, 27):
            assert code.pair_from(q_len, kv_len, packs, pl, w) == sum(1 for x in longest if x >= w)


def test_shares_of_a_cluster_cover_every_tile(code):
    for parts in (2, 4, 8):
        for n0 in range(0, 70):
            for n1 in (0, max(0, n0 - 1), n0):
                got = []
                for rank in range(parts):
                    out = (ctypes.c_int * 8)()
                    code.pair_share(n0, n1, 9000, 8000, parts, rank, out)
                    got.append(list(out))
                if max(n0, n1) <= 5:                              # stays whole, with the first CTA
                    assert [x[:2] for x in got] == [[1, 0]] + [[0, 0]] * (parts - 1) and got[0][2:] == [0, n0, n1, 9000, 8000, 1000]
                    continue
                for rank, (some, shared, first, a, b, kv_len, pos_off, row) in enumerate(got):
                    assert some and shared and first % 128 == 0 and (kv_len, pos_off, row) == (9000 - first, 8000 - first, 1000 + first)
                    assert rank == 0 or first // 128 == rank * -(-max(n0, n1) // parts)
                for n, i in ((n0, 3), (n1, 4)):
                    at = 0
                    for x in got:
                        assert x[i] == 0 or x[2] // 128 == at     # from where the share before ended
                        at += x[i]
                    assert at == n


def test_clusters_have_room(code):
    for sms in (148, 132, 64):
        for pairs in range(1, 200):
            for tiles in (1, 7, 8, 12, 13, 16, 31, 32, 256):
                for rows in (1, 16, 17, 4096):
                    for exact in (0, 1):
                        parts = code.pair_parts(pairs, tiles, exact, rows, sms)
                        assert parts in (1, 2, 4, 8) and (parts == 1 or parts * pairs <= sms and tiles >= parts and tiles > 7)


def test_clusters_of_the_f32_kernel_have_room(code):
    for blocks in range(1, 200):
        for tiles in range(1, 70):
            parts = code.f32_pair_parts(blocks, tiles, 148)
            assert parts == 1 or tiles >= parts and blocks <= {2: 74, 4: 33, 8: 15}[parts]     # at the same time: as the SMs lie


def test_a_grid_of_clusters_has_no_more_than_its_pairs(code):
    for group in GROUPS:
        for pairs in range(1, 75):
            for tiles in (8, 13, 16, 32, 64, 256):
                for streams in (1, 2, 3, 8, 24, 37):
                    parts = code.pair_parts(pairs * streams, tiles, 0, 4096, 148)
                    band = code.pair_band(pairs, tiles, group, parts)
                    assert 1 <= band <= min(8, pairs)
                    assert parts == 1 or -(-pairs // band) * band * streams * parts <= 148
