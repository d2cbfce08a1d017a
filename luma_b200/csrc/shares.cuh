// How the kernels share work out among CTAs: arithmetic alone, on the host and on the device (each CTA does it for itself, from lengths that the host does not know).
#pragma once

#include <cuda_runtime.h>

namespace fa {

// Division of n < 2^31 by a divisor the host knows, as a product with its rounded-up inverse (Granlund and Montgomery, "Division by
// invariant integers using multiplication"): a product, a sum and a shift. With the division operator, a CTA made ten divisions by run-time values one after
// the other before its first copy was requested, and knew its extents 1700 clocks from its start (timeline), on an SM with nothing else to do.
struct FastDiv {
    unsigned mul, shift;
    int d;
    FastDiv() = default;
    __host__ explicit FastDiv(int divisor) : mul(0), shift(0), d(divisor) {
        while ((1u << shift) < (unsigned)d) ++shift;
        mul = (unsigned)((((1ULL << shift) - (unsigned)d) << 32) / (unsigned)d) + 1u;
    }
    __host__ __device__ __forceinline__ int div(int n) const {
#ifdef __CUDA_ARCH__
        const unsigned high = __umulhi((unsigned)n, mul);
#else
        const unsigned high = (unsigned)(((unsigned long long)(unsigned)n * mul) >> 32);
#endif
        return (int)((high + (unsigned)n) >> shift);
    }
};

// Query heads of a GQA group that share a tile of the tensor-core prefill kernel: the largest power of two, up to the 32 rows that a warp
// stores at a time, that divides the group.
__host__ __device__ inline int pack_of(int group) {
    const int low = group & -group;
    return low < 32 ? low : 32;
}
// Pairs of 128-row tiles that q_len query tokens make for a KV head there.
__host__ __device__ inline long long prefill_pairs(int group, long long q_len) {
    const int pack = pack_of(group);
    return ((long long)(group / pack) * ((q_len * pack + 127) / 128) + 1) / 2;
}

// Whether n clusters find room at the same time, with one CTA to an SM: as the SMs lie, 33 clusters of four and 15 of eight do on 148.
inline bool clusters_fit(long long n, int ctas, int sms) { return (ctas == 8 ? 21 : ctas == 4 ? 9 : 4) * n <= 2LL * sms; }

// CTAs that share the keys of a tile pair there: of `pairs` pairs in all over up to `tiles` K/V tiles (`exact`: over as many), `rows` rows per KV head and sequence (rule and times
// where it is launched).
inline int prefill_parts(long long pairs, long long tiles, bool exact, long long rows, int sms) {
    if (tiles <= (rows <= 16 && exact ? 7 : 12)) return 1;
    if (clusters_fit(pairs, 8, sms) && tiles >= (rows > 16 ? 32 : 16)) return 8;
    return clusters_fit(pairs, 4, sms) ? 4 : clusters_fit(pairs, 2, sms) ? 2 : 1;
}

// Tile pairs of a stream (sequence, KV head) that sit next to each other in the grid there.
inline int prefill_band(int pairs, long long kv_tiles, int group, int parts) {
    int band = 1;
    while (parts == 1 && band < 8 && band * 2 <= pairs && (long long)(band * 2) * 2 * 8 <= kv_tiles * group) band *= 2;
    return band;
}

// CTAs that share the keys of a row block of the f32 kernel on the tensor cores: of `blocks` in all over `tiles` K/V tiles (tile_f32_tcgen05.cu).
inline int f32_parts(long long blocks, long long tiles, int sms) {
    int c = 1;
    while (c < 8 && clusters_fit(blocks, 2 * c, sms) && tiles >= c * 2) c *= 2;
    return c;
}

// ---- few-row calls (decode_splitk.cu) ----

// What a sequence weighs in the cut: its units, and behind them `cost` units for what it costs a CTA to begin and to end one (its query rows, the merge of the warps' parts, the
// count). Cut by the units alone, the CTAs with the end of a sequence in their share came to their own end 2 to 4 us behind the others (us, before and so: 8 x 4000 contiguous,
// where eight of 37 columns hold one, 27.9 and 26.7; 8 x 512-2048 15.2 and 13.7; 16 x 7 tokens over 1217-4869, 8/2 heads 26.9 and 24.6; 16 x 91-367, 8 heads of 64 11.9 and 9.6).
__host__ __device__ __forceinline__ unsigned rows_span(int units, int cost) { return units > 0 ? (unsigned)(units + cost) : 0u; }
// Where the columns get little more than a unit each there is nothing to even out, and a cost would leave columns empty.
__host__ __device__ __forceinline__ int rows_cost(unsigned total_units, int columns, int seq_cost) { return total_units <= (unsigned)columns + (unsigned)columns / 8u ? 0 : seq_cost; }

// The cut of `total` units into columns: the first `more` columns have share + 1 units, the others share
// (or, forced, every column at least `forced` units). All in 32 bits: a 64-bit division here cost a microsecond of a small call.
struct Cut {
    unsigned share, more;
    __host__ __device__ __forceinline__ Cut(unsigned total, unsigned columns, unsigned forced) {
        share = total / columns;
        more = total - share * columns;
        if (share < forced || (share == forced && more == 0u)) {   // (never less than covers them all, whatever bound the host had)
            share = forced;
            more = 0u;
        }
    }
    __host__ __device__ __forceinline__ unsigned first(unsigned c) const { return share * c + min(c, more); }
    __host__ __device__ __forceinline__ unsigned column_of(unsigned unit) const {
        const unsigned split = more * (share + 1u);
        return unit < split ? unit / (share + 1u) : more + (unit - split) / share;
    }
};

// ---- tile pairs (prefill_tcgen05.cu) ----

constexpr int kBlockM = 128;   // query rows per tile
constexpr int kBlockN = 128;   // keys per K/V tile

// Extents of one sequence. Query row i sits at global position pos_off + i and sees keys
// j < kv_len with j <= pos_off + i (bottom-right aligned for the varlen and kv-cache entry points).
struct SeqExtent {
    int q_len, kv_len, pos_off;   // (positions fit 32 bits: the last one is below kv_len or, batched, kv_seq_len + q_seq_len; see start_pos)
    long long o_row0;     // first row of this sequence in o (rows of o_heads * 128 elements)
    int q_crow, q_cb;     // TMA coordinates (row, batch) of the sequence's first q row
    int kv_crow, kv_cb;   // same for contiguous K/V (unused when paged)
};

struct TileInfo {
    int valid;    // this query tile exists
    int head;     // query head, the first of those that share the tile
    int row0;     // first row, in rows of query token x head of the tile
    int n_kv;     // K/V tiles it needs
};

// One tile pair, as the CTA's roles find it in shared memory.
struct Item {
    int some;            // 0: nothing is left, the CTA ends
    int seq, kv_head;
    SeqExtent sq;
    TileInfo t[2];
};

// ... and its share of the keys, where a cluster has the pair. Not in Item, which the other instantiations carry in the registers of a producer that has none left.
struct Share {
    int first_key;       // where it begins (a multiple of a tile); kv_len, pos_off and kv_crow of the pair's `sq` count from there
    int some;            // the CTAs of the cluster share the keys (0: there are too few, or there is no pair)
};

// Tiles that the query tokens of a sequence fill for `pack` heads.
static_assert(kBlockM == 1 << 7, "rows of a tile");
__host__ __device__ __forceinline__ int row_blocks(int q_len, int pack_log2) { return (q_len + (kBlockM >> pack_log2) - 1) >> (7 - pack_log2); }

// One past the last query token of tile `idx` of a sequence, or of its last tile.
__host__ __device__ __forceinline__ int tile_token_end(const SeqExtent& a, int idx, const FastDiv& by_packs, int pack_log2, int num_mb) {
    const int mb = idx < by_packs.d * num_mb ? by_packs.div(idx) : num_mb - 1;
    return min((mb + 1) * (kBlockM >> pack_log2), a.q_len);
}

template <bool kMask>
__host__ __device__ __forceinline__ TileInfo tile_info(const SeqExtent& a, int pair, int t, int kvh, const FastDiv& by_packs, int pack_log2, int num_mb) {
    TileInfo ti;
    // Tile 0 takes the later index of the pair: where the pair is two consecutive row blocks of the same heads,
    // that is the longer tile, and tile 0 is the one whose copies are requested first and whose
    // products the issuer serves first in every step, so the tile that decides when the CTA ends is never
    // the one that waits (S = 2048 MHA: 887-892 against 851 TFLOP/s).
    const int idx = pair * 2 + (1 - t);
    const int packs = by_packs.d;
    ti.valid = idx < packs * num_mb;
    const int mb = ti.valid ? by_packs.div(idx) : 0;
    ti.head = (kvh * packs + (ti.valid ? idx - mb * packs : 0)) << pack_log2;
    ti.row0 = mb * kBlockM;
    const int last_token = (min(ti.row0 + kBlockM, a.q_len << pack_log2) - 1) >> pack_log2;
    const int last_key = min(a.kv_len - 1, a.pos_off + last_token);
    ti.n_kv = ti.valid && last_key >= 0 ? last_key / kBlockN + 1 : 0;   // 0: the tile sees no key at all
    if (kMask && a.pos_off + (ti.row0 >> pack_log2) >= a.kv_len) ti.n_kv = 0;   // all its rows sit in padding
    return ti;
}

// Tile pairs of one sequence whose longer tile sees at least w K/V tiles (w <= 0: all): pair p holds tiles 2p and
// 2p + 1, tile i the row block i / packs.
__host__ __device__ __forceinline__ int pairs_from(int q_len, int kv_len, int packs, int pack_log2, int w) {
    if (q_len <= 0) return 0;
    const int pairs = (packs * row_blocks(q_len, pack_log2) + 1) / 2;
    if (w <= 0) return pairs;
    const long long key = (long long)(w - 1) * kBlockN;            // such a tile sees this key ...
    const long long token = key - ((long long)kv_len - q_len);     // ... and so does this query token or a later one
    if (key >= kv_len || token >= q_len) return 0;
    return pairs - (int)((max(token, 0LL) << pack_log2) / kBlockM) * packs / 2;
}

// The share of a pair's keys that is this CTA's, of `parts` equal ones in whole tiles. A pair of up to five tiles stays whole, with the first CTA (the host knows a bound only: 2 x 147 tokens
// over 609 keys with room for 2048, 8/2 heads, shared by four 18.9 us, alone 17.5).
__host__ __device__ __forceinline__ Share take_share(Item& w, int parts, int rank) {
    const int most = max(w.t[0].n_kv, w.t[1].n_kv), per = (most + parts - 1) / parts;
    if (most <= 5) {
        w.some = w.some && rank == 0;
        return Share{0, 0};
    }
#pragma unroll
    for (int t = 0; t < 2; ++t) w.t[t].n_kv = max(0, min(per, w.t[t].n_kv - rank * per));
    const int first_key = rank * per * kBlockN;
    w.sq.kv_len -= first_key;
    w.sq.pos_off -= first_key;
    w.sq.kv_crow += first_key;
    return Share{first_key, 1};
}

}  // namespace fa
