// The arithmetic by which CTAs share work (luma_b200/csrc/shares.cuh) for tests/test_cut_code.py, which calls it on the host.
#include "../../luma_b200/csrc/shares.cuh"

using namespace fa;

namespace {
SeqExtent extent(int q_len, int kv_len, int pos_off) {
    SeqExtent e{};
    e.q_len = q_len;
    e.kv_len = kv_len;
    e.pos_off = pos_off;
    return e;
}
}  // namespace

extern "C" {
unsigned cut_span(int units, int cost) { return rows_span(units, cost); }
int cut_cost(unsigned total_units, int columns, int seq_cost) { return rows_cost(total_units, columns, seq_cost); }
void cut_firsts(unsigned total, unsigned columns, unsigned forced, unsigned* first) {
    const Cut cut(total, columns, forced);
    for (unsigned c = 0; c <= columns; ++c) first[c] = cut.first(c);
}
unsigned cut_column_of(unsigned total, unsigned columns, unsigned forced, unsigned unit) { return Cut(total, columns, forced).column_of(unit); }
int divided(int n, int d) { return FastDiv(d).div(n); }
int pair_pack(int group) { return pack_of(group); }
long long pair_count(int group, long long q_len) { return prefill_pairs(group, q_len); }
int pair_blocks(int q_len, int pack_log2) { return row_blocks(q_len, pack_log2); }
int pair_from(int q_len, int kv_len, int packs, int pack_log2, int w) { return pairs_from(q_len, kv_len, packs, pack_log2, w); }
int pair_token_end(int q_len, int idx, int packs, int pack_log2) { return tile_token_end(extent(q_len, 0, 0), idx, FastDiv(packs), pack_log2, row_blocks(q_len, pack_log2)); }
// {valid, head, row0, n_kv} of tile t of a pair
void pair_tile(int q_len, int kv_len, int pos_off, int pair, int t, int kv_head, int packs, int pack_log2, int mask, int* out) {
    const SeqExtent e = extent(q_len, kv_len, pos_off);
    const FastDiv by(packs);
    const int blocks = row_blocks(q_len, pack_log2);
    const TileInfo ti = mask ? tile_info<true>(e, pair, t, kv_head, by, pack_log2, blocks) : tile_info<false>(e, pair, t, kv_head, by, pack_log2, blocks);
    out[0] = ti.valid;
    out[1] = ti.head;
    out[2] = ti.row0;
    out[3] = ti.n_kv;
}
// {some, shared, first key, tiles of tile 0 and 1, kv_len, pos_off, kv_crow} of the CTA's share
void pair_share(int n0, int n1, int kv_len, int pos_off, int parts, int rank, int* out) {
    Item w{};
    w.some = 1;
    w.sq = extent(0, kv_len, pos_off);
    w.sq.kv_crow = 1000;
    w.t[0].n_kv = n0;
    w.t[1].n_kv = n1;
    const Share share = take_share(w, parts, rank);
    const int all[8] = {w.some, share.some, share.first_key, w.t[0].n_kv, w.t[1].n_kv, w.sq.kv_len, w.sq.pos_off, w.sq.kv_crow};
    for (int i = 0; i < 8; ++i) out[i] = all[i];
}
int pair_parts(long long pairs, long long tiles, int exact, long long rows, int sms) { return prefill_parts(pairs, tiles, exact != 0, rows, sms); }
int f32_pair_parts(long long blocks, long long tiles, int sms) { return f32_parts(blocks, tiles, sms); }
int pair_band(int pairs, long long tiles, int group, int parts) { return prefill_band(pairs, tiles, group, parts); }
}
