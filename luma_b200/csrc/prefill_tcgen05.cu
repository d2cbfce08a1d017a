// Causal, GQA-capable flash-attention prefill forward for sm_100a: TMA-fed Q/K/V tiles,
// tcgen05.mma with the S and O accumulators in tensor memory, online softmax in registers,
// warp-specialised roles. Handles f16/bf16 storage with head_size 128, 64, or 32 on zero-padded 64-column tiles (template parameter D;
// the layout comments below give the D = 128 figures) for the batched entry point (optional
// key-padding mask: template parameter kMask), chunked prefill over a paged cache, and the packed varlen entry point (with
// or without the packed buffers' row counts). Replaces flash_attn_kernel
// (luma-flash-attn/kernels/flash_attn_func.cu:29-226), flash_attn_prefill_kernel
// (kernels/flash_attn_with_kvcache.cu:157-277) and flash_attn_varlen_kernel
// (kernels/flash_attn_varlen_func.cu:35-199), one-thread-per-query-row scalar kernels.
//
// One CTA (384 threads, 1 per SM) works on a pair of query tiles of 128 rows that share a batch
// element and a KV head — two consecutive row blocks of the heads that share a tile (tile 0 the later one) — and streams that KV head's K/V tiles
// (128 keys) past both. The rows of a tile are query token x head of the GQA group (as many heads as a power of two divides the group by, see pack_of): a tile
// of 128 rows is 32 tokens of four heads, so that a sequence's last tile is partly empty once and not once for every head, and a few tokens fill one
// tile together. A tile of 128 tokens for each head, and so (us): 1 x 658, 32/8 heads 15.0 and 13.7; 6 x 450-900 padded prompts at head size 64 76.2 and 68.5; 64 x 16
// tokens over 4096 keys, 32/8 heads 400 and 189; 24 packed prompts of 17-2000, head size 64 250 and 243; row counts that fill the tiles either way, the same within 1 %. Then
// it takes over the pair of a CTA of the grid that has not started (clusterlaunchcontrol), until none is left
// (an instantiation of one pair for grids where that wins nothing, see launch_variant):
//   warps 0-3 / 4-7 : softmax warpgroup of query tile 0 / 1 — one thread per query row: read S
//                     from tensor memory (tcgen05.ld), running max / sum in registers (exp2 with
//                     the scale folded in), write P as packed 16-bit back over S (tcgen05.st),
//                     rescale O in tensor memory only when the row max moved by more than 2^8,
//                     final normalisation of O, staged in shared memory and written with bulk
//                     tensor stores (and LSE); setmaxnreg gives these warps 208 registers
//   warp 8 / 10     : TMA producers — warp 8 finds the tile pairs, loads Q and the K tiles; warp 10 the V tiles; two 2-stage rings
//                     that run on across the pairs
//   warp 9          : MMA issuer — S_t = Q_t K^T (SS form), O_t += P_t V (P from tensor memory),
//                     completion signalled with tcgen05.commit on mbarriers; the warp runs converged
//                     and one elected lane issues
//   warp 11         : sets the barriers up
// While one warpgroup runs its softmax the tensor core works on the other tile; while the warpgroups normalise and write O, the next
// pair's Q and first K and V tiles arrive and its first S is computed. With a CTA for every pair, 4 to 5 us of each were set-up, first copies and
// last stores with nothing beside them: 24 packed prompts of 17-2000 tokens at head size 64 332 us, 267 so; 8 x 1000 at head size 64, 32/8 heads 77 and 64; 4 x 2048
// MHA 160 and 155; 2 x 8192 GQA, 64 steps to a pair, 937-948 and 945-952.
// Tensor memory (512 columns): S0 | S1 | O0 | O1, 128 fp32 columns each; P_t aliases S_t.
// Shared memory: Q 2 x 32 KiB, K ring 2 x 32 KiB, V ring 2 x 32 KiB, all 128-byte swizzled
// exactly as TMA writes them, so the MMA descriptors address them in place; 32 KiB for the softmax warps' rows on their way out.
//
// Every wait on an mbarrier is bounded (about 2 s of wall clock); on expiry the CTA records a
// status word in global memory, stops waiting everywhere, drains its own TMA copies, frees its
// tensor memory and returns.
#include <cuda.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "tcgen05.cuh"

namespace fa {

namespace {

// head size D (64 or 128) is a template parameter of the kernel
constexpr int kStages = 2;     // depth of the K and V rings
static_assert(kStages == 2, "step_full and step_done have an entry per stage, found by the parity of the step (j & 1, phase j >> 1) throughout the kernel");
// A third V stage measured 5 % slower on every prefill workload when there was room for one, without the softmax warps' output rows (1165
// against 1228 TFLOP/s at S = 8192); the issuer does not wait for the copies.
constexpr int kThreads = 384;   // three warpgroups: softmax 0, softmax 1, and producers + issuer (+ an idle warp)
constexpr int kLoadWarp = 8;
constexpr int kMmaWarp = 9;
constexpr int kLoadWarpV = 10;   // V-ring producer (K ring and Q: kLoadWarp)
constexpr int kHalfBytes = kBlockN * 64 * 2;   // 16 KiB: one 64-column half, 128 rows x 128 B
template <int D> struct TileBytes { static constexpr int value = kBlockN * D * 2; };   // one half at D = 64, two at D = 128
constexpr float kRescaleThreshold = 8.0f;            // log2 units

// Which element pairs take their exponential on the FMA pipe (a quintic) instead of the special-function unit: one in six at head size 128, one in eight at 64. It costs issue slots
// and registers that the special-function unit's time does not buy back at a larger share, at head size 64 at that already. us from a graph for a share of 1/8, 1/7, 1/6, 1/5: 2 x 8192 GQA 807.6, 802.7, 797.7,
// 807.8; 4 x 2048 MHA 129.4, 128.7, 128.1, 129.3; 4 chunks of 512 137.8, 136.2, 136.5, 135.8, with 32 decoding sequences 219.1, 218.4, 215.6, 216.2; 24 packed prompts of 1000 225.8, 227.8,
// 227.9, 230.1. At head size 64, 1/8, 1/6, 1/5, 1/4: 2 x 4096 189.7, 195.6, 191.8, 197.7; 8 x 1000 65.3, 67.0, 66.4, 70.6; 24 packed prompts of 17-2000 250.8, 256.8, 256.7, 261.6. The error of the
// log-sum-exp against 64 bits is the same for 1/8 and 1/6 (rms 2.1-3.9e-7 over 100-4096 tokens).
template <int D> __device__ __forceinline__ constexpr bool fma_pipe_exp(int i) { return D == 128 ? i % 6 == 5 : (i & 7) == 7; }

constexpr int kOutBytes = 4096;     // a softmax warp's rows on their way out: 32 of 128 bytes
constexpr int kDone = 4;            // entries of step_done, see there

template <int D>
struct SharedStorage {
    alignas(1024) unsigned char q[2][TileBytes<D>::value];
    alignas(1024) unsigned char k[kStages][TileBytes<D>::value];
    alignas(1024) unsigned char v[kStages][TileBytes<D>::value];
    alignas(1024) unsigned char out[8][kOutBytes];
    alignas(16) unsigned char answer[16];   // what the request for another tile pair brought (written by the hardware)
    Item item[2];                   // tile pair i of the CTA in entry i & 1
    Share share;                    // of item[0]
    alignas(8) unsigned long long item_full[2];   // K producer -> all roles: the entry holds the next tile pair
    unsigned long long item_empty[2];   // V producer, issuer, softmax warps -> K producer: it has been read
    unsigned long long answered;    // hardware -> K producer: `answer` is there
    unsigned long long q_full[2];
    unsigned long long k_first;     // copy engine -> MMA: K tile 0 of a tile pair
    unsigned long long step_full[2];    // copy engine -> MMA: what a step reads, its V tile and the tile pair's next K tile; step g of the CTA in entry g & 1
    // MMA -> producers: what was issued before this has finished. The issuer commits once per tile pair for the first S and once for every step; commit c is in
    // entry c & 3. A producer that waits for commit c can fall behind by up to three (tile pairs of one step: a step, the next pair's first S, its step), with two
    // entries it would find the phase it waits for gone, and wait for good.
    unsigned long long step_done[kDone];
    unsigned long long s_full[2];   // MMA -> softmax: S_t ready
    unsigned long long o_full[2];   // MMA -> softmax: O_t final (a barrier of its own: the next pair's first S_t may be ready before anybody has looked at this)
    unsigned long long p_ready[2][2];   // softmax -> MMA: keys 0-63 of P_t written and O_t rescaled ([0][t]), keys 64-127 written ([1][t])
    unsigned long long v_tail;      // copy engine -> V producer: the sequence's last, partly filled V tile has landed
    unsigned long long drain;       // MMA issuer, at its end: every product issued has finished
    unsigned int tmem_base;
    volatile int abort_flag;
    int left_out;                   // test hook: 1 + the step whose K tile was never requested, 0: none
};
static_assert(sizeof(SharedStorage<128>) + 1024 <= 232448, "fits the shared memory of an SM");

constexpr int kMaxPeers = 8;
#ifdef FA_TRACE
constexpr int kCtaLogEntries = 2048;
#endif
constexpr unsigned long long kWaitLimitNs = 2000000000ULL;   // default bound of every mbarrier wait

struct PrefillArgs {
    // Output: n_out buffers of (batch, q_seq_len, o_heads, 128), each receiving this launch's heads
    // at head offset o_head0. n_out == 1 with o_heads == q_heads is the ordinary call; with n_out > 1
    // the buffers are the same tensor on every GPU of a head-sharded group (peer memory over
    // NVLink), which makes the output all-gather part of the epilogue.
    void* o[kMaxPeers];
    int n_out, o_heads, o_head0;
    int o_by_32;        // o[0] is 32-byte aligned (and so is every row of every head)
    int peer0;          // n_out > 1: the buffer this CTA's rows go to first; each CTA walks the buffers from there
    int multicast;      // o[0] is an NVSwitch multicast address of the group's output tensors: one multimem.st reaches all of them
    float* lse;         // (batch, q_heads, q_seq_len) of this call, or null
    float* lse_peers[kMaxPeers];   // n_lse > 0: (batch, o_heads, q_seq_len) on every GPU of the group, written at head o_head0
    int n_lse;
    int* status;        // word in mapped host memory, set to non-zero when a bounded wait expired
    unsigned long long wait_ns;    // bound of every mbarrier wait
    int test_skip_k;    // test hook: the K producer leaves out tile (test_skip_k - 1), so that a wait runs out; 0 = off
#ifdef FA_TRACE
    int staged_store;   // 1 = stage O rows in shared memory and store whole rows even for a single output
    long long* trace;  // optional timeline of one CTA (clock64 stamps), null unless the "prefill_trace" option is set
    int trace_y;       // blockIdx.y of the traced CTA (option "prefill_trace_y", default 0 = the heaviest)
    long long* cta_log;  // optional per-CTA {start ns, end ns, SM id} records ("prefill_trace" = 3), up to kCtaLogEntries
#endif
    int batch, q_seq_len, kv_seq_len, q_heads, kv_heads, start_pos;
    int d_real;     // head size of the tensors: D, or 32 when the D = 64 kernel runs a head size of 32 on zero-padded tiles
    int pack_log2;          // of the query heads that share a tile (pack_of): row r is query token r >> pack_log2, head r % pack of them
    FastDiv by_packs, by_kv_heads, by_band;   // groups of `pack` query heads per KV head; KV heads; band
    int parts;      // CTAs (of a cluster) that share the keys of a tile pair; 1: the pair has a CTA of its own
    int streams_z;  // (batch, KV head) streams per blockIdx.z
    int band;       // tile pairs of one (batch, KV head) that sit next to each other in blockIdx.x
    // Launch order of the bands (blockIdx.y), heaviest = 0. spread_w == 0: heaviest first. Otherwise the
    // first spread_w rows of the grid are every spread_m-th band (a first wave that mixes all weights,
    // so that CTAs end at spread-out times from the start), the other bands follow heaviest first.
    int spread_w, spread_m;
    // Paged calls: ordered != 0: the CTA finds its tile pair on the device (find_item); pairs: tile pairs per (sequence, KV head) at most.
    int ordered, pairs;
    // which entry point the problem came from (fa::Mode) and its per-sequence descriptors
    int mode;                   // MODE_BATCH: uniform q_seq_len / kv_seq_len / start_pos
    const void* q;              // MODE_VARLEN: the packed q / k / v buffers themselves, for the tiles at their very end
    const void* k;
    const void* v;
    const unsigned char* mask;  // MODE_BATCH: optional (batch, kv_seq_len) key-padding mask, 1 = valid key
    const int* cu_q;            // MODE_VARLEN: packed row offsets of q / o
    const int* cu_k;            // MODE_VARLEN: packed row offsets (or, paged, lengths by difference) of k / v
    const int* context_lens;    // MODE_KVCACHE: cached length per sequence, query tokens included
    const int* block_tables;    // paged K/V: (batch, max_blocks) logical -> physical block
    int paged, block_size, max_blocks;
    int q_bounded, kv_bounded;  // MODE_VARLEN: the caller gave the packed buffers' rows, their tensor maps end there
    int behind_few;             // the few-row kernel was launched ahead: this one does not wait for it, but ends behind it
    int skip_rows;              // MODE_VARLEN: sequences of at most this many (query token, group head) rows are not this launch's; 0: none
    float scale_log2;
};

// ---- PTX wrappers -------------------------------------------------------------------------
// Bounded wait. Returns false when the wait was abandoned (time limit, or another thread of the
// CTA already gave up); the caller then falls through to the end of the kernel.
// The bound is counted in SM clocks (cheap to read, unlike the global nanosecond timer): wait_ns x 2 clocks, i.e. at least
// wait_ns of wall time at any SM clock up to 2 GHz.
// The status word lives in mapped host memory (the host reads it without touching the device), so it
// is written with a plain store: the code of one of the waits that expired.
template <typename Storage>
__device__ __forceinline__ bool mbar_wait(Storage& sm, unsigned long long* bar, unsigned parity, const PrefillArgs& a,
                                          int where) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    const long long limit = (long long)(a.wait_ns * 2ULL);
#pragma unroll 1
    for (unsigned spin = 1;; ++spin) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((spin & 63u) == 0u) {
            if (sm.abort_flag) return false;
            if (clock64() - t0 > limit) {
                sm.abort_flag = 1;
                *reinterpret_cast<volatile int*>(a.status) = where;
                __threadfence_system();
                return false;
            }
        }
    }
}

// The same for the producers. A look suspends until the phase is complete, or some 8000 clocks, so what follows the first one is seldom reached: it is a function of its own, out of the
// producers' loops, whose instructions share the SM's instruction cache with the softmax steps. 24 packed prompts of 17-2000 tokens, head size 64 267 us with it in each of the loops'
// waits, 254 so; 4 chunks of 512 143.3 and 142.5; 4 x 2048 MHA 129.8 and 129.2.
__device__ __noinline__ bool mbar_wait_on(unsigned bar, unsigned parity, unsigned abort_flag, long long limit, int* status, int where) {
    const long long t0 = clock64();
#pragma unroll 1
    for (unsigned spin = 1;; ++spin) {
        if (mbar_try_wait_at(bar, parity)) return true;
        if ((spin & 63u) == 0u) {
            if (shared_flag(abort_flag)) return false;
            if (clock64() - t0 > limit) {
                set_shared_flag(abort_flag);
                *reinterpret_cast<volatile int*>(status) = where;
                __threadfence_system();
                return false;
            }
        }
    }
}
template <typename Storage>
__device__ __forceinline__ bool producer_wait(Storage& sm, unsigned long long* bar, unsigned parity, const PrefillArgs& a, int where) {
    if (mbar_try_wait(bar, parity)) return true;
    return mbar_wait_on(smem_u32(bar), parity, smem_u32((const void*)&sm.abort_flag), (long long)(a.wait_ns * 2ULL), a.status, where);
}

// The end of a producer after an abort: none of its copies may be in flight when the CTA ends. These waits ignore the abort flag and depend on the copy engine
// alone (bounded all the same). A step's barrier also wants the arrival of the other ring's producer, which may have given up before that step, so each of them
// makes its arrivals for the two steps after its last one here. Two are enough: a stage is filled for step x once step x - 2 has finished, so neither ring is more
// than two steps ahead. And no phase gets a third arrival, which the hardware would take for an error while bytes are missing: one per ring and step,
// the one for step x when the phase of step x - 2 has been seen complete.
//   given    : steps that have this ring's arrival, or a copy that brings it
//   left_out : 1 + a step before them that the test hook left without, or 0
//   single   : what else is on its way, two bits each from bit 0: whether, and the parity of its phase (answer, Q of tile 0 and 1, K tile 0, V tail)
template <typename Storage>
__device__ __noinline__ void settle_copies(Storage& sm, int given, int left_out, unsigned single) {
    const unsigned long long begin = global_timer_ns();
    auto landed = [&](unsigned long long* bar, unsigned parity) {
#pragma unroll 1
        while (!mbar_try_wait(bar, parity & 1u))
            if (global_timer_ns() - begin >= 100000000ULL) return false;
        return true;
    };
#pragma unroll 1
    for (int i = 0; i < 5; ++i) {
        unsigned long long* const bar = i == 0 ? &sm.answered : i < 3 ? &sm.q_full[i - 1] : i == 3 ? &sm.k_first : &sm.v_tail;
        if ((single >> (2 * i)) & 1u) landed(bar, single >> (2 * i + 1));
    }
#pragma unroll 1
    for (int i = left_out > 0 ? -1 : 0; i < 2; ++i) {
        const int x = i < 0 ? left_out - 1 : given + i;
        if (x < 2 || landed(&sm.step_full[x & 1], (unsigned)((x - 2) >> 1))) mbar_arrive(&sm.step_full[x & 1]);
    }
}

// The end of a producer: false where its copies have to be looked after (above). As long as nobody gives up, every copy has landed when the issuer has come to its end.
template <typename Storage>
__device__ __forceinline__ bool all_read(Storage& sm, bool alive, const PrefillArgs& a, int where) {
    return alive && producer_wait(sm, &sm.drain, 0u, a, where) && !sm.abort_flag;   // (an issuer that gives up says so before it ends)
}

__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, unsigned long long* bar, int c0, int c1,
                                            int c2, int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];\n" ::"r"(
            smem_u32(dst)),
        "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
        : "memory");
}

// The same box as far as L2.
__device__ __forceinline__ void tma_prefetch_4d(const CUtensorMap* map, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global.tile [%0, {%1, %2, %3, %4}];\n" ::"l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}

// Bulk tensor store shared -> global of one box, tracked by the issuing thread's bulk group.
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, const void* src, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];\n" ::"l"(map),
                 "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
                 : "memory");
}

// 16 bytes to an NVSwitch multicast address: the switch replicates the store into the same offset of
// every GPU's memory bound to the multicast object (the bits are stored as they are).
__device__ __forceinline__ void multimem_st16(void* mc_addr, const uint4& w) {
    asm volatile("multimem.st.global.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(mc_addr), "r"(w.x), "r"(w.y), "r"(w.z), "r"(w.w)
                 : "memory");
}

// Asks for a tile pair of a CTA that has not started (which then never does); the answer arrives as 16 bytes on the barrier.
__device__ __forceinline__ void request_pair(void* answer, unsigned long long* bar) {
    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];\n" ::"r"(smem_u32(answer)), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ bool read_answer(const void* answer, int& x, int& y, int& z) {
    unsigned got;
    asm volatile(
        "{\n.reg .pred p;\n.reg .b128 h;\nld.shared.b128 h, [%4];\n"
        "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\nselp.u32 %0, 1, 0, p;\n"
        "mov.b32 %1, 0;\nmov.b32 %2, 0;\nmov.b32 %3, 0;\n"
        "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%1, %2, %3, _}, h;\n}\n"
        : "=r"(got), "=r"(x), "=r"(y), "=r"(z)
        : "r"(smem_u32(answer))
        : "memory");
    return got != 0;
}

// 32 bytes from registers, in one store where the buffer is aligned to them, else in two of 16.
__device__ __forceinline__ void store_32(void* to, const unsigned (&w)[8], bool whole) {
    if (whole) {
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"l"(to), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]),
                     "r"(w[7])
                     : "memory");
    } else {
        *static_cast<uint4*>(to) = make_uint4(w[0], w[1], w[2], w[3]);
        *(static_cast<uint4*>(to) + 1) = make_uint4(w[4], w[5], w[6], w[7]);
    }
}

// Maxima that are NaN where an operand is.
__device__ __forceinline__ float max_nan(float a, float b) {
    float d;
    asm("max.NaN.f32 %0, %1, %2;\n" : "=f"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ float max3_nan(float a, float b, float c) {
    float d;
    asm("max.NaN.f32 %0, %1, %2, %3;\n" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// Two f32 lanes in one 64-bit register for the packed FMA-pipe instructions of sm_100.
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(unsigned long long r, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;\n" : "=f"(a), "=f"(b) : "l"(r));
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// 2^x for two x on the FMA pipe instead of the special-function unit: x = n + f with n the
// nearest integer (magic-number rounding), a quintic for 2^f on [-0.5, 0.5] and n added to the exponent field. The quintic: constant term 1, so that
// a row's largest score weighs exactly 1; the others the minimax fit of relative error, moved by single bits to the smallest error of the
// f32 evaluation. 1.9e-7 at most, 2.2e-8 low on average, against ex2.approx's measured 1.4e-7 and 4.6e-8. A quartic (2.7e-6) showed in the f32 sums of the
// rows' first tile: error of LSE over 128 tokens with scores N(0,1) at most 9.9e-7, rms 2.4e-7, instead of 7.9e-7 and 2.2e-7 (8 x 128 x 8 rows,
// bf16, against 64 bits), and 7e-7 where one key takes all of a row's weight. x is clamped at -200, where that addition gives a negative integer, and those become zeros: 2^x for x
// below -126.5, -inf (a masked score) among them, is an exact zero or below 2^-126. A NaN becomes the largest finite number (the addition takes one from
// its exponent): infinite in 16 bits, but not in the row's sum, so the caller looks for NaN and +inf among the scores itself (see the row maximum).
__device__ __forceinline__ void ex2_fma2(float x0, float x1, float& p0, float& p1) {
    const unsigned long long x2 = pack2(max_nan(x0, -200.0f), max_nan(x1, -200.0f));
    const unsigned long long t2 = add2(x2, pack2(12582912.0f, 12582912.0f));   // 1.5 * 2^23
    const unsigned long long n2 = add2(t2, pack2(-12582912.0f, -12582912.0f));
    const unsigned long long f2 = fma2(n2, pack2(-1.0f, -1.0f), x2);
    unsigned long long p2 = fma2(pack2(0.0013202913105f, 0.0013202913105f), f2, pack2(0.0096749374643f, 0.0096749374643f));
    p2 = fma2(p2, f2, pack2(0.0555104725063f, 0.0555104725063f));
    p2 = fma2(p2, f2, pack2(0.2402218878270f, 0.2402218878270f));
    p2 = fma2(p2, f2, pack2(0.6931467056274f, 0.6931467056274f));
    p2 = fma2(p2, f2, pack2(1.0f, 1.0f));
    float t0, t1, q0, q1;
    unpack2(t2, t0, t1);
    unpack2(p2, q0, q1);
    p0 = __int_as_float(max(__float_as_int(q0) + (__float_as_int(t0) << 23), 0));
    p1 = __int_as_float(max(__float_as_int(q1) + (__float_as_int(t1) << 23), 0));
}

// Timeline slots: role (0/1 = softmax warpgroup, 2 = MMA issuer, 3 = K producer, by tile pair) x step of the CTA, over its tile pairs (< 60) x event (< 8).
// Compiled in with -DFA_TRACE only; the default build carries none of it.
[[maybe_unused]] constexpr int kTraceSteps = 60;
#ifdef FA_TRACE
__device__ __forceinline__ void trace_event(long long* trace, int role, int j, int ev) {
    if (trace != nullptr && j < kTraceSteps) trace[(role * kTraceSteps + j) * 8 + ev] = clock64();
}
#define FA_TRACE_EVENT(role, j, ev) trace_event(trace, role, j, ev)
#define FA_TRACE_PARAM(x) , long long* x
#define FA_TRACE_ARG(x) , x
#else
#define FA_TRACE_EVENT(role, j, ev) ((void)0)
#define FA_TRACE_PARAM(x)
#define FA_TRACE_ARG(x)
#endif

__device__ __forceinline__ SeqExtent seq_extent(const PrefillArgs& a, int s) {
    SeqExtent e;
    if (a.mode == MODE_BATCH) {
        e.q_len = a.q_seq_len; e.kv_len = a.kv_seq_len; e.pos_off = a.start_pos;
        e.o_row0 = (long long)s * a.q_seq_len;
        e.q_crow = 0; e.q_cb = s; e.kv_crow = 0; e.kv_cb = s;
    } else if (a.mode == MODE_VARLEN) {
        const int q0 = a.cu_q[s], k0 = a.cu_k[s];
        e.q_len = a.cu_q[s + 1] - q0; e.kv_len = a.cu_k[s + 1] - k0; e.pos_off = e.kv_len - e.q_len;
        e.o_row0 = q0;
        e.q_crow = q0; e.q_cb = 0; e.kv_crow = k0; e.kv_cb = 0;
    } else {
        e.q_len = a.q_seq_len; e.kv_len = a.context_lens[s]; e.pos_off = e.kv_len - e.q_len;
        e.o_row0 = (long long)s * a.q_seq_len;
        e.q_crow = 0; e.q_cb = s; e.kv_crow = 0; e.kv_cb = 0;
    }
    return e;
}

// The launch order of chunks of prompts over long contexts, whose lengths the host does not know: CTA `index`
// of the grid takes the index-th tile pair of the call, heaviest first (K/V tiles, in classes of an eighth of the longest
// range, so that the pairs of one K/V stream stay neighbours and meet in L2). In grid order (sequences as they
// come) a long context that comes late ends alone (times beside the rule that asks for it, in launch_variant).
// Run by one whole warp; a lane holds 8 neighbouring sequences at most.
constexpr int kOrderPerLane = 8;
constexpr int kOrderMax = 32 * kOrderPerLane;
constexpr int kOrderClasses = 8;

// Returns {sequence or -1, KV head, pair}.
__device__ __forceinline__ int3 find_item(const PrefillArgs& a, int index, int lane) {
    const int packs = a.by_packs.d, pl = a.pack_log2, group = packs << pl;
    int ql[kOrderPerLane], kl[kOrderPerLane];
    const int per = (a.batch + 31) / 32;
    int most = 0;
#pragma unroll
    for (int i = 0; i < kOrderPerLane; ++i) {
        ql[i] = kl[i] = 0;
        if (i >= per) break;
        const int k = lane * per + i;
        if (k >= a.batch) continue;
        const SeqExtent e = seq_extent(a, k);
        if (e.q_len <= 0 || e.q_len * group <= a.skip_rows) continue;
        // (a sequence longer than the call's max_seqlen_q has the grid's pairs and no more)
        const int cut = max(0, e.q_len - ((a.pairs * 2 + packs - 1) / packs * kBlockM >> pl));
        ql[i] = e.q_len - cut;
        kl[i] = e.kv_len - cut;
        most = max(most, kl[i] > 0 ? (kl[i] - 1) / kBlockN + 1 : 0);
    }
    most = __reduce_max_sync(0xffffffffu, most);
    const int width = max(1, (most + kOrderClasses - 1) / kOrderClasses);
    auto count = [&](int c, int (&x)[kOrderPerLane]) -> int {   // pairs in classes 0 .. c, per sequence and in all
        int sum = 0;
#pragma unroll
        for (int i = 0; i < kOrderPerLane; ++i) {
            x[i] = 0;
            if (i >= per) break;
            x[i] = c < 0 ? 0 : min(a.pairs, pairs_from(ql[i], kl[i], packs, pl, c >= kOrderClasses ? 0 : most - (c + 1) * width + 1));
            sum += x[i];
        }
        return __reduce_add_sync(0xffffffffu, sum) * a.kv_heads;
    };
    int upto[kOrderPerLane], before[kOrderPerLane];
    if (index >= count(kOrderClasses, upto)) return make_int3(-1, 0, 0);
    int lo = 0, hi = kOrderClasses;   // the first class whose running count passes the index
    while (lo < hi) {
        const int mid = (lo + hi) / 2;
        if (count(mid, upto) > index) hi = mid; else lo = mid + 1;
    }
    int rest = index - count(lo - 1, before);
    count(lo, upto);
    int mine = 0;
#pragma unroll
    for (int i = 0; i < kOrderPerLane; ++i) {
        if (i >= per) break;
        mine += (upto[i] - before[i]) * a.kv_heads;
    }
    int incl = mine;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += o;
    }
    const int owner = __ffs(__ballot_sync(0xffffffffu, incl > rest)) - 1;
    rest -= incl - mine;   // meaningful on the owner
    int s = 0, kvh = 0, pair = 0;
    bool found = false;
#pragma unroll
    for (int i = 0; i < kOrderPerLane; ++i) {
        if (i >= per) break;
        const int here = upto[i] - before[i];
        if (found) continue;
        if (rest < here * a.kv_heads) {
            found = true;
            s = lane * per + i;
            kvh = rest / here;
            const int pairs = min(a.pairs, pairs_from(ql[i], kl[i], packs, pl, 0));
            pair = pairs - 1 - before[i] - (rest - kvh * here);
        } else {
            rest -= here * a.kv_heads;
        }
    }
    return make_int3(__shfl_sync(0xffffffffu, s, owner), __shfl_sync(0xffffffffu, kvh, owner), __shfl_sync(0xffffffffu, pair, owner));
}

// One K or V tile (128 keys x D dims, D / 64 halves of 64 columns), tile index j.
//   contiguous: boxes of 128 rows starting at the sequence's row kv_crow + 128 j;
//   paged     : one box per page and half (block_size rows), requested by one whole warp; lane i holds the tile's page i
//               (page_of_lane) and requests it. Pages past the sequence's last one are requested at block -1, which is out of range for the
//               tensor map and therefore arrives as zeros.
// A paged tile is 16 copies at a page of 16 tokens: the lanes look their pages up before the ring stage is free, so
// that the request follows the release at once. Looked up and requested page by page by one thread after the release,
// a tile came about a thousand clocks later, which the two-stage rings do not hide: 3.6 % of a step of 4 chunks of 512 over
// 1024-8192 tokens (page 16).
__device__ __forceinline__ int page_of_lane(const PrefillArgs& a, int kv_len, int s, int j, int lane, int first_key) {
    const int per_tile = kBlockN / a.block_size;
    const int pg = j * per_tile + lane;
    return lane < per_tile && pg < (kv_len + a.block_size - 1) / a.block_size ? a.block_tables[(long long)s * a.max_blocks + first_key / a.block_size + pg] : -1;
}

// Contiguous K/V: called by one lane.
template <int D, bool kPaged>
__device__ __forceinline__ void load_kv_tile(const PrefillArgs& a, int kv_crow, int kv_cb, int kvh, unsigned char* dst,
                                             const CUtensorMap* map, unsigned long long* bar, int j, int page, int lane) {
    if (!kPaged) {
        mbar_expect_tx(bar, TileBytes<D>::value);
        tma_load_4d(dst, map, bar, 0, kvh, kv_crow + j * kBlockN, kv_cb);
        if (D == 128) tma_load_4d(dst + kHalfBytes, map, bar, 64, kvh, kv_crow + j * kBlockN, kv_cb);
        return;
    }
    if (lane == 0) mbar_expect_tx(bar, TileBytes<D>::value);
    __syncwarp();
    if (lane < kBlockN / a.block_size) {
        tma_load_4d(dst + lane * a.block_size * 128, map, bar, 0, kvh, 0, page);
        if (D == 128) tma_load_4d(dst + kHalfBytes + lane * a.block_size * 128, map, bar, 64, kvh, 0, page);
    }
    __syncwarp();
}

// A 128-row tile of a packed (varlen) buffer that would reach past the buffer's last row, fetched by
// one warp with plain loads: the reference's varlen signature does not say how many rows the packed
// buffers hold, so their tensor maps carry no row bound, and a bulk copy must never be asked for
// rows that may not exist. Rows past the end are written as zeros (what an out-of-range bulk copy
// delivers). Same shared-memory image as the bulk copies: 64-column halves, 128 B per row, 16-byte
// chunks XOR-swizzled by the row. The barrier's phase is completed by one plain arrival.
// All of a lane's copies are in flight together (cp.async): one trip to memory for a tile. As loads into registers, four at a time, a
// tile was 16 trips one after the other, and a CTA at the end of the buffers waited for two Q tiles, K and V so: 4 prompts of 38-155 tokens, 32/8 heads, through the
// plain entry point 27 us, 23 so; 4 of 235-941, 8/2 heads, 39 and 31. (With the row counts given nothing comes this way, see q_open: 36 and 12 us, 38 and 22.)
template <int D>
__device__ __forceinline__ void edge_tile_copy(unsigned char* dst, const void* base, int heads, int head, long long row_start,
                                               long long total_rows, unsigned long long* bar, int lane, int d_real, int pack_log2 = 0) {
    constexpr int kChunksPerRow = D / 8;   // 16-byte chunks per row of the tile (columns past d_real are zeros)
    const long long left = (total_rows - row_start) << pack_log2;   // rows of the tile: those of 1 << pack_log2 heads for each row of the buffer
    const int nrows = left < 0 ? 0 : (left > kBlockN ? kBlockN : (int)left);
    const unsigned char* src = static_cast<const unsigned char*>(base);
    const unsigned to = smem_u32(dst);
#pragma unroll 4
    for (int idx = lane; idx < kBlockN * kChunksPerRow; idx += 32) {
        const int r = idx / kChunksPerRow, cc = idx % kChunksPerRow;
        const bool real = r < nrows && cc * 8 < d_real;
        const unsigned char* from = real ? src + ((row_start + (r >> pack_log2)) * heads + head + (r & ((1 << pack_log2) - 1))) * (long long)(d_real * 2) + cc * 16 : src;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(to + (cc >> 3) * kHalfBytes + r * 128 + (((cc & 7) ^ (r & 7)) << 4)), "l"(from),
                     "r"(real ? 16 : 0)   // 0: nothing is read, zeros are written
                     : "memory");
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");   // generic-proxy writes -> tensor-core reads
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}

// The SM clock in units of 1024: 32 bits hold 36 minutes at 2 GHz, more than the longest bound of a wait.
__device__ __forceinline__ unsigned clock_1024() { return (unsigned)(clock64() >> 10); }

constexpr unsigned kApart = 950;   // clocks between the two tiles' first S at head size 64

// The MMA issuer, run by one whole warp (converged). Its loop is written for few instructions. What a scheduler executes in a loop comes at full rate
// up to 512 instructions (8 KiB), beyond that at one in 3 clocks, beyond 2048 in 6 (`clock64` around loops of that many independent multiply-adds); the
// softmax warps' unrolled steps pass between two steps of the issuer, which finds its own anew every time. The tensor pipe stood still meanwhile: 300 clocks from the issuer's last commit of a step to its first look at the next barrier, 150 for
// a look at one that had long completed (45 alone), with or without the copies. Step of 128 keys at S = 8192 GQA 3100 -> 2840 clocks,
// 884 -> 833 us; 4 x 2048 MHA 157.5 -> 147.8 us; head size 64, 2 x 8192 GQA 755 -> 699 us.
//   * a function of its own, so that the compiler sees what is the same for the whole warp (everything is, or is broadcast here): inside
//     the kernel it takes them for divergent, for the early returns and per-sequence loads before them;
//   * nothing is in the loop for the sake of the next tile pair: with a look for it behind a tile's last step (so that its first S would be issued beside the other
//     tile's last products) 24 packed prompts took 299 us instead of 275, 4 x 2048 MHA 159 instead of 154.5, 2 x 8192 GQA 965 instead of 947;
//   * a wait that runs out is looked after at the end of its step, which goes on without waiting on what happens to be in shared memory and
//     reports nothing as done. Leaving at each wait doubled the code after it.
template <typename T, int D, bool kOnePair>
__device__ __noinline__ void issue_products(unsigned sm_addr, unsigned tmem, int* status, unsigned long long wait_ns FA_TRACE_PARAM(trace)) {
    using Storage = SharedStorage<D>;
    sm_addr = __shfl_sync(0xffffffffu, sm_addr, 0);
    tmem = __shfl_sync(0xffffffffu, tmem, 0);
    const unsigned idesc_qk = make_idesc<T>(false, kBlockN);
    const unsigned idesc_pv = make_idesc<T>(true, D);   // N = head size
    const unsigned long long dq = make_desc(sm_addr + (unsigned)offsetof(Storage, q), 16, 1024);
    const unsigned long long dk = make_desc(sm_addr + (unsigned)offsetof(Storage, k), 16, 1024);
    const unsigned long long dv = make_desc(sm_addr + (unsigned)offsetof(Storage, v), kHalfBytes, 1024);
    constexpr unsigned kTileStep = TileBytes<D>::value >> 4;   // from one tile's descriptor to the next one's
    unsigned patience = (unsigned)(wait_ns >> 9) + 1u;   // the bound as in mbar_wait, in units of 1024 SM clocks
    int expired = 0;   // code of the wait that was the first to be given up; none has any patience from then on
    auto wait = [&](size_t bar, unsigned parity, int where) {
        const unsigned t0 = clock_1024();
#pragma unroll 1
        while (!__any_sync(0xffffffffu, mbar_try_wait_at(sm_addr + (unsigned)bar, parity))) {
            if (__any_sync(0xffffffffu, clock_1024() - t0 >= patience || shared_flag(sm_addr + (unsigned)offsetof(Storage, abort_flag)))) {
                if (expired == 0) expired = where;
                patience = 0;
                break;
            }
        }
    };
    // S_t = Q_t K^T : D / 16 K-steps over d; both operands K-major, 128 B swizzle
    auto issue_s = [&](int t, unsigned long long kd) {
        const unsigned long long qd = dq + t * kTileStep;
        if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk) {
                const unsigned inc = ((kk >> 2) * kHalfBytes + (kk & 3) * 32) >> 4;
                tc_mma_ss(tmem + t * 128, qd + inc, kd + inc, idesc_qk, kk > 0);
            }
        }
    };
    // O_t += P_t V : 4 K-steps of 16 keys; A = P from tensor memory (packed 16-bit, 8 columns
    // per step), B = V MN-major: 64-column halves 16 KiB apart, 8-key groups 1 KiB apart
    auto issue_pv = [&](int t, int half, unsigned long long vd, bool accumulate) {
        if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
                tc_mma_ts(tmem + 256 + t * 128, tmem + t * 128 + half * 32 + kk * 8, vd + half * 512 + kk * (2048 >> 4), idesc_pv, kk > 0 || accumulate);
        }
    };
    // Nothing is reported as done after a wait has run out: a producer that took a stage for free out of turn would arrive on a barrier whose phase
    // has both its arrivals but not all its bytes, which the hardware takes for an error.
    auto commit = [&](size_t bar) {
        if (expired == 0 && elect_one()) asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(sm_addr + (unsigned)bar) : "memory");
    };
    unsigned s0_at = 0;
    unsigned g = 0, done = 0, pairs = 0;      // steps, commits on step_done and tile pairs with a step so far
    unsigned loads0 = 0, loads1 = 0, steps0 = 0, steps1 = 0;   // tiles of Q, steps of each query tile
#pragma unroll 1
    for (unsigned it = 0; expired == 0; ++it) {
        const unsigned entry = sm_addr + (unsigned)offsetof(Storage, item) + (it & 1u) * (unsigned)sizeof(Item);
        wait(offsetof(Storage, item_full) + 8 * (it & 1u), (it >> 1) & 1u, 18);
        if (expired != 0) break;
        // n0, n1: K/V tiles that query tile 0 and 1 need (0: none, or no such tile)
        const int some = __shfl_sync(0xffffffffu, shared_int(entry + (unsigned)offsetof(Item, some)), 0);
        const int n0 = __shfl_sync(0xffffffffu, shared_int(entry + (unsigned)(offsetof(Item, t) + offsetof(TileInfo, n_kv))), 0);
        const int n1 = __shfl_sync(0xffffffffu, shared_int(entry + (unsigned)(offsetof(Item, t) + sizeof(TileInfo) + offsetof(TileInfo, n_kv))), 0);
        if (elect_one()) mbar_arrive_at(sm_addr + (unsigned)offsetof(Storage, item_empty) + 8 * (it & 1u));
        if (some == 0) break;
        const int n_max = max(n0, n1);
        if (n_max <= 0) {
            if (kOnePair) break;
            continue;
        }
        // The copies were requested in the order Q0, K0, Q1: the first S of tile 0 is issued as soon as
        // its two operands are there, without waiting for the other tile's Q.
        const unsigned long long kd0 = dk + (g & 1u) * kTileStep;
#pragma unroll 1
        for (int t = 0; t < 2; ++t) {
            if ((t == 0 ? n0 : n1) <= 0) continue;
            wait(offsetof(Storage, q_full) + 8 * t, (t == 0 ? loads0++ : loads1++) & 1u, 10);
            wait(offsetof(Storage, k_first), pairs & 1u, 11);
            if (D == 64) {
                // Two tiles that start together stay together, in each other's way at the exponentials (2900 clocks a step); near half a step apart they stay
                // so as well and take 2570. Where the pair has the steps to win the delay back.
                if (t == 1 && n0 >= 6)
                    while ((unsigned)clock64() - s0_at < kApart) {}
                s0_at = (unsigned)clock64();
            }
            tc_fence_after();
            issue_s(t, kd0);
            commit(offsetof(Storage, s_full) + 8 * t);
        }
        ++pairs;
        commit(offsetof(Storage, step_done) + 8 * (done++ & (kDone - 1)));
        FA_TRACE_EVENT(2, (int)g, 7);       // Q and the first K tile have landed
#pragma unroll 1
        for (int j = 0; j < n_max && expired == 0; ++j, ++g) {
            const unsigned s = g & 1u;   // stage of this step's V tile; the next K tile is in the other one
            const unsigned long long vd = dv + s * kTileStep, kd = dk + (s ^ 1u) * kTileStep;
            wait(offsetof(Storage, step_full) + 8 * s, (g >> 1) & 1u, 13);
            FA_TRACE_EVENT(2, (int)g, 4);
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const int n_kv = t == 0 ? n0 : n1;
                if (j < n_kv) {
                    // the first 64 keys of P_t arrive while the softmax still works on the other 64:
                    // their half of P.V leaves the critical path
                    const unsigned ph = (t == 0 ? steps0++ : steps1++) & 1u;
                    wait(offsetof(Storage, p_ready) + 8 * t, ph, 14 + t);
                    FA_TRACE_EVENT(2, (int)g, t * 2);
                    tc_fence_after();
                    issue_pv(t, 0, vd, j > 0);
                    wait(offsetof(Storage, p_ready) + 16 + 8 * t, ph, 16 + t);
                    FA_TRACE_EVENT(2, (int)g, 5 + t);
                    tc_fence_after();
                    issue_pv(t, 1, vd, true);
                    const bool more = j + 1 < n_kv;
                    if (more) issue_s(t, kd);
                    commit((more ? offsetof(Storage, s_full) : offsetof(Storage, o_full)) + 8 * t);
                    FA_TRACE_EVENT(2, (int)g, t * 2 + 1);
                }
            }
            commit(offsetof(Storage, step_done) + 8 * (done++ & (kDone - 1)));
        }
        if (kOnePair) break;
    }
    if (expired != 0 && !shared_flag(sm_addr + (unsigned)offsetof(Storage, abort_flag))) {   // (else another warp of the CTA gave up and reported it)
        set_shared_flag(sm_addr + (unsigned)offsetof(Storage, abort_flag));
        *reinterpret_cast<volatile int*>(status) = expired;
        __threadfence_system();
    }
    // Tensor memory is freed at the end of the kernel, in error paths while the softmax warps have long left: every product issued here has to
    // finish first (bounded; depends on the tensor pipe alone). Otherwise the last P.V is what the epilogue waits for as well.
    __syncwarp();
    expired = 0;
    commit(offsetof(Storage, drain));
    const unsigned long long t_begin = global_timer_ns();
    while (!mbar_try_wait_at(sm_addr + (unsigned)offsetof(Storage, drain), 0u) && global_timer_ns() - t_begin < 100000000ULL) {}
}

// One past the last key below `end` that the sequence's key-padding mask lets anybody see; 0: none. Run by one whole warp, 512 keys at a time from the end.
__device__ __noinline__ int seen_below(const unsigned char* mask_row, int end, int lane) {
#pragma unroll 1
    for (; end > 0; end -= 512) {
        int last = 0;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int key = end - 1 - lane - 32 * i;
            const bool there = key >= 0 && mask_row[max(key, 0)] != 0;
            last = max(last, there ? key + 1 : 0);
        }
        last = __reduce_max_sync(0xffffffffu, last);
        if (last > 0) return last;
    }
    return 0;
}

// The tile pair that CTA (bx, by, bz) of the grid stands for; false: there is none, or nothing to do for it. Run by one whole warp.
template <bool kMask, bool kPaged>
__device__ __forceinline__ bool find_pair(const PrefillArgs& a, int bx, int by, int bz, int lane, Item& w) {
    int pair;
    if (kPaged && a.ordered) {
        const int3 item = find_item(a, bx, lane);
        w.seq = item.x; w.kv_head = item.y; pair = item.z;
        if (w.seq < 0) return false;
    } else {
        // x = (batch element, KV head) x `band` neighbouring tile pairs, y = band of pairs,
        // heaviest (latest rows) first. Pairs are handed out in index order, so the `band` pairs that walk
        // the same K/V stream start together and meet its tiles in L2 instead of each pulling them from
        // HBM, while the order across bands stays heaviest first.
        // z = group of K/V streams: the grid runs group after group (each heaviest first), so that the
        // K/V of the streams in flight stay within L2 when every tile pair of a stream re-reads its stream's prefix
        const int x_band = a.by_band.div(bx);
        const int stream_id = bz * a.streams_z + x_band;
        if (stream_id >= a.kv_heads * a.batch) return false;   // the last group may be short
        w.seq = a.by_kv_heads.div(stream_id);
        w.kv_head = stream_id - w.seq * a.kv_heads;
        const int rank_y = launch_rank(by, a.spread_w, a.spread_m);   // this row's rank by weight, 0 = heaviest
        pair = ((int)gridDim.y - 1 - rank_y) * a.band + (a.band - 1 - (bx - x_band * a.band));
    }
    w.sq = seq_extent(a, w.seq);
    if ((w.sq.q_len << a.pack_log2) * a.by_packs.d <= a.skip_rows) return false;   // the few-row kernel's
    const int num_mb = row_blocks(w.sq.q_len, a.pack_log2);
    if (kMask) {
        // Padding behind a pair's last key that counts is not walked: the pair's keys end there, and a tile all of whose rows sit in padding (their output is zeros) sees none.
        const int last = tile_token_end(w.sq, pair * 2 + 1, a.by_packs, a.pack_log2, num_mb);   // one past the pair's last query token
        const int end = min(w.sq.kv_len, w.sq.pos_off + last);
        if (end > 0) w.sq.kv_len = seen_below(a.mask + (long long)w.seq * a.kv_seq_len, end, lane);
    }
    w.t[0] = tile_info<kMask>(w.sq, pair, 0, w.kv_head, a.by_packs, a.pack_log2, num_mb);
    w.t[1] = tile_info<kMask>(w.sq, pair, 1, w.kv_head, a.by_packs, a.pack_log2, num_mb);
    return w.t[0].valid || w.t[1].valid;   // (a sequence may be shorter than the grid's row range)
}

// Clusters: every thread of its CTAs takes part in every phase, and all waits of all roles end, so these do.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;\n" ::: "memory"); }
__device__ __forceinline__ unsigned peer_addr(const void* p, int rank) {   // the same place in another CTA's shared memory
    unsigned at;
    asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(at) : "r"(smem_u32(p)), "r"(rank));
    return at;
}

// The end of a pair whose keys are shared out over a cluster: every CTA has O over its share, unnormalised, and each row's reference and sum, lays them down where K and V were, and
// finishes 128 / parts rows of either tile from what all CTAs have: the rows' weights first, a thread a row, then a warp's lanes along the rows, 16 bytes each, eight loads in flight. What counts
// is the number of instructions, which come in for the first time at some 24 clocks each, and of trips to the other CTAs (some 800 clocks): two full tiles of 128 columns took
// 8 us by stores of 16 bytes into the other CTAs' rows, 7 with 16 loads in flight and the weights found by every lane, 4 so (device timer, clusters of two).
// Run by the eight softmax warps. `have`: the CTA has a pair, and this thread's tile is final.
template <typename T, int D, bool kMask>
__device__ __forceinline__ void split_rows(const PrefillArgs& a, SharedStorage<D>& sm, bool have, int t, int r, int warp, int lane, unsigned o_addr, int n_kv, float m, float l) {
    const int parts = a.parts, rank = (int)blockIdx.x & (parts - 1), share = kBlockM / parts;
    float* const rows = reinterpret_cast<float*>(sm.k[0]);   // K's and V's rings: (tile, row, D), 16-byte chunks swizzled by the row
    static_assert(offsetof(SharedStorage<D>, v) == offsetof(SharedStorage<D>, k) + sizeof(sm.k) && sizeof(sm.k) + sizeof(sm.v) >= 2 * kBlockM * D * 4, "the rings hold the rows of both tiles");
    float2* const ml = reinterpret_cast<float2*>(sm.out[0]);   // (tile, row)
    float* const weights = reinterpret_cast<float*>(sm.out[1]);   // (tile, row of the share, CTA)
    static_assert(sizeof(float2) * 2 * kBlockM <= kOutBytes && sizeof(float) * 2 * kBlockM / 2 * 8 <= kOutBytes, "fit");
    ml[t * kBlockM + r] = have ? make_float2(m, l) : make_float2(__int_as_float(0x7fffffff), __int_as_float(0x7fffffff));   // (else a wait ran out: the rows are undefined)
    const Item& w = sm.item[0];
    const int pl = a.pack_log2;
    if (have && n_kv > 0 && w.t[t].row0 + (warp & 3) * 32 < w.sq.q_len << pl) {   // (a warp whose rows exist)
        tc_fence_after();
        float* const mine = rows + (t * kBlockM + r) * D;
#pragma unroll 1
        for (int c = 0; c < D / 32; ++c) {
            float ov[32];
            tc_ld32(o_addr + c * 32, ov);
            tc_wait_ld();
#pragma unroll
            for (int i = 0; i < 8; ++i)
                *reinterpret_cast<float4*>(mine + (((c * 8 + i) ^ (r & 7)) << 2)) = make_float4(ov[4 * i], ov[4 * i + 1], ov[4 * i + 2], ov[4 * i + 3]);
        }
    }
    cluster_arrive();
    cluster_wait();
    const bool some = w.some && w.t[t].valid;
    const int rows_left = some ? (w.sq.q_len << pl) - w.t[t].row0 - rank * share : 0;   // rows of this share that exist
    if (r < share && r < rows_left) {
        const int row = w.t[t].row0 + rank * share + r, token = row >> pl, head = w.t[t].head + (row & ((1 << pl) - 1));
        float2 y[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            y[c] = make_float2(-INFINITY, 0.0f);
            if (c < parts) asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];\n" : "=f"(y[c].x), "=f"(y[c].y) : "r"(peer_addr(ml + t * kBlockM + rank * share + r, c)) : "memory");
        }
        // the row's reference and sum over all keys: the sum is NaN where one of the shares saw a NaN or +inf, as in a tile of one CTA
        float top = y[0].x, sum = 0.0f;
#pragma unroll
        for (int c = 1; c < 8; ++c) top = max_nan(top, y[c].x);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            y[c].x = y[c].x == -INFINITY ? 0.0f : ex2(y[c].x - top);
            sum = fmaf(y[c].x, y[c].y, sum);
        }
        bool q_ok = true;
        if (kMask) {
            const int pos = w.sq.pos_off + sm.share.first_key + token;
            q_ok = pos >= 0 && pos < w.sq.kv_len + sm.share.first_key && a.mask[(long long)w.seq * a.kv_seq_len + pos] != 0;
        }
        const bool seen = sum > 0.0f && top < INFINITY && q_ok;
        // (a share whose reference moved on behind its NaN has it in its sum and its O alone)
        const float inv = seen ? 1.0f / sum : sum != sum ? sum : 0.0f;
#pragma unroll
        for (int c = 0; c < 8; ++c)
            if (c < parts) weights[(t * share + r) * parts + c] = y[c].x * inv;
        if (a.lse != nullptr) a.lse[((long long)w.seq * a.q_heads + head) * a.q_seq_len + token] = seen ? (top + log2f(sum)) * 0.6931471805599453f : -INFINITY;
    }
    asm volatile("barrier.cta.sync 3, 256;\n" ::: "memory");   // the weights are there
    if (rows_left > 0) {
        constexpr int kLanes = D / 4, kRows = 32 / kLanes, kDeep = 4;   // lanes to a row; rows of a warp's load; loads of a part in flight
        const int col = (lane % kLanes) * 4;
#pragma unroll 1
        for (int i0 = (warp & 3) * kRows + lane / kLanes; i0 < share; i0 += 4 * kRows * kDeep) {
            float4 o[kDeep];
#pragma unroll
            for (int k = 0; k < kDeep; ++k) o[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 1
            for (int c = 0; c < parts; c += 2) {
                float4 x[2][kDeep];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const unsigned from = peer_addr(rows + (t * kBlockM + rank * share) * D, c + h);
#pragma unroll
                    for (int k = 0; k < kDeep; ++k) {
                        const int i = min(i0 + k * 4 * kRows, share - 1);
                        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n"
                                     : "=f"(x[h][k].x), "=f"(x[h][k].y), "=f"(x[h][k].z), "=f"(x[h][k].w)
                                     : "r"(from + i * (D * 4) + (((lane % kLanes) ^ ((rank * share + i) & 7)) << 4))
                                     : "memory");
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int k = 0; k < kDeep; ++k) {
                        const float by = weights[(t * share + min(i0 + k * 4 * kRows, share - 1)) * parts + c + h];
                        if (by != 0.0f) {   // (where a share saw no key, what lies there is nothing of ours)
                            o[k].x = fmaf(by, x[h][k].x, o[k].x);
                            o[k].y = fmaf(by, x[h][k].y, o[k].y);
                            o[k].z = fmaf(by, x[h][k].z, o[k].z);
                            o[k].w = fmaf(by, x[h][k].w, o[k].w);
                        }
                    }
            }
#pragma unroll
            for (int k = 0; k < kDeep; ++k) {
                const int i = i0 + k * 4 * kRows, row = w.t[t].row0 + rank * share + i;
                if (i < min(share, rows_left) && col < a.d_real) {
                    const long long at = ((w.sq.o_row0 + (row >> pl)) * a.o_heads + a.o_head0 + w.t[t].head + (row & ((1 << pl) - 1))) * a.d_real + col;
                    *reinterpret_cast<uint2*>(static_cast<T*>(a.o[0]) + at) = make_uint2(pack16<T>(o[k].x, o[k].y), pack16<T>(o[k].z, o[k].w));
                }
            }
        }
    }
    cluster_arrive();   // nobody's shared memory goes while another reads it
    cluster_wait();
}

// kMask: the call carries a key-padding mask (a separate instantiation, so that calls without one
// pay nothing for it in the softmax loop)
// kPaged: paged K/V, whose tiles are gathered page by page and whose tile pairs may be ordered on the device (a separate instantiation as
// well: with the code of the two in it the contiguous calls' kernel took 375 us for 24 prompts of 17-2000 tokens at d = 64,
// 364 without; 2 x 8192 GQA 1047 against 1027)
// kOnePair: a CTA works on its own tile pair and no other; nobody looks for a next one.
// kSplit (of those): the CTAs of a cluster share the keys of a tile pair and merge their rows through distributed shared memory.
template <typename T, int D, bool kMask, bool kPaged, bool kOnePair, bool kSplit>
__global__ void __launch_bounds__(kThreads, 1)
prefill_tcgen05_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map,
                       const __grid_constant__ CUtensorMap v_map, const __grid_constant__ CUtensorMap o_map, const PrefillArgs a) {
    extern __shared__ unsigned char smem_raw[];
    using Storage = SharedStorage<D>;
    Storage& sm = *reinterpret_cast<Storage*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
#ifdef FA_TRACE
    const long long t_entry = clock64();
    const unsigned long long ns_entry = a.cta_log != nullptr ? global_timer_ns() : 0ULL;
#endif

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);   // (the same for the whole warp, which the compiler sees only so)
    const int lane = threadIdx.x & 31;
    // A few-row kernel launched behind this one may start once every tile pair here is taken: it fills the SMs that run out of them.
    if (a.skip_rows > 0 && (kOnePair || !a.behind_few)) asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    // Packed buffers end at row cu_seqlens[num_seqs]; where the tensor map does not end with the buffer, a tile that reaches past that row is not asked
    // of the copy engine but fetched by the producer warp (see edge_tile_copy). A map that does gives zeros there like any other.
    const bool packed = a.mode == MODE_VARLEN;

    // Register budget: the kernel is compiled for 168 registers per thread (384 threads); the
    // producer/issuer warpgroup hands most of its share to the two softmax warpgroups, which
    // keep a whole 128-column score row per thread in registers.
    if (warp >= 8) {
    // One instruction for the four warps, as the instruction wants it, and ahead of what they do first: the softmax warps wait for the registers that all four give back. Behind
    // the K producer's first copies (which have no use for more than 88) 2 x 128, 32/8 heads took 7.2 us instead of 6.6 from a graph, 2 x 433 MHA 11.0 and 10.7.
    asm volatile("setmaxnreg.dec.sync.aligned.u32 88;\n");
    // Packed buffers whose ends the tensor maps do not know.
    const bool q_open = packed && !a.q_bounded, kv_open = packed && !a.paged && !a.kv_bounded;
    if (warp == kLoadWarp) {
        // ------------------------------ tile pairs, Q and K tiles ------------------------------
        // The warps run their loops whole; lane 0 issues the bulk copies (a paged tile: a lane per page), and all lanes share the
        // plain-load copy of a tile at the very end of a packed buffer.
        Item w;
        bool begun = false;   // the first tile pair's first copies have been requested
        // The CTA's own tile pair, and its first copies at once, in as few instructions as that takes: all of them come in for the first time here, and
        // in the loop below, with its waits and cases, the first S came 1600 to 2300 clocks later (a fifth of a call of one short wave).
        w.some = find_pair<kMask, kPaged>(a, kSplit ? (int)blockIdx.x / a.parts : (int)blockIdx.x, (int)blockIdx.y, (int)blockIdx.z, lane, w);
        Share share{0, 0};
        if (kSplit) {
            if (w.some) share = take_share(w, a.parts, (int)blockIdx.x % a.parts);
            if (lane == 0) sm.share = share;   // (with the pair, or with the word that there is none)
        }
        asm volatile("barrier.cta.sync 1, 96;\n" ::: "memory");   // the barriers have been initialised
        begun = w.some && max(w.t[0].n_kv, w.t[1].n_kv) > 0 && !q_open && !kv_open && a.test_skip_k != 1;
        if (begun && (kPaged || lane == 0)) {
            const int page = kPaged ? page_of_lane(a, w.sq.kv_len, w.seq, 0, lane, share.first_key) : -1;
            if (lane == 0 && w.t[0].n_kv > 0) {
                mbar_expect_tx(&sm.q_full[0], TileBytes<D>::value);
                tma_load_4d(sm.q[0], &q_map, &sm.q_full[0], 0, w.t[0].head, w.sq.q_crow + (w.t[0].row0 >> a.pack_log2), w.sq.q_cb);
                if (D == 128) tma_load_4d(sm.q[0] + kHalfBytes, &q_map, &sm.q_full[0], 64, w.t[0].head, w.sq.q_crow + (w.t[0].row0 >> a.pack_log2), w.sq.q_cb);
            }
            load_kv_tile<D, kPaged>(a, w.sq.kv_crow, w.sq.kv_cb, w.kv_head, sm.k[0], &k_map, &sm.k_first, 0, page, lane);
            if (lane == 0 && w.t[1].n_kv > 0) {
                mbar_expect_tx(&sm.q_full[1], TileBytes<D>::value);
                tma_load_4d(sm.q[1], &q_map, &sm.q_full[1], 0, w.t[1].head, w.sq.q_crow + (w.t[1].row0 >> a.pack_log2), w.sq.q_cb);
                if (D == 128) tma_load_4d(sm.q[1] + kHalfBytes, &q_map, &sm.q_full[1], 64, w.t[1].head, w.sq.q_crow + (w.t[1].row0 >> a.pack_log2), w.sq.q_cb);
            }
        }
        if (lane == 0 && w.some) {   // (published here, the other roles have read it when the first scores come)
            sm.item[0] = w;
            mbar_arrive(&sm.item_full[0]);
        }
        __syncwarp();
        const long long tot_q = q_open ? (long long)a.cu_q[a.batch] : 0;
        const long long tot_k = kv_open ? (long long)a.cu_k[a.batch] : 0;
        int g = 0, commits = 0;              // steps and commits on step_done of the tile pairs before this one
        int k_free0 = -1, k_free1 = -1;      // the commit that frees each K stage (-1: free)
        unsigned scores0 = 0, scores1 = 0;   // S of each query tile so far: its Q is free when the last one has finished
        bool q_used0 = false, q_used1 = false;   // (and has to be waited for: by the pair before this one)
        int first_s = -1;                    // the commit of the last pair's first S, where that pair had one step (else it has been waited for)
        int given = 0;                       // steps whose K arrival has been made or comes with a copy that has been requested
        unsigned q_loads0 = 0, q_loads1 = 0, firsts = 0, requests = 0, answers = 0;   // firsts: K tiles 0 that have been requested
        bool alive = true;
#ifdef FA_TRACE
        long long* const trace = (a.trace != nullptr && blockIdx.x == 0 && blockIdx.y == (unsigned)a.trace_y && blockIdx.z == 0 && lane == 0) ? a.trace : nullptr;
#endif
        auto wait_commit = [&](int c) { return c < 0 || __all_sync(0xffffffffu, producer_wait(sm, &sm.step_done[c & (kDone - 1)], (unsigned)(c / kDone) & 1u, a, 1)); };
        auto ask = [&]() {
            if (lane == 0) {
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");   // (the answer before has been read)
                mbar_expect_tx(&sm.answered, 16);
                request_pair(sm.answer, &sm.answered);
            }
            ++requests;
            FA_TRACE_EVENT(3, (int)requests, 0);
        };
        const bool have = w.some;            // the CTA's own tile pair is published
        bool owed = false;                   // the arrival that the last step of the pair before waits for, in place of another K tile
        auto owed_commit = [&]() { return (g & 1) ? k_free1 : k_free0; };
        for (unsigned it = 0;; ++it) {
            if (owed) {
                const int c = owed_commit();
                if (c < 0 || __all_sync(0xffffffffu, mbar_test_at(smem_u32(&sm.step_done[c & (kDone - 1)]), (unsigned)(c / kDone) & 1u))) {
                    if (lane == 0) mbar_arrive(&sm.step_full[(g - 1) & 1]);
                    given = g;
                    owed = false;
                }
            }
            // The next tile pair with something to do: this CTA's own first, then those of CTAs that have not started. Asked for when the pair at hand has its
            // last K tile requested, two to three steps before its end: whoever comes to its end first takes the next one. Asked for at a
            // pair's beginning, the order heaviest first was lost for the second half of 4 chunks of 512 (256 pairs on 148 SMs): 174 us instead of
            // 153. The answer takes 1100 to 3100 clocks, what follows from it until the first copy 2000 more.
            if (it > 0) w.some = 0;
            if (!kOnePair && !w.some) {
                if (requests == answers) ask();
                if (it >= 2) alive = __all_sync(0xffffffffu, mbar_wait(sm, &sm.item_empty[it & 1u], ((it >> 1) - 1u) & 1u, a, 5));
                while (alive) {
                    int bx, by, bz;
                    alive = __all_sync(0xffffffffu, mbar_wait(sm, &sm.answered, answers & 1u, a, 6));
                    if (!alive) break;
                    ++answers;
                    FA_TRACE_EVENT(3, (int)answers, 1);
                    const bool got = read_answer(sm.answer, bx, by, bz);
                    __syncwarp();
                    if (!got) break;   // every tile pair is taken
                    w.some = find_pair<kMask, kPaged>(a, bx, by, bz, lane, w);
                    if (w.some) break;
                    ask();
                }
                if (!alive) break;
            }
            if (!w.some) w.t[0].n_kv = w.t[1].n_kv = 0;
            if (lane == 0 && (kOnePair ? it == 0 && !w.some : it > 0 || !have)) {
                sm.item[it & 1u] = w;
                mbar_arrive(&sm.item_full[it & 1u]);
            }
            FA_TRACE_EVENT(3, (int)it, 2);
            if (owed) {
                alive = wait_commit(owed_commit());
                if (!alive) break;
                if (lane == 0) mbar_arrive(&sm.step_full[(g - 1) & 1]);
                given = g;
                owed = false;
            }
            if (!w.some) break;
            const int kv_len = w.sq.kv_len, kv_crow = w.sq.kv_crow, kv_cb = w.sq.kv_cb, seq = w.seq, kv_head = w.kv_head;
            const int n0 = w.t[0].n_kv, n1 = w.t[1].n_kv, n_max = max(n0, n1);
            if (n_max <= 0) {
                if (kOnePair) break;
                ask();
                continue;
            }
            if (it > 0 && !q_open && lane == 0) {   // its Q on the way to L2 while the tiles before it are still in use
                if (n0 > 0) {
                    tma_prefetch_4d(&q_map, 0, w.t[0].head, w.sq.q_crow + (w.t[0].row0 >> a.pack_log2), w.sq.q_cb);
                    if (D == 128) tma_prefetch_4d(&q_map, 64, w.t[0].head, w.sq.q_crow + (w.t[0].row0 >> a.pack_log2), w.sq.q_cb);
                }
                if (n1 > 0) {
                    tma_prefetch_4d(&q_map, 0, w.t[1].head, w.sq.q_crow + (w.t[1].row0 >> a.pack_log2), w.sq.q_cb);
                    if (D == 128) tma_prefetch_4d(&q_map, 64, w.t[1].head, w.sq.q_crow + (w.t[1].row0 >> a.pack_log2), w.sq.q_cb);
                }
            }
            int page = kPaged ? page_of_lane(a, kv_len, seq, 0, lane, share.first_key) : -1;
            auto load_k = [&](int j) {   // K tile j of the pair is what step g + j - 1 reads besides its V tile, and arrives on its barrier (tile 0: on its own)
                const int e = (g + j) & 1;
                unsigned long long* const bar = j == 0 ? &sm.k_first : &sm.step_full[e ^ 1];
                const bool skip = a.test_skip_k == j + 1;   // (the test hook's tile is never requested, the issuer's wait for it runs out)
                if (skip) {
                    if (lane == 0) sm.left_out = j > 0 ? g + j : 0;
                } else if (kv_open && (long long)kv_crow + (long long)(j + 1) * kBlockN > tot_k) {
                    edge_tile_copy<D>(sm.k[e], a.k, a.kv_heads, kv_head, (long long)kv_crow + (long long)j * kBlockN, tot_k, bar, lane, a.d_real);
                } else if (kPaged || lane == 0) {
                    load_kv_tile<D, kPaged>(a, kv_crow, kv_cb, kv_head, sm.k[e], &k_map, bar, j, page, lane);
                }
                (e ? k_free1 : k_free0) = commits + j;
                if (j > 0) given = g + j;
                else if (!skip) ++firsts;
                if (kPaged && j + 1 < n_max) page = page_of_lane(a, kv_len, seq, j + 1, lane, share.first_key);
            };
            // (a tile that sees no key needs no Q: the issuer leaves it out)
            auto load_q = [&](const TileInfo ti, unsigned char* to, unsigned long long* bar, unsigned& loads) {
                if (ti.n_kv <= 0) return;
                ++loads;
                const int token0 = ti.row0 >> a.pack_log2;
                if (q_open && (long long)w.sq.q_crow + token0 + (kBlockM >> a.pack_log2) > tot_q) {
                    edge_tile_copy<D>(to, a.q, a.q_heads, ti.head, (long long)w.sq.q_crow + token0, tot_q, bar, lane, a.d_real, a.pack_log2);
                } else if (lane == 0) {
                    mbar_expect_tx(bar, TileBytes<D>::value);
                    tma_load_4d(to, &q_map, bar, 0, ti.head, w.sq.q_crow + token0, w.sq.q_cb);
                    if (D == 128) tma_load_4d(to + kHalfBytes, &q_map, bar, 64, ti.head, w.sq.q_crow + token0, w.sq.q_cb);
                }
            };
            // K tile 0 and the Q tiles: of the first pair in the order that the issuer wants them; else K first, which comes free first, then the Q tile that does, of
            // two row blocks of one head the shorter one, tile 1.
            auto wait_q = [&](int t, unsigned scores) { return __all_sync(0xffffffffu, producer_wait(sm, &sm.s_full[t], (scores - 1u) & 1u, a, 8)); };
            if (it == 0 && begun) {
                k_free0 = 0;
                firsts = 1;
                q_loads0 = n0 > 0;
                q_loads1 = n1 > 0;
                if (kPaged && n_max > 1) page = page_of_lane(a, kv_len, seq, 1, lane, share.first_key);
            } else
#pragma unroll 1
            for (int n = 0; n < 3; ++n) {
                if (n == (it == 0 ? 1 : 0)) {
                    alive = wait_commit(first_s) &&   // the last pair's K tile 0 has left its barrier
                            wait_commit((g & 1) ? k_free1 : k_free0);
                    if (!alive) break;
                    load_k(0);
                    FA_TRACE_EVENT(3, (int)it, 3);
                } else {
                    const int t = it == 0 ? n >> 1 : 2 - n;
                    if (t ? q_used1 : q_used0) alive = wait_q(t, t ? scores1 : scores0);
                    if (!alive) break;
                    load_q(t ? w.t[1] : w.t[0], sm.q[t], &sm.q_full[t], t ? q_loads1 : q_loads0);
                    FA_TRACE_EVENT(3, (int)it, 4 + t);
                }
            }
            if (!alive) break;
            for (int j = 1; j < n_max; ++j) {
                alive = wait_commit(((g + j) & 1) ? k_free1 : k_free0);
                if (!alive) break;
                load_k(j);
            }
            if (!alive) break;
            owed = true;
            // (waits are for commits of late only, see step_done: where this pair had no use for a Q tile, that has long been free)
            first_s = n_max == 1 ? commits : -1;
            q_used0 = n0 > 0;
            q_used1 = n1 > 0;
            scores0 += (unsigned)max(n0, 0);
            scores1 += (unsigned)max(n1, 0);
            commits += n_max + 1;
            g += n_max;
        }
        if (lane == 0) {
            if (!all_read(sm, alive, a, 3))
                settle_copies(sm, given, sm.left_out,
                              (unsigned)(answers != requests) | (answers & 1u) << 1 | (unsigned)(q_loads0 > 0) << 2 | ((q_loads0 - 1u) & 1u) << 3 |
                                  (unsigned)(q_loads1 > 0) << 4 | ((q_loads1 - 1u) & 1u) << 5 | (unsigned)(firsts > 0) << 6 | ((firsts - 1u) & 1u) << 7);
        }
    } else if (warp == kLoadWarpV) {
        // ------------------------------ V tiles ------------------------------
        // A producer of its own: with a paged cache a tile is one copy per page and 64-column half plus a block-table read per page, and a single
        // thread issuing both rings cannot keep up with the tensor pipe at small page sizes.
        asm volatile("barrier.cta.sync 1, 96;\n" ::: "memory");   // the barriers have been initialised
        const long long tot_k = kv_open ? (long long)a.cu_k[a.batch] : 0;
        int g = 0, commits = 0;
        int v_free0 = -1, v_free1 = -1;
        unsigned tails = 0;
        bool alive = true, tail_pending = false;   // tail_pending: the tail tile's copy was issued and v_tail not yet seen complete
        int given = 0;                         // as in the K producer
        for (unsigned it = 0;; ++it) {
            alive = __all_sync(0xffffffffu, producer_wait(sm, &sm.item_full[it & 1u], (it >> 1) & 1u, a, 7));
            if (!alive) break;
            const Item w = sm.item[it & 1u];
            const Share share = kSplit ? sm.share : Share{0, 0};
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.item_empty[it & 1u]);
            if (!w.some) break;
            const SeqExtent& sq = w.sq;
            const int n_max = max(w.t[0].n_kv, w.t[1].n_kv);
            if (n_max <= 0) {
                if (kOnePair) break;
                continue;
            }
            // The sequence's last V tile, when the sequence does not end on a tile boundary, holds rows
            // that are not this sequence's: the unwritten rest of its last page, or the next sequence
            // of a packed buffer. P is exactly zero there, but 0 x NaN (an uninitialised pool, a page
            // recycled from other use) would still poison the whole output row, so those rows are
            // cleared in shared memory before the tile is handed to the MMA issuer: its copy completes
            // on a barrier of its own, the producer warp zeroes the rows and then completes the
            // ring's barrier with a plain arrival. (Garbage in K is harmless: the score mask is a select.)
            const bool tail_fix = (a.paged || packed) && (sq.kv_len % kBlockN) != 0;
            const int tail_j = sq.kv_len > 0 ? (sq.kv_len - 1) / kBlockN : -1;
            int page = kPaged ? page_of_lane(a, sq.kv_len, w.seq, 0, lane, share.first_key) : -1;
            for (int j = 0; j < n_max; ++j) {
                const int e = (g + j) & 1;
                const int c = e ? v_free1 : v_free0;
                if (c >= 0) alive = __all_sync(0xffffffffu, producer_wait(sm, &sm.step_done[c & (kDone - 1)], (unsigned)(c / kDone) & 1u, a, 2));
                if (!alive) break;
                const bool fix = tail_fix && j == tail_j;
                unsigned long long* const bar = fix ? &sm.v_tail : &sm.step_full[e];
                if (kv_open && (long long)sq.kv_crow + (long long)(j + 1) * kBlockN > tot_k)
                    edge_tile_copy<D>(sm.v[e], a.v, a.kv_heads, w.kv_head, (long long)sq.kv_crow + (long long)j * kBlockN, tot_k, bar, lane, a.d_real);
                else if (kPaged || lane == 0)
                    load_kv_tile<D, kPaged>(a, sq.kv_crow, sq.kv_cb, w.kv_head, sm.v[e], &v_map, bar, j, page, lane);
                (e ? v_free1 : v_free0) = commits + j + 1;
                if (kPaged && j + 1 < n_max) page = page_of_lane(a, sq.kv_len, w.seq, j + 1, lane, share.first_key);
                if (!fix) {
                    given = g + j + 1;
                    continue;
                }
                tail_pending = true;
                alive = __all_sync(0xffffffffu, producer_wait(sm, &sm.v_tail, tails & 1u, a, 4));
                if (!alive) break;
                tail_pending = false;
                ++tails;
                const int first = sq.kv_len - j * kBlockN;   // first row of the tile that is not this sequence's
                constexpr int kChunksPerHalfRow = 8;        // 128 B per row and 64-column half
                const int n_chunks = (kBlockN - first) * kChunksPerHalfRow;
                for (int h = 0; h < D / 64; ++h)
                    for (int idx = lane; idx < n_chunks; idx += 32)
                        *reinterpret_cast<uint4*>(sm.v[e] + h * kHalfBytes + first * 128 + idx * 16) = make_uint4(0u, 0u, 0u, 0u);
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");   // generic-proxy writes -> tensor-core reads
                __syncwarp();
                if (lane == 0) mbar_arrive(&sm.step_full[e]);
                given = g + j + 1;
            }
            if (!alive) break;
            if (kOnePair) break;
            commits += n_max + 1;
            g += n_max;
        }
        if (lane == 0) {
            if (!all_read(sm, alive, a, 9)) settle_copies(sm, given, 0, (unsigned)tail_pending << 8 | (tails & 1u) << 9);
        }
    } else if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(smem_u32(&sm.tmem_base)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
        tc_fence_before();
        asm volatile("barrier.cta.sync 2, 320;\n" ::: "memory");
        tc_fence_after();
#ifdef FA_TRACE
        // only the heaviest CTA of the first (batch, KV head) records its timeline, one thread per role
        long long* const trace = (a.trace != nullptr && blockIdx.x == 0 && blockIdx.y == (unsigned)a.trace_y && blockIdx.z == 0 && lane == 0) ? a.trace : nullptr;
        // slot kTraceSteps - 1 of each role holds the CTA's life cycle instead of a kv step
        if (trace != nullptr) {
            trace[(2 * kTraceSteps + kTraceSteps - 1) * 8 + 0] = t_entry;
            FA_TRACE_EVENT(2, kTraceSteps - 1, 1);   // set-up (barriers, tensor memory) done
        }
#endif
        issue_products<T, D, kOnePair>(smem_u32(&sm), sm.tmem_base, a.status, a.wait_ns FA_TRACE_ARG(trace));
    } else {
        // ------------------------------ set-up ------------------------------
        // By the warp that has nothing else to do, while the K producer finds out what the CTA's first tile pair is.
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];\n" ::"l"(&q_map) : "memory");
            asm volatile("prefetch.tensormap [%0];\n" ::"l"(&k_map) : "memory");
            asm volatile("prefetch.tensormap [%0];\n" ::"l"(&v_map) : "memory");
            sm.abort_flag = 0;
            sm.left_out = 0;
            for (int i = 0; i < 2; ++i) {
                mbar_init(&sm.item_full[i], 1);
                mbar_init(&sm.item_empty[i], 10);
                mbar_init(&sm.q_full[i], 1);
                mbar_init(&sm.s_full[i], 1);
                mbar_init(&sm.o_full[i], 1);
                mbar_init(&sm.p_ready[0][i], 128);
                mbar_init(&sm.p_ready[1][i], 128);
                mbar_init(&sm.step_full[i], 2);
            }
            for (int i = 0; i < kDone; ++i) mbar_init(&sm.step_done[i], 1);
            mbar_init(&sm.answered, 1);
            mbar_init(&sm.k_first, 1);
            mbar_init(&sm.v_tail, 1);
            mbar_init(&sm.drain, 1);
            asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        }
        __syncwarp();
        asm volatile("barrier.cta.arrive 1, 96;\n" ::: "memory");    // the producers
        asm volatile("barrier.cta.arrive 2, 320;\n" ::: "memory");   // issuer and softmax warps, which wait for tensor memory as well
        // This grid's completion stands for the few-row kernel's that was launched ahead of it (whose CTAs have all started when this one begins), so its CTAs end behind that. In this warp, which has nothing else to do: at the
        // end of every CTA the look whether there is one took 0.1 us of each call. Calls of one pair to a CTA never have one (see launch_variant).
        if (!kOnePair && a.behind_few) asm volatile("griddepcontrol.wait;\n" ::: "memory");
    }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 208;\n");
        // ------------------------------ softmax warpgroups ------------------------------
        asm volatile("barrier.cta.sync 2, 320;\n" ::: "memory");   // barriers and tensor memory
        tc_fence_after();
        const unsigned tmem = sm.tmem_base;
        const int t = warp >> 2;
        const int r = (warp & 3) * 32 + lane;                  // row within the tile == TMEM lane
        const unsigned lane_base = (unsigned)((warp & 3) * 32) << 16;
        const unsigned s_addr = tmem + lane_base + t * 128;
        const unsigned o_addr = tmem + lane_base + 256 + t * 128;
        unsigned steps = 0, tiles = 0;    // of this query tile so far: steps, and tiles with a step
        [[maybe_unused]] bool have = false;
        [[maybe_unused]] int last_n = 0;
        [[maybe_unused]] float last_m = 0.0f, last_l = 0.0f;
        bool alive = true;
#ifdef FA_TRACE
        long long* trace = (a.trace != nullptr && blockIdx.x == 0 && blockIdx.y == (unsigned)a.trace_y && blockIdx.z == 0 && lane == 0 && (warp & 3) == 0) ? a.trace : nullptr;
#endif
#pragma unroll 1
        for (unsigned it = 0; alive && (!kOnePair || it == 0); ++it) {
        alive = __all_sync(0xffffffffu, mbar_wait(sm, &sm.item_full[it & 1u], (it >> 1) & 1u, a, 22 + t));
        if (!alive) break;
        const bool some = sm.item[it & 1u].some != 0;
        const int b = sm.item[it & 1u].seq;
        const SeqExtent sq = sm.item[it & 1u].sq;
        const TileInfo ti = sm.item[it & 1u].t[t];
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.item_empty[it & 1u]);
        if (!some) break;
        const int first_key = kSplit ? sm.share.first_key : 0;
        const int row = ti.row0 + r, pl = a.pack_log2;
        const int pos = sq.pos_off + (row >> pl);   // global position of this row's query token
        // the last key that this row sees, and the last that every row of the tile sees (-1: none)
        const int last_seen = max(-1, min(pos, sq.kv_len - 1)), all_see = max(-1, min(sq.pos_off + (ti.row0 >> pl), sq.kv_len - 1));
        float m = -INFINITY;   // reference max, log2 domain (may lag the true max by <= 2^8)
        float l = 0.0f;

        for (int j = 0; j < ti.n_kv && alive; ++j) {
            alive = __all_sync(0xffffffffu, mbar_wait(sm, &sm.s_full[t], steps & 1u, a, 20 + t));
            if (!alive) break;
            ++steps;
            FA_TRACE_EVENT(t, (int)steps - 1, 0);
            tc_fence_after();
            const int key0 = j * kBlockN;
            // mask only where the causal diagonal or the end of K/V cuts through this tile
            const bool need_mask = key0 + kBlockN - 1 > all_see;
            const int limit = need_mask ? max(-1, min(last_seen - key0, kBlockN)) : kBlockN;

            // Masked scores become -inf, whose P is an exact zero from either exponential, so a masked tile runs the code of the others. (A form of its own
            // for the aligned diagonal, which left out the chunks of 32 keys that a warp does not see, and one for other masked tiles were straight-line
            // code run once per tile: 2 x 8192 GQA 967 us with them, 948 without. Leaving unseen chunks out behind a branch in this
            // code: 990 us, for what the compiler no longer interleaves.)
            // Key-padding mask (batched entry point): the tile's validity bytes become a ballot per chunk of 32; a tile whose real keys are all
            // valid (the usual case, padding sits at one end) runs as if there were no mask.
            unsigned valid[4];
            bool masked = need_mask;
            if (kMask) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int kk = key0 + c * 32 + lane;
                    const bool real = kk < sq.kv_len;
                    valid[c] = __ballot_sync(0xffffffffu, real && a.mask[(long long)b * a.kv_seq_len + first_key + (real ? kk : 0)] != 0);
                    masked = masked || valid[c] != __ballot_sync(0xffffffffu, real);
                }
            }
            float sv[4][32];
#pragma unroll
            for (int c = 0; c < 4; ++c) tc_ld32(s_addr + c * 32, sv[c]);
            tc_wait_ld();
            if (masked) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int n = limit + 1 - c * 32;
                    unsigned seen = n >= 32 ? 0xffffffffu : (n <= 0 ? 0u : (1u << n) - 1u);   // keys that this row sees of the chunk
                    if (kMask) seen &= valid[c];
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        if (!((seen >> i) & 1u)) sv[c][i] = -INFINITY;
                }
            }
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int i = 0; i < 32; i += 2) mx4[(i >> 1) & 3] = max3_nan(mx4[(i >> 1) & 3], sv[c][i], sv[c][i + 1]);
            // A row that sees a NaN outputs NaN whichever unit takes that key's exponential: its maximum is NaN, and with it the reference below, every
            // exponential of the tile and the row's sum from here on. A +inf stays the reference to the end, where the epilogue sees it.
            const float mx = max_nan(max3_nan(mx4[0], mx4[1], mx4[2]), mx4[3]) * a.scale_log2;   // scale > 0 is guaranteed by the dispatcher
            FA_TRACE_EVENT(t, (int)steps - 1, 1);

            float alpha = 1.0f;
            bool changed = false;
            if (!(mx <= m + kRescaleThreshold)) {   // also for the first finite max (m == -inf) and where either is NaN
                alpha = ex2(m - mx);                // 0 when m == -inf
                m = mx;
                changed = true;
            }
            if (j > 0 && __any_sync(0xffffffffu, changed)) {
                // rescale this warp's 32 rows of O in tensor memory (rows that did not move use 1.0)
#pragma unroll 1
                for (int c = 0; c < D / 32; ++c) {
                    float ov[32];
                    tc_ld32(o_addr + c * 32, ov);
                    tc_wait_ld();
                    unsigned ou[32];
#pragma unroll
                    for (int i = 0; i < 32; ++i) ou[i] = __float_as_uint(ov[i] * alpha);
                    tc_st32(o_addr + c * 32, ou);
                }
            }
            const float m_use = (m == -INFINITY) ? 0.0f : m;
            // exp2(s * scale - m) two columns at a time: packed FMA for the argument and the row sum
            const unsigned long long scale2 = pack2(a.scale_log2, a.scale_log2);
            const unsigned long long neg_m2 = pack2(-m_use, -m_use);
            unsigned long long sum2 = pack2(0.0f, 0.0f);
#pragma unroll
            for (int h = 0; h < 2; ++h) {   // 64 keys
                unsigned pu[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    const float(&x)[32] = sv[h * 2 + (i >> 4)];
                    const int ii = (i & 15) * 2;
                    float x0, x1, e0, e1;
                    unpack2(fma2(pack2(x[ii], x[ii + 1]), scale2, neg_m2), x0, x1);
                    if (fma_pipe_exp<D>(i)) {
                        ex2_fma2(x0, x1, e0, e1);
                    } else {
                        e0 = ex2(x0);
                        e1 = ex2(x1);
                    }
                    sum2 = add2(sum2, pack2(e0, e1));
                    pu[i] = pack16<T>(e0, e1);
                }
                tc_st32(s_addr + h * 32, pu);
                tc_wait_st();
                tc_fence_before();
                mbar_arrive(&sm.p_ready[h][t]);
                if (h == 0) FA_TRACE_EVENT(t, (int)steps - 1, 2);
            }
            float sum_lo, sum_hi;
            unpack2(sum2, sum_lo, sum_hi);
            l = l * alpha + (sum_lo + sum_hi);
            FA_TRACE_EVENT(t, (int)steps - 1, 3);
        }

        // epilogue: O_t is final once the commit after the last P.V has arrived
        if (alive && ti.n_kv > 0)
            alive = __all_sync(0xffffffffu, mbar_wait(sm, &sm.o_full[t], tiles++ & 1u, a, 30 + t));
        FA_TRACE_EVENT(t, max(0, (int)steps - 1), 4);
        if (kSplit && sm.share.some) {
            have = alive;
            last_n = ti.n_kv;
            last_m = m;
            last_l = l;
            break;
        }
        if (alive && ti.valid) {
            tc_fence_after();
            const int rows_end = sq.q_len << pl, token = row >> pl, head = ti.head + (row & ((1 << pl) - 1));
            const bool row_ok = row < rows_end;
            // with a padding mask a query row at a padded (or out-of-range) position outputs zeros (flash_attn_func.cu:77-84)
            bool q_ok = true;
            if (kMask) q_ok = row_ok && pos >= 0 && pos < sq.kv_len && a.mask[(long long)b * a.kv_seq_len + pos] != 0;
            const bool seen = l > 0.0f && m < INFINITY && q_ok;   // (false where a score was NaN, l NaN, or +inf, m +inf: 0 times that row's NaN or infinity is NaN)
            const float inv = seen ? 1.0f / l : 0.0f;
            // a bulk store writes every row of its box that lies inside the tensor: in a packed buffer the
            // rows after this sequence belong to the next one, so a tile that overhangs the end of its
            // sequence is written row by row
#ifdef FA_TRACE
            const bool staged_only = a.staged_store != 0;
#else
            constexpr bool staged_only = false;
#endif
            unsigned char* const stage = sm.out[warp];
            const bool bulk_ok = a.n_out == 1 && !a.multicast && !staged_only && (a.mode != MODE_VARLEN || ti.row0 + kBlockM <= rows_end);
            if (bulk_ok) {
                // Single output: the rows go out as bulk tensor stores. Each warp lays its 32 rows down in
                // shared memory in the 128-byte-swizzled box layout, 64 columns at a time, and one lane issues one store of 32 rows x 64 columns. Plain 16-byte stores
                // of 32 different rows per instruction would fill the SM's memory pipeline for thousands
                // of clocks and hold up the barrier traffic of the other tile's last steps. Rows past the
                // end of the sequence are outside the tensor map and are not written.
                // Where no tile pair follows, the second half goes through the Q tile's shared memory and need not wait until the first has been read (0.4 us).
                const bool last = D == 128 && (kOnePair || __all_sync(0xffffffffu, mbar_test_at(smem_u32(&sm.item_full[(it + 1u) & 1u]), ((it + 1u) >> 1) & 1u) && sm.item[(it + 1u) & 1u].some == 0));
#pragma unroll 1
                for (int h = 0; h < D / 64; ++h) {   // a half's copy is on its way while the next one is read and scaled
                    unsigned char* const half = h > 0 && last ? sm.q[t] + (warp & 3) * kOutBytes : stage;
                    float ov[2][32];
                    __syncwarp();   // (one lane has stored)
                    tc_ld32(o_addr + h * 64, ov[0]);
                    tc_ld32(o_addr + h * 64 + 32, ov[1]);
                    tc_wait_ld();
                    if (ti.n_kv == 0) {   // the tile saw no key: tensor memory holds nothing of ours, the rows are zeros
#pragma unroll
                        for (int i = 0; i < 32; ++i) ov[0][i] = ov[1][i] = 0.0f;
                    }
                    if (lane == 0 && !(h > 0 && last)) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");   // what was laid down here before has been read
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 8; ++i) {   // 16-byte chunk i of the 64-column half
                        const float* o8 = &ov[i >> 2][8 * (i & 3)];
                        uint4 w;
                        w.x = pack16<T>(o8[0] * inv, o8[1] * inv);
                        w.y = pack16<T>(o8[2] * inv, o8[3] * inv);
                        w.z = pack16<T>(o8[4] * inv, o8[5] * inv);
                        w.w = pack16<T>(o8[6] * inv, o8[7] * inv);
                        *reinterpret_cast<uint4*>(half + lane * 128 + ((i ^ (lane & 7)) << 4)) = w;
                    }
                    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");   // generic-proxy writes -> bulk copy reads
                    __syncwarp();
                    if (lane == 0) {
                        tma_store_4d(&o_map, half, h * 64, a.o_head0 + ti.head, sq.q_crow + ((ti.row0 + (warp & 3) * 32) >> pl), sq.q_cb);
                        asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
                    }
                }
            } else if (a.n_out == 1 && !a.multicast && !staged_only) {
                // A tile that overhangs its sequence: the rows that exist, from registers in 32-byte stores (whole sectors).
#pragma unroll 1
                for (int c = 0; c < D / 32; ++c) {
                    float ov[32];
                    __syncwarp();   // (lanes whose rows exist have stored)
                    tc_ld32(o_addr + c * 32, ov);
                    tc_wait_ld();
                    T* const to = static_cast<T*>(a.o[0]) + ((sq.o_row0 + token) * a.o_heads + a.o_head0 + head) * a.d_real + c * 32;
                    if (row_ok && c * 32 < a.d_real) {
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            unsigned w[8];
#pragma unroll
                            for (int x = 0; x < 8; ++x) w[x] = ti.n_kv == 0 ? 0u : pack16<T>(ov[16 * i + 2 * x] * inv, ov[16 * i + 2 * x + 1] * inv);
                            store_32(to + i * 16, w, a.o_by_32 != 0);
                        }
                    }
                }
            } else {
                // Several GPUs' buffers: this warp's rows (2 D bytes each, 16 at a time at D = 128) through shared memory, so that the global stores are whole rows: D / 8 lanes x 16 B contiguous,
                // 256 / D rows per instruction. That matters most for the peer copies, which cross NVLink.
                constexpr int kRowBytes = D * 2;
                constexpr int kChunks = D / 8;          // 16-byte chunks per row
                constexpr int kRowsAtOnce = kOutBytes / kRowBytes;
                if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");   // (an earlier tile's bulk stores)
                __syncwarp();
    #pragma unroll 1
                for (int part = 0; part < 32 / kRowsAtOnce; ++part) {
    #pragma unroll 1
                for (int c = 0; c < D / 32; ++c) {
                    float ov[32];
                    __syncwarp();   // (some lanes have written their rows)
                    tc_ld32(o_addr + c * 32, ov);
                    tc_wait_ld();
                    if (ti.n_kv == 0) {   // the tile saw no key: tensor memory holds nothing of ours, the rows are zeros
                    #pragma unroll
                        for (int i = 0; i < 32; ++i) ov[i] = 0.0f;
                    }
                    if (lane / kRowsAtOnce == part) {
                        const int rr = lane % kRowsAtOnce;
    #pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            uint4 w;
                            w.x = pack16<T>(ov[8 * i] * inv, ov[8 * i + 1] * inv);
                            w.y = pack16<T>(ov[8 * i + 2] * inv, ov[8 * i + 3] * inv);
                            w.z = pack16<T>(ov[8 * i + 4] * inv, ov[8 * i + 5] * inv);
                            w.w = pack16<T>(ov[8 * i + 6] * inv, ov[8 * i + 7] * inv);
                            const int ch = c * 4 + i;   // 16-byte chunk of the row, XOR-swizzled against bank conflicts
                            *reinterpret_cast<uint4*>(stage + rr * kRowBytes + ((ch ^ (rr & (kChunks - 1))) << 4)) = w;
                        }
                    }
                }
                __syncwarp();
                {
                    const int ch = lane & (kChunks - 1);
                    const int sub = lane / kChunks;
                    constexpr int kRowsPerStep = 32 / kChunks;
                    const int part_row0 = ti.row0 + (warp & 3) * 32 + part * kRowsAtOnce;
    #pragma unroll 4
                    for (int n = 0; n < kRowsAtOnce / kRowsPerStep; ++n) {
                        const int rr = n * kRowsPerStep + sub;
                        const int grow = part_row0 + rr;
                        if (grow < rows_end && ch * 8 < a.d_real) {
                            const uint4 w = *reinterpret_cast<const uint4*>(stage + rr * kRowBytes + ((ch ^ (rr & (kChunks - 1))) << 4));
                            const long long o_off = ((sq.o_row0 + (grow >> pl)) * a.o_heads + a.o_head0 + ti.head + (grow & ((1 << pl) - 1))) * a.d_real + ch * 8;
                            // every GPU of a group starts its walk at a different buffer (peer0 = its own
                            // index + 1), so that at no time all of them store to the same GPU
                            if (a.multicast) {
                                // one store into the multicast address: the switch writes it into every GPU's tensor
                                multimem_st16(static_cast<T*>(a.o[0]) + o_off, w);
                            } else {
                                int pe = a.peer0;
                                for (int n_pe = 0; n_pe < a.n_out; ++n_pe) {
                                    *reinterpret_cast<uint4*>(static_cast<T*>(a.o[pe]) + o_off) = w;
                                    pe = pe + 1 == a.n_out ? 0 : pe + 1;
                                }
                            }
                        }
                    }
                }
                __syncwarp();   // the rows are written again by the next part
                }
            }
            if (row_ok && (a.lse != nullptr || a.n_lse > 0)) {
                const float lse_val = seen ? (m + log2f(l)) * 0.6931471805599453f : -INFINITY;
                if (a.lse != nullptr) a.lse[((long long)b * a.q_heads + head) * a.q_seq_len + token] = lse_val;
                // head-sharded call: the same value into the (batch, o_heads, q_seq_len) LSE of every GPU of the group
                const long long g_off = ((long long)b * a.o_heads + a.o_head0 + head) * a.q_seq_len + token;
                for (int n = 0; n < a.n_lse; ++n) a.lse_peers[n][g_off] = lse_val;
            }
            FA_TRACE_EVENT(t, max(0, (int)steps - 1), 5);       // epilogue stores issued
        }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");   // shared memory stays valid until read
        if constexpr (kSplit) {
            __syncthreads();   // the products of both tiles have finished, nobody reads K or V any more
            if (sm.share.some) split_rows<T, D, kMask>(a, sm, have, t, r, warp, lane, tmem + lane_base + 256 + t * 128, last_n, last_m, last_l);
        }
    }
    if (kSplit && warp >= 8) {
        __syncthreads();           // (every role has ended: what the K producer found out is there, and the same in all CTAs of the cluster)
        if (sm.share.some) {   // the phases of split_rows, where every thread of a cluster is counted
            cluster_arrive();
            cluster_wait();
            cluster_arrive();
            cluster_wait();
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;\n" ::"r"(sm.tmem_base) : "memory");
    }
#ifdef FA_TRACE
    if (a.cta_log != nullptr && threadIdx.x == 0) {
        const int idx = blockIdx.y * gridDim.x + blockIdx.x;
        if (idx < kCtaLogEntries) {
            unsigned smid;
            asm volatile("mov.u32 %0, %%smid;\n" : "=r"(smid));
            a.cta_log[idx * 3 + 0] = (long long)ns_entry;
            a.cta_log[idx * 3 + 1] = (long long)global_timer_ns();
            a.cta_log[idx * 3 + 2] = (long long)smid;
        }
    }
#endif
}

// ---- host side ---------------------------------------------------------------------------
using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                              const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn get_encode_fn() {
    static EncodeFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, []() {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess) {
            fn = reinterpret_cast<EncodeFn>(p);
        } else {
            cudaGetLastError();
        }
    });
    return fn;
}

// (batch, seq, heads, 128) 16-bit tensor viewed as 4-D {d, head, seq, batch}; box = 64 x 1 x 128 x 1 (out: 64 x 1 x 32 x 1, what a softmax warp lays down at a time)
// seq <= 0: a packed buffer whose row count the caller did not give (batch is 1 then). The row extent is
// set beyond any buffer and the kernel never asks for a box that reaches past the real last row.
// pack: heads that share a tile, in neighbouring rows of a token: 64 x pack x 128 / pack x 1 (out: 64 x pack x 32 / pack x 1)
bool encode_map(CUtensorMap* map, const void* base, int dtype, int d, int batch, int seq, int heads, int pack = 1, bool out = false) {
    EncodeFn fn = get_encode_fn();
    if (fn == nullptr) return false;
    const bool unbounded = seq <= 0;
    const cuuint64_t rows = unbounded ? (cuuint64_t)0x7fffffff : (cuuint64_t)seq;
    const cuuint64_t dims[4] = {(cuuint64_t)d, (cuuint64_t)heads, rows, (cuuint64_t)batch};
    // the stride of the batch axis is never used when batch is 1; it only has to be a legal value
    const cuuint64_t strides[3] = {(cuuint64_t)d * 2, (cuuint64_t)heads * d * 2,
                                   unbounded ? (cuuint64_t)heads * d * 2 * 128 : (cuuint64_t)seq * heads * d * 2};
    const cuuint32_t box[4] = {64, (cuuint32_t)pack, (out ? 32u : (cuuint32_t)kBlockM) / (cuuint32_t)pack, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUtensorMapDataType dt = dtype == DT_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    const CUresult rc = fn(map, dt, 4, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return rc == CUDA_SUCCESS;
}

// Paged cache (num_blocks, block_size, heads, 128) viewed as 4-D {d, head, slot in block, block};
// box = 64 x 1 x block_size x 1: one page of one head and one 64-column half per copy. The C ABI
// does not say how many blocks the pool has, so the block extent is set far beyond any pool; only
// block ids read from the table are ever requested (and -1 for "no page": out of range, zeros).
bool encode_paged_map(CUtensorMap* map, const void* base, int dtype, int d, int block_size, int heads) {
    EncodeFn fn = get_encode_fn();
    if (fn == nullptr) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)d, (cuuint64_t)heads, (cuuint64_t)block_size, (cuuint64_t)1 << 30};
    const cuuint64_t strides[3] = {(cuuint64_t)d * 2, (cuuint64_t)heads * d * 2, (cuuint64_t)block_size * heads * d * 2};
    if (strides[2] >= ((cuuint64_t)1 << 40)) return false;
    const cuuint32_t box[4] = {64, 1, (cuuint32_t)block_size, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUtensorMapDataType dt = dtype == DT_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    const CUresult rc = fn(map, dt, 4, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return rc == CUDA_SUCCESS;
}

// Status words, one per device, in mapped pinned host memory: a kernel whose bounded wait ran out
// stores the wait's code there, and the host reads it at the next entry-point call without
// touching the device. One portable allocation for all devices, a cache line per device.
constexpr int kMaxDevices = 64;
constexpr int kStatusStride = 32;   // ints (128 bytes) between two devices' words
std::mutex g_status_mutex;
int* g_status_host = nullptr;

int* status_word() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    std::lock_guard<std::mutex> lock(g_status_mutex);
    if (g_status_host == nullptr) {
        void* p = nullptr;
        if (cudaHostAlloc(&p, sizeof(int) * kStatusStride * kMaxDevices, cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        std::memset(p, 0, sizeof(int) * kStatusStride * kMaxDevices);
        g_status_host = static_cast<int*>(p);
    }
    return g_status_host + dev * kStatusStride;
}

#ifdef FA_TRACE
// Per-device debug area in device memory: (from byte 256) the optional timeline, from byte 16384 the CTA log.
constexpr size_t kDebugBytes = 16384 + kCtaLogEntries * 24;
unsigned char* g_debug_area[kMaxDevices] = {nullptr};

unsigned char* debug_area() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    std::lock_guard<std::mutex> lock(g_status_mutex);
    if (g_debug_area[dev] == nullptr) {
        void* p = nullptr;
        if (cudaMalloc(&p, kDebugBytes) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        cudaMemset(p, 0, kDebugBytes);
        g_debug_area[dev] = static_cast<unsigned char*>(p);
    }
    return g_debug_area[dev];
}
#endif

template <typename T, int D, bool kMask, bool kPaged>
int launch_variant(const AttnParams& p, cudaStream_t stream) {
    CUtensorMap qm, km, vm, om;
    // packed varlen buffers are one "batch" of total rows
    const bool packed = p.mode == MODE_VARLEN;
    const int q_batch = packed ? 1 : p.num_seqs, q_rows = packed ? p.total_q : p.q_seq_len;
    const int k_batch = packed ? 1 : p.num_seqs, k_rows = packed ? p.total_k : p.kv_seq_len;
    // head size 32 runs on the D = 64 kernel: the maps carry the real inner extent (32), the 64-column
    // boxes read zeros past it and bulk stores write nothing there
    const int d_real = p.head_size;
    const int group = p.q_heads / p.kv_heads, pack = pack_of(group);
    bool ok = encode_map(&qm, p.q, p.dtype, d_real, q_batch, q_rows, p.q_heads, pack);
    // The output as boxes of 32 rows. Bulk stores are used for a single, local output
    // only: a head-sharded call (n_out > 0) stores every copy with plain stores, and no tensor map is
    // ever made over another GPU's memory — the kernel's fourth map is then a second one over q, unused.
    if (p.n_out > 0) om = qm;
    else ok = ok && encode_map(&om, p.o, p.dtype, d_real, q_batch, q_rows, p.q_heads, pack, true);
    if (p.paged) {
        ok = ok && encode_paged_map(&km, p.k, p.dtype, d_real, p.block_size, p.kv_heads) &&
             encode_paged_map(&vm, p.v, p.dtype, d_real, p.block_size, p.kv_heads);
    } else {
        ok = ok && encode_map(&km, p.k, p.dtype, d_real, k_batch, k_rows, p.kv_heads) &&
             encode_map(&vm, p.v, p.dtype, d_real, k_batch, k_rows, p.kv_heads);
    }
    if (!ok) return -1;  // let the SIMT kernel take it
    int* status = status_word();
    if (status == nullptr) return -1;

    PrefillArgs a{};
    if (p.n_out > 0) {
        if (p.n_out > kMaxPeers || p.n_lse > kMaxPeers) return -1;
        for (int i = 0; i < p.n_out; ++i) a.o[i] = p.o_peers[i];
        for (int i = 0; i < p.n_lse; ++i) a.lse_peers[i] = p.lse_peers[i];
        a.n_out = p.n_out;
        a.n_lse = p.n_lse;
        a.o_heads = p.o_heads;
        a.o_head0 = p.o_head0;
        // with equal shards this GPU's index in the group is o_head0 / q_heads: start one past it
        a.peer0 = (p.o_head0 / p.q_heads + 1) % p.n_out;
        a.multicast = p.multicast;
    } else {
        a.o[0] = p.o;
        a.o_by_32 = (reinterpret_cast<uintptr_t>(p.o) & 31) == 0;
        a.n_out = 1;
        a.o_heads = p.q_heads;
        a.o_head0 = 0;
    }
    a.lse = p.lse;
    a.status = status;
    a.wait_ns = get_option_prefill_wait_us() > 0 ? (unsigned long long)get_option_prefill_wait_us() * 1000ULL : kWaitLimitNs;
    a.test_skip_k = get_option_prefill_test_skip_k();
#ifdef FA_TRACE
    {
        unsigned char* dbg = get_option_prefill_trace() != 0 ? debug_area() : nullptr;
        a.staged_store = get_option_prefill_trace() == 2 ? 1 : 0;
        a.trace_y = get_option_prefill_trace_y();
        a.cta_log = (dbg != nullptr && get_option_prefill_trace() == 3) ? reinterpret_cast<long long*>(dbg + 16384) : nullptr;
        a.trace = (dbg != nullptr && get_option_prefill_trace() == 1) ? reinterpret_cast<long long*>(dbg + 256) : nullptr;
    }
#endif
    a.batch = p.num_seqs;
    a.q_seq_len = p.q_seq_len;
    a.kv_seq_len = p.kv_seq_len;
    a.q_heads = p.q_heads;
    a.kv_heads = p.kv_heads;
    a.start_pos = std::min(p.start_pos, p.kv_seq_len);   // (behind the keys there is nothing more to see)
    a.d_real = d_real;
    a.mode = p.mode;
    a.q = p.q;
    a.k = p.k;
    a.v = p.v;
    a.mask = p.mode == MODE_BATCH ? static_cast<const unsigned char*>(p.mask) : nullptr;
    a.cu_q = p.cu_q;
    a.cu_k = p.cu_k;
    a.context_lens = p.context_lens;
    a.block_tables = p.block_tables;
    a.paged = p.paged;
    a.block_size = p.block_size;
    a.max_blocks = p.max_blocks;
    a.q_bounded = p.total_q > 0;
    a.kv_bounded = p.total_k > 0;
    a.scale_log2 = p.scale * 1.4426950408889634f;

    const int packs = group / pack;
    while ((1 << a.pack_log2) < pack) ++a.pack_log2;
    const int pairs = (packs * row_blocks(p.q_seq_len, a.pack_log2) + 1) / 2;
    const size_t smem = sizeof(SharedStorage<D>) + 1024;
    const MixedFewRows few = prepare_mixed_few_rows(p, stream);   // its workspace is this call's until both kernels are launched
    a.skip_rows = few.max_rows;
    const long long kv_rows = p.mode == MODE_KVCACHE ? (long long)p.max_blocks * p.block_size : p.kv_seq_len;   // upper bound per sequence
    const long long all = (long long)p.num_seqs * p.kv_heads * pairs;
    // Where the tile pairs leave SMs without one, a cluster of 2, 4 or 8 CTAs shares the keys of each, as many as find room at the same time (one CTA to an SM; 33 clusters of four and 15
    // of eight, as the SMs lie), for a cluster of eight with four tiles for each. It takes 2 us (a few rows) to 7 (full tiles of 128 columns and eight CTAs) more, a tile 1.5. us from a graph,
    // alone and shared by 2, 4, 8: 1 x 512 tokens over 8192, 32/8 heads 108, 70; 1 x 64 over 8192 105, 64, 41, 31; 5 x 84 over 339-5439, 8 heads of 64 57, 36; 1 x 2048, 8 heads 28.7, 23.6; 2 x 64 over
    // 30000, 32/8 heads of 64 354, 192, 103, 115 (16 clusters of eight, in two rounds); 8 x 1 token over 1022, 8/2 heads 15.0, 12.6, 9.8; 4 x 1 over 544, 32/8 heads of 64 10.0, 9.8.
    // More than a few rows over at most 12 tiles stay alone: their results have the bits of the same rows in a call that fills the device. So do a few rows where there may be no more than 12 (over
    // pages, whose lengths the host does not know: 2 x 6 over 361 with room for 1024, 32 heads 13.0 alone, 14.8 as a cluster that finds too few to share) or are no more than 7 tiles.
    const int parts = p.n_out > 0 || a.skip_rows > 0 ? 1 : prefill_parts(all, (kv_rows + kBlockN - 1) / kBlockN, p.mode == MODE_BATCH, (long long)p.q_seq_len * group, sm_count());
    a.parts = parts;
    // Band width: the pairs of a band start together, so their work must be about equal or the
    // heaviest-first order is lost (at S = 2048 without GQA, bands of 2 cost 13 %). A band of w
    // pairs spans 2w / group row blocks, i.e. that many K/V tiles of difference between its lightest
    // and heaviest pair: keep that within an eighth of the longest K/V range, at most 8 pairs (16 measured no better). Clusters all run at the same time, and a band that the pairs do not fill would be clusters without
    // any, for which there may be no room (3 x 65 tokens over 640, 64/8 heads, 72 clusters of two for the 3 pairs of each KV head: with bands of two another 24 17.8 us, a CTA to a pair 14.6).
    const int band = get_option_prefill_band() > 0 ? std::min(get_option_prefill_band(), pairs) : prefill_band(pairs, std::max(1LL, (kv_rows + kBlockN - 1) / kBlockN), group, parts);
    a.band = band;
    a.by_band = FastDiv(band);
    a.by_kv_heads = FastDiv(p.kv_heads);
    a.by_packs = FastDiv(packs);
    // Head-sharded call (every CTA ends with stores to the other GPUs): heaviest-first makes the SMs end
    // their CTAs in waves, each wave a burst on the links that stalls every SM in it. A first wave that
    // mixes all weights staggers the SMs for the rest of the launch; the rest stays heaviest first, which
    // keeps the tail balanced.
    {
        const int rows = (pairs + band - 1) / band;
        const int per_row = p.kv_heads * p.num_seqs * band;
        const int w = (sm_count() + per_row - 1) / per_row;
        const int m = w > 0 ? rows / w : 0;
        const bool spread = p.n_out > 1 && get_option_prefill_order() != 1 && m >= 2;
        a.spread_w = spread ? w : 0;
        a.spread_m = spread ? m : 0;
    }
    if ((long long)p.kv_heads * p.num_seqs * band > 0x7fffffffLL) return -1;
    // Groups of K/V streams (blockIdx.z). Every tile pair of a (batch, KV head) stream re-reads the stream's
    // K/V prefix; with many streams and no sharing inside a launch band the prefixes in flight exceed L2 and
    // come from HBM again (B=4, H=32, S=2048: 523 MB read for 201 MB of q, k and v). Running the streams in
    // groups of about 16 MiB of K/V keeps the re-reads in L2 (the same launch: 201 MB read, 823 -> 851-871
    // TFLOP/s; 4 groups 843, 12-32 groups 810-834); within a group the order is unchanged.
    int groups = 1;
    {
        const long long streams = (long long)p.kv_heads * p.num_seqs;
        const long long kv_bytes_per_stream = 2LL * (p.mode == MODE_KVCACHE ? (long long)p.max_blocks * p.block_size : p.kv_seq_len) * D * 2;
        const long long budget = 16LL << 20;
        if (get_option_prefill_groups() > 0) groups = get_option_prefill_groups();
        else if (parts == 1 && band == 1 && pairs > 1 && p.n_out <= 1 && streams * kv_bytes_per_stream > 2 * budget)
            groups = (int)std::min<long long>(streams, (streams * kv_bytes_per_stream + budget - 1) / budget);
        else if (band > 1 && p.n_out <= 1 && (p.mode == MODE_BATCH || p.mode == MODE_VARLEN) && p.num_seqs >= 2 &&
                 streams * kv_bytes_per_stream > (48LL << 20) * (p.mode == MODE_VARLEN ? 2 : 1)) {
            // GQA launches share K/V inside a band already; running whole batch elements (sequences) one after
            // the other, about 48 MiB of K/V at a time, still keeps more of q, k, v and o in L2 and with it
            // power for the tensor pipe: B=2, Hq=32, Hkv=8, S=8192 1235-1237 against 1223-1225 TFLOP/s; 32 packed
            // prompts of 1024-8192 tokens 1015-1075 against 989-993 (12 to 20 groups). A packed call gives only
            // the longest sequence: the others are taken as half as long on average.
            const long long per_elem = (long long)p.kv_heads * kv_bytes_per_stream / (p.mode == MODE_VARLEN ? 2 : 1);
            const long long elems = std::max<long long>(1, (48LL << 20) / per_elem);
            groups = (int)((p.num_seqs + elems - 1) / elems);
        }
        if (groups > 65535) groups = 65535;
        if (groups < 1) groups = 1;
    }
    const int streams_per_group = (int)(((long long)p.kv_heads * p.num_seqs + groups - 1) / groups);
    a.streams_z = streams_per_group;
    dim3 grid(streams_per_group * band, (pairs + band - 1) / band, groups);
    a.pairs = pairs;
    // Ordered: chunks of prompts, at most half as long as the context may be. Whole prompts keep grid order, which is heaviest
    // first for them already. Finding its pair costs a CTA 1 to 2 us; what it wins is one late long pair, about a fifth of the longest pair's
    // 1.5 to 1.7 us per K/V tile, and nothing where all pairs start at once. So: more than one wave of pairs, and at least five tiles in the longest for
    // each. 4 chunks of 300 over 2048-8192 keys (the longest last), 32/8 heads (1.3 waves) 138-152 us in grid order, 110 ordered; 16 chunks of 300 over
    // 512-2048, 32/32 heads (7 waves) 161-172 and 166-186; 4 chunks of 64 over 128-512 (less than a wave) 17-19 and 19-21.
    const PackedMix mix = packed_mix(p);
    const long long few_pairs = (packs + 1) / 2;   // of a sequence whose rows fit one block
    const double waves = (double)(mix.prompts * pairs + (a.skip_rows > 0 ? 0 : mix.few * few_pairs)) * p.kv_heads / sm_count();
    long long ctas = all;
    if (p.total_q > 0)   // a sequence of n tokens has (packs * ceil(n * pack / 128) + 1) / 2 pairs
        ctas = std::min(ctas, p.kv_heads * ((packs * (((long long)p.total_q * pack + 127LL * p.num_seqs) / 128) + p.num_seqs) / 2));
    // ... and where most of the grid would be empty CTAs of sequences that are left to the few-row kernel: a launch in order has no more than
    // the rows can make (one chunk of 512 with 128 tokens over 128-2048, 32/8 heads: 8256 CTAs or 2644, 191 us or 153).
    const bool worth_ordering = (waves > 1.0 && (double)((kv_rows + kBlockN - 1) / kBlockN) > 5.0 * waves) || (a.skip_rows > 0 && all > 2 * ctas);
    if (kPaged && p.num_seqs >= 2 && p.num_seqs <= kOrderMax && 2LL * p.q_seq_len <= kv_rows && get_option_prefill_band() <= 0 &&
        get_option_prefill_groups() <= 0 && (worth_ordering || get_option_prefill_order() == 2)) {
        a.ordered = 1;
        if (ctas <= 0 || ctas > 0x7fffffffLL) return -1;
        grid = dim3((unsigned)ctas);
    }
    // Where the grid has no more CTAs than the device has SMs there is no pair to take over, and such a call runs without the loop over pairs, whose counters and cases cost the
    // step (up to 2 %) and, over pages, the producers' registers. us with the loop and without, from a graph: 1 x 658, 32/8 heads 15.2 and 14.9; 2 x 433 MHA 11.4 and
    // 10.9; 1 x 4096, 4/4 heads 52.2 and 51.2; 3 x 5 tokens over 46-747 18.7 and 17.7; 16 x 64 tokens over 1024-8192, 8/8 heads 104 and 101.6. Not asking for a pair alone, in the same
    // code, gave 0.1 us. Nor has a call in order much to take over: a CTA that has asked starts a pair about 2 us later, and those that start by themselves take
    // the next one just as well (4 chunks of 512 over 1024-8192 140 and 138, 4 of 300 over 2048-8192 124.8 and 123.4, 8 of 512 246 and 247). With few-row sequences left out
    // a grid in order has empty CTAs, which are cheaper to take over (serve steps of 4 chunks with 32 tokens 226 and 228, 6 with 40 310 and 318), and so are short pairs at head size
    // 64 (8 x 200 over 512-4096, 32/8 heads 68.5 and 69.6). Contiguous K/V at head size 64: no difference (1 x 449, 64/8 heads of 32 11.6 either way; 1 x 2048, 8/8 heads 26.8 and
    // 27.3), and none is built.
    if (parts > 1) {
        const auto kernel = prefill_tcgen05_kernel<T, D, kMask, kPaged, true, true>;
        cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (err == cudaSuccess) {
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(grid.x * (unsigned)parts, grid.y, grid.z);
            cfg.blockDim = dim3(kThreads);
            cfg.dynamicSmemBytes = smem;
            cfg.stream = stream;
            cudaLaunchAttribute attr{};
            attr.id = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim.x = (unsigned)parts;
            attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
            cfg.attrs = &attr;
            cfg.numAttrs = 1;
            cudaLaunchKernelEx(&cfg, kernel, qm, km, vm, om, a);
        }
        if (err != cudaSuccess) {
            set_last_errorf("prefill_tcgen05_kernel: %s", cudaGetErrorString(err));
            cudaGetLastError();
            return FLASH_ATTN_ERR_CUDA;
        }
        const int rc = check_launch("prefill_tcgen05_kernel");
        if (rc == FLASH_ATTN_OK) note_path("prefill_tcgen05", 1, parts == 8 ? "cluster 8" : parts == 4 ? "cluster 4" : "cluster 2");
        return rc;
    }
    constexpr bool kOneWave = D == 128 || kPaged;
    const bool one_pair = kOneWave && !(few.plan.wide && a.skip_rows > 0) && ((long long)grid.x * grid.y * grid.z <= sm_count() || (D == 128 && a.ordered && a.skip_rows == 0));
    const auto kernel = one_pair ? prefill_tcgen05_kernel<T, D, kMask, kPaged, kOneWave, false> : prefill_tcgen05_kernel<T, D, kMask, kPaged, false, false>;
    const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) {
        set_last_errorf("prefill_tcgen05_kernel: %s", cudaGetErrorString(err));
        cudaGetLastError();
        return FLASH_ATTN_ERR_CUDA;
    }
    a.behind_few = a.skip_rows > 0 && few.plan.wide;
    int rc = a.behind_few ? launch_mixed_few_rows(p, few, stream) : FLASH_ATTN_OK;
    if (rc != FLASH_ATTN_OK) return rc;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = a.behind_few ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, qm, km, vm, om, a);
    rc = check_launch("prefill_tcgen05_kernel");
    if (rc == FLASH_ATTN_OK && a.skip_rows > 0 && !a.behind_few) rc = launch_mixed_few_rows(p, few, stream);
    if (rc == FLASH_ATTN_OK) note_path("prefill_tcgen05", a.skip_rows > 0 ? 2 : 1, a.behind_few ? "few rows ahead" : a.skip_rows > 0 ? "few rows behind" : one_pair ? "one pair" : "pairs");
    return rc;
}

template <typename T, int D>
int launch_typed(const AttnParams& p, cudaStream_t stream) {
    if (p.mask != nullptr) return launch_variant<T, D, true, false>(p, stream);
    return p.paged ? launch_variant<T, D, false, true>(p, stream) : launch_variant<T, D, false, false>(p, stream);
}

}  // namespace

int* prefill_status_word() { return status_word(); }

int prefill_take_status() {
    int* status = status_word();
    if (status == nullptr) return 0;
    volatile int* w = status;
    const int h = *w;
    if (h != 0) *w = 0;
    return h;
}

int prefill_device_status() {
    int* status = status_word();
    if (status == nullptr) return -1;
    if (cudaDeviceSynchronize() != cudaSuccess) {
        cudaGetLastError();
        return -1;
    }
    return prefill_take_status();
}

int prefill_debug_read(void* dst, int bytes) {
#ifdef FA_TRACE
    unsigned char* dbg = debug_area();
    int* status = status_word();
    if (dbg == nullptr || status == nullptr || dst == nullptr || bytes <= 0) return -1;
    const size_t n = (size_t)bytes < kDebugBytes ? (size_t)bytes : kDebugBytes;
    if (cudaMemcpy(dst, dbg, n, cudaMemcpyDeviceToHost) != cudaSuccess) {
        cudaGetLastError();
        return -1;
    }
    if (n >= sizeof(int)) std::memcpy(dst, status, sizeof(int));
    return (int)n;
#else
    (void)dst;
    (void)bytes;
    return -1;   // the timeline is compiled in with -DFA_TRACE only
#endif
}

int launch_prefill_tcgen05(const AttnParams& p, cudaStream_t stream) {
    // batched entry point, chunked prefill over a paged cache (whole pages must tile the 128-key
    // K/V tile), and the packed varlen entry point. The reference's varlen signature does not say how
    // many rows the packed buffers have: their tensor maps then carry no row bound, and the kernel
    // fetches the tiles at the very end of the buffers with plain loads (edge_tile_copy).
    if (p.mask != nullptr && p.mode != MODE_BATCH) return -1;
    if (p.mode == MODE_KVCACHE) {
        if (!p.paged || p.max_blocks <= 0) return -1;
    } else if (p.mode == MODE_VARLEN) {
        if (p.paged && p.max_blocks <= 0) return -1;
    } else if (p.mode != MODE_BATCH) {
        return -1;
    }
    if (p.paged && (p.block_size < 8 || p.block_size > 128 || (128 % p.block_size) != 0)) return -1;
    if (p.dtype != DT_F16 && p.dtype != DT_BF16) return -1;
    if (p.head_size != 32 && p.head_size != 64 && p.head_size != 128) return -1;
    if (!(p.scale > 0.0f)) return -1;
    // (the dispatcher tries the split-K kernel first: single-token calls of the kv-cache entry point never get here, other calls
    // with few query rows where this kernel is the faster one for them)
    uintptr_t align = reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k) |
                      reinterpret_cast<uintptr_t>(p.v) | reinterpret_cast<uintptr_t>(p.o);
    for (int i = 0; i < p.n_out && i < 8; ++i) align |= reinterpret_cast<uintptr_t>(p.o_peers[i]);
    if (align & 15) return -1;
    if (prefill_pairs(p.q_heads / p.kv_heads, p.q_seq_len) > 65535) return -1;
    if (p.head_size == 64 || p.head_size == 32) return p.dtype == DT_BF16 ? launch_typed<__nv_bfloat16, 64>(p, stream) : launch_typed<__half, 64>(p, stream);
    return p.dtype == DT_BF16 ? launch_typed<__nv_bfloat16, 128>(p, stream) : launch_typed<__half, 128>(p, stream);
}

}  // namespace fa
