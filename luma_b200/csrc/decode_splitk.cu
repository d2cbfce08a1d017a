// Attention of a few query rows per sequence over a long K/V range, f16/bf16 storage, head_size 32, 64 or 128:
// single-token decode over the paged cache above all, and also a handful of speculated tokens, decoding over
// contiguous K/V, and the decoding sequences of a packed mixed batch.
//
// Replaces flash_attn_decode_kernel (luma-flash-attn/kernels/flash_attn_with_kvcache.cu:22-116;
// launch :123-145), which walks the context one token at a time with one warp per query head and
// re-reads K/V once per query head of a GQA group.
//
// Here the path is HBM-bound by construction:
//   * the query rows that share a KV head (every head of the GQA group x every query token) are the rows of
//     one tensor-core tile: a CTA reads each K/V row once and serves all of them, 16 rows at a time;
//   * the K/V ranges of all sequences are laid end to end in units of 64 tokens and cut into equal
//     shares, one per CTA slot of the device ("columns"; every KV head has its own CTA per column): all CTAs do
//     the same number of units whatever the lengths are, and each reads its share through one copy pipeline
//     that runs on across the sequence boundaries. The host knows only the width of the block table, so the
//     cut is made on the device, by every warp for itself, from the lengths;
//   * rows are gathered through the block table with 16-byte cp.async copies into a per-warp ring
//     of shared-memory stages (3 tiles of 16 tokens in flight per warp, 2 CTAs per SM), no
//     CTA-wide barrier inside a sequence;
//   * Q.K^T and P.V run on tensor cores (mma.sync m16n8k16, f32 accumulate) — at 8 query heads per KV
//     head scalar FMA could not keep up with the memory system;
//   * a sequence that lies inside one column is finished there; one that is cut leaves unnormalised f32
//     partials (acc, m, l) in a workspace, and the CTA that finishes its part last merges them, always in
//     column order, with log-sum-exp weights.
// Token -> slot arithmetic is that of block_slot() in common.cuh (reference: kernels/common.cuh:89-108).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <mutex>
#include <type_traits>

#include "common.cuh"

namespace fa {

namespace {

constexpr int kFour = 4;     // warps of a CTA (kWarps below)
constexpr int kWide = 8;     // ... of a launch that has part of the SMs to itself, one CTA to each (see prepare_mixed_few_rows)
constexpr int kTile = 16;    // tokens per tile (one mma K step for P.V, two N blocks for Q.K^T)
template <int kWarps> constexpr int unit_of = kWarps * kTile;   // tokens that the CTA's warps take at a time, the unit of the cut
constexpr int kStages = 3;   // tiles in flight per warp
constexpr int kRows = 16;    // query rows served per CTA (M of the mma)

// Where the finished rows go: one buffer of (rows, o_heads, D), or — head-sharded decode with
// the output all-gather fused in — the same tensor on every GPU of the group (peer memory, plain
// stores over NVLink), each receiving this call's heads at head offset o_head0.
struct RowsOut {
    void* o[8];
    int n_out, o_heads, o_head0, peer0;
    int halves;      // a buffer is aligned to its 2-byte elements only: rows are stored element by element
    float* lse;      // MODE_BATCH: (num_seqs, q_heads, q_seq_len) or null
};

constexpr int kMaxColumns = 65535;
constexpr int kCountBits = 20;   // of an arrival counter; the number of the call is above

struct RowsArgs {
    const void* q;
    const void* k;
    const void* v;
    const int* block_tables;
    const int* context_lens;   // MODE_KVCACHE
    const int* cu_q;           // MODE_VARLEN
    const int* cu_k;           // MODE_VARLEN
    float* ws_acc;       // (2 * CTAs, kRows, D) f32, unnormalised; slot 0 of a CTA: the sequence that began in an earlier column, slot 1: the one that goes on in the next
    float2* ws_ml;       // (2 * CTAs, kRows) {m (log2 domain), l}
    unsigned long long* arrived;   // (gridDim.x, num_seqs): `call` + the parts of a cut sequence that are in the workspace; zero between calls
    unsigned long long call;       // number of this call, in the bits above the count
    int mode, num_seqs, q_seq_len, kv_seq_len, start_pos;
    int q_heads, kv_heads, block_size, block_shift, max_blocks, paged;   // block_shift: log2 of the page size, -1 where it is no power of two
    int row_blocks;      // blocks of kRows query rows per KV head (blockIdx.x = KV head x row block)
    int capacity;        // keys that a sequence's row of the block table has room for; contiguous K/V: no limit
    int max_rows;        // sequences with more query rows than this (per KV head) are not this launch's
    int behind_prefill;  // launched behind the prefill kernel of the same call, which it does not depend on
    int forced_units;    // > 0: units per column (option "decode_chunk_tokens"); 0: equal shares
    int seq_cost;        // of a sequence, in units, beside its own units (see rows_span)
    float scale_log2;    // scale * log2(e)
    RowsOut out;
};

__device__ __forceinline__ void cp_async_16(void* smem, const void* gmem, bool valid) {
    const unsigned saddr = (unsigned)__cvta_generic_to_shared(smem);
    const int src_bytes = valid ? 16 : 0;  // 0 -> the 16 destination bytes are zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(saddr), "l"(gmem), "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

__device__ __forceinline__ void ldmatrix_x4(unsigned& r0, unsigned& r1, unsigned& r2, unsigned& r3,
                                            const void* smem) {
    const unsigned saddr = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(saddr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(unsigned& r0, unsigned& r1, unsigned& r2, unsigned& r3,
                                                  const void* smem) {
    const unsigned saddr = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(saddr));
}

template <typename T>
__device__ __forceinline__ void mma_16816(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1);
template <>
__device__ __forceinline__ void mma_16816<__nv_bfloat16>(float (&d)[4], const unsigned (&a)[4], unsigned b0,
                                                         unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void mma_16816<__half>(float (&d)[4], const unsigned (&a)[4], unsigned b0,
                                                  unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <typename T>
__device__ __forceinline__ unsigned pack2(float lo, float hi);
template <>
__device__ __forceinline__ unsigned pack2<__nv_bfloat16>(float lo, float hi) {
    __nv_bfloat162 t = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<unsigned*>(&t);
}
template <>
__device__ __forceinline__ unsigned pack2<__half>(float lo, float hi) {
    __half2 t = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<unsigned*>(&t);
}

__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}

// Shared memory of one CTA:
//   ring : kWarps x kStages x {K tile, V tile}, each tile kTile rows of D elements, 16-byte chunks
//          XOR-swizzled by the row (row & 7; row & 3 at head_size 32, whose rows hold only four chunks) against
//          ldmatrix bank conflicts
//   merge: the warps' partials of a finished sequence, up to 8 rows whole or 16 rows kMergeCols columns at a time — beside
//          the ring, which already holds tiles of the next sequence by then
template <int D, int kWarps>
struct Smem {
    static constexpr int kRowBytes = D * 2;
    static constexpr int kSwz = (D / 8 - 1) < 7 ? (D / 8 - 1) : 7;   // XOR mask of the 16-byte chunk index: stays inside the row
    static constexpr int kTileBytes = kTile * kRowBytes;
    static constexpr int kStageBytes = 2 * kTileBytes;
    static constexpr int kWarpBytes = kStages * kStageBytes;
    static constexpr int kRingBytes = kWarps * kWarpBytes;
    static constexpr int kMergeCols = D < 64 ? D : 64;
    static constexpr int kMergePitch = kMergeCols + 2;   // the row's m and l in the last two
    static constexpr int kMergeBytes = kWarps * kRows * kMergePitch * 4;
    static constexpr int kBytes = kRingBytes + kMergeBytes + 16;
    // CTAs per SM by shared memory (228 KiB, 1 KiB of it reserved per CTA) and registers
    static constexpr int kCtasPerSm = kWarps == kWide ? 1 : D == 128 ? 2 : (D == 64 ? 3 : 4);
    static_assert(kBytes <= 232448, "fits the shared memory of an SM");
};

// Extents of one sequence: its query rows and the keys it sees. Query token i sits at global position
// pos_off + i and sees keys j < kv_len with j <= pos_off + i; of a length beyond what the block table holds, kv_len is the part
// that it holds.
struct RowsSeq {
    int q_len, kv_len, pos_off;
    long long q_row0, kv_row0;
};

template <int kMode>
__device__ __forceinline__ RowsSeq rows_seq(const RowsArgs& a, int s) {
    RowsSeq r;
    if (kMode == MODE_KVCACHE) {
        r.q_len = a.q_seq_len;
        const int len = a.context_lens[s];
        r.kv_len = min(len, a.capacity);
        r.pos_off = len - r.q_len;
        r.q_row0 = (long long)s * a.q_seq_len;
        r.kv_row0 = 0;
    } else if (kMode == MODE_BATCH) {
        r.q_len = a.q_seq_len;
        r.kv_len = a.kv_seq_len;
        r.pos_off = a.start_pos;
        r.q_row0 = (long long)s * a.q_seq_len;
        r.kv_row0 = (long long)s * a.kv_seq_len;
    } else {
        const int q0 = a.cu_q[s], k0 = a.cu_k[s];
        r.q_len = a.cu_q[s + 1] - q0;
        const int len = a.cu_k[s + 1] - k0;
        r.kv_len = min(len, a.capacity);
        r.pos_off = len - r.q_len;
        r.q_row0 = q0;
        r.kv_row0 = k0;
    }
    return r;
}

// Keys that the last query token sees.
__device__ __forceinline__ int rows_visible(const RowsSeq& r) {
    const long long v = min((long long)r.kv_len, (long long)r.pos_off + r.q_len);
    return v > 0 ? (int)v : 0;
}

// Units of the sequence for the row block that starts at query row `row0`; 0: nothing to do there. A sequence
// whose rows see no key has one unit all the same: somebody has to write its zeros.
template <int kWarps>
__device__ __forceinline__ int rows_units(const RowsArgs& a, const RowsSeq& r, int group, int row0) {
    constexpr int kUnit = unit_of<kWarps>;
    const int rows = r.q_len * group;
    if (rows <= row0 || rows > a.max_rows) return 0;
    return max(1, (rows_visible(r) + kUnit - 1) / kUnit);
}

// One arrival; returns how many came before it. Everything the CTA's threads wrote before their last barrier is visible to
// whoever sees the count (release), and what earlier arrivals published is visible to this CTA after its next barrier (acquire).
// Whatever an earlier call left there (calls that overlapped on one buffer, which spoils their results, leave counts that are
// not zero) is below this call's number and does not count: the maximum lifts it, ahead of the addition to the same word,
// and costs no trip of its own, as nothing waits for it.
__device__ __forceinline__ unsigned long long arrive_acq_rel(unsigned long long* count, unsigned long long call) {
    unsigned long long before;
    asm volatile("red.relaxed.gpu.global.max.u64 [%0], %1;\n" ::"l"(count), "l"(call) : "memory");
    asm volatile("atom.add.acq_rel.gpu.global.u64 %0, [%1], 1;\n" : "=l"(before) : "l"(count) : "memory");
    return before - call;
}

// Two finished neighbours of an output row, to every output buffer.
template <typename T>
__device__ __forceinline__ void store_pair(const RowsOut& out, long long row, int head, int D, int d, unsigned both) {
    const long long off = (row * out.o_heads + out.o_head0 + head) * D + d;
    int pe = out.peer0;
    for (int n = 0; n < out.n_out; ++n) {
        T* const at = static_cast<T*>(out.o[pe]) + off;
        if (out.halves) {
            reinterpret_cast<unsigned short*>(at)[0] = (unsigned short)both;
            reinterpret_cast<unsigned short*>(at)[1] = (unsigned short)(both >> 16);
        } else {
            *reinterpret_cast<unsigned*>(at) = both;
        }
        pe = pe + 1 == out.n_out ? 0 : pe + 1;
    }
}

// Merges the parts of a cut sequence: warp w takes rows w, w + 4, ..., RW of them, a lane D / 32 neighbouring
// elements of each. The CTA runs alone at the end of its column here, so what counts is the number of dependent
// trips to L2 (about 0.6 us each) and of instructions, which come in for the first time: the first partials are asked for together with every part's (m, l), in all 16 rows of
// partials in flight per lane, and where a row goes is found by one lane and told to the others. With the partials asked for behind the weights, and
// every lane finding each row's place, a merge of 13 parts of 4 rows took 2.1 us, of 2-5 parts of 16 rows 6 to 8 us, of which 0.65 and 3 to 5 behind the sums (device timer); 16 sequences
// x 4 tokens over 512-8192 64.4 us a step, 8 x 4000 contiguous 28.7, one of 777 tokens 9.1.
template <typename T, int D, int RW, int kWarps>
__device__ __forceinline__ void merge_parts(const RowsArgs& a, float* scratch, long long q_row0, int s, int kvh, int row0, int group, int nrows, int c_first, int parts, int warp, int lane) {
    constexpr int E = D / 32;
    constexpr int kAtOnce = 16 / RW;      // parts in flight per row
    constexpr int kChunk = 64;            // parts whose weights sit in shared memory at a time
    static_assert(kRows / 2 * (D + 2) <= kRows * Smem<D, kWarps>::kMergePitch, "half of the rows fit the merge buffer whole");
    static_assert(kRows * kChunk * 4 <= Smem<D, kWarps>::kMergeBytes, "weights of a chunk fit the merge buffer");
    const unsigned grid_x = gridDim.x;
    const float* const acc0 = a.ws_acc + ((long long)blockIdx.x * (2 * kRows) + warp) * D + lane * E;   // of this warp's first row, slot 0 of column 0
    const float2* const ml0 = a.ws_ml + (long long)blockIdx.x * (2 * kRows) + warp;
    auto slot_of = [&](int c) { return (unsigned)c * grid_x * 2u + (c == c_first ? 1u : 0u); };   // (fits: the workspace has 2 kRows D floats for each)
    float o[RW][E], m[RW], l[RW];
#pragma unroll
    for (int k = 0; k < RW; ++k) {
        m[k] = -INFINITY;
        l[k] = 0.0f;
#pragma unroll
        for (int e = 0; e < E; ++e) o[k][e] = 0.0f;
    }
#pragma unroll 1
    for (int p0 = 0; p0 < parts; p0 += kChunk) {
        const int n = min(kChunk, parts - p0);
        float x[RW][kAtOnce][E];
        auto ask = [&](int i0) {
#pragma unroll
            for (int i = 0; i < kAtOnce; ++i) {
                const float* const part = acc0 + (unsigned long long)slot_of(c_first + p0 + i0 + i) * (kRows * D);
#pragma unroll
                for (int k = 0; k < RW; ++k) {
#pragma unroll
                    for (int e = 0; e < E; ++e) x[k][i][e] = 0.0f;
                    if (warp + k * kWarps < nrows && i0 + i < n) {
                        const float* const src = part + k * kWarps * D;
                        if constexpr (E == 4) {
                            const float4 y = __ldcg(reinterpret_cast<const float4*>(src));
                            x[k][i][0] = y.x; x[k][i][1] = y.y; x[k][i][2] = y.z; x[k][i][3] = y.w;
                        } else if constexpr (E == 2) {
                            const float2 y = __ldcg(reinterpret_cast<const float2*>(src));
                            x[k][i][0] = y.x; x[k][i][1] = y.y;
                        } else {
                            x[k][i][0] = __ldcg(src);
                        }
                    }
                }
            }
        };
        float2 y[RW][2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float2* const part = ml0 + (unsigned long long)slot_of(c_first + p0 + h * 32 + lane) * kRows;
#pragma unroll
            for (int k = 0; k < RW; ++k) {
                y[k][h] = make_float2(-INFINITY, 0.0f);
                if (warp + k * kWarps < nrows && h * 32 + lane < n) y[k][h] = __ldcg(part + k * kWarps);
            }
        }
        ask(0);
#pragma unroll
        for (int k = 0; k < RW; ++k) {
            float mx = fmaxf(y[k][0].x, y[k][1].x);
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
            mx = fmaxf(mx, m[k]);
            const float before = m[k] == -INFINITY ? 0.0f : fast_exp2(m[k] - mx);
            m[k] = mx;
            l[k] *= before;
#pragma unroll
            for (int e = 0; e < E; ++e) o[k][e] *= before;
            const float w0 = y[k][0].x == -INFINITY ? 0.0f : fast_exp2(y[k][0].x - mx);
            const float w1 = y[k][1].x == -INFINITY ? 0.0f : fast_exp2(y[k][1].x - mx);
            scratch[(k * kWarps + warp) * kChunk + lane] = w0;
            scratch[(k * kWarps + warp) * kChunk + 32 + lane] = w1;
            l[k] += w0 * y[k][0].y + w1 * y[k][1].y;   // this lane's share
        }
        __syncwarp();
#pragma unroll 1
        for (int i0 = 0;;) {
#pragma unroll
            for (int i = 0; i < kAtOnce; ++i)
#pragma unroll
                for (int k = 0; k < RW; ++k) {
                    const float w = scratch[(k * kWarps + warp) * kChunk + min(i0 + i, n - 1)];
#pragma unroll
                    for (int e = 0; e < E; ++e) o[k][e] = fmaf(w, x[k][i][e], o[k][e]);
                }
            i0 += kAtOnce;
            if (i0 >= n) break;
            ask(i0);
        }
        __syncwarp();
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int k = 0; k < RW; ++k) l[k] += __shfl_xor_sync(0xffffffffu, l[k], off);
    // lane k, k + RW, ... : row k's place, maximum and sum
    const int mine = lane & (RW - 1), r = warp + mine * kWarps, t = (row0 + r) / group, h = kvh * group + (row0 + r) - t * group;
    const long long at = ((q_row0 + t) * a.out.o_heads + a.out.o_head0 + h) * D;
    float m1 = m[0], l1 = l[0];
#pragma unroll
    for (int k = 1; k < RW; ++k)
        if (mine == k) {
            m1 = m[k];
            l1 = l[k];
        }
    const float inv1 = l1 > 0.0f ? 1.0f / l1 : 0.0f;
    if (a.out.lse != nullptr && lane < RW && r < nrows)
        a.out.lse[((long long)s * a.q_heads + h) * a.q_seq_len + t] = l1 > 0.0f ? (m1 + log2f(l1)) * 0.6931471805599453f : -INFINITY;
    unsigned both[RW][(E + 1) / 2];
    long long to[RW];
#pragma unroll
    for (int k = 0; k < RW; ++k) {
        const float inv = __shfl_sync(0xffffffffu, inv1, k);
        to[k] = __shfl_sync(0xffffffffu, at, k) + lane * E;
        if constexpr (E >= 2) {
#pragma unroll
            for (int e = 0; e < E; e += 2) both[k][e / 2] = pack2<T>(o[k][e] * inv, o[k][e + 1] * inv);
        } else {
            const float up = __shfl_down_sync(0xffffffffu, o[k][0], 1);
            both[k][0] = pack2<T>(o[k][0] * inv, up * inv);   // (even lanes')
        }
    }
    int pe = a.out.peer0;
#pragma unroll 1
    for (int n = 0; n < a.out.n_out; ++n) {
        T* const base = static_cast<T*>(a.out.o[pe]);
#pragma unroll
        for (int k = 0; k < RW; ++k) {
            if (warp + k * kWarps >= nrows || (E == 1 && (lane & 1) != 0)) continue;
#pragma unroll
            for (int e = 0; e < (E + 1) / 2; ++e) {
                if (a.out.halves) {
                    reinterpret_cast<unsigned short*>(base + to[k])[2 * e] = (unsigned short)both[k][e];
                    reinterpret_cast<unsigned short*>(base + to[k])[2 * e + 1] = (unsigned short)(both[k][e] >> 16);
                } else {
                    reinterpret_cast<unsigned*>(base + to[k])[e] = both[k][e];
                }
            }
        }
        pe = pe + 1 == a.out.n_out ? 0 : pe + 1;
    }
}

// kMode: the entry point. With the three of them behind branches, every place that looks at a sequence had
// the code of all three, which a small call brings in for the first time (1 x 777 tokens 8.7 us a step, 8.3 so; 2 x 62-250, 32 heads 10.1 and 9.1).
template <typename T, int D, int kMode, int kWarps>
__global__ void __launch_bounds__(kWarps * 32, Smem<D, kWarps>::kCtasPerSm) decode_splitk_kernel(const __grid_constant__ RowsArgs a) {
    using S = Smem<D, kWarps>;
    constexpr int kThreads = kWarps * 32, kUnit = unit_of<kWarps>;
    constexpr int kChunksPerRow = D / 8;          // 16-byte chunks per K/V row
    constexpr int kCopiesPerLane = kChunksPerRow / 2;  // a lane copies half a row of K and of V
    constexpr int kKSteps = D / 16;
    constexpr int kDBlocks = D / 8;
    extern __shared__ __align__(128) unsigned char smem_raw[];

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2;   // mma row group
    const int c4 = lane & 3;

    // Launched with programmatic stream serialisation: the grid may be set up while the kernel before it
    // drains, and touches nothing in global memory before that kernel has finished (returns at once
    // when the launch carries no programmatic dependency). The next kernel may be set up likewise.
    // Behind a prefill kernel (packed mixed batch) it starts when that kernel's last CTAs have started and fills
    // the SMs that they leave: what both read was written before the prefill kernel began. Every CTA then waits at
    // its end instead, so that this grid's completion stands for both.
    const bool behind = a.behind_prefill != 0;
    // Ahead of a prefill kernel of the same call, which does not wait for this one but for what came before both: that has finished when it may start.
    // (Known at compile time, or every launch waits for its first load before it lets the next one begin: one of 777 tokens, 32/8 heads 7.4 us from a graph, 7.65 with a flag of the launch's.)
    constexpr bool ahead = kWarps == kWide;
    if (!ahead) asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    if (!behind) asm volatile("griddepcontrol.wait;\n" ::: "memory");
    if (ahead) asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");

    // KV heads vary fastest across the grid: the CTAs that read the adjacent 256-byte slices of the
    // same token rows (one slice per KV head) are launched together, which keeps DRAM pages open.
    const int kvh = blockIdx.x / a.row_blocks;
    const int row0 = (blockIdx.x - kvh * a.row_blocks) * kRows;   // first query row of this CTA (row = token x group + head in group)
    const int column = blockIdx.y;
    int columns = gridDim.y;
    const int group = a.q_heads / a.kv_heads;

    // The cut: total units, this column's share of them, and the sequence its first unit lies in.
    unsigned total = 0, seq_first = 0;   // seq_first: unit at which sequence `s` begins
    int s = 0, cost = 0;
    unsigned u_begin, u_end;
    if (kMode == MODE_BATCH) {
        const int units = rows_units<kWarps>(a, rows_seq<kMode>(a, 0), group, row0);
        cost = rows_cost((unsigned)units * (unsigned)a.num_seqs, columns, a.seq_cost);
        const unsigned per = rows_span(units, cost);
        total = per * (unsigned)a.num_seqs;
        columns = (int)min((unsigned)columns, max(total, 1u));   // never an empty column between two others
        const Cut cut(total, (unsigned)columns, (unsigned)a.forced_units);
        u_begin = cut.first(column);
        u_end = min(total, cut.first(column + 1));
        if (column >= columns || u_begin >= u_end) {   // fewer units than columns
            if (behind) asm volatile("griddepcontrol.wait;\n" ::: "memory");
            return;
        }
        s = (int)(u_begin / per);
        seq_first = per * (unsigned)s;
    } else {
        // four neighbouring sequences per lane, 128 at a time; the last 128's counts stay in registers: units, and sequences that have any
        int mine[4], lane_sum = 0, upto = 0, lane_seqs = 0, upto_seqs = 0;
        auto count = [&](int s0) {
            lane_sum = lane_seqs = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int si = s0 + lane * 4 + i;
                mine[i] = si < a.num_seqs ? rows_units<kWarps>(a, rows_seq<kMode>(a, si), group, row0) : 0;
                lane_sum += mine[i];
                lane_seqs += mine[i] > 0 ? 1 : 0;
            }
            upto = lane_sum;
            upto_seqs = lane_seqs;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int o = __shfl_up_sync(0xffffffffu, upto, off), q = __shfl_up_sync(0xffffffffu, upto_seqs, off);
                if (lane >= off) {
                    upto += o;
                    upto_seqs += q;
                }
            }
        };
        int s0 = 0;
        unsigned seqs = 0;
#pragma unroll 1
        for (;; s0 += 128) {
            count(s0);
            total += (unsigned)__shfl_sync(0xffffffffu, upto, 31);
            seqs += (unsigned)__shfl_sync(0xffffffffu, upto_seqs, 31);
            if (s0 + 128 >= a.num_seqs) break;
        }
        cost = rows_cost(total, columns, a.seq_cost);
        total += seqs * (unsigned)cost;
        columns = (int)min((unsigned)columns, max(total, 1u));   // never an empty column between two others
        const Cut cut(total, (unsigned)columns, (unsigned)a.forced_units);
        u_begin = cut.first(column);
        u_end = min(total, cut.first(column + 1));
        if (column >= columns || u_begin >= u_end) {   // fewer units than columns
            if (behind) asm volatile("griddepcontrol.wait;\n" ::: "memory");
            return;
        }
        if (s0 > 0) s0 = 0;          // more than 128 sequences: walk them again from the start
        else s0 = -1;
#pragma unroll 1
        for (;;) {
            if (s0 >= 0) count(s0);
            const unsigned past = __ballot_sync(0xffffffffu, seq_first + (unsigned)(upto + upto_seqs * cost) > u_begin);
            if (past != 0u) {   // always before the sequences run out: u_begin < total
                const int at = __ffs(past) - 1;
                unsigned f = seq_first + (unsigned)(upto - lane_sum + (upto_seqs - lane_seqs) * cost);
                int si = max(s0, 0) + lane * 4;
#pragma unroll
                for (int i = 0; i < 3; ++i)
                    if (f + rows_span(mine[i], cost) <= u_begin && si == max(s0, 0) + lane * 4 + i) {
                        f += rows_span(mine[i], cost);
                        ++si;
                    }
                s = __shfl_sync(0xffffffffu, si, at);
                seq_first = __shfl_sync(0xffffffffu, f, at);
                break;
            }
            seq_first += (unsigned)(__shfl_sync(0xffffffffu, upto, 31) + __shfl_sync(0xffffffffu, upto_seqs, 31) * cost);
            s0 += 128;
        }
    }

    const T* __restrict__ qg = static_cast<const T*>(a.q);
    const T* __restrict__ kg = static_cast<const T*>(a.k);
    const T* __restrict__ vg = static_cast<const T*>(a.v);
    const long long kv_pitch = (long long)a.kv_heads * D;

    unsigned char* ring = smem_raw + warp * S::kWarpBytes;

    // ---- copy side: a cursor of its own over the CTA's units ------------------------------------------
    // Copies of one tile: a K/V row (D*2 bytes) is moved by kChunksPerRow adjacent lanes, 16 bytes
    // each, so one warp instruction reads whole rows (full 128-byte lines). Lane r < 16 looks up the
    // slot of token row r once per tile, two tiles ahead (the look-up is a load of its own, of a
    // microsecond under load); the other lanes get it by shuffle.
    constexpr int kRowsPerInstr = 32 / kChunksPerRow;      // 2 (D=128) or 4 (D=64)
    constexpr int kInstrPerTile = kTile / kRowsPerInstr;   // 8 or 4
    static_assert(kCopiesPerLane == kInstrPerTile, "a lane issues one 16-byte copy per instruction");
    const int cp_ch = lane % kChunksPerRow;
    const int cp_sub = lane / kChunksPerRow;
    int cp_s = s;
    unsigned cp_first = seq_first;                     // unit at which sequence cp_s begins
    RowsSeq cp_seq = rows_seq<kMode>(a, s);
    int cp_units = rows_units<kWarps>(a, cp_seq, group, row0);
    int cp_vis = rows_visible(cp_seq);
    int cp_tok = (int)(u_begin - seq_first) * kUnit;   // first token of the unit to look up next
    int cp_end = (int)min((unsigned)cp_units, u_end - cp_first) * kUnit;   // tokens of it that are this CTA's
    int cp_looked = 0, cp_issued = 0;                  // units looked up and asked for
    // on to the next sequence that has units here
    auto cp_next_seq = [&]() {
        while (cp_tok >= cp_end) {
            cp_first += rows_span(cp_units, cost);
            if (cp_first >= u_end) return;
            cp_seq = rows_seq<kMode>(a, ++cp_s);
            cp_units = rows_units<kWarps>(a, cp_seq, group, row0);
            cp_vis = rows_visible(cp_seq);
            cp_tok = 0;
            cp_end = (int)min((unsigned)cp_units, u_end - cp_first) * kUnit;
        }
    };
    cp_next_seq();
    auto look_up = [&]() -> long long {   // element offset of this lane's token row in the caches, -1 past the visible keys
        const int j = cp_tok + warp * kTile + (lane & 15);
        if (j >= cp_vis) return -1;
        long long slot;
        if (kMode == MODE_KVCACHE || (kMode == MODE_VARLEN && a.paged)) {
            const int page = a.block_shift >= 0 ? j >> a.block_shift : j / a.block_size;
            slot = a.block_tables[cp_s * a.max_blocks + page] * a.block_size + (j - page * a.block_size);
        } else {
            slot = cp_seq.kv_row0 + j;
        }
        return slot * kv_pitch + (long long)kvh * D;
    };
    auto look_up_next = [&]() -> long long {
        if (cp_tok >= cp_end) return -1;
        const long long off = look_up();
        ++cp_looked;
        cp_tok += kUnit;
        if (cp_tok >= cp_end) cp_next_seq();
        return off;
    };
    long long cp_off = look_up_next();
    long long cp_off2 = look_up_next();
    int cp_stage = 0;
    auto issue = [&]() {
        if (cp_issued < cp_looked) {
            unsigned char* kst = ring + cp_stage * S::kStageBytes;
            unsigned char* vst = kst + S::kTileBytes;
#pragma unroll
            for (int i = 0; i < kInstrPerTile; ++i) {
                const int row = i * kRowsPerInstr + cp_sub;
                const long long off = __shfl_sync(0xffffffffu, cp_off, row);
                const bool valid = off >= 0;
                const long long src = (valid ? off : 0) + cp_ch * 8;
                const int dst = row * S::kRowBytes + ((cp_ch ^ (row & S::kSwz)) << 4);
                cp_async_16(kst + dst, kg + src, valid);
                cp_async_16(vst + dst, vg + src, valid);
            }
            cp_stage = cp_stage + 1 == kStages ? 0 : cp_stage + 1;
            ++cp_issued;
            cp_off = cp_off2;
            cp_off2 = look_up_next();
        }
        cp_async_commit();  // committed even when empty so that group counting stays uniform
    };

#pragma unroll
    for (int it = 0; it < kStages - 1; ++it) issue();

    // ---- compute side: sequence after sequence ----------------------------------------------------------
    float* const merge = reinterpret_cast<float*>(smem_raw + S::kRingBytes);
    int* const last_flag = reinterpret_cast<int*>(smem_raw + S::kRingBytes + S::kMergeBytes);
    const int cta = blockIdx.y * gridDim.x + blockIdx.x;
    int stage = 0;
    unsigned u = u_begin;
    while (u < u_end) {
        const RowsSeq seq = rows_seq<kMode>(a, s);
        const int units = rows_units<kWarps>(a, seq, group, row0);
        if (u >= seq_first + (unsigned)units) {   // not this launch's, or ended
            seq_first += rows_span(units, cost);
            u = max(u, seq_first);
            ++s;
            continue;
        }
        const int vis = rows_visible(seq);
        const int nrows = min(kRows, seq.q_len * group - row0);   // query rows served here
        const unsigned seg_end = min(u_end, seq_first + (unsigned)units);
        const bool starts = u == seq_first, ends = seg_end == seq_first + (unsigned)units;

        // Q fragments of the A operand, straight from global: rows g and g+8; and the last key each of them sees.
        unsigned qa[kKSteps][4];
        int lim0 = -1, lim1 = -1;
        {
            const bool v0 = g < nrows, v1 = g + 8 < nrows;
            const int r0 = row0 + g, r1 = row0 + g + 8;
            const int t0 = r0 / group, t1 = r1 / group;
            const unsigned* q0 = reinterpret_cast<const unsigned*>(qg + ((seq.q_row0 + t0) * a.q_heads + kvh * group + (r0 - t0 * group)) * D);
            const unsigned* q1 = reinterpret_cast<const unsigned*>(qg + ((seq.q_row0 + t1) * a.q_heads + kvh * group + (r1 - t1 * group)) * D);
#pragma unroll
            for (int kk = 0; kk < kKSteps; ++kk) {
                qa[kk][0] = v0 ? q0[kk * 8 + c4] : 0u;
                qa[kk][1] = v1 ? q1[kk * 8 + c4] : 0u;
                qa[kk][2] = v0 ? q0[kk * 8 + 4 + c4] : 0u;
                qa[kk][3] = v1 ? q1[kk * 8 + 4 + c4] : 0u;
            }
            lim0 = (int)min((long long)seq.kv_len - 1, (long long)seq.pos_off + t0);
            lim1 = (int)min((long long)seq.kv_len - 1, (long long)seq.pos_off + t1);
        }
        const int lim_all = min(seq.kv_len, seq.pos_off + 1);   // keys below this are seen by every row

        float acc[kDBlocks][4];
#pragma unroll
        for (int n = 0; n < kDBlocks; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0f;
        float m0 = -INFINITY, m1 = -INFINITY;  // running max of rows g and g+8 (log2 domain)
        float l0 = 0.0f, l1 = 0.0f;            // this lane's share of the running sums

        int tok = (int)(u - seq_first) * kUnit + warp * kTile;   // first token of this warp's tile
        for (; u < seg_end; ++u, tok += kUnit) {
            issue();
            cp_async_wait<kStages - 1>();
            __syncwarp();
            const unsigned char* kst = ring + stage * S::kStageBytes;
            const unsigned char* vst = kst + S::kTileBytes;
            stage = stage + 1 == kStages ? 0 : stage + 1;
            if (tok >= vis) continue;   // past the last visible key: this warp has no tile in the sequence's last unit

            // S = Q K^T : 16 query rows x 16 tokens as two N blocks of 8 tokens
            float sc[2][4];
#pragma unroll
            for (int nb = 0; nb < 2; ++nb) sc[nb][0] = sc[nb][1] = sc[nb][2] = sc[nb][3] = 0.0f;
            {
                const int mi = lane >> 3;                    // which 8x8 matrix this lane addresses
                const int tr = ((mi >> 1) << 3) + (lane & 7);  // token row
#pragma unroll
                for (int kk = 0; kk < kKSteps; ++kk) {
                    const int ch = 2 * kk + (mi & 1);
                    unsigned b0, b1, b2, b3;
                    ldmatrix_x4(b0, b1, b2, b3, kst + tr * S::kRowBytes + ((ch ^ (tr & S::kSwz)) << 4));
                    mma_16816<T>(sc[0], qa[kk], b0, b1);
                    mma_16816<T>(sc[1], qa[kk], b2, b3);
                }
            }

            // scale, mask (only tiles that reach past the first query token's position need it), online
            // softmax over this tile's 16 tokens
            const bool cut = tok + kTile > lim_all;
            float tmax0 = -INFINITY, tmax1 = -INFINITY;
#pragma unroll
            for (int nb = 0; nb < 2; ++nb) {
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int j = tok + nb * 8 + 2 * c4 + e;
                    sc[nb][e] *= a.scale_log2;
                    sc[nb][2 + e] *= a.scale_log2;
                    if (cut) {
                        if (j > lim0) sc[nb][e] = -INFINITY;
                        if (j > lim1) sc[nb][2 + e] = -INFINITY;
                    }
                    tmax0 = fmaxf(tmax0, sc[nb][e]);
                    tmax1 = fmaxf(tmax1, sc[nb][2 + e]);
                }
            }
            tmax0 = fmaxf(tmax0, __shfl_xor_sync(0xffffffffu, tmax0, 1));
            tmax0 = fmaxf(tmax0, __shfl_xor_sync(0xffffffffu, tmax0, 2));
            tmax1 = fmaxf(tmax1, __shfl_xor_sync(0xffffffffu, tmax1, 1));
            tmax1 = fmaxf(tmax1, __shfl_xor_sync(0xffffffffu, tmax1, 2));
            const float mp0 = m0, mp1 = m1;
            m0 = fmaxf(m0, tmax0);
            m1 = fmaxf(m1, tmax1);
            // a row that has seen no key yet keeps m = -inf: exp2(-inf - 0) is an exact zero
            const float mu0 = m0 == -INFINITY ? 0.0f : m0, mu1 = m1 == -INFINITY ? 0.0f : m1;
            const float alpha0 = fast_exp2(mp0 - mu0), alpha1 = fast_exp2(mp1 - mu1);
            float ps0 = 0.0f, ps1 = 0.0f;
#pragma unroll
            for (int nb = 0; nb < 2; ++nb) {
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    sc[nb][e] = fast_exp2(sc[nb][e] - mu0);
                    sc[nb][2 + e] = fast_exp2(sc[nb][2 + e] - mu1);
                    ps0 += sc[nb][e];
                    ps1 += sc[nb][2 + e];
                }
            }
            l0 = l0 * alpha0 + ps0;
            l1 = l1 * alpha1 + ps1;
#pragma unroll
            for (int n = 0; n < kDBlocks; ++n) {
                acc[n][0] *= alpha0;
                acc[n][1] *= alpha0;
                acc[n][2] *= alpha1;
                acc[n][3] *= alpha1;
            }

            // O += P V : P (16 rows x 16 tokens) re-used from the accumulator layout as the A operand
            unsigned pa[4];
            pa[0] = pack2<T>(sc[0][0], sc[0][1]);
            pa[1] = pack2<T>(sc[0][2], sc[0][3]);
            pa[2] = pack2<T>(sc[1][0], sc[1][1]);
            pa[3] = pack2<T>(sc[1][2], sc[1][3]);
            {
                const int mi = lane >> 3;
                const int tr = ((mi & 1) << 3) + (lane & 7);
#pragma unroll
                for (int n = 0; n < kDBlocks; n += 2) {
                    const int ch = n + (mi >> 1);
                    unsigned b0, b1, b2, b3;
                    ldmatrix_x4_trans(b0, b1, b2, b3, vst + tr * S::kRowBytes + ((ch ^ (tr & S::kSwz)) << 4));
                    mma_16816<T>(acc[n], pa, b0, b1);
                    mma_16816<T>(acc[n + 1], pa, b2, b3);
                }
            }
            __syncwarp();  // the stage may be refilled by the next issue()
        }

        // ---- the warps' parts of this sequence, merged through shared memory ----------------------------
        // row sums: fold the four lanes that share a row
        l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
        l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
        l1 += __shfl_xor_sync(0xffffffffu, l1, 1);
        l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
        // Up to 8 rows fit the buffer whole; 16 go through it 64 columns at a time. Rows that do not exist are not written: a CTA does this once per
        // sequence with nothing of its own in flight but the ring, which is what batches of short contexts are made of
        // (256 x 128-512 tokens: 32/32 heads 294 us with all 16 rows in two passes, 259 so; 32/8 heads 86.5 and 82). The two are
        // separate code: with the pitch in a variable 16 sequences x 4 tokens x 4 heads lost 1.5 %.
        const int slot = 2 * cta + (starts ? 1 : 0);
        auto merge_warps = [&](auto few) {
            constexpr bool kFew = decltype(few)::value;
            constexpr int kCols = kFew ? D : S::kMergeCols, kPitch = kCols + 2, kSlots = kFew ? kRows / 2 : kRows;
            auto merge_ml = [&](int w, int r) { return reinterpret_cast<float2*>(merge + (w * kSlots + r) * kPitch + kCols); };
            float* const mine = merge + warp * kSlots * kPitch;
            if (c4 == 0) {
                if (!kFew || g < nrows) *merge_ml(warp, g) = make_float2(m0, l0);
                if (!kFew) *merge_ml(warp, g + 8) = make_float2(m1, l1);
            }
#pragma unroll
            for (int pass = 0; pass < D / kCols; ++pass) {
#pragma unroll
                for (int n = 0; n < kCols / 8; ++n) {
                    const int d = n * 8 + 2 * c4;
                    const float(&x)[4] = acc[pass * (kCols / 8) + n];
                    if (!kFew || g < nrows) *reinterpret_cast<float2*>(mine + g * kPitch + d) = make_float2(x[0], x[1]);
                    if (!kFew) *reinterpret_cast<float2*>(mine + (g + 8) * kPitch + d) = make_float2(x[2], x[3]);
                }
                __syncthreads();
                for (int idx = threadIdx.x; idx < nrows * (kCols / 2); idx += kThreads) {
                    const int r = idx / (kCols / 2);
                    const int d = (idx - r * (kCols / 2)) * 2;
                    float2 ml[kWarps];
                    float mstar = -INFINITY;
#pragma unroll
                    for (int w = 0; w < kWarps; ++w) {
                        ml[w] = *merge_ml(w, r);
                        mstar = fmaxf(mstar, ml[w].x);
                    }
                    float ox = 0.0f, oy = 0.0f, l = 0.0f;
#pragma unroll
                    for (int w = 0; w < kWarps; ++w) {
                        const float wgt = ml[w].x == -INFINITY ? 0.0f : fast_exp2(ml[w].x - mstar);
                        const float2 x = *reinterpret_cast<const float2*>(merge + (w * kSlots + r) * kPitch + d);
                        ox += wgt * x.x;
                        oy += wgt * x.y;
                        l += wgt * ml[w].y;
                    }
                    const int dd = pass * kCols + d;
                    if (starts && ends) {   // the whole sequence: finished here
                        const float inv = l > 0.0f ? 1.0f / l : 0.0f;   // reference: flash_attn_with_kvcache.cu:109
                        const int t = (row0 + r) / group, h = kvh * group + (row0 + r) - t * group;
                        const unsigned w2 = pack2<T>(ox * inv, oy * inv);
                        store_pair<T>(a.out, seq.q_row0 + t, h, D, dd, w2);
                        if (dd == 0 && a.out.lse != nullptr)
                            a.out.lse[((long long)s * a.q_heads + h) * a.q_seq_len + t] = l > 0.0f ? (mstar + log2f(l)) * 0.6931471805599453f : -INFINITY;
                    } else {
                        *reinterpret_cast<float2*>(a.ws_acc + ((long long)slot * kRows + r) * D + dd) = make_float2(ox, oy);
                        if (dd == 0) a.ws_ml[(long long)slot * kRows + r] = make_float2(mstar, l);
                    }
                }
                __syncthreads();   // the buffer is written again by the next pass or sequence
            }
        };
        if (nrows <= kRows / 2) merge_warps(std::true_type{});
        else merge_warps(std::false_type{});

        if (!(starts && ends)) {
            // ---- a cut sequence: whoever brings the last part merges all of them, in column order --------
            const Cut cut(total, (unsigned)columns, (unsigned)a.forced_units);
            const int c_first = (int)cut.column_of(seq_first);
            const int parts = (int)cut.column_of(seq_first + (unsigned)units - 1u) - c_first + 1;
            // (the last pass of the merge above ended with a barrier: every thread's partials are before this)
            if (threadIdx.x == 0) {
                unsigned long long* cnt = a.arrived + (long long)blockIdx.x * a.num_seqs + s;
                const int last = arrive_acq_rel(cnt, a.call) == (unsigned long long)(parts - 1);
                if (last) *cnt = 0ull;   // as it was found: a captured launch runs again under the same number
                *last_flag = last;
            }
            __syncthreads();
            if (*last_flag) {
                const int rows_per_warp = (nrows + kWarps - 1) / kWarps;
                if (rows_per_warp == 1) merge_parts<T, D, 1, kWarps>(a, merge, seq.q_row0, s, kvh, row0, group, nrows, c_first, parts, warp, lane);
                else if (rows_per_warp == 2) merge_parts<T, D, 2, kWarps>(a, merge, seq.q_row0, s, kvh, row0, group, nrows, c_first, parts, warp, lane);
                else merge_parts<T, D, 4, kWarps>(a, merge, seq.q_row0, s, kvh, row0, group, nrows, c_first, parts, warp, lane);
                __syncthreads();   // the merge buffer is written again by the next sequence
            }
        }
    }
    cp_async_wait<0>();
    if (behind) asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

// The grid: one CTA per KV head (x row block) and column, as many columns as fill the device's CTA slots in
// one wave or, where that leaves too many slots empty (many KV heads), in two.
int num_columns(int per_column, int ctas_per_sm, int sms) {
    const long long slots = (long long)ctas_per_sm * sms;
    const int one = (int)std::max<long long>(1, slots / per_column);
    const int two = (int)std::max<long long>(1, 2 * slots / per_column);
    const bool one_fills = (long long)one * per_column * 100 >= slots * 95 || 2LL * one * per_column >= (long long)two * per_column;
    return one_fills ? one : two;
}

// `rows`: query rows per KV head at most; `max_tokens`: upper bound of a sequence's visible keys.
// `wide_sms` > 0: a launch of wide CTAs on about so many SMs.
template <int D>
RowsPlan plan_rows(int num_seqs, int kv_heads, int rows, long long max_tokens, bool allow_forced, int wide_sms = 0) {
    RowsPlan r;
    r.row_blocks = (rows + kRows - 1) / kRows;
    const long long per_column = (long long)kv_heads * r.row_blocks;
    if (per_column > 0x7fffffffLL) return r;   // columns == 0: not this kernel's
    const int kUnit = wide_sms > 0 ? unit_of<kWide> : unit_of<kFour>;
    r.wide = wide_sms > 0 ? 1 : 0;
    r.columns = r.wide ? (int)std::max(1LL, wide_sms / per_column) : num_columns((int)per_column, Smem<D, kFour>::kCtasPerSm, sm_count());
    const long long most_units = (long long)num_seqs * std::max(1LL, (max_tokens + kUnit - 1) / kUnit);
    if (!r.wide && allow_forced && get_option_decode_chunk() > 0) {
        r.forced_units = (get_option_decode_chunk() + kUnit - 1) / kUnit;
        while ((most_units + r.forced_units - 1) / r.forced_units > 4096) r.forced_units *= 2;
        r.columns = (int)((most_units + r.forced_units - 1) / r.forced_units);
    }
    r.columns = (int)std::min<long long>(std::min(r.columns, kMaxColumns), most_units);
    const size_t slots = (size_t)2 * per_column * r.columns;
    r.acc_bytes = slots * kRows * D * sizeof(float);
    r.partial_bytes = r.acc_bytes + slots * kRows * sizeof(float2);
    r.counter_bytes = (size_t)per_column * num_seqs * sizeof(unsigned long long);
    return r;
}

std::atomic<unsigned long long> g_calls{0};   // launches of this kernel, of any type and on any device

template <typename T, int D, int kMode, int kWarps>
int launch_rows_as(RowsArgs& a, const RowsPlan& plan, cudaStream_t stream) {
    using S = Smem<D, kWarps>;
    static_assert(kMaxColumns < (1 << kCountBits), "the parts of a sequence fit the count");
    a.row_blocks = plan.row_blocks;
    a.forced_units = plan.forced_units;
    // (us for costs of 0, 2, 3, 4, 6: 64 x 512-8192 180.4, 180.3, 180.7-182, 181.2, 186; 8 x 4000 contiguous 27.9, 27.3, 26.7, 26.2, 25.9; 4 x 2369 15.9, 13.2, 13.8, 13.9, 13.9; with 16
    // rows 43 x 4 tokens over 200-3000 67.0, 63.6, 62.6, 61.1, 59.5; 64 x 2 over 100-1600, 64/8 heads 59.3, 56.7, 54.4, 53.3, 51.6; 16 x 4 over 512-8192 58.6, 58.2, 58.9, 57.5, 58.4)
    const int rows = a.max_rows < kRows ? a.max_rows : kRows;
    a.seq_cost = plan.forced_units > 0 ? 0 : rows > 8 ? 5 : 3;
    static std::atomic<unsigned long long> ready{0};   // devices whose copy of this kernel has its shared-memory limit raised
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err == cudaSuccess && (dev >= 64 || !((ready.load(std::memory_order_acquire) >> dev) & 1ULL))) {
        err = cudaFuncSetAttribute(decode_splitk_kernel<T, D, kMode, kWarps>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kBytes);
        if (err == cudaSuccess && dev < 64) ready.fetch_or(1ULL << dev, std::memory_order_release);
    }
    if (err != cudaSuccess) {
        set_last_errorf("decode_splitk_kernel: %s", cudaGetErrorString(err));
        cudaGetLastError();
        return FLASH_ATTN_ERR_CUDA;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(a.kv_heads * plan.row_blocks), (unsigned)plan.columns);
    cfg.blockDim = dim3(kWarps * 32);
    cfg.dynamicSmemBytes = S::kBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, decode_splitk_kernel<T, D, kMode, kWarps>, a);
    return check_launch("decode_splitk_kernel");
}

template <typename T, int D>
int launch_rows(RowsArgs& a, const RowsPlan& plan, cudaStream_t stream) {
    a.call = (g_calls.fetch_add(1, std::memory_order_relaxed) + 1) << kCountBits;
    for (int i = 0; i < a.out.n_out; ++i) a.out.halves |= (reinterpret_cast<uintptr_t>(a.out.o[i]) & 3) != 0;
    if constexpr (D >= 64)
        if (plan.wide) return launch_rows_as<T, D, MODE_VARLEN, kWide>(a, plan, stream);
    return a.mode == MODE_KVCACHE ? launch_rows_as<T, D, MODE_KVCACHE, kFour>(a, plan, stream)
           : a.mode == MODE_BATCH ? launch_rows_as<T, D, MODE_BATCH, kFour>(a, plan, stream)
                                  : launch_rows_as<T, D, MODE_VARLEN, kFour>(a, plan, stream);
}

int log2_or_minus1(int v) {
    for (int i = 0; i < 31; ++i)
        if (v == (1 << i)) return i;
    return -1;
}

// What can fail before anything is launched: the plan and its workspace. -1: not this kernel's; FLASH_ATTN_ERR_CUDA (no
// message yet): no memory for it, which is a failure only where no other kernel can take the call.
template <int D>
int prepare_typed(const AttnParams& p, int rows, cudaStream_t stream, RowsPlan& plan, Workspace& ws, int wide_sms) {
    const long long max_tokens = p.mode == MODE_KVCACHE ? (long long)p.max_blocks * p.block_size : p.kv_seq_len;
    if (max_tokens <= 0) return -1;
    // (behind a prefill kernel, whose SMs come free one after the other, smaller shares were no faster: 4 chunks of 512 with 32
    // decoding sequences 248-252 us with one share per CTA slot, 256 with two, 253-257 with three)
    plan = plan_rows<D>(p.num_seqs, p.kv_heads, rows, max_tokens, true, wide_sms);
    if (plan.columns <= 0) return -1;
    ws = decode_workspace(stream, plan.partial_bytes, plan.counter_bytes);
    return ws.partials != nullptr ? FLASH_ATTN_OK : FLASH_ATTN_ERR_CUDA;
}

template <typename T, int D>
int launch_typed(const AttnParams& p, int max_rows, bool behind_prefill, const RowsPlan& plan, const Workspace& ws, cudaStream_t stream) {
    RowsArgs a{};
    a.behind_prefill = behind_prefill && !plan.wide ? 1 : 0;
    a.q = p.q; a.k = p.k; a.v = p.v;
    a.block_tables = p.block_tables;
    a.context_lens = p.context_lens;
    a.cu_q = p.cu_q;
    a.cu_k = p.cu_k;
    a.ws_acc = reinterpret_cast<float*>(ws.partials);
    a.ws_ml = reinterpret_cast<float2*>(ws.partials + plan.acc_bytes);
    a.arrived = ws.counters;
    a.mode = p.mode;
    a.num_seqs = p.num_seqs;
    a.q_seq_len = p.q_seq_len;
    a.kv_seq_len = p.kv_seq_len;
    a.start_pos = p.start_pos;
    a.q_heads = p.q_heads;
    a.kv_heads = p.kv_heads;
    a.block_size = p.block_size;
    a.block_shift = log2_or_minus1(p.block_size);
    a.max_blocks = p.max_blocks;
    a.paged = p.paged;
    a.capacity = p.paged ? (int)std::min(0x7fffffffLL, (long long)p.max_blocks * p.block_size) : 0x7fffffff;
    a.max_rows = max_rows;
    a.scale_log2 = p.scale * 1.4426950408889634f;
    if (p.n_out > 0) {
        for (int i = 0; i < p.n_out && i < 8; ++i) a.out.o[i] = p.o_peers[i];
        a.out.n_out = p.n_out;
        a.out.o_heads = p.o_heads;
        a.out.o_head0 = p.o_head0;
        a.out.peer0 = (p.o_head0 / p.q_heads + 1) % p.n_out;
    } else {
        a.out.o[0] = p.o;
        a.out.n_out = 1;
        a.out.o_heads = p.q_heads;
    }
    a.out.lse = p.lse;
    const int rc = launch_rows<T, D>(a, plan, stream);
    if (rc == FLASH_ATTN_OK) note_path("decode_splitk", 1);
    return rc;
}

}  // namespace

namespace {

// 16-bit storage, 16-byte aligned K/V rows (cp.async); q is read four bytes at a time.
bool rows_kernel_takes(const AttnParams& p) {
    if (p.dtype != DT_F16 && p.dtype != DT_BF16) return false;
    if (p.head_size != 32 && p.head_size != 64 && p.head_size != 128) return false;
    if (p.mask != nullptr || p.n_lse > 0 || p.multicast) return false;
    if ((reinterpret_cast<uintptr_t>(p.k) | reinterpret_cast<uintptr_t>(p.v)) & 15) return false;
    return (reinterpret_cast<uintptr_t>(p.q) & 3) == 0;
}

int prepare_rows(const AttnParams& p, int rows, cudaStream_t stream, RowsPlan& plan, Workspace& ws, int wide_sms = 0) {
    return p.head_size == 128 ? prepare_typed<128>(p, rows, stream, plan, ws, wide_sms)
           : p.head_size == 64 ? prepare_typed<64>(p, rows, stream, plan, ws, wide_sms)
                               : prepare_typed<32>(p, rows, stream, plan, ws, 0);
}

int launch_prepared(const AttnParams& p, int max_rows, bool behind_prefill, const RowsPlan& plan, const Workspace& ws, cudaStream_t stream) {
    if (p.dtype == DT_BF16) {
        return p.head_size == 128 ? launch_typed<__nv_bfloat16, 128>(p, max_rows, behind_prefill, plan, ws, stream)
               : p.head_size == 64 ? launch_typed<__nv_bfloat16, 64>(p, max_rows, behind_prefill, plan, ws, stream)
                                   : launch_typed<__nv_bfloat16, 32>(p, max_rows, behind_prefill, plan, ws, stream);
    }
    return p.head_size == 128 ? launch_typed<__half, 128>(p, max_rows, behind_prefill, plan, ws, stream)
           : p.head_size == 64 ? launch_typed<__half, 64>(p, max_rows, behind_prefill, plan, ws, stream)
                               : launch_typed<__half, 32>(p, max_rows, behind_prefill, plan, ws, stream);
}

}  // namespace

int launch_decode_splitk(const AttnParams& p, cudaStream_t stream) {
    if (p.mode != MODE_KVCACHE || p.q_seq_len != 1 || !rows_kernel_takes(p)) return -1;
    const int rows = p.q_heads / p.kv_heads;
    RowsPlan plan;
    Workspace ws;
    const int rc = prepare_rows(p, rows, stream, plan, ws);
    if (rc == FLASH_ATTN_ERR_CUDA)
        set_last_errorf("flash_attn_with_kvcache: could not allocate %zu bytes of split-K workspace", plan.partial_bytes + plan.counter_bytes);
    return rc == FLASH_ATTN_OK ? launch_prepared(p, rows, false, plan, ws, stream) : rc;
}

// ---- this kernel or the prefill kernel, for calls that both take: the time of each, in microseconds, from what the host knows.
// Prefill kernel: a CTA per pair of 128-row tiles, one per SM; a CTA walks its K/V range at 1.5 us per 128 keys after 6.6 us of set-up. (Measured again
// since that kernel's issuer, set-up and softmax step got shorter, calls of one wave: 27-31 us at 2048 keys, 41-55 at 4096, 95-109 at 8192, where this says
// 31, 55 and 103.)
static long long longest_keys(const AttnParams& p) { return p.mode == MODE_KVCACHE ? (long long)p.max_blocks * p.block_size : p.kv_seq_len; }
static long long tile_pairs(const AttnParams& p, long long q_len) { return ((long long)(p.q_heads / p.kv_heads) * ((q_len + 127) / 128) + 1) / 2 * p.kv_heads; }
static double prefill_us(const AttnParams& p, double pairs, double setup = 6.6) {
    return std::max(1.0, pairs / sm_count()) * (setup + 1.5 * (double)((longest_keys(p) + 127) / 128));
}
// This kernel: a CTA slot takes 1.04 us per unit of 64 keys (16 rows of one KV head; 0.91 where several row blocks read the same K/V) and 2.2 us
// + 0.15 us a row per sequence, most of it the merge of its warps' parts; some sequence of more than one unit is always cut, and the merge of its
// parts is another 0.6 us a row.
static double rows_us(const AttnParams& p, long long seqs, long long rows) {
    const long long slots = (long long)sm_count() * (p.head_size == 128 ? Smem<128, kFour>::kCtasPerSm : p.head_size == 64 ? Smem<64, kFour>::kCtasPerSm : Smem<32, kFour>::kCtasPerSm);
    constexpr int kUnit = unit_of<kFour>;
    const double units = (double)((longest_keys(p) + kUnit - 1) / kUnit), nrows = (double)std::min<long long>(kRows, rows);
    const double blocks_per_slot = (double)(seqs * p.kv_heads * ((rows + kRows - 1) / kRows)) / (double)slots;
    return 4.4 + ((rows > kRows ? 0.91 : 1.04) * units + 2.2 + 0.15 * nrows) * blocks_per_slot + (units > 1.0 ? 0.6 * nrows : 0.0);
}

// Prefill kernel, the few rows of a sequence in one tile for as many heads as share one, clusters for the keys where they find room: 4 us a wave and 1.4 us per 128 keys, 4 more for a cluster.
static double prefill_few_rows_us(const AttnParams& p, long long rows) {
    const long long pairs = prefill_pairs(p.q_heads / p.kv_heads, p.q_seq_len) * p.kv_heads * p.num_seqs, tiles = (longest_keys(p) + 127) / 128;
    const int parts = prefill_parts(pairs, tiles, p.mode == MODE_BATCH, rows, sm_count());
    const double waves = std::max(1.0, (double)pairs / sm_count());
    return std::ceil(waves) * 4.0 + waves * 1.4 * (double)((tiles + parts - 1) / parts) + (parts > 1 ? 4.0 : 0.0);
}

// Up to four row blocks of 16 (query token x group head) rows, each of which reads the K/V rows again, from L2; the prefill kernel reads K/V once and has them in one tile
// where the heads of a group share it. Both kernels over 154 shapes of 1-64 sequences x 1-32 tokens, 64-32768 keys, groups of 1, 4 and 8: the choice takes on average 6 % more than the
// faster kernel for each (9 % with a tile for every head in the estimate, and with all calls of one wave over up to 12 tiles left to the prefill kernel). us there and here:
// 32 x 12 tokens over 1031-4126, 32/8 heads 81 and 139; 41 x 8 over 1375, 64/8 78 and 142; 16 x 4 over 216, 64/8 9.6 and 17.3; 8 x 2 over 1010, 32/8 17.7 and 13.3; 16 x 8 over 400,
// 8 heads of 64 12.9 and 10.6; 16 x 4 over 8192, 32/8 96 and 92. The estimate has to say half for the prefill kernel: it does not know the lengths, and equal shares suit unequal ones.
// Two groups of calls stay with one kernel whatever the estimates say, because programs and tests know them there: up to 64 pairs, counted by heads, over up to 12 tiles with the prefill
// kernel (4 x 1 over 544, 32/8 heads of 64 9.6 and 6.0), and up to 4 sequences by the estimates of a tile for every head (1 x 64 over 8192, 32 heads 33 and 68).
// Of the calls of one wave of pairs, counted by heads, over up to 12 tiles, four row blocks and, without GQA, short ranges stay with the prefill kernel too, where the estimates are not fine enough: 1008 shapes of 3-37 sequences x 1-16
// tokens over 66-1500 keys take 0.79 of what the prefill kernel takes for all, but of 635 that came here these were up to a quarter slower (there and here: 9 x 16 over 1200, 32/8 heads of 64 20.3 and 25.3; 3 x 8 over 500,
// 32 of 64 9.6 and 11.9; 12 x 8 over 200, 8 of 128 7.9 and 9.1) and the others at most 12 % (18 x 16 over 1500, 8 of 128 23.7 and 26.5).
int launch_few_rows(const AttnParams& p, bool prefill_takes_it, cudaStream_t stream) {
    if (p.n_out > 0 || !rows_kernel_takes(p)) return -1;
    const long long rows = (long long)p.q_seq_len * (p.q_heads / p.kv_heads);
    if (rows <= 0 || rows > 4 * kRows) return -1;
    const double pairs = (double)tile_pairs(p, p.q_seq_len) * p.num_seqs;
    if (longest_keys(p) <= 12 * 128 && pairs <= 64) return -1;
    if (prefill_takes_it) {
        if (longest_keys(p) <= 12 * 128 && pairs <= sm_count() && (rows > 3 * kRows || (p.q_heads == p.kv_heads && longest_keys(p) <= (p.num_seqs > 4 ? 3 : 4) * 128))) return -1;
        const double here = rows_us(p, p.num_seqs, rows);
        if (p.num_seqs > 4 ? prefill_few_rows_us(p, rows) < 0.575 * here : here >= prefill_us(p, pairs)) return -1;
    }
    RowsPlan plan;
    Workspace ws;
    if (prepare_rows(p, (int)rows, stream, plan, ws) != FLASH_ATTN_OK) return -1;   // the prefill kernel needs no memory of the library's
    return launch_prepared(p, (int)rows, false, plan, ws, stream);
}

// A packed batch of prompts (or chunks of them) and sequences with few rows: from the number of rows, as many sequences with max_seqlen_q
// rows as they make; the others may have few.
PackedMix packed_mix(const AttnParams& p) {
    PackedMix m{p.num_seqs, 0};
    if (p.mode != MODE_VARLEN || p.total_q <= 0) return m;
    if (p.q_seq_len > 1) m.prompts = std::min<long long>(p.num_seqs, std::max<long long>(1, ((long long)p.total_q - p.num_seqs + p.q_seq_len - 2) / (p.q_seq_len - 1)));
    else m.prompts = 0;
    m.few = p.num_seqs - m.prompts;
    return m;
}

// Whether the few-row sequences of a packed batch are better off behind the prefill kernel than in its grid, where each takes a
// CTA per two heads of its group: only where they make waves of those, by the estimates above (14 us of set-up for a CTA of a packed batch) and a
// seventh more, since the second launch
// starts when that kernel's last CTA has. Over 238 paged mixes (1-6 prompts, chunks of 64 or 512, 0-128 single tokens, contexts of
// 64-8192, four head layouts) no mix is then slower than with everything in the prefill grid, and the choice is 2 % off the better one on average:
// 4 x 512 with 32 tokens over 512-8192, 32/8 heads: 435 us in one grid, 231 so; with 1 token: 131 in one grid, 152 with two kernels, which
// one grid keeps. With the prefill kernel as it is now, 102 mixes drawn anew: two are more than 1.2 % slower than one grid (5.5 %: 53 us for 50; 2.7 %), two more than
// 5 % slower than with two kernels always (29 us for 23, 24.3 for 22.8, both 512 keys at most). Without the row count of the packed buffers (the C ABI's plain entry point) nothing is known of the mix, and
// long contexts go to two kernels.
static bool mixed_few_rows_are_better(const AttnParams& p) {
    if (p.total_q <= 0) return longest_keys(p) > 12 * 128 || tile_pairs(p, p.q_seq_len) * p.num_seqs > sm_count();
    const PackedMix m = packed_mix(p);
    if (m.few <= 0) return false;
    const double prompts = (double)m.prompts * tile_pairs(p, p.q_seq_len), few = (double)m.few * tile_pairs(p, 1);
    return prefill_us(p, prompts + few, 14.0) > 1.15 * (prefill_us(p, prompts, 14.0) + rows_us(p, m.few, p.q_heads / p.kv_heads));
}

// A mixed batch's two kernels side by side: the few-row kernel first, in CTAs of eight warps on part of the SMs, the prefill kernel behind it without waiting, on the others and then on all. How
// many SMs, and whether at all (0: behind, on all of them), by estimates from what the host knows: tile pairs of 6.6 us and 1.5 us per 128 keys; a wide CTA reads 42 GB/s (each warp's chain of products and
// exponentials) and takes 2 us for the end of each sequence, all SMs read 6.3 TB/s. One after the other the two leave the memory idle, then the tensor cores, and a last wave half empty, so that side by side is the faster up to an
// estimate a fifth above. us a pass, behind and beside: 4 chunks of 512 with 32 tokens over 512-8192, 32/8 heads 236.6 and 231.9 (on 80 SMs; 72 238, 56 244, 48 260, 96 250); 2 of 512 with 8 over
// 512-8192 139 and 116; 2 of 300 with 64 over 300-4800 173 and 161; one of 67 with 15 over 338-5418, 64/8 heads 118 and 79; one of 329 with 72 over 162-2593, 8/2 heads 76 and 46; one of 113 with 19 over
// 15-240, 32 heads of 64 24.6 and 22.8; estimated well above a fifth, and left: 5 of 72 with 43 over 113-1822, 32 heads of 64 102 (122-173 beside). Over the shortest contexts the launch that has to
// come first costs more than it wins (5 of up to 83 with 13 over 5-83, 32/8 heads from a graph 16 and 26; 4 of up to 169 with 9 over 10-169 19 and 22). Short sequences over many KV heads are ends above
// all: 3 of up to 200 with 40 over 12-200, 32/32 heads 37 behind, 49 beside on the SMs that the rate alone would give, 39 so; one of 128 with 16 over 16-260, 32/8 heads of 64 15.7, 18.6, 14.1. 160 mixes of
// contexts up to 200-900, from a graph: 0.949 of behind on average, 0.957 without the ends, 0.960 with 3 us; the slowest against behind 1.07, 1.33 and 1.06.
static int wide_sms(const AttnParams& p) {
    if (p.head_size < 64 || p.total_q <= 0 || longest_keys(p) < 192 || get_option_decode_chunk() > 0) return 0;
    const PackedMix m = packed_mix(p);
    const double keys = (double)longest_keys(p), sms = sm_count();
    const double pair = 6.6 + 1.5 * std::ceil(keys / 128.0), pairs = (double)m.prompts * (double)prefill_pairs(p.q_heads / p.kv_heads, p.q_seq_len) * p.kv_heads;
    const double bytes = (double)m.few * keys * p.kv_heads * p.head_size * 4.0, rate = 42e3 * p.head_size / 128.0;   // bytes, and bytes per us of a wide CTA
    const double ends = 2.0 * m.few * p.kv_heads;   // us of a CTA
    double best = 1.2 * (std::max(1.0, pairs / sms) * pair + bytes / 6.3e6 + ends / (2 * sms));
    int n = 0;
    for (int k = p.kv_heads; k <= 2 * (int)sms / 3; k += p.kv_heads) {
        const double few = bytes / std::min(k * rate, 6.3e6) + ends / k, all = std::max(std::max(few, pair), (pairs * pair + k * few) / sms);
        if (all < best) {
            best = all;
            n = k;
        }
    }
    return n;
}

MixedFewRows prepare_mixed_few_rows(const AttnParams& p, cudaStream_t stream) {
    MixedFewRows few;
    if (p.mode != MODE_VARLEN || p.num_seqs < 2 || p.n_out > 0 || !rows_kernel_takes(p)) return few;
    const int group = p.q_heads / p.kv_heads;
    // one row block: the CTA slots are shared out before anybody knows how many rows the sequences have
    // prompts packed back to back with their own K/V: few rows would see few keys
    if (group > kRows || (!p.paged && p.kv_seq_len <= p.q_seq_len) || !mixed_few_rows_are_better(p)) return few;
    if (prepare_rows(p, kRows, stream, few.plan, few.ws, wide_sms(p)) == FLASH_ATTN_OK) few.max_rows = kRows;
    return few;
}

int launch_mixed_few_rows(const AttnParams& p, const MixedFewRows& few, cudaStream_t stream) {
    return launch_prepared(p, few.max_rows, true, few.plan, few.ws, stream);
}

// ---------------------------------------------------------------------------------------------
// Decode without any allocation: the split-K partials live in a fixed array that is part of the
// library image instead of a cudaMalloc'ed workspace.
//
// Who needs this: a serving engine that hands all of HBM to its own pool at start-up leaves
// nothing for a library-side cudaMalloc to find, so the ordinary decode entry point can fail (or
// fragment the pool) the first time it has to size its workspace; and a caller in the middle of
// a latency-critical step cannot afford cudaMalloc / cudaFree, which take the driver's allocation
// lock and synchronise the whole device. For them the scratch is paid for once, when the library
// is loaded: every GPU whose context loads libflash_attn holds kStaticScratchBytes of it until
// the process exits, whether or not this entry point is ever called. "Loaded" is meant literally:
// with CUDA's default lazy module loading the array gets its memory when the first kernel or
// symbol of this translation unit is touched on a device — possibly the first call here — so a
// caller that is about to give away all free memory makes one small call first (or sets
// CUDA_MODULE_LOADING=EAGER); an out-of-memory answer at that point is reported as such.
//
// In host code `g_static_scratch` is only a handle for the symbol, not a device address; the
// device address is fetched once per device with cudaGetSymbolAddress (with that device current)
// and passed to the same kernel the ordinary path launches.
// ---------------------------------------------------------------------------------------------
namespace {

constexpr size_t kStaticScratchBytes = size_t(16) << 20;   // 16 MiB per GPU
constexpr size_t kStaticCounterBytes = size_t(1) << 20;    // of these, the arrival counters (at most 63 550 x 8 bytes within the entry point's limit)
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

constexpr int kMaxDevices = 64;
std::mutex g_static_mutex;
unsigned char* g_static_ptr[kMaxDevices] = {nullptr};

// Device address of the static scratch on the CURRENT device; resolved on first use per device.
unsigned char* static_scratch_ptr() {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
        cudaGetLastError();
        set_last_error("flash_attn_decode_bf16_noalloc: cannot identify the current device");
        return nullptr;
    }
    std::lock_guard<std::mutex> lock(g_static_mutex);
    if (g_static_ptr[dev] == nullptr) {
        void* ptr = nullptr;
        const cudaError_t err = cudaGetSymbolAddress(&ptr, g_static_scratch);
        if (err != cudaSuccess || ptr == nullptr) {
            cudaGetLastError();
            if (err == cudaErrorMemoryAllocation) {
                // lazy module loading: this first call is what backs the array, and no memory is left for it
                set_last_errorf("flash_attn_decode_bf16_noalloc: the library's %zu-byte scratch array could not be backed with "
                                "device memory. CUDA loads device code lazily: make the first call on each device before "
                                "the application reserves all device memory, or set CUDA_MODULE_LOADING=EAGER",
                                kStaticScratchBytes);
            } else {
                set_last_errorf("flash_attn_decode_bf16_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(err));
            }
            return nullptr;
        }
        g_static_ptr[dev] = static_cast<unsigned char*>(ptr);
    }
    return g_static_ptr[dev];
}

template <int D>
int launch_static(const void* q, const void* k, const void* v, void* o, const int* block_tables,
                  const int* context_lens, int num_seqs, int q_heads, int kv_heads, int block_size,
                  int max_blocks, float scale, cudaStream_t stream) {
    using T = __nv_bfloat16;
    const int group = q_heads / kv_heads;
    const long long max_tokens = (long long)max_blocks * block_size;

    // the documented limit of this entry point: one (acc, m, l) row per (sequence, head)
    const size_t row_bytes = (size_t)D * sizeof(float) + sizeof(float2);
    const size_t rows1 = (size_t)num_seqs * q_heads;
    if (rows1 * row_bytes > kStaticScratchBytes) {
        set_last_errorf("flash_attn_decode_bf16_noalloc: num_seqs*q_heads = %zu exceeds the static scratch "
                        "(%zu bytes hold at most %zu rows of head_size %d); use flash_attn_with_kvcache_bf16",
                        rows1, kStaticScratchBytes, kStaticScratchBytes / row_bytes, D);
        return FLASH_ATTN_ERR_INVALID_SHAPE;
    }
    // Within that limit the counters (one per sequence and row block of a KV head, at most one per row)
    // fit their part of the array; the partials are bounded by the device's CTA slots, not by the call
    // (two waves of 2 x 148 CTAs at head size 128: 9.8 MB).
    RowsPlan plan = plan_rows<D>(num_seqs, kv_heads, group, max_tokens, false);
    while (plan.columns > 1 && plan.partial_bytes > kStaticScratchBytes - kStaticCounterBytes) {
        const size_t per = plan.partial_bytes / plan.columns;
        --plan.columns;
        plan.partial_bytes -= per;
        plan.acc_bytes = (size_t)2 * kv_heads * plan.row_blocks * plan.columns * kRows * D * sizeof(float);
    }
    if (plan.columns <= 0 || plan.counter_bytes > kStaticCounterBytes) {
        set_last_error("flash_attn_decode_bf16_noalloc: grid dimensions out of range");
        return FLASH_ATTN_ERR_INVALID_SHAPE;
    }

    unsigned char* ws = static_scratch_ptr();
    if (ws == nullptr) return FLASH_ATTN_ERR_CUDA;

    RowsArgs a{};
    a.q = q; a.k = k; a.v = v;
    a.block_tables = block_tables;
    a.context_lens = context_lens;
    a.arrived = reinterpret_cast<unsigned long long*>(ws);   // zero in the library image, and again after every call
    a.ws_acc = reinterpret_cast<float*>(ws + kStaticCounterBytes);
    a.ws_ml = reinterpret_cast<float2*>(ws + kStaticCounterBytes + plan.acc_bytes);
    a.mode = MODE_KVCACHE;
    a.num_seqs = num_seqs;
    a.q_seq_len = 1;
    a.q_heads = q_heads;
    a.kv_heads = kv_heads;
    a.block_size = block_size;
    a.block_shift = log2_or_minus1(block_size);
    a.max_blocks = max_blocks;
    a.paged = 1;
    a.capacity = (int)std::min(0x7fffffffLL, max_tokens);
    a.max_rows = group;
    a.scale_log2 = scale * 1.4426950408889634f;
    a.out.o[0] = o;
    a.out.n_out = 1;
    a.out.o_heads = q_heads;
    // A captured launch keeps its number, which is lower than that of calls made since: the graph clears the counters itself.
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) cudaGetLastError();
    if (status == cudaStreamCaptureStatusActive) cudaMemsetAsync(ws, 0, plan.counter_bytes, stream);
    const int rc = launch_rows<T, D>(a, plan, stream);
    if (rc == FLASH_ATTN_OK) note_path("decode_splitk_static", 1);
    return rc;
}

}  // namespace
}  // namespace fa

extern "C" int flash_attn_decode_bf16_noalloc(const flash_attn_bf16_t* q, const flash_attn_bf16_t* k_cache,
                                              const flash_attn_bf16_t* v_cache, flash_attn_bf16_t* o,
                                              const int* block_tables, const int* context_lens, int num_seqs,
                                              int q_heads, int kv_heads, int head_size, int block_size,
                                              int max_blocks, float scale, void* stream) {
    using namespace fa;
    set_last_error("");
    cudaGetLastError();
    if (!q || !k_cache || !v_cache || !o || !block_tables || !context_lens) {
        set_last_error("flash_attn_decode_bf16_noalloc: null pointer argument");
        return FLASH_ATTN_ERR_NULL_PTR;
    }
    if (num_seqs <= 0 || q_heads <= 0 || kv_heads <= 0 || q_heads % kv_heads != 0 || block_size <= 0 || max_blocks <= 0) {
        set_last_error("flash_attn_decode_bf16_noalloc: num_seqs/heads/block_size/max_blocks must be > 0 and "
                       "q_heads a multiple of kv_heads");
        return FLASH_ATTN_ERR_INVALID_SHAPE;
    }
    if (head_size != 64 && head_size != 128) {
        set_last_error("flash_attn_decode_bf16_noalloc: head_size must be 64 or 128");
        return FLASH_ATTN_ERR_INVALID_SHAPE;
    }
    if (((reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) & 15) ||
        (reinterpret_cast<uintptr_t>(q) & 3)) {
        set_last_error("flash_attn_decode_bf16_noalloc: k_cache/v_cache must be 16-byte aligned, q 4-byte aligned");
        return FLASH_ATTN_ERR_INVALID_SHAPE;
    }
    // launch on the device that owns q, and resolve the scratch address on that same device
    int prev = -1;
    bool switched = false;
    cudaPointerAttributes attr;
    if (cudaPointerGetAttributes(&attr, q) == cudaSuccess && attr.type == cudaMemoryTypeDevice &&
        cudaGetDevice(&prev) == cudaSuccess && attr.device != prev) {
        if (cudaSetDevice(attr.device) != cudaSuccess) {
            cudaGetLastError();
            set_last_error("flash_attn_decode_bf16_noalloc: could not select the device that owns q");
            return FLASH_ATTN_ERR_CUDA;
        }
        switched = true;
    }
    cudaGetLastError();
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const int rc = head_size == 128
                       ? launch_static<128>(q, k_cache, v_cache, o, block_tables, context_lens, num_seqs, q_heads,
                                            kv_heads, block_size, max_blocks, scale, st)
                       : launch_static<64>(q, k_cache, v_cache, o, block_tables, context_lens, num_seqs, q_heads,
                                           kv_heads, block_size, max_blocks, scale, st);
    if (switched) cudaSetDevice(prev);
    return rc;
}
