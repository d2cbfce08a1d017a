// f32 storage on the tcgen05 tensor cores without giving up f32: every operand is split into three bf16 terms that together hold its 24 bits
// (Henry, Tang and Heinecke, "Leveraging the bfloat16 Artificial Intelligence Datatype For Higher-Precision Computations", 2019), and a product of two operands is
// the six term products of at least 2^-16 of the largest. Takes the problems that fill its tiles or leave SMs over from tile_f32.cu, whose warp-wide products run at an
// eighth of the rate (rule in launch_for). Replaces the same kernels of the reference: flash_attn_kernel
// (luma-flash-attn/kernels/flash_attn_func.cu:29-226), flash_attn_varlen_kernel (kernels/flash_attn_varlen_func.cu:35-199), flash_attn_prefill_kernel
// (kernels/flash_attn_with_kvcache.cu:157-277).
//
// A CTA has 128 query rows that share a KV head (row = query token x group + head in the group) and walks the K/V tiles of 64 keys that they see. Sixteen worker warps, four
// threads to a row, move the tiles in (f32, registers, one tile ahead), split them once for all rows into planes in shared memory, run the softmax and split the weights into
// tensor memory; a seventeenth warp issues the products. The scores of the next tile are computed beside this tile's softmax (at head size 128 behind its weights' product: tensor
// memory has no room for both), a tile's weights times V beside the next tile's softmax. Where blocks are few, a cluster of CTAs shares the keys of each and merges through
// distributed shared memory. Sums start from zero for every tile and are added to the running output in f32, since the tensor cores truncate when they accumulate: relative error
// against 64 bits, causal, N(0,1), 256-1500 tokens, norm by norm over all rows: 1.0-1.8e-7, log-sum-exp 2.3-3.2e-7 rms; the warp-wide products 1.1-1.9e-7 and 2.5-3.3e-7.
// What bounds it: issue slots of the workers (650 instructions a warp and step, half of them the splitting), 4000 clocks a tile; the products take 1600. 17 warps leave 96 registers a thread: 108-372 bytes of spill stores
// at head size 64, 376-924 at 128 (-Xptxas -v). us a call, warp-wide products -> this: 1 x 256, 8 heads of 64 11.9 -> 9.4; 2 x 979, 8 of 64 97 -> 36.5; 3 x 552, 8/2 of 64 50.5 -> 23.7; 3 x 301, 16/4 of 32
// 26.0 -> 12.0; 1 x 1024, 16/4 of 128 158 -> 100; 4 x 2048, 8 of 128 875 -> 507.
#include <atomic>

#include "common.cuh"
#include "tcgen05.cuh"
#include "tile_f32.cuh"

namespace fa {

namespace {

constexpr int kShares = 4;                  // threads of a row, each with a quarter of the keys and of the columns of O
constexpr int kWorkers = 128 * kShares;
constexpr int kWarps = kWorkers / 32;
constexpr int kThreads = kWorkers + 32;     // and the warp that issues the products
constexpr int kM = 128;                     // rows of a CTA: query token x head of the GQA group
constexpr int kN = 64;                      // keys of a tile
constexpr int kBlock = kN * 128;            // bytes of 64 rows of 64 columns of one term
// A row's maxima by the tile's parity: behind the barrier of its rows' warps (tile j) a warp may run on and write the next tile's maximum, while another has not yet read this one's (nothing
// else that it waits for needs that read). It writes into the same half again behind the barrier of tile j + 1, which the other reaches after its reads of tile j.
constexpr int kMaxBuffers = 2;
// Tiles of mask bytes: the two warps that bring tile j + 1 are behind the scores of tile j, that is behind what every warp did before it gave K of tile j. Warps of another quad may then still read
// the mask of tile j - 1 (at head sizes 32 and 64), not that of tile j - 2. Four and not three: the index is a mask.
constexpr int kMaskBuffers = 4;

// A product of three terms by three, without the three products below 2^-24, is six matrix products, into sums by their order (0: leading times leading; 1: leading times middle; 2: the others),
// which are added in f32 when they are read, the smallest first. Products are promised to add in the order of their issue where accumulator and shape are the same (PTX ISA, pipelined
// tcgen05 instructions), so no two of them that differ in shape share a column. The scores' leading term times K's leading and middle one is one product of both sums; the other four
// go to the third, with the middle term times the leading one, which belongs to order 1: what the tensor cores cut off there is 2^-8 of what they cut off in order 0. One instruction for each term
// of A on neighbouring blocks of B, in shapes of 192, 128 and 64 columns that overlapped, had a quarter less to read from shared memory, and no promise (us from a graph, so and with these: 1 x 256, 8 heads of 64 9.31 and 9.42;
// 2 x 979 37.7 and 36.4; 4 x 1000, 8 of 32 46.4 and 47.0; 1 x 1024, 16/4 of 128 101.3 and 103.9; six products of one shape for the scores 9.5, 36.6, 47.1, 106.1).
template <int D>
struct Plan {
    static constexpr int kHalves = D == 128 ? 2 : 1;               // blocks of 64 columns (head size 32: half of one, zeros behind)
    static constexpr int kCols = kHalves * 64;                     // columns of a tile of V and of O
    static constexpr int kQHalf = kM * 128, kQPlane = kHalves * kQHalf;
    // K: by half and term (the three terms of 64 columns are neighbouring rows), V: by term and half (neighbouring columns)
    static constexpr int kK = 3 * kQPlane, kV = kK + 3 * kHalves * kBlock, kRed = kV + 3 * kHalves * kBlock;
    static constexpr int kVis = kRed + kMaxBuffers * kShares * kM * 4, kMl = kVis + kMaskBuffers * kN, kAt = kMl + kM * 8, kBar = kAt + kM * 8, kBytes = kBar + 80 + 1024;   // (1024: the planes are aligned to that)
    // Tensor memory: the scores' three sums, the weights' three terms, O's sums. At head size 128 the weights lie over the scores' third sum and behind it, and O's small orders share one.
    static constexpr bool kOver = D == 128;
    static constexpr int kP = kOver ? 2 * kN : 3 * kN, kO = kOver ? 4 * kN : 3 * kN + 3 * kN / 2, kOrders = kOver ? 2 : 3;
    static_assert(kO + kOrders * kCols <= 512, "fits tensor memory");
};

struct Args {
    AttnParams p;
    int* status;
    unsigned long long wait_ns;
    int clusters;   // CTAs that share the keys of a row block
    int o_by_32;
    FastDiv by_group;
};

__device__ __forceinline__ void tc_st8(unsigned taddr, const unsigned (&u)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"r"(taddr), "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]),
                 "r"(u[6]), "r"(u[7])
                 : "memory");
}
__device__ __forceinline__ void tc_ld8(unsigned taddr, float* r) {
    unsigned* u = reinterpret_cast<unsigned*>(r);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tc_ld16(unsigned taddr, float* r) {
    unsigned* u = reinterpret_cast<unsigned*>(r);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]),
                   "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ unsigned peer_addr(unsigned addr, int rank) {
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(a) : "r"(addr), "r"(rank));
    return a;
}
__device__ __forceinline__ float4 peer_float4(unsigned addr) {
    float4 x;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w) : "r"(addr) : "memory");
    return x;
}
__device__ __forceinline__ float2 peer_float2(unsigned addr) {
    float2 x;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];\n" : "=f"(x.x), "=f"(x.y) : "r"(addr) : "memory");
    return x;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;\n" ::: "memory");
}

__device__ __forceinline__ void commit(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}

// What follows the first look of a wait, which suspends for some 8000 clocks: false when the limit has run out, here or for somebody else of the CTA. The wait's code goes to the status word, and
// nobody in the CTA waits any more. A function, or in line where registers come out better so, which is what decides (us from a graph, in line and as a function: 4 x 2048, 8 heads of 128 528.8 and 506; 1 x 1024,
// shared by two CTAs, 56.0 and 57.0; 4 x 1000, 8 of 32 47.1 and 44.8; 2 x 979, 8 of 64 36.4 and 37.3; 8 x 1024 102.4 and 105.0).
__device__ __forceinline__ bool wait_in_line(unsigned bar, unsigned parity, unsigned given_up, long long limit, int* status, int where) {
    const long long t0 = clock64();
#pragma unroll 1
    for (unsigned spin = 1; !mbar_try_wait_at(bar, parity); ++spin) {
        if ((spin & 63u) != 0u) continue;
        if (shared_flag(given_up)) return false;
        if (clock64() - t0 > limit) {
            set_shared_flag(given_up);
            *reinterpret_cast<volatile int*>(status) = where;
            __threadfence_system();
            return false;
        }
    }
    return true;
}
__device__ __noinline__ bool wait_called(unsigned bar, unsigned parity, unsigned given_up, long long limit, int* status, int where) {
    return wait_in_line(bar, parity, given_up, limit, status, where);
}
// The issuer's products, in functions of their own: unrolled among the workers' code their descriptors cost everybody registers (head size 128: 1164 bytes of spill stores, 916 rolled up, 840 so).
// At head size 64 rolled up where they come in for the first time (the scores of clusters, whose CTAs have a tile or two; what reads inputs anew every time: 1 x 256, 8 heads 10.94 us and 10.83) or where that is the
// faster form (the sums; 8 x 1024, 8 heads 102.6 and 101.8; with the scores rolled up as well 104.0).
template <int D, bool kFirst, bool kSmall, bool kRolled>   // the first two sums, the third
__device__ __noinline__ void issue_scores(unsigned tmem, unsigned long long dq, unsigned long long dk, unsigned long long* s_full) {
    using S = Plan<D>;
    const unsigned x = tmem, z = tmem + 2 * kN;
    tc_fence_after();
    if (elect_one()) {
#pragma unroll
        for (int t = 0; t < (kSmall ? 3 : 1); ++t)
#pragma unroll (kRolled ? 1 : D / 16)
            for (int kk = 0; kk < D / 16; ++kk) {
                const unsigned long long q = dq + ((t * S::kQPlane + (kk >> 2) * S::kQHalf + (kk & 3) * 32) >> 4), k = dk + (((kk >> 2) * 3 * kBlock + (kk & 3) * 32) >> 4);
                if (kFirst && t == 0) tc_mma_ss(x, q, k, make_idesc<__nv_bfloat16>(false, 2 * kN), kk > 0);
                if (!kSmall) continue;
#pragma unroll
                for (int u = t == 0 ? 2 : 0; t + u < 3; ++u) tc_mma_ss(z, q, k + (u * kBlock >> 4), make_idesc<__nv_bfloat16>(false, kN), t + kk > 0);
            }
        if (kSmall) commit(s_full);   // (the same lane is elected every time: its products before are behind the barrier as well)
    }
    __syncwarp();
}
template <int D>
__device__ __noinline__ void issue_sums(unsigned tmem, unsigned long long dv, unsigned long long* o_full) {
    using S = Plan<D>;
    const unsigned o0 = tmem + S::kO, o1 = tmem + S::kO + S::kCols, o2 = tmem + S::kO + (S::kOrders - 1) * S::kCols;
    tc_fence_after();
    if (elect_one()) {
#pragma unroll (D == 64 ? 1 : 4)
        for (int kk = 0; kk < 4; ++kk) {
            const unsigned p = tmem + S::kP + kk * 8, p1 = p + kN / 2, p2 = p + kN;
            const unsigned long long v = dv + (kk * 2048 >> 4), v1 = v + (S::kHalves * kBlock >> 4), v2 = v + (2 * S::kHalves * kBlock >> 4);
            tc_mma_ts(o0, p, v, make_idesc<__nv_bfloat16>(true, S::kCols), kk > 0);
            tc_mma_ts(o1, p, v1, make_idesc<__nv_bfloat16>(true, S::kCols), kk > 0);
            tc_mma_ts(o1, p1, v, make_idesc<__nv_bfloat16>(true, S::kCols), true);
            tc_mma_ts(o2, p, v2, make_idesc<__nv_bfloat16>(true, S::kCols), kk > 0 || S::kOrders == 2);
            tc_mma_ts(o2, p1, v1, make_idesc<__nv_bfloat16>(true, S::kCols), true);
            tc_mma_ts(o2, p2, v, make_idesc<__nv_bfloat16>(true, S::kCols), true);
        }
        commit(o_full);
    }
    __syncwarp();
}

// kPlain: contiguous K/V and no key-padding mask (look-ups and mask in the loop cost it registers and a tenth of its instructions).
template <int D, bool kCluster, bool kPlain>
__global__ void __launch_bounds__(kThreads, 1) tile_f32_tcgen05_kernel(const __grid_constant__ Args a) {
    using S = Plan<D>;
    constexpr int kVec = D / 4;                              // float4 of a row
    constexpr int kStep = kWorkers / kVec;                   // rows that the workers move at a time
    constexpr int kLoads = kN / kStep, kQLoads = kM / kStep;
    constexpr int kKeys = kN / kShares, kOut = D / kShares;              // keys of a tile and columns of O that a thread has of its row
    extern __shared__ unsigned char smem_raw[];
    unsigned char* const sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    float(*const red)[kM] = reinterpret_cast<float(*)[kM]>(sm + S::kRed);
    unsigned char* const vis = sm + S::kVis;
    float2* const ml = reinterpret_cast<float2*>(sm + S::kMl);
    long long* const out_at = reinterpret_cast<long long*>(sm + S::kAt);
    unsigned long long* const bars = reinterpret_cast<unsigned long long*>(sm + S::kBar);
    unsigned long long* const s_full = bars;         // issuer -> workers: scores
    unsigned long long* const o_full = bars + 1;     // ... and a tile's O
    unsigned long long* const k_ready = bars + 2;    // workers -> issuer: K's terms are in shared memory
    unsigned long long* const s_free = bars + 3;     // ... the scores have been read
    unsigned long long* const pv_ready = bars + 4;   // ... the weights and V's terms are there, and O has been read
    unsigned long long* const drain = bars + 5;
    unsigned* const tmem_base = reinterpret_cast<unsigned*>(bars + 6);
    volatile int* const given_up = reinterpret_cast<volatile int*>(tmem_base + 1);

    const AttnParams& p = a.p;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int s = blockIdx.z, kvh = blockIdx.y;
    const int group = a.by_group.d;
    const SeqInfo si = seq_info(p, s);
    const int rows = si.q_len * group;
    const int parts = kCluster ? a.clusters : 1, rank = kCluster ? (int)blockIdx.x & (parts - 1) : 0;   // (a power of two)
    const int row0 = (kCluster ? (int)(gridDim.x - 1 - blockIdx.x) >> (31 - __clz(parts)) : (int)(gridDim.x - 1 - blockIdx.x)) * kM;   // latest (longest) rows first
    if (row0 >= rows) return;                                // (all CTAs of a cluster)

    // keys past the last row's position are never visible
    const int last_token = a.by_group.div(min(rows, row0 + kM) - 1);
    const int kv_end = (int)max(0LL, min((long long)si.kv_len, (long long)si.pos_off + last_token + 1));
    const int tiles = (kv_end + kN - 1) / kN;
    const int per = kCluster ? (tiles + parts - 1) >> (31 - __clz(parts)) : tiles;
    const int first = rank * per, n = max(0, min(tiles, first + per) - first);   // this CTA's tiles
    const uint8_t* const mask_row = !kPlain && p.mask ? p.mask + (long long)s * p.kv_seq_len : nullptr;
    const float scale = p.scale * 1.4426950408889634f;

    // Bounded: the wait's code goes to the status word, and nobody in the CTA waits any more.
    constexpr bool kWaitInLine = D == 64 || (D == 128 && kCluster);
    auto wait = [&](unsigned long long* bar, unsigned parity, int where) {
        if (mbar_try_wait(bar, parity)) return true;
        const auto on = kWaitInLine ? wait_in_line : wait_called;
        return on(smem_u32(bar), parity, smem_u32((const void*)given_up), (long long)(a.wait_ns * 2ULL), a.status, where);
    };

    float acc[kOut], m = -INFINITY, l = 0.0f;   // of this thread's row: its columns of O, the maximum of the raw scores so far, the sum over its keys
    float u = 0.0f;                             // the reference: that maximum, scaled and rounded (0 until a key has been seen)
    const int quad = warp & 3, part = warp >> 2;   // tensor memory lanes 32 * quad ..., which quarter of keys and columns
    const int r = quad * 32 + lane, row = row0 + r, token = a.by_group.div(row), head = kvh * group + row - token * group;
    const long long pos = (long long)si.pos_off + token;
#pragma unroll
    for (int i = 0; i < kOut; ++i) acc[i] = 0.0f;

    if (warp == kWarps) {
        // ------------------------------ issuer ------------------------------
        if (lane == 0) {
            mbar_init(s_full, 1);
            mbar_init(o_full, 1);
            mbar_init(k_ready, kWarps);
            mbar_init(s_free, kWarps);
            mbar_init(pv_ready, kWarps);
            mbar_init(drain, 1);
            *given_up = 0;
            asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        }
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(smem_u32(tmem_base)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        const unsigned tmem = __shfl_sync(0xffffffffu, *tmem_base, 0), base = __shfl_sync(0xffffffffu, smem_u32(sm), 0);
        const unsigned long long dq = make_desc(base, 16, 1024), dk = make_desc(base + S::kK, 16, 1024), dv = make_desc(base + S::kV, kBlock, 1024);
        auto scores = [&]() { issue_scores<D, true, true, D == 64 && kCluster>(tmem, dq, dk, s_full); };
        auto sums = [&]() { issue_sums<D>(tmem, dv, o_full); };
        bool alive = n == 0 || __all_sync(0xffffffffu, wait(k_ready, 0u, 60));
        if (alive && n > 0) scores();
#pragma unroll 1
        for (int j = 0; j < n && alive; ++j) {
            const unsigned phase = (unsigned)j & 1u;
            const bool more = j + 1 < n;
            if (!S::kOver && more) {
                alive = __all_sync(0xffffffffu, wait(k_ready, phase ^ 1u, 61) && wait(s_free, phase, 62));
                if (!alive) break;
                scores();
            }
            alive = __all_sync(0xffffffffu, wait(pv_ready, phase, 63));
            if (!alive) break;
            sums();
            if (S::kOver && more) {
                // The third sum goes over the weights that sums() reads, and no order is promised there: it waits for their product. Behind the first two sums' products, or in a cluster with
                // them (us from a graph: 4 x 2048, 8 heads 506 and 517; 1 x 1024, shared by two CTAs, 57.7 and 56.9; without the wait 523 with more spills, and 55.2)
                alive = __all_sync(0xffffffffu, wait(k_ready, phase ^ 1u, 64) && (!kCluster || wait(o_full, phase, 65)));
                if (!alive) break;
                if (!kCluster) {
                    issue_scores<D, true, false, false>(tmem, dq, dk, s_full);
                    alive = __all_sync(0xffffffffu, wait(o_full, phase, 65));
                    if (!alive) break;
                }
                issue_scores<D, kCluster, true, false>(tmem, dq, dk, s_full);
            }
        }
    } else {
        // ------------------------------ workers ------------------------------
        const float* __restrict__ qg = static_cast<const float*>(p.q);
        const int vec = tid % kVec, at_row = tid / kVec;   // of a tile, this thread moves four columns of rows at_row, + kStep, ...
        const long long pitch = (long long)p.kv_heads * D, col = (long long)kvh * D + vec * 4;
        const long long in_seq = si.kv_row0 * pitch + col;
        auto fetch = [&](const void* base, float4 (&x)[kLoads], int tile, bool is_v) {
            const int key0 = tile * kN + at_row;
            const float* const from = static_cast<const float*>(base);
#pragma unroll
            for (int i = 0; i < kLoads; ++i) {
                const int key = key0 + i * kStep;
                x[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                // a padded key's weight is an exact zero, but zero times what may lie in its row of V need not be
                if (key < kv_end && (!is_v || mask_row == nullptr || mask_row[key] != 0))
                    x[i] = __ldg(reinterpret_cast<const float4*>(from + (!kPlain && p.paged ? block_slot(p.block_tables, s, p.max_blocks, key, p.block_size) * pitch + col : key * pitch + in_seq)));
            }
        };
        // Four columns of a row into the three terms' planes: 64 columns are 128 bytes, 16-byte chunks swizzled by the row.
        auto put = [&](unsigned at, int plane_bytes, int of_row, const float4& x) {
            unsigned h0, m0, l0, h1, m1, l1;
            split3(x.x, x.y, h0, m0, l0);
            split3(x.z, x.w, h1, m1, l1);
            at += of_row * 128 + ((((vec & 15) >> 1) ^ (of_row & 7)) << 4) + (vec & 1) * 8;
            asm volatile("st.shared.v2.b32 [%0], {%1, %2};\n" ::"r"(at), "r"(h0), "r"(h1) : "memory");
            asm volatile("st.shared.v2.b32 [%0], {%1, %2};\n" ::"r"(at + plane_bytes), "r"(m0), "r"(m1) : "memory");
            asm volatile("st.shared.v2.b32 [%0], {%1, %2};\n" ::"r"(at + 2 * plane_bytes), "r"(l0), "r"(l1) : "memory");
        };
        const unsigned base = smem_u32(sm), half_of = vec >> 4;
        auto put_k = [&](const float4 (&x)[kLoads]) {
#pragma unroll
            for (int i = 0; i < kLoads; ++i) put(base + S::kK + half_of * 3 * kBlock, kBlock, at_row + i * kStep, x[i]);
        };
        auto put_v = [&](const float4 (&x)[kLoads]) {
#pragma unroll
            for (int i = 0; i < kLoads; ++i) put(base + S::kV + half_of * kBlock, S::kHalves * kBlock, at_row + i * kStep, x[i]);
        };
        auto put_vis = [&](int tile) {
            if (mask_row != nullptr && tid < kN) vis[(tile & (kMaskBuffers - 1)) * kN + tid] = tile * kN + tid < kv_end ? mask_row[tile * kN + tid] : 0;
        };
        auto tell = [&](unsigned long long* bar) {   // what this warp has done before is seen by the issuer and the products
            __syncwarp();
            if (lane == 0) mbar_arrive(bar);
        };

        float4 kr[kLoads], vr[kLoads];
        {
            float4 q[kQLoads];
#pragma unroll
            for (int i = 0; i < kQLoads; ++i) {
                const int rr = row0 + at_row + i * kStep, t = a.by_group.div(rr);
                q[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (rr < rows) q[i] = __ldg(reinterpret_cast<const float4*>(qg + ((si.q_row0 + t) * p.q_heads + kvh * group + rr - t * group) * D + vec * 4));
            }
            if (n > 0) {
                fetch(p.k, kr, first, false);
                fetch(p.v, vr, first, true);
                put_vis(first);
            }
#pragma unroll
            for (int i = 0; i < kQLoads; ++i) put(base + half_of * S::kQHalf, S::kQPlane, at_row + i * kStep, q[i]);
        }
        if (n > 0) {
            put_k(kr);
            if (n > 1) fetch(p.k, kr, first + 1, false);
        }
        if (D == 32)   // the other half of V's columns: zeros
            for (int idx = tid; idx < 3 * kN * 8; idx += kWorkers) {
                const int term = idx / (kN * 8), of_row = idx / 8 % kN, c = idx % 8;
                if ((c ^ (of_row & 7)) >= 4) *reinterpret_cast<uint4*>(sm + S::kV + term * kBlock + of_row * 128 + c * 16) = make_uint4(0u, 0u, 0u, 0u);
            }
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");   // the products read what was written
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        tell(k_ready);
        const unsigned mine = *tmem_base + ((unsigned)(quad * 32) << 16);

        const int lim = (int)max(-1LL, min((long long)si.kv_len - 1, pos));
        const int all_see = (int)max(0LL, min((long long)si.kv_len, (long long)si.pos_off + a.by_group.div(row0) + 1));   // keys below: seen by every row
        // After a wait that ran out, the workers go through the rest of their steps without waiting: their warps meet at barriers of their own.
        auto wait_warp = [&](unsigned long long* bar, unsigned parity, int where) {
            wait(bar, parity, where);
            __syncwarp();
        };
        float alpha = 1.0f;
        // O of a tile, smallest orders first, onto the running output (rescaled by the alpha of its tile)
        auto add_o = [&](float by) {
            const unsigned from = mine + S::kO + part * kOut;
#pragma unroll
            for (int c = 0; c < kOut; c += (kOut < 16 ? 8 : 16)) {
                constexpr int kAt = kOut < 16 ? 8 : 16;
                float x[S::kOrders][kAt];
#pragma unroll
                for (int o = 0; o < S::kOrders; ++o) {
                    if constexpr (kAt == 8) tc_ld8(from + o * S::kCols + c, x[o]);
                    else tc_ld16(from + o * S::kCols + c, x[o]);
                }
                tc_wait_ld();
#pragma unroll
                for (int i = 0; i < kAt; ++i) {
                    float small = x[S::kOrders - 1][i];
                    if (S::kOrders == 3) small += x[1][i];
                    acc[c + i] = fmaf(acc[c + i], by, x[0][i] + small);
                }
            }
        };
#pragma unroll 1
        for (int j = 0; j < n; ++j) {
            const unsigned phase = (unsigned)j & 1u;
            const int tile = first + j;
            wait_warp(s_full, phase, 70);
            tc_fence_after();
            float sc[kKeys];
            {
                float x1[kKeys], x2[kKeys];
                tc_ld16(mine + 2 * kN + part * kKeys, x2);
                tc_ld16(mine + kN + part * kKeys, x1);
                tc_ld16(mine + part * kKeys, sc);
                tc_wait_ld();
#pragma unroll
                for (int i = 0; i < kKeys; ++i) sc[i] += x1[i] + x2[i];
            }
            tc_fence_before();
            if (!S::kOver) tell(s_free);
            if (j + 1 < n) {
                put_vis(tile + 1);
                put_k(kr);
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                tell(k_ready);
                if (j + 2 < n) fetch(p.k, kr, tile + 2, false);
            }
            const int key0 = tile * kN + part * kKeys;
            if (tile * kN + kN > all_see || mask_row != nullptr) {
#pragma unroll
                for (int i = 0; i < kKeys; ++i)
                    if (key0 + i > lim || (mask_row != nullptr && vis[(tile & (kMaskBuffers - 1)) * kN + part * kKeys + i] == 0)) sc[i] = -INFINITY;
            }
            float mx4[4] = {m, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int i = 0; i < kKeys; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], sc[i]);
            float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
            float(*const maxima)[kM] = red + (j & 1) * kShares;
            maxima[part][r] = mx;
            asm volatile("barrier.cta.sync %0, 128;\n" ::"r"(1 + quad) : "memory");   // the warps of these rows (which have read their scores)
            if (S::kOver) tc_fence_after();   // their loads come before this warp's weights, which go where the scores lie (tile 0 has no other fence until then)
            mx = fmaxf(fmaxf(maxima[0][r], maxima[1][r]), fmaxf(maxima[2][r], maxima[3][r]));
            const float before = u, by = alpha;
            u = mx == -INFINITY ? 0.0f : __fmul_rn(mx, scale);
            alpha = m == -INFINITY ? 0.0f : ex2(before - u);   // 1 exactly while the maximum stays
            m = mx;
            float sum4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int i = 0; i < kKeys; ++i) {
                sc[i] = ex2(fmaf(sc[i], scale, -u));
                sum4[i & 3] += sc[i];
            }
            l = l * alpha + ((sum4[0] + sum4[1]) + (sum4[2] + sum4[3]));
            if (j > 0) {
                wait_warp(o_full, phase ^ 1u, 71);   // the weights' place and V's are free, O can be read
                tc_fence_after();
                add_o(by);
            }
            put_v(vr);
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            if (j + 1 < n) fetch(p.v, vr, tile + 1, true);
            {
                unsigned hi[kKeys / 2], mid[kKeys / 2], lo[kKeys / 2];
#pragma unroll
                for (int i = 0; i < kKeys / 2; ++i) split3(sc[2 * i], sc[2 * i + 1], hi[i], mid[i], lo[i]);
                const unsigned to = mine + S::kP + part * kKeys / 2;
                tc_st8(to, hi);
                tc_st8(to + kN / 2, mid);
                tc_st8(to + kN, lo);
            }
            tc_wait_st();
            tc_fence_before();
            tell(pv_ready);
        }
        if (n > 0) {
            wait_warp(o_full, (unsigned)(n - 1) & 1u, 72);
            tc_fence_after();
            add_o(alpha);
        }
        __syncwarp();
        asm volatile("barrier.cta.sync %0, 128;\n" ::"r"(1 + quad) : "memory");   // (the maxima have been read)
        red[part][r] = l;
        tc_fence_before();
    }

    // ---- the end: the row's sum, then the shares of the cluster -------------------------------------------
    float probe = 0.0f * l;   // NaN where any of the sums is not finite
#pragma unroll
    for (int i = 0; i < kOut; ++i) probe = fmaf(0.0f, acc[i], probe);
    const bool again = __syncthreads_or(probe != 0.0f);
    const bool left = *given_up != 0;
    if (warp == kWarps) {   // every product issued has finished before tensor memory goes (bounded; the tensor pipe alone decides)
        tc_fence_after();
        if (left) {
            if (elect_one()) commit(drain);
            __syncwarp();
            const unsigned long long t0 = global_timer_ns();
            while (!mbar_try_wait(drain, 0u) && global_timer_ns() - t0 < 100000000ULL) {}
        }
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;\n" ::"r"(*tmem_base) : "memory");
    }
    // with a padding mask a query row at a padded (or out-of-range) position outputs zeros (flash_attn_func.cu:77-84)
    const bool counts = row < rows && (mask_row == nullptr || (pos >= 0 && pos < si.kv_len && mask_row[pos] != 0));
    const long long o_at = ((si.q_row0 + token) * p.q_heads + head) * D, lse_at = ((long long)s * p.q_heads + head) * p.q_seq_len + token;

    if (!kCluster) {
        if (left || warp == kWarps) return;
        if (again) {
            plain_rows<D, kWarps>(p, s, kvh, row0, min(rows, row0 + kM));
            return;
        }
        if (row >= rows) return;
        l = (red[0][r] + red[1][r]) + (red[2][r] + red[3][r]);
        const bool ok = l > 0.0f && counts;
        const float inv = ok ? 1.0f / l : 0.0f;
#pragma unroll
        for (int i = 0; i < kOut; ++i) acc[i] = ok ? quotient(acc[i], l, inv) : 0.0f;
        float* const to = static_cast<float*>(p.o) + o_at + part * kOut;
#pragma unroll
        for (int i = 0; i < kOut; i += 8) {
            if (a.o_by_32) {
                asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"l"(to + i), "f"(acc[i]), "f"(acc[i + 1]), "f"(acc[i + 2]),
                             "f"(acc[i + 3]), "f"(acc[i + 4]), "f"(acc[i + 5]), "f"(acc[i + 6]), "f"(acc[i + 7])
                             : "memory");
            } else {
                *reinterpret_cast<float4*>(to + i) = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
                *reinterpret_cast<float4*>(to + i + 4) = make_float4(acc[i + 4], acc[i + 5], acc[i + 6], acc[i + 7]);
            }
        }
        if (p.lse != nullptr && part == 0) p.lse[lse_at] = ok ? (u + log2f(l)) * 0.6931471805599453f : -INFINITY;
        return;
    }

    // Every CTA lays its rows down where its tiles were, and finishes a share of the rows from all of them.
    float* const laid = reinterpret_cast<float*>(sm);   // (kM, D), 16-byte chunks swizzled by the row
    constexpr int kChunks = D / 4;
    if (warp < kWarps) {
#pragma unroll
        for (int i = 0; i < kOut; i += 4) {
            const int c = part * (kOut / 4) + i / 4;
            *reinterpret_cast<float4*>(laid + r * D + ((c ^ (r & 7)) << 2)) = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
        }
        if (part == 0) {
            ml[r] = make_float2(m == -INFINITY ? m : u, again || left ? NAN : (red[0][r] + red[1][r]) + (red[2][r] + red[3][r]));
            out_at[r] = counts ? o_at : -1 - o_at;   // (rows that count for nothing: zeros)
        }
    }
    cluster_sync();
    const int share = kM / parts, r_begin = rank * share, r_end = min(r_begin + share, rows - row0);
    bool spoilt = false;   // by what one of the CTAs met
    if (warp < kWarps) {
        const int c = tid % kChunks;
        for (int rr = r_begin + tid / kChunks; rr < r_end; rr += kWorkers / kChunks) {
            const unsigned ml_at = smem_u32(ml + rr), acc_at = smem_u32(laid + rr * D + ((c ^ (rr & 7)) << 2));
            float2 x[8];
            float4 y[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                x[k] = make_float2(-INFINITY, 0.0f);
                y[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (k < parts) {
                    x[k] = peer_float2(peer_addr(ml_at, k));
                    y[k] = peer_float4(peer_addr(acc_at, k));
                }
            }
            float top = -INFINITY, sum = 0.0f;
#pragma unroll
            for (int k = 0; k < 8; ++k) top = fmaxf(top, x[k].x);
            float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float w = x[k].x == -INFINITY ? 0.0f : ex2(x[k].x - top);
                sum = x[k].x == -INFINITY && !isnan(x[k].y) ? sum : fmaf(w, x[k].y, sum);
                o.x = fmaf(w, y[k].x, o.x);
                o.y = fmaf(w, y[k].y, o.y);
                o.z = fmaf(w, y[k].z, o.z);
                o.w = fmaf(w, y[k].w, o.w);
            }
            spoilt = spoilt || isnan(sum);
            const long long at = out_at[rr], to = at < 0 ? -1 - at : at;
            const bool ok = sum > 0.0f && at >= 0;
            const float inv = ok ? 1.0f / sum : 0.0f;
            *reinterpret_cast<float4*>(static_cast<float*>(p.o) + to + c * 4) = ok ? make_float4(quotient(o.x, sum, inv), quotient(o.y, sum, inv), quotient(o.z, sum, inv), quotient(o.w, sum, inv)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (p.lse != nullptr && c == 0) {
                const int t = a.by_group.div(row0 + rr);
                p.lse[((long long)s * p.q_heads + kvh * group + row0 + rr - t * group) * p.q_seq_len + t] = ok ? (top + log2f(sum)) * 0.6931471805599453f : -INFINITY;
            }
        }
    }
    spoilt = __syncthreads_or(spoilt);
    cluster_sync();   // nobody's shared memory goes while another reads it
    if (spoilt && warp < kWarps) plain_rows<D, kWarps>(p, s, kvh, row0 + r_begin, row0 + r_end);
}

template <int D, bool kCluster, bool kPlain>
int launch_one(const AttnParams& p, int clusters, cudaStream_t stream) {
    using S = Plan<D>;
    static std::atomic<unsigned long long> ready{0};   // devices whose copy of this kernel has its shared-memory limit raised
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err == cudaSuccess && (dev >= 64 || !((ready.load(std::memory_order_acquire) >> dev) & 1ULL))) {
        err = cudaFuncSetAttribute(tile_f32_tcgen05_kernel<D, kCluster, kPlain>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kBytes);
        if (err == cudaSuccess && dev < 64) ready.fetch_or(1ULL << dev, std::memory_order_release);
    }
    if (err != cudaSuccess) {
        set_last_errorf("tile_f32_tcgen05_kernel: %s", cudaGetErrorString(err));
        cudaGetLastError();
        return FLASH_ATTN_ERR_CUDA;
    }
    Args a{};
    a.p = p;
    a.status = prefill_status_word();
    if (a.status == nullptr) return -1;
    a.wait_ns = get_option_prefill_wait_us() > 0 ? (unsigned long long)get_option_prefill_wait_us() * 1000ULL : 2000000000ULL;
    a.clusters = clusters;
    a.o_by_32 = (reinterpret_cast<uintptr_t>(p.o) & 31) == 0;
    a.by_group = FastDiv(p.q_heads / p.kv_heads);
    const long long rows = (long long)p.q_seq_len * (p.q_heads / p.kv_heads);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)((rows + kM - 1) / kM * clusters), (unsigned)p.kv_heads, (unsigned)p.num_seqs);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = S::kBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)clusters;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = kCluster ? 1 : 0;
    cudaLaunchKernelEx(&cfg, tile_f32_tcgen05_kernel<D, kCluster, kPlain>, a);
    const int rc = check_launch("tile_f32_tcgen05_kernel");
    if (rc == FLASH_ATTN_OK) note_path("tile_f32", 1, clusters == 8 ? "tcgen05 cluster 8" : clusters == 4 ? "tcgen05 cluster 4" : clusters == 2 ? "tcgen05 cluster 2" : "tcgen05");
    return rc;
}

template <int D>
int launch_for(const AttnParams& p, cudaStream_t stream) {
    const long long rows = (long long)p.q_seq_len * (p.q_heads / p.kv_heads), streams = (long long)p.kv_heads * p.num_seqs;
    const long long blocks = (rows + kM - 1) / kM * streams;
    const long long keys = p.mode == MODE_KVCACHE ? (long long)p.max_blocks * p.block_size : p.kv_seq_len;
    const long long tiles = (keys + kN - 1) / kN;
    // Few blocks: the keys of each are shared out over a cluster of 2, 4 or 8 CTAs, as long as all clusters find room at the same time, with a tile for each CTA. us with
    // one CTA to a block and so: 1 x 256, 8 heads of 64 15.5 and 9.2; 1 x 512, 8 of 32 19.2 and 9.6; 3 x 552, 8/2 heads of 64 (54 blocks, 9 tiles) 26.3 either way. 36 blocks in clusters of four, some of which
    // had to wait for a place, and of two: 1 x 280, 16/4 heads of 64 17.8 and 13.7, of 32 14.4 and 10.8.
    const int c = f32_parts(blocks, tiles, sm_count());
    // The other kernel (tile_f32.cu) keeps what leaves this one's 128 rows empty with a CTA to a block (us there and here: 32 x 1 token over 600, 8 heads of 64 29 and 52; 64 x 4 over
    // 512 81 and 94; 1 x 4 over 4096, 32/8 heads, shared by 8 CTAs 123 and 23), and problems of up to three tiles that give it a CTA of 16 rows (32 at head size 128) for
    // about every SM, which have no time to win back this one's set-up (2 x 113, 8/2 heads of 64 7.9 and 9.4; 1 x 192, 8 of 64 10.4 and 11.3; 2 x 91, 16/4 of 128 14.0 and
    // 14.5; at head size 32 up to 2.2 for an SM: 4 x 128, 8 heads 6.4 and 7.9; 4 x 73, 16/4 6.7 and 7.8; 4 x 160, 8/2 8.7 and 9.2, 8/8 9.7 and 8.8; 3 x 160 7.7 and 10.0; 3 x 95, 16/4 6.4 and 7.8; 4 x 96, 2.6 of them, 9.3 and 8.0; but 4 x 130, 16/4 of 64, 3.5 CTAs for an SM, 17.4 and 11.5; 1 x 160, 8 of 128 19.9 and 18.7).
    // Two tiles of head size 64 up to 1.65 for an SM (3 x 80, 16/4 9.3 and 9.8; with 1.7 of them 4 x 128, 8 heads the same; with 2 of them 3 x 97, 16/4 11.0 and 9.8), one tile up to as many rounds of two CTAs to an SM there as of one here
    // (4 x 64, 16/4 of 64 7.2 and 8.3; 24 x 48, 8 of 64 12.6 and 14.0, of 32 8.3 and 10.8), and at head size 32 up to five tiles where it has a CTA for each SM at most (1 x 200, 8 heads 7.0 and 7.7; 1 x 256 7.8 and 8.0; 1 x 280, 8/2 8.8 and 9.3; but with 160 of its CTAs 1 x 320, 8 heads 10.4 and 9.3, with 200
    // 1 x 200, 16/4 9.0 and 8.0).
    const long long small = (rows + (D == 128 ? 31 : 15)) / (D == 128 ? 32 : 16) * streams, sms = sm_count();
    const bool one_round = 20 * small <= (D == 32 ? 44 : D == 64 && tiles == 2 ? 33 : 30) * sms;
    if ((rows <= 16 && c == 1) || (tiles <= (D < 128 ? 3 : 2) && one_round) || (D < 128 && tiles == 1 && (small + 2 * sms - 1) / (2 * sms) <= (blocks + sms - 1) / sms) || (D == 32 && tiles <= 5 && small <= sms)) return -1;
    const bool plain = p.mask == nullptr && !p.paged;
    if (c > 1) return plain ? launch_one<D, true, true>(p, c, stream) : launch_one<D, true, false>(p, c, stream);
    return plain ? launch_one<D, false, true>(p, 1, stream) : launch_one<D, false, false>(p, 1, stream);
}

}  // namespace

int launch_tile_f32_tcgen05(const AttnParams& p, cudaStream_t stream) {
    return p.head_size == 128 ? launch_for<128>(p, stream) : p.head_size == 64 ? launch_for<64>(p, stream) : launch_for<32>(p, stream);
}

}  // namespace fa
