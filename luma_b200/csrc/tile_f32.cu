// f32 storage on the tensor cores without giving up f32 (the splitting is that of Henry, Tang and Heinecke, "Leveraging the
// bfloat16 Artificial Intelligence Datatype For Higher-Precision Computations", 2019): every operand is split into three bf16 terms that together
// hold its 24 bits (x = hi + mid + lo exactly, each term the rounded rest of the one before), and a product of two
// operands is the six term products of at least 2^-16 of the largest (hi hi, hi mid, mid hi, mid mid, hi lo,
// lo hi; what is left out is below 2^-24). Replaces the scalar kernel (tile_simt.cu) for f32 tensors through the
// batched, packed and chunked-prefill entry points: flash_attn_kernel (luma-flash-attn/kernels/flash_attn_func.cu:29-226),
// flash_attn_varlen_kernel (kernels/flash_attn_varlen_func.cu:35-199), flash_attn_prefill_kernel
// (kernels/flash_attn_with_kvcache.cu:157-277).
//
// The tensor cores truncate when they add into an f32 accumulator, a bias that would grow with the number of keys. So
// sums start from zero in every K/V tile, small terms first, and a tile's sum is added to the running output with an
// ordinary rounded f32 addition: fewer roundings per result than one fused multiply-add per key has. Measured against
// f64 (causal, N(0,1), 256-1500 tokens, norm by norm over all rows): relative error 1.1-1.9e-7 where the scalar kernel has 2.0-3.9e-7.
// What bounds it: the dependent products of a score or output block (one warp or two per scheduler), then the splitting of
// the tiles. B=1, H=8, S=256, d=64: 88 -> 13 us; B=1, S=718, 8/2 heads, d=32: 164 -> 22.5; B=2, S=509, 16/4 heads, d=128:
// 337 -> 88 us (scalar kernel -> this one, per call).
//
// A CTA of four warps owns 16 * WR query rows that share a KV head (row = query token x group + head in the group)
// and walks the K/V tiles they see. Tiles come in as f32 (registers, one tile ahead), are split once for all
// rows and lie in shared memory as three bf16 planes each, XOR-swizzled for ldmatrix. WR = 4: a warp per 16 rows. Small
// problems leave most SMs without a CTA that way; there a CTA takes 16 or 32 rows and WK = 4 / WR warps share the keys
// of every tile, merging with log-sum-exp weights at the end.
#include <atomic>

#include "common.cuh"
#include "tile_f32.cuh"

namespace fa {

namespace {

constexpr int kThreads = 128;
constexpr int kWarps = 4;

template <int D, int WR>
struct Shape {
    static constexpr int kWk = kWarps / WR;                        // warps that share the keys of a tile
    static constexpr int kRows = 16 * WR;
    static constexpr int kKeys = D == 128 ? 32 : 64;               // keys per tile: 16 KiB of f32 K and V each, 64 registers per thread in flight
    static constexpr int kKeysPerWarp = kKeys / kWk;
    static constexpr int kRowBytes = D * 2;
    static constexpr int kSwz = (D / 8 - 1) < 7 ? (D / 8 - 1) : 7;
    static constexpr int kPlane = kKeys * kRowBytes;
    static constexpr int kQPlane = kRows * kRowBytes;
    static constexpr int kKvBytes = 6 * kPlane;
    static constexpr int kMergeBytes = kWk > 1 ? kWarps * 16 * (D + 2) * 4 : 0;
    static constexpr int kTileBytes = kKvBytes > kMergeBytes ? kKvBytes : kMergeBytes;
    static constexpr int kBytes = kTileBytes + 3 * kQPlane + kKeys;   // ... and the tile's padding-mask bytes
    static_assert(kKeysPerWarp % 16 == 0, "P.V takes 16 keys per product");
};

__device__ __forceinline__ void ldmatrix_x4(unsigned& r0, unsigned& r1, unsigned& r2, unsigned& r3, const void* smem) {
    const unsigned saddr = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(saddr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(unsigned& r0, unsigned& r1, unsigned& r2, unsigned& r3, const void* smem) {
    const unsigned saddr = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(saddr));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <int D, int WR>
__global__ void __launch_bounds__(kThreads, 2) tile_f32_kernel(const __grid_constant__ AttnParams p) {
    using S = Shape<D, WR>;
    constexpr int kNb = S::kKeysPerWarp / 8;       // blocks of 8 keys a warp scores per tile
    constexpr int kVec = D / 4;                    // float4 per K/V row
    constexpr int kLoads = S::kKeys * kVec / kThreads;
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char* const kp = smem;                       // K planes hi, mid, lo
    unsigned char* const vp = smem + 3 * S::kPlane;       // V planes
    unsigned char* const qp = smem + S::kTileBytes;       // Q planes
    unsigned char* const vis = qp + 3 * S::kQPlane;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int wr = warp / S::kWk, wk = warp % S::kWk;
    const int g = lane >> 2, c4 = lane & 3;
    const int s = blockIdx.z, kvh = blockIdx.y;
    const int group = p.q_heads / p.kv_heads;
    const SeqInfo si = seq_info(p, s);
    const int rows = si.q_len * group;
    const int row0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * S::kRows;   // latest (longest) rows first
    if (row0 >= rows) return;

    const float* __restrict__ qg = static_cast<const float*>(p.q);
    const float* __restrict__ kg = static_cast<const float*>(p.k);
    const float* __restrict__ vg = static_cast<const float*>(p.v);
    float* __restrict__ og = static_cast<float*>(p.o);
    const long long kv_pitch = (long long)p.kv_heads * D;
    const uint8_t* mask_row = p.mask ? p.mask + (long long)s * p.kv_seq_len : nullptr;

    // keys past the last row's position are never visible
    const int last_token = (min(rows, row0 + S::kRows) - 1) / group;
    const int kv_end = (int)max(0LL, min((long long)si.kv_len, (long long)si.pos_off + last_token + 1));

    // One tile ahead in registers: thread t moves float4 t % kVec of keys t / kVec, + kThreads / kVec, ...
    float4 kr[kLoads], vr[kLoads];
    auto fetch = [&](int key0) {
#pragma unroll
        for (int i = 0; i < kLoads; ++i) {
            const int j = key0 + (i * kThreads + tid) / kVec;
            kr[i] = vr[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (j < kv_end) {
                const long long row = p.paged ? (long long)block_slot(p.block_tables, s, p.max_blocks, j, p.block_size) : si.kv_row0 + j;
                const long long off = row * kv_pitch + (long long)kvh * D + (tid % kVec) * 4;
                kr[i] = *reinterpret_cast<const float4*>(kg + off);
                // a padded key's weight is an exact zero, but zero times what may lie there need not be
                if (mask_row == nullptr || mask_row[j] != 0) vr[i] = *reinterpret_cast<const float4*>(vg + off);
            }
        }
    };
    auto put = [&](unsigned char* plane0, int plane_bytes, int row, int vec, const float4& x) {
        unsigned h0, m0, l0, h1, m1, l1;
        split3(x.x, x.y, h0, m0, l0);
        split3(x.z, x.w, h1, m1, l1);
        const int at = row * S::kRowBytes + (((vec >> 1) ^ (row & S::kSwz)) << 4) + (vec & 1) * 8;
        *reinterpret_cast<uint2*>(plane0 + at) = make_uint2(h0, h1);
        *reinterpret_cast<uint2*>(plane0 + plane_bytes + at) = make_uint2(m0, m1);
        *reinterpret_cast<uint2*>(plane0 + 2 * plane_bytes + at) = make_uint2(l0, l1);
    };
    fetch(0);
    for (int idx = tid; idx < S::kRows * kVec; idx += kThreads) {
        const int r = idx / kVec, vec = idx % kVec;
        float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (row0 + r < rows) {
            const int t = (row0 + r) / group, h = kvh * group + (row0 + r) - t * group;
            x = *reinterpret_cast<const float4*>(qg + ((si.q_row0 + t) * p.q_heads + h) * D + vec * 4);
        }
        put(qp, S::kQPlane, r, vec, x);
    }

    // the two rows of this lane: their position, whether they exist
    const int r0 = row0 + wr * 16 + g, r1 = r0 + 8;
    const int t0 = r0 / group, t1 = r1 / group;
    const long long pos0 = (long long)si.pos_off + t0, pos1 = (long long)si.pos_off + t1;
    const int lim0 = (int)max(-1LL, min((long long)si.kv_len - 1, pos0)), lim1 = (int)max(-1LL, min((long long)si.kv_len - 1, pos1));
    const int warp_last = min(rows - 1, row0 + wr * 16 + 15) / group;     // this warp's last token
    const long long warp_end = min((long long)kv_end, (long long)si.pos_off + warp_last + 1);
    const int all_see = (int)max(0LL, min((long long)si.kv_len, (long long)si.pos_off + (row0 + wr * 16) / group + 1));   // keys below: seen by every row

    float acc[D / 8][4];
#pragma unroll
    for (int n = 0; n < D / 8; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0f;
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.0f, l1 = 0.0f;
    const float scale = p.scale * 1.4426950408889634f;

    for (int key0 = 0; key0 < kv_end; key0 += S::kKeys) {
        __syncthreads();   // the tile before this one has been read
#pragma unroll
        for (int i = 0; i < kLoads; ++i) {
            const int row = (i * kThreads + tid) / kVec;
            put(kp, S::kPlane, row, tid % kVec, kr[i]);
            put(vp, S::kPlane, row, tid % kVec, vr[i]);
        }
        if (mask_row != nullptr && tid < S::kKeys) vis[tid] = key0 + tid < kv_end ? mask_row[key0 + tid] : 0;
        __syncthreads();
        if (key0 + S::kKeys < kv_end) fetch(key0 + S::kKeys);

        const int first = wk * S::kKeysPerWarp;        // this warp's keys within the tile
        if ((long long)key0 + first >= warp_end || row0 + wr * 16 >= rows) continue;

        // ---- scores: 16 rows x kKeysPerWarp keys --------------------------------------------------------
        float sc[kNb][4];
#pragma unroll
        for (int nb = 0; nb < kNb; ++nb) sc[nb][0] = sc[nb][1] = sc[nb][2] = sc[nb][3] = 0.0f;
        {
            const int mi = lane >> 3;
            const int q_row = wr * 16 + ((mi & 1) << 3) + (lane & 7);   // A: rows 0-7 / 8-15 of k 0-7, then of k 8-15
            const int k_row = ((mi >> 1) << 3) + (lane & 7);            // B: tokens 0-7 with k 0-7 / 8-15, then tokens 8-15
            // small terms first, the product of the two hi terms last
#pragma unroll
            for (int pass = 0; pass < 2; ++pass)
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk) {
                    unsigned qa[3][4];
#pragma unroll
                    for (int t = 0; t < (pass == 0 ? 3 : 1); ++t)
                        ldmatrix_x4(qa[t][0], qa[t][1], qa[t][2], qa[t][3],
                                    qp + t * S::kQPlane + q_row * S::kRowBytes + (((2 * kk + (mi >> 1)) ^ (q_row & S::kSwz)) << 4));
#pragma unroll
                    for (int nb = 0; nb < kNb; nb += 2) {
                        const int row = first + nb * 8 + k_row;
                        const int at = row * S::kRowBytes + (((2 * kk + (mi & 1)) ^ (row & S::kSwz)) << 4);
                        unsigned b[3][4];
#pragma unroll
                        for (int t = 0; t < (pass == 0 ? 3 : 1); ++t)
                            ldmatrix_x4(b[t][0], b[t][1], b[t][2], b[t][3], kp + t * S::kPlane + at);
                        if (pass == 0) {
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                mma_bf16(sc[nb + h], qa[2], b[0][2 * h], b[0][2 * h + 1]);
                                mma_bf16(sc[nb + h], qa[1], b[1][2 * h], b[1][2 * h + 1]);
                                mma_bf16(sc[nb + h], qa[0], b[2][2 * h], b[2][2 * h + 1]);
                                mma_bf16(sc[nb + h], qa[1], b[0][2 * h], b[0][2 * h + 1]);
                                mma_bf16(sc[nb + h], qa[0], b[1][2 * h], b[1][2 * h + 1]);
                            }
                        } else {
#pragma unroll
                            for (int h = 0; h < 2; ++h) mma_bf16(sc[nb + h], qa[0], b[0][2 * h], b[0][2 * h + 1]);
                        }
                    }
                }
        }

        // ---- scale, mask, online softmax ------------------------------------------------------------------
        const bool cut = key0 + first + S::kKeysPerWarp > all_see || mask_row != nullptr;
        float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
        for (int nb = 0; nb < kNb; ++nb)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int y = first + nb * 8 + 2 * c4 + e, j = key0 + y;
                sc[nb][e] *= scale;
                sc[nb][2 + e] *= scale;
                if (cut) {
                    const bool padded = mask_row != nullptr && vis[y] == 0;
                    if (j > lim0 || padded) sc[nb][e] = -INFINITY;
                    if (j > lim1 || padded) sc[nb][2 + e] = -INFINITY;
                }
                mx0 = fmaxf(mx0, sc[nb][e]);
                mx1 = fmaxf(mx1, sc[nb][2 + e]);
            }
        mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1));
        mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
        mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1));
        mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
        const float n0 = fmaxf(m0, mx0), n1 = fmaxf(m1, mx1);
        const float u0 = n0 == -INFINITY ? 0.0f : n0, u1 = n1 == -INFINITY ? 0.0f : n1;   // a row that has seen no key yet
        const float a0 = ex2(m0 - u0), a1 = ex2(m1 - u1);
        m0 = n0;
        m1 = n1;
        float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
        for (int nb = 0; nb < kNb; ++nb)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                sc[nb][e] = ex2(sc[nb][e] - u0);
                sc[nb][2 + e] = ex2(sc[nb][2 + e] - u1);
                s0 += sc[nb][e];
                s1 += sc[nb][2 + e];
            }
        l0 = l0 * a0 + s0;
        l1 = l1 * a1 + s1;

        // ---- O += P V ---------------------------------------------------------------------------------------
        unsigned pa[kNb / 2][3][4];
#pragma unroll
        for (int kk = 0; kk < kNb / 2; ++kk)
#pragma unroll
            for (int h = 0; h < 2; ++h) {   // registers 0, 1: keys 0-7 of the step (rows g, g + 8), 2, 3: keys 8-15
                split3(sc[2 * kk + h][0], sc[2 * kk + h][1], pa[kk][0][2 * h], pa[kk][1][2 * h], pa[kk][2][2 * h]);
                split3(sc[2 * kk + h][2], sc[2 * kk + h][3], pa[kk][0][2 * h + 1], pa[kk][1][2 * h + 1], pa[kk][2][2 * h + 1]);
            }
        {
            const int mi = lane >> 3;
            const int v_row = ((mi & 1) << 3) + (lane & 7);
#pragma unroll
            for (int n = 0; n < D / 8; n += 2) {
                float c[2][4];
#pragma unroll
                for (int h = 0; h < 2; ++h) c[h][0] = c[h][1] = c[h][2] = c[h][3] = 0.0f;
#pragma unroll
                for (int pass = 0; pass < 2; ++pass)
#pragma unroll
                    for (int kk = 0; kk < kNb / 2; ++kk) {
                        const int row = first + kk * 16 + v_row;
                        const int at = row * S::kRowBytes + (((n + (mi >> 1)) ^ (row & S::kSwz)) << 4);
                        unsigned b[3][4];
#pragma unroll
                        for (int t = 0; t < (pass == 0 ? 3 : 1); ++t)
                            ldmatrix_x4_trans(b[t][0], b[t][1], b[t][2], b[t][3], vp + t * S::kPlane + at);
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            if (pass == 0) {
                                mma_bf16(c[h], pa[kk][2], b[0][2 * h], b[0][2 * h + 1]);
                                mma_bf16(c[h], pa[kk][1], b[1][2 * h], b[1][2 * h + 1]);
                                mma_bf16(c[h], pa[kk][0], b[2][2 * h], b[2][2 * h + 1]);
                                mma_bf16(c[h], pa[kk][1], b[0][2 * h], b[0][2 * h + 1]);
                                mma_bf16(c[h], pa[kk][0], b[1][2 * h], b[1][2 * h + 1]);
                            } else {
                                mma_bf16(c[h], pa[kk][0], b[0][2 * h], b[0][2 * h + 1]);
                            }
                        }
                    }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    acc[n + h][0] = fmaf(acc[n + h][0], a0, c[h][0]);
                    acc[n + h][1] = fmaf(acc[n + h][1], a0, c[h][1]);
                    acc[n + h][2] = fmaf(acc[n + h][2], a1, c[h][2]);
                    acc[n + h][3] = fmaf(acc[n + h][3], a1, c[h][3]);
                }
            }
        }
    }

    float probe = 0.0f * l0 + 0.0f * l1;   // NaN where any of the sums is not finite
#pragma unroll
    for (int n = 0; n < D / 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) probe = fmaf(0.0f, acc[n][e], probe);
    if (__syncthreads_or(probe != 0.0f)) {
        plain_rows<D, kWarps>(p, s, kvh, row0, min(rows, row0 + S::kRows));
        return;
    }

    l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
    l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 1);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 2);

    if (S::kWk > 1) {   // the key shares of the same rows, through shared memory (the tiles are dead); warp wk == 0 goes on with the sum
        __syncthreads();
        float* const mine = reinterpret_cast<float*>(smem) + warp * 16 * (D + 2);
        if (wk > 0) {
#pragma unroll
            for (int n = 0; n < D / 8; ++n) {
                *reinterpret_cast<float2*>(mine + g * (D + 2) + n * 8 + 2 * c4) = make_float2(acc[n][0], acc[n][1]);
                *reinterpret_cast<float2*>(mine + (g + 8) * (D + 2) + n * 8 + 2 * c4) = make_float2(acc[n][2], acc[n][3]);
            }
            if (c4 == 0) {
                *reinterpret_cast<float2*>(mine + g * (D + 2) + D) = make_float2(m0, l0);
                *reinterpret_cast<float2*>(mine + (g + 8) * (D + 2) + D) = make_float2(m1, l1);
            }
        }
        __syncthreads();
        if (wk > 0) return;
#pragma unroll
        for (int w = 1; w < S::kWk; ++w) {
            const float* other = mine + w * 16 * (D + 2);
            const float2 o0 = *reinterpret_cast<const float2*>(other + g * (D + 2) + D);
            const float2 o1 = *reinterpret_cast<const float2*>(other + (g + 8) * (D + 2) + D);
            const float n0 = fmaxf(m0, o0.x), n1 = fmaxf(m1, o1.x);
            const float u0 = n0 == -INFINITY ? 0.0f : n0, u1 = n1 == -INFINITY ? 0.0f : n1;
            const float a0 = ex2(m0 - u0), a1 = ex2(m1 - u1), b0 = ex2(o0.x - u0), b1 = ex2(o1.x - u1);
            m0 = n0;
            m1 = n1;
            l0 = l0 * a0 + o0.y * b0;
            l1 = l1 * a1 + o1.y * b1;
#pragma unroll
            for (int n = 0; n < D / 8; ++n) {
                const float2 x = *reinterpret_cast<const float2*>(other + g * (D + 2) + n * 8 + 2 * c4);
                const float2 y = *reinterpret_cast<const float2*>(other + (g + 8) * (D + 2) + n * 8 + 2 * c4);
                acc[n][0] = acc[n][0] * a0 + x.x * b0;
                acc[n][1] = acc[n][1] * a0 + x.y * b0;
                acc[n][2] = acc[n][2] * a1 + y.x * b1;
                acc[n][3] = acc[n][3] * a1 + y.y * b1;
            }
        }
    }

#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int r = half ? r1 : r0, t = half ? t1 : t0;
        if (r >= rows) continue;
        const int h = kvh * group + r - t * group;
        const long long pos = half ? pos1 : pos0;
        const float m = half ? m1 : m0, l = half ? l1 : l0;
        // with a padding mask a query row at a padded (or out-of-range) position outputs zeros (flash_attn_func.cu:77-84)
        const bool ok = l > 0.0f && (mask_row == nullptr || (pos >= 0 && pos < si.kv_len && mask_row[pos] != 0));
        const float inv = ok ? 1.0f / l : 0.0f;
        float* dst = og + ((si.q_row0 + t) * p.q_heads + h) * D + 2 * c4;
#pragma unroll
        for (int n = 0; n < D / 8; ++n)
            *reinterpret_cast<float2*>(dst + n * 8) = make_float2(acc[n][2 * half] * inv, acc[n][2 * half + 1] * inv);
        if (p.lse != nullptr && c4 == 0)
            p.lse[((long long)s * p.q_heads + h) * p.q_seq_len + t] = ok ? (m + log2f(l)) * 0.6931471805599453f : -INFINITY;
    }
}

template <int D, int WR>
int launch_one(const AttnParams& p, cudaStream_t stream) {
    using S = Shape<D, WR>;
    static std::atomic<unsigned long long> ready{0};   // devices whose copy of this kernel has its shared-memory limit raised
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err == cudaSuccess && (dev >= 64 || !((ready.load(std::memory_order_acquire) >> dev) & 1ULL))) {
        err = cudaFuncSetAttribute(tile_f32_kernel<D, WR>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kBytes);
        if (err == cudaSuccess && dev < 64) ready.fetch_or(1ULL << dev, std::memory_order_release);
    }
    if (err != cudaSuccess) {
        set_last_errorf("tile_f32_kernel: %s", cudaGetErrorString(err));
        cudaGetLastError();
        return FLASH_ATTN_ERR_CUDA;
    }
    const long long rows = (long long)p.q_seq_len * (p.q_heads / p.kv_heads);
    dim3 grid((unsigned)((rows + S::kRows - 1) / S::kRows), (unsigned)p.kv_heads, (unsigned)p.num_seqs);
    tile_f32_kernel<D, WR><<<grid, kThreads, S::kBytes, stream>>>(p);
    const int rc = check_launch("tile_f32_kernel");
    if (rc == FLASH_ATTN_OK) note_path("tile_f32", 1, "mma");
    return rc;
}

}  // namespace

int launch_tile_f32(const AttnParams& p, cudaStream_t stream) {
    if (p.dtype != DT_F32 || (p.head_size != 32 && p.head_size != 64 && p.head_size != 128)) return -1;
    if (p.mode == MODE_KVCACHE && p.q_seq_len == 1) return -1;   // one row per head: nothing for a 16-row tile
    if (p.n_out > 0 || p.num_seqs > 65535 || p.kv_heads > 65535) return -1;
    if ((reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k) | reinterpret_cast<uintptr_t>(p.v) | reinterpret_cast<uintptr_t>(p.o)) & 15)
        return -1;
    const long long rows = (long long)p.q_seq_len * (p.q_heads / p.kv_heads);
    if (rows > 0x7fffffffLL - 64) return -1;
    const int rc = launch_tile_f32_tcgen05(p, stream);
    if (rc >= 0) return rc;
    const bool large = (rows + 63) / 64 * p.kv_heads * p.num_seqs >= 2LL * sm_count();   // two CTAs per SM
    if (p.head_size == 128) return large ? launch_one<128, 4>(p, stream) : launch_one<128, 2>(p, stream);
    if (p.head_size == 64) return large ? launch_one<64, 4>(p, stream) : launch_one<64, 1>(p, stream);
    return large ? launch_one<32, 4>(p, stream) : launch_one<32, 1>(p, stream);
}

}  // namespace fa
