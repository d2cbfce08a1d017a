// What the two kernels for f32 storage share: the split of f32 values into three bf16 terms, and rows in plain f32.
#pragma once

#include "common.cuh"
#include "tcgen05.cuh"

namespace fa {
namespace {

// Two values less a packed bf16 pair.
__device__ __forceinline__ float2 less(float x, float y, unsigned pair) {
    float2 d;
    asm("{\n.reg .b64 a, b, c;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nsub.rn.f32x2 c, a, b;\nmov.b64 {%0, %1}, c;\n}\n"
        : "=f"(d.x), "=f"(d.y)
        : "f"(x), "f"(y), "r"(pair << 16), "r"(pair & 0xffff0000u));
    return d;
}
// Two values -> three packed bf16 pairs whose sum is the pair (the differences are exact).
__device__ __forceinline__ void split3(float x, float y, unsigned& hi, unsigned& mid, unsigned& lo) {
    hi = pack16<__nv_bfloat16>(x, y);
    float2 rest = less(x, y, hi);
    mid = pack16<__nv_bfloat16>(rest.x, rest.y);
    rest = less(rest.x, rest.y, mid);
    lo = pack16<__nv_bfloat16>(rest.x, rest.y);
}

// x / y for many x, given 1 / y rounded to nearest: a product, its remainder and one correction (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", 1990), which
// round to nearest while nothing underflows: the bits of the division operator, whose code at the end of a kernel, for 16 or 32 columns of a row, takes longer (tile_f32_tcgen05.cu, us: 1 x 256, 8 heads of 64
// 11.08 and 10.77 so; 4 x 2048, 8 of 128 523 and 506).
__host__ __device__ __forceinline__ float quotient(float x, float y, float inv) {
    const float q = x * inv;
    return fmaf(fmaf(-q, y, x), inv, q);
}

// The rows of a CTA that met a value that does not survive the split, one key at a time in plain f32, as tile_simt.cu
// does it: a warp per row (the CTA's first kWarps). An infinity minus itself, and infinity times the other operand's small terms, are NaN where the
// product is not, and so is zero weight times a row that a query does not see; the same holds for a value that rounds
// to a bf16 infinity. Each leaves a NaN in the sums that it reaches, which is where the kernel looks, once at its end.
template <int D, int kWarps>
__device__ __noinline__ void plain_rows(const AttnParams& p, int s, int kvh, int row0, int row_end) {
    const SeqInfo si = seq_info(p, s);
    const uint8_t* mask_row = p.mask ? p.mask + (long long)s * p.kv_seq_len : nullptr;
    constexpr int E = D / 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, group = p.q_heads / p.kv_heads;
    const float* kg = static_cast<const float*>(p.k);
    const float* vg = static_cast<const float*>(p.v);
    for (int r = row0 + warp; r < row_end; r += kWarps) {
        const int t = r / group, h = kvh * group + r - t * group;
        const long long pos = (long long)si.pos_off + t, at = ((si.q_row0 + t) * p.q_heads + h) * D;
        const int end = (int)max(0LL, min((long long)si.kv_len, pos + 1));
        float q[E], acc[E], m = -INFINITY, l = 0.0f;
        for (int e = 0; e < E; ++e) {
            q[e] = static_cast<const float*>(p.q)[at + lane + 32 * e];
            acc[e] = 0.0f;
        }
        for (int j = 0; j < end; ++j) {
            if (mask_row != nullptr && mask_row[j] == 0) continue;
            const long long row = p.paged ? (long long)block_slot(p.block_tables, s, p.max_blocks, j, p.block_size) : si.kv_row0 + j;
            const long long off = (row * p.kv_heads + kvh) * D + lane;
            float part = 0.0f;
            for (int e = 0; e < E; ++e) part = fmaf(q[e], kg[off + 32 * e], part);
            for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
            const float sc = part * p.scale, m_new = fmaxf(m, sc);
            const float alpha = __expf(m - m_new), pr = __expf(sc - m_new);
            l = l * alpha + pr;
            for (int e = 0; e < E; ++e) acc[e] = acc[e] * alpha + pr * vg[off + 32 * e];
            m = m_new;
        }
        const bool ok = l > 0.0f && (mask_row == nullptr || (pos >= 0 && pos < si.kv_len && mask_row[pos] != 0));
        const float inv = ok ? 1.0f / l : 0.0f;
        for (int e = 0; e < E; ++e) static_cast<float*>(p.o)[at + lane + 32 * e] = acc[e] * inv;
        if (p.lse != nullptr && lane == 0)
            p.lse[((long long)s * p.q_heads + h) * p.q_seq_len + t] = ok ? m + __logf(l) : -INFINITY;
    }
}

}  // namespace
}  // namespace fa
