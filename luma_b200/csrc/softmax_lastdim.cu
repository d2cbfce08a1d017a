// Row softmax over the last dimension for sm_100a: the kernel of the math-path attention
// (scores -> probabilities). Replaces softmax_{f32,f16,bf16} of luma-cuda/kernels/nn.cu:21-76,
// which reads every row three times (max, sum, normalise) with one element per load and does its
// arithmetic in the storage type. Here a row is read once with 16-byte loads, kept in registers,
// reduced in f32 (running max and sum merged across lanes with the online-softmax rule of
// luma-cpu/src/kernels/nn.rs:39-56) and written once, rounded to nearest even: the kernel is bound
// by HBM at 2 * rows * row_size * sizeof(T) bytes.
// 32 elements per thread throughout (4 vectors of 16-bit storage, 8 of f32):
//   rows of up to 1024 elements  : one warp per row (several short rows at a time), no shared memory
//   rows of up to 32768 elements : one CTA of 64 .. 1024 threads per row, one shared-memory exchange
//   longer rows                  : one CTA per row, two passes over the row (read twice)
// Where rows begin on no 16-byte boundary, the first and the last kind read as wide as every row's beginning allows, two elements or one (template
// parameter V; a warp's loads still cover whole lines), the second kind in the aligned vectors that cover the row (RAGGED). Until then all such rows
// went through the last kind in single elements. Before and now, us: 42983 rows of 162 bf16 223 and 14, 20000 of 1001 f32 152 and 28 (of 1000: 27), 60000 of 4099 bf16 789 and 189,
// 8000 of 16383 bf16 340 and 105.
#include "common.cuh"
#include "../../include/luma_nn_kernels.h"

namespace fa {
namespace {

constexpr float kLog2e = 1.4426950408889634f;

template <int BYTES> struct Word;
template <> struct Word<2> { using type = unsigned short; };
template <> struct Word<4> { using type = unsigned; };
template <> struct Word<8> { using type = uint2; };
template <> struct Word<16> { using type = uint4; };

template <typename T, int V>
__device__ __forceinline__ void load_vec(const T* p, float (&x)[V]) {
    const auto raw = *reinterpret_cast<const typename Word<V * (int)sizeof(T)>::type*>(p);
    const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
    for (int i = 0; i < V; ++i) x[i] = to_f32<T>(e[i]);
}
template <typename T, int V>
__device__ __forceinline__ void store_vec(T* p, const float (&x)[V]) {
    typename Word<V * (int)sizeof(T)>::type raw;
    T* e = reinterpret_cast<T*>(&raw);
#pragma unroll
    for (int i = 0; i < V; ++i) e[i] = from_f32<T>(x[i]);
    *reinterpret_cast<typename Word<V * (int)sizeof(T)>::type*>(p) = raw;
}

// Where a row that begins anywhere lies in aligned vectors: vector v of it begins at element v * V of `src` and `dst`, and its own elements are
// [head, end) of those; head == 0 and end % V == 0 unless RAGGED. All loads come first and `unpack` after, so that what the ends of a row cost stays
// behind the last load.
template <typename T, bool RAGGED>
struct RowWindow {
    static constexpr int V = 16 / (int)sizeof(T);
    const T* src;
    T* dst;
    int head, end;
    int first, last;   // vectors at [first, last) lie inside the tensor whole; the others are read element by element
    bool whole_stores;
    // [in, stop): the whole tensor, outside of which nothing is read
    __device__ __forceinline__ RowWindow(const T* in, const T* stop, T* out, long long row, int n) : src(in + row * n), dst(out + row * n), head(0), end(n) {
        if (RAGGED) {
            head = (int)((reinterpret_cast<uintptr_t>(src) & 15) / sizeof(T));
            src -= head;
            dst -= head;
            end += head;
            first = src < in ? V : 0;
            last = stop - src < end + V ? (int)(stop - src) / V * V : end + V;
            whole_stores = (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
        }
    }
    __device__ __forceinline__ uint4 load(int col) const {
        uint4 raw = make_uint4(0u, 0u, 0u, 0u);
        if (col >= first && col < last && col < end) raw = *reinterpret_cast<const uint4*>(src + col);
        return raw;
    }
    // one bit per element of the vector at col that is the row's
    __device__ __forceinline__ unsigned own(int col) const {
        return (((1u << V) - 1u) << max(head - col, 0)) & ((1u << min(max(end - col, 0), V)) - 1u);
    }
    __device__ __forceinline__ void unpack(int col, const uint4& raw, float (&x)[V]) const {
        const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
        for (int i = 0; i < V; ++i) x[i] = to_f32<T>(e[i]);
        if (col < head || col + V > end) {
            const unsigned mine = own(col);
            if (col < first || col >= last) {
#pragma unroll
                for (int i = 0; i < V; ++i)
                    if ((mine >> i) & 1u) x[i] = to_f32<T>(src[col + i]);
            }
#pragma unroll
            for (int i = 0; i < V; ++i)
                if (!((mine >> i) & 1u)) x[i] = -INFINITY;
        }
    }
    __device__ __forceinline__ void store(int col, const float (&x)[V]) const {
        if (!RAGGED || (col >= head && col + V <= end && whole_stores)) {
            store_vec<T, V>(dst + col, x);
            return;
        }
        const unsigned mine = own(col);
#pragma unroll
        for (int i = 0; i < V; ++i)
            if ((mine >> i) & 1u) dst[col + i] = from_f32<T>(x[i]);
    }
};

__device__ __forceinline__ float fast_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}

// (m, s) = running max and sum of exp(x - m); merging two partial results
__device__ __forceinline__ void merge(float& m, float& s, float m2, float s2) {
    const float mn = fmaxf(m, m2);
    // exp2f(-inf - -inf) would be NaN: an empty partial (s == 0) contributes nothing
    const float a = s == 0.0f ? 0.0f : s * exp2f((m - mn) * kLog2e);
    const float b = s2 == 0.0f ? 0.0f : s2 * exp2f((m2 - mn) * kLog2e);
    m = mn;
    s = a + b;
}
__device__ __forceinline__ void warp_merge(float& m, float& s) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const float m2 = __shfl_xor_sync(0xffffffffu, m, off);
        const float s2 = __shfl_xor_sync(0xffffffffu, s, off);
        merge(m, s, m2, s2);
    }
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
    return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// One warp works on R rows at a time, each row in VPT vectors per lane (R * VPT vectors = 32 elements per lane).
template <typename T, int V, int VPT, int R>
__global__ void __launch_bounds__(256) softmax_warp_kernel(const T* __restrict__ in, T* __restrict__ out, long long rows, int n) {
    const int lane = threadIdx.x & 31;
    const long long row0 = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * R;
    if (row0 >= rows) return;
    float x[R][VPT][V];
    float m[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        m[r] = -INFINITY;
        const bool live = row0 + r < rows;
        const T* src = in + (row0 + r) * n;
#pragma unroll
        for (int v = 0; v < VPT; ++v) {
            const int col = (v * 32 + lane) * V;
            if (live && col < n) {
                load_vec<T, V>(src + col, x[r][v]);
            } else {
#pragma unroll
                for (int i = 0; i < V; ++i) x[r][v][i] = -INFINITY;
            }
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
        for (int v = 0; v < VPT; ++v)
#pragma unroll
            for (int i = 0; i < V; ++i) m[r] = fmaxf(m[r], x[r][v][i]);
        float s = 0.0f;
        const float ml = m[r] == -INFINITY ? 0.0f : m[r] * kLog2e;   // a lane that saw only -inf: exp2(-inf) = 0
#pragma unroll
        for (int v = 0; v < VPT; ++v)
#pragma unroll
            for (int i = 0; i < V; ++i) {
                x[r][v][i] = fast_ex2(fmaf(x[r][v][i], kLog2e, -ml));   // exp(x - m_lane)
                s += x[r][v][i];
            }
        // exp(x - m_row) / s_row = exp(x - m_lane) * exp(m_lane - m_row) / s_row: the row max first, then
        // every lane's sum rescaled once; a row of -inf only gives NaN (as the reference's arithmetic does)
        const float mr = warp_max(m[r]);
        const float rescale = (m[r] == -INFINITY && mr != -INFINITY) ? 0.0f : fast_ex2((m[r] - mr) * kLog2e);
        const float sr = warp_sum(s * rescale);
        const float f = rescale / sr;
        if (row0 + r < rows) {
            T* dst = out + (row0 + r) * n;
#pragma unroll
            for (int v = 0; v < VPT; ++v) {
                const int col = (v * 32 + lane) * V;
                if (col < n) {
#pragma unroll
                    for (int i = 0; i < V; ++i) x[r][v][i] *= f;
                    store_vec<T, V>(dst + col, x[r][v]);
                }
            }
        }
    }
}

// One CTA of THREADS threads per row, or (RAGGED) of as many warps as the row's vectors need; VPT vectors per thread; one exchange through shared memory.
template <typename T, bool RAGGED, int VPT, int THREADS>
__global__ void __launch_bounds__(THREADS) softmax_block_kernel(const T* __restrict__ in, T* __restrict__ out, int n) {
    constexpr int V = 16 / (int)sizeof(T);
    __shared__ float sh_m[THREADS / 32], sh_s[THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, threads = RAGGED ? blockDim.x : THREADS, warps = threads >> 5;
    const RowWindow<T, RAGGED> w(in, in + (long long)gridDim.x * n, out, (long long)blockIdx.x, n);
    float x[VPT][V];
    if constexpr (RAGGED) {
        uint4 raw[VPT];
#pragma unroll
        for (int v = 0; v < VPT; ++v) raw[v] = w.load((v * threads + threadIdx.x) * V);
#pragma unroll
        for (int v = 0; v < VPT; ++v) w.unpack((v * threads + threadIdx.x) * V, raw[v], x[v]);
    } else {
#pragma unroll
        for (int v = 0; v < VPT; ++v) {
            const int col = (v * THREADS + threadIdx.x) * V;
            if (col < n) {
                load_vec<T, V>(w.src + col, x[v]);
            } else {
#pragma unroll
                for (int i = 0; i < V; ++i) x[v][i] = -INFINITY;
            }
        }
    }
    float m = -INFINITY;
#pragma unroll
    for (int v = 0; v < VPT; ++v)
#pragma unroll
        for (int i = 0; i < V; ++i) m = fmaxf(m, x[v][i]);
    float s = 0.0f;
    const float ml = m == -INFINITY ? 0.0f : m * kLog2e;   // a thread that saw only -inf: exp2(-inf) = 0
#pragma unroll
    for (int v = 0; v < VPT; ++v)
#pragma unroll
        for (int i = 0; i < V; ++i) {
            x[v][i] = fast_ex2(fmaf(x[v][i], kLog2e, -ml));
            s += x[v][i];
        }
    // row max through shared memory, every thread's sum rescaled once, then the row sum
    float mw = warp_max(m);
    if (lane == 0) sh_m[warp] = mw;
    __syncthreads();
    const float mr = warp_max(lane < warps ? sh_m[lane] : -INFINITY);
    const float rescale = (m == -INFINITY && mr != -INFINITY) ? 0.0f : fast_ex2((m - mr) * kLog2e);
    const float sw = warp_sum(s * rescale);
    if (lane == 0) sh_s[warp] = sw;
    __syncthreads();
    const float sr = warp_sum(lane < warps ? sh_s[lane] : 0.0f);
    const float f = rescale / sr;
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
        const int col = (v * threads + threadIdx.x) * V;
        if (col < w.end) {
#pragma unroll
            for (int i = 0; i < V; ++i) x[v][i] *= f;
            w.store(col, x[v]);
        }
    }
}

constexpr int kStreamThreads = 512;

// Any row length: one CTA per row, pass 1 reduces (m, s) online, pass 2 re-reads and writes.
template <typename T, int V>
__global__ void __launch_bounds__(kStreamThreads) softmax_stream_kernel(const T* __restrict__ in, T* __restrict__ out, int n) {
    __shared__ float sh_m[kStreamThreads / 32], sh_s[kStreamThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const T* src = in + (long long)blockIdx.x * n;
    T* dst = out + (long long)blockIdx.x * n;
    float m = -INFINITY, s = 0.0f;
    for (unsigned c = threadIdx.x * V; c < (unsigned)n; c += kStreamThreads * V) {   // (up to a stride beyond n, which may be near 2^31)
        float x[V];
        load_vec<T, V>(src + c, x);
        float mv = x[0];
#pragma unroll
        for (int i = 1; i < V; ++i) mv = fmaxf(mv, x[i]);
        const float ref = mv == -INFINITY ? 0.0f : mv;   // (a NaN beside -inf reaches the sum so)
        float sv = 0.0f;
#pragma unroll
        for (int i = 0; i < V; ++i) sv += fast_ex2((x[i] - ref) * kLog2e);
        merge(m, s, mv, sv);
    }
    warp_merge(m, s);
    if (lane == 0) { sh_m[warp] = m; sh_s[warp] = s; }
    __syncthreads();
    m = lane < kStreamThreads / 32 ? sh_m[lane] : -INFINITY;
    s = lane < kStreamThreads / 32 ? sh_s[lane] : 0.0f;
    warp_merge(m, s);
    const float ml = m * kLog2e, inv = 1.0f / s;
    for (unsigned c = threadIdx.x * V; c < (unsigned)n; c += kStreamThreads * V) {
        float x[V];
        load_vec<T, V>(src + c, x);
#pragma unroll
        for (int i = 0; i < V; ++i) x[i] = fast_ex2(fmaf(x[i], kLog2e, -ml)) * inv;
        store_vec<T, V>(dst + c, x);
    }
}

template <typename T, int V>
int launch_softmax(const T* in, T* out, long long rows, int n, cudaStream_t stream) {
    // 32 elements per thread (4 vectors of 16-bit, 8 of f32): few enough registers for 4 CTAs of 256
    // threads per SM, whose loads, arithmetic and stores then overlap; with 128 elements per thread
    // (one resident CTA) a bf16 row of 4096 reached 0.54 of the copy bandwidth
    constexpr int P = 32 / V;
    constexpr int kWide = 16 / (int)sizeof(T);
    // the longest row of one CTA: 32 elements for each of 1024 threads, of which a row that begins anywhere may leave kWide - 1 unused ahead of it
    constexpr int kLongest = 32768 - (V == kWide ? 0 : kWide - 1);
    const int vecs = n / V;
    const int warps = 8;
    const unsigned grid = (unsigned)rows;
    if (vecs <= 32 * P) {
        // a warp takes R rows of P / R vectors per lane at a time
        auto per_warp = [&](auto kernel, int r) {
            kernel<<<(unsigned)((rows + (long long)warps * r - 1) / ((long long)warps * r)), warps * 32, 0, stream>>>(in, out, rows, n);
        };
        if (P >= 8 && vecs <= 32 * (P / 8)) per_warp(softmax_warp_kernel<T, V, P >= 8 ? P / 8 : P, P >= 8 ? 8 : 1>, 8);
        else if (vecs <= 32 * (P / 4)) per_warp(softmax_warp_kernel<T, V, P / 4, 4>, 4);
        else if (vecs <= 32 * (P / 2)) per_warp(softmax_warp_kernel<T, V, P / 2, 2>, 2);
        else per_warp(softmax_warp_kernel<T, V, P, 1>, 1);
        note_path("softmax_warp", 1);
    } else if (n <= kLongest) {
        if constexpr (V == kWide) {
            if (vecs <= 64 * P) softmax_block_kernel<T, false, P, 64><<<grid, 64, 0, stream>>>(in, out, n);
            else if (vecs <= 128 * P) softmax_block_kernel<T, false, P, 128><<<grid, 128, 0, stream>>>(in, out, n);
            else if (vecs <= 256 * P) softmax_block_kernel<T, false, P, 256><<<grid, 256, 0, stream>>>(in, out, n);
            else if (vecs <= 512 * P) softmax_block_kernel<T, false, P, 512><<<grid, 512, 0, stream>>>(in, out, n);
            else softmax_block_kernel<T, false, P, 1024><<<grid, 1024, 0, stream>>>(in, out, n);
        } else {
            // Rows as long as this pay for aligned vectors with masked ends; in single elements a bf16 row of 4099 took 415 us where this takes 189
            // (60000 rows), one of 1413 86 and 57 (f16, 46713 rows). CTAs of just as many warps as a row needs: in CTAs of a power of two,
            // lengths just above one had twice the threads. Two CTAs of more than 512 threads do not fit an SM's registers: just
            // above, each thread takes a vector more, five instead of four in 16 bits (up to a quarter above), nine instead of eight in f32 (up to an eighth):
            // 8000 rows of 16383 bf16 105 us, 155 without.
            constexpr int kEach = 32 / kWide;
            const unsigned all = (unsigned)(n + 2 * kWide - 2) / kWide;   // (a row begins up to kWide - 1 elements into its first vector)
            auto fit = [&](unsigned each) { return (all + each * 32 - 1) / (each * 32) * 32; };
            const unsigned threads = fit(kEach);
            if (threads <= 128) softmax_block_kernel<T, true, kEach, 128><<<grid, threads, 0, stream>>>(in, out, n);
            else if (threads <= 256) softmax_block_kernel<T, true, kEach, 256><<<grid, threads, 0, stream>>>(in, out, n);
            else if (threads <= 512) softmax_block_kernel<T, true, kEach, 512><<<grid, threads, 0, stream>>>(in, out, n);
            else if (fit(kEach + 1) <= 512) softmax_block_kernel<T, true, kEach + 1, 512><<<grid, fit(kEach + 1), 0, stream>>>(in, out, n);
            else softmax_block_kernel<T, true, kEach, 1024><<<grid, threads, 0, stream>>>(in, out, n);
        }
        note_path("softmax_block", 1);
    } else {
        softmax_stream_kernel<T, V><<<grid, kStreamThreads, 0, stream>>>(in, out, n);
        note_path("softmax_stream", 1);
    }
    return check_launch("softmax_last_dim");
}

template <typename T>
int softmax_impl(const void* in, void* out, long long rows, int n, void* stream) {
    set_last_error("");
    cudaGetLastError();
    if (in == nullptr || out == nullptr) {
        set_last_error("luma_softmax: input/output must not be null");
        return FLASH_ATTN_ERR_NULL_PTR;
    }
    if (rows <= 0 || n <= 0 || rows > 0x7fffffffLL) {
        set_last_error("luma_softmax: num_rows and row_size must be > 0 (num_rows < 2^31)");
        return FLASH_ATTN_ERR_INVALID_SHAPE;
    }
    cudaPointerAttributes attr;
    int prev = -1;
    if (cudaPointerGetAttributes(&attr, in) == cudaSuccess && attr.type == cudaMemoryTypeDevice) {
        cudaGetDevice(&prev);
        if (prev != attr.device) cudaSetDevice(attr.device);
        else prev = -1;
    } else {
        cudaGetLastError();
    }
    const T* const src = static_cast<const T*>(in);
    T* const dst = static_cast<T*>(out);
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    constexpr int kWide = 16 / (int)sizeof(T);
    const uintptr_t both = reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out) | (uintptr_t)((size_t)n * sizeof(T));   // every row's beginning
    const int rc = both % 16 == 0 ? launch_softmax<T, kWide>(src, dst, rows, n, st)
                   : both % (2 * sizeof(T)) == 0 ? launch_softmax<T, 2>(src, dst, rows, n, st)
                                                 : launch_softmax<T, 1>(src, dst, rows, n, st);
    if (prev >= 0) cudaSetDevice(prev);
    return rc;
}

}  // namespace
}  // namespace fa

extern "C" {
int luma_softmax_f32(const float* input, float* output, long long num_rows, int row_size, void* stream) {
    return fa::softmax_impl<float>(input, output, num_rows, row_size, stream);
}
int luma_softmax_f16(const flash_attn_f16_t* input, flash_attn_f16_t* output, long long num_rows, int row_size, void* stream) {
    return fa::softmax_impl<__half>(input, output, num_rows, row_size, stream);
}
int luma_softmax_bf16(const flash_attn_bf16_t* input, flash_attn_bf16_t* output, long long num_rows, int row_size, void* stream) {
    return fa::softmax_impl<__nv_bfloat16>(input, output, num_rows, row_size, stream);
}
}
