// Memory-bound element-wise and reduction kernels: GELU forward/backward,
// dropout (Philox counter, mask regenerated in the backward), bias gradient
// (column sum), 16-bit -> fp32 gradient accumulation, embedding gather and its
// scatter-add backward, micro-batch row pack/unpack.
//
// They take the place of the ATen element-wise kernels the reference launches
// one node at a time from its interpreter (src/torch/TorchDriver.cpp:566) and of
// the pad / slice / cat helpers of src/torch/TorchUtil.cpp:785-843,1091-1136.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "debug_check.cuh"
#include "launch.cuh"
#include "philox.cuh"
#include "tc_common.cuh"

namespace rb {

template <typename T>
__device__ __forceinline__ void ld8e(const T* p, float (&v)[8]) {
    uint4 q = *reinterpret_cast<const uint4*>(p);
    const T* e = reinterpret_cast<const T*>(&q);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = to_f32<T>(e[j]);
}
template <typename T>
__device__ __forceinline__ void st8e(T* p, const float (&v)[8]) {
    uint4 q;
    T* e = reinterpret_cast<T*>(&q);
#pragma unroll
    for (int j = 0; j < 8; ++j) e[j] = from_f32<T>(v[j]);
    *reinterpret_cast<uint4*>(p) = q;
}

// mode 0: y = gelu(x); mode 1: y = dy * gelu'(x)
template <typename T>
__global__ void gelu_kernel(const T* __restrict__ x, const T* __restrict__ dy, T* __restrict__ y,
                            size_t n, int mode) {
    const size_t nv = n / 8;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < nv;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        float a[8], o[8];
        ld8e(x + i * 8, a);
        if (mode == 0) {
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] = gelu_erf(a[j]);
        } else {
            float d[8];
            ld8e(dy + i * 8, d);
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] = d[j] * gelu_erf_grad(a[j]);
        }
        st8e(y + i * 8, o);
    }
    if (blockIdx.x == 0 && threadIdx.x < n % 8) {
        const size_t i = nv * 8 + threadIdx.x;
        const float a = to_f32<T>(x[i]);
        y[i] = from_f32<T>(mode == 0 ? gelu_erf(a) : to_f32<T>(dy[i]) * gelu_erf_grad(a));
    }
}

// y = keep ? x * scale : 0, mask from (seed, offset, linear index)
template <typename T>
__global__ void dropout_kernel(const T* __restrict__ x, T* __restrict__ y, size_t n, uint32_t thr,
                               float scale, uint64_t seed, uint64_t offset) {
    const size_t nv = n / 8;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < nv;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        float a[8];
        ld8e(x + i * 8, a);
        bool k[8];
        keep8(seed, offset, i * 8, thr, k);
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] = k[j] ? a[j] * scale : 0.f;
        st8e(y + i * 8, a);
    }
    if (blockIdx.x == 0 && threadIdx.x < n % 8) {
        const size_t i = nv * 8 + threadIdx.x;
        const Philox4 r = philox4x32(seed, offset, i >> 3);
        const uint32_t w = r.v[(i & 7) >> 1];
        const uint32_t bits = (i & 1) ? (w >> 16) : (w & 0xffffu);
        y[i] = from_f32<T>(bits >= thr ? to_f32<T>(x[i]) * scale : 0.f);
    }
}

// out[n] (+)= sum_m x[m, n]; x is [M, N] row-major 16-bit, out fp32.
// grid (ceil(N/64), SPLIT); block (32, 8): thread handles 2 columns.
template <typename T>
__global__ void colsum_kernel(const T* __restrict__ x, float* __restrict__ out, int M, int N,
                              long long ld) {
    __shared__ float red[8][65];
    const int col = blockIdx.x * 64 + threadIdx.x * 2;
    float s0 = 0.f, s1 = 0.f;
    if (col < N) {
        for (int m = blockIdx.y * 8 + threadIdx.y; m < M; m += gridDim.y * 8) {
            const T* p = x + static_cast<long long>(m) * ld + col;
            if (col + 1 < N) {
                s0 += to_f32<T>(p[0]);
                s1 += to_f32<T>(p[1]);
            } else {
                s0 += to_f32<T>(p[0]);
            }
        }
    }
    red[threadIdx.y][threadIdx.x * 2] = s0;
    red[threadIdx.y][threadIdx.x * 2 + 1] = s1;
    __syncthreads();
    if (threadIdx.y == 0) {
#pragma unroll
        for (int w = 1; w < 8; ++w) {
            s0 += red[w][threadIdx.x * 2];
            s1 += red[w][threadIdx.x * 2 + 1];
        }
        if (col < N) atomicAdd(out + col, s0);
        if (col + 1 < N) atomicAdd(out + col + 1, s1);
    }
}

// Vector variant: a thread owns 8 adjacent columns (one 16-byte load per row), a block of (32, 8)
// covers 256 columns; rows are strided over threadIdx.y and blockIdx.y.  Needs N % 8 == 0,
// ld % 8 == 0 and a 16-byte aligned base.
template <typename T>
__global__ void colsum_vec_kernel(const T* __restrict__ x, float* __restrict__ out, int M, int N,
                                  long long ld) {
    __shared__ float red[8][256 + 8];
    const int col = blockIdx.x * 256 + threadIdx.x * 8;
    float s[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) s[j] = 0.f;
    if (col < N) {
        const int step = gridDim.y * 8;
        int m = blockIdx.y * 8 + threadIdx.y;
        // two rows in flight per iteration
        for (; m + step < M; m += 2 * step) {
            float a[8], b[8];
            ld8e(x + static_cast<long long>(m) * ld + col, a);
            ld8e(x + static_cast<long long>(m + step) * ld + col, b);
#pragma unroll
            for (int j = 0; j < 8; ++j) s[j] += a[j] + b[j];
        }
        if (m < M) {
            float a[8];
            ld8e(x + static_cast<long long>(m) * ld + col, a);
#pragma unroll
            for (int j = 0; j < 8; ++j) s[j] += a[j];
        }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) red[threadIdx.y][threadIdx.x * 8 + j] = s[j];
    __syncthreads();
    const int t = threadIdx.y * 32 + threadIdx.x;  // 256 threads, one column each
    float acc = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) acc += red[w][t];
    const int c = blockIdx.x * 256 + t;
    if (c < N) atomicAdd(out + c, acc);
}

// The gradients of three stacked projections, each into a tensor of its own: a third of the rows of one [3 n] block of
// weights (fp32 or 16-bit) and of one fp32 vector of biases, rounded to 16 bits.  Small calls are bound by the host: with a
// copy or conversion per tensor (six launches) a forward and backward of 6 x 197 tokens x 768 took 189 us, with this
// one launch 153.
struct Unstack3 {
    const void* w;
    const float* b;   // may be null
    void *wd[3], *bd[3];
    long long wn, bn;   // elements of one part, multiples of 8
};
template <typename T, typename SrcT>
__global__ void __launch_bounds__(256) unstack3_kernel(const Unstack3 u) {
    grid_trigger();
    grid_wait();
    const long long wv = u.wn / 8, bv = u.b ? u.bn / 8 : 0, total = 3 * (wv + bv);
    for (long long i = blockIdx.x * 256LL + threadIdx.x; i < total; i += gridDim.x * 256LL) {
        const bool is_w = i < 3 * wv;
        const long long k = is_w ? i : i - 3 * wv, n = is_w ? wv : bv;
        const int part = static_cast<int>(k / n);
        T* dst = static_cast<T*>(is_w ? u.wd[part] : u.bd[part]) + (k - part * n) * 8;
        if (std::is_same_v<SrcT, float> || !is_w) {
            const float4* src = reinterpret_cast<const float4*>(is_w ? static_cast<const float*>(u.w) : u.b) + k * 2;
            const float4 lo = src[0], hi = src[1];
            const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
            st8e(dst, v);
        } else {
            *reinterpret_cast<uint4*>(dst) = static_cast<const uint4*>(u.w)[k];
        }
    }
}

// dst(fp32) += src(16-bit) * scale
template <typename T>
__global__ void accum_kernel(float* __restrict__ dst, const T* __restrict__ src, size_t n,
                             float scale) {
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<size_t>(gridDim.x) * blockDim.x)
        dst[i] += to_f32<T>(src[i]) * scale;
}

// dst(16-bit) = src(fp32) * scale
template <typename T>
__global__ void cast_kernel(T* __restrict__ dst, const float* __restrict__ src, size_t n,
                            float scale) {
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<size_t>(gridDim.x) * blockDim.x)
        dst[i] = from_f32<T>(src[i] * scale);
}

// out[r, :] = table[ids[r], :]  (H % 8 == 0); one warp per row
template <typename T>
__global__ void embed_fwd_kernel(const long long* ids, const T* table, T* out, int rows, int H, long long vocab) {
    grid_trigger();
    grid_wait();
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= rows) return;
    long long id = ids[warp];
    const bool ok = id >= 0 && id < vocab;
    const uint4* src = reinterpret_cast<const uint4*>(table + (ok ? id : 0) * H);
    uint4* dst = reinterpret_cast<uint4*>(out + static_cast<long long>(warp) * H);
    for (int i = lane; i < H / 8; i += 4 * 32) {
        uint4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = ok && i + u * 32 < H / 8 ? src[i + u * 32] : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i + u * 32 < H / 8) dst[i + u * 32] = v[u];
    }
}

// dtable(fp32)[ids[r], :] += dout[r, :] ; rows with id == padding_idx are skipped
template <typename T>
__global__ void embed_bwd_kernel(const long long* __restrict__ ids, const T* __restrict__ dout,
                                 float* __restrict__ dtable, int rows, int H, long long vocab,
                                 long long padding_idx) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= rows) return;
    const long long id = ids[warp];
    if (id < 0 || id >= vocab || id == padding_idx) return;
    const T* src = dout + static_cast<long long>(warp) * H;
    float* dst = dtable + id * H;
    for (int i = lane; i < H; i += 32) atomicAdd(dst + i, to_f32<T>(src[i]));
}

// Vector variant of embed_bwd_kernel: a thread owns 4 adjacent columns (8 bytes per row) of STRIP consecutive rows and
// keeps their sum in registers for as long as the id stays the same.  Not memory but the atomic units bound this:
// a segment table has two rows, so in the scalar kernel every token of a batch adds to one of two addresses per
// column; equal neighbours (segments, padding) cost one reduction per strip here.  Ids that differ cost the same
// 32-byte sectors as before in a quarter of the instructions.  (8 columns per thread, as two 16-byte reductions 32
// bytes apart from lane to lane, touches every sector twice and was slower than the scalar kernel on such ids.)
// Word, position and segment tables for 32 x 512 tokens x 1024: 107 -> 32.5 us; begun beside the end of the kernel before,
// as are the lookups, 43.6 -> 39.7 us one behind the other.
template <typename T, int STRIP>
__global__ void __launch_bounds__(256)
    embed_bwd_vec_kernel(const long long* ids, const T* dout, float* dtable, int rows, int nv, long long vocab,
                         long long padding_idx) {
    grid_trigger();
    grid_wait();
    constexpr int FLIGHT = STRIP < 8 ? STRIP : 8;   // rows on their way at a time
    const long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    const long long strip = t / nv;
    const int vec = static_cast<int>(t - strip * nv);
    const long long r0 = strip * STRIP;
    if (r0 >= rows) return;
    const int n = static_cast<int>(min(static_cast<long long>(STRIP), rows - r0));
    const long long ld = static_cast<long long>(nv) * 4;
    const T* src = dout + r0 * ld + vec * 4;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    long long cur = -1;   // the id whose sum `acc` holds; -1: none
    auto flush = [&]() {
        if (cur < 0) return;
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dtable + cur * ld + vec * 4), "f"(acc[0]),
                     "f"(acc[1]), "f"(acc[2]), "f"(acc[3])
                     : "memory");
    };
#pragma unroll
    for (int k0 = 0; k0 < STRIP; k0 += FLIGHT) {
        if (k0 >= n) break;
        long long id[FLIGHT];
        uint2 q[FLIGHT];
#pragma unroll
        for (int u = 0; u < FLIGHT; ++u) {
            id[u] = -1;
            if (k0 + u < n) {
                id[u] = ids[r0 + k0 + u];
                if (id[u] < 0 || id[u] >= vocab || id[u] == padding_idx) id[u] = -1;
                q[u] = *reinterpret_cast<const uint2*>(src + (k0 + u) * ld);
            }
        }
#pragma unroll
        for (int u = 0; u < FLIGHT; ++u) {
            if (id[u] < 0) continue;
            const T* e = reinterpret_cast<const T*>(&q[u]);
            if (id[u] != cur) {
                flush();
                cur = id[u];
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[j] = to_f32<T>(e[j]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[j] += to_f32<T>(e[j]);
            }
        }
    }
    flush();
}

// Row copy between two row-major buffers with different row offsets; used to
// pack micro-batch slices and pipeline send buffers.  bytes_per_row % 16 == 0.
__global__ void rowcopy_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst,
                               long long rows, long long vec_per_row, long long src_ld,
                               long long dst_ld) {
    const long long total = rows * vec_per_row;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const long long r = i / vec_per_row, c = i - r * vec_per_row;
        dst[r * dst_ld + c] = src[r * src_ld + c];
    }
}

static inline int grid_for(size_t work, int threads) {
    size_t g = (work + threads - 1) / threads;
    const size_t cap = 148 * 16;
    return static_cast<int>(g < 1 ? 1 : (g > cap ? cap : g));
}

}  // namespace rb

using namespace rb;

extern "C" int rb_gelu(const void* x, const void* dy, void* y, long long n, int mode, int dtype,
                       void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (n <= 0) return 0;
    if (off16(x, dy, y)) return -5;
    const int g = grid_for(n / 8 + 1, 256);
    if (dtype == 1)
        gelu_kernel<__nv_bfloat16><<<g, 256, 0, st>>>(static_cast<const __nv_bfloat16*>(x),
                                                     static_cast<const __nv_bfloat16*>(dy),
                                                     static_cast<__nv_bfloat16*>(y), n, mode);
    else
        gelu_kernel<__half><<<g, 256, 0, st>>>(static_cast<const __half*>(x),
                                              static_cast<const __half*>(dy),
                                              static_cast<__half*>(y), n, mode);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

extern "C" int rb_dropout(const void* x, void* y, long long n, float p, uint64_t seed,
                          uint64_t offset, int dtype, void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (n <= 0) return 0;
    if (off16(x, y)) return -5;
    const uint32_t thr = drop_threshold(p);
    const float scale = 1.f / (1.f - p);
    const int g = grid_for(n / 8 + 1, 256);
    if (dtype == 1)
        dropout_kernel<__nv_bfloat16><<<g, 256, 0, st>>>(static_cast<const __nv_bfloat16*>(x),
                                                        static_cast<__nv_bfloat16*>(y), n, thr,
                                                        scale, seed, offset);
    else
        dropout_kernel<__half><<<g, 256, 0, st>>>(static_cast<const __half*>(x),
                                                 static_cast<__half*>(y), n, thr, scale, seed,
                                                 offset);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// out must be zeroed by the caller unless it accumulates on purpose
extern "C" int rb_colsum(const void* x, float* out, int M, int N, long long ld, int dtype,
                         void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (M <= 0 || N <= 0) return 0;
    if (N % 8 == 0 && ld % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0) {
        const int cols = (N + 255) / 256;
        int split = (148 * 6 + cols - 1) / cols;  // about six blocks per SM in total
        const int max_split = (M + 15) / 16;
        if (split > max_split) split = max_split;
        if (split < 1) split = 1;
        dim3 grid(cols, split), block(32, 8);
        if (dtype == 1)
            colsum_vec_kernel<__nv_bfloat16><<<grid, block, 0, st>>>(static_cast<const __nv_bfloat16*>(x), out, M,
                                                                    N, ld);
        else
            colsum_vec_kernel<__half><<<grid, block, 0, st>>>(static_cast<const __half*>(x), out, M, N, ld);
        return cudaGetLastError() == cudaSuccess ? 0 : -1;
    }
    int split = (M + 255) / 256;
    if (split > 64) split = 64;
    dim3 grid((N + 63) / 64, split), block(32, 8);
    if (dtype == 1)
        colsum_kernel<__nv_bfloat16><<<grid, block, 0, st>>>(static_cast<const __nv_bfloat16*>(x),
                                                            out, M, N, ld);
    else
        colsum_kernel<__half><<<grid, block, 0, st>>>(static_cast<const __half*>(x), out, M, N, ld);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

extern "C" int rb_accum_f32(float* dst, const void* src, long long n, float scale, int dtype,
                            void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (n <= 0) return 0;
    const int g = grid_for(n, 256);
    if (dtype == 1)
        accum_kernel<__nv_bfloat16><<<g, 256, 0, st>>>(dst, static_cast<const __nv_bfloat16*>(src),
                                                      n, scale);
    else
        accum_kernel<__half><<<g, 256, 0, st>>>(dst, static_cast<const __half*>(src), n, scale);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

extern "C" int rb_cast_from_f32(void* dst, const float* src, long long n, float scale, int dtype,
                                void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (n <= 0) return 0;
    const int g = grid_for(n, 256);
    if (dtype == 1)
        cast_kernel<__nv_bfloat16><<<g, 256, 0, st>>>(static_cast<__nv_bfloat16*>(dst), src, n,
                                                     scale);
    else
        cast_kernel<__half><<<g, 256, 0, st>>>(static_cast<__half*>(dst), src, n, scale);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// w: [3, wn] fp32 (w_fp32 != 0) or 16-bit; b: [3, bn] fp32 or null; all addresses on 16-byte boundaries
extern "C" int rb_unstack3(const void* w, int w_fp32, const float* b, void* const* wd, void* const* bd, long long wn,
                           long long bn, int dtype, void* stream) {
    if (wn % 8 || (b && bn % 8)) return -2;
    Unstack3 u = {w, b, {wd[0], wd[1], wd[2]}, {nullptr, nullptr, nullptr}, wn, bn};
    for (int i = 0; i < 3 && b; ++i) u.bd[i] = bd[i];
    if (wn <= 0) return 0;
    if (off16(w, b) || off16(u.wd[0], u.wd[1], u.wd[2], u.bd[0], u.bd[1], u.bd[2])) return -5;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int g = grid_for(3 * (wn + (b ? bn : 0)) / 8, 256);
    const auto kern = dtype == 1 ? (w_fp32 ? unstack3_kernel<__nv_bfloat16, float> : unstack3_kernel<__nv_bfloat16, uint16_t>)
                                 : (w_fp32 ? unstack3_kernel<__half, float> : unstack3_kernel<__half, uint16_t>);
    return launch_after(kern, g, 256, 0, st, u) == cudaSuccess ? 0 : -1;
}

extern "C" int rb_embed_fwd(const long long* ids, const void* table, void* out, int rows, int H,
                            long long vocab, int dtype, void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (rows <= 0) return 0;
    RB_DEBUG_ARG(H % 8 == 0, "rb_embed_fwd: H must be a multiple of 8");
    if (H % 8) return -2;
    if (off16(table, out)) return -5;
    RB_DEBUG_RANGE(ids, rows, 0, vocab, -1 - vocab, st);
    const int g = (rows * 32 + 255) / 256;
    const cudaError_t e =
        dtype == 1 ? launch_after(embed_fwd_kernel<__nv_bfloat16>, g, 256, 0, st, ids, static_cast<const __nv_bfloat16*>(table),
                                  static_cast<__nv_bfloat16*>(out), rows, H, vocab)
                   : launch_after(embed_fwd_kernel<__half>, g, 256, 0, st, ids, static_cast<const __half*>(table),
                                  static_cast<__half*>(out), rows, H, vocab);
    return e == cudaSuccess ? 0 : -1;
}

extern "C" int rb_embed_bwd(const long long* ids, const void* dout, float* dtable, int rows, int H,
                            long long vocab, long long padding_idx, int dtype, void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (rows <= 0) return 0;
    RB_DEBUG_RANGE(ids, rows, 0, vocab, padding_idx, st);
    if (H % 4 == 0 && ((reinterpret_cast<uintptr_t>(dout) | reinterpret_cast<uintptr_t>(dtable)) & 15) == 0) {
        const int nv = H / 4;
        // long strips save reductions where ids repeat, short ones keep the GPU busy on small batches: below
        // a million 4-element groups strips of 16 rows leave less than four warps per scheduler
        const bool longer = static_cast<long long>(rows) * nv >= (1LL << 20);
        const int strip = longer ? 16 : 4;
        const long long threads = (static_cast<long long>(rows) + strip - 1) / strip * nv;
        const unsigned blocks = static_cast<unsigned>((threads + 255) / 256);
        auto go = [&](auto* d) {
            using T = std::remove_const_t<std::remove_pointer_t<decltype(d)>>;
            return launch_after(longer ? embed_bwd_vec_kernel<T, 16> : embed_bwd_vec_kernel<T, 4>, blocks, 256, 0, st, ids, d,
                                dtable, rows, nv, vocab, padding_idx);
        };
        const cudaError_t e =
            dtype == 1 ? go(static_cast<const __nv_bfloat16*>(dout)) : go(static_cast<const __half*>(dout));
        return e == cudaSuccess ? 0 : -1;
    }
    const int g = (rows * 32 + 255) / 256;
    if (dtype == 1)
        embed_bwd_kernel<__nv_bfloat16><<<g, 256, 0, st>>>(
            ids, static_cast<const __nv_bfloat16*>(dout), dtable, rows, H, vocab, padding_idx);
    else
        embed_bwd_kernel<__half><<<g, 256, 0, st>>>(ids, static_cast<const __half*>(dout), dtable,
                                                   rows, H, vocab, padding_idx);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// src/dst row strides in bytes; bytes_per_row, strides and both bases 16 B aligned
extern "C" int rb_rowcopy(const void* src, void* dst, long long rows, long long bytes_per_row,
                          long long src_stride_bytes, long long dst_stride_bytes, void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (rows <= 0 || bytes_per_row <= 0) return 0;
    RB_DEBUG_ARG(((bytes_per_row | src_stride_bytes | dst_stride_bytes) & 15) == 0,
                 "rb_rowcopy: row length and strides must be multiples of 16 bytes");
    RB_DEBUG_ARG(((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0,
                 "rb_rowcopy: both buffers must be 16-byte aligned");
    RB_DEBUG_ARG(src_stride_bytes >= bytes_per_row && dst_stride_bytes >= bytes_per_row,
                 "rb_rowcopy: a row stride shorter than the row makes rows overlap");
    if ((bytes_per_row | src_stride_bytes | dst_stride_bytes) & 15) return -2;
    if ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) return -2;
    const long long vpr = bytes_per_row / 16;
    const int g = grid_for(static_cast<size_t>(rows * vpr), 256);
    rowcopy_kernel<<<g, 256, 0, st>>>(static_cast<const uint4*>(src), static_cast<uint4*>(dst),
                                      rows, vpr, src_stride_bytes / 16, dst_stride_bytes / 16);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}
