// Convolution support kernels and batch normalisation for channels-last (NHWC) activations.
//
// A convolution runs as a tcgen05 GEMM (gemm_tcgen05.cu): a 1x1 convolution IS a GEMM over the
// [N*H*W, C] view of an NHWC tensor, and a k x k convolution becomes one after `im2col` lays the k*k
// shifted windows of every output pixel side by side ([N*Ho*Wo, k*k*C], tap-major).  For the wide
// ResNets this framework is benchmarked on (C >= 512) the gathered matrix is read at more than 1000
// FLOP per byte, so the gather is a small fraction of the GEMM time.  `col2im` is the adjoint (input
// gradient), written as a gather so that no atomics are needed.
//
// Batch normalisation over [R = N*H*W, C]: per-channel sums in fp32 (one pass, 16-byte loads, 8 channels
// per thread), then one element-wise pass that normalises, optionally adds a residual and applies ReLU.
// Backward: one reduction pass (sum dy, sum dy * xhat, with the ReLU mask taken from the saved output),
// one element-wise pass.  Running statistics are updated by the finalising kernel, per replica (no
// cross-rank synchronisation), like the reference, which runs aten::batch_norm inside each replica's
// TorchScript interpreter (src/torch/TorchDriver.cpp:566) and treats the statistics as non-gradient
// parameters (src/comp/ParamStorage.cpp:209-211).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "launch.cuh"
#include "tc_common.cuh"

namespace rb {

template <typename T>
__device__ __forceinline__ void ld8(const T* p, float (&v)[8]) {
    const uint4 q = *reinterpret_cast<const uint4*>(p);
    const T* e = reinterpret_cast<const T*>(&q);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = to_f32<T>(e[j]);
}
template <typename T>
__device__ __forceinline__ void st8(T* p, const float (&v)[8]) {
    uint4 q;
    q.x = pack2<T>(v[0], v[1]);
    q.y = pack2<T>(v[2], v[3]);
    q.z = pack2<T>(v[4], v[5]);
    q.w = pack2<T>(v[6], v[7]);
    *reinterpret_cast<uint4*>(p) = q;
}

// ---------------------------------------------------------------------------------------------------
// im2col / col2im, NHWC, square kernel k, stride s, padding pad.  C % 8 == 0.
// cols[(n, ho, wo), (ky, kx, c)] = x[n, ho*s - pad + ky, wo*s - pad + kx, c]  (0 outside)
// ---------------------------------------------------------------------------------------------------
template <typename T>
__global__ void im2col_kernel(const T* __restrict__ x, T* __restrict__ cols, int N, int H, int W, int C, int Ho,
                              int Wo, int k, int s, int pad) {
    // one thread per (output pixel, 8 channels): the pixel coordinates are decoded once, the taps are a loop
    const int cv = C / 8;
    const long long total = static_cast<long long>(N) * Ho * Wo * cv;
    const long long row_len = static_cast<long long>(k) * k * C;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int c8 = static_cast<int>(i % cv);
        const long long pix = i / cv;
        const int wo = static_cast<int>(pix % Wo);
        const int ho = static_cast<int>((pix / Wo) % Ho);
        const int n = static_cast<int>(pix / (static_cast<long long>(Wo) * Ho));
        const T* xin = x + static_cast<long long>(n) * H * W * C + c8 * 8;
        T* out = cols + pix * row_len + c8 * 8;
        for (int ky = 0; ky < k; ++ky) {
            const int h = ho * s - pad + ky;
            const bool hin = h >= 0 && h < H;
#pragma unroll 3
            for (int kx = 0; kx < k; ++kx) {
                const int w = wo * s - pad + kx;
                uint4 v = make_uint4(0, 0, 0, 0);
                if (hin && w >= 0 && w < W)
                    v = *reinterpret_cast<const uint4*>(xin + (static_cast<long long>(h) * W + w) * C);
                *reinterpret_cast<uint4*>(out + static_cast<long long>(ky * k + kx) * C) = v;
            }
        }
    }
}

// dx[n, h, w, c] = sum over the taps (ky, kx) and output pixels that read (h, w) of dcols
template <typename T>
__global__ void col2im_kernel(const T* __restrict__ dcols, T* __restrict__ dx, int N, int H, int W, int C, int Ho,
                              int Wo, int k, int s, int pad) {
    const int cv = C / 8;
    const long long total = static_cast<long long>(N) * H * W * cv;
    const long long row_len = static_cast<long long>(k) * k * C;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int c8 = static_cast<int>(i % cv);
        long long r = i / cv;
        const int w = static_cast<int>(r % W);
        r /= W;
        const int h = static_cast<int>(r % H);
        const int n = static_cast<int>(r / H);
        float acc[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = 0.f;
        for (int ky = 0; ky < k; ++ky) {
            const int hn = h + pad - ky;
            if (hn < 0 || hn % s) continue;
            const int ho = hn / s;
            if (ho >= Ho) continue;
            for (int kx = 0; kx < k; ++kx) {
                const int wn = w + pad - kx;
                if (wn < 0 || wn % s) continue;
                const int wo = wn / s;
                if (wo >= Wo) continue;
                float v[8];
                ld8(dcols + ((static_cast<long long>(n) * Ho + ho) * Wo + wo) * row_len +
                        (static_cast<long long>(ky) * k + kx) * C + c8 * 8,
                    v);
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[j] += v[j];
            }
        }
        st8(dx + i * 8, acc);
    }
}

// ---------------------------------------------------------------------------------------------------
// Operands of the implicit-GEMM convolution
// ---------------------------------------------------------------------------------------------------
// out [N, H + pad, W + pad, C] = x [N, H, W, C] with zero columns behind every row and zero rows behind every image;
// one block per padded image row.  Bound by memory: one pass that reads x once and writes every output vector once (a
// generic pad clears the output and then copies the interior with a strided kernel: 32 x 28 x 28 x 1024 took 80 us
// that way; this takes 16.4 us, of which a launch beside the end of the kernel before saves 1.6).
__global__ void __launch_bounds__(256)
    pad_nhwc_kernel(const uint4* x, uint4* out, int H, int W, int cv, int pad) {
    grid_trigger();
    grid_wait();
    const int Wp = W + pad, Hp = H + pad;
    const int n = blockIdx.x / Hp, y = blockIdx.x - n * Hp;
    uint4* o = out + static_cast<long long>(blockIdx.x) * Wp * cv;
    const uint4* row = x + (static_cast<long long>(n) * H + y) * W * cv;
    const int live = y < H ? W * cv : 0;
    for (int i = threadIdx.x; i < Wp * cv; i += 4 * 256) {
        uint4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = i + u * 256 < live ? row[i + u * 256] : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i + u * 256 < Wp * cv) o[i + u * 256] = v[u];
    }
}

// A filter [Co, Ci, taps] as the GEMM reads it, [Co, taps, Ci]; 16-bit elements, Ci a multiple of 8.  A block takes CH
// channels of one filter through shared memory, so that both sides move in 16-byte pieces of consecutive addresses (a
// generic strided copy reads 2 bytes of every 18: 1024 x 1024 x 3 x 3 took 258 us that way and takes 10.3 us here,
// 2048 x 2048 333 and 39 us).  The padded rows shift the banks by four from tap to tap.  CH shrinks as the taps grow, to stay below 48 KiB.
template <int CH>
__global__ void __launch_bounds__(256)
    pack_taps_kernel(const uint16_t* src, uint16_t* dst, int Ci, int taps, int chunks) {
    grid_trigger();
    grid_wait();
    constexpr int LD = CH + 8;
    extern __shared__ uint4 pack_smem[];
    uint16_t* tile = reinterpret_cast<uint16_t*>(pack_smem);  // [taps][LD]
    const int co = blockIdx.x / chunks, c0 = (blockIdx.x - co * chunks) * CH, nc = min(CH, Ci - c0);
    const uint4* from = reinterpret_cast<const uint4*>(src + (static_cast<long long>(co) * Ci + c0) * taps);
    const int pieces = nc * taps / 8, row = nc / 8;
    for (int v = threadIdx.x; v < pieces; v += 256) {
        const uint4 q = from[v];
        const uint16_t* e = reinterpret_cast<const uint16_t*>(&q);
        int c = v * 8 / taps, t = v * 8 - c * taps;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            tile[t * LD + c] = e[j];
            if (++t == taps) t = 0, ++c;
        }
    }
    __syncthreads();
    uint16_t* to = dst + static_cast<long long>(co) * taps * Ci + c0;
    for (int v = threadIdx.x; v < pieces; v += 256) {
        const int t = v / row, c = (v - t * row) * 8;
        *reinterpret_cast<uint4*>(to + static_cast<long long>(t) * Ci + c) = *reinterpret_cast<const uint4*>(tile + t * LD + c);
    }
}
// The same for 2 x 2 and 3 x 3 filters, 256 channels a block: the 8 * TAPS values of eight channels lie in shared memory as
// they came, one word more apart, so that a thread's eight gathered values and its neighbours' are in different banks.
// us, the kernel above and this: 64 x 64 x 3 x 3 1.7 -> 1.4, 1024 x 1024 10.3 -> 6.0, 2048 x 2048 39 -> 28 (5.3 TB/s),
// 1024 x 1024 x 2 x 2 6.6 -> 3.8.  (There a thread's values go to shared memory one by one, four to a bank.)
template <int TAPS>
__global__ void __launch_bounds__(TAPS * 32)
    pack_few_kernel(const uint4* src, uint4* dst, int Ci, int chunks) {
    constexpr int LD = 8 * TAPS / 2 + 1;   // words of eight channels
    __shared__ uint32_t tile[32 * LD];
    grid_wait();
    const int co = blockIdx.x / chunks, g0 = (blockIdx.x - co * chunks) * 32, ng = min(32, Ci / 8 - g0);   // groups of 8
    const int i = threadIdx.x, t = i >> 5, lane = i & 31;
    if (i < ng * TAPS) {
        const uint4 q = src[(static_cast<long long>(co) * (Ci / 8) + g0) * TAPS + i];
        uint32_t* to = tile + i / TAPS * LD + i % TAPS * 4;
        to[0] = q.x, to[1] = q.y, to[2] = q.z, to[3] = q.w;
    }
    __syncthreads();
    if (lane >= ng) return;
    const uint16_t* e = reinterpret_cast<const uint16_t*>(tile + lane * LD) + t;
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = e[2 * j * TAPS] | static_cast<uint32_t>(e[(2 * j + 1) * TAPS]) << 16;
    dst[(static_cast<long long>(co) * TAPS + t) * (Ci / 8) + g0 + lane] = make_uint4(w[0], w[1], w[2], w[3]);
}
template <int TAPS>
static int pack_few_launch(const void* src, void* dst, int Co, int Ci, cudaStream_t st) {
    const int chunks = (Ci + 255) / 256;
    if (static_cast<long long>(Co) * chunks > 0x7fffffffLL) return -2;
    return launch_after(pack_few_kernel<TAPS>, static_cast<unsigned>(Co) * chunks, TAPS * 32, 0, st,
                        static_cast<const uint4*>(src), static_cast<uint4*>(dst), Ci, chunks) == cudaSuccess ? 0 : -1;
}
template <int CH>
static int pack_taps_launch(const void* src, void* dst, int Co, int Ci, int taps, cudaStream_t st) {
    const int chunks = (Ci + CH - 1) / CH;
    if (static_cast<long long>(Co) * chunks > 0x7fffffffLL) return -2;
    return launch_after(pack_taps_kernel<CH>, static_cast<unsigned>(Co) * chunks, 256, taps * (CH + 8) * 2, st,
                        static_cast<const uint16_t*>(src), static_cast<uint16_t*>(dst), Ci, taps, chunks) == cudaSuccess
               ? 0
               : -1;
}

// The weight gradient comes out of its GEMM as src [Co, taps, Ci] fp32 and belongs into a [Co, Ci, taps] tensor:
// added to an fp32 gradient buffer (ADD) or rounded to a 16-bit gradient.  A block takes 128 channels of one
// filter through shared memory so that both sides are touched in whole lines; the row stride shifts the banks by four
// from tap to tap.  For filters from 4 x 4 to 9 x 9 (and any number of channels): a strided copy reads 4 bytes of every
// 4 * taps, which costs it 107 us for 1024 x 1024 x 5 x 5 (added to fp32) where this takes 72.  Smaller filters have the
// kernel below: here a block's loads, its barrier and its stores follow one another with little in flight.
constexpr int FOLD_C = 128, FOLD_LD = FOLD_C + 4;
template <typename OutT, bool ADD>
__global__ void __launch_bounds__(256)
    wgrad_fold_kernel(const float* __restrict__ src, OutT* __restrict__ dst, int Ci, int taps) {
    extern __shared__ float tile[];  // [taps][FOLD_LD]
    const int c0 = blockIdx.x * FOLD_C, nc = min(FOLD_C, Ci - c0);
    const long long co = blockIdx.y;
    src += co * taps * Ci + c0;
    dst += (co * Ci + c0) * taps;
#pragma unroll 5
    for (int i = threadIdx.x; i < taps * FOLD_C; i += 256) {
        const int t = i / FOLD_C, c = i - t * FOLD_C;
        if (c < nc) tile[t * FOLD_LD + c] = src[static_cast<long long>(t) * Ci + c];
    }
    __syncthreads();
#pragma unroll 5
    for (int i = threadIdx.x; i < taps * nc; i += 256) {
        const int c = i / taps, t = i - c * taps;
        const float v = tile[t * FOLD_LD + c];
        if constexpr (ADD)
            dst[i] += v;
        else
            dst[i] = from_f32<OutT>(v);
    }
}

// The same for the filters of 2 x 2 and 3 x 3, whose taps are known to the compiler: what is added to, and the 256
// channels of every tap (a warp has one), are on their way to a block before it waits for either, in 16-byte pieces, and
// the results leave in such.  Bound by memory.  us, the strided operation and this, added to fp32 and rounded to 16 bits:
// 512 x 512 x 3 x 3 8.4 -> 3.7 and 8.4 -> 2.9, 1024 x 1024 24.7 -> 10.7 and 20.6 -> 7.7, 2048 x 2048 (from memory) 121 -> 66
// and 80 -> 36, 1024 x 1024 x 2 x 2 12.5 -> 5.9 and 10.6 -> 3.9; 128 channels a block: 11.5 where this takes 10.7.
constexpr int FEW_C = 256;
template <typename OutT, bool ADD, int TAPS>
__global__ void __launch_bounds__(TAPS * 32)
    wgrad_fold_few_kernel(const float* src, OutT* dst, int Ci, int chunks) {
    constexpr int U = FEW_C / 128, LD = FEW_C + 4, V = 16 / sizeof(OutT);
    constexpr int OUTS = FEW_C / V / 32;   // vectors of the result a thread writes
    __shared__ __align__(16) float tile[TAPS * LD];
    grid_wait();
    const int co = blockIdx.x / chunks, c0 = (blockIdx.x - co * chunks) * FEW_C, nc = min(FEW_C, Ci - c0);
    src += static_cast<long long>(co) * TAPS * Ci + c0;
    dst += (static_cast<long long>(co) * Ci + c0) * TAPS;
    const int nv = nc * TAPS / V;
    uint4 old[OUTS];
    if constexpr (ADD) {
#pragma unroll
        for (int u = 0; u < OUTS; ++u) {
            const int i = threadIdx.x + u * TAPS * 32;
            if (i < nv) old[u] = reinterpret_cast<const uint4*>(dst)[i];
        }
    }
    float4 in[U];
    const int t = threadIdx.x >> 5, lane = threadIdx.x & 31;   // a warp has a tap
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int c = (u * 32 + lane) * 4;
        if (c < nc) in[u] = *reinterpret_cast<const float4*>(src + static_cast<long long>(t) * Ci + c);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) *reinterpret_cast<float4*>(tile + t * LD + (u * 32 + lane) * 4) = in[u];
    __syncthreads();
#pragma unroll
    for (int u = 0; u < OUTS; ++u) {
        const int i = threadIdx.x + u * TAPS * 32;
        if (i >= nv) break;
        float v[V];
#pragma unroll
        for (int j = 0; j < V; ++j) {
            const int e = i * V + j, c = e / TAPS;
            v[j] = tile[(e - c * TAPS) * LD + c];
        }
        if constexpr (ADD) {
            const float* o = reinterpret_cast<const float*>(&old[u]);
            reinterpret_cast<float4*>(dst)[i] = make_float4(o[0] + v[0], o[1] + v[1], o[2] + v[2], o[3] + v[3]);
        } else {
            st8(dst + i * V, v);
        }
    }
}
template <int TAPS>
static int wgrad_fold_few(const float* src, void* dst, int Co, int Ci, int dtype, cudaStream_t st) {
    const int chunks = (Ci + FEW_C - 1) / FEW_C;
    if (static_cast<long long>(Co) * chunks > 0x7fffffffLL) return -2;
    const unsigned grid = static_cast<unsigned>(Co) * chunks;
    const cudaError_t e =
        dtype == 2   ? launch_after(wgrad_fold_few_kernel<float, true, TAPS>, grid, TAPS * 32, 0, st, src,
                                    static_cast<float*>(dst), Ci, chunks)
        : dtype == 1 ? launch_after(wgrad_fold_few_kernel<__nv_bfloat16, false, TAPS>, grid, TAPS * 32, 0, st, src,
                                    static_cast<__nv_bfloat16*>(dst), Ci, chunks)
                     : launch_after(wgrad_fold_few_kernel<__half, false, TAPS>, grid, TAPS * 32, 0, st, src,
                                    static_cast<__half*>(dst), Ci, chunks);
    return e == cudaSuccess ? 0 : -1;
}

// ---------------------------------------------------------------------------------------------------
// batch norm
// ---------------------------------------------------------------------------------------------------
__device__ __forceinline__ void ldf8(const float* p, float (&v)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(p);
    const float4 b = *reinterpret_cast<const float4*>(p + 4);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}
// parameters may be views of a flat buffer that start at any element
__device__ __forceinline__ void ldf8_any(const float* p, float (&v)[8]) {
    if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
        ldf8(p, v);
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = p[j];
    }
}

// A thread owns 8 adjacent channels (16 bytes a row) in every kernel here; a block of (BX, 256 / BX) threads covers
// BX * 8 channels, rows are strided over threadIdx.y and blockIdx.y.  BX follows the channel count, so that a layer of
// 64 channels does not leave three quarters of its threads without one.
// Sums over a block's rows: part[blockIdx.y][0][c] = sum_r a(r, c), part[blockIdx.y][1][c] = sum_r a(r, c) * b(r, c)
//   MODE 0 (statistics):  a = x,                 b = x
//   MODE 1 (backward):    a = dy masked by relu, b = xhat = (x - mean) * rstd
template <typename T, int MODE, int BX>
__global__ void __launch_bounds__(256)
    bn_reduce_kernel(const T* x, const T* dy, const T* y, const float* mean, const float* rstd, float* part, long long R,
                     int C, int relu) {
    constexpr int TY = 256 / BX;
    __shared__ float red[2][TY][BX * 8 + 8];
    grid_wait();
    const int col = (blockIdx.x * BX + threadIdx.x) * 8;
    float s0[8], s1[8], mu[8], rs[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) s0[j] = s1[j] = 0.f, mu[j] = 0.f, rs[j] = 1.f;
    if (col < C) {
        if (MODE == 1) {
#pragma unroll
            for (int j = 0; j < 8; ++j) mu[j] = mean[col + j], rs[j] = rstd[col + j];
        }
        for (long long r = blockIdx.y * TY + threadIdx.y; r < R; r += static_cast<long long>(gridDim.y) * TY) {
            float a[8];
            ld8(x + r * C + col, a);
            if (MODE == 0) {
#pragma unroll
                for (int j = 0; j < 8; ++j) s0[j] += a[j], s1[j] = fmaf(a[j], a[j], s1[j]);
            } else {
                float g[8];
                ld8(dy + r * C + col, g);
                if (relu) {
                    float o[8];
                    ld8(y + r * C + col, o);
#pragma unroll
                    for (int j = 0; j < 8; ++j) g[j] = o[j] > 0.f ? g[j] : 0.f;
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) s0[j] += g[j], s1[j] = fmaf(g[j], (a[j] - mu[j]) * rs[j], s1[j]);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        red[0][threadIdx.y][threadIdx.x * 8 + j] = s0[j];
        red[1][threadIdx.y][threadIdx.x * 8 + j] = s1[j];
    }
    __syncthreads();
    const int t = threadIdx.y * BX + threadIdx.x;
    if (t >= BX * 8) return;
    float a0 = 0.f, a1 = 0.f;
#pragma unroll
    for (int w = 0; w < TY; ++w) a0 += red[0][w][t], a1 += red[1][w][t];
    const int c = blockIdx.x * BX * 8 + t;
    part += blockIdx.y * 2LL * C;
    if (c < C) {
        part[c] = a0;
        part[C + c] = a1;
    }
}

// The blocks' sums added up, in fp64 and in a fixed order: total[0 .. 2 C).  (By atomics, in the order they arrived, the last
// bits of a total changed from run to run, and a result of the norm that lies next to zero fell on either side of the ReLU,
// with dy or 0 for its gradient.)  Bound by latency: a block has 16 columns only, and 128 rows on their way at a time.
__global__ void __launch_bounds__(512) bn_total_kernel(const float* part, int parts, int C, float* total) {
    __shared__ double red[16][16];
    grid_trigger();
    grid_wait();
    const int t = threadIdx.x, col = blockIdx.x * 16 + (t & 3) * 4;   // (2 C is a multiple of 16)
    double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 5
    for (int r = t >> 2; r < parts; r += 128) {
        const float4 v = *reinterpret_cast<const float4*>(part + r * 2LL * C + col);
        s[0] += v.x, s[1] += v.y, s[2] += v.z, s[3] += v.w;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) s[j] += __shfl_xor_sync(0xffffffffu, s[j], o);
        if ((t & 31) < 4) red[t >> 5][t * 4 % 16 + j] = s[j];
    }
    __syncthreads();
    if (t >= 16) return;
    double sum = 0.0;
#pragma unroll
    for (int w = 0; w < 16; ++w) sum += red[w][t];
    total[blockIdx.x * 16 + t] = static_cast<float>(sum);
}

// y = act(x * scale + shift (+ residual)) with scale = rstd gamma and shift = beta - mean scale.  Every thread derives
// its 8 channels' scale and shift from the two sums itself (a kernel of C threads in between cost 3 us and a launch for
// a few hundred cycles of arithmetic: 32 x 14 x 14 x 2048 with residual 13.6 + 3.1 -> 12.6 us, its backward below 18.6 +
// 2.2 -> 17.3 us); the first row of blocks also writes mean, rstd and the running statistics (momentum, unbiased
// variance).  Bound by memory: four rows of a thread are on their way at a time, the first while the coefficients are
// computed, and rows are taken from the last one on, because the reduction has just read those and they are still in
// the L2 cache.
template <typename T, int BX>
__global__ void __launch_bounds__(256)
    bn_apply_kernel(const T* x, const T* res, const float* part, const float* gamma, const float* beta, float* mean,
                    float* rstd, float* run_mean, float* run_var, T* y, long long R, int C, float eps, float momentum,
                    int relu) {
    constexpr int TY = 256 / BX;
    const int col = (blockIdx.x * BX + threadIdx.x) * 8;
    grid_wait();
    if (col >= C) return;
    const long long step = static_cast<long long>(gridDim.y) * TY;
    long long r0 = blockIdx.y * TY + threadIdx.y;
    uint4 qx[4], qr[4];   // (loads written out: the compiler may not move one before another row's store)
    auto fetch = [&](long long r0) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const long long r = r0 + u * step;
            if (r >= R) break;
            qx[u] = *reinterpret_cast<const uint4*>(x + (R - 1 - r) * C + col);
            if (res) qr[u] = *reinterpret_cast<const uint4*>(res + (R - 1 - r) * C + col);
        }
    };
    fetch(r0);   // beside the coefficients' arithmetic
    float sc[8], sh[8], p0[8], p1[8];
    ldf8(part + col, p0);
    ldf8(part + C + col, p1);
    ldf8_any(gamma + col, sc);
    ldf8_any(beta + col, sh);
    const float inv = 1.f / static_cast<float>(R);
    const bool writer = blockIdx.y == 0 && threadIdx.y == 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int c = col + j;
        const float m = p0[j] * inv;
        const float var = fmaxf(p1[j] * inv - m * m, 0.f);
        const float rs = rsqrtf(var + eps);
        sc[j] = rs * sc[j];
        sh[j] = sh[j] - m * sc[j];
        if (writer) {
            mean[c] = m;
            rstd[c] = rs;
            if (run_mean) {
                const float unbiased = R > 1 ? var * static_cast<float>(R) / static_cast<float>(R - 1) : var;
                run_mean[c] = (1.f - momentum) * run_mean[c] + momentum * m;
                run_var[c] = (1.f - momentum) * run_var[c] + momentum * unbiased;
            }
        }
    }
    while (r0 < R) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const long long r = r0 + u * step;
            if (r >= R) break;
            float v[8], o[8];
            ld8(reinterpret_cast<const T*>(&qx[u]), v);
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] = fmaf(v[j], sc[j], sh[j]);
            if (res) {
                float rr[8];
                ld8(reinterpret_cast<const T*>(&qr[u]), rr);
#pragma unroll
                for (int j = 0; j < 8; ++j) o[j] += rr[j];
            }
            if (relu) {
#pragma unroll
                for (int j = 0; j < 8; ++j) o[j] = fmaxf(o[j], 0.f);
            }
            st8(y + (R - 1 - r) * C + col, o);
        }
        fetch(r0 += 4 * step);
    }
}

// dx = A g + B x + Cc, g = dy masked by relu, with A = gamma rstd, B = -A rstd sum(g xhat) / R and
// Cc = -A sum(g) / R - B mean derived per thread from the two sums; dres = g (optional).  The first row of blocks adds
// the sums to the fp32 gradients of beta and gamma when it is given their buffers.
template <typename T, int BX>
__global__ void __launch_bounds__(256)
    bn_bwd_apply_kernel(const T* x, const T* dy, const T* y, const float* part, const float* mean, const float* rstd,
                        const float* gamma, float* dgamma, float* dbeta, T* dx, T* dres, long long R, int C, int relu) {
    constexpr int TY = 256 / BX;
    const int col = (blockIdx.x * BX + threadIdx.x) * 8;
    grid_wait();
    if (col >= C) return;
    float A[8], B[8], Cc[8], p0[8], p1[8], rs[8], mu[8];
    ldf8(part + col, p0);
    ldf8(part + C + col, p1);
    ldf8_any(gamma + col, A);
    ldf8(rstd + col, rs);
    ldf8(mean + col, mu);
    const float inv = 1.f / static_cast<float>(R);
    const bool writer = blockIdx.y == 0 && threadIdx.y == 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int c = col + j;
        A[j] = A[j] * rs[j];
        B[j] = -A[j] * rs[j] * p1[j] * inv;
        Cc[j] = -A[j] * p0[j] * inv - B[j] * mu[j];
        if (writer && dgamma) dgamma[c] += p1[j];
        if (writer && dbeta) dbeta[c] += p0[j];
    }
    const long long step = static_cast<long long>(gridDim.y) * TY;
    for (long long r0 = blockIdx.y * TY + threadIdx.y; r0 < R; r0 += 2 * step) {  // (two rows' loads, as above)
        uint4 qx[2], qd[2], qy[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const long long r = r0 + u * step;
            if (r >= R) break;
            qx[u] = *reinterpret_cast<const uint4*>(x + (R - 1 - r) * C + col);
            qd[u] = *reinterpret_cast<const uint4*>(dy + (R - 1 - r) * C + col);
            if (relu) qy[u] = *reinterpret_cast<const uint4*>(y + (R - 1 - r) * C + col);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const long long r = r0 + u * step;
            if (r >= R) break;
            float v[8], g[8], o[8];
            ld8(reinterpret_cast<const T*>(&qx[u]), v);
            ld8(reinterpret_cast<const T*>(&qd[u]), g);
            if (relu) {
                float yy[8];
                ld8(reinterpret_cast<const T*>(&qy[u]), yy);
#pragma unroll
                for (int j = 0; j < 8; ++j) g[j] = yy[j] > 0.f ? g[j] : 0.f;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] = fmaf(A[j], g[j], fmaf(B[j], v[j], Cc[j]));
            st8(dx + (R - 1 - r) * C + col, o);
            if (dres) st8(dres + (R - 1 - r) * C + col, g);
        }
    }
}

// Grid of the batch-norm kernels: blocks of BX * 8 channels, and as many row groups as give the whole grid about
// `per_sm` blocks per SM, each with four rows or more per thread.  per_sm is what an SM holds at once of the kernel with
// its registers (40 to 101 a thread), so that there is one wave: 4 for the reductions, 2 for the element-wise passes (at four
// with half the rows in flight, or held to 64 registers, those take longer).  The reductions' grid also decides which rows
// make up a sum, and with it the last bits of the statistics: four blocks per SM, as it was when sums met by atomics.
// Forward + backward in a captured graph, one B200 (us), at ordinary launches with atomics into memory that a memset had
// cleared, and now: 6272 x 2048 with residual and ReLU 15.6 + 34.1 -> 16.1 + 33.5, 25088 x 1024 with ReLU 23.4 + 63.1 -> 26.3
// + 57.5, 100352 x 256 with both 40.6 + 76.1 -> 36.1 + 67.8, 401408 x 64 with ReLU 26.0 + 65.0 -> 25.5 + 56.4.  With atomics,
// and a kernel that clears in the place of the memset, these take 15.1 + 32.3, 25.5 + 56.0, 36.9 + 67.2 and 26.0 + 54.6: what a
// fixed order costs.  (fp64 atomics, whose order hardly shows, take as long: 29.3 + 54 at 401408 x 64.)
// Neither the reductions nor the passes let the next kernel begin by grid_trigger(): a GEMM that does waits on the SMs with its
// shared memory, and the first-level cache that this leaves to them costs more (a 1x1 convolution of 32 x 14 x 14 x 2048 with
// its norm, forward and backward, 131.6 us of device time with the triggers, 120.3 without, 128.5 at ordinary launches).
template <int BX>
static dim3 bn_grid(long long R, int C, int per_sm) {
    const int cols = (C + BX * 8 - 1) / (BX * 8);
    long long split = (R + 4 * (256 / BX) - 1) / (4 * (256 / BX));
    const long long want = (148LL * per_sm + cols - 1) / cols;
    if (split > want) split = want;
    return dim3(cols, static_cast<unsigned>(split < 1 ? 1 : split));
}

// the reductions' blocks along the rows
static long long bn_parts(long long R, int C) {
    return (C >= 256 ? bn_grid<32>(R, C, 4) : C > 64 ? bn_grid<16>(R, C, 4) : bn_grid<8>(R, C, 4)).y;
}

// total: fp32 [2, C], and behind it the parts
template <typename T, int MODE, int BX>
static cudaError_t bn_reduce(const T* x, const T* dy, const T* y, const float* mean, const float* rstd, float* total, long long R,
                             int C, int relu, cudaStream_t st) {
    const dim3 grid = bn_grid<BX>(R, C, 4);
    float* part = total + 2LL * C;
    const cudaError_t e = launch_after(bn_reduce_kernel<T, MODE, BX>, grid, dim3(BX, 256 / BX), 0, st, x, dy, y, mean, rstd, part,
                                       R, C, relu);
    if (e != cudaSuccess) return e;
    return launch_after(bn_total_kernel, C / 8, 512, 0, st, part, static_cast<int>(grid.y), C, total);
}

template <typename T, int BX>
static int bn_fwd_launch(const void* x, const void* res, const float* gamma, const float* beta, void* y, float* part,
                         float* mean, float* rstd, float* run_mean, float* run_var, long long R, int C, float eps,
                         float momentum, int relu, cudaStream_t st) {
    const dim3 block(BX, 256 / BX);
    const T* xt = static_cast<const T*>(x);
    if (bn_reduce<T, 0, BX>(xt, nullptr, nullptr, nullptr, nullptr, part, R, C, 0, st) != cudaSuccess) return -1;
    const cudaError_t e = launch_after(bn_apply_kernel<T, BX>, bn_grid<BX>(R, C, 2), block, 0, st, xt,
                                       static_cast<const T*>(res), part, gamma, beta, mean, rstd, run_mean, run_var,
                                       static_cast<T*>(y), R, C, eps, momentum, relu);
    return e == cudaSuccess ? 0 : -1;
}
template <typename T, int BX>
static int bn_bwd_launch(const void* x, const void* dy, const void* y, const float* mean, const float* rstd,
                         const float* gamma, float* part, float* dgamma, float* dbeta, void* dx, void* dres, long long R,
                         int C, int relu, cudaStream_t st) {
    const dim3 block(BX, 256 / BX);
    const T *xt = static_cast<const T*>(x), *dt = static_cast<const T*>(dy), *yt = static_cast<const T*>(y);
    if (bn_reduce<T, 1, BX>(xt, dt, yt, mean, rstd, part, R, C, relu, st) != cudaSuccess) return -1;
    const cudaError_t e = launch_after(bn_bwd_apply_kernel<T, BX>, bn_grid<BX>(R, C, 2), block, 0, st, xt, dt, yt, part, mean,
                                       rstd, gamma, dgamma, dbeta, static_cast<T*>(dx), static_cast<T*>(dres), R, C, relu);
    return e == cudaSuccess ? 0 : -1;
}

static inline int ew_grid(long long n) {
    long long g = (n + 255) / 256;
    const long long cap = 148LL * 16;
    return static_cast<int>(g < 1 ? 1 : (g > cap ? cap : g));
}

}  // namespace rb

// dtype: 1 = bf16, 0 = fp16
extern "C" int rb_im2col(const void* x, void* cols, int N, int H, int W, int C, int k, int s, int pad, int dtype,
                         void* stream) {
    using namespace rb;
    if (C % 8 || k < 1 || s < 1) return -2;
    const int Ho = (H + 2 * pad - k) / s + 1, Wo = (W + 2 * pad - k) / s + 1;
    if (Ho <= 0 || Wo <= 0) return -2;
    if (off16(x, cols)) return -5;
    const long long total = static_cast<long long>(N) * Ho * Wo * k * k * (C / 8);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (dtype == 1)
        im2col_kernel<__nv_bfloat16><<<ew_grid(total), 256, 0, st>>>(
            static_cast<const __nv_bfloat16*>(x), static_cast<__nv_bfloat16*>(cols), N, H, W, C, Ho, Wo, k, s, pad);
    else
        im2col_kernel<__half><<<ew_grid(total), 256, 0, st>>>(static_cast<const __half*>(x),
                                                             static_cast<__half*>(cols), N, H, W, C, Ho, Wo, k, s, pad);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

extern "C" int rb_col2im(const void* dcols, void* dx, int N, int H, int W, int C, int k, int s, int pad, int dtype,
                         void* stream) {
    using namespace rb;
    if (C % 8 || k < 1 || s < 1) return -2;
    const int Ho = (H + 2 * pad - k) / s + 1, Wo = (W + 2 * pad - k) / s + 1;
    if (Ho <= 0 || Wo <= 0) return -2;
    if (off16(dcols, dx)) return -5;
    const long long total = static_cast<long long>(N) * H * W * (C / 8);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (dtype == 1)
        col2im_kernel<__nv_bfloat16><<<ew_grid(total), 256, 0, st>>>(
            static_cast<const __nv_bfloat16*>(dcols), static_cast<__nv_bfloat16*>(dx), N, H, W, C, Ho, Wo, k, s, pad);
    else
        col2im_kernel<__half><<<ew_grid(total), 256, 0, st>>>(static_cast<const __half*>(dcols),
                                                             static_cast<__half*>(dx), N, H, W, C, Ho, Wo, k, s, pad);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// x [N, H, W, C] -> out [N, H + pad, W + pad, C], 16-bit elements, zeros behind every row and image
extern "C" int rb_pad_nhwc(const void* x, void* out, int N, int H, int W, int C, int pad, void* stream) {
    if (C % 8 || pad < 0 || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out)) & 15)) return -2;
    if (N <= 0 || H <= 0 || W <= 0) return 0;
    return rb::launch_after(rb::pad_nhwc_kernel, static_cast<unsigned>(N) * (H + pad), 256, 0, static_cast<cudaStream_t>(stream),
                            static_cast<const uint4*>(x), static_cast<uint4*>(out), H, W, C / 8, pad) == cudaSuccess
               ? 0
               : -1;
}

// 16-bit filter src [Co, Ci, taps] -> dst [Co, taps, Ci]
extern "C" int rb_pack_taps(const void* src, void* dst, int Co, int Ci, int taps, void* stream) {
    using namespace rb;
    if (Co <= 0 || Ci <= 0 || taps <= 0) return 0;
    if (Ci % 8 || taps > 1024 || ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15)) return -2;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (taps == 9) return pack_few_launch<9>(src, dst, Co, Ci, st);
    if (taps == 4) return pack_few_launch<4>(src, dst, Co, Ci, st);
    const auto fits = [&](int ch) { return taps * (ch + 8) * 2 <= 48 * 1024; };
    if (fits(256)) return pack_taps_launch<256>(src, dst, Co, Ci, taps, st);
    return fits(64) ? pack_taps_launch<64>(src, dst, Co, Ci, taps, st) : pack_taps_launch<16>(src, dst, Co, Ci, taps, st);
}

// rb_wgrad_fold for 4 or 9 taps, Ci a multiple of 8, both addresses on 16-byte boundaries
extern "C" int rb_wgrad_fold_few(const float* src, void* dst, int Co, int Ci, int taps, int dtype, void* stream) {
    using namespace rb;
    if (Co <= 0 || Ci <= 0 || taps <= 0) return 0;
    if (Ci % 8 || (taps != 4 && taps != 9)) return -2;
    if (off16(src, dst)) return -5;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return taps == 4 ? wgrad_fold_few<4>(src, dst, Co, Ci, dtype, st) : wgrad_fold_few<9>(src, dst, Co, Ci, dtype, st);
}

// src fp32 [Co, taps, Ci] into dst [Co, Ci, taps]; dtype 2: added to fp32, 1 / 0: written as bf16 / fp16
extern "C" int rb_wgrad_fold(const float* src, void* dst, int Co, int Ci, int taps, int dtype, void* stream) {
    using namespace rb;
    if (Co <= 0 || Ci <= 0 || taps <= 0) return 0;
    const int smem = taps * FOLD_LD * static_cast<int>(sizeof(float));
    if (smem > 48 * 1024 || Co > 65535) return -2;
    const dim3 grid((Ci + FOLD_C - 1) / FOLD_C, Co);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (dtype == 2)
        wgrad_fold_kernel<float, true><<<grid, 256, smem, st>>>(src, static_cast<float*>(dst), Ci, taps);
    else if (dtype == 1)
        wgrad_fold_kernel<__nv_bfloat16, false><<<grid, 256, smem, st>>>(src, static_cast<__nv_bfloat16*>(dst), Ci, taps);
    else
        wgrad_fold_kernel<__half, false><<<grid, 256, smem, st>>>(src, static_cast<__half*>(dst), Ci, taps);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

#define RB_BN_DISPATCH(FN, ...)                                                                       \
    (C >= 256 ? (dtype == 1 ? FN<__nv_bfloat16, 32>(__VA_ARGS__) : FN<__half, 32>(__VA_ARGS__))       \
     : C > 64 ? (dtype == 1 ? FN<__nv_bfloat16, 16>(__VA_ARGS__) : FN<__half, 16>(__VA_ARGS__))       \
              : (dtype == 1 ? FN<__nv_bfloat16, 8>(__VA_ARGS__) : FN<__half, 8>(__VA_ARGS__)))

// Floats that `part` of the two entries below has to hold.
extern "C" long long rb_bn_part_floats(long long R, int C) {
    return C % 8 || C <= 0 || R <= 0 ? 0 : (1 + rb::bn_parts(R, C)) * 2 * C;
}

// Forward statistics + normalisation.  part: fp32 scratch (rb_bn_part_floats); mean / rstd: fp32 [C] outputs;
// run_mean / run_var may be null (evaluation of a frozen layer is not handled here: pass training only).
extern "C" int rb_bn_fwd(const void* x, const void* res, const float* gamma, const float* beta, void* y, float* part,
                         float* mean, float* rstd, float* run_mean, float* run_var, long long R, int C, float eps,
                         float momentum, int relu, int dtype, void* stream) {
    using namespace rb;
    if (C % 8 || R <= 0) return -2;
    if (off16(x, res, y, part)) return -5;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return RB_BN_DISPATCH(bn_fwd_launch, x, res, gamma, beta, y, part, mean, rstd, run_mean, run_var, R, C, eps, momentum,
                          relu, st);
}

// Backward.  part: fp32 scratch (rb_bn_part_floats); on return its first C floats are d beta and the next C d gamma, which are
// also added to dbeta_acc / dgamma_acc when those are given.
extern "C" int rb_bn_bwd(const void* x, const void* dy, const void* y, const float* mean, const float* rstd,
                         const float* gamma, float* part, float* dgamma_acc, float* dbeta_acc, void* dx, void* dres,
                         long long R, int C, int relu, int dtype, void* stream) {
    using namespace rb;
    if (C % 8 || R <= 0) return -2;
    if (off16(x, dy, y, dx, dres) || off16(mean, rstd, part)) return -5;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return RB_BN_DISPATCH(bn_bwd_launch, x, dy, y, mean, rstd, gamma, part, dgamma_acc, dbeta_acc, dx, dres, R, C, relu, st);
}
