// Fused  y = LayerNorm( dropout(x) + residual )  forward and backward.
//
// One warp owns one row; a lane holds NCHUNK groups of 8 consecutive elements
// (16-byte loads), so a row of H = 256 * NCHUNK elements is read exactly once
// and kept in registers.  The forward also writes z = dropout(x) + residual
// (the LayerNorm input, needed by the backward) and the per-row mean / rstd.
// The backward produces dz (gradient of the residual branch), dx (dz through
// the dropout mask, regenerated from the Philox counter) and per-CTA partial
// sums of dgamma / dbeta in a scratch buffer that a second kernel reduces.
//
// These take the place of aten::layer_norm / aten::dropout / aten::add nodes of
// the traced graph that the reference executes one by one
// (src/torch/TorchDriver.cpp:566; dropout train flag: src/graph/ConvertGraph.cpp:469-484).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cstdlib>
#include <stdint.h>

#include "launch.cuh"
#include "philox.cuh"
#include "tc_common.cuh"

namespace rb {

constexpr int LN_WARPS = 8;
constexpr int LN_THREADS = LN_WARPS * 32;

template <typename T>
__device__ __forceinline__ void ld8(const T* p, float (&v)[8]) {
    uint4 q = *reinterpret_cast<const uint4*>(p);
    const T* e = reinterpret_cast<const T*>(&q);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = to_f32<T>(e[j]);
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8], const __nv_bfloat16*) {
    return make_uint4(pack2<__nv_bfloat16>(v[0], v[1]), pack2<__nv_bfloat16>(v[2], v[3]),
                      pack2<__nv_bfloat16>(v[4], v[5]), pack2<__nv_bfloat16>(v[6], v[7]));
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8], const __half*) {
    return make_uint4(pack2<__half>(v[0], v[1]), pack2<__half>(v[2], v[3]), pack2<__half>(v[4], v[5]),
                      pack2<__half>(v[6], v[7]));
}
template <typename T>
__device__ __forceinline__ void unpack8(const uint4& q, float (&v)[8]) {
    const T* e = reinterpret_cast<const T*>(&q);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = to_f32<T>(e[j]);
}
// 16 bytes from global to this thread's own place in shared memory, asynchronously
__device__ __forceinline__ void cp_async16(uint4* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Sum over the WPR warps that share a row.  Only those warps meet (a named barrier per row slot), and the two
// halves of `sm` take turns, so one barrier per sum is enough: a half is written again only after everybody has
// passed the barrier of the other one.
template <int WPR>
__device__ __forceinline__ float2 group_sum(float2 v, float2 (*sm)[LN_WARPS], int& turn, int warp, int lane) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
    if constexpr (WPR > 1) {
        if (lane == 0) sm[turn][warp] = v;
        asm volatile("bar.sync %0, %1;" ::"r"(1 + warp / WPR), "n"(32 * WPR) : "memory");
        const int base = (warp / WPR) * WPR;
        v = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < WPR; ++i) {
            const float2 w = sm[turn][base + i];
            v.x += w.x;
            v.y += w.y;
        }
        turn ^= 1;
    }
    return v;
}

// Rows a thread has on their way while it works on one.  Both kernels are bound by memory, and what kept them
// from it was latency: a row is one dependent chain load -> reduce -> store, so the bytes in flight were those
// of the resident warps' current rows.  Each thread now fetches its own 16-byte pieces of the next rows into
// its own places of a shared-memory ring (no barrier is needed to read them back), three deep or more.  16384 x 1024
// bf16 with dropout and residual (134 MB each way, 20 us at the copy bandwidth): forward 32.3 -> 28.0 us, backward
// 34.8 -> 29.9 us; 387 x 4096: 4.7 -> 4.0 and 7.2 -> 6.7 us.
template <int NCHUNK>
struct LnRing {
    static constexpr int STAGES = NCHUNK <= 2 ? 4 : 3;
    static constexpr int BYTES = STAGES * 2 * NCHUNK * LN_THREADS * 16;   // two input matrices
    static constexpr int FWD_CTAS = 3 * (BYTES + 1024) <= 227 * 1024 ? 3 : 2;
};

// A row of H = 256 * NCHUNK * WPR elements is shared by WPR warps.
template <typename T, int NCHUNK, int WPR>
__global__ void __launch_bounds__(LN_THREADS, LnRing<NCHUNK>::FWD_CTAS)
    ln_fwd_kernel(const T* x, const T* residual, const T* gamma, const T* beta, T* __restrict__ y, T* __restrict__ z_out,
                  float* __restrict__ mean_out, float* __restrict__ rstd_out, int rows, float eps, uint32_t thr, float scale,
                  uint64_t seed, uint64_t offset) {
    constexpr int H = NCHUNK * 256 * WPR;
    constexpr int RPB = LN_WARPS / WPR;  // rows per CTA per iteration
    constexpr int STAGES = LnRing<NCHUNK>::STAGES;
    grid_trigger();
    grid_wait();
    extern __shared__ uint4 ring[];  // [STAGES][x, residual][NCHUNK][LN_THREADS]
    __shared__ float2 sm[2][LN_WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = warp / WPR, part = warp % WPR;
    const long long step = static_cast<long long>(gridDim.x) * RPB;
    const int col0 = (part * NCHUNK * 32 + lane) * 8;
    auto place = [&](int stage, int which, int c) { return ring + ((stage * 2 + which) * NCHUNK + c) * LN_THREADS + threadIdx.x; };
    auto fetch = [&](int stage, long long row) {
        if (row < rows) {
#pragma unroll
            for (int c = 0; c < NCHUNK; ++c) {
                cp_async16(place(stage, 0, c), x + row * H + col0 + c * 256);
                if (residual) cp_async16(place(stage, 1, c), residual + row * H + col0 + c * 256);
            }
        }
        cp_async_commit();
    };
    long long row = static_cast<long long>(blockIdx.x) * RPB + slot;
#pragma unroll
    for (int k = 0; k < STAGES - 1; ++k) fetch(k, row + k * step);
    int stage = 0, turn = 0;
    for (; row < rows; row += step) {
        fetch(stage == 0 ? STAGES - 1 : stage - 1, row + (STAGES - 1) * step);
        cp_async_wait<STAGES - 1>();
        const size_t base = static_cast<size_t>(row) * H;
        float v[NCHUNK][8];
        float s = 0.f;
#pragma unroll
        for (int c = 0; c < NCHUNK; ++c) {
            const int col = col0 + c * 256;
            unpack8<T>(*place(stage, 0, c), v[c]);
            if (thr) {
                bool k[8];
                keep8(seed, offset, base + col, thr, k);
#pragma unroll
                for (int j = 0; j < 8; ++j) v[c][j] = k[j] ? v[c][j] * scale : 0.f;
            }
            if (residual) {
                float r[8];
                unpack8<T>(*place(stage, 1, c), r);
#pragma unroll
                for (int j = 0; j < 8; ++j) v[c][j] += r[j];
            }
            if (z_out) {
                const uint4 q = pack8(v[c], static_cast<const T*>(nullptr));
                *reinterpret_cast<uint4*>(z_out + base + col) = q;
                // the backward reads z in storage precision: normalise the same values
                unpack8<T>(q, v[c]);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) s += v[c][j];
        }
        const float mean = group_sum<WPR>(make_float2(s, 0.f), sm, turn, warp, lane).x * (1.f / H);
        float sq = 0.f;
#pragma unroll
        for (int c = 0; c < NCHUNK; ++c)
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float d = v[c][j] - mean;
                sq += d * d;
            }
        const float rstd = rsqrtf(group_sum<WPR>(make_float2(sq, 0.f), sm, turn, warp, lane).x * (1.f / H) + eps);
        if (lane == 0 && part == 0) {
            mean_out[row] = mean;
            rstd_out[row] = rstd;
        }
        // gamma / beta are re-read per row (they stay in L1) instead of costing 16 * NCHUNK registers
#pragma unroll
        for (int c = 0; c < NCHUNK; ++c) {
            const int col = col0 + c * 256;
            float o[8], g[8], b[8];
            ld8(gamma + col, g);
            ld8(beta + col, b);
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] = (v[c][j] - mean) * rstd * g[j] + b[j];
            *reinterpret_cast<uint4*>(y + base + col) = pack8(o, static_cast<const T*>(nullptr));
        }
        if (++stage == STAGES) stage = 0;
    }
}

// scratch layout: partial[blockIdx][0][H] = dgamma, partial[blockIdx][1][H] = dbeta
template <typename T, int NCHUNK, int WPR>
__global__ void __launch_bounds__(LN_THREADS, 2)
    ln_bwd_kernel(const T* dy, const T* z, const T* gamma, const float* mean_in, const float* rstd_in,
                  T* __restrict__ dz_out, T* __restrict__ dx_out, float* __restrict__ partial,
                  int rows, uint32_t thr, float scale, uint64_t seed, uint64_t offset) {
    constexpr int H = NCHUNK * 256 * WPR;
    constexpr int RPB = LN_WARPS / WPR;
    constexpr int STAGES = LnRing<NCHUNK>::STAGES;
    grid_trigger();
    grid_wait();
    extern __shared__ uint4 ring[];  // [STAGES][dy, z][NCHUNK][LN_THREADS]
    __shared__ float red[LN_WARPS][256 + 8];
    __shared__ float2 sm[2][LN_WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = warp / WPR, part = warp % WPR;
    const long long step = static_cast<long long>(gridDim.x) * RPB;
    const int col0 = (part * NCHUNK * 32 + lane) * 8;
    auto place = [&](int stage, int which, int c) { return ring + ((stage * 2 + which) * NCHUNK + c) * LN_THREADS + threadIdx.x; };
    auto fetch = [&](int stage, long long row) {
        if (row < rows) {
#pragma unroll
            for (int c = 0; c < NCHUNK; ++c) {
                cp_async16(place(stage, 0, c), dy + row * H + col0 + c * 256);
                cp_async16(place(stage, 1, c), z + row * H + col0 + c * 256);
            }
        }
        cp_async_commit();
    };
    // gamma stays in registers where they suffice; wider threads read it again from L1 (spills otherwise)
    constexpr bool KEEP_G = NCHUNK <= 2;
    float kept[KEEP_G ? NCHUNK : 1][8], dg[NCHUNK][8], db[NCHUNK][8];
#pragma unroll
    for (int c = 0; c < NCHUNK; ++c) {
        if constexpr (KEEP_G) ld8(gamma + col0 + c * 256, kept[c]);
#pragma unroll
        for (int j = 0; j < 8; ++j) dg[c][j] = db[c][j] = 0.f;
    }
    auto get_gamma = [&](int c, float (&g)[8]) {
        if constexpr (KEEP_G) {
#pragma unroll
            for (int j = 0; j < 8; ++j) g[j] = kept[c][j];
        } else {
            ld8(gamma + col0 + c * 256, g);
        }
    };
    long long row = static_cast<long long>(blockIdx.x) * RPB + slot;
#pragma unroll
    for (int k = 0; k < STAGES - 1; ++k) fetch(k, row + k * step);
    float mean = row < rows ? mean_in[row] : 0.f, rstd = row < rows ? rstd_in[row] : 0.f;
    int stage = 0, turn = 0;
    for (; row < rows; row += step) {
        fetch(stage == 0 ? STAGES - 1 : stage - 1, row + (STAGES - 1) * step);
        // the next row's statistics, used one iteration later
        const bool more = row + step < rows;
        const float mean_next = more ? mean_in[row + step] : 0.f, rstd_next = more ? rstd_in[row + step] : 0.f;
        cp_async_wait<STAGES - 1>();
        const size_t base = static_cast<size_t>(row) * H;
        float2 s = make_float2(0.f, 0.f);
#pragma unroll
        for (int c = 0; c < NCHUNK; ++c) {
            float d[8], zz[8], g[8];
            unpack8<T>(*place(stage, 0, c), d);
            unpack8<T>(*place(stage, 1, c), zz);
            get_gamma(c, g);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float xh = (zz[j] - mean) * rstd, w = d[j] * g[j];
                s.x += w;
                s.y += w * xh;
                dg[c][j] += d[j] * xh;
                db[c][j] += d[j];
            }
        }
        s = group_sum<WPR>(s, sm, turn, warp, lane);
        const float s1 = s.x * (1.f / H), s2 = s.y * (1.f / H);
#pragma unroll(NCHUNK <= 2 ? NCHUNK : 1)
        for (int c = 0; c < NCHUNK; ++c) {
            const int col = col0 + c * 256;
            // read again from the ring: cheaper than 16 * NCHUNK registers held across the sum
            float d[8], zz[8], g[8], o[8];
            unpack8<T>(*place(stage, 0, c), d);
            unpack8<T>(*place(stage, 1, c), zz);
            get_gamma(c, g);
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] = rstd * (d[j] * g[j] - s1 - (zz[j] - mean) * rstd * s2);
            *reinterpret_cast<uint4*>(dz_out + base + col) = pack8(o, static_cast<const T*>(nullptr));
            if (dx_out) {
                if (thr) {
                    bool k[8];
                    keep8(seed, offset, base + col, thr, k);
#pragma unroll
                    for (int j = 0; j < 8; ++j) o[j] = k[j] ? o[j] * scale : 0.f;
                }
                *reinterpret_cast<uint4*>(dx_out + base + col) = pack8(o, static_cast<const T*>(nullptr));
            }
        }
        mean = mean_next;
        rstd = rstd_next;
        if (++stage == STAGES) stage = 0;
    }
    // reduce the per-warp partials across the CTA, one 256-column slab at a time
    float* out_g = partial + static_cast<size_t>(blockIdx.x) * 2 * H;
    float* out_b = out_g + H;
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
        for (int c = 0; c < NCHUNK; ++c) {
            __syncthreads();
#pragma unroll
            for (int j = 0; j < 8; ++j) red[warp][lane * 8 + j] = pass == 0 ? dg[c][j] : db[c][j];
            __syncthreads();
            const int t = threadIdx.x;  // 256 threads, 256 columns
#pragma unroll
            for (int pt = 0; pt < WPR; ++pt) {
                float s = 0.f;
#pragma unroll
                for (int sl = 0; sl < RPB; ++sl) s += red[sl * WPR + pt][t];
                (pass == 0 ? out_g : out_b)[(pt * NCHUNK + c) * 256 + t] = s;
            }
        }
    }
}

// dgamma[h] (+)= sum_blocks partial[b][0][h]; dbeta likewise.  grid = 2H/32 blocks of (32, 32): bound by the
// latency of its loads, so a thread has ten of them at most, four in flight (296 x 2048 floats: 5.2 -> 3.7 us).
template <typename OutT>
__global__ void __launch_bounds__(1024)
    ln_bwd_reduce_kernel(const float* partial, OutT* dgamma, OutT* dbeta, int nblocks, int H, int accumulate) {
    grid_trigger();
    grid_wait();
    __shared__ float red[32][33];
    const int col2 = blockIdx.x * 32 + threadIdx.x;  // in [0, 2H)
    float s = 0.f;
#pragma unroll 4
    for (int b = threadIdx.y; b < nblocks; b += 32) s += partial[static_cast<size_t>(b) * 2 * H + col2];
    red[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y == 0) {
#pragma unroll
        for (int w = 1; w < 32; ++w) s += red[w][threadIdx.x];
        OutT* dst = col2 < H ? dgamma + col2 : dbeta + (col2 - H);
        *dst = from_f32<OutT>(accumulate ? to_f32<OutT>(*dst) + s : s);
    }
}

// Shared memory above 48 KiB has to be asked for once per kernel and device.
template <typename K>
static bool ln_allow_smem(K kern, int bytes, bool (&done)[64]) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    if (done[dev & 63]) return true;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return false;
    done[dev & 63] = true;
    return true;
}

template <typename T, int NCHUNK, int WPR>
static int launch_fwd(const void* x, const void* res, const void* g, const void* b, void* y,
                      void* z, float* mean, float* rstd, int rows, float eps, float p,
                      uint64_t seed, uint64_t offset, cudaStream_t st) {
    const uint32_t thr = p > 0.f ? drop_threshold(p) : 0u;
    const float scale = p > 0.f ? 1.f / (1.f - p) : 1.f;
    constexpr int RPB = LN_WARPS / WPR;
    // one wave of resident CTAs: each works through its rows with the next ones on their way
    int grid = (rows + RPB - 1) / RPB;
    const int cap = 148 * LnRing<NCHUNK>::FWD_CTAS;
    if (grid > cap) grid = cap;
    static bool allowed[64] = {false};
    if (!ln_allow_smem(ln_fwd_kernel<T, NCHUNK, WPR>, LnRing<NCHUNK>::BYTES, allowed)) return -1;
    const cudaError_t e = launch_after(ln_fwd_kernel<T, NCHUNK, WPR>, grid, LN_THREADS, LnRing<NCHUNK>::BYTES, st,
                                       static_cast<const T*>(x), static_cast<const T*>(res), static_cast<const T*>(g),
                                       static_cast<const T*>(b), static_cast<T*>(y), static_cast<T*>(z), mean, rstd, rows,
                                       eps, thr, scale, seed, offset);
    return e == cudaSuccess ? 0 : -1;
}

template <typename T, int NCHUNK, int WPR>
static int launch_bwd(const void* dy, const void* z, const void* g, const float* mean,
                      const float* rstd, void* dz, void* dx, float* partial, int grid, int rows,
                      float p, uint64_t seed, uint64_t offset, cudaStream_t st) {
    const uint32_t thr = p > 0.f ? drop_threshold(p) : 0u;
    const float scale = p > 0.f ? 1.f / (1.f - p) : 1.f;
    static bool allowed[64] = {false};
    if (!ln_allow_smem(ln_bwd_kernel<T, NCHUNK, WPR>, LnRing<NCHUNK>::BYTES, allowed)) return -1;
    const cudaError_t e = launch_after(ln_bwd_kernel<T, NCHUNK, WPR>, grid, LN_THREADS, LnRing<NCHUNK>::BYTES, st,
                                       static_cast<const T*>(dy), static_cast<const T*>(z), static_cast<const T*>(g), mean,
                                       rstd, static_cast<T*>(dz), static_cast<T*>(dx), partial, rows,
                                       thr, scale, seed, offset);
    return e == cudaSuccess ? 0 : -1;
}

}  // namespace rb

#define RB_LN_DISPATCH(T, FN, ...)                      \
    switch (H / 256) {                                  \
        case 1: return rb::FN<T, 1, 1>(__VA_ARGS__);    \
        case 2: return rb::FN<T, 2, 1>(__VA_ARGS__);    \
        case 3: return rb::FN<T, 3, 1>(__VA_ARGS__);    \
        case 4: return rb::FN<T, 2, 2>(__VA_ARGS__);    \
        case 6: return rb::FN<T, 3, 2>(__VA_ARGS__);    \
        case 8: return rb::FN<T, 2, 4>(__VA_ARGS__);    \
        case 12: return rb::FN<T, 3, 4>(__VA_ARGS__);   \
        case 16: return rb::FN<T, 4, 4>(__VA_ARGS__);   \
        default: return -2;                             \
    }

// 1 when H is a width the register-resident kernels cover
extern "C" int rb_ln_supported(int H) {
    if (H % 256) return 0;
    switch (H / 256) {
        case 1: case 2: case 3: case 4: case 6: case 8: case 12: case 16: return 1;
        default: return 0;
    }
}

// number of CTAs (= rows of the scratch buffer) the backward uses for `rows`
extern "C" int rb_ln_bwd_grid(int rows) {
    int grid = (rows + 1) / 2;
    const int cap = 148 * 2;
    return grid > cap ? cap : (grid < 1 ? 1 : grid);
}

// dtype: 0 fp16, 1 bf16.  residual / z may be null (z == x then).
extern "C" int rb_ln_fwd(const void* x, const void* residual, const void* gamma, const void* beta,
                         void* y, void* z, float* mean, float* rstd, int rows, int H, float eps,
                         float p, uint64_t seed, uint64_t offset, int dtype, void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (rows <= 0) return 0;
    if (rb::off16(x, residual, gamma, beta, y, z)) return -5;
    if (dtype == 1) {
        RB_LN_DISPATCH(__nv_bfloat16, launch_fwd, x, residual, gamma, beta, y, z, mean, rstd, rows,
                       eps, p, seed, offset, st)
    } else {
        RB_LN_DISPATCH(__half, launch_fwd, x, residual, gamma, beta, y, z, mean, rstd, rows, eps, p,
                       seed, offset, st)
    }
}

namespace rb {
static int ln_bwd_rows(const void* dy, const void* z, const void* gamma, const float* mean, const float* rstd, void* dz,
                       void* dx, float* partial, int grid, int rows, int H, float p, uint64_t seed, uint64_t offset,
                       int dtype, cudaStream_t st) {
    if (dtype == 1) {
        RB_LN_DISPATCH(__nv_bfloat16, launch_bwd, dy, z, gamma, mean, rstd, dz, dx, partial, grid, rows, p, seed, offset, st)
    } else {
        RB_LN_DISPATCH(__half, launch_bwd, dy, z, gamma, mean, rstd, dz, dx, partial, grid, rows, p, seed, offset, st)
    }
}
template <typename OutT>
static int ln_bwd_sums(const float* partial, void* dgamma, void* dbeta, int grid, int H, int accumulate, cudaStream_t st) {
    return launch_after(ln_bwd_reduce_kernel<OutT>, 2 * H / 32, dim3(32, 32), 0, st, partial, static_cast<OutT*>(dgamma),
                        static_cast<OutT*>(dbeta), grid, H, accumulate) == cudaSuccess
               ? 0
               : -1;
}
// An empty batch contributes nothing: the parameters' gradients are zero, or stay what they were.
static int ln_bwd_empty(void* dgamma, void* dbeta, size_t bytes, int accumulate, cudaStream_t st) {
    if (accumulate) return 0;
    return cudaMemsetAsync(dgamma, 0, bytes, st) == cudaSuccess && cudaMemsetAsync(dbeta, 0, bytes, st) == cudaSuccess ? 0 : -1;
}
}  // namespace rb

// `partial` is scratch of rb_ln_bwd_grid(rows) * 2 * H floats.  dgamma / dbeta are
// fp32 [H]; accumulate != 0 adds to them.  dx (may be null): dz through the dropout mask, or dz once more without dropout.
extern "C" int rb_ln_bwd(const void* dy, const void* z, const void* gamma, const float* mean,
                         const float* rstd, void* dz, void* dx, float* dgamma, float* dbeta,
                         float* partial, int rows, int H, float p, uint64_t seed, uint64_t offset,
                         int accumulate, int dtype, void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (rows <= 0) return rb::ln_bwd_empty(dgamma, dbeta, H * sizeof(float), accumulate, st);
    if (rb::off16(dy, z, gamma, dz, dx)) return -5;
    const int grid = rb_ln_bwd_grid(rows);
    const int rc = rb::ln_bwd_rows(dy, z, gamma, mean, rstd, dz, dx, partial, grid, rows, H, p, seed, offset, dtype, st);
    return rc ? rc : rb::ln_bwd_sums<float>(partial, dgamma, dbeta, grid, H, accumulate, st);
}

// the same with dgamma / dbeta written in the 16-bit type of the operands (rounded from the fp32 sums)
extern "C" int rb_ln_bwd16(const void* dy, const void* z, const void* gamma, const float* mean, const float* rstd,
                           void* dz, void* dx, void* dgamma, void* dbeta, float* partial, int rows, int H, float p,
                           uint64_t seed, uint64_t offset, int dtype, void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (rows <= 0) return rb::ln_bwd_empty(dgamma, dbeta, H * 2, 0, st);
    if (rb::off16(dy, z, gamma, dz, dx)) return -5;
    const int grid = rb_ln_bwd_grid(rows);
    const int rc = rb::ln_bwd_rows(dy, z, gamma, mean, rstd, dz, dx, partial, grid, rows, H, p, seed, offset, dtype, st);
    if (rc) return rc;
    return dtype == 1 ? rb::ln_bwd_sums<__nv_bfloat16>(partial, dgamma, dbeta, grid, H, 0, st)
                      : rb::ln_bwd_sums<__half>(partial, dgamma, dbeta, grid, H, 0, st);
}

// ---------------------------------------------------------------------------
// Allocation-free variant of rb_ln_bwd (declared and documented in norm_noalloc.h)
// ---------------------------------------------------------------------------
#include <atomic>

#include "norm_noalloc.h"

// Scratch for the per-CTA partial sums of dgamma / dbeta.  In host code this name is only a
// stand-in for the symbol: kernels must be given the address cudaGetSymbolAddress returns.
static __device__ __align__(256) float g_ln_noalloc_scratch[RB_LN_NOALLOC_MAX_FLOATS];

// One cached address per device.  The slots are atomics: two host threads that make their first call on a
// device at the same time both resolve the symbol and store the same value, which is harmless.
static float* ln_noalloc_scratch_ptr() {
    static std::atomic<float*> ptrs[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    float* p = ptrs[dev].load(std::memory_order_acquire);
    if (!p) {
        if (cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_ln_noalloc_scratch) != cudaSuccess) return nullptr;
        ptrs[dev].store(p, std::memory_order_release);
    }
    return p;
}

extern "C" const char* rb_ln_bwd_noalloc_strerror(int code) {
    switch (code) {
        case RB_LN_NOALLOC_OK: return "ok";
        case RB_LN_NOALLOC_LAUNCH_FAILED: return "kernel launch failed";
        case RB_LN_NOALLOC_BAD_WIDTH: return "unsupported row width H (supported: 256, 512, 768, 1024, 1536, 2048, 3072, 4096)";
        case RB_LN_NOALLOC_NO_SYMBOL: return "could not resolve the device address of the built-in scratch array";
        case RB_LN_NOALLOC_TOO_LARGE: return "rows x H needs more scratch than the built-in array holds (RB_LN_NOALLOC_MAX_FLOATS)";
        default: return "unknown error";
    }
}

extern "C" int rb_ln_bwd_noalloc(const void* dy, const void* z, const void* gamma, const float* mean,
                                 const float* rstd, void* dz, void* dx, float* dgamma, float* dbeta, int rows,
                                 int H, float p, uint64_t seed, uint64_t offset, int accumulate, int dtype,
                                 void* stream) {
    if (rows <= 0) {   // writes zero gradients unless it accumulates; needs no scratch
        const int rc = rb_ln_bwd(dy, z, gamma, mean, rstd, dz, dx, dgamma, dbeta, nullptr, rows, H, p, seed, offset,
                                 accumulate, dtype, stream);
        return rc == 0 ? RB_LN_NOALLOC_OK : RB_LN_NOALLOC_LAUNCH_FAILED;
    }
    if (!rb_ln_supported(H)) return RB_LN_NOALLOC_BAD_WIDTH;
    const long long need = static_cast<long long>(rb_ln_bwd_grid(rows)) * 2 * H;
    if (need > RB_LN_NOALLOC_MAX_FLOATS) return RB_LN_NOALLOC_TOO_LARGE;
    float* scratch = ln_noalloc_scratch_ptr();
    if (!scratch) return RB_LN_NOALLOC_NO_SYMBOL;
    const int rc = rb_ln_bwd(dy, z, gamma, mean, rstd, dz, p > 0.f ? dx : nullptr, dgamma, dbeta, scratch, rows, H, p, seed, offset,
                             accumulate, dtype, stream);
    return rc == 0 ? RB_LN_NOALLOC_OK : (rc == -2 ? RB_LN_NOALLOC_BAD_WIDTH : RB_LN_NOALLOC_LAUNCH_FAILED);
}
