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

#include <type_traits>

#include "launch.cuh"
#include "philox.cuh"
#include "tc_common.cuh"

namespace rb {

constexpr int LN_WARPS = 8;
constexpr int LN_THREADS = LN_WARPS * 32;

// Eight 16-bit values as four pairs of fp32: both kernels are bound by issue slots as much as by memory (a row's bytes pass
// an SM in some 175 cycles, and at 220 instructions a warp and row, dropout apart, that is what four schedulers take), so
// what has a two-wide form uses it, and gamma and beta stay in registers where they suffice.
template <typename T>
__device__ __forceinline__ void unpack_pairs(const uint4& q, uint64_t (&v)[4]) {
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if constexpr (std::is_same_v<T, __nv_bfloat16>) {
            v[j] = f2_pack_bits(w[j] << 16, w[j] & 0xffff0000u);
        } else {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
            v[j] = f2_pack(f.x, f.y);
        }
    }
}
template <typename T>
__device__ __forceinline__ uint4 pack_pairs(const uint64_t (&v)[4]) {
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float a, b;
        f2_unpack(v[j], a, b);
        w[j] = pack2<T>(a, b);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}
template <typename T>
__device__ __forceinline__ void load_pairs(const T* p, uint64_t (&v)[4]) {
    unpack_pairs<T>(*reinterpret_cast<const uint4*>(p), v);
}
__device__ __forceinline__ uint64_t f2_both(float x) { return f2_pack(x, x); }
__device__ __forceinline__ float f2_sum(uint64_t v) {
    float a, b;
    f2_unpack(v, a, b);
    return a + b;
}
// v * scale where the element is kept, else zero
__device__ __forceinline__ void drop_pairs(uint64_t (&v)[4], const bool (&k)[8], uint64_t scale2) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float a, b;
        f2_unpack(f2_mul(v[j], scale2), a, b);
        v[j] = f2_pack(k[2 * j] ? a : 0.f, k[2 * j + 1] ? b : 0.f);
    }
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

// Rows a thread has on their way while it works on one.  A row is one dependent chain load -> reduce -> store, and the bytes
// in flight would be those of the resident warps' current rows.  Each thread fetches its own 16-byte pieces of the next rows
// into its own places of a shared-memory ring (no barrier is needed to read them back), three deep or more.
// Time, and at the copy bandwidth (us, bf16; backward with the sums' reduction): 16384 x 1024 with dropout and residual forward
// 28.7 -> 27.2 (20.5), backward 33.5 -> 31.3 (20.5); without 15.2 -> 12.9 (10.3) and 23.6 -> 19.9 (15.4); 8192 x 2048 24.5
// -> 21.1 and 25.2 -> 24.7; 4096 x 4096 25.4 -> 24.8 and 33.4 -> 30.0; before that, of one row at a time, 32.3 and 34.8 at
// 16384 x 1024 with dropout.
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
    constexpr bool KEEP = NCHUNK <= 2;   // wider threads read gamma and beta again from L1 for every row
    uint64_t kept_g[KEEP ? NCHUNK : 1][4], kept_b[KEEP ? NCHUNK : 1][4];
    if constexpr (KEEP) {
#pragma unroll
        for (int c = 0; c < NCHUNK; ++c) {
            load_pairs(gamma + col0 + c * 256, kept_g[c]);
            load_pairs(beta + col0 + c * 256, kept_b[c]);
        }
    }
    const uint64_t scale2 = f2_both(scale);
    long long row = static_cast<long long>(blockIdx.x) * RPB + slot;
#pragma unroll
    for (int k = 0; k < STAGES - 1; ++k) fetch(k, row + k * step);
    int stage = 0, turn = 0;
    for (; row < rows; row += step) {
        fetch(stage == 0 ? STAGES - 1 : stage - 1, row + (STAGES - 1) * step);
        cp_async_wait<STAGES - 1>();
        const size_t base = static_cast<size_t>(row) * H;
        uint64_t v[NCHUNK][4];
        uint64_t s2 = f2_both(0.f);
#pragma unroll
        for (int c = 0; c < NCHUNK; ++c) {
            const int col = col0 + c * 256;
            unpack_pairs<T>(*place(stage, 0, c), v[c]);
            if (thr) {
                bool k[8];
                keep8(seed, offset, base + col, thr, k);
                drop_pairs(v[c], k, scale2);
            }
            if (residual) {
                uint64_t r[4];
                unpack_pairs<T>(*place(stage, 1, c), r);
#pragma unroll
                for (int j = 0; j < 4; ++j) v[c][j] = f2_add(v[c][j], r[j]);
            }
            if (z_out) {
                const uint4 q = pack_pairs<T>(v[c]);
                *reinterpret_cast<uint4*>(z_out + base + col) = q;
                // the backward reads z in storage precision: normalise the same values
                unpack_pairs<T>(q, v[c]);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) s2 = f2_add(s2, v[c][j]);
        }
        const float mean = group_sum<WPR>(make_float2(f2_sum(s2), 0.f), sm, turn, warp, lane).x * (1.f / H);
        const uint64_t minus_mean = f2_both(-mean);
        uint64_t sq2 = f2_both(0.f);
#pragma unroll
        for (int c = 0; c < NCHUNK; ++c)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                v[c][j] = f2_add(v[c][j], minus_mean);
                sq2 = f2_fma(v[c][j], v[c][j], sq2);
            }
        const float rstd = rsqrtf(group_sum<WPR>(make_float2(f2_sum(sq2), 0.f), sm, turn, warp, lane).x * (1.f / H) + eps);
        if (lane == 0 && part == 0) {
            mean_out[row] = mean;
            rstd_out[row] = rstd;
        }
        const uint64_t rstd2 = f2_both(rstd);
#pragma unroll
        for (int c = 0; c < NCHUNK; ++c) {
            const int col = col0 + c * 256;
            uint64_t g[4], b[4];
            if constexpr (KEEP) {
#pragma unroll
                for (int j = 0; j < 4; ++j) g[j] = kept_g[c][j], b[j] = kept_b[c][j];
            } else {
                load_pairs(gamma + col, g);
                load_pairs(beta + col, b);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) v[c][j] = f2_fma(f2_mul(v[c][j], rstd2), g[j], b[j]);
            *reinterpret_cast<uint4*>(y + base + col) = pack_pairs<T>(v[c]);
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
    // a row's 16-bit values stay in registers across its sum where they suffice, else they are read again from the ring
    // (16384 x 1024 24.0 -> 19.4 us; of 4096 elements a row, held: 49 us for 30)
    constexpr bool HOLD = NCHUNK <= 2 && WPR <= 2;
    uint64_t kept[KEEP_G ? NCHUNK : 1][4], dg[NCHUNK][4], db[NCHUNK][4];
#pragma unroll
    for (int c = 0; c < NCHUNK; ++c) {
        if constexpr (KEEP_G) load_pairs(gamma + col0 + c * 256, kept[c]);
#pragma unroll
        for (int j = 0; j < 4; ++j) dg[c][j] = db[c][j] = f2_both(0.f);
    }
    auto get_gamma = [&](int c, uint64_t (&g)[4]) {
        if constexpr (KEEP_G) {
#pragma unroll
            for (int j = 0; j < 4; ++j) g[j] = kept[c][j];
        } else {
            load_pairs(gamma + col0 + c * 256, g);
        }
    };
    const uint64_t scale2 = f2_both(scale);
    long long row = static_cast<long long>(blockIdx.x) * RPB + slot;
#pragma unroll
    for (int k = 0; k < STAGES - 1; ++k) fetch(k, row + k * step);
    float mean = row < rows ? mean_in[row] : 0.f, rstd = row < rows ? rstd_in[row] : 0.f;
    int stage = 0, turn = 0;
    for (; row < rows; row += step) {
        // the next row's statistics, used one iteration later
        const bool more = row + step < rows;
        const float mean_next = more ? mean_in[row + step] : 0.f, rstd_next = more ? rstd_in[row + step] : 0.f;
        cp_async_wait<STAGES - 2>();
        const size_t base = static_cast<size_t>(row) * H;
        const uint64_t minus_mean = f2_both(-mean), rstd2 = f2_both(rstd);
        uint64_t sx = f2_both(0.f), sy = sx;
        uint4 hd[HOLD ? NCHUNK : 1], hz[HOLD ? NCHUNK : 1];
#pragma unroll
        for (int c = 0; c < NCHUNK; ++c) {
            uint64_t d[4], zz[4], g[4];
            const uint4 qd = *place(stage, 0, c), qz = *place(stage, 1, c);
            if constexpr (HOLD) hd[c] = qd, hz[c] = qz;
            unpack_pairs<T>(qd, d);
            unpack_pairs<T>(qz, zz);
            get_gamma(c, g);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint64_t xh = f2_mul(f2_add(zz[j], minus_mean), rstd2), w = f2_mul(d[j], g[j]);
                sx = f2_add(sx, w);
                sy = f2_fma(w, xh, sy);
                dg[c][j] = f2_fma(d[j], xh, dg[c][j]);
                db[c][j] = f2_add(db[c][j], d[j]);
            }
        }
        // (here, behind the loads of this row and before the wait for the other warps: at the top of the loop 24.0 us, not 22)
        fetch(stage == 0 ? STAGES - 1 : stage - 1, row + (STAGES - 1) * step);
        const float2 s = group_sum<WPR>(make_float2(f2_sum(sx), f2_sum(sy)), sm, turn, warp, lane);
        // o = rstd (d g - s1 - xh s2), with s1 and s2 the means of s.x and s.y.  (Not with rstd^2 taken out of the loop: it is
        // out of fp32's range where rstd itself and every term are not.)
        const uint64_t c1 = f2_both(-s.x * (1.f / H)), c2 = f2_both(-s.y * (1.f / H));
#pragma unroll(NCHUNK <= 2 ? NCHUNK : 1)
        for (int c = 0; c < NCHUNK; ++c) {
            const int col = col0 + c * 256;
            uint64_t d[4], zz[4], g[4], o[4];
            if constexpr (HOLD) {
                unpack_pairs<T>(hd[c], d);
                unpack_pairs<T>(hz[c], zz);
            } else {
                unpack_pairs<T>(*place(stage, 0, c), d);
                unpack_pairs<T>(*place(stage, 1, c), zz);
            }
            get_gamma(c, g);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                o[j] = f2_mul(rstd2, f2_fma(d[j], g[j], f2_fma(f2_mul(f2_add(zz[j], minus_mean), rstd2), c2, c1)));
            *reinterpret_cast<uint4*>(dz_out + base + col) = pack_pairs<T>(o);
            if (dx_out) {
                if (thr) {
                    bool k[8];
                    keep8(seed, offset, base + col, thr, k);
                    drop_pairs(o, k, scale2);
                }
                *reinterpret_cast<uint4*>(dx_out + base + col) = pack_pairs<T>(o);
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
            for (int j = 0; j < 4; ++j)
                f2_unpack(pass == 0 ? dg[c][j] : db[c][j], red[warp][lane * 8 + 2 * j], red[warp][lane * 8 + 2 * j + 1]);
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
