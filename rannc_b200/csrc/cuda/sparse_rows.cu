// Rows of zeros in the gradient of a wide output layer.
//
// The loss of masked-LM pre-training looks at 15 % of the positions, and padding counts nowhere: most rows of the gradient
// that reaches the vocabulary projection are zero.  Its two products, two thirds of the layer's work, multiply them all the
// same.  Here the rows that count are found and gathered on the device, and the products run over those (gemm_tcgen05.h:
// rows_ctl); which form runs is decided there too, since the host does not wait.  Nothing is assumed about where dy comes from
// and nothing is kept: every backward looks at the rows it is given.
//
// The results are those of the products over all rows, infinities and NaN included.  A row of dy that is zero adds 0 * x to the
// weight gradient: nothing, where x is finite, and a row whose x is not counts as one that is not zero.  Its own input
// gradient is 0 * W, zero or NaN column by column and the same for every such row: a row of zeros behind the gathered ones
// goes through the product, and its result is theirs.
//
// 8192 rows, 1024 to 30528, 15 % of the rows not zero: 649 -> 272 us for the backward, of which looking 81 (5.2 TB/s),
// gathering 25, the two products 150; what it costs where every row counts, and the rule for when to look, stand in
// host/ops.cpp (gather_room).
#include "sparse_rows.h"

#include "gemm_tcgen05.h"

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "launch.cuh"
#include "tc_common.cuh"

namespace rb {

// A warp looks at a row.  One that is not zero shows in its first 512 bytes nearly always; a row of zeros is read to its end:
// bound by memory, four loads of a thread in flight.
__global__ void __launch_bounds__(256)
    rows_live_kernel(const uint4* dy, long long ldv, const uint4* x, long long x_ldv, int rows, int nv, int x_nv,
                     uint32_t exponent, uint8_t* live) {
    grid_trigger();
    grid_wait();
    const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= rows) return;
    const uint4* d = dy + row * ldv;
    auto bits = [](const uint4& q) { return q.x | q.y | q.z | q.w; };
    bool found = __any_sync(0xffffffffu, lane < nv && bits(d[lane]) != 0);
    for (int i = 32; i < nv && !found; i += 128) {
        uint32_t any = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i + u * 32 + lane < nv) any |= bits(d[i + u * 32 + lane]);
        found = __any_sync(0xffffffffu, any != 0);
    }
    if (!found) {
        // infinity or NaN: all bits of the exponent set, in either half of a word
        const uint32_t low = exponent & 0xffffu, high = exponent & 0xffff0000u;
        auto odd = [&](uint32_t w) { return (w & low) == low || (w & high) == high; };
        bool any = false;
        for (int i = lane; i < x_nv; i += 32) {
            const uint4 q = x[row * x_ldv + i];
            any = any || odd(q.x) || odd(q.y) || odd(q.z) || odd(q.w);
        }
        found = __any_sync(0xffffffffu, any);
    }
    if (lane == 0) live[row] = found;
}

// One block numbers the rows that count: each thread takes a run of rows, counts its flags and, behind the sums of all, goes
// through them once more.
__global__ void __launch_bounds__(1024)
    rows_plan_kernel(const uint8_t* live, int rows, int room, int32_t* idx, int32_t* pos, int32_t* ctl) {
    grid_trigger();
    grid_wait();
    __shared__ int sums[32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int run = (rows + 1023) / 1024, first = min(rows, t * run), last = min(rows, first + run);
    int n = 0;
    for (int r = first; r < last; ++r) n += live[r];
    int before = n;   // inclusive sums over the warp, then over the warps
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before += v;
    }
    if (lane == 31) sums[warp] = before;
    __syncthreads();
    if (warp == 0) {
        int s = sums[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += v;
        }
        sums[lane] = s;
    }
    __syncthreads();
    const int count = sums[31];
    const bool use = count > 0 && count < room;
    if (t == 0) {
        ctl[0] = count;
        ctl[1] = use;
    }
    if (!use) return;
    int k = before - n + (warp ? sums[warp - 1] : 0);
    for (int r = first; r < last; ++r) {
        const bool on = live[r] != 0;
        if (on) idx[k] = r;
        pos[r] = on ? k++ : -1;
    }
}

// Blocks take the gathered rows in turn; four loads of a thread in flight, bound by memory.
__global__ void __launch_bounds__(256)
    rows_gather_kernel(const uint4* dy, long long ldv, const uint4* x, long long x_ldv, int nv, int x_nv, const int32_t* idx,
                       const int32_t* ctl, uint4* dy_out, uint4* x_out, float4* dx32) {
    grid_trigger();
    grid_wait();
    if (!ctl[1]) return;
    const int count = ctl[0], padded = (count + 64) / 64 * 64;
    const uint4 zero = make_uint4(0, 0, 0, 0);
    for (int r = blockIdx.x; r < padded; r += gridDim.x) {
        const bool real = r < count;
        const long long src = real ? idx[r] : 0;
        auto copy = [&](const uint4* from, uint4* to, int n) {
            for (int i = threadIdx.x; i < n; i += 1024) {
                uint4 q[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) q[u] = real && i + u * 256 < n ? from[i + u * 256] : zero;
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (i + u * 256 < n) to[i + u * 256] = q[u];
            }
        };
        copy(dy + src * ldv, dy_out + static_cast<long long>(r) * nv, nv);
        copy(x + src * x_ldv, x_out + static_cast<long long>(r) * x_nv, x_nv);
        if (dx32 && r <= count)
            for (int i = threadIdx.x; i < 2 * x_nv; i += 256)
                dx32[static_cast<long long>(r) * 2 * x_nv + i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

// A block has 256 columns of SCATTER_ROWS rows, a thread 8 columns of every eighth row.  The parts of the row of zeros, which
// most rows get, are added up once for those.
constexpr int SCATTER_ROWS = 32;
template <typename T>
__global__ void __launch_bounds__(256)
    rows_scatter_kernel(const float4* dx32, uint4* dx, int rows, int nv, const int32_t* pos, const int32_t* ctl, bool in_parts) {
    grid_trigger();
    grid_wait();
    if (!ctl[1]) return;
    const int col = blockIdx.y * 32 + (threadIdx.x & 31);
    if (col >= nv) return;
    const int parts = in_parts ? ctl[2] : 1;
    const long long step = in_parts ? static_cast<long long>(ctl[3]) * 2 * nv : 0;
    auto total = [&](int k) {
        const float4* src = dx32 + static_cast<long long>(k) * 2 * nv + 2 * col;
        float4 a = src[0], b = src[1];
#pragma unroll 4
        for (int s = 1; s < parts; ++s) {
            const float4 c = src[s * step], d = src[s * step + 1];
            a.x += c.x, a.y += c.y, a.z += c.z, a.w += c.w;
            b.x += d.x, b.y += d.y, b.z += d.z, b.w += d.w;
        }
        return make_uint4(pack2<T>(a.x, a.y), pack2<T>(a.z, a.w), pack2<T>(b.x, b.y), pack2<T>(b.z, b.w));
    };
    const int first = blockIdx.x * SCATTER_ROWS + (threadIdx.x >> 5);
    int k[SCATTER_ROWS / 8];
#pragma unroll
    for (int u = 0; u < SCATTER_ROWS / 8; ++u) k[u] = first + 8 * u < rows ? pos[first + 8 * u] : -1;
    const uint4 left_out = total(ctl[0]);
#pragma unroll
    for (int u = 0; u < SCATTER_ROWS / 8; ++u) {
        const int row = first + 8 * u;
        if (row < rows) dx[static_cast<long long>(row) * nv + col] = k[u] < 0 ? left_out : total(k[u]);
    }
}

}  // namespace rb

using namespace rb;

extern "C" int rb_rows_plan(const void* dy, long long ld, const void* x, long long x_ld, int rows, int cols, int x_cols, int room,
                            uint8_t* live, int32_t* idx, int32_t* pos, int32_t* ctl, int dtype, void* stream) {
    if (rows <= 0 || cols <= 0 || x_cols <= 0 || room <= 0 || cols % 8 || x_cols % 8 || ld % 8 || x_ld % 8 || room % 64) return -2;
    if (off16(dy, x)) return -5;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const uint32_t e = dtype == 1 ? 0x7f807f80u : 0x7c007c00u;
    if (launch_after(rows_live_kernel, (rows + 7) / 8, 256, 0, st, static_cast<const uint4*>(dy), ld / 8,
                     static_cast<const uint4*>(x), x_ld / 8, rows, cols / 8, x_cols / 8, e, live) != cudaSuccess)
        return -1;
    return launch_after(rows_plan_kernel, 1, 1024, 0, st, static_cast<const uint8_t*>(live), rows, room, idx, pos, ctl) ==
                   cudaSuccess
               ? 0
               : -1;
}

extern "C" int rb_rows_gather(const void* dy, long long ld, const void* x, long long x_ld, int cols, int x_cols,
                              const int32_t* idx, const int32_t* ctl, void* dy_out, void* x_out, float* dx32, void* stream) {
    if (cols % 8 || x_cols % 8 || ld % 8 || x_ld % 8) return -2;
    if (off16(dy, x, dy_out, x_out, dx32)) return -5;
    // (about four blocks of 256 threads to an SM: 64 KiB on their way there)
    return launch_after(rows_gather_kernel, num_sms() * 4, 256, 0, static_cast<cudaStream_t>(stream), static_cast<const uint4*>(dy),
                        ld / 8, static_cast<const uint4*>(x), x_ld / 8, cols / 8, x_cols / 8, idx, ctl,
                        static_cast<uint4*>(dy_out), static_cast<uint4*>(x_out),
                        reinterpret_cast<float4*>(dx32)) == cudaSuccess
               ? 0
               : -1;
}

static int rows_scatter(const float* dx32, void* dx, int rows, int x_cols, const int32_t* pos, const int32_t* ctl, int dtype,
                        bool in_parts, void* stream) {
    if (rows <= 0) return 0;
    if (x_cols % 8) return -2;
    if (off16(dx32, dx)) return -5;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    auto kern = dtype == 1 ? rows_scatter_kernel<__nv_bfloat16> : rows_scatter_kernel<__half>;
    const dim3 grid((rows + SCATTER_ROWS - 1) / SCATTER_ROWS, (x_cols / 8 + 31) / 32);
    return launch_after(kern, grid, 256, 0, st, reinterpret_cast<const float4*>(dx32), static_cast<uint4*>(dx), rows,
                        x_cols / 8, pos, ctl, in_parts) == cudaSuccess
               ? 0
               : -1;
}
extern "C" int rb_rows_scatter(const float* dx32, void* dx, int rows, int x_cols, const int32_t* pos, const int32_t* ctl,
                               int dtype, void* stream) {
    return rows_scatter(dx32, dx, rows, x_cols, pos, ctl, dtype, false, stream);
}
extern "C" int rb_rows_scatter_parts(const float* dx32, void* dx, int rows, int x_cols, const int32_t* pos, const int32_t* ctl,
                                     int dtype, void* stream) {
    return rows_scatter(dx32, dx, rows, x_cols, pos, ctl, dtype, true, stream);
}
