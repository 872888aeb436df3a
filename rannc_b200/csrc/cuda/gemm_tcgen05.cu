// Dense GEMM on the 5th-generation tensor cores (tcgen05 + TMEM + TMA), sm_100a.
//
//   D[b] = epilogue( alpha * op(A[b]) * op(B[b]) )      op(A): M x K, op(B): K x N
//
// A is "K-major" when stored [M, K] row-major and "MN-major" when stored
// [K, M] row-major; B is K-major when stored [N, K] (the nn.Linear weight
// layout) and MN-major when stored [K, N].  The three GEMMs of a linear layer
// map onto it without a transposed copy:
//   forward  Y  = X  W^T : A = X  (K-major),  B = W  (K-major)
//   dgrad    dX = dY W   : A = dY (K-major),  B = W  (MN-major)
//   wgrad    dW = dY^T X : A = dY (MN-major), B = X  (MN-major)
//
// Structure: persistent CTAs (one per SM), 128 x 256 output tile (128 or 64 columns for small problems), K step 64,
// 4-stage TMA->smem ring (6 or 8 with narrower tiles), fp32 accumulators double-buffered in TMEM (2 x 256
// columns) so the epilogue of tile i overlaps the main loop of tile i+1.
// Warp 0 = TMA producer, warp 1 = MMA issuer, the next eight (sixteen with an activation) = epilogue, the last two =
// column sums of A where asked for (with K = 1024 a tile's main loop is only 16 k steps, and four warps could not
// drain a 128 x 256 accumulator in that time); the epilogue writes through shared memory and the copy engine.
//
// PAIR variant (cta_group::2): two CTAs of a cluster -- the two SMs of a TPC -- share a 256 x 256 tile.
// Each CTA loads its own 128 rows of A and HALF of the B tile (so a k step moves 32 KiB per SM instead
// of 48 KiB, and shared memory, which the products read too, takes that much less in),
// one lane of the first CTA issues the MMAs for both, and each CTA keeps and drains the accumulator of
// its own 128 rows.  Completion of both CTAs' loads is counted on the first CTA's barrier; stage-free
// and accumulator-full signals go to both CTAs with one multicast commit.  No load is multicast.
//
// This kernel takes the place of the cuBLAS calls the reference reaches through
// aten::linear / aten::matmul in its TorchScript interpreter
// (src/torch/TorchDriver.cpp:566) and in src/distop/DistMatmul.cpp:97-214.
#include "gemm_tcgen05.h"

#include <algorithm>
#include <cstdlib>
#include <mutex>

#include "launch.cuh"
#include "tc_common.cuh"

namespace rb {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int A_STAGE_BYTES = BM * BK * 2;  // 16 KiB
constexpr int SUM_WARPS = 2;                         // column sums of A: one per 64-column chunk of its tile
constexpr int GROUP_M = 8;
constexpr int EPI_BYTES = 32 * 1024;                 // staging memory of the epilogue warps

// TN: columns of the output tile.  A wide tile moves the fewest bytes per multiplication; a problem with too few
// 256-wide tiles to give every SM one takes 128 or 64 columns instead (single-CTA kernel only).
// EW: epilogue warps, 8 or 16: two or four per TMEM lane quarter, each with 128 or 64 of the tile's 256 columns (and 32 at
// least: with a 64-column tile half of sixteen have nothing to do).  Sixteen where an activation is part of the epilogue
// (see there).  Each owns 4 or 2 KiB of shared memory in which it lays out 32 x 32 blocks of the tile (16-bit: 64-byte rows,
// two blocks or one; fp32: 128-byte rows, eight warps only; both swizzled as the tensor map of D says) that the copy engine
// then writes, or adds, to global memory.
template <bool PAIR, int TN, int EW>
struct Cfg {
    static_assert(TN == 256 || (!PAIR && (TN == 128 || TN == 64)), "unsupported tile");
    static constexpr int B_ROWS = PAIR ? TN / 2 : TN;       // extent of the B tile one CTA loads
    static constexpr int B_STAGE_BYTES = B_ROWS * BK * 2;   // 8 / 16 / 32 KiB
    static constexpr int STAGE_BYTES = A_STAGE_BYTES + B_STAGE_BYTES;
    static constexpr int STAGES = 192 * 1024 / STAGE_BYTES;  // 6 (pair) / 4 / 6 / 8
    static constexpr int SMEM_BYTES =
        STAGES * STAGE_BYTES + EPI_BYTES + 1024 /*align slack*/ + 384 /*barriers*/;
    static constexpr int TILE_M = PAIR ? 2 * BM : BM;       // rows of the output tile of a CTA (pair)
    static constexpr int TMEM_COLS = 2 * TN;                // two accumulators
    static constexpr int EPI_THREADS = 32 * EW;
    static constexpr int THREADS = 64 + EPI_THREADS + 32 * SUM_WARPS;
    static constexpr int PARTS = TN / 32 < EW / 4 ? TN / 32 : EW / 4;   // column groups of the tile
    static constexpr int PART_COLS = TN / PARTS;
    static constexpr int DRAIN_WARPS = 4 * PARTS;
};

struct GemmKernelParams {
    int M, N, K, batch;
    int a_major, b_major;
    int num_m_blocks, num_n_blocks, num_tiles, num_kb;
    int base_tiles, split_k, kb_per_split;  // split-K: num_tiles = base_tiles * split_k
    // the last, partly filled wave of tiles [tail_first, base_tiles) in an arrangement of its own (see Tail): 0 tiles: none
    int tail_first, tail_tiles, tail_split, tail_kb, tail_units;
    int partial;                            // a work item may hold part of a tile's K: results are added
    int rs_nranks, rs_cols;                 // reduce-scatter epilogue: column block j -> rs_peer[j]
    void* rs_peer[8];
    // all-gather prologue: B is assembled in local memory from column shards held by the ranks of a group
    int ag_nranks, ag_my_idx, ag_rows, ag_cols;  // shard r = [ag_rows, ag_cols] at ag_src[r]
    const void* ag_src[8];
    void* ag_dst;                                // [ag_rows, ag_nranks * ag_cols] (the B operand)
    unsigned int* ag_flags;                      // [8] counters, zero at launch: CTAs done copying shard r
    void* D;
    const void* bias;
    const void* residual;
    const void* aux_in;
    void* aux_out;
    long long ldd, strideD;
    float alpha;
    int flags;
    int* err;
    // implicit-GEMM convolution: see RbGemmArgs
    int conv_kb_per_tap, conv_b_tap_cols;
    int wgrad_taps, wgrad_cols;
    int map_hp, map_wp, map_h, map_w, map_pad;
    int conv_shift[49];
    // 1: the epilogue goes through shared memory and the copy engine (tensor maps of D and of the auxiliary
    // matrix); 0: every thread stores its own row (mapped rows, peers' memory, unaligned outputs)
    int staged;
    // MN-major operands: 1: all 64-column chunks of a stage in one copy (tensor map [chunk][row][64]); 0: one copy each
    int a_merged, b_merged;
    // 1: the bias / the matrices beside the output / the output start their rows on 16-byte boundaries
    int bias_al, in_al, out_al;
    float* a_colsum;   // not null: column sums of the stored A (MN-major) are added here
    int* rows_ctl;   // see RbGemmArgs
    int rows_mode, rows_out;
};

// A product whose rows were gathered on the device (RbGemmArgs::rows_ctl): how many there are, and whether this form of the
// product is the one in use, is read here.  (The host cannot choose: it does not wait for the device.)
constexpr int ROWS_DRAIN_STEPS = 6;   // what a part costs besides its own steps (as DRAIN_STEPS below)
__device__ __forceinline__ void apply_rows(GemmKernelParams& p, int units, bool first) {
    const int count = p.rows_ctl[0], gathered = p.rows_ctl[1];
    if ((p.rows_mode != RB_GEMM_ROWS_ALL) != (gathered != 0)) {
        p.num_tiles = 0;   // the other form runs
        return;
    }
    if (p.rows_mode == RB_GEMM_ROWS_K) {
        // rows up to the next whole step are zero; whole tiles, as for any short K
        p.num_kb = (count + BK - 1) / BK;
        p.kb_per_split = p.num_kb;
        p.tail_tiles = 0;
        p.num_tiles = p.base_tiles;
    } else if (p.rows_mode == RB_GEMM_ROWS_M) {
        // one more row, of zeros: its product stands for every row that was left out
        p.num_m_blocks = (count + 1 + 2 * BM - 1) / (2 * BM);
        p.base_tiles = p.num_m_blocks * p.num_n_blocks;
        // few tiles and a long K (the layer's outputs): parts whose waves take the fewest steps, each with its drain, and
        // three eighths of a step for every tile of a part that is written and read once more (512 KiB from L2)
        const int part_rows = p.num_m_blocks * 2 * BM;
        int split = 1, best = 0x7fffffff;
        for (int s = 1; s <= 16 && s * 4 <= p.num_kb && s * part_rows <= p.rows_out; ++s) {
            const int cost = (p.base_tiles * s + units - 1) / units * ((p.num_kb + s - 1) / s + ROWS_DRAIN_STEPS) +
                             p.base_tiles * s * 3 / 8;
            if (cost < best) best = cost, split = s;
        }
        p.kb_per_split = (p.num_kb + split - 1) / split;
        p.split_k = (p.num_kb + p.kb_per_split - 1) / p.kb_per_split;
        p.num_tiles = p.base_tiles * p.split_k;
        if (first) p.rows_ctl[2] = p.split_k, p.rows_ctl[3] = part_rows;
    }
}

__device__ __forceinline__ void tile_coords(const GemmKernelParams& p, int tile, int& mb, int& nb,
                                            int& b, int& kb_begin, int& kb_end) {
    if (p.tail_tiles > 0 && tile >= p.tail_first) {
        const int r = tile - p.tail_first;
        int t = r % p.tail_tiles;
        if (p.tail_split > 1) {   // equal parts of K, one wave of them
            kb_begin = r / p.tail_tiles * p.tail_kb;
            kb_end = min(p.num_kb, kb_begin + p.tail_kb);
        } else if (r < p.tail_tiles) {   // owners: the first tail_kb steps of a tile each
            kb_begin = 0;
            kb_end = p.tail_kb;
        } else {   // helpers: the rest of one tile after another
            const int round = r / p.tail_units, x = r - round * p.tail_units - p.tail_tiles;
            t = round * (p.tail_units - p.tail_tiles) + x;
            kb_begin = p.tail_kb;
            kb_end = p.num_kb;
            if (x < 0 || t >= p.tail_tiles) t = kb_end = 0;   // (an owner's place in a later round: nothing to do)
        }
        tile = p.tail_first + t;
    } else {
        kb_begin = 0;
        if (p.split_k > 1) {
            const int ks = static_cast<unsigned>(tile) / static_cast<unsigned>(p.base_tiles);
            tile -= ks * p.base_tiles;
            kb_begin = ks * p.kb_per_split;
        }
        kb_end = min(p.num_kb, kb_begin + p.kb_per_split);
    }
    // (every role of every CTA does this for every tile, the epilogue between two tiles: a division is some 40 cycles)
    unsigned t = tile;
    b = 0;
    if (p.batch > 1) {
        const unsigned per_batch = p.num_m_blocks * p.num_n_blocks;
        b = t / per_batch;
        t -= b * per_batch;
    }
    const unsigned group_sz = GROUP_M * p.num_n_blocks;
    const unsigned g = t / group_sz;
    const int first_m = g * GROUP_M;
    const unsigned gm = min(GROUP_M, p.num_m_blocks - first_m);
    t -= g * group_sz;
    nb = gm == GROUP_M ? t / GROUP_M : t / gm;
    mb = first_m + (t - nb * gm);
}

template <int N, typename T>
__device__ __forceinline__ void load_n(const T* ptr, bool vec_ok, int valid, float (&v)[N]) {
    if (vec_ok) {
        if constexpr (sizeof(T) == 2) {
            const uint4* p4 = reinterpret_cast<const uint4*>(ptr);
#pragma unroll
            for (int i = 0; i < N / 8; ++i) {
                uint4 q = p4[i];
                const T* e = reinterpret_cast<const T*>(&q);
#pragma unroll
                for (int j = 0; j < 8; ++j) v[i * 8 + j] = to_f32<T>(e[j]);
            }
        } else {
            const float4* p4 = reinterpret_cast<const float4*>(ptr);
#pragma unroll
            for (int i = 0; i < N / 4; ++i) {
                float4 q = p4[i];
                v[i * 4 + 0] = q.x;
                v[i * 4 + 1] = q.y;
                v[i * 4 + 2] = q.z;
                v[i * 4 + 3] = q.w;
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < N; ++j) v[j] = (j < valid) ? to_f32<T>(ptr[j]) : 0.f;
    }
}

template <int N, typename T>
__device__ __forceinline__ void store_n(T* ptr, bool vec_ok, int valid, const float (&v)[N]) {
    if (vec_ok) {
        if constexpr (sizeof(T) == 2) {
            uint4* p4 = reinterpret_cast<uint4*>(ptr);
#pragma unroll
            for (int i = 0; i < N / 8; ++i) {
                uint4 q;
                T* e = reinterpret_cast<T*>(&q);
#pragma unroll
                for (int j = 0; j < 8; ++j) e[j] = from_f32<T>(v[i * 8 + j]);
                p4[i] = q;
            }
        } else {
            float4* p4 = reinterpret_cast<float4*>(ptr);
#pragma unroll
            for (int i = 0; i < N / 4; ++i)
                p4[i] = make_float4(v[i * 4], v[i * 4 + 1], v[i * 4 + 2], v[i * 4 + 3]);
        }
    } else {
#pragma unroll
        for (int j = 0; j < N; ++j)
            if (j < valid) ptr[j] = from_f32<T>(v[j]);
    }
}

__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[32]) { tmem_ld32(taddr, r); }
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[16]) { tmem_ld16(taddr, r); }

// ROWS: the sizes are completed by apply_rows
template <typename InT, typename OutT, bool PAIR, int BN, int EPI_WARPS, bool ROWS>
__global__ void __launch_bounds__(Cfg<PAIR, BN, EPI_WARPS>::THREADS, 1)
    gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA,
                        const __grid_constant__ CUtensorMap tmB,
                        const __grid_constant__ CUtensorMap tmD,
                        const __grid_constant__ CUtensorMap tmAux, const GemmKernelParams params) {
    using C = Cfg<PAIR, BN, EPI_WARPS>;
    constexpr int STAGES = C::STAGES, STAGE_BYTES = C::STAGE_BYTES, B_STAGE_BYTES = C::B_STAGE_BYTES;
    constexpr int TILE_M = C::TILE_M, TMEM_COLS = C::TMEM_COLS;
    constexpr int EPI_THREADS = C::EPI_THREADS, EPI_STAGE_BYTES = EPI_BYTES / EPI_WARPS;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                               ~static_cast<uintptr_t>(1023));
    uint8_t* sA = smem;
    uint8_t* sB = smem + STAGES * A_STAGE_BYTES;
    uint8_t* sEpi = smem + STAGES * STAGE_BYTES;   // [EPI_WARPS][EPI_STAGE_BYTES]
    uint64_t* bars = reinterpret_cast<uint64_t*>(sEpi + EPI_BYTES);
    uint64_t* full = bars;                  // [STAGES]
    uint64_t* empty = bars + STAGES;        // [STAGES]
    uint64_t* tfull = bars + 2 * STAGES;    // [2]
    uint64_t* tempty = bars + 2 * STAGES + 2;  // [2]
    uint64_t* aux_full = bars + 2 * STAGES + 4;  // [EPI_WARPS] a warp's block of the auxiliary matrix has arrived
    uint64_t* used = aux_full + EPI_WARPS;       // [STAGES] a_colsum: the MMAs have read the stage, the sums may
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(used + STAGES);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    // (the same for all lanes, for the compiler too: what the issuing warps compute from it stays in uniform registers)
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int lane = threadIdx.x & 31;
    // PAIR: rank of this CTA in its pair; the first CTA issues the MMAs and owns the `full` / `tempty` counts
    const uint32_t crank = PAIR ? cluster_ctarank() : 0u;
    const int tile0 = PAIR ? static_cast<int>(blockIdx.x >> 1) : static_cast<int>(blockIdx.x);
    const int tile_step = PAIR ? static_cast<int>(gridDim.x >> 1) : static_cast<int>(gridDim.x);

    __shared__ std::conditional_t<ROWS, GemmKernelParams, char> s_params;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], params.a_colsum ? SUM_WARPS : 1);
            mbar_init(&used[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&tfull[a], 1);
            mbar_init(&tempty[a], (PAIR ? 2 : 32) * C::DRAIN_WARPS);   // PAIR: one arrival per epilogue warp of both CTAs
        }
        for (int w = 0; w < EPI_WARPS; ++w) mbar_init(&aux_full[w], 1);
        *abort_flag = 0;
        fence_mbar_init();
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
        if (params.staged) {
            tma_prefetch_desc(&tmD);
            if (params.flags & (RB_GEMM_AUX_OUT | RB_GEMM_DGELU)) tma_prefetch_desc(&tmAux);
        }
    }
    if (warp == 2) {
        if (PAIR) {
            tmem_alloc_pair(tmem_slot, TMEM_COLS);
            tmem_relinquish_pair();
        } else {
            tmem_alloc(tmem_slot, TMEM_COLS);
            tmem_relinquish();
        }
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync_all();   // the peer's barriers exist before anything signals them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    grid_trigger();
    grid_wait();   // all of the above runs beside the end of the kernel before
    if constexpr (ROWS) {
        if (threadIdx.x == 0) {
            s_params = params;
            apply_rows(s_params, tile_step, blockIdx.x == 0);
        }
        __syncthreads();
    }
    const GemmKernelParams& p = [&]() -> const GemmKernelParams& {
        if constexpr (ROWS)
            return s_params;
        else
            return params;
    }();

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        // One lane issues every copy and the warp goes along: behind a branch for that lane, coordinates and addresses
        // would have to be moved to the uniform registers for each instruction (16384 x 4096 x 1024, B MN-major: 128.4 ->
        // 126.1 us; 4096 x 1024 x 6144 into fp32, both MN-major: 61.3 -> 58.4).
        // What a step costs this one warp bounds the whole kernel: the products of a step take 512 cycles, the copy engine
        // brings a step's bytes in some 300 (a loop that only copies: 100 to 115 bytes a cycle and SM, in either layout), but
        // a step that chose its layout, its tap and its form of copy anew took 530 cycles (K-major) to 609 (MN-major) on an
        // otherwise idle SM, and 790 beside a busy epilogue, which takes turns with it at the scheduler.  So a tile's steps
        // are cut into runs without a decision in them -- one copy per operand, of one form, whose coordinates move on by
        // constants -- and the next stage's barrier is asked before it is needed.  Cycles a step (one tile's products / its
        // steps): 8192^3 K-major 530 -> 510, MN-major 609 -> 510; 16384 x 4096 x 1024 with bias 600 -> 485, with GELU and
        // second output 790 -> 540 (now the accumulators are waited for); 4096 x 1024 x 16384 into fp32 690 -> 563.  Back to
        // back under the power cap, where fewer cycles mean a lower clock (us): 117.6 -> 97.9 with bias, 129 -> 107 weight
        // gradient, 428 -> 373 head (8192 x 30528 x 1024), 441 -> 365 its weight gradient; 32 x 1024 x 1024 9.7 -> 7.9.
        const uint32_t el = elect_one();
        int stage = 0;
        uint32_t phase = 0;
        uint32_t ag_ready = 0;
        bool ok = true;
        const bool a_k = p.a_major == 0, b_k = p.b_major == 0, a_merged = p.a_merged, b_merged = p.b_merged;
        const bool gather = p.ag_nranks > 1, conv = p.conv_kb_per_tap > 0;
        // an MN-major operand whose columns are no whole number of 64-column chunks takes a copy per chunk
        const bool chunked = !(a_k || a_merged) || !(b_k || b_merged);
        // PAIR: both CTAs' bytes are counted on the first CTA's barrier
        const uint32_t full0 = PAIR ? mapa_shared(smem_u32(full), 0) : smem_u32(full);
        uint32_t empty_now = mbar_test_wait(&empty[0], 1);
        for (int tile = tile0; tile < p.num_tiles && ok; tile += tile_step) {
            int mb, nb, b, kb_begin, kb_end;
            tile_coords(p, tile, mb, nb, b, kb_begin, kb_end);
            const int m0 = mb * TILE_M + static_cast<int>(crank) * BM;
            const int n0 = nb * BN + (PAIR ? static_cast<int>(crank) * (BN / 2) : 0);
            // position along K in A and in B, and the rows (columns) of each: A's (K-major) shift with the filter tap,
            // B's (MN-major) move on by a block of columns per tap
            int ak = kb_begin * BK, am = m0, bk = ak, bn = n0;
            int tap = 0, shift0 = 0, left = 0x7fffffff;   // steps until the next tap, or until a gathered K wraps around
            if (conv) {
                tap = kb_begin / p.conv_kb_per_tap;
                ak -= tap * p.conv_kb_per_tap * BK;
                am = m0 + p.conv_shift[tap];
                left = p.conv_kb_per_tap - ak / BK;
                if (!b_k) {
                    bk = ak;
                    bn = n0 + tap * p.conv_b_tap_cols;
                }
            } else if (p.wgrad_taps > 0) {
                // column block -> filter tap: the tap's rows are shifted; past the last tap the columns lie outside
                // the matrix and read as zero.  (Of several chunks, this is the first.)
                const int t = min(n0 / p.wgrad_cols, p.wgrad_taps - 1);
                bn = n0 - t * p.wgrad_cols;
                shift0 = p.conv_shift[t];
                bk += shift0;
            } else if (gather && b_k) {
                // start with the k-range this rank holds itself
                const int own = p.ag_my_idx * (p.ag_cols / BK);
                ak = bk = (kb_begin + own < p.num_kb ? kb_begin + own : kb_begin + own - p.num_kb) * BK;
                left = p.num_kb - ak / BK;
            }
            int todo = kb_end - kb_begin;
            while (todo > 0 && ok) {
                // a run of steps that only move along K: coordinates of the operands' maps
                // (four-dimensional, whatever the layout) and what they move on by
                int run = min(todo, left);
                todo -= run;
                int a0 = a_k ? ak : (a_merged ? 0 : am), a1 = a_k ? am : ak;
                int b0 = b_k ? bk : (b_merged ? 0 : bn), b1 = b_k ? bn : bk;
                const int a2 = a_merged ? am >> 6 : 0, b2 = b_merged ? bn >> 6 : 0;
                const int da0 = a_k ? BK : 0, da1 = BK - da0, db0 = b_k ? BK : 0, db1 = BK - db0;
                for (; run > 0; --run) {
                    if (gather) {
                        // wait until every CTA has copied the shard this step reads into the local B buffer
                        const int shard = (b_k ? b0 : n0) / p.ag_cols;
                        if (!(ag_ready & (1u << shard))) {
                            bool got = false;
                            const uint64_t t0 = globaltimer_ns();
                            for (uint32_t it = 0; it < RB_MBAR_SPIN_LIMIT; ++it) {
                                if (__any_sync(0xffffffffu, *abort_flag)) break;
                                unsigned int v;
                                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p.ag_flags + shard) : "memory");
                                if (__all_sync(0xffffffffu, v >= gridDim.x)) {
                                    got = true;
                                    break;
                                }
                                if ((it & 0xff) == 0xff && __any_sync(0xffffffffu, globaltimer_ns() - t0 > RB_WAIT_LIMIT_NS)) break;
                                __nanosleep(64);
                            }
                            if (!got) {
                                *abort_flag = 1;
                                ok = false;
                                break;
                            }
                            asm volatile("fence.proxy.async.global;" ::: "memory");
                            ag_ready |= 1u << shard;
                        }
                    }
                    // (asked about at the end of the step before: the answer is there by now)
                    if (!__all_sync(0xffffffffu, empty_now) && !mbar_wait_warp(&empty[stage], phase ^ 1, abort_flag)) {
                        ok = false;
                        break;
                    }
                    uint8_t* a_dst = sA + stage * A_STAGE_BYTES;
                    uint8_t* b_dst = sB + stage * B_STAGE_BYTES;
                    const uint32_t fb = full0 + stage * 8;
                    if (!PAIR || crank == 0) mbar_arrive_expect_tx_el(&full[stage], (PAIR ? 2 : 1) * STAGE_BYTES, el);
                    auto load = [&](uint8_t* dst, const CUtensorMap* m, int c0, int c1, int c2) {
                        if constexpr (PAIR)
                            tma_load_4d_pair(dst, m, fb, c0, c1, c2, b, el);
                        else
                            tma_load_4d_el(dst, m, &full[stage], c0, c1, c2, b, el);
                    };
                    load(a_dst, &tmA, a0, a1, a2);
                    load(b_dst, &tmB, b0, b1, b2);
                    if (chunked) {
                        if (!a_k && !a_merged) {
#pragma unroll 1
                            for (int c = 1; c < BM / 64; ++c) load(a_dst + c * (BK * 128), &tmA, a0 + c * 64, a1, 0);
                        }
                        if (!b_k && !b_merged) {
#pragma unroll 1
                            for (int c = 1; c < C::B_ROWS / 64; ++c) {
                                int cx = b0 + c * 64, cy = b1;
                                if (p.wgrad_taps > 0) {
                                    cx = n0 + c * 64;
                                    const int t = min(cx / p.wgrad_cols, p.wgrad_taps - 1);
                                    cx -= t * p.wgrad_cols;
                                    cy += p.conv_shift[t] - shift0;
                                }
                                load(b_dst + c * (BK * 128), &tmB, cx, cy, 0);
                            }
                        }
                    }
                    a0 += da0;
                    a1 += da1;
                    b0 += db0;
                    b1 += db1;
                    if (++stage == STAGES) {
                        stage = 0;
                        phase ^= 1;
                    }
                    empty_now = mbar_test_wait(&empty[stage], phase ^ 1);
                }
                if (todo > 0) {   // (behind the last tap there is no further step)
                    ak = 0;
                    if (conv) {
                        left = p.conv_kb_per_tap;
                        am = m0 + p.conv_shift[++tap];
                        if (b_k) {
                            bk = b0;
                        } else {
                            bk = 0;
                            bn += p.conv_b_tap_cols;
                        }
                    } else {
                        left = 0x7fffffff;
                        bk = 0;
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (crank == 0) {
            // ---------------- MMA issuer (PAIR: the first CTA issues for both) ----------------
            // (one lane issues, the warp goes along: as above)
            const uint32_t el = elect_one();
            constexpr int fmt = (sizeof(InT) == 2 && std::is_same<InT, __nv_bfloat16>::value) ? 1 : 0;
            const uint32_t idesc = make_idesc_f16(fmt, p.a_major, p.b_major, TILE_M, BN);
            // per-UMMA_K (16 elements) advance of the smem start address, in the descriptors' units of 16 bytes
            const uint32_t a_kstep = (p.a_major == 0) ? 32u / 16 : 2048u / 16;
            const uint32_t b_kstep = (p.b_major == 0) ? 32u / 16 : 2048u / 16;
            // descriptors of the first stage (their low halves): the address of any other is added
            const uint32_t a_desc = desc_lo_sw128(smem_u32(sA), (p.a_major == 0) ? 16u : BK * 128u);
            const uint32_t b_desc = desc_lo_sw128(smem_u32(sB), (p.b_major == 0) ? 16u : BK * 128u);
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            int it = 0;
            for (int tile = tile0; tile < p.num_tiles && ok; tile += tile_step) {
                int mb_, nb_, b_, kb_begin, kb_end;
                tile_coords(p, tile, mb_, nb_, b_, kb_begin, kb_end);
                if (kb_begin >= kb_end) continue;
                const int acc = it & 1;
                const uint32_t acc_phase = (it >> 1) & 1;
                ++it;
                if (!mbar_wait_warp(&tempty[acc], acc_phase ^ 1, abort_flag)) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * BN;
                for (int kb = kb_begin; kb < kb_end; ++kb) {
                    if (!mbar_wait_warp(&full[stage], phase, abort_flag)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t da0 = a_desc + static_cast<uint32_t>(stage) * (A_STAGE_BYTES / 16);
                    const uint32_t db0 = b_desc + static_cast<uint32_t>(stage) * (B_STAGE_BYTES / 16);
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) {
                        const uint32_t da = da0 + k * a_kstep, db = db0 + k * b_kstep;
                        if constexpr (PAIR)
                            umma_f16_pair_lo(d_tmem, da, db, idesc, (kb > kb_begin || k > 0) ? 1u : 0u, el);
                        else
                            umma_f16_lo(d_tmem, da, db, idesc, (kb > kb_begin || k > 0) ? 1u : 0u, el);
                    }
                    // frees the stage (PAIR: in both CTAs), or hands it on to the warps that sum its columns
                    uint64_t* done = p.a_colsum ? &used[stage] : &empty[stage];
                    if (el) {
                        if constexpr (PAIR)
                            umma_commit_pair(done, 3);
                        else
                            umma_commit(done);
                    }
                    if (++stage == STAGES) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (ok && el) {
                    if constexpr (PAIR)
                        umma_commit_pair(&tfull[acc], 3);
                    else
                        umma_commit(&tfull[acc]);
                }
            }
        }
    } else if (warp >= 2 + EPI_WARPS) {
        if (p.a_colsum) {
            // ---------------- column sums of A (bias gradient beside a weight gradient) ----------------
            // A = dy is stored [K, M] and passes through shared memory anyway: a separate kernel reads it once more
            // from memory (98 us for 8192 x 30528).  The n-blocks of a tile row share the work: block nb sums the k
            // steps congruent to nb, so every row is added exactly once and a summed step (16 KiB of shared-memory
            // reads) comes once per num_n_blocks steps.
            const int c = warp - (2 + EPI_WARPS);   // 64-column chunk of the tile
            const int piece = lane & 7, kr = lane >> 3;
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int tile = tile0; tile < p.num_tiles && ok; tile += tile_step) {
                int mb, nb, b, kb_begin, kb_end;
                tile_coords(p, tile, mb, nb, b, kb_begin, kb_end);
                float s[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) s[j] = 0.f;
                bool any = false;
                for (int kb = kb_begin; kb < kb_end; ++kb) {
                    if (!mbar_wait_warp(&used[stage], phase, abort_flag)) {
                        ok = false;
                        break;
                    }
                    if (kb % p.num_n_blocks == nb) {
                        any = true;
                        const uint8_t* rows = sA + stage * A_STAGE_BYTES + c * (BK * 128);
#pragma unroll 8
                        for (int r = kr; r < BK; r += 4) {
                            const uint4 q4 = *reinterpret_cast<const uint4*>(rows + r * 128 + ((piece ^ (r & 7)) << 4));
                            const InT* e = reinterpret_cast<const InT*>(&q4);
#pragma unroll
                            for (int j = 0; j < 8; ++j) s[j] += to_f32<InT>(e[j]);
                        }
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&empty[stage]);
                    if (++stage == STAGES) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (any && ok) {
                    const int m0 = mb * TILE_M + static_cast<int>(crank) * BM + c * 64 + piece * 8;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        s[j] += __shfl_xor_sync(0xffffffffu, s[j], 8);
                        s[j] += __shfl_xor_sync(0xffffffffu, s[j], 16);
                        if (kr == 0 && m0 + j < p.M) atomicAdd(p.a_colsum + m0 + j, s[j]);
                    }
                }
            }
        }
    } else {
        // ---------------- epilogue (the EPI_WARPS warps from 2 on) ----------------
        if (p.ag_nranks > 1) {
            // all-gather prologue: the epilogue threads of every CTA copy their share of each peer's
            // shard into the local B buffer (plain 16-byte peer loads), in the order the k loop consumes
            // them (own shard first); a counter per shard tells the TMA producers when it is whole
            const int t = threadIdx.x - 64;
            const int vec_per_row = p.ag_cols / 8;
            const long long total = static_cast<long long>(p.ag_rows) * vec_per_row;
            const long long dst_ld = static_cast<long long>(p.ag_nranks) * p.ag_cols;
            for (int rr = 0; rr < p.ag_nranks; ++rr) {
                const int r = (p.ag_my_idx + rr) % p.ag_nranks;   // the order in which the k loop needs them
                const uint4* src = reinterpret_cast<const uint4*>(p.ag_src[r]);
                InT* dst = reinterpret_cast<InT*>(p.ag_dst) + static_cast<long long>(r) * p.ag_cols;
                for (long long i = static_cast<long long>(blockIdx.x) * EPI_THREADS + t; i < total;
                     i += static_cast<long long>(gridDim.x) * EPI_THREADS * 4) {
                    uint4 v[4];
                    long long idx[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        idx[u] = i + static_cast<long long>(u) * gridDim.x * EPI_THREADS;
                        if (idx[u] < total) v[u] = src[idx[u]];
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        if (idx[u] < total) {
                            const long long row = idx[u] / vec_per_row, c = idx[u] - row * vec_per_row;
                            *reinterpret_cast<uint4*>(dst + row * dst_ld + c * 8) = v[u];
                        }
                    }
                }
                asm volatile("fence.proxy.async.global;" ::: "memory");
                __threadfence();
                asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory");
                if (t == 0) atomicAdd(p.ag_flags + r, 1u);
            }
        }
        const int q = warp & 3;  // TMEM lane quarter this warp may access
        constexpr int PARTS = C::PARTS, PART_COLS = C::PART_COLS;
        const int part = (warp - 2) >> 2;    // which columns of the tile this warp drains
        const int row_in_tile = q * 32 + lane;
        const int first_tile = part < PARTS ? tile0 : p.num_tiles;
        // activations and 16-bit matrices beside the output: not with eight warps and a 16-bit output (see dispatch)
        constexpr bool OUT16 = sizeof(OutT) == 2, ACT = EPI_WARPS == 16 || !OUT16;
        const bool has_bias = p.flags & RB_GEMM_BIAS;
        const bool has_res = p.flags & RB_GEMM_RESIDUAL;
        const bool act_gelu = ACT && (p.flags & RB_GEMM_GELU);
        const bool act_dgelu = ACT && (p.flags & RB_GEMM_DGELU);
        const bool aux_out = ACT && (p.flags & RB_GEMM_AUX_OUT);
        const bool accum = p.flags & RB_GEMM_ACCUM;
        const bool bias_al = p.bias_al, in_al = p.in_al, out_al = p.out_al;
        auto release_acc = [&](int acc) {
            tc_fence_before();
            if constexpr (PAIR) {
                // the accumulator may be overwritten once the epilogue warps of BOTH CTAs have drained it.  (With a release
                // at cluster scope this took 1200 to 2500 cycles, a sixth of what a tile of K = 1024 takes: bias + GELU +
                // second output 160.7 -> 151.7 us, GELU gradient 162.6 -> 152.8, B MN-major 126.2 -> 121.4, 16384 x 4096.)
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&tempty[acc]), 0));
            } else {
                mbar_arrive(&tempty[acc]);
            }
        };
        int it = 0;
        if (p.staged) {
            // A thread that stores (or loads) its own row makes every 16-byte access of its warp touch 32 lines, 32 cycles
            // each: for two 16-bit outputs alone as long as a main loop of K = 1024 (8200 cycles).  Rows therefore go to the
            // staging block (conflict-free by the swizzle) and the copy engine moves 32 x 32 blocks; it also clips them to
            // M x N, adds fp32 blocks to D (accumulation, split K) and fetches the auxiliary block one step ahead.
            // 8192 x 30528 x 1024: 426 -> 386 us; weight gradient 4096 x 1024 x 16384: 122 -> 116 us.  Larger blocks (32 x
            // 64, or 128 rows per four warps) hold up the loads for longer: GELU 131 -> 138 us, plain 108 -> 112.
            //
            // Sixteen warps for an activation: a block is a chain of tensor-memory load, bias, GELU (64 instructions of the
            // special-function unit a thread), staging and copy, 2700 cycles long, and with two warps to a scheduler that
            // is 11000 a tile, behind which the products of K = 1024 (8200) wait.  Four to a scheduler hide each other's
            // latency: 16384 x 4096 x 1024 with GELU and second output 137 -> 121 us, GELU gradient 132 -> 123, 2000 x 3072
            // x 768 with GELU and second output 21.7 -> 18.7.  Without an activation a block is short, and the extra warps
            // only take turns with the one that issues the copies: 96.5 -> 100.4 with bias, fp32 sums 114 -> 122; those keep
            // eight.  (GELU's value and the one before it share a block's place: the second is written once the first has
            // left, which its arithmetic covers.)
            uint8_t* stage_buf = sEpi + (warp - 2) * EPI_STAGE_BYTES;
            constexpr int SLOTS = EPI_STAGE_BYTES / (OUT16 ? 2048 : 4096);   // blocks the staging memory holds
            uint64_t* abar = &aux_full[warp - 2];
            uint32_t aux_phase = 0;
            uint32_t turn = 0;   // which slot the next block takes: counted over tiles, whose blocks may be odd in number
            const uint32_t sw64 = (lane >> 1) & 3, sw128 = lane & 7;
            const bool add_out = !OUT16 && (accum || p.partial);
            // lays a row of 32 16-bit values out in a block
            auto put_row = [&](uint8_t* block, const float (&v)[32], auto type) {
                using T = decltype(type);
#pragma unroll
                for (int g = 0; g < 4; ++g)
                    *reinterpret_cast<uint4*>(block + lane * 64 + ((g ^ sw64) << 4)) =
                        make_uint4(pack2<T>(v[g * 8], v[g * 8 + 1]), pack2<T>(v[g * 8 + 2], v[g * 8 + 3]),
                                   pack2<T>(v[g * 8 + 4], v[g * 8 + 5]), pack2<T>(v[g * 8 + 6], v[g * 8 + 7]));
            };
            bool ok = true;
            for (int tile = first_tile; tile < p.num_tiles && ok; tile += tile_step) {
                int mb, nb, b, kb_begin, kb_end;
                tile_coords(p, tile, mb, nb, b, kb_begin, kb_end);
                if (kb_begin >= kb_end) continue;
                const int acc = it & 1;
                const uint32_t acc_phase = (it >> 1) & 1;
                ++it;
                const int row0 = mb * TILE_M + static_cast<int>(crank) * BM + q * 32;
                const int col0 = nb * BN + part * PART_COLS;
                const bool row_ok = row0 + lane < p.M;
                int d_row = row0;
                if constexpr (ROWS && !OUT16)   // (parts one below the other)
                    if (p.rows_mode == RB_GEMM_ROWS_M) d_row += kb_begin / p.kb_per_split * p.num_m_blocks * TILE_M;
                // blocks of this warp that hold part of the matrix
                const int nblk = row0 < p.M ? max(0, min(PART_COLS / 32, (p.N - col0 + 31) / 32)) : 0;
                auto fetch_aux = [&](int c) {   // (one lane; the block before has left its place)
                    tma_store_wait_read<0>();
                    mbar_arrive_expect_tx(abar, 2048);
                    tma_load_3d(stage_buf, &tmAux, abar, col0 + c * 32, row0, b);
                };
                if (OUT16 && act_dgelu && nblk > 0 && lane == 0) fetch_aux(0);
                if (!mbar_wait_warp(&tfull[acc], acc_phase, abort_flag)) break;
                tc_fence_after();
                if (nblk == 0) release_acc(acc);
                const long long row_off = static_cast<long long>(b) * p.strideD +
                                          static_cast<long long>(row_ok ? row0 + lane : 0) * p.ldd;
                const uint32_t t_acc = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * BN + part * PART_COLS;
#pragma unroll 1
                for (int c = 0; c < nblk; ++c) {
                    const int col = col0 + c * 32;
                    uint32_t r[32];
                    tmem_ld32(t_acc + c * 32, r);
                    tmem_ld_wait();
                    if (c == nblk - 1) release_acc(acc);
                    const int valid = min(32, p.N - col);
                    const bool full_chunk = valid == 32;
                    float v[32];
                    const uint64_t alpha2 = f2_pack(p.alpha, p.alpha);
                    if (has_bias) {
                        float t[32];
                        load_n(reinterpret_cast<const InT*>(p.bias) + col, full_chunk && bias_al, valid, t);
#pragma unroll
                        for (int j = 0; j < 32; j += 2)
                            f2_unpack(f2_fma(f2_pack_bits(r[j], r[j + 1]), alpha2, f2_pack(t[j], t[j + 1])), v[j], v[j + 1]);
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; j += 2)
                            f2_unpack(f2_mul(f2_pack_bits(r[j], r[j + 1]), alpha2), v[j], v[j + 1]);
                    }
                    // the block that is about to be overwritten has been read by the copy engine
                    auto wait_slot = [&] {
                        if (lane == 0) tma_store_wait_read<SLOTS - 1>();
                        __syncwarp();
                    };
                    if (OUT16 && aux_out) {   // the value before the activation, in storage precision
                        wait_slot();
                        put_row(stage_buf, v, InT());
                        fence_proxy_async();
                        __syncwarp();
                        if (lane == 0) {
                            tma_store_3d(&tmAux, stage_buf, col, row0, b);
                            tma_store_commit();
                        }
                    }
                    if (act_gelu) {
#pragma unroll
                        for (int j = 0; j < 32; j += 2) gelu_erf2(v[j], v[j + 1]);
                    }
                    if (OUT16 && act_dgelu) {
                        if (!mbar_wait_warp(abar, aux_phase, abort_flag)) {
                            ok = false;
                            break;
                        }
                        aux_phase ^= 1;
#pragma unroll
                        for (int g = 0; g < 4; ++g) {
                            const uint4 x = *reinterpret_cast<const uint4*>(stage_buf + lane * 64 + ((g ^ sw64) << 4));
                            const InT* e = reinterpret_cast<const InT*>(&x);
#pragma unroll
                            for (int j = 0; j < 8; j += 2)
                                gelu_erf_grad2(to_f32<InT>(e[j]), to_f32<InT>(e[j + 1]), v[g * 8 + j], v[g * 8 + j + 1]);
                        }
                        __syncwarp();   // every lane has its row: the output takes its place
                    }
                    if (has_res && row_ok) {
                        float t[32];
                        load_n(reinterpret_cast<const InT*>(p.residual) + row_off + col, full_chunk && in_al, valid, t);
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] += t[j];
                    }
                    if (OUT16 && accum && row_ok) {
                        float t[32];
                        load_n(reinterpret_cast<const OutT*>(p.D) + row_off + col, full_chunk && out_al, valid, t);
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] += t[j];
                    }
                    if (!(OUT16 && act_dgelu)) wait_slot();
                    uint8_t* dst = stage_buf + (SLOTS > 1 && (turn & 1) ? 2048 : 0);
                    ++turn;
                    if constexpr (OUT16) {
                        put_row(dst, v, OutT());
                    } else {
#pragma unroll
                        for (int g = 0; g < 8; ++g)
                            *reinterpret_cast<float4*>(dst + lane * 128 + ((g ^ sw128) << 4)) =
                                make_float4(v[g * 4], v[g * 4 + 1], v[g * 4 + 2], v[g * 4 + 3]);
                    }
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) {
                        if (add_out)
                            tma_reduce_add_3d(&tmD, dst, col, d_row, b);
                        else
                            tma_store_3d(&tmD, dst, col, d_row, b);
                        tma_store_commit();
                        if (OUT16 && act_dgelu && c + 1 < nblk) fetch_aux(c + 1);
                    }
                }
            }
            // the staging memory must outlive the copies that read it; their writes are complete when the kernel is
            if (lane == 0) tma_store_wait_read<0>();
        }
        constexpr int DC = EPI_WARPS == 16 ? 16 : 32;   // columns at a time: sixteen warps leave a thread 96 registers
        for (int tile = p.staged ? p.num_tiles : first_tile; tile < p.num_tiles; tile += tile_step) {
            int mb, nb, b, kb_begin, kb_end;
            tile_coords(p, tile, mb, nb, b, kb_begin, kb_end);
            if (kb_begin >= kb_end) continue;
            const int acc = it & 1;
            const uint32_t acc_phase = (it >> 1) & 1;
            ++it;
            if (!mbar_wait_warp(&tfull[acc], acc_phase, abort_flag)) break;
            tc_fence_after();
            int row = mb * TILE_M + static_cast<int>(crank) * BM + row_in_tile;
            bool row_ok = row < p.M;
            if (p.map_hp > 0 && row_ok) {
                // rows are positions of a zero-padded image grid: only the interior is stored
                const int per_img = p.map_hp * p.map_wp;
                const int img = row / per_img;
                const int rem = row - img * per_img;
                const int yy = rem / p.map_wp - p.map_pad;
                const int xx = rem - (rem / p.map_wp) * p.map_wp - p.map_pad;
                row_ok = yy >= 0 && yy < p.map_h && xx >= 0 && xx < p.map_w;
                row = (img * p.map_h + yy) * p.map_w + xx;
            }
            const long long row_off = static_cast<long long>(b) * p.strideD +
                                      static_cast<long long>(row_ok ? row : 0) * p.ldd;
#pragma unroll 1
            for (int c = part * (PART_COLS / DC); c < (part + 1) * (PART_COLS / DC); ++c) {
                const int col = nb * BN + c * DC;
                if (col >= p.N) break;
                uint32_t r[DC];
                tmem_ld(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * BN + c * DC, r);
                tmem_ld_wait();
                if (!row_ok) continue;
                const int valid = min(DC, p.N - col);
                const bool full_chunk = valid == DC;
                float v[DC];
#pragma unroll
                for (int j = 0; j < DC; ++j) v[j] = __uint_as_float(r[j]) * p.alpha;
                if constexpr (std::is_same<OutT, float>::value) {
                    if (p.partial || p.rs_nranks > 1) {
                        // partial sums (a K slice, and/or one replica's share of a reduce-scatter):
                        // accumulate with vector reductions.  With rs_nranks > 1 the output columns
                        // are split in equal blocks and block j lives in rank j's buffer, so the
                        // reduction goes to that peer's memory over NVLink.
                        float* dptr = reinterpret_cast<float*>(p.D) + row_off + col;
                        if (p.rs_nranks > 1) {
                            const int owner = col / p.rs_cols;
                            dptr = reinterpret_cast<float*>(p.rs_peer[owner]) + row_off + (col - owner * p.rs_cols);
                        }
                        if (full_chunk && out_al) {
#pragma unroll
                            for (int j = 0; j < DC; j += 4)
                                asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dptr + j),
                                             "f"(v[j]), "f"(v[j + 1]), "f"(v[j + 2]), "f"(v[j + 3])
                                             : "memory");
                        } else {
#pragma unroll
                            for (int j = 0; j < DC; ++j)
                                if (j < valid) atomicAdd(dptr + j, v[j]);
                        }
                        continue;
                    }
                }
                if (has_bias) {
                    float t[DC];
                    load_n(reinterpret_cast<const InT*>(p.bias) + col, full_chunk && bias_al, valid, t);
#pragma unroll
                    for (int j = 0; j < DC; ++j) v[j] += t[j];
                }
                if (aux_out)
                    store_n(reinterpret_cast<InT*>(p.aux_out) + row_off + col, full_chunk && in_al,
                            valid, v);
                if (act_gelu) {
#pragma unroll
                    for (int j = 0; j < DC; ++j) v[j] = gelu_erf(v[j]);
                }
                if (act_dgelu) {
                    float t[DC];
                    load_n(reinterpret_cast<const InT*>(p.aux_in) + row_off + col,
                           full_chunk && in_al, valid, t);
#pragma unroll
                    for (int j = 0; j < DC; ++j) v[j] *= gelu_erf_grad(t[j]);
                }
                if (has_res) {
                    float t[DC];
                    load_n(reinterpret_cast<const InT*>(p.residual) + row_off + col,
                           full_chunk && in_al, valid, t);
#pragma unroll
                    for (int j = 0; j < DC; ++j) v[j] += t[j];
                }
                OutT* dptr = reinterpret_cast<OutT*>(p.D) + row_off + col;
                if (accum) {
                    float t[DC];
                    load_n(dptr, full_chunk && out_al, valid, t);
#pragma unroll
                    for (int j = 0; j < DC; ++j) v[j] += t[j];
                }
                store_n(dptr, full_chunk && out_al, valid, v);
            }
            release_acc(acc);
        }
    }

    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        if (threadIdx.x == 0) {
            atomicExch(params.err, ERR_MBAR_TIMEOUT);
            // let bulk copies that may still be in flight land before the CTA's
            // shared memory is released
            const long long t0 = clock64();
            while (clock64() - t0 < 2000000) {
            }
        }
        __syncthreads();
    }
    // PAIR: neither CTA leaves (or frees tensor memory) while the other may still signal its barriers or
    // its MMAs may still write this CTA's accumulators
    if (PAIR) cluster_sync_all();
    if (warp == 2) {
        tc_fence_after();
        if (PAIR)
            tmem_dealloc_pair(tmem_base, TMEM_COLS);
        else
            tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                             &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

int make_tmap_4d(CUtensorMap* out, const void* base, int fmt, uint64_t d0, uint64_t d1, uint64_t d2,
                 uint64_t d3, uint64_t s1, uint64_t s2, uint64_t s3, uint32_t b0, uint32_t b1) {
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) return -100;
    cuuint64_t dims[4] = {d0, d1, d2, d3};
    cuuint64_t strides[3] = {s1, s2, s3};
    cuuint32_t box[4] = {b0, b1, 1, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUtensorMapDataType dt =
        fmt == 1 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    CUresult r = CUDA_SUCCESS;
    for (int attempt = 0; attempt < 2; ++attempt) {
        r = fn(out, dt, 4, const_cast<void*>(base), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_ERROR_INVALID_CONTEXT) break;
        // a thread that has made no runtime call yet (an autograd worker whose first operator is ours) has
        // no context bound for driver entry points: bind the device's primary context and try again
        cudaFree(nullptr);
    }
    return r == CUDA_SUCCESS ? 0 : -static_cast<int>(r) - 1000;
}

// fp32 tensor, 4-D, 128-byte swizzle: box [b0 <= 32 elements, b1 rows, 1, 1]
int make_tmap_4d_f32(CUtensorMap* out, const void* base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t d3,
                     uint64_t s1, uint64_t s2, uint64_t s3, uint32_t b0, uint32_t b1) {
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) return -100;
    cuuint64_t dims[4] = {d0, d1, d2, d3};
    cuuint64_t strides[3] = {s1, s2, s3};
    cuuint32_t box[4] = {b0, b1, 1, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = CUDA_SUCCESS;
    for (int attempt = 0; attempt < 2; ++attempt) {
        r = fn(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<void*>(base), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_ERROR_INVALID_CONTEXT) break;
        cudaFree(nullptr);
    }
    return r == CUDA_SUCCESS ? 0 : -static_cast<int>(r) - 1000;
}

// An MN-major operand [rows, 64 * chunks] as [chunk][row][64]: box of `n` chunks x 64 rows, 128-byte swizzle
static int make_tmap_chunks(CUtensorMap* out, const void* base, int fmt, uint64_t rows, uint64_t chunks, uint64_t batch,
                            uint64_t row_bytes, uint64_t batch_bytes, uint32_t n) {
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) return -100;
    cuuint64_t dims[4] = {64, rows, chunks, batch};
    cuuint64_t strides[3] = {row_bytes, 128, batch_bytes};
    cuuint32_t box[4] = {64, BK, n, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = CUDA_SUCCESS;
    for (int attempt = 0; attempt < 2; ++attempt) {
        r = fn(out, fmt == 1 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4,
               const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_ERROR_INVALID_CONTEXT) break;
        cudaFree(nullptr);   // a thread without a context yet: see make_tmap_4d
    }
    return r == CUDA_SUCCESS ? 0 : -static_cast<int>(r) - 1000;
}

// A matrix the GEMM's epilogue writes (or reads) in 32 x 32 blocks: 16-bit elements with 64-byte swizzled block
// rows, fp32 with 128-byte ones.  Blocks are clipped to d0 x d1 by the copy engine.
static int make_tmap_block32(CUtensorMap* out, const void* base, bool fp32, int fmt, uint64_t d0, uint64_t d1,
                             uint64_t d2, uint64_t s1_bytes, uint64_t s2_bytes) {
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) return -100;
    cuuint64_t dims[3] = {d0, d1, d2};
    cuuint64_t strides[2] = {s1_bytes, s2_bytes};
    cuuint32_t box[3] = {32, 32, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    const CUtensorMapDataType dt = fp32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                        : (fmt == 1 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16);
    const CUresult r = fn(out, dt, 3, const_cast<void*>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE,
                          fp32 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : -static_cast<int>(r) - 1000;
}

static __device__ int g_error_word = 0;

int* error_word_ptr() {
    // one address per device
    static int* ptrs[64] = {nullptr};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return nullptr;
    if (!ptrs[dev]) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_error_word) != cudaSuccess) return nullptr;
        ptrs[dev] = static_cast<int*>(p);
    }
    return ptrs[dev];
}

int num_sms() {
    static int n[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return 148;
    if (!n[dev] && cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148;
    return n[dev];
}

template <typename InT, typename OutT, bool PAIR, int TN, int EW, bool ROWS = false>
static int launch(const RbGemmArgs& a, const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmD,
                  const CUtensorMap& tmAux, const GemmKernelParams& p, cudaStream_t stream) {
    auto kern = gemm_tcgen05_kernel<InT, OutT, PAIR, TN, EW, ROWS>;
    constexpr int smem = Cfg<PAIR, TN, EW>::SMEM_BYTES, GEMM_THREADS = Cfg<PAIR, TN, EW>::THREADS;
    static bool attr_set[64] = {false};
    static int max_clusters[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (!attr_set[dev & 63]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return -static_cast<int>(e);
        attr_set[dev & 63] = true;
    }
    if (!PAIR) {
        int grid = p.num_tiles < num_sms() ? p.num_tiles : num_sms();
        if (a.max_ctas > 0 && grid > a.max_ctas) grid = a.max_ctas;
        const cudaError_t e = launch_after(kern, grid, GEMM_THREADS, smem, stream, tmA, tmB, tmD, tmAux, p);
        return e == cudaSuccess ? 0 : -static_cast<int>(e);
    }
    // one cluster of two CTAs per TPC; persistent over the pair tiles
    if (!max_clusters[dev & 63]) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.blockDim = dim3(GEMM_THREADS, 1, 1);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        cfg.gridDim = dim3(num_sms(), 1, 1);
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) n = num_sms() / 2;
        max_clusters[dev & 63] = n;
    }
    int clusters = !ROWS && p.num_tiles < max_clusters[dev & 63] ? p.num_tiles : max_clusters[dev & 63];
    if (a.max_ctas > 1 && clusters > a.max_ctas / 2) clusters = a.max_ctas / 2;
    const cudaError_t e = launch_after_clusters(kern, 2, 2 * clusters, GEMM_THREADS, smem, stream, tmA, tmB, tmD, tmAux, p);
    return e == cudaSuccess ? 0 : -static_cast<int>(e);
}

template <typename InT>
static int dispatch(const RbGemmArgs& a, bool pair, int tn, const CUtensorMap& tmA, const CUtensorMap& tmB,
                    const CUtensorMap& tmD, const CUtensorMap& tmAux, const GemmKernelParams& p, cudaStream_t st) {
    // what the epilogue has to do decides on its warps; fp32 results with an activation are rare and stay on eight
    const bool act = a.out_dtype == 0 && (a.flags & (RB_GEMM_GELU | RB_GEMM_DGELU | RB_GEMM_AUX_OUT));
#define RB_GEMM_LAUNCH(PAIR, TN)                                                                \
    return a.out_dtype == 1 ? launch<InT, float, PAIR, TN, 8>(a, tmA, tmB, tmD, tmAux, p, st) \
           : act            ? launch<InT, InT, PAIR, TN, 16>(a, tmA, tmB, tmD, tmAux, p, st)  \
                            : launch<InT, InT, PAIR, TN, 8>(a, tmA, tmB, tmD, tmAux, p, st)
    if (a.rows_ctl)
        return a.out_dtype == 1 ? launch<InT, float, true, 256, 8, true>(a, tmA, tmB, tmD, tmAux, p, st)
                                : launch<InT, InT, true, 256, 8, true>(a, tmA, tmB, tmD, tmAux, p, st);
    if (pair) RB_GEMM_LAUNCH(true, 256);
    if (tn == 64) RB_GEMM_LAUNCH(false, 64);
    if (tn == 128) RB_GEMM_LAUNCH(false, 128);
    RB_GEMM_LAUNCH(false, 256);
#undef RB_GEMM_LAUNCH
}

// RB_GEMM_PAIR_GATHER=1 also puts the gather -> GEMM variant on the pair kernel (same prologue code).  Measured
// with four local slices it is no faster there (0.230 ms against 0.223 ms for M 8192, N = K = 4096: the
// prologue copy, not the main loop, is what the variant adds), so it stays on the single-CTA kernel; the
// scatter epilogue does gain from the pair kernel (0.224 ms against 0.248 ms) and uses it.
static bool pair_gather_enabled() {
    static int v = -1;
    if (v < 0) {
        const char* e = getenv("RB_GEMM_PAIR_GATHER");
        v = (e && e[0] == '1') ? 1 : 0;
    }
    return v == 1;
}

// RB_GEMM_PAIR=0 keeps every GEMM on the single-CTA kernel
static bool pair_enabled() {
    static int v = -1;
    if (v < 0) {
        const char* e = getenv("RB_GEMM_PAIR");
        v = (e && e[0] == '0') ? 0 : 1;
    }
    return v == 1;
}

// How a product is cut up: the kernel variant, its output tiles, and the parts K is split into.
struct Tiling {
    bool pair;
    int tn, m_blocks, n_blocks, split;
    int tail_tiles, tail_split, tail_kb;   // see Tail
};
// The tiles that do not fill the last wave of the CTA pairs, of a product that is added to an fp32 matrix: K is shared out
// so that every pair has something to do.
//  - No more tiles than half the pairs (37 of 74): K in `split` equal parts, one wave of them.
//  - More: each tile's pair takes the first `kb` steps, all in step, so that operands are shared through L2; the pairs left
//    over take the remaining steps of one tile after another, in at most six rounds.
// What it is worth (us, whole tiles -> shared; the matrix comes from memory, as a gradient buffer does; w + t: full waves
// and tiles left over):
//     w + t          K = 1024       1536           2048           4096           8192
//     1 + 14         27.5 -> 26.7   32.8 -> 28.7   36.9 -> 32.8   57.3 -> 43.1   94.2 -> 65.6
//     1 + 36                        32.8 -> 30.8   36.9 -> 34.8   57.4 -> 51.1   96.3 -> 79.9
//     3 + 34                        57.3 -> 55.3   65.6 -> 62.5   102 -> 94.2    184 -> 167
//     6 + 36                        88.1 -> 86.1   102 -> 98.3    176 -> 166     347 -> 328
//     1 + 46 (two rounds)           37.9 -> 37.9   42.0 -> 39.9   62.5 -> 56.4   104 -> 91.2
//     3 + 50 (three)                                              104 -> 100     187 -> 178
//     1 + 58 (four)                                               61.4 -> 57.5   100 -> 95.2
//     1 + 62 (six) by 16384: 185 -> 178
// and with copies that took longer to issue, where it is not used: 1 + 36 and 3 + 34 by 512 25.5 -> 25.6 and 42.0 -> 43.0, by
// 1024 30.7 -> 29.6 and 50.2 -> 52.1; 2 + 68 (twelve rounds) and 1 + 70 (eighteen) by 16384 327 -> 328 and 217 -> 222.
// With a short K the matrix bounds the product and a part's addition to it costs what the part saves: from 24 steps on, or
// where one full wave is followed by a third of one at most.  Beyond six rounds the helpers' additions eat up the gain.
// Only behind full waves: with fewer tiles than pairs its parts are longer than those of the even split below, and the tensor
// core's sums lose with length (4096 x 1024 by 16384, 64 tiles: 101.0 -> 99.1 us, relative error 2.1e-6 -> 1.6e-5; with parts
// as long as before, summed in registers, 100.9 us).  Behind full waves parts are shorter than the whole tiles they replace.
struct Tail {
    int split, kb;       // split > 1: equal parts of kb steps; 1: owners and helpers; 0: whole tiles
    double cost;         // in k steps of the longest chain of a pair
};
// What a part costs besides its own steps.  (An estimate.  With anything from 4 to 10 the sizes above are cut up the same way
// but for helpers' cases up to K = 4096, whose times differ by 4 % at most.)
constexpr double DRAIN_STEPS = 6.0;
constexpr int TAIL_ROUNDS = 6, TAIL_STEPS = 24;   // see above
static Tail choose_tail(int tiles, int units, int num_kb) {
    Tail t = {0, num_kb, num_kb + DRAIN_STEPS};
    if (tiles <= 0 || tiles >= units) return t;
    if (2 * tiles <= units) {
        const int s = std::min(units / tiles, num_kb / 4);
        if (s > 1) {
            const int kb = (num_kb + s - 1) / s;
            t = {(num_kb + kb - 1) / kb, kb, kb + DRAIN_STEPS};
        }
        return t;
    }
    const int rounds = (tiles + units - tiles - 1) / (units - tiles);
    if (rounds > TAIL_ROUNDS) return t;
    const int kb = static_cast<int>((rounds * (num_kb + DRAIN_STEPS) - DRAIN_STEPS) / (rounds + 1) + 0.999);
    if (kb < num_kb && num_kb - kb >= 4) t = {1, kb, std::max(kb + DRAIN_STEPS, rounds * (num_kb - kb + DRAIN_STEPS))};
    return t;
}
static Tiling choose_tiling(const RbGemmArgs& a) {
    // The pair kernel (256 x 256 tile over two SMs) serves every GEMM with enough work to fill the GPU:
    // enough tiles, or few tiles and a long K that is split (weight gradients); the gather prologue and the
    // scatter epilogue are the same code in both variants.  Small problems stay on the single-CTA kernel.
    const bool accum32 = a.out_dtype == 1 && a.flags == RB_GEMM_ACCUM;
    Tiling t;
    t.pair = a.rows_ctl || (pair_enabled() && (a.ag_nranks <= 1 || pair_gather_enabled()));
    if (t.pair && !a.rows_ctl) {
        const long long pt = ((a.M + 2 * BM - 1) / (2 * BM)) * ((a.N + 255) / 256) * a.batch;
        const long long kbs = (a.K + BK - 1) / BK;
        if (pt < num_sms() / 2 && !(accum32 && a.M > BM && pt * (kbs / 4) >= num_sms() / 2)) t.pair = false;
    }
    t.m_blocks = static_cast<int>(t.pair ? (a.M + 2 * BM - 1) / (2 * BM) : (a.M + BM - 1) / BM);
    const int num_kb = static_cast<int>((a.K + BK - 1) / BK);
    const int units = t.pair ? num_sms() / 2 : num_sms();   // CTAs (or CTA pairs) that run at once
    // Few output tiles and a long K (weight gradients): split K over CTAs and accumulate with
    // reductions.  Only for fp32 outputs that accumulate and have no other epilogue work.
    auto split_for = [&](int tiles) {
        int split = 1;
        if (accum32 && tiles < units && num_kb >= 8) {
            double best = 0.0;
            for (int s = 1; s <= 32 && s * 4 <= num_kb; ++s) {
                const int work = tiles * s;
                const int waves = (work + units - 1) / units;
                const double eff = static_cast<double>(work) / (waves * units) - 0.005 * s;
                if (eff > best + 1e-9) {
                    best = eff;
                    split = s;
                }
            }
        }
        return split;
    };
    t.tn = 256;
    if (!t.pair && a.ag_nranks <= 1 && a.rs_nranks <= 1) {
        if (a.tile_n == 64 || a.tile_n == 128 || a.tile_n == 256) {
            t.tn = a.tile_n;
        } else {
            // Narrow tiles move more bytes per product but keep more SMs busy.  Estimated cycles: k steps one CTA
            // does, each bound by its loads (48 / 32 / 24 KiB), plus the last tile's epilogue.  Measured with 256 /
            // 128 / 64 columns (us): 32 x 1024 x 1024 8.8 / 6.8 / 6.5; 351 x 3072 x 768 8.7 / 7.0 / 6.7;
            // 1182 x 768 x 3072 18.9 / 14.9 / 14.1; 2000 x 1024 x 1024 10.2 / 8.1 / 11.1;
            // 1182 x 2304 x 768 9.2 / 10.1 / 12.2.  The rule took the best or one within 3 % in 87 of 89 shapes (8 and 32 x
            // 4096 x 1024: 128 columns are 0.2 to 1 us faster than the 64 it takes).
            double best = 1e30;
            for (int w : {256, 128, 64}) {
                const int tiles = t.m_blocks * static_cast<int>((a.N + w - 1) / w * a.batch);
                const int s = split_for(tiles);
                const double steps = static_cast<double>((tiles * s + units - 1) / units) * ((num_kb + s - 1) / s);
                const double cost = steps * (w == 256 ? 768 : (w == 128 ? 512 : 384)) + 12.0 * w;
                if (cost < 0.98 * best) {
                    best = cost;
                    t.tn = w;
                }
            }
        }
    }
    t.n_blocks = static_cast<int>((a.N + t.tn - 1) / t.tn);
    const int tiles = t.m_blocks * t.n_blocks * static_cast<int>(a.batch);
    t.split = a.rows_ctl && a.rows_mode == RB_GEMM_ROWS_K ? 1 : split_for(tiles);   // (K is known on the device alone)
    t.tail_tiles = t.tail_split = t.tail_kb = 0;
    const int left = tiles % units;
    if (accum32 && t.pair && tiles > units && a.rs_nranks <= 1 && a.ag_nranks <= 1 && !a.in_order &&
        (num_kb >= TAIL_STEPS || (num_kb >= 8 && tiles < 2 * units && 3 * left <= units))) {
        const Tail tail = choose_tail(left, units, num_kb);
        // what the last wave takes less has to be worth it over all of them
        if (tail.split > 0 && num_kb + DRAIN_STEPS - tail.cost > 0.01 * (tiles / units + 1) * num_kb) {
            t.tail_tiles = left;
            t.tail_split = tail.split;
            t.tail_kb = tail.kb;
        }
    }
    return t;
}

}  // namespace rb

extern "C" int rb_gemm(const RbGemmArgs* a, void* stream_) {
    using namespace rb;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (a->M <= 0 || a->N <= 0 || a->batch <= 0) return 0;
    if (a->K <= 0) {
        // a sum of nothing (the weight gradient of an empty batch) is zero; no caller has an epilogue for it
        if (a->flags == RB_GEMM_ACCUM) return 0;
        if (a->flags || a->map_hp > 0) return -9;
        const size_t es = a->out_dtype == 1 ? 4 : 2;
        for (int64_t b = 0; b < a->batch; ++b)
            if (cudaMemset2DAsync(static_cast<char*>(a->D) + b * a->strideD * es, a->ldd * es, 0, a->N * es, a->M,
                                  stream) != cudaSuccess)
                return -4;
        return 0;
    }
    // TMA needs 16-byte aligned bases and row strides
    if ((reinterpret_cast<uintptr_t>(a->A) & 15) || (reinterpret_cast<uintptr_t>(a->B) & 15) ||
        (a->lda % 8) || (a->ldb % 8) || (a->batch > 1 && ((a->strideA % 8) || (a->strideB % 8))))
        return -2;
    GemmKernelParams p;
    p.M = static_cast<int>(a->M);
    p.N = static_cast<int>(a->N);
    p.K = static_cast<int>(a->K);
    p.batch = static_cast<int>(a->batch);
    p.a_major = a->a_major;
    p.b_major = a->b_major;
    const Tiling tiling = choose_tiling(*a);
    const bool pair = tiling.pair;
    const int tn = tiling.tn;
    p.num_m_blocks = tiling.m_blocks;
    p.num_kb = (p.K + BK - 1) / BK;
    p.num_n_blocks = tiling.n_blocks;
    p.base_tiles = p.num_m_blocks * p.num_n_blocks * p.batch;
    p.ag_nranks = a->ag_nranks > 1 ? a->ag_nranks : 0;
    p.ag_my_idx = a->ag_my_idx;
    p.ag_rows = a->ag_rows;
    p.ag_cols = a->ag_cols;
    p.ag_dst = const_cast<void*>(a->B);
    p.ag_flags = static_cast<unsigned int*>(a->ag_flags);
    for (int r = 0; r < 8; ++r) p.ag_src[r] = a->ag_nranks > 1 ? a->ag_src[r] : nullptr;
    if (p.ag_nranks > 1) {
        // shards are column blocks of the stored B matrix: [rows, ag_cols] each, ag_cols a multiple of the tile
        const long long stored_cols = a->b_major == 0 ? a->K : a->N;
        if (a->ag_nranks > 8 || a->batch != 1 || !a->ag_flags || a->ag_cols % 256 ||
            static_cast<long long>(a->ag_cols) * a->ag_nranks != stored_cols || a->ldb != stored_cols)
            return -6;
        cudaMemsetAsync(a->ag_flags, 0, 8 * sizeof(unsigned int), stream);
    }
    p.split_k = 1;
    p.rs_nranks = a->rs_nranks > 1 ? a->rs_nranks : 0;
    p.rs_cols = a->rs_nranks > 1 ? static_cast<int>(a->N / a->rs_nranks) : 0;
    for (int r = 0; r < 8; ++r) p.rs_peer[r] = a->rs_nranks > 1 ? a->rs_peer[r] : nullptr;
    if (p.rs_nranks > 1 && (a->out_dtype != 1 || a->flags != RB_GEMM_ACCUM || a->N % a->rs_nranks || p.rs_cols % 32 ||
                            a->rs_nranks > 8 || a->batch != 1))
        return -5;
    p.split_k = tiling.split;
    p.kb_per_split = (p.num_kb + p.split_k - 1) / p.split_k;
    p.split_k = (p.num_kb + p.kb_per_split - 1) / p.kb_per_split;
    p.num_tiles = p.base_tiles * p.split_k;
    p.tail_tiles = tiling.tail_tiles;
    p.tail_first = p.base_tiles - tiling.tail_tiles;
    p.tail_split = tiling.tail_split;
    p.tail_kb = tiling.tail_kb;
    p.tail_units = num_sms() / 2;
    p.partial = p.split_k > 1 || p.tail_tiles > 0;
    if (p.tail_tiles > 0) {
        const int helpers = p.tail_units - p.tail_tiles;
        p.num_tiles = p.tail_first + (p.tail_split > 1 ? p.tail_tiles * p.tail_split
                                                       : p.tail_units * ((p.tail_tiles + helpers - 1) / helpers));
    }
    p.D = a->D;
    p.bias = a->bias;
    p.residual = a->residual;
    p.aux_in = a->aux_in;
    p.aux_out = a->aux_out;
    p.ldd = a->ldd;
    p.strideD = a->strideD;
    p.alpha = a->alpha;
    p.flags = a->flags;
    p.err = error_word_ptr();
    if (!p.err) return -3;
    p.conv_kb_per_tap = 0;
    p.conv_b_tap_cols = 0;
    p.map_hp = a->map_hp;
    p.map_wp = a->map_wp;
    p.map_h = a->map_h;
    p.map_w = a->map_w;
    p.map_pad = a->map_pad;
    for (int t = 0; t < 49; ++t) p.conv_shift[t] = 0;
    if (a->conv_taps > 0) {
        // A must be K-major with conv_c (a multiple of the k step) columns; no batch, gather or scatter
        if (a->conv_taps > 49 || a->a_major != 0 || a->conv_c % BK || a->lda != a->conv_c || a->batch != 1 ||
            a->K != static_cast<int64_t>(a->conv_taps) * a->conv_c || a->ag_nranks > 1 || a->rs_nranks > 1 ||
            (a->b_major != 0 && a->conv_b_tap_cols % 8))
            return -7;
        p.conv_kb_per_tap = a->conv_c / BK;
        p.conv_b_tap_cols = a->conv_b_tap_cols;
        for (int t = 0; t < a->conv_taps; ++t) p.conv_shift[t] = a->conv_shift[t];
    }
    p.a_colsum = a->a_colsum;
    p.rows_ctl = a->rows_ctl;
    p.rows_mode = a->rows_mode;
    p.rows_out = a->rows_out;
    const bool rows_m = a->rows_ctl && a->rows_mode == RB_GEMM_ROWS_M;
    if (a->rows_ctl) {
        // plain products of one matrix; what is gathered along K is cut into whole tiles
        if (a->batch != 1 || a->ag_nranks > 1 || a->rs_nranks > 1 || a->conv_taps > 0 || a->wgrad_taps > 0 || a->map_hp > 0 ||
            (a->flags & ~RB_GEMM_ACCUM) || a->rows_mode < RB_GEMM_ROWS_ALL || a->rows_mode > RB_GEMM_ROWS_M ||
            (rows_m && (a->a_major != 0 || a->out_dtype != 1 || a->flags || a->rows_out % 256 || a->rows_out < a->M)))
            return -10;
    }
    if (a->a_colsum && (a->a_major != 1 || a->batch != 1 || a->ag_nranks > 1)) return -8;
    p.wgrad_taps = 0;
    p.wgrad_cols = 1;
    if (a->wgrad_taps > 0) {
        // a 64-column block of B must lie within one tap
        if (a->wgrad_taps > 49 || a->conv_taps > 0 || a->b_major != 1 || a->conv_c % 64 || a->conv_c <= 0 ||
            a->N != static_cast<int64_t>(a->wgrad_taps) * a->conv_c || a->batch != 1 ||
            a->ag_nranks > 1 || a->rs_nranks > 1)
            return -7;
        p.wgrad_taps = a->wgrad_taps;
        p.wgrad_cols = a->conv_c;
        for (int t = 0; t < a->wgrad_taps; ++t) p.conv_shift[t] = a->conv_shift[t];
    }
    if (a->map_hp > 0 && (a->batch != 1 || a->rs_nranks > 1 || a->map_wp <= 0)) return -7;

    p.bias_al = !off16(a->bias);
    p.in_al = !off16(a->residual, a->aux_in, a->aux_out) && a->ldd % 8 == 0 && (a->batch == 1 || a->strideD % 8 == 0);
    const int64_t per16 = a->out_dtype == 1 ? 4 : 8;
    p.out_al = !off16(a->D) && a->ldd % per16 == 0 && (a->batch == 1 || a->strideD % per16 == 0);
    for (int r = 0; r < p.rs_nranks; ++r) p.out_al = p.out_al && !off16(a->rs_peer[r]);

    CUtensorMap tmA, tmB;
    int rc;
    const uint64_t sA = a->batch > 1 ? a->strideA * 2 : (a->a_major == 0 ? a->M : a->K) * a->lda * 2;
    const uint64_t sB = a->batch > 1 ? a->strideB * 2 : (a->b_major == 0 ? a->N : a->K) * a->ldb * 2;
    // An MN-major operand of whole 64-column chunks is seen as [chunk][row][64], so that one copy brings all chunks of a
    // stage.  The copies are issued one by one, and with two or four per operand and stage it was their number, not
    // the bytes, that kept the tensor core waiting (4096 x 1024 x 32768: its pipe 69 % active that way and 73 % now,
    // 210 -> 190 us): 8192 x 4096 x 8192, both operands MN-major, 421 -> 391 us, with fp32 accumulation 434 -> 402 us;
    // 1024 x 9216 x 26912 445 -> 366 us.  A last chunk that the matrix fills only in part would read past its rows, and
    // column blocks that straddle filter taps need a shift each: those keep a copy per chunk.
    const int b_cols = pair ? 128 : tn;   // columns of B one CTA loads
    p.a_merged = a->a_major == 1 && a->M % 64 == 0;
    p.b_merged = a->b_major == 1 && (a->conv_taps > 0    ? a->conv_b_tap_cols % 64 == 0
                                     : a->wgrad_taps > 0 ? a->conv_c % b_cols == 0
                                                         : a->N % 64 == 0);
    if (a->conv_taps > 0)
        rc = make_tmap_4d(&tmA, a->A, a->in_dtype, a->conv_c, a->M, 1, 1, a->lda * 2, sA, sA, BK, BM);
    else if (a->a_major == 0)
        rc = make_tmap_4d(&tmA, a->A, a->in_dtype, a->K, a->M, 1, a->batch, a->lda * 2, sA, sA, BK, BM);
    else if (p.a_merged)
        rc = make_tmap_chunks(&tmA, a->A, a->in_dtype, a->K, a->M / 64, a->batch, a->lda * 2, sA, BM / 64);
    else
        rc = make_tmap_4d(&tmA, a->A, a->in_dtype, a->M, a->K, 1, a->batch, a->lda * 2, sA, sA, 64, BK);
    if (rc) return rc;
    // stored columns of an MN-major B: with filter taps [conv_c rows, conv_taps * conv_b_tap_cols] (tap t's block starts
    // at column t * conv_b_tap_cols), for a weight gradient the activation's conv_c
    const uint64_t stored = a->conv_taps > 0    ? static_cast<uint64_t>(a->conv_taps) * a->conv_b_tap_cols
                            : a->wgrad_taps > 0 ? a->conv_c
                                                : a->N;
    const uint64_t b_rows = a->conv_taps > 0 ? a->conv_c : a->K;
    const uint64_t sB1 = a->conv_taps > 0 ? static_cast<uint64_t>(a->conv_c) * a->ldb * 2 : sB;
    if (a->b_major == 0)
        rc = make_tmap_4d(&tmB, a->B, a->in_dtype, a->K, a->N, 1, a->batch, a->ldb * 2, sB, sB, BK, b_cols);
    else if (p.b_merged)
        rc = make_tmap_chunks(&tmB, a->B, a->in_dtype, b_rows, stored / 64, a->batch, a->ldb * 2, sB1, b_cols / 64);
    else
        rc = make_tmap_4d(&tmB, a->B, a->in_dtype, stored, b_rows, 1, a->batch, a->ldb * 2, sB1, sB1, 64, BK);
    if (rc) return rc;

    // The staged epilogue wants outputs the copy engine can address: plain rows in this GPU's memory, 16-byte
    // aligned bases and row strides.  Its staging blocks of an auxiliary matrix are 16-bit ones, so an fp32 output
    // with one, or an output that both reads and writes an auxiliary matrix, stays on the direct path, as do mapped
    // rows (padded image grids) and peers' buffers (reduce-scatter).
    CUtensorMap tmD = tmA, tmAux = tmA;
    const bool fp32_out = a->out_dtype == 1;
    const int64_t out_es = fp32_out ? 4 : 2;
    const bool aux_w = a->flags & RB_GEMM_AUX_OUT, aux_r = a->flags & RB_GEMM_DGELU;
    const void* aux = aux_w ? a->aux_out : a->aux_in;
    auto addressable = [&](const void* ptr, int64_t es) {
        return !(reinterpret_cast<uintptr_t>(ptr) & 15) && (a->ldd * es) % 16 == 0 && a->ldd >= a->N &&
               (a->batch == 1 || (a->strideD > 0 && (a->strideD * es) % 16 == 0));
    };
    p.staged = a->map_hp <= 0 && p.rs_nranks <= 1 && addressable(a->D, out_es) && !(aux_w && aux_r) &&
               !(fp32_out && (aux_w || aux_r)) && (!(aux_w || aux_r) || addressable(aux, 2));
    if (p.staged) {
        const int64_t sd = a->batch > 1 ? a->strideD : a->M * a->ldd;
        rc = make_tmap_block32(&tmD, a->D, fp32_out, a->in_dtype, a->N, rows_m ? a->rows_out : a->M, a->batch, a->ldd * out_es,
                               (rows_m ? a->rows_out * a->ldd : sd) * out_es);
        if (!rc && (aux_w || aux_r))
            rc = make_tmap_block32(&tmAux, aux, false, a->in_dtype, a->N, a->M, a->batch, a->ldd * 2, sd * 2);
        if (rc) p.staged = 0;
    }
    if (rows_m && !p.staged) return -10;   // (only the staged epilogue keeps the parts apart)

    return a->in_dtype == 1 ? dispatch<__nv_bfloat16>(*a, pair, tn, tmA, tmB, tmD, tmAux, p, stream)
                            : dispatch<__half>(*a, pair, tn, tmA, tmB, tmD, tmAux, p, stream);
}

// Parts that the K dimension of an fp32 [M, N] += product is split into: 1 when its tiles fill the GPU by themselves
extern "C" int rb_gemm_splits(long long M, long long N, long long K) {
    RbGemmArgs a = {};
    a.M = M, a.N = N, a.K = K, a.batch = 1;
    a.out_dtype = 1;
    a.flags = RB_GEMM_ACCUM;
    return M > 0 && N > 0 && K > 0 ? rb::choose_tiling(a).split : 1;
}

// Pairs of SMs that work on 256 x 256 tiles at once (0: pairs are switched off)
extern "C" int rb_gemm_pairs() { return rb::pair_enabled() ? rb::num_sms() / 2 : 0; }

// How the last wave of tiles of an fp32 [M, N] += product is summed: 0 whole tiles, 1 the first part of K by the tiles' own
// pairs of SMs and the rest by the pairs left over, n > 1: K in n parts
extern "C" int rb_gemm_last_wave(long long M, long long N, long long K, int in_order) {
    RbGemmArgs a = {};
    a.M = M, a.N = N, a.K = K, a.batch = 1;
    a.out_dtype = 1;
    a.flags = RB_GEMM_ACCUM;
    a.in_order = in_order;
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    const rb::Tiling t = rb::choose_tiling(a);
    return t.tail_tiles > 0 ? t.tail_split : 0;
}

// Copies the device error word into `host_dst` (pinned host memory) on `stream` without waiting: the caller
// reads the value once work enqueued before the copy has finished (an event, or the next synchronisation).
extern "C" int rb_error_peek_async(int* host_dst, void* stream) {
    int* p = rb::error_word_ptr();
    if (!p || !host_dst) return -3;
    return cudaMemcpyAsync(host_dst, p, sizeof(int), cudaMemcpyDeviceToHost, static_cast<cudaStream_t>(stream)) ==
                   cudaSuccess
               ? 0
               : -4;
}

// Reads (and clears) the device error word.  Synchronises the device.
extern "C" int rb_read_error(int clear) {
    int* p = rb::error_word_ptr();
    if (!p) return -3;
    int v = 0;
    if (cudaMemcpy(&v, p, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -4;
    if (clear && v) {
        int z = 0;
        cudaMemcpy(p, &z, sizeof(int), cudaMemcpyHostToDevice);
    }
    return v;
}
