// Fused multi-head attention backward on tcgen05 tensor cores (head dim 64).
//
// One CTA per SM walks a list of items, 128 keys of one (batch, head) each, and sweeps the query blocks of an item.  Per
// query block i it recomputes, with the keys on the TMEM lanes,
//     St  = K_j Q_i^T          dPt = V_j dO_i^T                (TMEM, 2 x 128 cols)
//     Pt  = exp(St*scale + bias - lse_i)      dSt = Pt * (dPt - delta_i)
// rounds both to 16 bits (four threads per key row) and feeds them back to the tensor core:
//     dK_j += dSt Q_i         dV_j += Pt  dO_i                 (TMEM accumulators)
//     dQ_i  = dSt^T K_j  -- the same dSt tile read as an MN-major A operand --
// dSt goes through swizzled shared memory (dQ wants it transposed); Pt returns to tensor memory, from where the
// tensor core takes it as its A operand: 64 KiB a step less on shared memory, which products, tiles and staging
// kept busy for two thirds of the time.  dQ_i is drained from TMEM into a swizzled fp32 staging tile and added to
// an fp32 scratch buffer by ONE bulk tensor reduction per half tile (the copy
// engine does the read-modify-write; the math threads do not wait for it); a
// last kernel converts the scratch to the 16-bit dQ.  (A sequence of one key block has nothing to add up: its dQ is
// rounded and stored at once.)  dK and dV leave by way of the same staging tile.  Q_i / dO_i stream through a 3-stage TMA
// ring.  Warps 0..15 = element math, warp 16 = loads and the S / dP products, warp 17 = the products with dSt and Pt,
// warps 18..21 = dQ, dK and dV drain, and the row statistics (lse, delta, dropout hash) of the blocks to come: the math
// warps' chain per query block is only "S / dP -> P / dS", without a barrier among them, and the drain of block i runs
// beside the math of block i + 1.  Of a block's products those that read dSt come first, so that its tile is free again
// before the next block's is ready.
//
// Every role runs on from item to item: blocks are counted over all items (barrier phases, ring stages, statistics), the
// next item's K and V are loaded while the last block is in work, its first S / dP stand ready when the math warps come, and
// dK and dV are drained beside its first block.  A CTA that did one item spent 7200 of 21200 cycles (S = 512) before its
// first product and behind its last, and 1800 until the next one began; now an item takes 15000, 3500 a block: two reads and
// some sixteen instructions an element of the math warps, and the barriers between them and the products.
//
// With the delta and conversion passes (us): 32 x 512 x 16 heads with bias and dropout 278 -> 227 with converged issuing
// warps (one thread's issuing of 32 products a step had bounded it), 220 -> 168 with items; 64 x 128 x 16 74 -> 51; 8 x 1024
// x 16 165 -> 136; 4 x 2048 x 16 without dropout 234 -> 220 to 232.  With no more items than SMs nothing overlaps, and what
// an item needs beside its products costs a little (6 x 197 x 12: 13.9 -> 14.8).
//
// Takes the place of the autograd graph the reference runs for the traced
// attention chain (src/torch/TorchDriver.cpp:642-847).
#include "attn.h"
#include "attn_common.cuh"
#include "launch.cuh"
#include "tc_common.cuh"

namespace rb {

constexpr int BQ = 128, BKEYS = 128;
constexpr int TILE = 128 * 64 * 2;       // 16 KiB
constexpr int SQ_BYTES = 128 * 128 * 2;  // 32 KiB
constexpr int BWD_MATH = 512;                  // warps 0..15: four threads per key row
constexpr int BWD_DRAIN = 128;                 // warps 18..21: move dQ, dK and dV out of tensor memory
constexpr int LOAD_WARP = BWD_MATH / 32, GRAD_WARP = LOAD_WARP + 1;
constexpr int BWD_THREADS = BWD_MATH + 64 + BWD_DRAIN;
constexpr int BWD_TMEM_COLS = 512;
constexpr int C_ST = 0, C_DPT = 128, C_DV = 256, C_DK = 320, C_DQ = 384, C_P = 448;   // P: 128 16-bit columns
constexpr int DQ_STAGE = 128 * 64 * 4;   // 32 KiB: [2 column halves][128 rows x 128 B]
constexpr int QD_STAGES = 3;             // Q / dO ring: block i + 2 is loaded while blocks i and i + 1 are in use
constexpr int STATS = 3 * 128;           // (lse, delta, row hash) of a query block
// K x 2, V + (Q, dO) x 3 stages + dSt + dQ staging + row statistics of two blocks + barriers
constexpr int BWD_SMEM = 3 * TILE + 2 * QD_STAGES * TILE + SQ_BYTES + DQ_STAGE + 2 * STATS * 4 + 256;

struct AttnBwdParams {
    int B, H, S;
    float scale, scale_log2;
    const float* key_bias;
    const float* lse;
    const float* delta;
    float* dq_accum;  // [B, S, H, 64] fp32
    uint32_t thr32;   // keep an element when its 32-bit hash >= thr32 (0: no dropout)
    float inv_keep;
    uint32_t seed;
    // walking the items (see Item): how far apart a CTA's are, and 2^32 / (key blocks, heads), rounded up (0: one)
    int step_kb, step_h, step_b;
    uint32_t inv_nq, inv_h;
    int* err;
};

// DQ16 (one key block): its product is all of dQ, which is rounded and stored at once
template <typename T, bool DQ16>
__global__ void __launch_bounds__(BWD_THREADS, 1)
    attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                    const __grid_constant__ CUtensorMap tmDQ, const __grid_constant__ CUtensorMap tmDK,
                    const __grid_constant__ CUtensorMap tmDV, const AttnBwdParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sK = smem;                                // [2]: the next item's comes beside this one's, which dQ reads to the end
    uint8_t* sV = smem + 2 * TILE;
    uint8_t* sQ = smem + 3 * TILE;                     // [QD_STAGES]
    uint8_t* sdO = smem + (3 + QD_STAGES) * TILE;      // [QD_STAGES]
    uint8_t* sdSt = smem + (3 + 2 * QD_STAGES) * TILE;
    uint8_t* sDQ = sdSt + SQ_BYTES;
    float* s_stats = reinterpret_cast<float*>(sDQ + DQ_STAGE);   // [2][-lse, -delta, row hash][128]
    uint64_t* bars = reinterpret_cast<uint64_t*>(s_stats + 2 * STATS);
    uint64_t* kv_full = bars;
    uint64_t* qd_full = bars + 1;     // [QD_STAGES]
    uint64_t* s_full = bars + 4;
    uint64_t* s_free = bars + 5;
    uint64_t* pds_ready = bars + 6;
    uint64_t* ds_done = bars + 7;     // dK and dQ of the step are done: dSt may be overwritten, dQ drained
    uint64_t* p_done = bars + 8;      // ... and dV: Pt may be
    uint64_t* dq_free = bars + 9;     // the previous bulk reduction has read the staging tile
    uint64_t* dq_ready = bars + 10;   // every drain thread has written its part of the staging tile
    uint64_t* dq_taken = bars + 11;   // dQ of the last step is out of tensor memory: the next may overwrite it
    uint64_t* stats_full = bars + 12;   // [2]
    // [QD_STAGES] every product that reads the stage is done: it may be loaded again.  A barrier per stage, whose next phase
    // cannot end before that load: p_done may be two blocks further by the time the loading warp looks, and a wait for a
    // phase's parity would then wait for the block after, whose products wait for the loading warp.
    uint64_t* qd_free = bars + 14;
    uint64_t* dkv_taken = bars + 14 + QD_STAGES;   // dK and dV of the last item are out of tensor memory
    uint64_t* k_free = bars + 15 + QD_STAGES;      // [2] every product that reads the K buffer is done
    uint64_t* dkv_free = bars + 17 + QD_STAGES;    // the last dQ reduction has read the staging tile: dK and dV go there
    uint64_t* dkv_ready = bars + 18 + QD_STAGES;   // every drain thread has written its rows of them
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 19 + QD_STAGES);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    // (the same for all lanes, for the compiler too: what the issuing warps compute from it stays in uniform registers)
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int nq = (p.S + BQ - 1) / BQ;   // query blocks, and key blocks
    const int nitems = nq * p.H * p.B;
    // An item: 128 keys of one (batch, head).  The CTA's items lie gridDim.x apart; what that is in key blocks, heads and
    // batch rows the host has worked out: a role that divided for every item would pay some 500 cycles, and the first loads
    // would wait for it.  (A block's index is below 2^16, so the products with the rounded-up inverses are exact.)
    struct Item {
        int at, kb, h, b;
    };
    auto first_item = [&] {
        const int at = blockIdx.x, bh = p.inv_nq ? __umulhi(at, p.inv_nq) : at, b = p.inv_h ? __umulhi(bh, p.inv_h) : bh;
        return Item{at, at - bh * nq, bh - b * p.H, b};
    };
    auto advance = [&](Item& x) {
        x.at += gridDim.x;
        x.kb += p.step_kb;
        x.h += p.step_h;
        x.b += p.step_b;
        if (x.kb >= nq) x.kb -= nq, ++x.h;
        if (x.h >= p.H) x.h -= p.H, ++x.b;
    };
    // query block j of an item, where j may lie in one of the CTA's items to come: false if there is none
    auto reach = [&](Item& x, int& j) {
        while (j >= nq) {
            j -= nq;
            advance(x);
        }
        return x.at < nitems;
    };

    if (threadIdx.x == 0) {
        mbar_init(kv_full, 1);
        for (int st = 0; st < QD_STAGES; ++st) {
            mbar_init(&qd_full[st], 1);
            mbar_init(&qd_free[st], 1);
        }
        mbar_init(s_full, 1);
        mbar_init(s_free, BWD_MATH);
        mbar_init(pds_ready, BWD_MATH);
        mbar_init(ds_done, 1);
        mbar_init(p_done, 1);
        mbar_init(dq_free, 1);
        mbar_init(dq_ready, BWD_DRAIN);
        mbar_init(dq_taken, BWD_DRAIN);
        mbar_init(dkv_taken, BWD_DRAIN);
        mbar_init(dkv_free, 1);
        mbar_init(dkv_ready, BWD_DRAIN);
        for (int u = 0; u < 2; ++u) {
            mbar_init(&stats_full[u], BWD_DRAIN);
            mbar_init(&k_free[u], 1);
        }
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == GRAD_WARP && lane < 7)
        tma_prefetch_desc(lane == 0 ? &tmK : lane == 1 ? &tmV : lane == 2 ? &tmQ : lane == 3 ? &tmdO : lane == 4 ? &tmDQ
                                         : lane == 5 ? &tmDK : &tmDV);
    if (warp == LOAD_WARP) {
        tmem_alloc(tmem_slot, BWD_TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    grid_trigger();
    grid_wait();   // all of the above runs beside the end of the kernel before
    constexpr int fmt = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;

    if (warp == LOAD_WARP) {
        // ------------- loads, and the S / dP products -------------
        // The whole warp goes through the loop and one lane's predicate lets the instructions through: a branch for that
        // lane would keep descriptors out of the uniform registers, and eight products then take 600 cycles to issue, not
        // 350 -- more with the math warps beside it.
        const uint32_t el = elect_one();
        const uint32_t id_s = make_idesc_f16(fmt, 0, 0, 128, 128);
        const uint32_t k_desc = desc_lo_sw128(smem_u32(sK), 16), v_desc = desc_lo_sw128(smem_u32(sV), 16);
        const uint32_t q_desc = desc_lo_sw128(smem_u32(sQ), 16), do_desc = desc_lo_sw128(smem_u32(sdO), 16);
        Item item = first_item();
        auto load_qd = [&](int j, int st) {
            Item x = item;
            if (!reach(x, j)) return;
            if (el) {
                mbar_arrive_expect_tx(&qd_full[st], 2 * TILE);
                tma_load_4d(sQ + st * TILE, &tmQ, &qd_full[st], 0, j * BQ, x.h, x.b);
                tma_load_4d(sdO + st * TILE, &tmdO, &qd_full[st], 0, j * BQ, x.h, x.b);
            }
        };
        auto more = [&](int j) {
            Item x = item;
            return reach(x, j);
        };
        bool ok = true;
        int st = 0, next = 2;   // stage of a block, and of the block after the next (which the block before was in)
        uint32_t phase = 0, free_phase = 1;   // (of the block before: it is 0 from block 1 on)
        int c = 0;                            // blocks so far, over all items
        auto load_kv = [&](const Item& x, int buf) {
            if (el) {
                mbar_arrive_expect_tx(kv_full, 2 * TILE);
                tma_load_4d(sK + buf * TILE, &tmK, kv_full, 0, x.kb * BKEYS, x.h, x.b);
                tma_load_4d(sV, &tmV, kv_full, 0, x.kb * BKEYS, x.h, x.b);
            }
        };
        if (item.at < nitems) {
            load_kv(item, 0);
            for (int j = 0; j < QD_STAGES; ++j) load_qd(j, j);
        }
        for (int k = 0; item.at < nitems && ok; advance(item), ++k) {
            const uint32_t kd = k_desc + (k & 1) * (TILE / 16);
            ok = mbar_wait_warp(kv_full, k & 1, abort_flag);
            for (int i = 0; i < nq && ok; ++i, ++c) {
                // S / dP of a block go to the tensor core as soon as the math warps have read the last block's: they run
                // behind that block's products, while its math is busy
                ok = mbar_wait_warp(&qd_full[st], phase, abort_flag) && (c == 0 || mbar_wait_warp(s_free, (c - 1) & 1, abort_flag));
                if (!ok) break;
                tc_fence_after();
                const uint32_t qa = q_desc + st * (TILE / 16), da = do_desc + st * (TILE / 16);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
                    umma_f16_lo(tmem + C_ST, kd + kk * 2, qa + kk * 2, id_s, kk != 0, el);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
                    umma_f16_lo(tmem + C_DPT, v_desc + kk * 2, da + kk * 2, id_s, kk != 0, el);
                if (el) umma_commit(s_full);
                // the stage the block before used is free once its products are done: the block after the next goes there
                // (in an item's last block behind the next item's K and V)
                if (i + 1 < nq) {
                    if (c >= 1 && more(i + 2)) {
                        ok = mbar_wait_warp(&qd_free[next], free_phase, abort_flag);
                        if (!ok) break;
                        load_qd(i + 2, next);
                    }
                    if (++next == QD_STAGES) {
                        next = 0;
                        free_phase ^= 1;
                    }
                }
                if (++st == QD_STAGES) {
                    st = 0;
                    phase ^= 1;
                }
            }
            // The next item's K and V, while this one's last block is in work: V's place is free with the last dP, K's other
            // buffer with the products of the item before.  (Loaded behind the last product that reads K, 4200 cycles passed
            // from there to the next item's first S, of 19000 an item at S = 512.)
            Item x = item;
            advance(x);
            if (ok && x.at < nitems) {
                ok = mbar_wait_warp(s_full, (c - 1) & 1, abort_flag) &&
                     (k == 0 || mbar_wait_warp(&k_free[(k + 1) & 1], ((k - 1) >> 1) & 1, abort_flag));
                if (!ok) break;
                load_kv(x, (k + 1) & 1);
            }
            if (ok && c >= 2 && more(nq + 1)) {
                ok = mbar_wait_warp(&qd_free[next], free_phase, abort_flag);
                if (!ok) break;
                load_qd(nq + 1, next);
            }
            if (++next == QD_STAGES) {
                next = 0;
                free_phase ^= 1;
            }
        }
    } else if (warp == GRAD_WARP) {
        // ------------- the products with dSt and Pt.  A warp of its own: one that issued all products took 4400 cycles
        // a step, between the math warps that share its scheduler, and S / dP queued behind them -------------
        const uint32_t el = elect_one();
        const uint32_t id_kn = make_idesc_f16(fmt, 0, 1, 128, 64);  // A K-major, B MN-major
        const uint32_t id_nn = make_idesc_f16(fmt, 1, 1, 128, 64);  // A MN-major, B MN-major
        const uint32_t ds_k = desc_lo_sw128(smem_u32(sdSt), 16), ds_n = desc_lo_sw128(smem_u32(sdSt), SQ_BYTES / 2);
        const uint32_t k_desc = desc_lo_sw128(smem_u32(sK), 8192);
        const uint32_t q_desc = desc_lo_sw128(smem_u32(sQ), 8192), do_desc = desc_lo_sw128(smem_u32(sdO), 8192);
        int st = 0, c = 0;
        uint32_t phase = 0;
        bool ok = true;
        Item item = first_item();
        for (int k = 0; item.at < nitems && ok; advance(item), ++k) {
            // dK and dV of the last item must have left tensor memory
            if (k > 0 && !mbar_wait_warp(dkv_taken, (k - 1) & 1, abort_flag)) break;
            const uint32_t kd = k_desc + (k & 1) * (TILE / 16);
            for (int i = 0; i < nq; ++i, ++c) {
                ok = mbar_wait_warp(&qd_full[st], phase, abort_flag) && mbar_wait_warp(pds_ready, c & 1, abort_flag);
                if (!ok) break;
                tc_fence_after();
                const uint32_t qa = q_desc + st * (TILE / 16), da = do_desc + st * (TILE / 16);
#pragma unroll
                for (int x = 0; x < 8; ++x)
                    umma_f16_lo(tmem + C_DK, ds_k + (x >> 2) * (SQ_BYTES / 32) + (x & 3) * 2, qa + x * 128, id_kn,
                                (i | x) != 0, el);
                // dQ of the previous step must have left tensor memory before this step's product replaces it
                if (c > 0) {
                    ok = mbar_wait_warp(dq_taken, (c - 1) & 1, abort_flag);
                    if (!ok) break;
                    tc_fence_after();
                }
#pragma unroll
                for (int x = 0; x < 8; ++x)
                    umma_f16_lo(tmem + C_DQ, ds_n + x * 128, kd + x * 128, id_nn, x != 0, el);
                if (el) umma_commit(ds_done);
#pragma unroll
                for (int x = 0; x < 8; ++x)
                    umma_f16_ts_lo(tmem + C_DV, tmem + C_P + x * 8, da + x * 128, id_kn, (i | x) != 0, el);
                Item x = item;
                int ahead = i + QD_STAGES;
                const bool reload = reach(x, ahead);
                if (el) {
                    if (reload) umma_commit(&qd_free[st]);   // (waited for, so it arrives while the block lives)
                    umma_commit(p_done);
                }
                if (++st == QD_STAGES) {
                    st = 0;
                    phase ^= 1;
                }
            }
            Item x = item;
            int ahead = 2 * nq;   // (waited for by the load of the item after the next)
            if (ok && reach(x, ahead) && el) umma_commit(&k_free[k & 1]);
        }
    } else if (warp > GRAD_WARP) {
        // ------------- drain: thread r owns query row r of dQ (TMEM lane r), and key row r of dK and dV -------------
        const int r = (warp & 3) * 32 + lane;
        const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
        const uint32_t sw = r & 7;
        const bool issuer = threadIdx.x == BWD_MATH + 64;
        // row statistics: thread t looks after row t of every query block, two buffers.  Both sums are negated (the
        // element-wise chain adds them); past the end of the sequence lse is +inf, and probabilities come out as
        // exp2(-inf) = 0.
        const int t = threadIdx.x - (BWD_MATH + 64);
        Item item = first_item();
        int first = 0;   // blocks of the items before
        float lse = 0.f, delta = 0.f;
        uint32_t hash = 0;
        auto fetch_stats = [&](int j) {   // (volatile: the loads are not sunk to their use.  Not the read-only path: the
                                          // kernel before this one writes delta, and may still run when this one is resident)
            Item x = item;
            if (!reach(x, j)) return false;
            const int q = j * BQ + t;
            lse = INFINITY;
            delta = 0.f;
            if (q < p.S) {
                const long long row = (static_cast<long long>(x.b) * p.H + x.h) * p.S + q;
                asm volatile("ld.global.f32 %0, [%1];" : "=f"(lse) : "l"(p.lse + row));
                asm volatile("ld.global.f32 %0, [%1];" : "=f"(delta) : "l"(p.delta + row));
            }
            hash = drop_row_hash(p.seed, x.b, x.h, q, p.H, p.S);
            return true;
        };
        auto put_stats = [&](int j) {
            const int buf = (first + j) & 1;
            float* s = s_stats + buf * STATS;
            s[t] = lse * -1.4426950408889634f;
            s[128 + t] = -delta;
            reinterpret_cast<uint32_t*>(s)[256 + t] = hash;
            mbar_arrive(&stats_full[buf]);
        };
        if (item.at < nitems)
            for (int j = 0; j < 2; ++j)
                if (fetch_stats(j)) put_stats(j);
        bool ok = true;
        for (int k = 0; item.at < nitems && ok; advance(item), first += nq, ++k) {
            for (int i = 0; i < nq; ++i) {
                const int c = first + i;
                const bool more = fetch_stats(i + 2);
                ok = mbar_wait_warp(ds_done, c & 1, abort_flag);
                if (!ok) break;
                tc_fence_after();
                uint32_t v0[32], v1[32];
                tmem_ld32(tmem + lane_addr + C_DQ, v0);
                tmem_ld32(tmem + lane_addr + C_DQ + 32, v1);
                tmem_ld_wait();
                tc_fence_before();
                mbar_arrive(dq_taken);
                // dSt of this step has been read, so it had been written: the math threads are past this step's statistics,
                // whose buffer is that of the block after the next
                if (more) put_stats(i + 2);
                if (issuer) {
                    tma_store_wait_read<0>();   // the previous reduction no longer reads the staging tile
                    mbar_arrive(dq_free);
                }
                ok = mbar_wait_warp(dq_free, c & 1, abort_flag);
                if (!ok) break;
                uint8_t* row = sDQ + (r >> 3) * 1024 + sw * 128;
                if constexpr (DQ16) {
#pragma unroll
                    for (int g = 0; g < 8; ++g) {
                        uint32_t w[4];
#pragma unroll
                        for (int x = 0; x < 4; ++x) {
                            const int at = (g & 3) * 8 + 2 * x;
                            w[x] = pack2<T>(__uint_as_float(g < 4 ? v0[at] : v1[at]) * p.scale,
                                            __uint_as_float(g < 4 ? v0[at + 1] : v1[at + 1]) * p.scale);
                        }
                        *reinterpret_cast<uint4*>(row + ((static_cast<uint32_t>(g) ^ sw) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                } else {
#pragma unroll
                    for (int g = 0; g < 8; ++g) {
                        const uint32_t off = (static_cast<uint32_t>(g) ^ sw) << 4;
                        *reinterpret_cast<float4*>(row + off) =
                            make_float4(__uint_as_float(v0[g * 4]) * p.scale, __uint_as_float(v0[g * 4 + 1]) * p.scale,
                                        __uint_as_float(v0[g * 4 + 2]) * p.scale, __uint_as_float(v0[g * 4 + 3]) * p.scale);
                        *reinterpret_cast<float4*>(row + DQ_STAGE / 2 + off) =
                            make_float4(__uint_as_float(v1[g * 4]) * p.scale, __uint_as_float(v1[g * 4 + 1]) * p.scale,
                                        __uint_as_float(v1[g * 4 + 2]) * p.scale, __uint_as_float(v1[g * 4 + 3]) * p.scale);
                    }
                }
                fence_proxy_async();
                mbar_arrive(dq_ready);
                if (warp == GRAD_WARP + 1) {
                    ok = mbar_wait_warp(dq_ready, c & 1, abort_flag);
                    if (!ok) break;
                    if (issuer) {
                        if constexpr (DQ16) {
                            tma_store_4d(&tmDQ, sDQ, 0, i * BQ, item.h, item.b);
                        } else {
                            tma_reduce_add_4d(&tmDQ, sDQ, 0, i * BQ, item.h, item.b);
                            tma_reduce_add_4d(&tmDQ, sDQ + DQ_STAGE / 2, 32, i * BQ, item.h, item.b);
                        }
                        tma_store_commit();
                    }
                }
            }
            // dK and dV: thread r owns key row r.  These warps have little to do, and the math warps go on to the next item: as
            // their task it was 3300 of an item's 19000 cycles (S = 512).  Rounded, they wait in registers for the stores, so
            // that tensor memory is free for the next item's products.
            ok = ok && mbar_wait_warp(p_done, (first + nq - 1) & 1, abort_flag);
            if (!ok) break;
            tc_fence_after();
            uint32_t e[2][32];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                uint32_t v[16];
                tmem_ld16(tmem + lane_addr + (u < 4 ? C_DK : C_DV) + (u & 3) * 16, v);
                tmem_ld_wait();
                const float f = u < 4 ? p.scale : p.inv_keep;
#pragma unroll
                for (int x = 0; x < 8; ++x)
                    e[u >> 2][(u & 3) * 8 + x] = pack2<T>(__uint_as_float(v[2 * x]) * f, __uint_as_float(v[2 * x + 1]) * f);
            }
            tc_fence_before();
            mbar_arrive(dkv_taken);
            // By way of the dQ staging tile, whose halves are a tile of 128 rows of 128 bytes each, and the copy engine.
            // (Stores of 32 bytes a thread kept the load / store unit from the math warps: 189 us for what takes 168.)
            // Behind the last item nobody loads V or the other K any more: there they need not wait for the last dQ.
            Item x = item;
            advance(x);
            const bool last = x.at >= nitems;
            uint8_t* dk_tile = last ? sK + ((k + 1) & 1) * TILE : sDQ;
            uint8_t* dv_tile = last ? sV : sDQ + DQ_STAGE / 2;
            if (!last) {
                if (issuer) {
                    tma_store_wait_read<0>();
                    mbar_arrive(dkv_free);
                }
                ok = mbar_wait_warp(dkv_free, k & 1, abort_flag);
                if (!ok) break;
            }
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int g = 0; g < 8; ++g)
                    *reinterpret_cast<uint4*>((u == 0 ? dk_tile : dv_tile) + (r >> 3) * 1024 + sw * 128 +
                                              ((static_cast<uint32_t>(g) ^ sw) << 4)) =
                        make_uint4(e[u][g * 4], e[u][g * 4 + 1], e[u][g * 4 + 2], e[u][g * 4 + 3]);
            fence_proxy_async();
            mbar_arrive(dkv_ready);
            if (warp == GRAD_WARP + 1) {
                ok = mbar_wait_warp(dkv_ready, k & 1, abort_flag);
                if (!ok) break;
                if (issuer) {
                    tma_store_4d(&tmDK, dk_tile, 0, item.kb * BKEYS, item.h, item.b);
                    tma_store_4d(&tmDV, dv_tile, 0, item.kb * BKEYS, item.h, item.b);
                    tma_store_commit();
                }
            }
        }
        // the staging tile must outlive the copies that read it; their sums are complete when the kernel is
        if (issuer) tma_store_wait_read<0>();
    } else {
        // threads r, r + 128, r + 256, r + 384: TMEM lane r = key row for St/dPt; `part` selects 32 of the 128 query columns
        const int r = threadIdx.x & 127;
        const int part = threadIdx.x >> 7;
        const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
        const uint64_t scale2 = f2_pack(p.scale_log2, p.scale_log2), keep2 = f2_pack(p.inv_keep, p.inv_keep);
        // the key's bias; -inf for keys past the end of the sequence: their probabilities come out as exp2(-inf) = 0
        auto fetch_bias = [&](const Item& x) {
            const int key = x.kb * BKEYS + r;
            if (x.at >= nitems || key >= p.S) return -INFINITY;
            return p.key_bias ? p.key_bias[static_cast<long long>(x.b) * p.S + key] : 0.f;
        };
        const uint32_t sw = r & 7;
        uint8_t* drow = sdSt + (part >> 1) * (SQ_BYTES / 2) + (r >> 3) * 1024 + sw * 128;
        bool ok = true;
        int blk = 0;
        Item item = first_item();
        float bias = fetch_bias(item);
        while (item.at < nitems && ok) {
            const uint32_t key_hash = drop_key_hash(p.seed, item.kb * BKEYS + r);
            const uint64_t kbias2 = f2_pack(bias * 1.4426950408889634f, bias * 1.4426950408889634f);
            advance(item);
            bias = fetch_bias(item);   // (the next item's: on its way for as long as this one takes)
            for (int i = 0; i < nq; ++i, ++blk) {
                if (!mbar_wait_warp(&stats_full[blk & 1], (blk >> 1) & 1, abort_flag) || !mbar_wait_warp(s_full, blk & 1, abort_flag)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const float* st_lse = s_stats + (blk & 1) * STATS + part * 32;
                const float* st_delta = st_lse + 128;
                const uint32_t* st_hash = reinterpret_cast<const uint32_t*>(st_lse + 256);
                // Pt / dSt of this thread's 32 columns, packed to 16 bits, held in registers: the whole
                // computation overlaps the tensor-core work of the previous step, whose operands still
                // occupy their places.  Pt carries the dropout mask without its 1 / (1 - p)
                // factor (dV is scaled once at the end); dSt = P (mask dP / (1 - p) - delta).
                uint32_t pk[16], dk[16];
                const uint32_t t_s = tmem + lane_addr + C_ST + part * 32, t_dp = tmem + lane_addr + C_DPT + part * 32;
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    uint32_t s_[16], d_[16];
                    tmem_ld16(t_s + c * 16, s_);
                    tmem_ld16(t_dp + c * 16, d_);
                    tmem_ld_wait();
                    if (c == 1) {
                        // both TMEM tiles are in registers: the next step's MMAs may overwrite them
                        tc_fence_before();
                        mbar_arrive(s_free);
                    }
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        // A CTA holds all of tensor memory, so per SM the MMAs of a query block wait for the P / dS of the one
                        // before and these threads for its S / dP.  Sixteen warps, four to a scheduler, hide each other's
                        // latency: with eight, of 64 columns a thread, the passes above took 246 and 175 us.  Some ten
                        // instructions per element; what has a two-wide form uses it -- P = 2^((S scale + bias) - lse), dS = P
                        // (mask dP / (1 - p) - delta).  The bias goes to the score first, as in the forward: where every key
                        // of a row carries a huge negative bias the score is rounded away in both, and P stays at most 1; bias
                        // - lse first would leave 2^(S scale).
                        const int qb = c * 16 + g * 4;
                        const ulonglong2 ls4 = *reinterpret_cast<const ulonglong2*>(st_lse + qb);
                        const ulonglong2 dl4 = *reinterpret_cast<const ulonglong2*>(st_delta + qb);
                        uint32_t rhv[4] = {0, 0, 0, 0};
                        if (p.thr32) {
                            const uint4 rh4 = *reinterpret_cast<const uint4*>(st_hash + qb);
                            rhv[0] = rh4.x, rhv[1] = rh4.y, rhv[2] = rh4.z, rhv[3] = rh4.w;
                        }
#pragma unroll
                        for (int x = 0; x < 4; x += 2) {
                            const int e = g * 4 + x;
                            const uint64_t nlse = x == 0 ? ls4.x : ls4.y, ndelta = x == 0 ? dl4.x : dl4.y;
                            float e0, e1;
                            f2_unpack(f2_add(f2_fma(f2_pack_bits(s_[e], s_[e + 1]), scale2, kbias2), nlse), e0, e1);
                            const float p0 = ex2_approx(e0), p1 = ex2_approx(e1);
                            uint64_t t;
                            float d0, d1;
                            if (p.thr32) {
                                const bool k0 = drop_keep(rhv[x], key_hash, p.thr32), k1 = drop_keep(rhv[x + 1], key_hash, p.thr32);
                                pk[(qb + x) / 2] = pack2<T>(k0 ? p0 : 0.f, k1 ? p1 : 0.f);
                                t = f2_fma(f2_pack_bits(k0 ? d_[e] : 0u, k1 ? d_[e + 1] : 0u), keep2, ndelta);
                            } else {
                                pk[(qb + x) / 2] = pack2<T>(p0, p1);
                                t = f2_add(f2_pack_bits(d_[e], d_[e + 1]), ndelta);
                            }
                            f2_unpack(f2_mul(f2_pack(p0, p1), t), d0, d1);
                            dk[(qb + x) / 2] = pack2<T>(d0, d1);
                        }
                    }
                }
                // the previous step's products read dSt and Pt: wait, then overwrite
                if (blk > 0 && !mbar_wait_warp(ds_done, (blk - 1) & 1, abort_flag)) {
                    ok = false;
                    break;
                }
#pragma unroll
                for (int g = 0; g < 4; ++g)
                    *reinterpret_cast<uint4*>(drow + ((static_cast<uint32_t>((part & 1) * 4 + g) ^ sw) << 4)) =
                        make_uint4(dk[g * 4], dk[g * 4 + 1], dk[g * 4 + 2], dk[g * 4 + 3]);
                fence_proxy_async();
                if (blk > 0 && !mbar_wait_warp(p_done, (blk - 1) & 1, abort_flag)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                tmem_st16(tmem + lane_addr + C_P + part * 16, pk);
                tmem_st_wait();
                tc_fence_before();
                mbar_arrive(pds_ready);
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        if (threadIdx.x == 0) {
            atomicExch(p.err, ERR_MBAR_TIMEOUT);
            const long long t0 = clock64();
            while (clock64() - t0 < 2000000) {
            }
        }
        __syncthreads();
    }
    if (warp == LOAD_WARP) {
        tc_fence_after();
        tmem_dealloc(tmem, BWD_TMEM_COLS);
    }
}

// delta[b,h,q] = sum_d dO[b,q,h,d] * O[b,q,h,d], D = 64, and the dQ scratch, if it is used, is cleared (a memset of its
// own cost as much as the rest of this pass).  Rows are taken in memory order ((b, q, h): h is the fastest index of
// a [B, S, H, D] tensor), 8 lanes x 16 bytes per row, two rows of a thread in flight: bound by memory.
template <typename T>
__global__ void __launch_bounds__(256)
    attn_delta_kernel(const T* O, const T* dO, float* __restrict__ delta, float* __restrict__ dq_accum, int B, int H, int S,
                      long long o_sb, long long o_ss, long long o_sh, long long d_sb, long long d_ss,
                      long long d_sh) {
    grid_trigger();
    grid_wait();
    const unsigned rows = static_cast<unsigned>(B) * S * H;   // < 2^31: checked by the caller
    const int sub = threadIdx.x & 7;
    // a block takes 64 consecutive rows: 32 and the 32 behind them
    const unsigned row0 = blockIdx.x * 64u + (threadIdx.x >> 3);
    uint4 ov[2], dv[2];
    long long at[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const unsigned row = row0 + u * 32u;
        ov[u] = dv[u] = make_uint4(0, 0, 0, 0);
        at[u] = -1;
        if (row < rows) {
            const unsigned bq = row / H, h = row - bq * H, b = bq / S, q = bq - b * S;
            ov[u] = *reinterpret_cast<const uint4*>(O + b * o_sb + q * o_ss + h * o_sh + sub * 8);
            dv[u] = *reinterpret_cast<const uint4*>(dO + b * d_sb + q * d_ss + h * d_sh + sub * 8);
            at[u] = (static_cast<long long>(b) * H + h) * S + q;
        }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        if (dq_accum && at[u] >= 0) {
            float4* z = reinterpret_cast<float4*>(dq_accum + static_cast<size_t>(row0 + u * 32u) * 64 + sub * 4);
            z[0] = make_float4(0.f, 0.f, 0.f, 0.f);   // 8 lanes cover the row in two runs of 128 bytes
            z[8] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        const T* oe = reinterpret_cast<const T*>(&ov[u]);
        const T* de = reinterpret_cast<const T*>(&dv[u]);
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) s = fmaf(to_f32<T>(oe[j]), to_f32<T>(de[j]), s);
        s += __shfl_xor_sync(0xffffffffu, s, 4);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        if (sub == 0 && at[u] >= 0) delta[at[u]] = s;
    }
}

// dQ[b,q,h,:] = (T) acc[b,q,h,:]
template <typename T>
__global__ void attn_dq_convert_kernel(const float* acc, T* __restrict__ dQ, int B,
                                       int H, int S, long long sb, long long ss, long long sh) {
    grid_trigger();
    grid_wait();
    const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;  // 8-element group
    const long long total = static_cast<long long>(B) * S * H * 8;
    if (i >= total) return;
    const int g = i & 7;
    const long long row = i >> 3;  // (b*S + q)*H + h
    const int h = row % H;
    const int q = (row / H) % S;
    const int b = row / (static_cast<long long>(H) * S);
    const float4 a = *reinterpret_cast<const float4*>(acc + row * 64 + g * 8);
    const float4 c = *reinterpret_cast<const float4*>(acc + row * 64 + g * 8 + 4);
    uint4 o;
    T* e = reinterpret_cast<T*>(&o);
    e[0] = from_f32<T>(a.x); e[1] = from_f32<T>(a.y); e[2] = from_f32<T>(a.z); e[3] = from_f32<T>(a.w);
    e[4] = from_f32<T>(c.x); e[5] = from_f32<T>(c.y); e[6] = from_f32<T>(c.z); e[7] = from_f32<T>(c.w);
    *reinterpret_cast<uint4*>(dQ + b * sb + q * ss + h * sh + g * 8) = o;
}

template <typename T>
static int launch_bwd(const RbAttnArgs& a, cudaStream_t st) {
    CUtensorMap tq, tk, tv, tdo;
    int rc;
    const uint64_t D = a.D, S = a.S, H = a.H, B = a.B;
    if ((rc = make_tmap_4d(&tq, a.Q, a.dtype, D, S, H, B, a.q_ss * 2, a.q_sh * 2, a.q_sb * 2, 64, 128))) return rc;
    if ((rc = make_tmap_4d(&tk, a.K, a.dtype, D, S, H, B, a.k_ss * 2, a.k_sh * 2, a.k_sb * 2, 64, 128))) return rc;
    if ((rc = make_tmap_4d(&tv, a.V, a.dtype, D, S, H, B, a.v_ss * 2, a.v_sh * 2, a.v_sb * 2, 64, 128))) return rc;
    if ((rc = make_tmap_4d(&tdo, a.dO, a.dtype, D, S, H, B, a.do_ss * 2, a.do_sh * 2, a.do_sb * 2, 64, 128))) return rc;
    const long long rows = static_cast<long long>(a.B) * a.H * a.S;
    if (rows >= (1LL << 31) - 64) return -2;
    CUtensorMap tdq, tdk, tdv;
    const bool dq16 = !rb_attn_bwd_adds(&a);
    if (!dq16 && !a.dq_accum) return -2;
    // (a dimension of one has any stride; the copy engine wants one it can take)
    auto stride = [](uint64_t n, int64_t s) { return static_cast<uint64_t>(n > 1 ? s * 2 : 128); };
    if (dq16)
        rc = make_tmap_4d(&tdq, a.dQ, a.dtype, D, S, H, B, stride(S, a.dq_ss), stride(H, a.dq_sh), stride(B, a.dq_sb), 64, 128);
    else
        rc = make_tmap_4d_f32(&tdq, a.dq_accum, 64, S, H, B, H * 64 * 4, 64 * 4, S * H * 64 * 4, 32, 128);
    if (rc) return rc;
    if ((rc = make_tmap_4d(&tdk, a.dK, a.dtype, D, S, H, B, stride(S, a.dk_ss), stride(H, a.dk_sh), stride(B, a.dk_sb), 64, 128)))
        return rc;
    if ((rc = make_tmap_4d(&tdv, a.dV, a.dtype, D, S, H, B, stride(S, a.dv_ss), stride(H, a.dv_sh), stride(B, a.dv_sb), 64, 128)))
        return rc;
    if (launch_after(attn_delta_kernel<T>, static_cast<unsigned>((rows + 63) / 64), 256, 0, st, static_cast<const T*>(a.O),
                     static_cast<const T*>(a.dO), a.delta, dq16 ? nullptr : a.dq_accum, a.B, a.H, a.S, a.o_sb, a.o_ss, a.o_sh,
                     a.do_sb, a.do_ss, a.do_sh) != cudaSuccess)
        return -1;
    AttnBwdParams p;
    p.B = a.B; p.H = a.H; p.S = a.S;
    p.scale = a.scale;
    p.scale_log2 = a.scale * 1.4426950408889634f;
    p.key_bias = a.key_bias;
    p.lse = a.lse;
    p.delta = a.delta;
    p.dq_accum = a.dq_accum;
    p.thr32 = drop_threshold(a.p_drop);
    p.inv_keep = a.p_drop > 0.f ? 1.f / (1.f - a.p_drop) : 1.f;
    p.seed = drop_seed(a.seed, a.offset);
    p.err = error_word_ptr();
    if (!p.err) return -3;
    auto kern = dq16 ? attn_bwd_kernel<T, true> : attn_bwd_kernel<T, false>;
    static bool attr_set[64][2] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (!attr_set[dev & 63][dq16]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_SMEM) != cudaSuccess)
            return -4;
        attr_set[dev & 63][dq16] = true;
    }
    const long long nitems = static_cast<long long>((a.S + BKEYS - 1) / BKEYS) * a.H * a.B;   // (< 2^31, as the rows)
    const int sms = num_sms();
    const unsigned grid = static_cast<unsigned>(nitems < sms ? nitems : sms);
    const unsigned nq = static_cast<unsigned>((a.S + BQ - 1) / BQ), nh = static_cast<unsigned>(a.H);
    p.step_kb = static_cast<int>(grid % nq);
    p.step_h = static_cast<int>(grid / nq % nh);
    p.step_b = static_cast<int>(grid / nq / nh);
    auto inverse = [](unsigned d) { return d == 1 ? 0u : static_cast<uint32_t>(((1ull << 32) + d - 1) / d); };
    p.inv_nq = inverse(nq);
    p.inv_h = inverse(nh);
    if (launch_after(kern, grid, BWD_THREADS, BWD_SMEM, st, tq, tk, tv, tdo, tdq, tdk, tdv, p) != cudaSuccess) return -1;
    if (dq16) return 0;
    const long long groups = rows * 8;
    return launch_after(attn_dq_convert_kernel<T>, static_cast<unsigned>((groups + 255) / 256), 256, 0, st,
                        static_cast<const float*>(a.dq_accum), static_cast<T*>(a.dQ), a.B, a.H, a.S, a.dq_sb, a.dq_ss,
                        a.dq_sh) == cudaSuccess
               ? 0
               : -1;
}

}  // namespace rb

// A sequence of one key block has nothing to add up in dQ: without the clearing of the scratch, the additions and the
// conversion 64 x 128 x 16 heads take 38.4 us in place of 50.8, 32 x 64 x 16 18.6 (23.4), 8 x 128 x 16 11.2 (14.0),
// 1 x 32 x 4 7.7 (9.7).  A kernel of its own: asked in the drain loop, it cost the longer sequences 1 %.  (Strides of dQ
// that the copy engine does not take go the way of those.)
extern "C" int rb_attn_bwd_adds(const RbAttnArgs* a) {
    auto takes = [](int n, int64_t s) { return n <= 1 || (s > 0 && s < (int64_t{1} << 39)); };
    return a->S > rb::BKEYS || !takes(a->S, a->dq_ss) || !takes(a->H, a->dq_sh) || !takes(a->B, a->dq_sb);
}

extern "C" int rb_attn_bwd(const RbAttnArgs* a, void* stream) {
    if (a->D != 64) return -2;
    if (a->B <= 0 || a->H <= 0 || a->S <= 0) return 0;
    // (the tensor maps check the bases and strides too, but of O and dQ)
    if (rb::off16(a->O, a->dQ, a->dK, a->dV) || (a->o_sb | a->o_ss | a->o_sh | a->dq_sb | a->dq_ss | a->dq_sh) % 8 ||
        (a->dk_sb | a->dk_ss | a->dk_sh | a->dv_sb | a->dv_ss | a->dv_sh) % 8)
        return -5;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return a->dtype == 1 ? rb::launch_bwd<__nv_bfloat16>(*a, st) : rb::launch_bwd<__half>(*a, st);
}
