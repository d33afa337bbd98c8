// Attention backward on sm_100a: dQ, dK, dV of softmax(Q K^T / sqrt(128)) V per head, from Q, K, V and dO.
//
// It takes the place of the reference's exact backward attention_bwd (engine/src/train.cu:216-242: five batched cuBLAS SGEMMs
// per head group around k_softmax_pad, train.cu:103-121, and k_dsoftmax, train.cu:124-131, with the [heads, Tq, Tk]
// probabilities P and their gradient dP materialised in the arena) for the LoRA trainer's two call sites (train.cu:334, 344).
// Here nothing of size Tq x Tk exists in memory: like the forward kernel the products are formed tile by tile on the tensor
// cores (fp16 operands, fp32 accumulation in TMEM) and P is recomputed from a per-row statistic.
//
// Three launches (kb_attn_bwd): the staging pre-pass (Q, K, V, dO -> fp16), the forward kernel in its RowStats form, which stores no
// O but leaves in the "stats" array L_i = log2 of the softmax denominator of row i (npad zero keys included) and
// D_i = sum_d dO[i, d] O[i, d] (= sum_j P_ij dP_ij, what k_dsoftmax sums; dO as the tensor cores see it, O in fp32), and this
// file's kernel, whose thread blocks play one of two roles:
//
//   BWD_DKV  one thread block per (key block j, head, image), query blocks i streamed through a ring:
//              S^T  = K_j Q_i^T            dP^T = V_j dO_i^T                      (two SS products into TMEM)
//              P^T  = 2^(c S^T - L_i)      dS^T = P^T (dP^T - D_i)                (softmax warps; fp16, written over dP^T)
//              dV_j += P^T dO_i            dK_j += dS^T Q_i                       (A operand from TMEM, B the same shared-memory
//                                                                                  tiles read MN-major)
//   BWD_DQ   one thread block per (query block i, head, image), key blocks j streamed:
//              S = Q_i K_j^T,  dP = dO_i V_j^T,  dS = 2^(c S - L_i) (dP - D_i),  dQ_i += dS K_j
//
// Two roles instead of one with atomics: every output element is written once by one thread block, in a fixed order, so
// results are bit-identical from run to run (the reference's are too). The price is that S and dP are formed twice.
// The npad zero keys only enter through L_i: their dP is 0 and their K is 0, so they add nothing to any gradient
// (train.cu:124 says the same of the reference). Rows past Tq or Tk are zero-filled by TMA; a zero Q/dO row has dS = 0 and
// adds nothing to dK / dV, a zero K row adds nothing to dQ, so ragged sizes need no masking - only finite statistics, which
// the stats array (padded to whole query blocks) always holds.
//
// TMEM (512 columns): T0 [0,128) S or S^T, T1 [128,256) dP or dP^T, acc0 [256,384), acc1 [384,512) (BWD_DQ: its first half holds dS).
// A step is a chain through the softmax warps (~2100 cycles: 1024 of them the MUFU unit's) next to four (BWD_DQ: three) products of 512
// cycles, so nothing but the products that have to may stand in that chain:
//   softmax phase 1: S^T read (T0 is free: the next step's S^T may go), P^T = 2^(c S^T - L) kept in registers;
//   softmax phase 2: dP^T read, P^T stored as fp16 over it ("READ1": dV may go), dS^T = P^T (dP^T - D) stored over it too ("DS");
//   issue order:     [READ0] S^T of the next step | [READ1] dV += P^T dO | [DS] dK += dS^T Q | dP^T of the next step
// (in-order execution of one thread's tcgen05.mma keeps dP^T from overwriting what dV and dK still read). Phase 1 of the next step
// runs under dV, dK and dP^T. Each of the eight softmax warps (lane quarter x column half) owns 64 columns of T0 / T1 and writes its
// fp16 results over those same columns, so no warp overwrites what another still has to read. In BWD_DQ dS has columns of its own, and
// dP of the next step need not wait for dQ. The streamed tiles have three and two stages: with two of each the tile of the next S was
// asked for when the step in front had freed it and came after it was wanted.
// Measured on B200 by clock stamps, cycles per step: P^T stored over S^T, whose next product therefore waited for dV, and two stages: BWD_DKV
// 3050, BWD_DQ 2780 -> 2580 and 2080 (with S^T and dP^T in one place in turn, so that S^T waited for dP^T to be read: 3090). An SS product costs the
// same with half the N, and taking its A operand from TMEM changed nothing.
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>

#include "attn_sm100.cuh"
#include "ptx.cuh"

namespace kb {

constexpr int BWD_DKV = 0, BWD_DQ = 1;
constexpr int BWD_THREADS = 384;                              // warps 0-7 softmax / epilogue, 8 MMA issue, 9 TMA loads, 10-11 idle
constexpr int BWD_SOFTMAX_REGS = 224, BWD_OTHER_REGS = 56;    // 384 x 168 = 256 x 224 + 128 x 56 (-Xptxas -v: 12 bytes of spill stores, 24 of loads)
constexpr int BWD_X0_STAGES = 3, BWD_X1_STAGES = 2;           // of the streamed tiles: X0 (Q_i or K_j), X1 (dO_i or V_j, with the statistics)
constexpr int BWD_STATS_BYTES = 1024;                         // the statistics of a query block
constexpr int BWD_SMEM = (2 + BWD_X0_STAGES + BWD_X1_STAGES) * TILE_BYTES + BWD_X1_STAGES * BWD_STATS_BYTES + 1024;   // resident pair, rings, control block
static_assert(BWD_SMEM <= 232448, "shared memory per thread block on sm_100");

struct BwdParams {
    int B, H, Tq, Tk;
    // BWD_DKV with few key blocks (cross-attention to a short context): the query blocks of a (key block, head, image) are cut
    // into qsplit ranges of q_per blocks, one thread block each, whose partial dK / dV go to scratch (image index s * B + b of
    // the output tensor maps) and are summed in a fixed order by bwd_reduce_kernel. qsplit = 1: no cut, outputs written directly.
    int qsplit, q_per;
    const float* stats;     // [B][H][ceil(Tq/128)][2][128]: L (log2 of the softmax denominator, in units of c * score), then D
    float scale_log2;       // c = log2(e) / sqrt(128)
    float scale;            // 1 / sqrt(128)
    uint32_t* status;
};

// T is the first product (S or S^T) or the second (dP or dP^T) of a step. READ, DS: one arrival per softmax warp
enum { BB_RES = 0, BB_X0FULL = 2, BB_X0EMPTY = BB_X0FULL + BWD_X0_STAGES, BB_X1FULL = BB_X0EMPTY + BWD_X0_STAGES, BB_X1EMPTY = BB_X1FULL + BWD_X1_STAGES,
       BB_TFULL = BB_X1EMPTY + BWD_X1_STAGES, BB_READ = BB_TFULL + 2, BB_DS = BB_READ + 2, BB_DSFREE, BB_ACC, BB_COUNT };

__device__ __forceinline__ void bulk_load_1d(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

// One thread block's work in either role: (blk, h, b) = (key block, head, image) for BWD_DKV, (query block, head, image) for BWD_DQ.
template <int MODE>
__device__ __forceinline__ void attn_bwd_body(const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV, const CUtensorMap& tmdO,
                                              const CUtensorMap& tmOut0, const CUtensorMap& tmOut1, const BwdParams& p, const int blk, const int h,
                                              const int b, const int part) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t base = smem_u32(smem_raw);
    if (base & 1023u) {                                           // never seen; without it every tile would be garbage
        if (threadIdx.x == 0) atomicOr(p.status, ST_TIMEOUT);
        return;
    }
    const uint32_t sR0 = base, sR1 = base + TILE_BYTES;            // resident: K_j, V_j (BWD_DKV) or Q_i, dO_i (BWD_DQ)
    constexpr int OFF_X1 = (2 + BWD_X0_STAGES) * TILE_BYTES, OFF_STATS = OFF_X1 + BWD_X1_STAGES * TILE_BYTES;
    const uint32_t sX0 = base + 2 * TILE_BYTES, sX1 = base + OFF_X1;
    uint8_t* const ctrl = smem_raw + OFF_STATS + BWD_X1_STAGES * BWD_STATS_BYTES;
    const uint32_t bars = smem_u32(ctrl);
    uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(ctrl + 256);
    volatile uint32_t* const abort_flag = reinterpret_cast<volatile uint32_t*>(ctrl + 260);
    static_assert(BB_COUNT * 8 <= 256, "barriers in front of the shared words");
    auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nqb = (p.Tq + BM - 1) / BM;
    const int i0 = MODE == BWD_DKV ? part * p.q_per : 0;           // first streamed block of this thread block
    const int n_it = MODE == BWD_DKV ? min(nqb - i0, p.q_per) : (p.Tk + BN - 1) / BN;

    if (tid == 0) {
        for (int i = 0; i < BB_COUNT; i++) mbar_init(bar(i), (i == BB_READ || i == BB_READ + 1 || i == BB_DS) ? 8u : 1u);   // one arrival per softmax warp
        *abort_flag = 0u;
        mbar_fence_init();
        fence_proxy_async_smem();
    }
    if (warp == 9 && lane == 0) { tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmdO); }
    if (warp == 8) {
        tmem_alloc(smem_u32(tmem_slot), TMEM_ALL_COLUMNS);
        tmem_relinquish();
    }
    pdl_launch();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    constexpr uint32_t tmem_base = 0;                             // see TMEM_ALL_COLUMNS and elect_one
    constexpr uint32_t T0 = 0u, T1 = 128u;
    // fp16 operands: BWD_DKV: a warp stores its P^T and its dS^T over its own 64 columns of dP^T, which it has read (contraction elements
    // [64 hh, 64 hh + 64) in columns [64 hh, 64 hh + 32) and [64 hh + 32, 64 hh + 64)); BWD_DQ: dS in columns of its own
    constexpr uint32_t TP = T1, TDS = MODE == BWD_DKV ? T1 + 32u : 384u, PIECE = MODE == BWD_DKV ? 64u : 32u;
    pdl_wait();

    if (warp < 8) {
        setmaxnreg_inc<BWD_SOFTMAX_REGS>();
        // ------------------------------------------------------------------ softmax warps: TMEM lane quarter x column half
        const int quarter = warp & 3, half = warp >> 2;
        const int r = quarter * 32 + lane;                          // row of the resident block (= TMEM lane)
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        const uint32_t tT0 = tmem_base + lane_base + T0, tT1 = tmem_base + lane_base + T1, tP = tmem_base + lane_base + TP, tDS = tmem_base + lane_base + TDS;
        const float c = p.scale_log2;
        float Lr = 0.f, Dr = 0.f;                                   // BWD_DQ: this row's statistics
        if (MODE == BWD_DQ) {
            const float* st = p.stats + (((size_t)b * p.H + h) * nqb + blk) * 256;
            Lr = __ldcg(st + r);
            Dr = __ldcg(st + 128 + r);
        }
        bool ok = true;
        for (int it = 0; it < n_it; ++it) {
            const int st1 = it % BWD_X1_STAGES;
            if (MODE == BWD_DKV) {                                  // the statistics come with the X1 tile
                ok = __all_sync(0xffffffffu, mbar_wait(bar(BB_X1FULL + st1), (uint32_t)(it / BWD_X1_STAGES) & 1u, abort_flag));
                if (!ok) break;
            }
            // ---- phase 1: P = 2^(c S - L) for this warp's 64 columns
            ok = __all_sync(0xffffffffu, mbar_wait(bar(BB_TFULL + 0), (uint32_t)it & 1u, abort_flag));
            if (!ok) break;
            tc_fence_after();
            const float* sStats = reinterpret_cast<const float*>(smem_raw + OFF_STATS + st1 * BWD_STATS_BYTES) + half * 64;
            float pv[64];
            {
                uint32_t s0[32], s1[32];
                tmem_ld32(tT0 + (uint32_t)(half * 64), s0);
                tmem_ld32(tT0 + (uint32_t)(half * 64 + 32), s1);
                tmem_wait_ld();
                reg_fence32(s0); reg_fence32(s1);
                tc_fence_before();                                  // S has been read: the next step's S may be formed
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(BB_READ + 0));
#pragma unroll
                for (int e = 0; e < 64; e += 4) {
                    float4 L4 = make_float4(Lr, Lr, Lr, Lr);
                    if (MODE == BWD_DKV) L4 = *reinterpret_cast<const float4*>(sStats + e);   // per column: the query row's statistic (a broadcast read)
                    const uint32_t* const sv = e < 32 ? s0 : s1;
                    pv[e] = ex2(fmaf(__uint_as_float(sv[e & 31]), c, -L4.x));
                    pv[e + 1] = ex2(fmaf(__uint_as_float(sv[(e & 31) + 1]), c, -L4.y));
                    pv[e + 2] = ex2(fmaf(__uint_as_float(sv[(e & 31) + 2]), c, -L4.z));
                    pv[e + 3] = ex2(fmaf(__uint_as_float(sv[(e & 31) + 3]), c, -L4.w));
                }
            }
            uint32_t pk[32];
            if (MODE == BWD_DKV) {
#pragma unroll
                for (int e = 0; e < 32; e++) pk[e] = pack16<DT_F16>(pv[2 * e], pv[2 * e + 1]);
                reg_fence32(pk);
            }
            // ---- phase 2: dS = P (dP - D)
            // The second product of this step is complete and with it every product in front of it, the previous step's dV and dK among them
            ok = __all_sync(0xffffffffu, mbar_wait(bar(BB_TFULL + 1), (uint32_t)it & 1u, abort_flag));
            if (!ok) break;
            tc_fence_after();
            {
                uint32_t d0[32], d1[32], dk[32];
                tmem_ld32(tT1 + (uint32_t)(half * 64), d0);
                tmem_ld32(tT1 + (uint32_t)(half * 64 + 32), d1);
                tmem_wait_ld();
                reg_fence32(d0); reg_fence32(d1);
                if (MODE == BWD_DKV) {                              // element pair (2c, 2c+1) of the contraction in column c
                    tmem_st32(tP + (uint32_t)half * PIECE, pk);
                    tmem_wait_st();
                }
                tc_fence_before();                                  // BWD_DKV: P^T is stored; BWD_DQ: dP has been read, the next step's may be formed
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(BB_READ + 1));
                if (MODE == BWD_DQ && tid == 0) mbar_arrive(bar(BB_X1EMPTY + st1));   // V_j has been multiplied
#pragma unroll
                for (int e = 0; e < 64; e += 4) {
                    float4 D4 = make_float4(Dr, Dr, Dr, Dr);
                    if (MODE == BWD_DKV) D4 = *reinterpret_cast<const float4*>(sStats + 128 + e);
                    const uint32_t* const dv = e < 32 ? d0 : d1;
                    dk[e >> 1] = pack16<DT_F16>(pv[e] * (__uint_as_float(dv[e & 31]) - D4.x), pv[e + 1] * (__uint_as_float(dv[(e & 31) + 1]) - D4.y));
                    dk[(e >> 1) + 1] = pack16<DT_F16>(pv[e + 2] * (__uint_as_float(dv[(e & 31) + 2]) - D4.z), pv[e + 3] * (__uint_as_float(dv[(e & 31) + 3]) - D4.w));
                }
                if (MODE == BWD_DQ && it > 0) {                     // the previous step's dQ has read dS and its K_j
                    ok = __all_sync(0xffffffffu, mbar_wait(bar(BB_DSFREE), (uint32_t)(it - 1) & 1u, abort_flag));
                    if (!ok) break;
                    tc_fence_after();
                    if (tid == 0) mbar_arrive(bar(BB_X0EMPTY + (it - 1) % BWD_X0_STAGES));
                }
                tmem_st32(tDS + (uint32_t)half * PIECE, dk);
            }
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(BB_DS));
        }
        // ------------------------------------------------------------------ epilogue: accumulators -> global
        // Each warp turns its 32 rows x 64 columns of an accumulator into two 32 x 32 fp32 boxes (128-byte rows, 128-byte
        // swizzle) in the stage area, which is free now, and one lane hands them to bulk tensor stores: rows past the end are
        // clipped by the tensor map. (Per-thread row stores, 32 scattered 16-byte pieces per instruction, took ~4 us per
        // thread block here, as they did in the projection GEMM.)
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait(bar(BB_ACC), 0u, abort_flag));
        if (ok) {
            tc_fence_after();
            uint8_t* const my_stage = smem_raw + 2 * TILE_BYTES + warp * 16384;          // four 4 KiB boxes per warp
#pragma unroll
            for (int a = 0; a < (MODE == BWD_DKV ? 2 : 1); a++) {
                const float k = (MODE == BWD_DKV && a == 0) ? 1.f : p.scale;   // dV unscaled; dK and dQ carry 1/sqrt(128)
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    uint32_t o[32];
                    tmem_ld32(tmem_base + lane_base + 256u + (uint32_t)(a * 128 + half * 64 + 32 * q), o);
                    tmem_wait_ld();
                    reg_fence32(o);
                    uint8_t* const box = my_stage + (a * 2 + q) * 4096 + lane * 128;
#pragma unroll
                    for (int cc = 0; cc < 8; cc++)
                        *reinterpret_cast<float4*>(box + ((cc ^ (lane & 7)) << 4)) =
                            make_float4(__uint_as_float(o[4 * cc]) * k, __uint_as_float(o[4 * cc + 1]) * k, __uint_as_float(o[4 * cc + 2]) * k,
                                        __uint_as_float(o[4 * cc + 3]) * k);
                }
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                const int row0 = blk * BM + quarter * 32;
                if (row0 < (MODE == BWD_DKV ? p.Tk : p.Tq)) {
#pragma unroll
                    for (int a = 0; a < (MODE == BWD_DKV ? 2 : 1); a++)
#pragma unroll
                        for (int q = 0; q < 2; q++)
                            tma_store_3d(a ? &tmOut1 : &tmOut0, smem_u32(my_stage + (a * 2 + q) * 4096), h * HD + half * 64 + 32 * q, row0,
                                         MODE == BWD_DKV ? part * p.B + b : b);
                    tma_store_commit();
                }
                tma_store_wait_read();                                       // the stage area goes away with the thread block
            }
        }
    } else {
        setmaxnreg_dec<BWD_OTHER_REGS>();
        if (warp == 8 && elect_one()) {
            // ------------------------------------------------------------------ MMA issue
            constexpr uint32_t IDESC_T = idesc_f16(0, 0, 0, 0, BM, BN);   // T = R X^T, both operands K-major (rows of 128 head channels)
            constexpr uint32_t IDESC_A = idesc_f16(0, 0, 0, 1, BM, HD);   // acc += (fp16 in TMEM) X, X MN-major (rows = contraction index)
            constexpr uint32_t DESC_HI = smem_desc_hi_sw128(1024);
            auto issue_T = [&](uint32_t d_tmem, uint32_t a_saddr, uint32_t b_saddr) {
                const uint32_t alo = smem_desc_lo(a_saddr, 16), blo = smem_desc_lo(b_saddr, 16);
                mma_ss_w<0>(d_tmem, alo, blo, DESC_HI, IDESC_T);
#pragma unroll
                for (int kk = 1; kk < 8; kk++) {
                    const uint32_t off = ((uint32_t)(kk >> 2) * HALF_BYTES + (uint32_t)(kk & 3) * 32u) >> 4;
                    mma_ss_w<1>(d_tmem, alo + off, blo + off, DESC_HI, IDESC_T);
                }
            };
            auto issue_A = [&](uint32_t d_tmem, uint32_t a_region, uint32_t b_saddr, bool first) {
                const uint32_t blo = smem_desc_lo(b_saddr, HALF_BYTES);
#pragma unroll
                for (int kk = 0; kk < 8; kk++) {
                    const uint32_t a_t = a_region + PIECE * (uint32_t)(kk >> 2) + (uint32_t)(8 * (kk & 3));
                    if (kk == 0 && first) mma_ts_w<0>(d_tmem, a_t, blo, DESC_HI, IDESC_A);
                    else mma_ts_w<1>(d_tmem, a_t, blo + (uint32_t)(kk * 128), DESC_HI, IDESC_A);
                }
            };
            auto x0 = [&](int it) { return sX0 + (uint32_t)(it % BWD_X0_STAGES) * TILE_BYTES; };
            auto x1 = [&](int it) { return sX1 + (uint32_t)(it % BWD_X1_STAGES) * TILE_BYTES; };
            auto x0_wait = [&](int it) { return mbar_wait(bar(BB_X0FULL + it % BWD_X0_STAGES), (uint32_t)(it / BWD_X0_STAGES) & 1u, abort_flag); };
            auto x1_wait = [&](int it) { return mbar_wait(bar(BB_X1FULL + it % BWD_X1_STAGES), (uint32_t)(it / BWD_X1_STAGES) & 1u, abort_flag); };
            auto step_wait = [&](int which, int it) { return mbar_wait(bar(which), (uint32_t)it & 1u, abort_flag); };
            auto first_T = [&](int it) { issue_T(tmem_base + T0, sR0, x0(it)); tc_commit(bar(BB_TFULL + 0)); };    // S / S^T
            auto second_T = [&](int it) { issue_T(tmem_base + T1, sR1, x1(it)); tc_commit(bar(BB_TFULL + 1)); };   // dP / dP^T
            bool good = mbar_wait(bar(BB_RES + 0), 0u, abort_flag) && x0_wait(0);
            if (good) {
                tc_fence_after();
                first_T(0);
                good = mbar_wait(bar(BB_RES + 1), 0u, abort_flag) && x1_wait(0);
                if (good) {
                    tc_fence_after();
                    second_T(0);
                }
            }
            // tiles are waited for in front of the softmax warps, whose signal is what the next product hangs on
            for (int it = 0; it < n_it && good; ++it) {
                const bool more = it + 1 < n_it;
                if (more) {
                    good = x0_wait(it + 1) && step_wait(BB_READ + 0, it);
                    if (!good) break;
                    tc_fence_after();
                    first_T(it + 1);
                    good = x1_wait(it + 1);
                    if (!good) break;
                }
                if (MODE == BWD_DKV) {
                    good = step_wait(BB_READ + 1, it);
                    if (!good) break;
                    tc_fence_after();
                    issue_A(tmem_base + 256u, tmem_base + TP, x1(it), it == 0);                           // dV += P^T dO_i
                    good = step_wait(BB_DS, it);
                    if (!good) break;
                    tc_fence_after();
                    issue_A(tmem_base + 384u, tmem_base + TDS, x0(it), it == 0);                          // dK += dS^T Q_i
                    if (more) {
                        tc_commit(bar(BB_X1EMPTY + it % BWD_X1_STAGES));                                 // this step's tiles are multiplied, its statistics read
                        second_T(it + 1);
                    }
                } else {
                    if (more) {
                        good = step_wait(BB_READ + 1, it);
                        if (!good) break;
                        tc_fence_after();
                        second_T(it + 1);
                    }
                    good = step_wait(BB_DS, it);
                    if (!good) break;
                    tc_fence_after();
                    issue_A(tmem_base + 256u, tmem_base + TDS, x0(it), it == 0);                          // dQ += dS K_j
                    if (more) tc_commit(bar(BB_DSFREE));
                }
            }
            if (good) tc_commit(bar(BB_ACC));
        } else if (warp == 9 && elect_one()) {
            // ------------------------------------------------------------------ TMA loads
            auto load_tile = [&](uint32_t dst, const CUtensorMap* tm, uint32_t mbar, int row0) {
                tma_load_3d(dst, tm, mbar, h * HD, row0, b);
                tma_load_3d(dst + HALF_BYTES, tm, mbar, h * HD + 64, row0, b);
            };
            // the resident pair, each tile in front of the first streamed one that it is multiplied with
            auto load_res = [&](int i) {
                mbar_expect_tx(bar(BB_RES + i), TILE_BYTES);
                load_tile(i ? sR1 : sR0, i == 0 ? (MODE == BWD_DKV ? &tmK : &tmQ) : (MODE == BWD_DKV ? &tmV : &tmdO), bar(BB_RES + i), blk * BM);
            };
            bool good = true;
            int issued0 = 0, issued1 = 0;
            for (int it = 0; it < n_it && good; ++it) {
                const int st0 = it % BWD_X0_STAGES, st1 = it % BWD_X1_STAGES;
                if (MODE == BWD_DQ) {
                    good = mbar_wait(bar(BB_X0EMPTY + st0), ((uint32_t)(it / BWD_X0_STAGES) & 1u) ^ 1u, abort_flag);
                    if (!good) break;
                }                                                     // BWD_DKV: step it - 3 was waited for in front of the last X1 tile
                if (it == 0) load_res(0);
                mbar_expect_tx(bar(BB_X0FULL + st0), TILE_BYTES);
                load_tile(sX0 + st0 * TILE_BYTES, MODE == BWD_DKV ? &tmQ : &tmK, bar(BB_X0FULL + st0), (i0 + it) * BM);
                issued0 = it + 1;
                good = mbar_wait(bar(BB_X1EMPTY + st1), ((uint32_t)(it / BWD_X1_STAGES) & 1u) ^ 1u, abort_flag);
                if (!good) break;
                if (it == 0) load_res(1);
                mbar_expect_tx(bar(BB_X1FULL + st1), TILE_BYTES + (MODE == BWD_DKV ? BWD_STATS_BYTES : 0));
                load_tile(sX1 + st1 * TILE_BYTES, MODE == BWD_DKV ? &tmdO : &tmV, bar(BB_X1FULL + st1), (i0 + it) * BM);
                if (MODE == BWD_DKV)
                    bulk_load_1d(base + OFF_STATS + st1 * BWD_STATS_BYTES, p.stats + (((size_t)b * p.H + h) * nqb + (i0 + it)) * 256, BWD_STATS_BYTES, bar(BB_X1FULL + st1));
                issued1 = it + 1;
            }
            if (!good || *abort_flag) {                               // let the copies already requested land before the memory goes away
                for (int i = 0; i < 2; i++) drain_wait(bar(BB_RES + i), 0u);
                for (int k = max(issued0 - BWD_X0_STAGES, 0); k < issued0; ++k) drain_wait(bar(BB_X0FULL + k % BWD_X0_STAGES), (uint32_t)(k / BWD_X0_STAGES) & 1u);
                for (int k = max(issued1 - BWD_X1_STAGES, 0); k < issued1; ++k) drain_wait(bar(BB_X1FULL + k % BWD_X1_STAGES), (uint32_t)(k / BWD_X1_STAGES) & 1u);
            }
        }
        __syncwarp();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 8) {
        if (lane == 0 && *abort_flag) atomicOr(p.status, ST_TIMEOUT);
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

// dk / dv [B*Tk, ld] = sum over the qsplit partial results [qsplit][B*Tk][cols] in scratch, in the order of the parts
// (bit-identical from run to run); one thread per four columns of a row, both tensors in one launch (blockIdx.y).
__global__ void bwd_reduce_kernel(float* dk, int ld_dk, float* dv, int ld_dv, const float* part_dk, const float* part_dv, int rows, int cols, int qsplit) {
    pdl_launch();
    pdl_wait();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t per_row = (size_t)cols / 4;
    if (i >= (size_t)rows * per_row) return;
    const size_t r = i / per_row, c4 = i % per_row;
    const float* src = blockIdx.y ? part_dv : part_dk;
    float* dst = blockIdx.y ? dv + r * (size_t)ld_dv + c4 * 4 : dk + r * (size_t)ld_dk + c4 * 4;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = 0; s < qsplit; s++) {
        const float4 v = __ldcg(reinterpret_cast<const float4*>(src + ((size_t)s * rows + r) * (size_t)cols) + c4);
        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    *reinterpret_cast<float4*>(dst) = acc;
}

// Both roles in ONE launch: thread blocks [0, n_dkv) are the dK/dV blocks, the rest the dQ blocks. The two halves are independent
// (disjoint outputs, common read-only inputs); launched together, the dQ blocks start on the SMs that the last, partial round of
// dK/dV blocks leaves idle: 2 x 512 blocks at the DiT size are 6.9 rounds on 148 SMs instead of 3.46 rounds twice, each rounded up.
__global__ void __launch_bounds__(BWD_THREADS, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                const __grid_constant__ CUtensorMap tmdO, const __grid_constant__ CUtensorMap tmDQ, const __grid_constant__ CUtensorMap tmDK,
                const __grid_constant__ CUtensorMap tmDV, const __grid_constant__ BwdParams p, const int n_dkv) {
    const int nkb = (p.Tk + BN - 1) / BN, nqb = (p.Tq + BM - 1) / BM;
    int idx = (int)blockIdx.x;
    if (idx < n_dkv) {
        const int part = idx % p.qsplit;
        idx /= p.qsplit;
        attn_bwd_body<BWD_DKV>(tmQ, tmK, tmV, tmdO, tmDV, tmDK, p, idx % nkb, (idx / nkb) % p.H, idx / (nkb * p.H), part);
    } else {
        idx -= n_dkv;
        attn_bwd_body<BWD_DQ>(tmQ, tmK, tmV, tmdO, tmDQ, tmDQ, p, idx % nqb, (idx / nqb) % p.H, idx / (nqb * p.H), 0);
    }
}

}  // namespace kb
