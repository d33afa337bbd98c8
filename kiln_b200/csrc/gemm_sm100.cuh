// fp16 GEMM for the projections around attention on sm_100a: C = epilogue(A[M,K] * W[N,K]^T), fp32 accumulation
// in TMEM, TMA-fed tcgen05 MMAs, persistent CTAs with two accumulator buffers so that the epilogue of one tile runs
// under the main loop of the next.
//
// Two shapes of the same kernel. PAIR: two CTAs of a cluster share one 256x256 tile through cta_group::2 MMAs; each
// loads its own 128 rows of A and 128 of the 256 W rows per 64-wide k step (32 KiB) and keeps its 128x256 half of the
// accumulator, so a CTA moves half the shared-memory bytes per flop of the single-CTA shape. That matters because
// measured on B200 a 128x128 single-CTA tile is bound by shared-memory bandwidth (TMA writes plus operand reads,
// about 100 B/clk/SM), not by the tensor pipe. Single: one CTA per 128x128 tile, for M <= 128 or when the pair shapes would
// fill the device worse, and where N is no multiple of 256 and the k range is short (the host decides).
//
// NARROW: the same pair on 224 or 192 columns, of any N, where that fills the rounds of tiles better (gemm_shape in routes.h has the rule and
// both sides measured). Each CTA then loads 112 or 96 W rows per k step, and a tile leaves in chunks of 32 columns: one fp32 box of 128-byte rows,
// or one fp16 box of 64-byte rows. Not for the head epilogue, whose tiles are whole heads.
//
// Split K (p.split_k = 2 or 4): with fewer tiles than half of the SMs the k steps of a tile are cut into split_k ranges, one CTA (or
// pair) each, all of a tile in one cluster. Every CTA leaves the accumulator rows that it does not finish in its own shared memory
// (the operand ring, which is free by then); after a cluster barrier the CTA that owns a quarter (split_k = 4) or a half of the rows
// adds the others' parts from there, in a fixed order, and runs the epilogue on them. No scratch memory, no atomics.
//
// It takes the place of the reference's fp16-activation GEMM tc16::k_gemm16 (engine/src/tcgemm16.cuh:57-175,
// host wrapper linear16 at engine/src/kernels.cu:559-609) with its four epilogues — fp32 store, fp16 store,
// fp16 GELU, gated add into the fp32 residual stream (engine/src/tcgemm16.cuh:145-174) — and adds a fifth that the
// attention path wants: EPI_HEADS16 treats every 128 output columns as one attention head and applies the
// per-head RMSNorm (engine/src/kernels.cu:656-666) and rotate-half RoPE (engine/src/kernels.cu:759-772) to the
// accumulator row before storing fp16 (how the epilogue warps share that work is described at the code). With it the
// Q and K projections emit exactly what the attention kernel consumes, and the separate rmsnorm / rope_half launches
// and the staging pre-pass disappear. Up to three weight matrices can share one launch (q, k, v of one activation).
// Outputs leave through TMA stores, the residual epilogue through a TMA reduce-add.
// (The reference accumulates each 32-wide k tile in fp16 before flushing to fp32; here every product is
// accumulated in fp32.)
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math.h>

#include "attn_sm100.cuh"   // pack16, ST_TIMEOUT
#include "ptx.cuh"

namespace kb {

constexpr int EPI_F32 = 0, EPI_F16 = 1, EPI_GELU16 = 2, EPI_RESID = 3, EPI_HEADS16 = 4;

constexpr int GB_M = 128;                                  // accumulator rows per CTA (TMEM lanes)
constexpr int GB_K = 64;                                   // k step: one 128-byte swizzle atom of fp16
constexpr int G_STAGE_BYTES = (GB_M + 128) * GB_K * 2;     // 32 KiB: this CTA's A rows then its W rows, each [128][64] fp16
// k steps in flight: 5 next to the head epilogue, whose warps turn 32 rows x 64 fp32 through shared memory, 6 next to the others, which stage
// one box at a time. A step takes the tensor pipe 0.2-0.3 us and its tiles come from L2 or HBM, a microsecond away. Measured on B200 with 3,
// 4, 5 stages (8 KB of staging per warp), 6 (4 KB): N 8192, K 2048, M 3456 (fp16) 100.7, 89.3, 85.1, 84.0 us, with GELU 107.7, 97.2, 92.5, 90.4;
// N 2048, K 8192 (residual), M 3456 114.2, 101.2, 94.2, 92.9, M 1536 -, 45.3, 40.2, 38.6; K 2048, M 1536 14.6, 14.7 with 5 and 6.
constexpr int G_MAX_STAGES = 6;
__host__ __device__ constexpr int g_stages(int epi) { return epi == EPI_HEADS16 ? 5 : 6; }
constexpr int G_EPI_WARPS = 8;                             // two per TMEM lane quarter, each taking every other column chunk
constexpr int G_THREADS = 32 * (G_EPI_WARPS + 4);          // warps 0-7 epilogue; third warpgroup: warp 8 MMA issue, warp 9 TMA loads, two idle
constexpr int G_GROUP_M = 8;                               // row tiles per raster group (engine/src/tcgemm16.cuh:18)
__host__ __device__ constexpr int g_staging_warp(int epi) { return epi == EPI_HEADS16 ? 8192 : 4096; }   // output being re-ordered, per epilogue warp
constexpr int G_SMEM = 6 * G_STAGE_BYTES + G_EPI_WARPS * 4096 + 2048 + 1024;   // = 227 KiB with the alignment slack, the same for every epilogue:
static_assert(g_stages(EPI_HEADS16) * G_STAGE_BYTES + G_EPI_WARPS * g_staging_warp(EPI_HEADS16) == g_stages(EPI_F32) * G_STAGE_BYTES + G_EPI_WARPS * g_staging_warp(EPI_F32), "ring and staging");

struct GemmParams {
    void* C;
    int ldc;
    int M, N, K;
    // Second product (LoRA side path, engine/src/tcgemm16.cuh:26-28): the accumulator of segment s also takes
    // A2_s[M, K2_s] * W2_s[N, K2_s]^T, as further k steps after the first product's, so every epilogue sees the sum.
    // K2 = 0: none. A last partial k step reads zeros past column K2 (the tensor maps fill out-of-range elements).
    int K2[3];
    int split_k;                   // CTAs (pairs) that share a tile's k steps: 1, 2, or 4 (not PAIR). > 1: one tile per cluster
    int tiles_m, tiles_n;          // in tiles of the launched shape (256x256 for PAIR, 128x128 otherwise)
    // Up to three weight matrices [N, K] share one launch (the q, k, v projections of one activation): column tile tn
    // belongs to segment tn / tiles_n_seg, which has its own W and C tensor maps and its own head epilogue settings.
    int tiles_n_seg;               // column tiles per segment (= tiles_n for a single matrix)
    const float* gate;             // EPI_RESID: C[r, c] += gate[c] * acc (null = 1)
    const __nv_bfloat16* head_w[3];   // EPI_HEADS16: RMSNorm weight[128] of the segment, or null
    int rope_on[3];                // EPI_HEADS16: the segment's heads are rotated (tables below)
    const float* rope_cos;         // EPI_HEADS16: tables [rope_T, 64] or null; row r uses table row r % rope_T
    const float* rope_sin;
    int rope_T;
    float eps;
    uint32_t* status;
};

struct alignas(64) GemmMaps {
    CUtensorMap w[3];              // per segment: the weight matrix, box 64 columns x 128 rows
    CUtensorMap c[3];              // per segment: the output, box as the epilogue stores it
    CUtensorMap a2[3];             // per segment: left operand [M, K2] of the second product (unused when K2 = 0)
    CUtensorMap w2[3];             // per segment: right operand [N, K2] of the second product
};

enum { GBAR_FULL = 0, GBAR_EMPTY = G_MAX_STAGES, GBAR_ACC_FULL = 2 * G_MAX_STAGES, GBAR_ACC_EMPTY = 2 * G_MAX_STAGES + 2, GBAR_COUNT = 2 * G_MAX_STAGES + 4 };

// v Phi(v) (engine/src/tcgemm16.cuh:55 takes erff) without the cancellation of 1 + erf in the negative tail and at half the instructions:
// with a = |v|, erfc(a / sqrt 2) = 2^(-a Q(a)) and v Phi(v) = (v + |v| - a 2^(-a Q(a))) / 2. Q is a polynomial fitted to
// -log2(erfc(a / sqrt 2)) / a on [0, 7] by weighted least squares (beyond 7 the term is below 1e-11, and Q is taken at 7); the weights were not
// kept, a^2 erfc(a / sqrt 2) + 1e-4 a on 2000 Chebyshev nodes gives a polynomial with the same errors. Against float64 over
// N(0,1) and [-9, 9] in fp32: rel. 2-norm 2.8e-8 and 1.3e-8, largest error 2.4e-7 (0.5 v (1 + erff): 3.8e-8, 1.8e-8, 4.5e-7); rounded to fp16 the same.
// Up-projection of 3456 rows, N 8192, K 2048, inside a CUDA graph: 91.4 -> 87.9 us (84.8 without any GELU).
__device__ __forceinline__ float gelu(float v) {
    const float a = fminf(fabsf(v), 7.f);
    float q = -2.5095840960887017e-09f;
    q = fmaf(q, a, 9.659256505756275e-08f);
    q = fmaf(q, a, -1.6297367437800858e-06f);
    q = fmaf(q, a, 1.5769759556860663e-05f);
    q = fmaf(q, a, -9.427715122001246e-05f);
    q = fmaf(q, a, 3.198326739948243e-04f);
    q = fmaf(q, a, -5.3875570301897824e-05f);
    q = fmaf(q, a, -6.906468421220779e-03f);
    q = fmaf(q, a, 5.242638662457466e-02f);
    q = fmaf(q, a, 0.4592227637767792f);
    q = fmaf(q, a, 1.151104211807251f);
    return 0.5f * ((v + fabsf(v)) - a * ex2(-(q * a)));
}

// tile w -> (row tile, column tile): groups of G_GROUP_M row tiles x every column tile, column-major inside a group, so
// the CTAs running at the same time share weight tiles in L2 (engine/src/tcgemm16.cuh:66-69)
__device__ __forceinline__ void gemm_tile(int w, const GemmParams& p, int& tm, int& tn) {
    const int per_group = G_GROUP_M * p.tiles_n;
    const int first = (w / per_group) * G_GROUP_M, gsz = min(p.tiles_m - first, G_GROUP_M), in_g = w % per_group;
    tm = first + in_g % gsz;
    tn = in_g / gsz;
}

// dst[r * ld + col0 + c] = fp16(scale * src[r, c]) for a bf16 LoRA matrix [rows, cols]: how the stacked operands of the
// second product are laid out, with the LoRA's scale folded into its up-projection (engine/src/kernels.cu:548-554)
__global__ void lora_pack_kernel(__half* dst, int ld, int col0, const __nv_bfloat16* src, int rows, int cols, float scale) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)rows * cols) return;
    const int r = (int)(i / cols), c = (int)(i % cols);
    dst[(size_t)r * ld + col0 + c] = __float2half_rn(scale * __bfloat162float(src[i]));
}

template <int EPI, bool PAIR, bool SPLIT, int BN = PAIR ? 256 : 128>
__global__ void __launch_bounds__(G_THREADS, 1)
gemm16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ GemmMaps maps, const GemmParams p) {
    static_assert(BN == (PAIR ? 256 : 128) || (PAIR && !SPLIT && EPI != EPI_HEADS16 && BN % 32 == 0 && BN < 256), "tile width");
    constexpr int BUF_COLS = PAIR ? 256 : 128;                            // TMEM columns from one accumulator buffer (BN of them used) to the next
    constexpr int W_ROWS = PAIR ? BN / 2 : BN;                            // W rows this CTA loads per k step
    constexpr uint32_t STAGE_TX = (GB_M + W_ROWS) * GB_K * 2;             // bytes of a stage in use
    constexpr int TILE_M = PAIR ? 256 : 128;                              // tile rows over the CTA group
    constexpr bool OUT32 = (EPI == EPI_F32 || EPI == EPI_RESID);
    constexpr bool NARROW = BN != BUF_COLS;
    // Columns per output chunk, which leaves as one or two boxes of 32 rows: 128-byte rows, or 64-byte rows where 64 16-bit columns do not
    // divide the tile. Every epilogue warp has a chunk: it has to hand its share of the accumulator back.
    constexpr int CW = NARROW ? 32 : OUT32 || !PAIR ? 64 : 128;
    constexpr int NCH = BN / CW, BOX_COLS = OUT32 || NARROW ? 32 : 64, BOXES = CW / BOX_COLS, BOX_BYTES = 32 * BOX_COLS * (OUT32 ? 4 : 2);
    static_assert(NCH >= 2, "a chunk for both warps of a lane quarter");
    constexpr int G_STAGES = g_stages(EPI), STAGING_WARP = g_staging_warp(EPI);
    constexpr uint32_t TMEM_COLS = 2 * BUF_COLS;

    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* const smem = smem_raw + (base - raw);
    const uint32_t sRing = base;
    uint8_t* const stage_out = smem + G_STAGES * G_STAGE_BYTES;
    uint8_t* const ctrl = stage_out + G_EPI_WARPS * STAGING_WARP;
    const uint32_t bars = sRing + G_STAGES * G_STAGE_BYTES + G_EPI_WARPS * STAGING_WARP;
    uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(ctrl + 512);
    volatile uint32_t* const abort_flag = reinterpret_cast<volatile uint32_t*>(ctrl + 516);
    auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int S = SPLIT ? p.split_k : 1;
    const uint32_t crank = (PAIR || SPLIT) ? cluster_ctarank() : 0u;
    const uint32_t rank = PAIR ? crank & 1u : 0u;                         // 0 issues the MMAs
    const uint32_t lead = crank - rank;                                   // the issuing CTA of this pair
    const int part = PAIR ? (int)(crank >> 1) : (int)crank;               // which range of the k steps
    const int group = (int)blockIdx.x / ((PAIR ? 2 : 1) * S);
    const int n_groups = (int)gridDim.x / ((PAIR ? 2 : 1) * S);
    // split K: the part that finishes a lane quarter, and the others' share of its accumulator ([column / 4][row][4] in their rings)
    auto owner = [&](int quarter) { return S == 4 ? quarter : S == 2 ? quarter >> 1 : 0; };
    auto add_parts = [&](float (&v)[32], int col, int row) {
        for (int o = 0; o < S; o++) {
            if (o == part) continue;
            const uint32_t src = mapa_u32(sRing, (uint32_t)o * (PAIR ? 2u : 1u) + rank) + (uint32_t)((col >> 2) * GB_M + row) * 16u;
#pragma unroll
            for (int e = 0; e < 8; e++) {
                const float4 x = ld_cluster_v4(src + (uint32_t)(e * GB_M * 16));
                v[4 * e] += x.x; v[4 * e + 1] += x.y; v[4 * e + 2] += x.z; v[4 * e + 3] += x.w;
            }
        }
    };
    // split K, all epilogue warps: leave what other parts finish in the ring, meet them; true if this warp has rows to finish
    auto exchange_parts = [&](uint32_t acc, int quarter, int half, bool ok) {
        if (ok && owner(quarter) != part) {
#pragma unroll 1
            for (int col = half * (BN / 2); col < (half + 1) * (BN / 2); col += 32) {
                uint32_t a[32];
                tmem_ld32(acc + (uint32_t)col, a);
                tmem_wait_ld();
                reg_fence32(a);
#pragma unroll
                for (int e = 0; e < 8; e++)
                    *reinterpret_cast<uint4*>(smem + ((col >> 2) + e) * (GB_M * 16) + (quarter * 32 + (threadIdx.x & 31)) * 16) =
                        make_uint4(a[4 * e], a[4 * e + 1], a[4 * e + 2], a[4 * e + 3]);
            }
        }
        __syncwarp();
        cluster_arrive();
        cluster_wait();
        return ok && owner(quarter) == part;
    };
    const int n_tiles = p.tiles_m * p.tiles_n, ksteps1 = p.K / GB_K;

    if (tid == 0) {
        for (int i = 0; i < GBAR_COUNT; i++) mbar_init(bar(i), (i >= GBAR_ACC_EMPTY) ? (PAIR ? 2u : 1u) * G_EPI_WARPS : 1u);   // acc_empty: one arrival per epilogue warp of the group
        *abort_flag = 0u;
        mbar_fence_init();
        fence_proxy_async_smem();
    }
    if (warp == G_EPI_WARPS + 1 && lane == 0) { tma_prefetch_desc(&tmA); tma_prefetch_desc(&maps.w[0]); tma_prefetch_desc(&maps.c[0]); }
    if (warp == G_EPI_WARPS) {
        tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);                       // two accumulator buffers
        tmem_relinquish();
    }
    pdl_launch();
    tc_fence_before();
    if (PAIR) { cluster_arrive(); cluster_wait(); } else __syncthreads();
    tc_fence_after();
    static_assert(!PAIR || TMEM_COLS == TMEM_ALL_COLUMNS, "a pair's accumulators are addressed from column 0");
    const uint32_t tmem_base = PAIR ? 0u : *tmem_slot;                    // see elect_one
    pdl_wait();

    if (warp < G_EPI_WARPS) {
        // the row buffers of the epilogue live in registers; -Xptxas -v reports spills for the cut k ranges only (single CTAs 12 bytes of
        // stores and 48 of loads, pairs with the head epilogue 12 and 8)
        setmaxnreg_inc<224>();
        // ------------------------------------------------------------------ epilogue: one output row per thread
        if constexpr (EPI == EPI_HEADS16) {
            // The two warps of a TMEM lane quarter split every head by RoPE half: warp half hs owns columns [32 hs, +32) and
            // their rotation partners [64 + 32 hs, +32). A thread normalises its row of the accumulator, the warp turns its
            // 32 rows x 64 values through shared memory, and the rotation runs after the turn, one (i, i + 64) pair per
            // lane per row: there a table row is one coalesced 128-byte read (measured: reading the tables in the
            // thread-per-row layout, 32 different lines per instruction, cost 4 us per tile). The 32 + 32 table values of
            // a lane are loaded once per tile, before the accumulator is waited for, and serve both heads of the tile.
            constexpr int NH = BN / 128;
            const int quarter = warp & 3, hs = warp >> 2;
            const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
            uint8_t* const my_stage = stage_out + warp * 32 * 256;        // 32 rows x 64 fp32, written and re-read by this warp only
            float* const ss_buf = reinterpret_cast<float*>(ctrl + 1024) + quarter * 64;
            volatile uint32_t* const ok_buf = reinterpret_cast<volatile uint32_t*>(ctrl + 640) + quarter * 2;
            const int pair_bar = 1 + quarter;
            uint4 w0[4], w1[4];                                           // RMSNorm weights of this warp's 32 + 32 columns (bf16)
            int w_seg = -1;                                               // segment they belong to
            uint32_t use[2] = {0, 0};
            int k = 0;
            for (int w = group; w < n_tiles; w += n_groups, ++k) {
                const int buf = k & 1;
                int tm, tn;
                gemm_tile(w, p, tm, tn);
                const int seg = tn / p.tiles_n_seg;
                const int m0 = tm * TILE_M + (int)rank * GB_M, n0 = (tn - seg * p.tiles_n_seg) * BN;
                const int row0 = m0 + quarter * 32;
                const int nrow = p.M - row0;
                const __nv_bfloat16* const head_w = seg == 0 ? p.head_w[0] : seg == 1 ? p.head_w[1] : p.head_w[2];
                const bool rope = (seg == 0 ? p.rope_on[0] : seg == 1 ? p.rope_on[1] : p.rope_on[2]) != 0;
                if (head_w && seg != w_seg) {                             // L1 hits after the first tile of a segment
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        w0[q] = reinterpret_cast<const uint4*>(head_w + hs * 32)[q];
                        w1[q] = reinterpret_cast<const uint4*>(head_w + 64 + hs * 32)[q];
                    }
                    w_seg = seg;
                }
                float cr[32], sr[32];
                if (rope) {
                    int tr = min(row0, p.M - 1) % p.rope_T;
#pragma unroll
                    for (int rr = 0; rr < 32; rr++) {
                        cr[rr] = p.rope_cos[(size_t)tr * 64 + hs * 32 + lane];
                        sr[rr] = p.rope_sin[(size_t)tr * 64 + hs * 32 + lane];
                        if (row0 + rr + 1 < p.M) tr = (tr + 1 == p.rope_T) ? 0 : tr + 1;
                    }
                }
                bool ok = __all_sync(0xffffffffu, mbar_wait(bar(GBAR_ACC_FULL + buf), use[buf] & 1u, abort_flag));
                ++use[buf];
                if (lane == 0) ok_buf[hs] = ok ? 1u : 0u;                 // leave only together: the pair meets at named barriers below
                named_bar_sync(pair_bar, 64);
                ok = ok_buf[0] != 0u && ok_buf[1] != 0u;
                named_bar_sync(pair_bar, 64);
                if (SPLIT) {
                    tc_fence_after();
                    ok = exchange_parts(tmem_base + lane_base + (uint32_t)(buf * BUF_COLS), quarter, hs, ok);
                }
                if (!ok) break;
                tc_fence_after();
#pragma unroll 1
                for (int h = 0; h < NH; h++) {
                    float x0[32], x1[32];
                    {
                        uint32_t a0[32], a1[32];
                        tmem_ld32(tmem_base + lane_base + (uint32_t)(buf * BUF_COLS + h * 128 + hs * 32), a0);
                        tmem_ld32(tmem_base + lane_base + (uint32_t)(buf * BUF_COLS + h * 128 + 64 + hs * 32), a1);
                        tmem_wait_ld();
                        reg_fence32(a0);
                        reg_fence32(a1);
#pragma unroll
                        for (int e = 0; e < 32; e++) { x0[e] = __uint_as_float(a0[e]); x1[e] = __uint_as_float(a1[e]); }
                    }
                    if (SPLIT) {
                        add_parts(x0, h * 128 + hs * 32, quarter * 32 + lane);
                        add_parts(x1, h * 128 + 64 + hs * 32, quarter * 32 + lane);
                    }
                    if (h == NH - 1) {                                    // this warp's share of the accumulator is in registers
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) {
                            if (PAIR && rank != 0) mbar_arrive_cluster(mapa_u32(bar(GBAR_ACC_EMPTY + buf), lead));
                            else mbar_arrive(bar(GBAR_ACC_EMPTY + buf));
                        }
                    }
                    if (head_w) {                                         // engine/src/kernels.cu:656-666
                        float ss = 0.f;
#pragma unroll
                        for (int e = 0; e < 32; e++) ss = fmaf(x0[e], x0[e], fmaf(x1[e], x1[e], ss));
                        ss_buf[hs * 32 + lane] = ss;
                        named_bar_sync(pair_bar, 64);
                        const float rs = rsqrtf((ss + ss_buf[(hs ^ 1) * 32 + lane]) * (1.f / 128.f) + p.eps);
                        named_bar_sync(pair_bar, 64);                     // both sums are read before the next head overwrites them
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            const uint32_t d0[4] = {w0[q].x, w0[q].y, w0[q].z, w0[q].w}, d1[4] = {w1[q].x, w1[q].y, w1[q].z, w1[q].w};
#pragma unroll
                            for (int m = 0; m < 4; m++) {                 // a bf16 is the top half of an fp32
                                x0[8 * q + 2 * m] = x0[8 * q + 2 * m] * rs * __uint_as_float(d0[m] << 16);
                                x0[8 * q + 2 * m + 1] = x0[8 * q + 2 * m + 1] * rs * __uint_as_float(d0[m] & 0xffff0000u);
                                x1[8 * q + 2 * m] = x1[8 * q + 2 * m] * rs * __uint_as_float(d1[m] << 16);
                                x1[8 * q + 2 * m + 1] = x1[8 * q + 2 * m + 1] * rs * __uint_as_float(d1[m] & 0xffff0000u);
                            }
                        }
                    }
                    if (lane == 0) tma_store_wait_read();                 // the boxes of the last head have left shared memory
                    __syncwarp();
                    uint8_t* const my_row = my_stage + lane * 256;
#pragma unroll
                    for (int j = 0; j < 8; j++) {                         // 16-byte pieces j (first half) and 8 + j (partners), XOR-swizzled by row
                        *reinterpret_cast<float4*>(my_row + ((j ^ (lane & 15)) << 4)) = make_float4(x0[4 * j], x0[4 * j + 1], x0[4 * j + 2], x0[4 * j + 3]);
                        *reinterpret_cast<float4*>(my_row + (((8 + j) ^ (lane & 15)) << 4)) = make_float4(x1[4 * j], x1[4 * j + 1], x1[4 * j + 2], x1[4 * j + 3]);
                    }
                    __syncwarp();
                    uint32_t pk[32];
#pragma unroll
                    for (int rr = 0; rr < 32; rr++) {
                        const uint8_t* src = my_stage + rr * 256 + (lane & 3) * 4;
                        float a = *reinterpret_cast<const float*>(src + (((lane >> 2) ^ (rr & 15)) << 4));
                        float b = *reinterpret_cast<const float*>(src + (((8 + (lane >> 2)) ^ (rr & 15)) << 4));
                        if (rope) {                                       // engine/src/kernels.cu:769-771
                            const float ra = a * cr[rr] - b * sr[rr];
                            b = b * cr[rr] + a * sr[rr];
                            a = ra;
                        }
                        const float other = __shfl_xor_sync(0xffffffffu, (lane & 1) ? a : b, 1);
                        pk[rr] = (lane & 1) ? pack16<DT_F16>(other, b) : pack16<DT_F16>(a, other);
                    }
                    // back into shared memory as two 32-row x 64-byte boxes (first half, partners), which leave by TMA
                    __syncwarp();
                    uint8_t* const my_out = my_stage + (lane & 1) * 2048 + (lane >> 1) * 4;
#pragma unroll
                    for (int rr = 0; rr < 32; rr++) *reinterpret_cast<uint32_t*>(my_out + rr * 64) = pk[rr];
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0 && nrow > 0) {
                        const int x = n0 + h * 128 + hs * 32;
                        tma_store_3d(&maps.c[seg], smem_u32(my_stage), x, row0, 0);
                        tma_store_3d(&maps.c[seg], smem_u32(my_stage) + 2048, x + 64, row0, 0);
                        tma_store_commit();
                    }
                }
            }
            if (lane == 0) tma_store_wait_read();
        } else {
            const int quarter = warp & 3, chunk0 = warp >> 2;                // TMEM lanes [32 quarter, +32); chunks chunk0, chunk0 + 2, ...
            const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
            constexpr int SLOTS = STAGING_WARP / BOX_BYTES;                  // boxes on their way out at a time
            static_assert(SLOTS == 1 || SLOTS == 2, "");
            uint8_t* const my_stage = stage_out + warp * STAGING_WARP;
            uint32_t use[2] = {0, 0};
            int k = 0, box_use = 0;
            for (int w = group; w < n_tiles; w += n_groups, ++k) {
                const int buf = k & 1;
                int tm, tn;
                gemm_tile(w, p, tm, tn);
                const int seg = tn / p.tiles_n_seg;
                const int m0 = tm * TILE_M + (int)rank * GB_M, n0 = (tn - seg * p.tiles_n_seg) * BN;
                bool ok = __all_sync(0xffffffffu, mbar_wait(bar(GBAR_ACC_FULL + buf), use[buf] & 1u, abort_flag));
                ++use[buf];
                if (SPLIT) {
                    tc_fence_after();
                    ok = exchange_parts(tmem_base + lane_base + (uint32_t)(buf * BUF_COLS), quarter, chunk0, ok);
                }
                if (!ok) break;                                               // warps are independent from here on
                tc_fence_after();
                const int nrow = p.M - (m0 + quarter * 32);                      // rows of this warp inside the matrix
#pragma unroll 1
                for (int ch = chunk0; ch < NCH; ch += 2) {
                    float v[CW];
                    {
                        uint32_t a[CW / 32][32];
#pragma unroll
                        for (int q = 0; q < CW / 32; q++) tmem_ld32(tmem_base + lane_base + (uint32_t)(buf * BUF_COLS + ch * CW + 32 * q), a[q]);
                        tmem_wait_ld();
#pragma unroll
                        for (int q = 0; q < CW / 32; q++) {
                            reg_fence32(a[q]);
#pragma unroll
                            for (int e = 0; e < 32; e++) v[32 * q + e] = __uint_as_float(a[q][e]);
                        }
                    }
                    if (SPLIT) {
#pragma unroll
                        for (int q = 0; q < CW / 32; q++) {
                            float x[32];
#pragma unroll
                            for (int e = 0; e < 32; e++) x[e] = v[32 * q + e];
                            add_parts(x, ch * CW + 32 * q, quarter * 32 + lane);
#pragma unroll
                            for (int e = 0; e < 32; e++) v[32 * q + e] = x[e];
                        }
                    }
                    if (ch + 2 >= NCH) {                                      // this warp's last chunk is in registers: the MMA warp may reuse it
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) {
                            if (PAIR && rank != 0) mbar_arrive_cluster(mapa_u32(bar(GBAR_ACC_EMPTY + buf), lead));
                            else mbar_arrive(bar(GBAR_ACC_EMPTY + buf));
                        }
                    }
                    if constexpr (EPI == EPI_GELU16) {
#pragma unroll
                        for (int c = 0; c < CW; c++) v[c] = gelu(v[c]);
                    }
                    if constexpr (EPI == EPI_RESID) {
                        if (p.gate && n0 + ch * CW < p.N) {
#pragma unroll
                            for (int c = 0; c < CW; c += 4) {
                                const float4 gt = *reinterpret_cast<const float4*>(p.gate + n0 + ch * CW + c);
                                v[c] *= gt.x; v[c + 1] *= gt.y; v[c + 2] *= gt.z; v[c + 3] *= gt.w;
                            }
                        }
                    }
                    // The 32 rows of the chunk go through shared memory as swizzled boxes and leave by TMA (measured: 32 row stores per
                    // warp took 3 us, the issue rate of plain global stores from eight warps; the bulk copy takes them off the warp).
                    // Behind the last tile the ring is free, of a cut k range (one tile per CTA) beyond what the other parts read there: a place
                    // for every box of the warp, and nobody waits for one to be read. Of a pair with a cut range half of the warps finish rows.
                    // (The cut ranges through the staging area, residual, N 2048, back to back: K 2048, M 128 9.2 us, here 9.0, M 300 9.9 -> 9.6,
                    // M 384 9.9 -> 9.6; K 8192, M 1024, pairs, 37.0 -> 36.6.)
                    const bool in_ring = SPLIT || w + n_groups >= n_tiles;
                    constexpr int READ_BY_PARTS = SPLIT ? BN / 4 * GB_M * 16 : 0;
                    static_assert(READ_BY_PARTS + (SPLIT && PAIR ? 4 : 8) * 4 * 4096 <= G_STAGES * G_STAGE_BYTES, "four places per warp");
                    const uint32_t place = READ_BY_PARTS + (SPLIT && PAIR ? (warp >> 2) * 2 + (warp & 1) : warp) * 4 * 4096;
#pragma unroll
                    for (int b = 0; b < BOXES; b++) {
                        uint8_t* const box = in_ring ? smem + place + ((ch >> 1) * BOXES + b) * 4096 : my_stage + (SLOTS == 2 ? box_use * BOX_BYTES : 0);
                        if (!in_ring) {
                            if (lane == 0) { if (SLOTS == 2) tma_store_wait_read_1(); else tma_store_wait_read(); }   // the box that was here has been read
                            box_use ^= 1;
                        }
                        __syncwarp();
#pragma unroll
                        for (int c = 0; c < BOX_BYTES / 512; c++) {           // 16-byte pieces of this thread's row
                            uint4 pk;
                            if constexpr (OUT32) {
                                const float* const u = v + b * 32 + 4 * c;
                                pk = make_uint4(__float_as_uint(u[0]), __float_as_uint(u[1]), __float_as_uint(u[2]), __float_as_uint(u[3]));
                            } else {
                                const float* const u = v + b * BOX_COLS + 8 * c;
                                pk.x = pack16<DT_F16>(u[0], u[1]); pk.y = pack16<DT_F16>(u[2], u[3]);
                                pk.z = pack16<DT_F16>(u[4], u[5]); pk.w = pack16<DT_F16>(u[6], u[7]);
                            }
                            if constexpr (BOX_BYTES == 4096) *reinterpret_cast<uint4*>(box + lane * 128 + ((c ^ (lane & 7)) << 4)) = pk;
                            else *reinterpret_cast<uint4*>(box + lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4)) = pk;
                        }
                        fence_proxy_async_smem();
                        __syncwarp();
                        const int x = n0 + ch * CW + b * BOX_COLS, y = m0 + quarter * 32;
                        if (lane == 0) {                                      // an empty group where nothing is stored, so that groups count boxes
                            if (nrow > 0 && x < p.N) {                        // a narrow last column tile stores only the boxes that begin inside it
                                if constexpr (EPI == EPI_RESID) tma_reduce_add_3d(&maps.c[seg], smem_u32(box), x, y, 0);
                                else tma_store_3d(&maps.c[seg], smem_u32(box), x, y, 0);
                            }
                            tma_store_commit();
                        }
                    }
                }
            }
            if (lane == 0) tma_store_wait_read();
        }
    } else if (warp == G_EPI_WARPS) {
        setmaxnreg_dec<56>();
        // ------------------------------------------------------------------ MMA issue (one lane of the group's first CTA)
        if (rank == 0 && elect_one()) {
            constexpr uint32_t IDESC = idesc_f16(0, 0, 0, 0, TILE_M, BN);
            uint32_t ring = 0, use[2] = {0, 0};
            bool good = true;
            int k = 0;
            for (int w = group; w < n_tiles && good; w += n_groups, ++k) {
                const int buf = k & 1;
                // the epilogues have drained this accumulator (passes at once for the first two tiles)
                good = mbar_wait(bar(GBAR_ACC_EMPTY + buf), (use[buf] & 1u) ^ 1u, abort_flag);
                ++use[buf];
                if (!good) break;
                tc_fence_after();
                int tm, tn;
                gemm_tile(w, p, tm, tn);
                const int ksteps = ksteps1 + (p.K2[tn / p.tiles_n_seg] + GB_K - 1) / GB_K;
                const int ks0 = ksteps * part / S, ks1 = ksteps * (part + 1) / S;
                for (int ks = ks0; ks < ks1 && good; ++ks, ++ring) {
                    const uint32_t st = ring % G_STAGES;
                    good = mbar_wait(bar(GBAR_FULL + st), (ring / G_STAGES) & 1u, abort_flag);
                    if (!good) break;
                    tc_fence_after();
                    const uint32_t a_s = sRing + st * G_STAGE_BYTES;
                    const uint64_t adesc = smem_desc_sw128(a_s, 16, 1024), wdesc = smem_desc_sw128(a_s + GB_M * GB_K * 2, 16, 1024);
#pragma unroll
                    for (int kk = 0; kk < 4; kk++) {
                        const uint32_t acc = (ks > ks0 || kk > 0) ? 1u : 0u;
                        if (PAIR) mma_ss_pair(tmem_base + (uint32_t)(buf * BUF_COLS), adesc + (uint64_t)(kk * 2), wdesc + (uint64_t)(kk * 2), IDESC, acc);
                        else mma_ss(tmem_base + (uint32_t)(buf * BUF_COLS), adesc + (uint64_t)(kk * 2), wdesc + (uint64_t)(kk * 2), IDESC, acc);
                    }
                    if (PAIR) tc_commit_pair(bar(GBAR_EMPTY + st), (uint16_t)(3u << lead)); else tc_commit(bar(GBAR_EMPTY + st));
                }
                if (good) {
                    if (PAIR) tc_commit_pair(bar(GBAR_ACC_FULL + buf), (uint16_t)(3u << lead)); else tc_commit(bar(GBAR_ACC_FULL + buf));
                }
            }
        }
        __syncwarp();
        if (SPLIT) { cluster_arrive(); cluster_wait(); }                  // the barrier of exchange_parts
    } else {
        setmaxnreg_dec<56>();
        // ------------------------------------------------------------------ TMA loads (one lane of every CTA)
        if (warp == G_EPI_WARPS + 1 && elect_one()) {
            uint32_t ring = 0;
            bool good = true;
            for (int w = group; w < n_tiles && good; w += n_groups) {
                int tm, tn;
                gemm_tile(w, p, tm, tn);
                const int seg = tn / p.tiles_n_seg;
                const int m0 = tm * TILE_M + (int)rank * GB_M, wrow0 = (tn - seg * p.tiles_n_seg) * BN + (int)rank * W_ROWS;
                const int ksteps = ksteps1 + (p.K2[seg] + GB_K - 1) / GB_K;
                const int ks1 = ksteps * (part + 1) / S;
                for (int ks = ksteps * part / S; ks < ks1 && good; ++ks, ++ring) {
                    const bool second = ks >= ksteps1;                    // the k steps of the second product follow the first's
                    const CUtensorMap* const tmL = second ? &maps.a2[seg] : &tmA;
                    const CUtensorMap* const tmW = second ? &maps.w2[seg] : &maps.w[seg];
                    const int k0 = (second ? ks - ksteps1 : ks) * GB_K;
                    const uint32_t st = ring % G_STAGES;
                    good = mbar_wait(bar(GBAR_EMPTY + st), ((ring / G_STAGES) & 1u) ^ 1u, abort_flag);
                    if (!good) break;
                    const uint32_t a_s = sRing + st * G_STAGE_BYTES;
                    if (PAIR) {
                        // both CTAs' bytes complete on the issuing CTA's barrier
                        if (rank == 0) mbar_expect_tx(bar(GBAR_FULL + st), 2 * STAGE_TX);
                        const uint32_t fb = mapa_u32(bar(GBAR_FULL + st), lead);
                        tma_load_3d_pair(a_s, tmL, fb, k0, m0, 0);
                        tma_load_3d_pair(a_s + GB_M * GB_K * 2, tmW, fb, k0, wrow0, 0);
                    } else {
                        mbar_expect_tx(bar(GBAR_FULL + st), G_STAGE_BYTES);
                        tma_load_3d(a_s, tmL, bar(GBAR_FULL + st), k0, m0, 0);
                        tma_load_3d(a_s + GB_M * GB_K * 2, tmW, bar(GBAR_FULL + st), k0, wrow0, 0);
                    }
                }
            }
            if (!good || *abort_flag) {
                // let the copies already requested land before the memory goes away: a bounded wait on the FULL barrier of every
                // stage with a request outstanding. In a pair those barriers live in the first CTA; the second one cannot poll
                // them and waits a fixed 20 us instead (both then meet at the cluster barrier below).
                if (!PAIR || rank == 0) {
                    for (uint32_t k = ring > (uint32_t)G_STAGES ? ring - G_STAGES : 0u; k < ring; ++k) drain_wait(bar(GBAR_FULL + k % G_STAGES), (k / G_STAGES) & 1u);
                } else {
                    const uint64_t t0 = globaltimer_ns();
                    while (globaltimer_ns() - t0 < 20000ull) {}
                }
            }
        }
        __syncwarp();
        if (SPLIT) { cluster_arrive(); cluster_wait(); }                  // the barrier of exchange_parts
    }
    tc_fence_before();
    if (PAIR || SPLIT) { cluster_arrive(); cluster_wait(); } else __syncthreads();   // split K: nobody leaves while its ring is read
    if (warp == G_EPI_WARPS) {
        if (lane == 0 && *abort_flag) atomicOr(p.status, ST_TIMEOUT);
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

}  // namespace kb
