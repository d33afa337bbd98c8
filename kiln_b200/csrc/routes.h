// Which schedule an attention call takes, how its backward cuts query ranges, which tile shape a GEMM takes and what a thread block of the
// pre-pass: rules on sizes only, plain host code (no CUDA headers), so that they can be tested without a device.
#pragma once
#include <stddef.h>
#include <stdint.h>

#ifdef __CUDACC__
#define KB_HOST_DEVICE __host__ __device__   // what the kernels are built from as well
#else
#define KB_HOST_DEVICE
#endif

namespace kb {

#ifndef KB_SPLIT_MARGIN
#define KB_SPLIT_MARGIN 7
#endif
constexpr int ROUTE_TILE = 128;   // query rows per tile, keys per block

// Balanced (item, key block) ranges per SM against whole items per SM, in key-block steps on the slowest SM. Measured on B200
// (4096 / 3456 / 2560 / 2048 / 1536 / 1024 tokens x 16 heads, device time inside a CUDA graph): a key-block step costs ~1.86 us
// and the balanced schedule a fixed ~15 us on top (one more segment to fill and drain per SM, the partial results written and
// merged; the cooperative launch itself measured free): it wins at 2560 and 3456 tokens (63.8 vs 83.5 us, 97.6 vs 111.7 us), ties
// or wins at 4096 (128.2 vs 127.4 us on one GPU, 126.9 vs 140.0 us on another), ties at 2048 and loses at 1536 and 1024 (36.8 vs
// 29.3 us, 28.7 vs 21.3 us). So it is taken when it saves at least eight steps.
inline bool split_pays(int n_items, int nb, int sm_count) {
    const long long steps = (long long)n_items * nb;
    if (nb < 2 || steps < 2LL * sm_count) return false;
    const long long whole = (long long)((n_items + sm_count - 1) / sm_count) * nb;
    const long long balanced = (steps + sm_count - 1) / sm_count + KB_SPLIT_MARGIN;
    return balanced < whole;
}

enum Route { ROUTE_WHOLE, ROUTE_BALANCED, ROUTE_KEYS };

// One 128-row query tile per item with its keys split over both streams (MODE_KEYS), against 256 rows and all keys (MODE_PAIR): a
// candidate while every item has an SM to itself, where it halves the steps of the longest item. It reads every K/V tile twice as
// often (128 KB per step and SM), and in more than one round the balanced or the whole-item schedule is as fast or faster. Measured
// on B200, 16 heads, fp16, device time, whole items -> this: 256 tokens 9.4 -> 6.9 us, 512 12.9 -> 9.4, 1000 20.7 -> 14.9,
// 1152 22.5 -> 15.6; beyond one round 1280 25.1 -> 28.4, 2048 35.3 -> 42.0, 3456 90.0 (balanced) -> 91.4.
//
// With few tiles and many keys the balanced schedule spreads the keys of an item over more SMs than one, at the price of merging
// sm_count / n_items parts. Both in units of 10 ns, fitted to 40 shapes: keys 5.5 us + 1.95 us per step of two blocks; balanced
// 13.5 us (9 with a single query tile, which has one stream) + 1.9 us per block step + 1.8 us per part. Measured, queries x keys x
// heads, balanced / keys: 128 x 16384 x 16 52 / 127 us, 256 x 16384 x 4 88 / 126, 512 x 8192 x 16 51 / 68, 4096 x 4096 x 2
// 35.3 / 36.9; the other way 256 x 4096 x 16 37.6 / 36.0, 1024 x 8192 x 16 73 / 71, 4096 x 4096 x 4 46 / 39, 1024 x 1024 x 16 25 / 15.
//
// room: the workspace holds the balanced schedule's partial results; may_keys: the call has a MODE_KEYS form (no peers).
inline Route attn_route(int B, int Tq, int Tk, int H, int sm_count, bool may_keys, bool room) {
    const int nb = (Tk + ROUTE_TILE - 1) / ROUTE_TILE;
    const int n_items = ((Tq + 2 * ROUTE_TILE - 1) / (2 * ROUTE_TILE)) * H * B, items_keys = ((Tq + ROUTE_TILE - 1) / ROUTE_TILE) * H * B;
    const bool balanced = room && split_pays(n_items, nb, sm_count);
    if (may_keys && nb >= 2 && items_keys <= sm_count) {
        const long long keys_cost = 550 + 195LL * ((nb + 1) / 2);
        const long long balanced_cost = (Tq > ROUTE_TILE ? 1350 : 900) + 190LL * (((long long)n_items * nb + sm_count - 1) / sm_count) + 180LL * sm_count / n_items;
        return balanced && balanced_cost < keys_cost ? ROUTE_BALANCED : ROUTE_KEYS;
    }
    return balanced ? ROUTE_BALANCED : ROUTE_WHOLE;
}

// A row-major matrix in memory, in bytes
struct MatBytes {
    const void* p;
    size_t rows, stride, width;
};
// Do two matrices share a byte? Exact for equal row strides (column slices of one buffer do not); for different ones, whether
// their address ranges meet.
inline bool share_bytes(const MatBytes& x, const MatBytes& y) {
    const MatBytes &lo = (uintptr_t)x.p <= (uintptr_t)y.p ? x : y, &hi = (uintptr_t)x.p <= (uintptr_t)y.p ? y : x;
    const size_t d = (uintptr_t)hi.p - (uintptr_t)lo.p;
    if (d >= (lo.rows - 1) * lo.stride + lo.width) return false;
    if (lo.stride != hi.stride) return true;
    const size_t off = d % lo.stride;
    return off < lo.width || off + hi.width > lo.stride;
}
// May an item read its raw Q tile while other items store their output? Yes if no output byte is a byte of Q, or if every (row,
// head) of the output lies exactly on its own Q, which only the item itself reads.
inline bool q_survives_output(const MatBytes& q, const MatBytes& out) {
    return !share_bytes(q, out) || (q.p == out.p && q.stride == out.stride && q.width == out.width);
}

// Backward: how the dK/dV role cuts its query blocks when there are too few (key block, head, image) triples to fill the GPU
// (cross-attention to a short context): parts of q_per query blocks each; 1 part = no cut.
inline void bwd_qsplit(int B, int Tq, int Tk, int H, int sm_count, int* qsplit, int* q_per) {
    const long long triples = (long long)B * H * ((Tk + 127) / 128);
    const int nqb = (Tq + 127) / 128;
    int want = (int)(sm_count / (triples > 0 ? triples : 1));
    if (want > nqb) want = nqb;
    if (want < 2) { *qsplit = 1; *q_per = nqb; return; }
    *q_per = (nqb + want - 1) / want;
    *qsplit = (nqb + *q_per - 1) / *q_per;
}

// Pre-pass: what a thread block takes. A unit is a warp, or with np = 1 the thread block; it takes prep_heads(np) (row, head) pairs of one row,
// or with few heads those of several rows. np: pieces of eight elements per lane, four of 16 bytes or two of 32; one where all of it is a few
// rows, as a lane with less to do is done sooner (never with RoPE, whose lanes hold two pieces).
// The line between few rows and many, 64 pairs per SM (9472), lies where neither is the better one for long. Measured on B200, back to back,
// many -> one: cross_kv, whose context has 8 heads, 512 rows fp32 10.2 -> 9.9 us, bf16 10.3 -> 9.9, 1024 rows 16.0 -> 15.6, 15.7 -> 15.4, 1184 (here)
// 21.2 -> 20.9, 20.8 -> 20.4, 2368 29.9 -> 30.6, 29.0 -> 28.6, 3000 34.0 -> 33.9, 32.5 -> 33.3; self-attention, 16 heads, three tensors, plain:
// 256 tokens 11.5 -> 11.4, 9.5 -> 9.6, 500 (24000 pairs) 14.4 -> 15.4, 12.3 -> 12.3, 1000 22.9 -> 23.5, 17.3 -> 18.9, 1536 40.7 -> 41.7, 32.7 -> 34.8.
constexpr int PREP_WARPS = 4;
KB_HOST_DEVICE constexpr int prep_units(int np) { return np == 1 ? 1 : PREP_WARPS; }
KB_HOST_DEVICE constexpr int prep_heads(int np) { return np == 1 ? 2 * PREP_WARPS : 2 * np; }
struct PrepLayout {
    int np;
    bool few;          // few heads (qk_prep_few_kernel)
    int heads;         // of a row, in a unit; few: the largest power of two that divides H, so that no lane is idle
    int rows, groups;  // rows of a thread block; thread blocks side by side that take a row's heads
};
// Few: where more than 3/8 of a unit's lanes would be idle, with RoPE 1/2 (there a row's table values serve two of its heads), of a unit of four
// heads 1/4. Measured on B200, back to back, a row to a unit -> few (half a warp per pair, which knows no rows), pre-pass alone, plain: 4096
// rows, 1 head fp32 4.7 -> 1.8 us (2.0), bf16 4.7 -> 1.5 (1.9), 2 heads fp32 4.7 -> 2.0 (2.2), 2048 rows, 4 heads bf16 2.5 -> 1.8 (2.1); RoPE,
// 8192 rows, 2 heads fp32 4.1 -> 3.1 (3.9), bf16 4.9 -> 3.2 (4.0), 5 heads fp32 7.9 -> 6.5 (6.3); the other way RoPE bf16, 4 heads, 512 rows
// 1.8 -> 2.1 (2.1), 4096 rows 3.0 -> 3.2 (3.9). Self-attention, plain, 1 head, 1536 tokens fp32 24.0 -> 20.3 (20.2), 4096 tokens bf16 44.9 -> 38.1
// (38.2), 2 heads, 1000 tokens fp32 18.8 -> 16.6 (16.8).
inline PrepLayout prep_layout(long long pairs, int H, bool in32, bool rope, int sm_count) {
    const int np = rope || pairs >= 64LL * sm_count ? (in32 ? 2 : 4) : 1, all = prep_heads(np), lanes = (H + all - 1) / all * all;
    PrepLayout l = {np, 8 * (lanes - H) > (all == 4 ? 2 : rope ? 4 : 3) * lanes, all, prep_units(np), lanes / all};
    if (l.few) {
        while (H % l.heads) l.heads /= 2;
        l.rows *= all / l.heads;
        l.groups = H / l.heads;
    }
    return l;
}

// GEMM: CTA pairs on 256x256 tiles when that fills the device better. Measured on B200 a CTA of a pair spends about 11/8 of the
// time a single CTA spends per 64-wide k step while doing twice the work, so compare waves x time per step (a step of a single CTA
// = 8 units of ~43 ns). Either shape cuts the k steps of its tiles over `split` CTAs (pairs) of a cluster when all clusters are
// resident at once; leaving, meeting and adding the parts costs about 3 us on single CTAs and 4 us on pairs (half of the warps run
// the epilogue of twice the columns). Measured on B200 inside a CUDA graph, whole k range -> split (* without dependent launches,
// which save 1.5 us): N 2048, K 8192: M 128 40.2* -> 16.3 us, 512 40.8* -> 25.3, 1024 41.6* -> 29.1; N 2048, K 2048: M 128 14.4* -> 9.2,
// 512 15.0* -> 11.0; with M 1024 (pairs, head epilogue) 14.7 -> 17.1, so not taken there. N 96 (a stacked LoRA), K 2048, M 1536: 13.4* -> 10.1.
constexpr int SPLIT_K_COST = 70, SPLIT_K_COST_PAIR = 95;
struct GemmShape {
    bool pair;
    int split;
    int width;   // columns of a tile
};
// The cheapest shape among those with `split` parts (0: any). max_clusters[1], [2]: resident clusters of 2 and 4 CTAs.
inline GemmShape gemm_cheapest(int M, int N, long long ksteps, int n_seg, int split, int sm_count, const int* max_clusters) {
    long long best = -1;
    GemmShape shape = {false, 1, 128};
    for (int pair = 1; pair >= 0; pair--) {
        if (pair && (N % 256 || M <= 128)) continue;
        const int tile = pair ? 256 : 128;
        const long long tiles = (long long)((M + tile - 1) / tile) * ((N + tile - 1) / tile) * n_seg;
        const long long unit = pair ? 11 : 8, groups = pair ? sm_count / 2 : sm_count;
        for (int s = 1; s <= (pair ? 2 : 4); s *= 2) {
            if ((split && s != split) || (s > 1 && (ksteps < 2 * s || tiles > max_clusters[pair ? s : s / 2]))) continue;
            const long long cost = ((tiles + groups - 1) / groups) * ((ksteps + s - 1) / s) * unit + (s == 1 ? 0 : pair ? SPLIT_K_COST_PAIR : SPLIT_K_COST);
            if (best < 0 || cost < best) { best = cost; shape = {pair != 0, s, tile}; }
        }
    }
    return shape;
}

// Narrow tiles: a CTA pair takes 224 or 192 columns where that is faster than the shape above. The cost of a launch whose k range is not cut, in
// units of ~3.9 ns: k steps x time of one x rounds of tiles, a last round that is not full charged six tenths and four tenths of its part (in
// long launches the thread blocks drift apart, and under the power cap time follows the work), and what a pair needs once more than a single
// CTA for twice the rows (1.2 us: filling, a longer epilogue). GELU keeps the epilogue warps of the wide chunks (tiles of 256 and 128 columns)
// busy longer than a k step's share of them, so those steps cost a tenth more. Measured on B200 with all widths forced, inside a CUDA graph, in
// single calls with pauses; sustained the differences grow (GELU, M 4096: 123, 108, 122 us):
//                          N 2048, residual                              N 8192, GELU (K 2048)
//   M       1536  1792  2048  2560  3456  4096   K 8192: 1536  3456     512  1024  2304  3456  3840  4096  8192   F16: 1536  3456  3840  F32: 3456
//   256     19.8  19.8  20.1  30.7  31.7  33.1           52.6  96.9    21.2  33.8  61.8  98.0 103.1 107.2 213.3        40.3  87.7  92.5       95.6
//   224     18.1  18.4  24.6  28.3  29.7  37.2           46.8  94.9    19.1  29.4  61.4  89.1  98.0 102.4 202.9        38.6  85.7  94.9       93.2
//   192     16.4  23.2  24.9  26.3  34.1  36.2           42.3 107.2    25.9  35.2  64.5  96.3 101.4 109.6 214.4        42.0  90.5  95.2       99.3
// and M 1100, K 1024, F16, 128 columns 21.9, 192 20.8; where N is no multiple of 256 (M 1537, N 2056, F16), 128, 224 columns: K 64 5.1, 6.8 us, 512 8.5, 8.9, 1024 11.3, 11.3, 2048 17.8, 16.7.
// The rule is within 3 % of the best width in each of 95 such measurements, 5.5 % sustained (tests/test_routes.py).
constexpr int GEMM_PAIR_FIXED = 300;
inline long long gemm_tile_cost(int M, int N, long long ksteps, int width, bool gelu, int sm_count) {
    const bool pair = width != 128;
    const int height = pair ? 256 : 128, unit = width == 256 ? (gelu ? 98 : 88) : width == 224 ? 80 : width == 192 ? 71 : gelu ? 64 : 59;
    const long long tiles = (long long)((M + height - 1) / height) * ((N + width - 1) / width), groups = pair ? sm_count / 2 : sm_count;
    return ksteps * unit * (6 * ((tiles + groups - 1) / groups) * groups + 4 * tiles) / groups + (pair ? 10 * GEMM_PAIR_FIXED : 0);
}
// n_seg weight matrices in one launch. any_n_seg: the outputs have to be the same to the bit whether the projections of an activation
// share a launch or not. The number of parts is the order of the sums (the tile shape is not), so it is then the one that suits three
// segments, for one and two as well: a split that would pay for a single projection only is left out (N 2048, K 2048: four parts up to
// M 256, two up to M 512; up to M 128 two parts are left). What that costs the single call, head epilogue, device time: M 128
// 9.1 us either way, M 256 10.2 -> 10.7, M 512 10.3 -> 11.1.
inline GemmShape gemm_shape(int M, int N, long long ksteps, int n_seg, bool any_n_seg, int sm_count, const int* max_clusters, bool any_width = false,
                            bool gelu = false) {
    const int split = any_n_seg ? gemm_cheapest(M, N, ksteps, 3, 0, sm_count, max_clusters).split : 0;
    GemmShape g = gemm_cheapest(M, N, ksteps, n_seg, split, sm_count, max_clusters);
    if (!any_width || n_seg > 1 || g.split > 1 || M <= 128) return g;
    long long best = gemm_tile_cost(M, N, ksteps, g.width, gelu, sm_count);
    for (int width = 224; width >= 192; width -= 32) {
        const long long cost = gemm_tile_cost(M, N, ksteps, width, gelu, sm_count);
        if (cost < best) { best = cost; g = {true, 1, width}; }
    }
    return g;
}

}  // namespace kb
