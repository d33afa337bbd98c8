// Row pre-pass for Q and K: per (token, head) RMSNorm with a bf16 weight[128] and rotate-half RoPE,
// written once as 16-bit operands for the attention kernel. It restates, fused into one pass,
//   k_rmsnorm_warp  engine/src/kernels.cu:656-666   y = x * rsqrt(mean(x^2) + eps) * w
//   k_rope_half     engine/src/kernels.cu:759-772   pairs (i, i+64): a*c - b*s, b*c + a*s, tables [T, 64]
// in the reference's order (norm, then RoPE; engine/src/dit.cu:464-468). With neither norm nor RoPE
// it is the fp32 -> 16-bit staging conversion the reference does inside its kernel
// (engine/src/tcflash.cuh:56-64).
// The attention kernel's tensor-core operands are always fp16 (as in the reference, which converts to
// fp16 while staging): bf16 and fp32 inputs are converted here, fp16 inputs that need neither norm nor
// RoPE skip this pass entirely.
// Bound by memory; a warp takes several heads of a row, see qk_prep_kernel.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include <type_traits>

#include "ptx.cuh"
#include "routes.h"

namespace kb {

// eight consecutive elements as fp32, and as they lie in memory
struct F8 { float v[8]; };
template <typename T> struct Raw8 { uint4 u[sizeof(T) / 2]; };
template <typename T> struct Io {
    static __device__ __forceinline__ Raw8<T> raw8(const T* p) {
        Raw8<T> r;
#pragma unroll
        for (int i = 0; i < (int)sizeof(T) / 2; i++) r.u[i] = reinterpret_cast<const uint4*>(p)[i];
        return r;
    }
    static __device__ __forceinline__ F8 f8(const Raw8<T>& r) {
        F8 f;
        if constexpr (sizeof(T) == 4) {
#pragma unroll
            for (int i = 0; i < 2; i++) {
                f.v[4 * i] = __uint_as_float(r.u[i].x); f.v[4 * i + 1] = __uint_as_float(r.u[i].y);
                f.v[4 * i + 2] = __uint_as_float(r.u[i].z); f.v[4 * i + 3] = __uint_as_float(r.u[i].w);
            }
        } else {
            const uint32_t w[4] = {r.u[0].x, r.u[0].y, r.u[0].z, r.u[0].w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if constexpr (std::is_same<T, __nv_bfloat16>::value) {   // a bf16 is the top half of an fp32
                    f.v[2 * i] = __uint_as_float(w[i] << 16); f.v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
                } else {
                    const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
                    f.v[2 * i] = h.x; f.v[2 * i + 1] = h.y;
                }
            }
        }
        return f;
    }
    static __device__ __forceinline__ F8 ld8(const T* p) { return f8(raw8(p)); }
    static __device__ __forceinline__ void st8(T* p, const F8& f) {
        if constexpr (sizeof(T) == 4) {
            reinterpret_cast<float4*>(p)[0] = make_float4(f.v[0], f.v[1], f.v[2], f.v[3]);
            reinterpret_cast<float4*>(p)[1] = make_float4(f.v[4], f.v[5], f.v[6], f.v[7]);
        } else {
            uint32_t w[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if constexpr (std::is_same<T, __nv_bfloat16>::value) {
                    const __nv_bfloat162 h = __floats2bfloat162_rn(f.v[2 * i], f.v[2 * i + 1]);
                    w[i] = *reinterpret_cast<const uint32_t*>(&h);
                } else {
                    const __half2 h = __floats2half2_rn(f.v[2 * i], f.v[2 * i + 1]);
                    w[i] = *reinterpret_cast<const uint32_t*>(&h);
                }
            }
            *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
};

// One launch stages up to five tensors (Q, K, V, or Q and the four context tensors of NAG).
struct PrepSeg {
    const void* in;              // [rows, ld_in], head h at columns h*128
    void* out;                   // [rows, ld_out]
    const __nv_bfloat16* w;      // RMSNorm weight[128] or null
    const float* cos_t;          // RoPE tables [T, 64] or null; row r uses table row r % T
    const float* sin_t;
    int rows, ld_in, ld_out, T;
    unsigned block0;             // first thread block of this segment in the launch
};
struct PrepParams {
    PrepSeg seg[5];
    int nseg, H;
    int heads_log2;              // qk_prep_few_kernel: log2 of PrepLayout::heads
    float eps;
    unsigned blocks;             // total thread blocks
    unsigned int* zero_ptr;      // optional: zero_n words the first thread block clears (counters and flags that the
    int zero_n;                  // attention kernel launched next on the stream expects at zero)
};

// Clears the words of a call that stages nothing (a kernel and not a memset, so that the chain of dependent launches holds).
__global__ void zero_words_kernel(unsigned int* ptr, int n) {
    pdl_launch();
    pdl_wait();
    for (int i = threadIdx.x; i < n; i += blockDim.x) ptr[i] = 0u;
}

// A warp takes 2 NP heads of a row: all its loads first (NP pieces of eight elements per lane), then head after head.
//   without RoPE: two heads side by side, lane `sub` of 16 holds elements [8 sub, 8 sub + 8);
//   with RoPE   : four heads side by side, lane `sub` of 8 holds elements [8 sub, 8 sub + 8) AND their rotation partners [64 + 8 sub, ...),
//                 so the rotation needs no shuffle, and a lane's 8 + 8 table values serve all its heads (NP = 1: never with RoPE).
// Bound by memory: the rows come from HBM, the 16-bit copies go to L2. NP (launch_prep_t) sets what a lane has in flight against how many
// lanes there are. Measured on B200 with three sets of inputs in turn, whole attention call, one piece per lane (two with RoPE) -> this:
// self-attention with norm and RoPE, bf16, 256 tokens 11.1 -> 10.0 us, 1000 21.6 -> 20.7, 1536 39.5 -> 38.0, 4096 144.5 -> 141.2 (NP 2: 10.2,
// 21.1, 38.5, 142.1; NP 8: 10.9, 21.7, 38.2, 143.8); fp32, whose pieces are 32 bytes, NP 2: 1000 tokens 23.4 -> 23.4, gradients at 1024
// 101.7 -> 100.0 (NP 4: 23.5, 100.0; 4096 tokens 151.8 -> 152.6); a context of 512 x 1024 fp32 for cross_kv 11.1 us with NP 1, 11.5 with 2; NP 1
// with the four warps of a block on one row 9.94 (fp32) and 9.95 (bf16), on four rows 10.37 and 9.90, half a warp per head (before) 10.18 and 10.05.
constexpr int PREP_THREADS = 32 * PREP_WARPS;   // routes.h (PrepLayout) says what a thread block takes

template <typename InT, typename OutT, int NP>
__global__ void __launch_bounds__(PREP_THREADS)
qk_prep_kernel(const __grid_constant__ PrepParams pp) {
    constexpr int ROWS = prep_units(NP), HEADS = prep_heads(NP), NI = NP > 1 ? NP / 2 : 1;
    pdl_launch();
    pdl_wait();
    if (blockIdx.x == 0 && blockIdx.y == 0)
        for (int i = threadIdx.x; i < pp.zero_n; i += PREP_THREADS) pp.zero_ptr[i] = 0u;
    int si = 0;
#pragma unroll
    for (int i = 1; i < 5; i++)
        if (i < pp.nseg && blockIdx.x >= pp.seg[i].block0) si = i;
    const PrepSeg& sg = pp.seg[si];
    const int lane = threadIdx.x & 31;
    const unsigned row = ROWS * (blockIdx.x - sg.block0) + (ROWS > 1 ? threadIdx.x >> 5 : 0u);
    if (row >= (unsigned)sg.rows) return;
    const int r = (int)row;
    const InT* const src = static_cast<const InT*>(sg.in) + (size_t)r * sg.ld_in;
    OutT* const dst = static_cast<OutT*>(sg.out) + (size_t)r * sg.ld_out;
    for (int h0 = (int)blockIdx.y * HEADS + (ROWS > 1 ? 0 : 2 * (int)(threadIdx.x >> 5)); h0 < pp.H; h0 += (int)gridDim.y * HEADS) {   // one round up to 65535 groups of heads
        if (NP > 1 && sg.cos_t) {
            const int sub = lane & 7, hl = h0 + (lane >> 3);     // heads hl, hl + 4, ...
            Raw8<InT> ra[NI], rb[NI];
#pragma unroll
            for (int i = 0; i < NI; i++) {
                const int h = min(hl + 4 * i, pp.H - 1);         // past the last head: read again, not stored
                ra[i] = Io<InT>::raw8(src + h * 128 + 8 * sub);
                rb[i] = Io<InT>::raw8(src + h * 128 + 64 + 8 * sub);
            }
            const size_t tr = (size_t)(r % sg.T) * 64 + 8 * sub;
            const F8 c = Io<float>::ld8(sg.cos_t + tr), s = Io<float>::ld8(sg.sin_t + tr);
            Raw8<__nv_bfloat16> wa, wb;
            if (sg.w) { wa = Io<__nv_bfloat16>::raw8(sg.w + 8 * sub); wb = Io<__nv_bfloat16>::raw8(sg.w + 64 + 8 * sub); }
#pragma unroll
            for (int i = 0; i < NI; i++) {
                F8 a = Io<InT>::f8(ra[i]), b = Io<InT>::f8(rb[i]);
                if (sg.w) {
                    float ss = 0.f;
#pragma unroll
                    for (int e = 0; e < 8; e++) ss += a.v[e] * a.v[e] + b.v[e] * b.v[e];
#pragma unroll
                    for (int o = 4; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                    const float rs = rsqrtf(ss * (1.f / 128.f) + pp.eps);
                    const F8 fa = Io<__nv_bfloat16>::f8(wa), fb = Io<__nv_bfloat16>::f8(wb);
#pragma unroll
                    for (int e = 0; e < 8; e++) { a.v[e] = a.v[e] * rs * fa.v[e]; b.v[e] = b.v[e] * rs * fb.v[e]; }
                }
                F8 x, y;
#pragma unroll
                for (int e = 0; e < 8; e++) {                    // engine/src/kernels.cu:769-771
                    x.v[e] = a.v[e] * c.v[e] - b.v[e] * s.v[e];
                    y.v[e] = b.v[e] * c.v[e] + a.v[e] * s.v[e];
                }
                if (hl + 4 * i < pp.H) {
                    Io<OutT>::st8(dst + (hl + 4 * i) * 128 + 8 * sub, x);
                    Io<OutT>::st8(dst + (hl + 4 * i) * 128 + 64 + 8 * sub, y);
                }
            }
            continue;
        }
        const int sub = lane & 15, hl = h0 + (lane >> 4);        // heads hl, hl + 2, ...
        Raw8<InT> rx[NP];
#pragma unroll
        for (int i = 0; i < NP; i++) rx[i] = Io<InT>::raw8(src + min(hl + 2 * i, pp.H - 1) * 128 + 8 * sub);
        Raw8<__nv_bfloat16> w;
        if (sg.w) w = Io<__nv_bfloat16>::raw8(sg.w + 8 * sub);
#pragma unroll
        for (int i = 0; i < NP; i++) {
            F8 x = Io<InT>::f8(rx[i]);
            if (sg.w) {                                           // block-uniform
                float ss = 0.f;
#pragma unroll
                for (int e = 0; e < 8; e++) ss += x.v[e] * x.v[e];
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                const float rs = rsqrtf(ss * (1.f / 128.f) + pp.eps);
                const F8 fw = Io<__nv_bfloat16>::f8(w);
#pragma unroll
                for (int e = 0; e < 8; e++) x.v[e] = x.v[e] * rs * fw.v[e];
            }
            if (hl + 2 * i < pp.H) Io<OutT>::st8(dst + (hl + 2 * i) * 128 + 8 * sub, x);
        }
    }
}

// The same with few heads, which would leave lanes of a unit (PrepLayout, which has both sides measured) idle: a unit takes 2^heads_log2 heads,
// a divisor of H, of each of several rows. A kernel of its own: written as one with the above, its places cost that one 3 % of cross_kv
// (fp32, 512 rows 9.85 -> 10.15 us).
template <typename InT, typename OutT, int NP>
__global__ void __launch_bounds__(PREP_THREADS)
qk_prep_few_kernel(const __grid_constant__ PrepParams pp) {
    constexpr int UNITS = prep_units(NP), HEADS = prep_heads(NP), NI = NP > 1 ? NP / 2 : 1;
    pdl_launch();
    pdl_wait();
    if (blockIdx.x == 0 && blockIdx.y == 0)
        for (int i = threadIdx.x; i < pp.zero_n; i += PREP_THREADS) pp.zero_ptr[i] = 0u;
    int si = 0;
#pragma unroll
    for (int i = 1; i < 5; i++)
        if (i < pp.nseg && blockIdx.x >= pp.seg[i].block0) si = i;
    const PrepSeg& sg = pp.seg[si];
    const int lane = threadIdx.x & 31;
    const int hs = pp.heads_log2, step = 1 << hs;
    const unsigned row0 = (UNITS * (blockIdx.x - sg.block0) + (NP > 1 ? threadIdx.x >> 5 : 0u)) * (unsigned)(HEADS >> hs);
    if (row0 >= (unsigned)sg.rows) return;
    const int last = sg.rows - 1 - (int)row0;                    // last row, from the unit's first on
    const InT* const src = static_cast<const InT*>(sg.in) + (size_t)row0 * sg.ld_in;
    OutT* const dst = static_cast<OutT*>(sg.out) + (size_t)row0 * sg.ld_out;
    const int k_warp = NP > 1 ? 0 : 2 * (int)(threadIdx.x >> 5);  // a warp's first pair of the unit
    for (int h0 = (int)blockIdx.y * step; h0 < pp.H; h0 += (int)gridDim.y * step) {   // one round up to 65535 groups of heads
        // pair k of the unit: its row, its place in the tensor, and is it one (past the last row or head: read again, not stored)
        auto row_of = [&](int k) { return min(k >> hs, last); };
        auto at = [&](int k, int ld) { return (size_t)row_of(k) * ld + (h0 + (k & (step - 1))) * 128; };
        auto live = [&](int k) { return (k >> hs) <= last; };
        if (NP > 1 && sg.cos_t) {
            const int sub = lane & 7, k0 = lane >> 3;            // pairs k0, k0 + 4, ...
            Raw8<InT> ra[NI], rb[NI];
#pragma unroll
            for (int i = 0; i < NI; i++) {
                ra[i] = Io<InT>::raw8(src + at(k0 + 4 * i, sg.ld_in) + 8 * sub);
                rb[i] = Io<InT>::raw8(src + at(k0 + 4 * i, sg.ld_in) + 64 + 8 * sub);
            }
            F8 c, s;
            auto table = [&](int k) {
                const size_t tr = (size_t)((row0 + (unsigned)row_of(k)) % (unsigned)sg.T) * 64 + 8 * sub;
                c = Io<float>::ld8(sg.cos_t + tr);
                s = Io<float>::ld8(sg.sin_t + tr);
            };
            table(k0);
            Raw8<__nv_bfloat16> wa, wb;
            if (sg.w) { wa = Io<__nv_bfloat16>::raw8(sg.w + 8 * sub); wb = Io<__nv_bfloat16>::raw8(sg.w + 64 + 8 * sub); }
#pragma unroll
            for (int i = 0; i < NI; i++) {
                if (i > 0) table(k0 + 4 * i);
                F8 a = Io<InT>::f8(ra[i]), b = Io<InT>::f8(rb[i]);
                if (sg.w) {
                    float ss = 0.f;
#pragma unroll
                    for (int e = 0; e < 8; e++) ss += a.v[e] * a.v[e] + b.v[e] * b.v[e];
#pragma unroll
                    for (int o = 4; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                    const float rs = rsqrtf(ss * (1.f / 128.f) + pp.eps);
                    const F8 fa = Io<__nv_bfloat16>::f8(wa), fb = Io<__nv_bfloat16>::f8(wb);
#pragma unroll
                    for (int e = 0; e < 8; e++) { a.v[e] = a.v[e] * rs * fa.v[e]; b.v[e] = b.v[e] * rs * fb.v[e]; }
                }
                F8 x, y;
#pragma unroll
                for (int e = 0; e < 8; e++) {                    // engine/src/kernels.cu:769-771
                    x.v[e] = a.v[e] * c.v[e] - b.v[e] * s.v[e];
                    y.v[e] = b.v[e] * c.v[e] + a.v[e] * s.v[e];
                }
                if (live(k0 + 4 * i)) {
                    Io<OutT>::st8(dst + at(k0 + 4 * i, sg.ld_out) + 8 * sub, x);
                    Io<OutT>::st8(dst + at(k0 + 4 * i, sg.ld_out) + 64 + 8 * sub, y);
                }
            }
            continue;
        }
        const int sub = lane & 15, k0 = (lane >> 4) + k_warp;   // pairs k0, k0 + 2, ...
        Raw8<InT> rx[NP];
#pragma unroll
        for (int i = 0; i < NP; i++) rx[i] = Io<InT>::raw8(src + at(k0 + 2 * i, sg.ld_in) + 8 * sub);
        Raw8<__nv_bfloat16> w;
        if (sg.w) w = Io<__nv_bfloat16>::raw8(sg.w + 8 * sub);
#pragma unroll
        for (int i = 0; i < NP; i++) {
            F8 x = Io<InT>::f8(rx[i]);
            if (sg.w) {                                           // block-uniform
                float ss = 0.f;
#pragma unroll
                for (int e = 0; e < 8; e++) ss += x.v[e] * x.v[e];
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                const float rs = rsqrtf(ss * (1.f / 128.f) + pp.eps);
                const F8 fw = Io<__nv_bfloat16>::f8(w);
#pragma unroll
                for (int e = 0; e < 8; e++) x.v[e] = x.v[e] * rs * fw.v[e];
            }
            if (live(k0 + 2 * i)) Io<OutT>::st8(dst + at(k0 + 2 * i, sg.ld_out) + 8 * sub, x);
        }
    }
}

}  // namespace kb
