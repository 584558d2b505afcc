// Device functions of the mixed-precision stage (FP32 gathers and
// convolutions with compensated sums, FP64 row constants and positions),
// shared by the single-quench kernel (dyn_mixed.cu) and the batched
// persistent kernel (dyn_batch.cu) so that both run the same arithmetic.
#pragma once
#include "dyn_epi.cuh"

namespace dyn {
namespace mixed {

struct FModel {
    int p, p2;
    float cA, cB, cC, cD;
};

// Packed FP32x2 arithmetic (fma.rn.f32x2 / mul.rn.f32x2 of the sm_100 family): one
// instruction for the (QK, QR) pair, each half rounded exactly as fmaf / __fmul_rn.
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
        "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
// w * x + c for both halves of x and c
__device__ __forceinline__ float2 ffma2s(float w, float2 x, float2 c) { return ffma2(make_float2(w, w), x, c); }
__device__ __forceinline__ float2 fmul2s(float w, float2 x) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
        "mov.b64 ra, {%2, %2};\n\tmov.b64 rb, {%3, %4};\n\t"
        "mul.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(w), "f"(x.x), "f"(x.y));
    return d;
}
// a * b as a fused step from +0: the assembler contracts a packed mul and a packed add or sub
// that uses its product into one fma, which takes the product's rounding out of an error-free
// sum; a fused step it leaves alone
__device__ __forceinline__ float2 fmul2(float2 a, float2 b) { return ffma2(a, b, make_float2(0.f, 0.f)); }
__device__ __forceinline__ float2 fadd2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "add.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 fsub2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "sub.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

template <int E>
__device__ __forceinline__ float fpow_c(float q) {
    if constexpr (E <= 0) return 1.0f;
    else if constexpr (E == 1) return q;
    else if constexpr (E == 2) return q * q;
    else if constexpr (E == 3) return (q * q) * q;
    else if constexpr (E == 4) { float s = q * q; return s * s; }
    else { float s = fpow_c<E / 2>(q); s = s * s; if constexpr (E & 1) s = s * q; return s; }
}
__device__ __forceinline__ float fpow_r(float q, int e) {
    float r = 1.0f, c = q;
    while (e > 0) { if (e & 1) r *= c; c *= c; e >>= 1; }
    return r;
}

template <int P, int P2>
struct SigF {
    __device__ __forceinline__ static void d12(const FModel& M, float q, float& a, float& b) {
        if constexpr (P >= 0) {
            a = fmaf(M.cA, fpow_c<P - 1>(q), M.cB * fpow_c<P2 - 1>(q));
            b = fmaf(M.cC, fpow_c<P - 2>(q), M.cD * fpow_c<P2 - 2>(q));
        } else {
            a = fmaf(M.cA, fpow_r(q, M.p - 1), M.cB * fpow_r(q, M.p2 - 1));
            b = fmaf(M.cC, fpow_r(q, M.p - 2), M.cD * fpow_r(q, M.p2 - 2));
        }
    }
    __device__ __forceinline__ static float d2(const FModel& M, float q) {
        if constexpr (P >= 0) return fmaf(M.cC, fpow_c<P - 2>(q), M.cD * fpow_c<P2 - 2>(q));
        else return fmaf(M.cC, fpow_r(q, M.p - 2), M.cD * fpow_r(q, M.p2 - 2));
    }
};

// FP32 stencil weights are tap-major: plane p holds the tap pair (2p, 2p+1)
// of every target (float2, the second tap zero for an odd depth), so the
// lanes of a warp, handling consecutive targets, read consecutive words.
// sum_d w[d] * x[d] over the m taps of target ij, taps in order.
__device__ __forceinline__ float2 dotfT(const float2* __restrict__ w, size_t L2, size_t ij,
                                        const float2* __restrict__ x, int m, bool ldg) {
    float2 acc = make_float2(0.f, 0.f);
    for (int d = 0; d < m; d += 2) {
        const float2 ww = __ldg(w + (size_t)(d >> 1) * L2 + ij);
        const float2 xa = ldg ? __ldg(x + d) : x[d];
        acc = ffma2s(ww.x, xa, acc);
        if (d + 1 < m) {
            const float2 xb = ldg ? __ldg(x + d + 1) : x[d + 1];
            acc = ffma2s(ww.y, xb, acc);
        }
    }
    return acc;
}

// sum_d w[d] * x[b + d] for a 10-tap segment in shared memory (the staged last row), read
// as six 16-byte loads from the even element at or below b, each tap selecting its element
// (the select form; the same sums as seg11s with shifted weights, up to the sign of an
// exact zero, with fewer live registers)
__device__ __forceinline__ float2 seg10s(const float w[10], const float2* arr, int b) {
    const int a = b & ~1;
    const bool sh = b & 1;
    const float4* p = reinterpret_cast<const float4*>(arr + a);
    float2 e[12];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const float4 v = p[k];
        e[2 * k] = make_float2(v.x, v.y);
        e[2 * k + 1] = make_float2(v.z, v.w);
    }
    float2 acc = make_float2(0.f, 0.f);
#pragma unroll
    for (int d = 0; d < 10; ++d) acc = ffma2s(w[d], sh ? e[d + 1] : e[d], acc);
    return acc;
}

// The ten stencil weights laid over the element pairs that start at the even
// element a = b & ~1 at or below the stencil start b: w11[k] = w[k - (b & 1)]
// (zero outside 0..9).  A segment sum then needs no per-element select, and
// one shift serves every segment whose start has the same parity.
__device__ __forceinline__ void shift_w(const float w[10], const bool sh, float w11[11]) {
    w11[0] = sh ? 0.f : w[0];
#pragma unroll
    for (int k = 1; k < 10; ++k) w11[k] = sh ? w[k - 1] : w[k];
    w11[10] = sh ? w[9] : 0.f;
}

// sum_k w11[k] * arr[a + k], k = 0..10, a even, from shared memory (the staged last row):
// five 16-byte loads and one 8-byte load, taps in order.  The zero tap leaves the sum of
// the ten others unchanged, so arr[a .. a+10] must be finite (the staged row is zero-filled
// past its end).
__device__ __forceinline__ float2 seg11s(const float w11[11], const float2* arr, int a) {
    const float4* p = reinterpret_cast<const float4*>(arr + a);
    float2 acc = make_float2(0.f, 0.f);
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        const float4 v = p[q];
        acc = ffma2s(w11[2 * q], make_float2(v.x, v.y), acc);
        acc = ffma2s(w11[2 * q + 1], make_float2(v.z, v.w), acc);
    }
    return ffma2s(w11[10], arr[a + 10], acc);
}

// the ten taps of target ij from the tap-major planes
__device__ __forceinline__ void load_w10(const float2* __restrict__ w, size_t L2, size_t ij, float wv[10]) {
#pragma unroll
    for (int d = 0; d < 5; ++d) {
        const float2 q = __ldg(w + d * L2 + ij);
        wv[2 * d] = q.x;
        wv[2 * d + 1] = q.y;
    }
}

// sum_d w[d] * x[d] of a history segment (read-only path), taps in order
template <int M>
__device__ __forceinline__ float2 dot_ldg(const float2* __restrict__ w, size_t L2, size_t ij,
                                          const float2* __restrict__ x, int m) {
    if constexpr (M == 10) {
        float wv[10];
        load_w10(w, L2, ij, wv);
        float2 acc = make_float2(0.f, 0.f);
#pragma unroll
        for (int d = 0; d < 10; ++d) acc = ffma2s(wv[d], __ldg(x + d), acc);
        return acc;
    } else {
        return dotfT(w, L2, ij, x, m, true);
    }
}

// A ten-tap sum as dot_ldg's over a segment of the history (start b in the whole array), read as
// six 16-byte loads from the even element at or below the start, every tap selecting its element.
// Reads up to two elements past a segment and uses none of them.
__device__ __forceinline__ float2 seg10(const float w[10], const float2* __restrict__ arr, size_t b) {
    const float4* p = reinterpret_cast<const float4*>(arr + (b & ~(size_t)1));
    const bool sh = b & 1;
    float2 e[12];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const float4 v = __ldg(p + k);
        e[2 * k] = make_float2(v.x, v.y);
        e[2 * k + 1] = make_float2(v.z, v.w);
    }
    float2 acc = make_float2(0.f, 0.f);
#pragma unroll
    for (int d = 0; d < 10; ++d) acc = ffma2s(w[d], sh ? e[d + 1] : e[d], acc);
    return acc;
}

// (h, l) + s, normalized (the double-float sum of namespace mdf)
__device__ __forceinline__ void shift_offset(float& h, float& l, float s) {
    const float t = __fadd_rn(h, s), bp = __fsub_rn(t, h);
    const float e = __fadd_rn(__fadd_rn(__fsub_rn(h, __fsub_rn(t, bp)), __fsub_rn(s, bp)), __fadd_rn(l, 0.f));
    h = __fadd_rn(t, e);
    l = __fsub_rn(e, __fsub_rn(h, t));
}

// TwoSum accumulation: s + c carries the sum to about twice FP32 precision
// (round-to-nearest intrinsics: a product passed as v is never fused into the sum)
__device__ __forceinline__ void two_sum_add(float& s, float& c, float v) {
    const float t = __fadd_rn(s, v);
    const float bp = __fsub_rn(t, s);
    c = __fadd_rn(c, __fadd_rn(__fsub_rn(s, __fsub_rn(t, bp)), __fsub_rn(v, bp)));
    s = t;
}

// (hi, lo) += (h2, l2) with TwoSum on the high parts
__device__ __forceinline__ void pair_add(float& h, float& l, float h2, float l2) {
    const float t = __fadd_rn(h, h2);
    const float bp = __fsub_rn(t, h);
    l = __fadd_rn(__fadd_rn(l, l2), __fadd_rn(__fsub_rn(h, __fsub_rn(t, bp)), __fsub_rn(h2, bp)));
    h = t;
}

// Reduce-scatter of 8 compensated sums over a warp (as warp_reduce8, in FP32
// pairs): lane l with (l & 3) == 0 ends with the warp total of value index
// warp_reduce8_index(l) as hi + lo.
__device__ __forceinline__ void warp_reduce8_pair(const float hv[8], const float lv[8], int lane, float& H, float& Lo) {
    float wh[4], wl[4];
    const bool b16 = lane & 16;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float sh = b16 ? hv[k] : hv[k + 4], sl = b16 ? lv[k] : lv[k + 4];
        wh[k] = b16 ? hv[k + 4] : hv[k];
        wl[k] = b16 ? lv[k + 4] : lv[k];
        pair_add(wh[k], wl[k], __shfl_xor_sync(0xffffffffu, sh, 16), __shfl_xor_sync(0xffffffffu, sl, 16));
    }
    const bool b8 = lane & 8;
    float xh[2], xl[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const float sh = b8 ? wh[k] : wh[k + 2], sl = b8 ? wl[k] : wl[k + 2];
        xh[k] = b8 ? wh[k + 2] : wh[k];
        xl[k] = b8 ? wl[k + 2] : wl[k];
        pair_add(xh[k], xl[k], __shfl_xor_sync(0xffffffffu, sh, 8), __shfl_xor_sync(0xffffffffu, sl, 8));
    }
    const bool b4 = lane & 4;
    float yh = b4 ? xh[1] : xh[0], yl = b4 ? xl[1] : xl[0];
    pair_add(yh, yl, __shfl_xor_sync(0xffffffffu, b4 ? xh[0] : xh[1], 4),
             __shfl_xor_sync(0xffffffffu, b4 ? xl[0] : xl[1], 4));
    pair_add(yh, yl, __shfl_xor_sync(0xffffffffu, yh, 2), __shfl_xor_sync(0xffffffffu, yl, 2));
    pair_add(yh, yl, __shfl_xor_sync(0xffffffffu, yh, 1), __shfl_xor_sync(0xffffffffu, yl, 1));
    H = yh;
    Lo = yl;
}

// Block-shared scratch of one target row
constexpr int RED_CAP = 256;  // per-warp partial sums held between folds (float pairs)
constexpr int MAX_SEG = 4096 / 32;  // 32-target segments of the longest row
template <int CAP>
struct B2Jobs {  // targets whose B2 sums a chunk of CAP targets has to form (CAP 0: none kept)
    unsigned short s[CAP ? 2 * CAP : 1];  // (local target << 1) | 0: S0, 1: S1
    unsigned short d[CAP ? 2 * CAP : 1];  // (local target << 1) | 0: D1, 1: D2
    int X[CAP ? CAP : 1];
    int n[2][2];  // [chunk parity][s, d]
};
struct RowShared {
    int seg[MAX_SEG + 1];  // B2 interval brackets: seg[w] = k(phi2[i][32 w] t), seg[nseg] = k(phi2[i][L-1] t)
    float c[4];            // B1 Hermite constants of the row (FP32)
    int bi[2];             // B1 floor index, cubic flag
    float2 red[RED_CAP];   // [chunk slot][warp][8] partial sums as (hi, lo)
};

// B2 brackets: phi2 is non-decreasing along a row (checked when the tables are
// loaded), so every target of 32-target segment w has its interval in
// [seg[w], seg[w + 1]]; one full search per segment, short ones per target (a stage
// that goes on from the previous one starts from each target's last row instead)
__device__ __forceinline__ void row_brackets(const DevCtx& c, const StageDev& sp, const int i, RowShared& sh) {
    if (!(sp.T > 0.0)) return;
    const int L = c.L, nseg = (L + 31) >> 5;
    const ListView lv{c.t1grid, sp.nrows, sp.T};
    for (int w = threadIdx.x; w <= nseg; w += blockDim.x) {
        const int j = w < nseg ? (w << 5) : L - 1;
        sh.seg[w] = floor_index(lv, __dmul_rn(c.phi2[(size_t)i * L + j], sp.T), 0, sp.nrows - 1);
    }
}
// Row set-up for target row i: stages the last history row (FP32 mirror) in
// shared memory, rounds the row's B1 weights to FP32 and brackets the B2
// intervals of its targets.  BATCH: the row's own work too, and the B1 row of a stage
// flagged `fresh` (after a rollback or an upload) is searched here.
template <bool BATCH>
__device__ __forceinline__ B1Row row_b1(const DevCtx& c, const StageDev& sp, const int i) {
    B1Row r = {};
    r.F = 1;
    if (sp.T > 0.0) {
        if (BATCH && sp.fresh)
            r = b1_row(c, search_pos(c.search, ListView{c.t1grid, sp.nrows, sp.T}, __dmul_rn(c.theta[i], sp.T)), sp.maxceil, sp.nrows);
        else
            r = c.b1[i];
    }
    if constexpr (BATCH) side_value(c, sp, r, i);
    return r;
}
template <bool BATCH>
__device__ __forceinline__ void row_setup(const DevCtx& c, const StageDev& sp, const int i, float2* s_lastf,
                                          RowShared& sh, const bool brackets) {
    const int L = c.L, tpb = blockDim.x;
    const float2* row = c.KRf + (size_t)(sp.nrows - 1) * L;
    for (int k = threadIdx.x; k < L; k += tpb) s_lastf[k] = row[k];
    if (threadIdx.x == 0) {
        s_lastf[L] = s_lastf[L + 1] = make_float2(0.f, 0.f);
        const B1Row r = row_b1<BATCH>(c, sp, i);
        sh.bi[0] = r.F; sh.bi[1] = r.cubic;
        sh.c[0] = (float)r.c0; sh.c[1] = (float)r.c1; sh.c[2] = (float)r.c2; sh.c[3] = (float)r.c3;
    }
    if (BATCH && threadIdx.x == 32) side_position(c, sp, sp.fresh ? sp.nrows : c.b1[i].F, i);
    if (brackets) row_brackets(c, sp, i, sh);
}

// The rows' own work (side_row) for rows blk*blockDim.x on, one thread a row
__device__ __forceinline__ void side_rows(const DevCtx& c, const StageDev& sp, const int blk) {
    const int i = blk * blockDim.x + threadIdx.x;
    if (i < c.L) side_row(c, sp, i);
}

// A non-negative FP64 value as an FP32 pair, h truncated, l the rest rounded: in the integer
// pipe, away from the FP64 pipe's conversions (each holds it as long as an FP64 FMA).  Below
// 2^-70 the rest is dropped.
__device__ __forceinline__ void split_f64(double v, float& h, float& l) {
    const int hi = __double2hiint(v), lo = __double2loint(v), ex = hi >> 20;
    if (ex < 1023 - 70) {
        h = __double2float_rn(v);
        l = 0.f;
        return;
    }
    h = __int_as_float(__funnelshift_l(lo, hi - (896 << 20), 3));
    l = __fmul_rn(__uint2float_rn((unsigned)lo & 0x1fffffffu), __int_as_float((ex - (1023 + 52 - 127)) << 23));
}

// Row X (clamped) and offset x = xh + xl of target ij in the history.  The plain form
// takes x from the FP32 inverse length alone (xl = 0), the (hi, lo) form from pairs.
// key > 0: the target's row at the previous stage, where the search starts.
template <bool DF>
__device__ __forceinline__ void b2_position(const DevCtx& c, const ListView& lv, const RowShared& sh, const size_t ij,
                                            const int j, const double t, const int maxX, const int key, int& X, float& xh,
                                            float& xl) {
    const double El = __dmul_rn(__ldg(c.phi2 + ij), t);
    const int k = key > 0 ? floor_index_near(lv, El, min(key, lv.n) - 1)
                          : floor_index(lv, El, sh.seg[j >> 5], sh.seg[(j >> 5) + 1]);
    xh = xl = 0.f;
    if (k >= lv.n - 1) {
        X = lv.n;
    } else {
        const double diff = __dsub_rn(El, lv.at(k));
        X = k + 1;
        if constexpr (DF) {
            const float2 il = __ldg(c.inv_len_f + k);
            float dh, dl;
            split_f64(diff, dh, dl);
            xh = __fmul_rn(dh, il.x);
            xl = __fmaf_rn(dh, il.x, -xh);
            xl = __fmaf_rn(dh, il.y, xl);
            xl = __fmaf_rn(dl, il.x, xl);
            if (xh >= 1.0f) { X = k + 2; shift_offset(xh, xl, -1.0f); }
        } else {
            xh = __fmul_rn(__double2float_rn(diff), __ldg(&c.inv_len_f[k].x));
            if (xh >= 1.0f) { X = k + 2; xh = xh - 1.0f; }
        }
    }
    if (X > maxX) {
        if constexpr (DF) shift_offset(xh, xl, __int2float_rn(X - maxX));
        else xh += __int2float_rn(X - maxX);
        X = maxX;
    }
    if (X < 1) {
        if constexpr (DF) shift_offset(xh, xl, -__int2float_rn(1 - X));
        else xh -= __int2float_rn(1 - X);
        X = 1;
    }
}

// Push the sums of one target on the chunk's lists, in lane order and sum by sum, one
// reservation per warp and list
template <int CAP>
__device__ __forceinline__ void b2_push(B2Jobs<CAP>& jb, const int par, const int tl, const int need) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    unsigned b[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) b[q] = __ballot_sync(0xffffffffu, need >> q & 1);
#pragma unroll
    for (int l = 0; l < 2; ++l) {
        const int n0 = __popc(b[2 * l]), tot = n0 + __popc(b[2 * l + 1]);
        if (tot == 0) continue;
        int base = 0;
        if (lane == 0) base = atomicAdd(&jb.n[par][l], tot);
        base = __shfl_sync(0xffffffffu, base, 0);
        unsigned short* out = l == 0 ? jb.s : jb.d;
        if (need >> (2 * l) & 1) out[base + __popc(b[2 * l] & lt)] = (unsigned short)(tl << 1);
        if (need >> (2 * l + 1) & 1) out[base + n0 + __popc(b[2 * l + 1] & lt)] = (unsigned short)(tl << 1 | 1);
    }
}

// One chunk of tpb*K targets of row i: A1/A2 from the staged row, B1 and B2
// from the FP32 history, Sigma, and the eight int.dat-weighted products with
// TwoSum accumulation; each warp's eight sums land in sh.red[slot][warp].
// Call after row_setup and a __syncthreads(); a block can run several chunks (slots)
// before one fold.
// SHIFT picks the segment form of the depth-10 A1/A2 gathers (shifted weights, seg11s, or
// per-tap selects, seg10s): same results, different instruction counts and register
// footprints.  CAP: targets of a chunk when the B2 sums are kept in planes (B2Mode; keep:
// this stage goes on from the previous one), 0 when every target forms its own.
template <int M, int K, int P, int P2, bool SHIFT, int CAP>
__device__ __forceinline__ void chunk_sums(const DevCtx& c, const StageDev& sp, const int ch, const int slot,
                                           const float2* s_lastf, RowShared& sh, const int i, B2Jobs<CAP>& jb,
                                           const int par, const bool keep) {
    const int L = c.L, tpb = blockDim.x;
    const size_t L2 = (size_t)L * L;
    const int nrows = sp.nrows;
    const double t = sp.T;
    const bool live = t > 0.0;
    const FModel Mf{c.M.p, c.M.p2, (float)c.M.cA, (float)c.M.cB, (float)c.M.cC, (float)c.M.cD};
    const int m = M > 0 ? M : c.m;
    const float bc0 = sh.c[0], bc1 = sh.c[1], bc2 = sh.c[2], bc3 = sh.c[3];
    const int F = sh.bi[0], cubic1 = sh.bi[1];
    const int maxX = sp.maxX;
    const float2 fill = c.KRf[0];
    const ListView lv{c.t1grid, nrows, t};

    [[maybe_unused]] int Xk[K];
    [[maybe_unused]] float xk[K];
    if constexpr (CAP > 0) {
#pragma unroll
        for (int kk = 0; kk < K; ++kk) {
            const int tl = kk * tpb + threadIdx.x, j = ch * tpb * K + tl;
            Xk[kk] = 1;
            xk[kk] = 0.f;
            int need = 0;
            if (live && j < L) {
                const size_t ij = (size_t)i * L + j;
                const int key = keep ? c.b2key[ij] : 0;
                float xl;
                b2_position<false>(c, lv, sh, ij, j, t, maxX, key, Xk[kk], xk[kk], xl);
                need = b2_need(Xk[kk], key, b2_dirty(sp), Xk[kk] < nrows - 1);
                jb.X[tl] = Xk[kk];
                if (Xk[kk] != key) c.b2key[ij] = Xk[kk];
            }
            b2_push(jb, par, tl, need);
        }
    }
    if constexpr (CAP > 0) {
        __syncthreads();
        const int ns = jb.n[par][0], nd = jb.n[par][1];
        if (threadIdx.x == 0) jb.n[par ^ 1][0] = jb.n[par ^ 1][1] = 0;
        for (int q = threadIdx.x; q < ns + nd; q += tpb) {
            const int job = q < ns ? jb.s[q] : jb.d[q - ns] | 0x10000, tl = (job & 0xffff) >> 1, second = job & 1;
            const size_t ij = (size_t)i * L + ch * tpb * K + tl;
            const size_t at = (size_t)(jb.X[tl] - 1) * (size_t)L + (size_t)__ldg(c.iB2 + ij);
            // S0, S1: (QK, QR) rows X-1, X; D1, D2: (dQK, dQR) rows X, X+1
            const float2* x = q < ns ? c.KRf + at + (second ? L : 0) : c.dKRf + at + (second ? 2 * (size_t)L : L);
            c.b2f[(size_t)((q < ns ? 0 : 2) + second) * L2 + ij] = dot_ldg<M>(c.wB2f, L2, ij, x, m);
        }
        __syncthreads();
    }

    float acc[8], cmp[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) { acc[k] = 0.f; cmp[k] = 0.f; }

#pragma unroll
    for (int kk = 0; kk < K; ++kk) {
        const int j = ch * tpb * K + kk * tpb + threadIdx.x;
        if (j < L) {
            const size_t ij = (size_t)i * L + j;
            float2 a1, a2, b1, b2;
            if (live) {
                if constexpr (M == 10 && SHIFT) {
                    float wv[10], w11[11];
                    const int sa1 = __ldg(c.iA1 + ij), sa2 = __ldg(c.iA2 + ij);
                    load_w10(c.wA1f, L2, ij, wv);
                    shift_w(wv, sa1 & 1, w11);
                    a1 = seg11s(w11, s_lastf, sa1 & ~1);
                    load_w10(c.wA2f, L2, ij, wv);
                    shift_w(wv, sa2 & 1, w11);
                    a2 = seg11s(w11, s_lastf, sa2 & ~1);
                } else if constexpr (M == 10) {
                    float wv[10];
                    load_w10(c.wA1f, L2, ij, wv);
                    a1 = seg10s(wv, s_lastf, __ldg(c.iA1 + ij));
                    load_w10(c.wA2f, L2, ij, wv);
                    a2 = seg10s(wv, s_lastf, __ldg(c.iA2 + ij));
                } else {
                    a1 = dotfT(c.wA1f, L2, ij, s_lastf + __ldg(c.iA1 + ij), m, false);
                    a2 = dotfT(c.wA2f, L2, ij, s_lastf + __ldg(c.iA2 + ij), m, false);
                }
                {
                    const float2 x0 = __ldg(c.KRf + (size_t)(F - 1) * L + j);
                    const float2 x1 = __ldg(c.KRf + (size_t)F * L + j);
                    const float2 d1 = __ldg(c.dKRf + (size_t)F * L + j);
                    // c0 x0 + c1 x1 - c2 d1 (- c3 d2), packed over (QK, QR)
                    float2 r = fmul2s(-bc2, d1);
                    if (cubic1) r = ffma2s(-bc3, __ldg(c.dKRf + (size_t)(F + 1) * L + j), r);
                    b1 = ffma2s(bc0, x0, ffma2s(bc1, x1, r));
                }
                {
                    int X;
                    float x;
                    if constexpr (CAP > 0) {
                        X = Xk[kk];
                        x = xk[kk];
                    } else {
                        float xl;
                        b2_position<false>(c, lv, sh, ij, j, t, maxX, 0, X, x, xl);
                    }
                    const float x2 = x * x, x3 = x2 * x;
                    const bool cubic2 = X < nrows - 1;
                    // the four segments (rows X-1, X of (QK, QR), rows X, X+1 of (dQK, dQR)),
                    // each folded into the Hermite sum as it completes
                    const size_t base = (size_t)(X - 1) * (size_t)L + (size_t)__ldg(c.iB2 + ij);
                    [[maybe_unused]] float wv[10];
                    if constexpr (CAP == 0 && M == 10) load_w10(c.wB2f, L2, ij, wv);
                    auto seg = [&](const int which) -> float2 {
                        if constexpr (CAP > 0) {
                            return c.b2f[(size_t)which * L2 + ij];
                        } else {
                            const float2* arr = which < 2 ? c.KRf : c.dKRf;
                            const size_t at = base + (size_t)(which == 0 ? 0 : which == 3 ? 2 : 1) * (size_t)L;
                            if constexpr (M == 10) return seg10(wv, arr, at);
                            else return dot_ldg<M>(c.wB2f, L2, ij, arr + at, m);
                        }
                    };
                    float2 r;
                    float e0;
                    if (cubic2) {
                        e0 = 1.f - 3.f * x2 + 2.f * x3;
                        const float e1 = x - 2.f * x2 + x3, e2 = 3.f * x2 - 2.f * x3;
                        const float e3 = (x3 - x2) * __ldg(&c.inv_dtr_f[X + 1].x);
                        r = fmul2s(e3, seg(3));
                        r = ffma2s(e2, seg(1), r);
                        r = ffma2s(e1, seg(2), r);
                    } else {
                        e0 = 1.f - x2;
                        r = fmul2s(x - x2, seg(2));
                        r = ffma2s(x2, seg(1), r);
                    }
                    b2 = ffma2s(e0, seg(0), r);
                }
            } else {
                a1 = a2 = b1 = b2 = fill;
            }
            float sKA1, dA1, sKB1, dB1, sKB2, dB2;
            SigF<P, P2>::d12(Mf, a1.x, sKA1, dA1);
            const float sRA1 = dA1 * a1.y;
            const float sRA2 = SigF<P, P2>::d2(Mf, a2.x) * a2.y;
            SigF<P, P2>::d12(Mf, b1.x, sKB1, dB1);
            const float sRB1 = dB1 * b1.y;
            SigF<P, P2>::d12(Mf, b2.x, sKB2, dB2);
            const float sRB2 = dB2 * b2.y;
            const float wj = __ldg(&c.integ_f[j].x);
            const float wRA2 = wj * sRA2, wQRA2 = wj * a2.y;
            const float v[8] = {wRA2 * b2.x, (wj * sRA1) * b1.x, (wj * sKA1) * b1.y, wQRA2 * sKB2,
                                (wj * a1.y) * sKB1, (wj * a1.x) * sRB1, wRA2 * b2.y, wQRA2 * sRB2};
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                // the first term of a TwoSum from zero is exact: (s, c) = (v, 0)
                if (kk == 0) acc[k] = v[k];
                else two_sum_add(acc[k], cmp[k], v[k]);
            }
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float H, Lo;
    warp_reduce8_pair(acc, cmp, lane, H, Lo);
    if ((lane & 3) == 0) sh.red[((slot * (tpb >> 5)) + warp) * 8 + warp_reduce8_index(lane)] = make_float2(H, Lo);
}

// After a __syncthreads() that follows the chunks of slots 0..ng-1 (chunks ch0..ch0+ng-1):
// the block's six sums of each chunk into part[ch][0..6)[i], warps added in order, compensated
// on the high parts, one conversion at the end.  Eight lanes a chunk in whole warps ((hi, lo): two
// of them idle; a loop bounded by ng measured 1.3 % slower over mixed lengths).  The plain form's
// eight sums (DF false) are paired here, the two ConvA sums that share their factor: across lanes
// in a kernel of one chunk; in the batch by the thread that stores them, because the exchange kept
// so much alive through its loop that it spilled at 48 registers (16 quenches at L = 1024: 1005 us
// a gather at 56, now 950; in the single kernel that form is the slower one, one RK54 step at
// L = 640 282 us against 270).
template <bool DF, bool BATCH>
__device__ __forceinline__ void fold_chunks(const DevCtx& c, const int i, const int ch0, const int ng, const RowShared& sh) {
    const int nw = blockDim.x >> 5;
    if constexpr (DF || !BATCH) {
        const int k = threadIdx.x & 7;
        for (int g = threadIdx.x >> 3; g < ((ng + 3) & ~3); g += blockDim.x >> 3) {
            float h = 0.f, l = 0.f;
            if (g < ng)
                for (int w = 0; w < nw; ++w) {
                    const float2 hl = sh.red[(g * nw + w) * 8 + k];
                    pair_add(h, l, hl.x, hl.y);
                }
            double v = (double)h + (double)l;
            int out = k;
            if constexpr (!DF) {
                const double next = __shfl_down_sync(0xffffffffu, v, 1);
                if (k == 1 || k == 4) v += next;
                out = k < 2 ? k : k == 2 || k == 5 ? 6 : k < 5 ? k - 1 : k - 2;
            }
            if (g < ng && out < 6) c.part[((size_t)(ch0 + g) * 6 + out) * c.L + i] = v;
        }
    } else {
        const auto sum = [&](const float2* r) {
            float h = 0.f, l = 0.f;
            for (int w = 0; w < nw; ++w) pair_add(h, l, r[8 * w].x, r[8 * w].y);
            return (double)h + (double)l;
        };
        for (int t = threadIdx.x; t < 6 * ng; t += blockDim.x) {
            const int g = t / 6, out = t - 6 * g, k = out + (out >= 2) + (out >= 4);
            const float2* r = sh.red + g * nw * 8 + k;
            double v = sum(r);
            if (out == 1 || out == 3) v += sum(r + 1);
            c.part[((size_t)ch0 * 6 + t) * c.L + i] = v;
        }
    }
}

}  // namespace mixed

// ---------------------------------------------------------------- (hi, lo) form
// Plain FP32 gathers go wrong over long runs through FP32 roundings that repeat
// step after step (the rounded weights and stored history, and the rounding of
// sums over them).  Here the weights and the stored (QK, QR) history carry FP32
// (hi, lo) pairs; the A1/A2 and B2 stencil sums add every product w x with its
// rounding error (TwoProd, TwoSum) and the cross terms (w_hi x_lo + w_lo x_hi); the gathered values stay
// (hi, lo) and everything that changes from stage to stage -- the B2 interval offset,
// the Hermite weights, B1, Sigma and the int.dat products -- runs in double-float
// (chunk_dd), so the stage derivatives carry no stage-to-stage FP32 rounding noise and
// the embedded error estimate sees the method's error, as in the FP64 form.  The
// derivative rows (dQK, dQR), a step's worth of change, stay single FP32.
//
// Double-float: an unevaluated sum h + l of two floats, ~44 bits.  Every operation is a
// round-to-nearest intrinsic or packed instruction, so the compiler never fuses a
// product into a following sum (which would break the error-free transformations and
// make the result depend on how a kernel was inlined).  The arithmetic is packed: two
// double-floats side by side (pr), the (QK, QR) pair of one point or the same quantity at
// two points, one FP32x2 instruction for both.
namespace mdf {
using namespace mixed;

struct ff {
    float h, l;
};
__device__ __forceinline__ ff ff_mul(ff a, ff b) {
    const float p = __fmul_rn(a.h, b.h);
    float e = __fmaf_rn(a.h, b.h, -p);
    e = __fmaf_rn(a.h, b.l, e);
    e = __fmaf_rn(a.l, b.h, e);
    return {p, e};
}

struct pr {
    float2 h, l;
};
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
__device__ __forceinline__ pr pr_both(ff v) { return {both(v.h), both(v.l)}; }
__device__ __forceinline__ pr pr_bcast(float4 v) { return {make_float2(v.x, v.y), make_float2(v.z, v.w)}; }
// a * b.  Products and sums are left unnormalized: the low word is the exact rounding
// error of the high one plus the cross terms, a few ulp of it at most, which every later
// operation takes as it is.
__device__ __forceinline__ pr pr_mul(pr a, pr b) {
    const float2 p = fmul2(a.h, b.h);
    float2 e = ffma2(a.h, b.h, fsub2(make_float2(0.f, 0.f), p));
    e = ffma2(a.h, b.l, e);
    e = ffma2(a.l, b.h, e);
    return {p, e};
}
// s + w x: the product with its rounding error, added with TwoSum.  (Adding the unrounded
// product in one fused step saves three operations of twelve, but where s and w x cancel the
// sum keeps bits below both that the error term then misses.)
__device__ __forceinline__ void pr_add_prod(pr& s, float2 w, float2 x) {
    const float2 p = fmul2(w, x), e = ffma2(w, x, fsub2(make_float2(0.f, 0.f), p));
    const float2 t = fadd2(s.h, p), bp = fsub2(t, s.h);
    const float2 d = fadd2(fsub2(s.h, fsub2(t, bp)), fsub2(p, bp));
    s.l = fadd2(s.l, fadd2(d, e));
    s.h = t;
}
// s + a * b with the cross terms of (hi, lo) factors
__device__ __forceinline__ void pr_acc(pr& s, pr a, pr b) {
    pr_add_prod(s, a.h, b.h);
    s.l = ffma2(a.h, b.l, s.l);
    s.l = ffma2(a.l, b.h, s.l);
}
__device__ __forceinline__ void pr_accf(pr& s, pr a, float2 b) {
    pr_add_prod(s, a.h, b);
    s.l = ffma2(a.l, b, s.l);
}
__device__ __forceinline__ pr pr_sub(pr a, pr b) {
    const float2 t = fsub2(a.h, b.h), bp = fsub2(t, a.h);
    const float2 e = fsub2(fsub2(a.h, fsub2(t, bp)), fadd2(b.h, bp));
    return {t, fadd2(e, fsub2(a.l, b.l))};
}
__device__ __forceinline__ pr pr_norm(pr a) {
    const float2 h = fadd2(a.h, a.l);
    return {h, fsub2(a.l, fsub2(h, a.h))};
}
// (s, l) += (h2, l2), TwoSum on the high parts (pair_add on both lanes)
__device__ __forceinline__ void pr_add(pr& s, pr v) {
    const float2 t = fadd2(s.h, v.h), bp = fsub2(t, s.h);
    s.l = fadd2(fadd2(s.l, v.l), fadd2(fsub2(s.h, fsub2(t, bp)), fsub2(v.h, bp)));
    s.h = t;
}

// Stencil weights: plane p holds the tap pair (2p, 2p+1) of every target as (hi, hi, lo, lo),
// a second tap past an odd depth zero.  History and the staged row: (QK, QR) as
// (hi, hi, lo, lo).  Sum over the taps of target ij, taps in order, from the element x on.
template <int M, bool LDG>
__device__ __forceinline__ pr gather(const float4* __restrict__ w, size_t L2, size_t ij, const float4* x, int m) {
    pr s;
    auto tap = [&](float wh, float wl, float4 v, bool first) {
        const pr xv = pr_bcast(v);
        if (first) s = pr_mul({both(wh), both(wl)}, xv);
        else pr_acc(s, {both(wh), both(wl)}, xv);
    };
    const int mm = M > 0 ? M : m;
#pragma unroll
    for (int d = 0; d < (M > 0 ? M : 1 << 20); d += 2) {
        if (d >= mm) break;
        const float4 q = __ldg(w + (size_t)(d >> 1) * L2 + ij);
        tap(q.x, q.z, LDG ? __ldg(x + d) : x[d], d == 0);
        if (d + 1 < mm) tap(q.y, q.w, LDG ? __ldg(x + d + 1) : x[d + 1], false);
    }
    return s;
}
// of a derivative-row segment with the high weights, in plain FP32
template <int M>
__device__ __forceinline__ float2 gather_f(const float4* __restrict__ w, size_t L2, size_t ij,
                                           const float2* __restrict__ x, int m) {
    float2 acc = make_float2(0.f, 0.f);
    const int mm = M > 0 ? M : m;
#pragma unroll
    for (int d = 0; d < (M > 0 ? M : 1 << 20); d += 2) {
        if (d >= mm) break;
        const float4 q = __ldg(w + (size_t)(d >> 1) * L2 + ij);
        acc = ffma2s(q.x, __ldg(x + d), acc);
        if (d + 1 < mm) acc = ffma2s(q.y, __ldg(x + d + 1), acc);
    }
    return acc;
}

// q^e as a left-to-right product chain, whether e is a template constant (the specialized
// models) or a run-time value (the generic kernel): both round alike, so a quench gives the
// same result in either kernel.  Times v.
template <int E>
__device__ __forceinline__ pr pow_times(pr q, int e, pr v) {
    if constexpr (E >= 0) {
        if constexpr (E == 0) {
            return v;
        } else {
            pr r = q;
#pragma unroll
            for (int k = 1; k < E; ++k) r = pr_mul(r, q);
            return pr_mul(r, v);
        }
    } else {
        if (e <= 0) return v;
        pr r = q;
        for (int k = 1; k < e; ++k) r = pr_mul(r, q);
        return pr_mul(r, v);
    }
}
// f'(q) and f''(q) at two points; cst: the model's coefficients.  Neighbouring exponents
// share their power, q^(p-1) (cA + cB q).
template <int P, int P2>
__device__ __forceinline__ void sigma(const float4* cst, int p, int p2, pr q, pr& d1, pr& d2) {
    constexpr int E1 = P < 0 ? -1 : P > 1 ? P - 1 : 0, E2 = P < 0 ? -1 : P > 2 ? P - 2 : 0;
    constexpr int G1 = P < 0 ? -1 : P2 > 1 ? P2 - 1 : 0, G2 = P < 0 ? -1 : P2 > 2 ? P2 - 2 : 0;
    if (P >= 0 ? P2 == P + 1 && P >= 2 : p2 == p + 1 && p >= 2) {
        pr a = pr_bcast(cst[0]), b = pr_bcast(cst[2]);
        pr_acc(a, pr_bcast(cst[1]), q);
        pr_acc(b, pr_bcast(cst[3]), q);
        d1 = pow_times<E1>(q, p - 1, a);
        d2 = pow_times<E2>(q, p - 2, b);
    } else {
        d1 = pow_times<E1>(q, p - 1, pr_bcast(cst[0]));
        pr_add(d1, pow_times<G1>(q, p2 - 1, pr_bcast(cst[1])));
        d2 = pow_times<E2>(q, p - 2, pr_bcast(cst[2]));
        pr_add(d2, pow_times<G2>(q, p2 - 2, pr_bcast(cst[3])));
    }
}

// Reduce-scatter of 6 compensated sums over a warp (as warp_reduce6)
__device__ __forceinline__ void warp_reduce6_pair(const float hv[6], const float lv[6], int lane, float& H, float& Lo) {
    const bool b16 = lane & 16, b8 = lane & 8, b4 = lane & 4;
    auto xc = [](float& h, float& l, float sh, float sl, int o) {
        pair_add(h, l, __shfl_xor_sync(0xffffffffu, sh, o), __shfl_xor_sync(0xffffffffu, sl, o));
    };
    float wh[3], wl[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        wh[k] = b16 ? hv[k + 3] : hv[k];
        wl[k] = b16 ? lv[k + 3] : lv[k];
        xc(wh[k], wl[k], b16 ? hv[k] : hv[k + 3], b16 ? lv[k] : lv[k + 3], 16);
    }
    float x0h = b8 ? wh[2] : wh[0], x0l = b8 ? wl[2] : wl[0], x1h = wh[1], x1l = wl[1];
    xc(x0h, x0l, b8 ? wh[0] : wh[2], b8 ? wl[0] : wl[2], 8);
    xc(x1h, x1l, wh[1], wl[1], 8);
    H = b4 ? x1h : x0h;
    Lo = b4 ? x1l : x0l;
    xc(H, Lo, b4 ? x0h : x1h, b4 ? x0l : x1l, 4);
    xc(H, Lo, H, Lo, 2);
    xc(H, Lo, H, Lo, 1);
}

// Per-row scratch: the staged newest row (dynamic shared memory, [L] (hi, hi, lo, lo)) and
// the constants every target of the row uses, each as (h, h, l, l): the model's cA..cD, the
// B1 weights c0, c1, -c2, -c3
struct RowConst {
    float4 model[4], b1[4];
};
__device__ __forceinline__ float4 quad(double v) {
    const float h = (float)v, l = (float)(v - (double)h);
    return make_float4(h, h, l, l);
}
template <bool BATCH>
__device__ __forceinline__ void row_setup(const DevCtx& c, const StageDev& sp, const int i, float4* s_row, RowShared& sh,
                                          RowConst& rc, const bool brackets) {
    const int L = c.L;
    const float4* row = c.KRq + (size_t)(sp.nrows - 1) * L;
    for (int k = threadIdx.x; k < L; k += blockDim.x) s_row[k] = row[k];
    if (threadIdx.x < 4) rc.model[threadIdx.x] = c.cq[threadIdx.x];
    if (threadIdx.x == 0) {
        const B1Row r = row_b1<BATCH>(c, sp, i);
        sh.bi[0] = r.F; sh.bi[1] = r.cubic;
        rc.b1[0] = quad(r.c0); rc.b1[1] = quad(r.c1); rc.b1[2] = quad(-r.c2); rc.b1[3] = quad(-r.c3);
    }
    if (BATCH && threadIdx.x == 32) side_position(c, sp, sp.fresh ? sp.nrows : c.b1[i].F, i);
    if (brackets) row_brackets(c, sp, i, sh);
}

// One chunk of tpb*K targets of row i, as chunk_sums, with everything that changes from
// stage to stage in double-float: the B2 interval offset, the Hermite weights, the gathered
// values (the compensated sums kept as (hi, lo)), Sigma and the int.dat products,
// accumulated as (hi, lo) pairs.  FP32 roundings that differ between the stages of
// one step would otherwise put a noise of ~1e-7 of |h| into every stage derivative,
// which the embedded error estimate sees: with delta_max = 1e-10 the controller
// then keeps the step ~1000x below the FP64 form's.  The roundings of the frozen
// inputs (the (hi, lo) weights and history, the FP32 derivative rows) vary smoothly
// with the stage time and cancel in the estimate.
template <int M, int K, int P, int P2, int CAP>
__device__ __forceinline__ void chunk_dd(const DevCtx& c, const StageDev& sp, const int ch, const int slot,
                                         const float4* s_row, const RowConst& rc, RowShared& sh, const int i,
                                         B2Jobs<CAP>& jb, const int par, const bool keep) {
    const int L = c.L, tpb = blockDim.x;
    const size_t L2 = (size_t)L * L;
    const int nrows = sp.nrows;
    const double t = sp.T;
    const bool live = t > 0.0;
    const int m = M > 0 ? M : c.m;
    const int maxX = sp.maxX;
    const ListView lv{c.t1grid, nrows, t};

    [[maybe_unused]] int Xk[K];
    [[maybe_unused]] ff xk[K];
    if constexpr (CAP > 0) {
#pragma unroll
        for (int kk = 0; kk < K; ++kk) {
            const int tl = kk * tpb + threadIdx.x, j = ch * tpb * K + tl;
            Xk[kk] = 1;
            xk[kk] = ff{0.f, 0.f};
            int need = 0;
            if (live && j < L) {
                const size_t ij = (size_t)i * L + j;
                const int key = keep ? c.b2key[ij] : 0;
                b2_position<true>(c, lv, sh, ij, j, t, maxX, key, Xk[kk], xk[kk].h, xk[kk].l);
                need = b2_need(Xk[kk], key, b2_dirty(sp), Xk[kk] < nrows - 1);
                jb.X[tl] = Xk[kk];
                if (Xk[kk] != key) c.b2key[ij] = Xk[kk];
            }
            b2_push(jb, par, tl, need);
        }
    }
    if constexpr (CAP > 0) {
        __syncthreads();
        const int ns = jb.n[par][0], nd = jb.n[par][1];
        if (threadIdx.x == 0) jb.n[par ^ 1][0] = jb.n[par ^ 1][1] = 0;
        // the compensated sums of (QK, QR) rows first, then the short ones of the derivative rows
        for (int q = threadIdx.x; q < ns; q += tpb) {
            const int tl = jb.s[q] >> 1, second = jb.s[q] & 1;
            const size_t ij = (size_t)i * L + ch * tpb * K + tl;
            const size_t at = (size_t)(jb.X[tl] - 1 + second) * (size_t)L + (size_t)__ldg(c.iB2 + ij);
            const pr v = gather<M, true>(c.wB2q, L2, ij, c.KRq + at, m);
            c.b2q[second * L2 + ij] = make_float4(v.h.x, v.h.y, v.l.x, v.l.y);
        }
        for (int q = threadIdx.x; q < nd; q += tpb) {
            const int tl = jb.d[q] >> 1, second = jb.d[q] & 1;
            const size_t ij = (size_t)i * L + ch * tpb * K + tl;
            const size_t at = (size_t)(jb.X[tl] + second) * (size_t)L + (size_t)__ldg(c.iB2 + ij);
            c.b2f[second * L2 + ij] = gather_f<M>(c.wB2q, L2, ij, c.dKRf + at, m);
        }
        __syncthreads();
    }

    // the six sums as three pairs: ConvR with QKB2 | QRB2, the two ConvA pairs, ConvR with Sigma B2
    pr accR = {}, accA = {}, accS = {};
#pragma unroll
    for (int kk = 0; kk < K; ++kk) {
        const int j = ch * tpb * K + kk * tpb + threadIdx.x;
        if (j < L) {
            const size_t ij = (size_t)i * L + j;
            pr a1, a2, b1, b2;  // the (QK, QR) pairs at the A1, A2, B1, B2 points
            if (live) {
                a1 = pr_norm(gather<M, false>(c.wA1q, L2, ij, s_row + __ldg(c.iA1 + ij), m));
                a2 = pr_norm(gather<M, false>(c.wA2q, L2, ij, s_row + __ldg(c.iA2 + ij), m));
                {
                    const int F = sh.bi[0];
                    const size_t r1 = (size_t)F * L + j;
                    b1 = pr_mul(pr_bcast(rc.b1[0]), pr_bcast(__ldg(c.KRq + (r1 - L))));
                    pr_acc(b1, pr_bcast(rc.b1[1]), pr_bcast(__ldg(c.KRq + r1)));
                    pr_accf(b1, pr_bcast(rc.b1[2]), __ldg(c.dKRf + r1));
                    if (sh.bi[1]) pr_accf(b1, pr_bcast(rc.b1[3]), __ldg(c.dKRf + (r1 + L)));
                    b1 = pr_norm(b1);
                }
                {
                    int X;
                    ff x;
                    if constexpr (CAP > 0) {
                        X = Xk[kk];
                        x = xk[kk];
                    } else {
                        b2_position<true>(c, lv, sh, ij, j, t, maxX, 0, X, x.h, x.l);
                    }
                    const bool cubic2 = X < nrows - 1;
                    pr S0, S1;
                    float2 D1, D2 = make_float2(0.f, 0.f);
                    if constexpr (CAP > 0) {
                        S0 = pr_bcast(c.b2q[ij]);
                        S1 = pr_bcast(c.b2q[L2 + ij]);
                        D1 = c.b2f[ij];
                        if (cubic2) D2 = c.b2f[L2 + ij];
                    } else {
                        const size_t base = (size_t)(X - 1) * (size_t)L + (size_t)__ldg(c.iB2 + ij);
                        S0 = gather<M, true>(c.wB2q, L2, ij, c.KRq + base, m);
                        S1 = gather<M, true>(c.wB2q, L2, ij, c.KRq + base + L, m);
                        D1 = gather_f<M>(c.wB2q, L2, ij, c.dKRf + base + L, m);
                        if (cubic2) D2 = gather_f<M>(c.wB2q, L2, ij, c.dKRf + base + 2 * L, m);
                    }
                    // S0 + e2 (S1 - S0) + e1 D1 + e3 D2 with, through y = 1 - x:
                    // e1 = x y^2, e2 = x^2 + 2 x^2 y, e3 = -x^2 y / ratio (cubic); x y, x^2 (quadratic)
                    const float yh = __fsub_rn(1.f, x.h);
                    const ff y{yh, __fsub_rn(__fsub_rn(__fsub_rn(1.f, yh), x.h), x.l)};
                    const ff xy = ff_mul(x, y), xx = ff_mul(x, x);
                    b2 = S0;
                    const pr dS = pr_sub(S1, S0);
                    if (cubic2) {
                        const ff x2y = ff_mul(xx, y), e1 = ff_mul(xy, y);
                        ff e2 = xx;
                        pair_add(e2.h, e2.l, 2.f * x2y.h, 2.f * x2y.l);
                        const float2 rt = __ldg(c.inv_dtr_f + X + 1);
                        const ff e3 = ff_mul(x2y, ff{-rt.x, -rt.y});
                        pr_acc(b2, pr_both(e2), dS);
                        pr_accf(b2, pr_both(e1), D1);
                        pr_accf(b2, pr_both(e3), D2);
                    } else {
                        pr_acc(b2, pr_both(xx), dS);
                        pr_accf(b2, pr_both(xy), D1);
                    }
                    b2 = pr_norm(b2);
                }
            } else {
                a1 = pr_bcast(c.KRq[0]);
                a2 = b1 = b2 = a1;
            }
            const float2 wj = __ldg(c.integ_f + j);
            // u = w R(A2), v = u f''(C(A2)); ConvR: v (C, R)(B2) and u (f'(C), f''(C) R)(B2)
            pr d1, d2;
            sigma<P, P2>(rc.model, c.M.p, c.M.p2,
                         pr{make_float2(a2.h.x, b2.h.x), make_float2(a2.l.x, b2.l.x)}, d1, d2);
            const ff u = ff_mul(ff{wj.x, wj.y}, ff{a2.h.y, a2.l.y});
            const pr vR = pr_mul(pr_both(ff_mul(u, ff{d2.h.x, d2.l.x})), b2);
            const ff sR = ff_mul(ff{d2.h.y, d2.l.y}, ff{b2.h.y, b2.l.y});
            const pr vS = pr_mul(pr_both(u), pr{make_float2(d1.h.y, sR.h), make_float2(d1.l.y, sR.l)});
            // ConvA: w (f''(C) R (A1) C(B1) + f'(C)(A1) R(B1)) and the same with A1, B1 exchanged
            sigma<P, P2>(rc.model, c.M.p, c.M.p2,
                         pr{make_float2(a1.h.x, b1.h.x), make_float2(a1.l.x, b1.l.x)}, d1, d2);
            pr vA = pr_mul(pr_mul(d2, pr{make_float2(a1.h.y, b1.h.y), make_float2(a1.l.y, b1.l.y)}),
                           pr{make_float2(b1.h.x, a1.h.x), make_float2(b1.l.x, a1.l.x)});
            pr_acc(vA, d1, pr{make_float2(b1.h.y, a1.h.y), make_float2(b1.l.y, a1.l.y)});
            vA = pr_mul(pr{both(wj.x), both(wj.y)}, vA);
            if (kk == 0) {
                accR = vR; accA = vA; accS = vS;
            } else {
                pr_add(accR, vR); pr_add(accA, vA); pr_add(accS, vS);
            }
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float hv[6] = {accR.h.x, accA.h.x, accS.h.x, accA.h.y, accR.h.y, accS.h.y};
    const float lw[6] = {accR.l.x, accA.l.x, accS.l.x, accA.l.y, accR.l.y, accS.l.y};
    float H, Lo;
    warp_reduce6_pair(hv, lw, lane, H, Lo);
    const int ri = warp_reduce6_index(lane);
    if ((lane & 3) == 0 && ri < 6) sh.red[((slot * (tpb >> 5)) + warp) * 8 + ri] = make_float2(H, Lo);
}

}  // namespace mdf

}  // namespace dyn
