// CUDA kernels of the GB300-native DYNAMITE hot path (FP64 form).
//
// Per RK stage the whole interpolate -> Sigma -> convolution -> RHS -> RK
// update -> r(t) chain of the reference (interpolateGPU, QKRstepGPU,
// drstep2GPU, appendAllGPU_ptr/replaceAllGPU_ptr, rstepGPU, RK54GPU...) runs
// as two kernels:
//
//   k_main (grid L x nch, and a few CTAs for the rows' own work): every
//     target (i, j) gathers its A1/A2/B1/B2 values from the history through
//     the stencil tables, evaluates Sigma, and accumulates the eight
//     int.dat-weighted products of the memory integrals in six sums (two pairs
//     share their factor).  Of size L^2 it writes what the next stage goes on
//     from: each target's history row and those of its four B2 sums that
//     changed.  The rows' own CTAs interpolate QK^{B1}[i,0] and rInt and search
//     the next stage's B1 positions.
//   k_epi (grid L/32, four warps a CTA): finishes the row reductions, forms the
//     EOM right-hand side and the RK stage combination, writes the history row,
//     accumulates r(t) (and dr/dt at stage 0) and forms the next stage's B1
//     rows; the last CTA to finish (atomic ticket) folds the per-CTA partials.
//
// A second, reference-order family of kernels ("exact") materializes the 16
// interpolation arrays and the RHS with the reference CPU build's operation
// order (no FMA contraction) for the C-ABI calls that mirror
// interpolateGPU/QKRstepGPU one to one.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include "dyn_epi.cuh"

namespace dyn {

// ------------------------------------------------------------------------
// Log-space response (the reference's -R option).  QK is interpolated as in
// the linear form; QR is interpolated as f = log QR with the derivatives
// g = dQR / QR and exponentiated, wherever every value it rests on is
// positive, and linearly otherwise.

// A1/A2 (index_vec.cu:185-226): lx holds log QR of the last row (QR itself
// where QR <= 0, as the reference's log slice does, index_vec.cu:367-375)
template <int M>
__device__ __forceinline__ double2 dot2s_log(const double* __restrict__ w, const double2* x, const double* lx, int m) {
    double qk = 0.0, qr = 0.0, sl = 0.0;
    bool ok = true;
    const int n = M > 0 ? M : m;
#pragma unroll
    for (int d = 0; d < n; ++d) {
        const double ww = __ldg(w + d);
        const double2 v = x[d];
        qk = fma(ww, v.x, qk);
        qr = fma(ww, v.y, qr);
        sl = fma(ww, lx[d], sl);
        ok = ok && v.y > 0.0;
    }
    return make_double2(qk, ok ? exp(sl) : qr);
}

// B1 (index_vec.cu:456-530) with the row's coefficients: r0, r1 the QR nodes,
// g1, g2 the stored dQR at the nodes' right neighbours; c3 = 0 on the
// quadratic branch
__device__ __forceinline__ double b1_log(double c0, double c1, double c2, double c3, double r0, double r1, double g1,
                                         double g2, double lin) {
    if (!(r0 > 0.0 && r1 > 0.0)) return lin;
    double f = c0 * log(r0) + c1 * log(r1) - c2 * (g1 / r0);
    if (c3 != 0.0) f -= c3 * (g2 / r1);
    return exp(f);
}

// ------------------------------------------------------------------------
// k_main: fused gathers + Sigma + convolution products for one stage.
// LOGR: QR gathers in log space (the last row's logs staged after it in
// shared memory).

// f' and f'' of a target: neighbouring exponents share their power, q^(P-1) (cA + cB q)
// and q^(P-2) (cC + cD q), one FP64 operation fewer each than Sig's two powers
template <int P, int P2>
struct SigT {
    __device__ __forceinline__ static double d1(const DModel& M, double q) {
        if constexpr (P >= 2 && P2 == P + 1) return ipow_c<P - 1>(q) * fma(M.cB, q, M.cA);
        else return Sig<P, P2>::d1(M, q);
    }
    __device__ __forceinline__ static double d2(const DModel& M, double q) {
        if constexpr (P >= 2 && P2 == P + 1) return ipow_c<P - 2>(q) * fma(M.cD, q, M.cC);
        else return Sig<P, P2>::d2(M, q);
    }
    __device__ __forceinline__ static void d12(const DModel& M, double q, double& a, double& b) {
        a = d1(M, q);
        b = d2(M, q);
    }
};

// One of the four B2 stencil sums of target ij (0: S0, 1: S1, 2: D1, 3: D2)
template <int M>
__device__ __forceinline__ double2 b2_sum(const DevCtx& c, const size_t ij, const int X, const int which, const int m) {
    const size_t at = (size_t)(X - 1) * c.L + __ldg(c.iB2 + ij) + (size_t)(which == 0 ? 0 : which == 3 ? 2 : 1) * c.L;
    return dot2g<M>(c.wB2 + ij * m, (which < 2 ? c.KR : c.dKR) + at, m);
}

// Bound by the FP64 pipe (2 lanes per SM and clock: a warp instruction holds it 16
// cycles whatever its lanes do), so what counts is FP64 instructions per target: ~200
// when every stage formed its four B2 sums (80), divided for its position (10) and kept
// eight row sums; ~130 with the sums kept, stored inverse interval lengths, shared powers
// and six row sums.  L = 512, 1500 rows: 111 us a stage before, 76 us after (pipe 86 %
// busy); the first stage of a call, which forms all sums through the list, 105 us.
//
// KEEP: the B2 sums live in planes over the stages of a call (B2Mode).  The targets
// that need a sum push it on a list in shared memory, the CTA's threads work the
// list off with full warps whatever targets it came from, and every target then
// reads its four sums back.  Without planes (KEEP false: the allocation-free
// right-hand side, or no memory for them) every target forms its own.
//
// SPLIT: two threads a target, two warps each for the halves that meet only in the row sums:
// the first half of the CTA its position and B2, the second A1, B1 and A2 meanwhile.  For
// lengths whose rows leave most schedulers without a warp, where a warp's own FP64 rate (one
// instruction in 64 cycles) bounds the stage; the same bits.
template <int M, int K, int P, int P2, bool LOGR, bool KEEP, bool SPLIT>
__global__ void __launch_bounds__(SPLIT ? 128 : 64) k_main(const DevCtx c, const int s) {
    static_assert(!SPLIT || (KEEP && K == 1));
    wait_prior_grid();
    const StageDev& sp = c.stages[s];
    const int L = c.L, nthr = blockDim.x, nside = (L + nthr - 1) / nthr;
    const int tpb = SPLIT ? 64 : nthr, tid = SPLIT ? threadIdx.x & 63 : threadIdx.x;  // target of the CTA
    const bool half0 = !SPLIT || threadIdx.x < 64, half1 = !SPLIT || threadIdx.x >= 64;
    if (blockIdx.y < nside) {  // the rows' own work, a row a thread
        const int r = blockIdx.y * nthr + threadIdx.x;
        if (blockIdx.x == 0 && r < L) side_row(c, sp, r);
        return;
    }
    // rows near theta = 1 first: most of their targets read the row being written, the longest work
    const int i = L - 1 - (blockIdx.y - nside);
    const size_t L2 = (size_t)L * L;
    const int nrows = sp.nrows;
    const double t = sp.T;
    const bool live = t > 0.0;
    extern __shared__ double2 s_last[];
    __shared__ double s_red[SPLIT ? 4 : 2][6];
    __shared__ double2 s_a2[SPLIT ? 64 : 1];
    __shared__ int s_X[KEEP ? 64 * K : 1];
    __shared__ unsigned short s_job[KEEP ? 4 * 64 * K : 1];  // (local target << 2) | sum
    __shared__ int s_njob;

    double* s_logR = reinterpret_cast<double*>(s_last + L);  // LOGR only: [L]

    const double2* KRl = c.KR + (size_t)(nrows - 1) * L;
    for (int k = threadIdx.x; k < L; k += nthr) {
        const double2 v = KRl[k];
        s_last[k] = v;
        if constexpr (LOGR) s_logR[k] = v.y > 0.0 ? log(v.y) : v.y;
    }
    if (threadIdx.x == 0) s_njob = 0;
    B1Row r1 = {};
    if (live) r1 = c.b1[i];

    const DModel Mo = c.M;
    const int m = M > 0 ? M : c.m;
    const int maxX = sp.maxX;
    const double2 fill = c.KR[0];
    const ListView lv{c.t1grid, nrows, t};
    const double* pos2_src = sp.b2_reuse >= 0
        ? (sp.b2_reuse == NSAVE ? c.posB2x : c.posB2x_saved + (size_t)sp.b2_reuse * L2) : nullptr;
    double* pos2_dst = sp.b2_save >= 0
        ? (sp.b2_save == NSAVE ? c.posB2x : c.posB2x_saved + (size_t)sp.b2_save * L2) : nullptr;
    const bool keep = KEEP && sp.b2_mode == B2_KEEP;
    const int dirty = b2_dirty(sp);
    __syncthreads();

    // ---- positions of the targets in the history: row X, offset x in its interval
    int X[K];
    double x[K];
    if (half0) {
#pragma unroll
    for (int kk = 0; kk < K; ++kk) {
        const int j = blockIdx.x * tpb * K + kk * tpb + tid;
        const size_t ij = (size_t)i * L + j;
        X[kk] = 1;
        x[kk] = 0.0;
        int need = 0;
        if (live && j < L) {
            const int key = keep ? c.b2key[ij] : 0;
            // position as the reference gives it, clamped to the rows there are
            const auto at_position = [&](const double pos2) {
                long long Xl = (long long)pos2;
                if (Xl > maxX) Xl = maxX;
                if (Xl < 1) Xl = 1;
                X[kk] = (int)Xl;
                x[kk] = __dsub_rn(pos2, (double)Xl);
                if (pos2_dst) pos2_dst[ij] = pos2;
            };
            if (pos2_src || sp.kind == KIND_RHS) {
                at_position(pos2_src ? pos2_src[ij] : search_pos(c.search, lv, __dmul_rn(__ldg(c.phi2 + ij), t)));
            } else {
                const double El = __dmul_rn(__ldg(c.phi2 + ij), t);
                const int k = key > 0 ? floor_index_near(lv, El, min(key, nrows) - 1) : floor_index(lv, El, 0, nrows - 1);
                const double tk = lv.at(k);
                if (off_interval(lv, El, k, tk)) {
                    at_position(search_pos_cold(c.search, lv.p, lv.n, lv.vlast, El));
                } else {
                    if (k >= nrows - 1) {
                        X[kk] = nrows;
                    } else {
                        x[kk] = okey(tk) == okey(El) ? 0.0 : __dmul_rn(__dsub_rn(El, tk), __ldg(c.inv_len + k));
                        X[kk] = k + 1;
                    }
                    if (pos2_dst) pos2_dst[ij] = (double)X[kk] + x[kk];
                    if (X[kk] > maxX) { x[kk] += (double)(X[kk] - maxX); X[kk] = maxX; }
                    if (X[kk] < 1) { x[kk] -= (double)(1 - X[kk]); X[kk] = 1; }
                }
            }
            if constexpr (KEEP) {
                need = b2_need(X[kk], key, dirty, X[kk] < nrows - 1);
                s_X[kk * tpb + tid] = X[kk];
                if (X[kk] != key) c.b2key[ij] = X[kk];
            }
        }
        if constexpr (KEEP) {
            // push this target's sums: one reservation per warp, sum by sum in lane order
            const unsigned lt = (1u << (threadIdx.x & 31)) - 1u;
            unsigned b[4];
            int tot = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                b[q] = __ballot_sync(0xffffffffu, need >> q & 1);
                tot += __popc(b[q]);
            }
            if (tot) {
                int base = 0;
                if ((threadIdx.x & 31) == 0) base = atomicAdd(&s_njob, tot);
                base = __shfl_sync(0xffffffffu, base, 0);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (need >> q & 1) s_job[base + __popc(b[q] & lt)] = (unsigned short)((kk * tpb + tid) << 2 | q);
                    base += __popc(b[q]);
                }
            }
        }
    }
    }
    // the stencils of the last row and B1 of a target
    const double bc0 = r1.c0, bc1 = r1.c1, bc2 = r1.c2, bc3 = r1.c3;
    const int F = r1.F, cubic1 = r1.cubic;
    const auto gather_a = [&](const size_t ij, const int j, double2& a1, double2& a2, double2& b1) {
        if constexpr (LOGR) {
            const int ia1 = __ldg(c.iA1 + ij), ia2 = __ldg(c.iA2 + ij);
            a1 = dot2s_log<M>(c.wA1 + ij * m, s_last + ia1, s_logR + ia1, m);
            a2 = dot2s_log<M>(c.wA2 + ij * m, s_last + ia2, s_logR + ia2, m);
        } else {
            a1 = dot2s<M>(c.wA1 + ij * m, s_last + __ldg(c.iA1 + ij), m);
            a2 = dot2s<M>(c.wA2 + ij * m, s_last + __ldg(c.iA2 + ij), m);
        }
        const double2 x0 = __ldg(c.KR + (size_t)(F - 1) * L + j);
        const double2 x1 = __ldg(c.KR + (size_t)F * L + j);
        const double2 d1 = __ldg(c.dKR + (size_t)F * L + j);
        b1.x = bc0 * x0.x + bc1 * x1.x - bc2 * d1.x;
        b1.y = bc0 * x0.y + bc1 * x1.y - bc2 * d1.y;
        double2 d2 = make_double2(0.0, 0.0);
        if (cubic1) {
            d2 = __ldg(c.dKR + (size_t)(F + 1) * L + j);
            b1.x -= bc3 * d2.x;
            b1.y -= bc3 * d2.y;
        }
        if constexpr (LOGR) b1.y = b1_log(bc0, bc1, bc2, cubic1 ? bc3 : 0.0, x0.y, x1.y, d1.y, d2.y, b1.y);
    };
    [[maybe_unused]] double2 sa1, sb1;
    if constexpr (SPLIT) {
        const int j = blockIdx.x * tpb + tid;
        if (half1 && live && j < L) gather_a((size_t)i * L + j, j, sa1, s_a2[tid], sb1);
    }
    if constexpr (KEEP) {
        __syncthreads();
        const int nj = s_njob;
        for (int q = threadIdx.x; q < nj; q += nthr) {
            const int job = s_job[q], tl = job >> 2, which = job & 3;
            const size_t ij = (size_t)i * L + blockIdx.x * tpb * K + tl;
            const double2 v = b2_sum<M>(c, ij, s_X[tl], which, m);
            c.b2s[which * L2 + ij] = v;
            if (LOGR && which < 2 && v.y > 0.0) reinterpret_cast<double*>(c.b2s + 4 * L2)[which * L2 + ij] = log(v.y);
        }
        __syncthreads();
    }

    double acc[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) acc[k] = 0.0;

#pragma unroll
    for (int kk = 0; kk < K; ++kk) {
        const int j = blockIdx.x * tpb * K + kk * tpb + tid;
        if (j < L) {
            const size_t ij = (size_t)i * L + j;
            double2 a1, a2, b1, b2;
            if (live) {
                if constexpr (!SPLIT) {
                    gather_a(ij, j, a1, a2, b1);
                } else {
                    a1 = sa1;
                    b1 = sb1;
                    a2 = s_a2[tid];
                }
                if (half0) {
                    const bool cubic2 = X[kk] < nrows - 1;
                    const double x1 = x[kk], x2 = x1 * x1;
                    double2 S0, S1, D1, D2 = make_double2(0.0, 0.0);
                    if constexpr (KEEP) {
                        S0 = c.b2s[ij];
                        S1 = c.b2s[L2 + ij];
                        D1 = c.b2s[2 * L2 + ij];
                        if (cubic2) D2 = c.b2s[3 * L2 + ij];
                    } else {
                        S0 = b2_sum<M>(c, ij, X[kk], 0, m);
                        S1 = b2_sum<M>(c, ij, X[kk], 1, m);
                        D1 = b2_sum<M>(c, ij, X[kk], 2, m);
                        if (cubic2) D2 = b2_sum<M>(c, ij, X[kk], 3, m);
                    }
                    // index_mat.cu:203-222: Hermite of log of the row sums; the logs are kept beside
                    // the sums (L = 519, 3400 rows: RK54 step 2.50 -> 2.39 ms)
                    const bool logs = LOGR && S0.y > 0.0 && S1.y > 0.0;
                    double l0 = 0.0, l1 = 0.0;
                    if (logs) {
                        const double* b2l = reinterpret_cast<const double*>(c.b2s + 4 * L2);
                        l0 = KEEP ? b2l[ij] : log(S0.y);
                        l1 = KEEP ? b2l[L2 + ij] : log(S1.y);
                    }
                    if (cubic2) {
                        // Hermite weights through y = x^3 - x^2: e1 = x - x^2 + y, e2 = x^2 - 2 y, e0 = 1 - e2
                        const double y = fma(x2, x1, -x2), e1 = (x1 - x2) + y, e2 = fma(-2.0, y, x2), e0 = 1.0 - e2;
                        const double e3 = y * c.inv_dtr[X[kk] + 1];
                        b2.x = fma(e3, D2.x, fma(e2, S1.x, fma(e1, D1.x, e0 * S0.x)));
                        b2.y = fma(e3, D2.y, fma(e2, S1.y, fma(e1, D1.y, e0 * S0.y)));
                        if (logs) b2.y = exp(e0 * l0 + e1 * (D1.y / S0.y) + e2 * l1 + e3 * (D2.y / S1.y));
                    } else {
                        const double e0 = 1.0 - x2, e2 = x1 - x2;
                        b2.x = fma(e2, D1.x, fma(x2, S1.x, e0 * S0.x));
                        b2.y = fma(e2, D1.y, fma(x2, S1.y, e0 * S0.y));
                        if (logs) b2.y = exp(e0 * l0 + x2 * l1 + e2 * (D1.y / S0.y));
                    }
                    if (c.rec) {
                        GatherRec* g = c.rec + ij;
                        if (!SPLIT) *g = GatherRec{a1, a2, b1, b2, x1, X[kk], 0};
                        else { g->a2 = a2; g->b2 = b2; g->x = x1; g->X = X[kk]; }
                    }
                }
                if (SPLIT && half1 && c.rec) { c.rec[ij].a1 = a1; c.rec[ij].b1 = b1; }
            } else {
                a1 = a2 = b1 = b2 = fill;
            }
            const double wj = __ldg(c.integ + j);
            if (half1) {
                double sKA1, dA1, sKB1, dB1;
                SigT<P, P2>::d12(Mo, a1.x, sKA1, dA1);
                SigT<P, P2>::d12(Mo, b1.x, sKB1, dB1);
                // ConvA(SigmaRA1, QKB1) + ConvA(SigmaKA1, QRB1)
                acc[1] = fma(wj, fma(sKA1, b1.y, (dA1 * a1.y) * b1.x), acc[1]);
                // ConvA(QRA1, SigmaKB1) + ConvA(QKA1, SigmaRB1)
                acc[3] = fma(wj, fma(a1.x, dB1 * b1.y, a1.y * sKB1), acc[3]);
            }
            if (half0) {
                double sKB2, dB2;
                SigT<P, P2>::d12(Mo, b2.x, sKB2, dB2);
                const double wQRA2 = wj * a2.y, wRA2 = wQRA2 * SigT<P, P2>::d2(Mo, a2.x);
                acc[0] = fma(wRA2, b2.x, acc[0]);            // ConvR(SigmaRA2, QKB2)
                acc[2] = fma(wQRA2, sKB2, acc[2]);           // ConvR(QRA2, SigmaKB2)
                acc[4] = fma(wRA2, b2.y, acc[4]);            // ConvR(SigmaRA2, QRB2)
                acc[5] = fma(wQRA2, dB2 * b2.y, acc[5]);     // ConvR(QRA2, SigmaRB2)
            }
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double r = warp_reduce6(acc, lane);
    const int ri = warp_reduce6_index(lane);
    if ((lane & 3) == 0 && ri < 6) s_red[warp][ri] = r;
    __syncthreads();
    if (threadIdx.x < 6) {
        double v = 0.0;
        for (int w = 0; w < (nthr >> 5); ++w) v += s_red[w][threadIdx.x];
        c.part[((size_t)blockIdx.x * 6 + threadIdx.x) * L + i] = v;
    }
}

// ------------------------------------------------------------------------
// k_epi: RHS, RK combination, history row, r(t), next positions.
template <int P, int P2, bool MIXED>
__global__ void __launch_bounds__(EPI_T) k_epi(const DevCtx c, const int s) {
    wait_prior_grid();
    const StageDev& sp = c.stages[s];
    const double inv = epi::rows<P, P2, MIXED>(c, sp, s, blockIdx.x, s == 0 && sp.fsal);
    if (!epi::elect_last(c, gridDim.x)) return;
    epi::fold<MIXED>(c, sp, s, gridDim.x, inv);
    if (threadIdx.x == 0) c.slots->counter = 0;
}

// ------------------------------------------------------------------------
// Positions and B1 rows of the current state (after init/upload/sparsify/rollback).
__global__ void k_pos_init(const DevCtx c, const int nrows) {
    const double T = c.t1grid[nrows - 1];
    const ListView lv{c.t1grid, nrows, T};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < c.L; i += gridDim.x * blockDim.x) {
        const double p = search_pos(c.search, lv, __dmul_rn(c.theta[i], T));
        c.posB1x[i] = p;
        c.b1[i] = b1_row(c, p, nrows - 1 < 1 ? 1 : nrows - 1, nrows);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) c.slots->counter = 0;
}

// ------------------------------------------------------------------------
// Reference-order ("exact") kernels: no contraction, the C++ expression
// order of the reference CPU build, so results on identical inputs are
// bit-identical to the reference compiled with -ffp-contract=off.
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dvd(double a, double b) { return __ddiv_rn(a, b); }

__device__ __forceinline__ double ip_exact(const double* w, const double2* x, int m, int comp) {
    double acc = 0.0;
    for (int d = 0; d < m; ++d) acc = add(acc, mul(w[d], comp ? x[d].y : x[d].x));
    return acc;
}

// exp(sum_d w_d log QR_d) when every QR_d > 0, else the linear value lin
// (index_vec.cpp:24-57, whose CPU form sums the logs in long double; this sum,
// like the reference's CUDA kernel index_vec.cu:185-226, is in double)
__device__ __forceinline__ double ip_log_exact(const double* w, const double2* x, int m, double lin) {
    double acc = 0.0;
    bool ok = true;
    for (int d = 0; d < m; ++d) {
        const double v = x[d].y;
        ok = ok && v > 0.0;
        acc = add(acc, mul(w[d], v > 0.0 ? log(v) : v));
    }
    return ok ? exp(acc) : lin;
}

// posB1x (given or searched), Floor clamp, B2 clamp (interpolation_core.cpp:19-114)
__global__ void k_pos_b1_exact(const DevCtx c, const int nrows, const double* pos1_given,
                               const double* pos2_given) {
    const int L = c.L;
    __shared__ double s_max[32];
    const double T = c.t1grid[nrows - 1];
    const ListView lv{c.t1grid, nrows, T};
    double mx = 0.0;
    for (int i = threadIdx.x; i < L; i += blockDim.x) {
        const double p = pos1_given ? pos1_given[i] : search_pos(c.search, lv, mul(c.theta[i], T));
        c.posB1x[i] = p;
        c.b1[i] = b1_row(c, p, nrows - 1 < 1 ? 1 : nrows - 1, nrows);
        mx = i == 0 ? p : fmax(mx, p);
    }
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
        double m = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m = fmax(m, s_max[w]);
        long long mc = (long long)ceil(m) - 1;
        c.slots->maxceil = (int)(mc < 1 ? 1 : mc);
        const double p = pos2_given ? pos2_given[(size_t)L * L - 1]
                                    : search_pos(c.search, lv, mul(c.phi2[(size_t)L * L - 1], T));
        c.slots->maxX = (int)(long long)(p - 0.5);
    }
}

// B1 (index_vec.cpp:63-136): C and R at time theta_i t, column j, by the cubic
// (quadratic at the last interval) Hermite of the history rows around posB1x[i],
// in the reference's operation order; log space for R with the -R option
__device__ __forceinline__ void b1_exact(const DevCtx& c, const int nrows, const int maxceil, const int i, const int j,
                                         double& vK, double& vR) {
    const int L = c.L;
    const double pos = c.posB1x[i];
    long long F = (long long)floor(pos);
    if (F < 1) F = 1; else if (F > maxceil) F = maxceil;
    const double wt = sub((double)F, pos);
    const double in3 = mul(wt, wt), in4 = mul(in3, wt);
    const double2 x0 = c.KR[(size_t)(F - 1) * L + j], x1 = c.KR[(size_t)F * L + j];
    const double2 d1 = c.dKR[(size_t)F * L + j];
    if (F < nrows - 1) {
        const double2 d2 = c.dKR[(size_t)(F + 1) * L + j];
        const double dr = c.dtr[F + 1];
        const double e0 = sub(sub(1.0, mul(3.0, in3)), mul(2.0, in4));
        const double e1 = add(mul(3.0, in3), mul(2.0, in4));
        const double e2 = add(add(wt, mul(2.0, in3)), in4);
        const double e3 = add(in3, in4);
        vK = sub(sub(add(mul(e0, x0.x), mul(e1, x1.x)), mul(e2, d1.x)), dvd(mul(e3, d2.x), dr));
        vR = sub(sub(add(mul(e0, x0.y), mul(e1, x1.y)), mul(e2, d1.y)), dvd(mul(e3, d2.y), dr));
        if (c.logr && x0.y > 0.0 && x1.y > 0.0)  // index_vec.cpp:89-100
            vR = exp(sub(sub(add(mul(e0, log(x0.y)), mul(e1, log(x1.y))), mul(e2, dvd(d1.y, x0.y))),
                         mul(dvd(e3, dr), dvd(d2.y, x1.y))));
    } else {
        const double e0 = sub(1.0, in3), e2 = add(wt, in3);
        vK = add(sub(mul(e0, x0.x), mul(e2, d1.x)), mul(in3, x1.x));
        vR = add(sub(mul(e0, x0.y), mul(e2, d1.y)), mul(in3, x1.y));
        if (c.logr && x0.y > 0.0 && x1.y > 0.0)  // index_vec.cpp:122-127
            vR = exp(sub(add(mul(e0, log(x0.y)), mul(in3, log(x1.y))), mul(e2, dvd(d1.y, x0.y))));
    }
}

// The B1 pair alone (what a save of the reference reads back as QK_B1/QR_B1), into
// caller arrays [L*L]; the t = 0 state gives the single row's values
__global__ void k_b1_exact(const DevCtx c, const int nrows, double* qk, double* qr) {
    const int L = c.L;
    const size_t L2 = (size_t)L * L;
    const bool live = c.t1grid[nrows - 1] > 0.0;
    const int maxceil = c.slots->maxceil;
    for (size_t ij = (size_t)blockIdx.x * blockDim.x + threadIdx.x; ij < L2; ij += (size_t)gridDim.x * blockDim.x) {
        double vK, vR;
        if (live) b1_exact(c, nrows, maxceil, (int)(ij / L), (int)(ij % L), vK, vR);
        else { vK = c.KR[0].x; vR = c.KR[0].y; }
        qk[ij] = vK;
        qr[ij] = vR;
    }
}

__global__ void k_interp_exact(const DevCtx c, const int nrows, const double* pos2_given) {
    const int L = c.L, m = c.m;
    const size_t L2 = (size_t)L * L;
    const double T = c.t1grid[nrows - 1];
    const bool live = T > 0.0;
    const ListView lv{c.t1grid, nrows, T};
    const DModel Mo = c.M;
    const double2* KRl = c.KR + (size_t)(nrows - 1) * L;
    const int maxceil = c.slots->maxceil, maxX = c.slots->maxX;
    for (size_t ij = (size_t)blockIdx.x * blockDim.x + threadIdx.x; ij < L2; ij += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(ij / L), j = (int)(ij % L);
        double v[8];
        double pos2 = pos2_given ? pos2_given[ij] : search_pos(c.search, lv, mul(c.phi2[ij], T));
        c.posB2x[ij] = pos2;
        if (!live) {
            for (int k = 0; k < 8; k += 2) { v[k] = c.KR[0].x; v[k + 1] = c.KR[0].y; }
        } else {
            // A1, A2: index_vec.cpp:15-61
            const double* w1 = c.wA1 + ij * m;
            const double* w2 = c.wA2 + ij * m;
            v[0] = ip_exact(w1, KRl + c.iA1[ij], m, 0);
            v[1] = ip_exact(w1, KRl + c.iA1[ij], m, 1);
            v[2] = ip_exact(w2, KRl + c.iA2[ij], m, 0);
            v[3] = ip_exact(w2, KRl + c.iA2[ij], m, 1);
            if (c.logr) {  // index_vec.cpp:24-57
                v[1] = ip_log_exact(w1, KRl + c.iA1[ij], m, v[1]);
                v[3] = ip_log_exact(w2, KRl + c.iA2[ij], m, v[3]);
            }
            // B1: index_vec.cpp:63-136
            b1_exact(c, nrows, maxceil, i, j, v[4], v[5]);
            // B2: index_mat.cpp:18-91
            {
                long long X = (long long)pos2;
                if (X > maxX) X = maxX;
                if (X < 1) X = 1;
                const double x = sub(pos2, (double)X), x2 = mul(x, x), x3 = mul(x2, x);
                const size_t base = (size_t)(X - 1) * L + c.iB2[ij];
                const double* w = c.wB2 + ij * m;
                for (int comp = 0; comp < 2; ++comp) {
                    const double S0 = ip_exact(w, c.KR + base, m, comp);
                    const double D1 = ip_exact(w, c.dKR + base + L, m, comp);
                    const double S1 = ip_exact(w, c.KR + base + L, m, comp);
                    double val;
                    if (X < nrows - 1) {
                        const double D2 = ip_exact(w, c.dKR + base + 2 * L, m, comp);
                        const double e0 = add(sub(1.0, mul(3.0, x2)), mul(2.0, x3));
                        const double e1 = add(sub(x, mul(2.0, x2)), x3);
                        const double e2 = sub(mul(3.0, x2), mul(2.0, x3));
                        const double e3 = add(-x2, x3);
                        val = add(add(add(mul(e0, S0), mul(e1, D1)), mul(e2, S1)), dvd(mul(e3, D2), c.dtr[X + 1]));
                        if (comp == 1 && c.logr && S0 > 0.0 && S1 > 0.0)  // index_mat.cpp:47-58
                            val = exp(add(add(add(mul(e0, log(S0)), mul(e1, dvd(D1, S0))), mul(e2, log(S1))),
                                          mul(dvd(e3, c.dtr[X + 1]), dvd(D2, S1))));
                    } else {
                        val = add(add(mul(sub(1.0, x2), S0), mul(x2, S1)), mul(sub(x, x2), D1));
                        if (comp == 1 && c.logr && S0 > 0.0 && S1 > 0.0)  // index_mat.cpp:76-82
                            val = exp(add(add(mul(sub(1.0, x2), log(S0)), mul(x2, log(S1))), mul(sub(x, x2), dvd(D1, S0))));
                    }
                    v[6 + comp] = val;
                }
            }
        }
        for (int k = 0; k < 8; ++k) c.ip[(size_t)k * L2 + ij] = v[k];
        // Sigma (math_sigma.cpp:7-62): SigmaK = f'(QK), SigmaR = f''(QK) QR
        for (int f = 0; f < 4; ++f) {
            c.ip[(size_t)(8 + 2 * f) * L2 + ij] = Df_x(Mo, v[2 * f]);
            c.ip[(size_t)(9 + 2 * f) * L2 + ij] = mul(DDf_x(Mo, v[2 * f]), v[2 * f + 1]);
        }
    }
}

// rInt: index_vec.cpp:138-156
__global__ void k_rint_exact(const DevCtx c, const int nrows) {
    const int L = c.L;
    const bool live = c.t1grid[nrows - 1] > 0.0;
    const int maxceil = c.slots->maxceil;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < L; i += gridDim.x * blockDim.x) {
        if (!live) { c.rint[i] = c.rvec[0]; continue; }
        const double pos = c.posB1x[i];
        long long F = (long long)floor(pos);
        if (F < 1) F = 1; else if (F > maxceil) F = maxceil;
        const double u = sub((double)F, pos), u2 = mul(u, u), u3 = mul(u, mul(u, u));
        double r;
        if (F < nrows - 1) {
            const double e0 = sub(sub(1.0, mul(3.0, u2)), mul(2.0, u3));
            const double e1 = add(mul(3.0, u2), mul(2.0, u3));
            const double e2 = add(add(u, mul(2.0, u2)), u3);
            r = sub(sub(add(mul(e0, c.rvec[F - 1]), mul(e1, c.rvec[F])), mul(e2, c.drvec[F])),
                    dvd(mul(add(u2, u3), c.drvec[F + 1]), c.dtr[F + 1]));
        } else {
            r = sub(add(mul(sub(1.0, u2), c.rvec[F - 1]), mul(u2, c.rvec[F])), mul(add(u, u2), c.drvec[F]));
        }
        c.rint[i] = r;
    }
}

// Sums in the reference's order.  The terms of a sum are formed by all threads, SUM_W columns
// at a time, in shared memory; one thread per sum adds them in column order.  So only the adds
// are a serial chain (512 of them ~13 us), not the loads and the products (L = 512: rstep 439
// -> 26 us, energy 257 -> 23, QKRstep, eight sums a row, 759 -> 36).
constexpr int SUM_W = 256;  // columns per block of terms, and threads of a CTA
template <int N>
using SumTerms = double[N][SUM_W + 1];  // + 1: the adding threads read different banks
// term(j, put) forms column j's N terms and hands them over with put(k, value); thread k < N
// returns sum k
template <int N, typename Term>
__device__ __forceinline__ double ordered_sums(const int L, SumTerms<N>& s_t, Term term) {
    double sum = 0.0;
    for (int j0 = 0; j0 < L; j0 += SUM_W) {
        const int w = min(SUM_W, L - j0);
        if (threadIdx.x < w) term(j0 + threadIdx.x, [&](int k, double v) { s_t[k][threadIdx.x] = v; });
        __syncthreads();
        if (threadIdx.x < N) {
            const double* t = s_t[threadIdx.x];
#pragma unroll 8
            for (int q = 0; q < w; ++q) sum = add(sum, t[q]);
        }
        __syncthreads();
    }
    return sum;
}

// QKstep / QRstep (time_steps.cpp:27-47, 94-100) on the materialized arrays, a CTA per row
__global__ void __launch_bounds__(SUM_W) k_qkr_exact(const DevCtx c, const int nrows, double2* out) {
    const int L = c.L, i = blockIdx.x;
    const size_t L2 = (size_t)L * L, row = (size_t)i * L;
    const DModel Mo = c.M;
    const double t = c.t1grid[nrows - 1];
    const double* ip = c.ip;
    const double2* q = c.KR + (size_t)(nrows - 1) * L;
    __shared__ SumTerms<8> s_t;
    __shared__ double s_sum[8];
    // ConvA/ConvR rows in convolution.cpp:5-50 order
    const double sum = ordered_sums<8>(L, s_t, [&](int j, auto put) {
        const double w = c.integ[j];
        const double* p = ip + row + j;
        const double wRA2 = mul(w, p[11 * L2]), wQRA2 = mul(w, p[3 * L2]);
        put(0, mul(wRA2, p[6 * L2]));                // SigmaRA2, QKB2
        put(1, mul(mul(w, p[9 * L2]), p[4 * L2]));   // SigmaRA1, QKB1
        put(2, mul(mul(w, p[8 * L2]), p[5 * L2]));   // SigmaKA1, QRB1
        put(3, mul(wQRA2, p[14 * L2]));              // QRA2, SigmaKB2
        put(4, mul(mul(w, p[1 * L2]), p[12 * L2]));  // QRA1, SigmaKB1
        put(5, mul(mul(w, p[0 * L2]), p[13 * L2]));  // QKA1, SigmaRB1
        put(6, mul(wRA2, p[7 * L2]));                // SigmaRA2, QRB2
        put(7, mul(wQRA2, p[15 * L2]));              // QRA2, SigmaRB2
    });
    if (threadIdx.x < 8) s_sum[threadIdx.x] = sum;
    __syncthreads();
    if (threadIdx.x != 0) return;
    const double th = c.theta[i];
    const double tA = mul(t, th), tR = mul(t, sub(1.0, th));
    const double rE = c.rint[L - 1];
    const double q0 = q[0].x;
    const double cR1 = mul(s_sum[0], tR), cA1 = mul(s_sum[1], tA), cA2 = mul(s_sum[2], tA);
    const double cR2 = mul(s_sum[3], tR), cA3 = mul(s_sum[4], tA), cA4 = mul(s_sum[5], tA);
    const double cR3 = mul(s_sum[6], tR), cR4 = mul(s_sum[7], tR);
    const double qb = ip[4 * L2 + row];
    const double fac1 = dvd(Df_x(Mo, q0), Mo.T0);
    const double d1 = add(add(add(add(mul(qb, fac1), mul(q[i].x, -rE)), cR1), cA1), cA2);
    const double fac2 = dvd(q0, Mo.T0);
    const double d2 = sub(add(add(add(add(mul(Df_x(Mo, qb), fac2), mul(q[i].y, mul(2.0, Mo.Gamma))), cR2), cA3), cA4),
                          mul(q[i].x, c.rint[i]));
    const double hK = add(d1, mul(d2, th));
    const double e1 = add(mul(q[i].y, -rE), cR3);
    const double e2 = sub(mul(q[i].y, c.rint[i]), cR4);
    out[i] = make_double2(hK, add(e1, mul(e2, th)));
}

// rstep (time_steps.cpp:83-92), one CTA
__global__ void __launch_bounds__(SUM_W) k_rstep_exact(const DevCtx c, const int nrows, double* out) {
    const DModel Mo = c.M;
    const double t = c.t1grid[nrows - 1];
    const double2* q = c.KR + (size_t)(nrows - 1) * c.L;
    __shared__ SumTerms<2> s_t;
    __shared__ double s_sum[2];
    const double sum = ordered_sums<2>(c.L, s_t, [&](int j, auto put) {
        const double2 v = q[j];
        const double tw = mul(t, c.integ[j]);
        put(0, mul(mul(tw, mul(DDf_x(Mo, v.x), v.y)), v.x));
        put(1, mul(mul(tw, Df_x(Mo, v.x)), v.y));
    });
    if (threadIdx.x < 2) s_sum[threadIdx.x] = sum;
    __syncthreads();
    if (threadIdx.x == 0)
        out[0] = add(add(add(Mo.Gamma, s_sum[0]), s_sum[1]), dvd(mul(Df_x(Mo, q[0].x), q[0].x), Mo.T0));
}

// drstep2 (time_steps.cpp:117-125), one CTA
__global__ void __launch_bounds__(SUM_W) k_drstep2_exact(const DevCtx c, const double* qK, const double* qR,
                                                         const double* dqK, const double* dqR, const double t, double* out) {
    const DModel Mo = c.M;
    __shared__ SumTerms<6> s_t;
    __shared__ double s_sum[6];
    const double sum = ordered_sums<6>(c.L, s_t, [&](int j, auto put) {
        const double q = qK[j], r = qR[j], dq = dqK[j], dr = dqR[j];
        const double sk = Df_x(Mo, q), sr = mul(DDf_x(Mo, q), r);
        const double dsk = add(mul(DDf_x(Mo, q), dq), mul(0.0, dr));
        const double dsr = add(mul(mul(DDDf_x(Mo, q), r), dq), mul(DDf_x(Mo, q), dr));
        const double w = c.integ[j], tw = mul(t, w);
        put(0, mul(mul(mul(1.0, w), sr), q));
        put(1, mul(mul(mul(1.0, w), sk), r));
        put(2, mul(mul(tw, dsr), q));
        put(3, mul(mul(tw, dsk), r));
        put(4, mul(mul(tw, sr), dq));
        put(5, mul(mul(tw, sk), dr));
    });
    if (threadIdx.x < 6) s_sum[threadIdx.x] = sum;
    __syncthreads();
    if (threadIdx.x != 0) return;
    const double dsk0 = add(mul(DDf_x(Mo, qK[0]), dqK[0]), mul(0.0, dqR[0])), sk0 = Df_x(Mo, qK[0]);
    const double term = dvd(add(mul(dsk0, qK[0]), mul(sk0, dqK[0])), Mo.T0);
    out[0] = add(add(add(add(add(add(s_sum[0], s_sum[1]), s_sum[2]), s_sum[3]), s_sum[4]), s_sum[5]), term);
}

// energy at t1grid.back() (time_steps.cu:641-674 with the CPU sum order), one CTA
__global__ void __launch_bounds__(SUM_W) k_energy_exact(const DevCtx c, const int nrows, double* out) {
    const DModel Mo = c.M;
    const double t = c.t1grid[nrows - 1];
    const double2* q = c.KR + (size_t)(nrows - 1) * c.L;
    __shared__ SumTerms<1> s_t;
    const double sum = ordered_sums<1>(c.L, s_t, [&](int j, auto put) {
        const double2 v = q[j];
        put(0, mul(mul(mul(t, c.integ[j]), Df_x(Mo, v.x)), v.y));
    });
    if (threadIdx.x == 0) out[0] = -add(sum, dvd(Df_x(Mo, q[0].x), Mo.T0));
}

// ConvA / ConvR on device arrays (convolution.cpp:5-50)
__global__ void __launch_bounds__(SUM_W) k_conv_exact(const DevCtx c, const int kind, const double* f, const double* g,
                                                      const int depth, const double t, double* out) {
    const int L = c.L, r = blockIdx.x;
    __shared__ SumTerms<1> s_t;
    const double sum = ordered_sums<1>(L, s_t, [&](int j, auto put) {
        const size_t e = (size_t)r * L + j;
        const double w = depth == 1 ? mul(t, c.integ[j]) : c.integ[j];
        put(0, mul(mul(w, f[e]), g[e]));
    });
    if (threadIdx.x != 0) return;
    if (depth == 1) out[0] = sum;
    else out[r] = mul(sum, kind == 0 ? mul(t, c.theta[r]) : mul(t, sub(1.0, c.theta[r])));
}

__global__ void k_search(const int mode, const double* list, const int nlist, const double* elem,
                         const size_t nelem, double* out) {
    const double last = list[nlist - 1];
    const ListView lv{list, nlist, last};
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < nelem; k += (size_t)gridDim.x * blockDim.x)
        out[k] = search_pos(mode, lv, __dmul_rn(elem[k], last));
}

// x / d correctly rounded for many x and one d: y = RN(1/d); q = x y is off by an ulp or two,
// one Newton correction q + (x - q d) y leaves it within one, and from there the same step
// rounds correctly (Markstein, IBM J. Res. Dev. 34, 1990).  Five FP64 instructions; the general
// division where y or the remainders could leave the normal range.
struct DivBy {
    double d, y;
    bool ok;
    __device__ __forceinline__ void set(double d_) {
        d = d_;
        y = dvd(1.0, d_);
        ok = fabs(d) > 1e-150 && fabs(d) < 1e150;
    }
    __device__ __forceinline__ double operator()(double x) const {
        const double m = fabs(x);
        if (!ok || !(m > 1e-120 && m < 1e120)) return m == 0.0 && ok ? 0.0 : dvd(x, d);
        double q = mul(x, y);
        q = fma(fma(-q, d, x), y, q);
        return fma(fma(-q, d, x), y, q);
    }
};

// Sparsify indicator of every node (bit 0 evaluated, bit 1 val < thr, bit 2 val >= thr): val is a
// sum over the columns in the reference's order.  A CTA takes SP_NODES evaluated nodes; its
// warps form the terms of 32 columns of a node side by side (coalesced rows), the node's own
// thread adds them in order.  Bound by the FP64 pipe (16 instructions a term: the two
// divisions share each row's divisor); n = 8000, L = 512: 847 us with a thread per node, whole
// divisions and strided reads; the whole sparsify pass 1.56 -> 0.68 ms.
constexpr int SP_NODES = 16, SP_T = 256;
__global__ void __launch_bounds__(SP_T) k_sparsify_flags(const DevCtx c, const int n, const int variant, const double thr,
                                                         unsigned char* flags) {
    const int L = c.L, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __shared__ double s_t[2][2][SP_NODES][33];  // [tile parity][QK, QR]: the adds of one tile run beside the next one's terms
    __shared__ double s_td2[SP_NODES], s_sc[SP_NODES];
    __shared__ DivBy s_by1[SP_NODES], s_by3[SP_NODES];
    // evaluated nodes: 2 <= i < n - 1, of variant 2 the even ones
    const int step = variant == 2 ? 2 : 1, e0 = blockIdx.x * SP_NODES;
    auto node = [&](int k) { return 2 + (e0 + k) * step; };
    if (threadIdx.x < SP_NODES) {
        const int k = threadIdx.x, i = node(k);
        if (i + 1 < n) {
            const double tl = c.t1grid[i - 2], tm = c.t1grid[i];
            s_td2[k] = sub(tm, tl);
            s_sc[k] = dvd(s_td2[k], 12.0);
            s_by1[k].set(sub(c.t1grid[i - 1], tl));
            s_by3[k].set(sub(c.t1grid[i + 1], tm));
        }
    }
    __syncthreads();
    double val = 0.0;  // of node(threadIdx.x), threadIdx.x < SP_NODES
    // variants 0, 1: all QK terms, then all QR terms; variant 2: the two of a column in turn
    const int passes = variant == 2 ? 1 : 2, tiles = (L + 31) / 32;
    for (int tile = 0; tile < passes * tiles; ++tile) {
        const int pass = tile >= tiles, j0 = (tile - pass * tiles) * 32;
        double(*t)[SP_NODES][33] = s_t[tile & 1];
        for (int k = warp; k < SP_NODES; k += SP_T / 32) {
            const int i = node(k), j = j0 + lane;
            if (i + 1 >= n || j >= L) continue;
            const double td2 = s_td2[k], sc = s_sc[k];
            const DivBy by1 = s_by1[k], by3 = s_by3[k];
            auto term = [&](double f1, double df1, double df2) {
                return fabs(mul(sc, sub(mul(2.0, f1), mul(td2, add(by1(df1), by3(df2))))));
            };
            const size_t at = (size_t)i * L + j;
            const double2 x0 = c.KR[at], x2 = c.KR[at - 2 * (size_t)L], d1 = c.dKR[at - L], d3 = c.dKR[at + L];
            if (variant == 2 || pass == 0) t[0][k][lane] = term(sub(x0.x, x2.x), d1.x, d3.x);
            if (variant == 2 || pass == 1) t[1][k][lane] = term(sub(x0.y, x2.y), d1.y, d3.y);
        }
        __syncthreads();
        if (threadIdx.x < SP_NODES && node(threadIdx.x) + 1 < n) {
            const int w = min(32, L - j0);
            for (int q = 0; q < w; ++q) {
                if (variant == 2) {
                    val = add(val, t[0][threadIdx.x][q]);
                    val = add(val, t[1][threadIdx.x][q]);
                } else {
                    val = add(val, t[pass][threadIdx.x][q]);
                }
            }
        }
    }
    if (threadIdx.x < SP_NODES) {
        const int i = node(threadIdx.x);
        if (i + 1 < n) {
            if (variant == 0) {
                const double tl = c.t1grid[i - 2], tm = c.t1grid[i];
                const double td1 = sub(c.t1grid[i - 1], tl), td2 = sub(tm, tl), td3 = sub(c.t1grid[i + 1], tm);
                const double f1 = sub(c.rvec[i], c.rvec[i - 2]);
                val = add(val, fabs(mul(dvd(td2, 12.0), sub(mul(2.0, f1), mul(td2, add(dvd(c.drvec[i - 1], td1),
                                                                                       dvd(c.drvec[i + 1], td3)))))));
            }
            flags[i] = (unsigned char)(1 | (val < thr ? 2 : 0) | (val >= thr ? 4 : 0));
        }
    }
    // the nodes nothing is evaluated for
    const int t = blockIdx.x * SP_T + threadIdx.x;
    for (int i = t; i < n; i += gridDim.x * SP_T)
        if (i < 2 || i + 1 >= n || (variant == 2 && (i & 1))) flags[i] = 0;
}

// Rows [r0, r0 + rows) of the compacted history into staging
__global__ void k_compact(const DevCtx c, const int* inds, const int* indsD, const double* tfac, const int r0,
                          const int rows, double2* KRn, double2* dKRn, double* rn, double* drn) {
    const int L = c.L;
    const size_t total = (size_t)rows * L;
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const int r = r0 + (int)(e / L), j = (int)(e % L);
        KRn[e] = c.KR[(size_t)inds[r] * L + j];
        const double f = tfac ? tfac[r] : 1.0;
        const double2 d = c.dKR[(size_t)indsD[r] * L + j];
        dKRn[e] = make_double2(mul(f, d.x), mul(f, d.y));
        if (j == 0) {
            rn[e / L] = c.rvec[inds[r]];
            drn[e / L] = mul(f, c.drvec[indsD[r]]);
        }
    }
}

__global__ void k_pack(const double* QK, const double* QR, double2* out, size_t count) {
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < count; e += (size_t)gridDim.x * blockDim.x)
        out[e] = make_double2(QK[e], QR[e]);
}
__global__ void k_unpack(const double2* in, double* QK, double* QR, size_t count) {
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < count; e += (size_t)gridDim.x * blockDim.x) {
        const double2 v = in[e];
        QK[e] = v.x;
        QR[e] = v.y;
    }
}

// FP64 throughput probe: 8 independent FMA chains per thread.
__global__ void k_fp64_probe(double* out, int iters) {
    double a[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = 1.0 + 1e-3 * (threadIdx.x + k);
    const double b = 0.999999, c = 1e-7;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int k = 0; k < 8; ++k) a[k] = fma(a[k], b, c);
    }
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += a[k];
    if (s == 12345.678) out[0] = s;  // keeps the chains live
}

// ------------------------------------------------------------------------
// launch wrappers
template <int M, int K, int P, int P2, bool LOGR, bool KEEP, bool SPLIT = false>
static cudaError_t launch_main_t(const DevCtx& c, int s, cudaStream_t st) {
    const int nthr = SPLIT ? 128 : c.tpb;
    dim3 grid(c.nch, c.L + (c.L + nthr - 1) / nthr), block(nthr);
    const size_t smem = (size_t)c.L * (LOGR ? sizeof(double2) + sizeof(double) : sizeof(double2));
    static std::atomic<unsigned long long> devs{0};
    const cudaError_t e = raise_smem_limit(k_main<M, K, P, P2, LOGR, KEEP, SPLIT>, smem, 4096 * (int)(smem / c.L), devs);
    if (e != cudaSuccess) return e;
    return launch_pdl(k_main<M, K, P, P2, LOGR, KEEP, SPLIT>, grid, block, smem, st, c, s);
}

// Lengths up to which k_main takes two threads a target (`run` of one RK54 step, one thread a target -> two:
// L = 64 166 -> 142 us, 128 172 -> 154, 192 198 -> 191, 224 230 -> 231, 320 325 -> 330): beyond
// 192 a row has four chunks and its warps fill the schedulers by themselves.
constexpr int SPLIT_L = 192;

template <int M, int P, int P2, bool LOGR>
static cudaError_t launch_main_kl(const DevCtx& c, int s, cudaStream_t st) {
    if (c.b2key && c.kpt == 1 && c.tpb == 64 && c.L <= SPLIT_L) return launch_main_t<M, 1, P, P2, LOGR, true, true>(c, s, st);
    if (c.b2key) return c.kpt == 1 ? launch_main_t<M, 1, P, P2, LOGR, true>(c, s, st)
                                   : launch_main_t<M, 2, P, P2, LOGR, true>(c, s, st);
    switch (c.kpt) {
        case 1: return launch_main_t<M, 1, P, P2, LOGR, false>(c, s, st);
        case 2: return launch_main_t<M, 2, P, P2, LOGR, false>(c, s, st);
        default: return launch_main_t<M, 4, P, P2, LOGR, false>(c, s, st);
    }
}

// the log-space form is built once, on the generic-exponent model
template <int M, int P, int P2>
static cudaError_t launch_main_k(const DevCtx& c, int s, cudaStream_t st) {
    return c.logr ? launch_main_kl<M, -1, -1, true>(c, s, st) : launch_main_kl<M, P, P2, false>(c, s, st);
}

template <int P, int P2>
static cudaError_t launch_stage_pp(const DevCtx& c, int s, cudaStream_t st, bool gather) {
    cudaError_t e = cudaSuccess;
    if (gather && c.mixed) e = launch_main_mixed(c, s, st);
    else if (gather) e = c.m == 10 ? launch_main_k<10, P, P2>(c, s, st) : launch_main_k<0, P, P2>(c, s, st);
    if (e != cudaSuccess) return e;
    const int G = (c.L + EPI_ROWS - 1) / EPI_ROWS;
    if (c.mixed) return launch_pdl(k_epi<P, P2, true>, dim3(G), dim3(EPI_T), 0, st, c, s);
    return launch_pdl(k_epi<P, P2, false>, dim3(G), dim3(EPI_T), 0, st, c, s);
}

cudaError_t launch_stage(const DevCtx& c, int s, cudaStream_t st, bool gather) {
    if (c.M.p == 3 && c.M.p2 == 4) return launch_stage_pp<3, 4>(c, s, st, gather);
    if (c.M.p == 3 && c.M.p2 == 0) return launch_stage_pp<3, 0>(c, s, st, gather);
    return launch_stage_pp<-1, -1>(c, s, st, gather);
}

// Nothing goes on from a lone right-hand side, so its B2 sums go to no planes: with / without
// them a call measures, at L = 256, 512, 1024, 2048: plain 70 / 60, 82 / 72, 159 / 120, 470 /
// 345 us; (hi, lo) 70 / 69, 92 / 84, 207 / 170, 819 / 698; FP64 82 / 81, 155 / 150, 430 / 416,
// 1559 / 1477.  FP64 up to SPLIT_L keeps them: two threads a target 59 us, one 63 (L = 33).
cudaError_t launch_rhs(const DevCtx& c, cudaStream_t st) {
    DevCtx one = c;
    if (c.mixed || c.L > SPLIT_L) one.b2key = nullptr;
    return launch_stage(one, 0, st);
}

template <int P, int P2>
static cudaError_t launch_main_pp(const DevCtx& c, int s, cudaStream_t st) {
    return c.m == 10 ? launch_main_k<10, P, P2>(c, s, st) : launch_main_k<0, P, P2>(c, s, st);
}

cudaError_t launch_main_only(const DevCtx& c, int s, cudaStream_t st) {
    if (c.mixed) return launch_main_mixed(c, s, st);
    if (c.M.p == 3 && c.M.p2 == 4) return launch_main_pp<3, 4>(c, s, st);
    if (c.M.p == 3 && c.M.p2 == 0) return launch_main_pp<3, 0>(c, s, st);
    return launch_main_pp<-1, -1>(c, s, st);
}

cudaError_t launch_epi_only(const DevCtx& c, int s, cudaStream_t st) {
    const int G = (c.L + EPI_ROWS - 1) / EPI_ROWS;
    if (c.mixed) {
        if (c.M.p == 3 && c.M.p2 == 4) k_epi<3, 4, true><<<G, EPI_T, 0, st>>>(c, s);
        else if (c.M.p == 3 && c.M.p2 == 0) k_epi<3, 0, true><<<G, EPI_T, 0, st>>>(c, s);
        else k_epi<-1, -1, true><<<G, EPI_T, 0, st>>>(c, s);
    } else {
        if (c.M.p == 3 && c.M.p2 == 4) k_epi<3, 4, false><<<G, EPI_T, 0, st>>>(c, s);
        else if (c.M.p == 3 && c.M.p2 == 0) k_epi<3, 0, false><<<G, EPI_T, 0, st>>>(c, s);
        else k_epi<-1, -1, false><<<G, EPI_T, 0, st>>>(c, s);
    }
    return cudaGetLastError();
}

cudaError_t launch_pos_init(const DevCtx& c, int nrows, cudaStream_t st) {
    k_pos_init<<<(c.L + 63) / 64, 64, 0, st>>>(c, nrows);
    return cudaGetLastError();
}

cudaError_t launch_interp_exact(const DevCtx& c, int nrows, const double* p1, const double* p2, cudaStream_t st) {
    k_pos_b1_exact<<<1, 256, 0, st>>>(c, nrows, p1, p2);
    const size_t L2 = (size_t)c.L * c.L;
    const int blocks = (int)((L2 + 255) / 256 < 4096 ? (L2 + 255) / 256 : 4096);
    k_interp_exact<<<blocks, 256, 0, st>>>(c, nrows, p2);
    k_rint_exact<<<(c.L + 127) / 128, 128, 0, st>>>(c, nrows);
    return cudaGetLastError();
}

cudaError_t launch_b1_exact(const DevCtx& c, int nrows, double* qk, double* qr, cudaStream_t st) {
    k_pos_b1_exact<<<1, 256, 0, st>>>(c, nrows, nullptr, nullptr);
    const size_t L2 = (size_t)c.L * c.L;
    const int blocks = (int)((L2 + 255) / 256 < 4096 ? (L2 + 255) / 256 : 4096);
    k_b1_exact<<<blocks, 256, 0, st>>>(c, nrows, qk, qr);
    return cudaGetLastError();
}

cudaError_t launch_qkr_exact(const DevCtx& c, int nrows, double2* out, cudaStream_t st) {
    k_qkr_exact<<<c.L, SUM_W, 0, st>>>(c, nrows, out);
    return cudaGetLastError();
}

cudaError_t launch_rstep_exact(const DevCtx& c, int nrows, double* out, cudaStream_t st) {
    k_rstep_exact<<<1, SUM_W, 0, st>>>(c, nrows, out);
    return cudaGetLastError();
}

cudaError_t launch_drstep2_exact(const DevCtx& c, const double* qK, const double* qR, const double* dqK,
                                 const double* dqR, double t, double* out, cudaStream_t st) {
    k_drstep2_exact<<<1, SUM_W, 0, st>>>(c, qK, qR, dqK, dqR, t, out);
    return cudaGetLastError();
}

cudaError_t launch_energy_exact(const DevCtx& c, int nrows, double* out, cudaStream_t st) {
    k_energy_exact<<<1, SUM_W, 0, st>>>(c, nrows, out);
    return cudaGetLastError();
}

cudaError_t launch_conv_exact(const DevCtx& c, int kind, const double* f, const double* g, size_t n, double t,
                              double* out, cudaStream_t st) {
    const int depth = (int)(n / c.L);
    k_conv_exact<<<depth, SUM_W, 0, st>>>(c, kind, f, g, depth, t, out);
    return cudaGetLastError();
}

cudaError_t launch_search(const DevCtx& c, const double* list, size_t nlist, const double* elem, size_t nelem,
                          double* out, cudaStream_t st) {
    const int blocks = (int)((nelem + 255) / 256 < 4096 ? (nelem + 255) / 256 : 4096);
    k_search<<<blocks > 0 ? blocks : 1, 256, 0, st>>>(c.search, list, (int)nlist, elem, nelem, out);
    return cudaGetLastError();
}

cudaError_t launch_sparsify_flags(const DevCtx& c, int n, int variant, double thr, unsigned char* flags,
                                  cudaStream_t st) {
    const int nodes = n < 4 ? 0 : variant == 2 ? (n - 2) / 2 : n - 3;
    k_sparsify_flags<<<std::max(1, (nodes + SP_NODES - 1) / SP_NODES), SP_T, 0, st>>>(c, n, variant, thr, flags);
    return cudaGetLastError();
}

// The history compacted in place: row r takes inds[r] and, scaled, derivative row indsD[r].
// Both are at or above r and increase, so chunks of rows go through the staging buffers in
// order without reaching rows still to be read.
cudaError_t launch_compact(const DevCtx& c, const int* inds, const int* indsD, const double* tfac, int k,
                           const CompactBuf& buf, cudaStream_t st) {
    const size_t L = c.L, per = buf.elems / L;  // rows staged at a time
    for (size_t r0 = 0; r0 < (size_t)k; r0 += per) {
        const size_t rows = std::min(per, (size_t)k - r0), total = rows * L;
        const int blocks = (int)((total + 255) / 256 < 8192 ? (total + 255) / 256 : 8192);
        k_compact<<<blocks, 256, 0, st>>>(c, inds, indsD, tfac, (int)r0, (int)rows, buf.KR, buf.dKR, buf.r, buf.dr);
        cudaError_t e = cudaGetLastError();
        auto back = [&](void* dst, const void* src, size_t bytes) {
            if (e == cudaSuccess) e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, st);
        };
        back(c.KR + r0 * L, buf.KR, total * sizeof(double2));
        back(c.dKR + r0 * L, buf.dKR, total * sizeof(double2));
        back(c.rvec + r0, buf.r, rows * sizeof(double));
        back(c.drvec + r0, buf.dr, rows * sizeof(double));
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t CompactBuf::reserve(size_t n, size_t L) {
    if (n > cap) {
        for (void* p : {(void*)flags, (void*)idx, (void*)tf, (void*)r, (void*)dr}) cudaFree(p);
        flags = nullptr;
        idx = nullptr;
        tf = r = dr = nullptr;
        cap = 0;
        cudaError_t e = cudaMalloc((void**)&flags, n);
        if (e == cudaSuccess) e = cudaMalloc((void**)&idx, 2 * n * sizeof(int));
        for (double** p : {&tf, &r, &dr})
            if (e == cudaSuccess) e = cudaMalloc((void**)p, n * sizeof(double));
        if (e != cudaSuccess) return e;
        cap = n;
    }
    // counted in elements, so that rows of any length share the bound
    const size_t want = std::min(n * L, (64u << 20) / (2 * sizeof(double2)));
    if (want > elems) {
        cudaFree(KR); cudaFree(dKR);
        KR = dKR = nullptr;
        elems = 0;
        cudaError_t e = cudaMalloc((void**)&KR, want * sizeof(double2));
        if (e == cudaSuccess) e = cudaMalloc((void**)&dKR, want * sizeof(double2));
        if (e != cudaSuccess) return e;
        elems = want;
    }
    return cudaSuccess;
}

void CompactBuf::release() {
    for (void* p : {(void*)flags, (void*)idx, (void*)tf, (void*)KR, (void*)dKR, (void*)r, (void*)dr}) cudaFree(p);
    *this = CompactBuf{};
}

cudaError_t launch_pack_rows(const double* QK, const double* QR, double2* out, size_t count, cudaStream_t st) {
    const int blocks = (int)((count + 255) / 256 < 8192 ? (count + 255) / 256 : 8192);
    k_pack<<<blocks > 0 ? blocks : 1, 256, 0, st>>>(QK, QR, out, count);
    return cudaGetLastError();
}

cudaError_t launch_fp64_probe(double* out, int blocks, int threads, int iters, cudaStream_t st) {
    k_fp64_probe<<<blocks, threads, 0, st>>>(out, iters);
    return cudaGetLastError();
}

cudaError_t launch_unpack_rows(const double2* in, double* QK, double* QR, size_t count, cudaStream_t st) {
    const int blocks = (int)((count + 255) / 256 < 8192 ? (count + 255) / 256 : 8192);
    k_unpack<<<blocks > 0 ? blocks : 1, 256, 0, st>>>(in, QK, QR, count);
    return cudaGetLastError();
}

// ------------------------------------------------------------------------
// Energy of every history row as the reference writes it at save time
// (computeEnergyHistoryKernel, io_output.cu:61-122):
//   E_k = -t_k (sum_j w_j f'(QK[k,j]) QR[k,j] + f'(QK[k,0]) / T0)
// (the T0 term carries the factor t_k there, unlike energyGPU's per-step E).
// One warp per row, lanes over the columns, a shuffle sum.
__global__ void k_energy_history(const DevCtx c, const int nrows, double* out) {
    const int lane = threadIdx.x & 31;
    const int k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (k >= nrows) return;  // whole warps: k is uniform over a warp
    const int L = c.L;
    const double2* row = c.KR + (size_t)k * L;
    double sum = 0.0;
    for (int j = lane; j < L; j += 32) {
        const double2 v = row[j];
        const double sk = Df_x(c.M, v.x);
        sum = fma(sk * v.y, c.integ[j], sum);
        if (j == 0) sum += sk / c.M.T0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) out[k] = -c.t1grid[k] * sum;
}

cudaError_t launch_energy_history(const DevCtx& c, int nrows, double* out, cudaStream_t st) {
    if (nrows <= 0) return cudaSuccess;
    k_energy_history<<<(nrows + 7) / 8, 256, 0, st>>>(c, nrows, out);
    return cudaGetLastError();
}

}  // namespace dyn
