// Stage epilogue of the DYNAMITE hot path as device functions, shared by the
// single-quench kernel k_epi (dyn_kernels.cu) and the batched epilogue
// (dyn_batch.cu): finish the row reductions, form the EOM right-hand side
// (QKstep/QRstep, time_steps.cpp:27-47,94-100), the RK stage combination
// (tableau or SERK2 recurrence, runge_kutta.cpp:19-252, runge_kutta.cu:397-487),
// write the history row (appendAll/replaceAll, time_steps.cpp:49-81,127-162),
// accumulate r(t) (rstep, time_steps.cpp:83-92), dr/dt at stage 0 (drstep2,
// time_steps.cpp:117-125) and, at the last stage, the error norm and the
// energy terms; the last CTA of a stage folds the per-CTA partials.
#pragma once
#include "dyn_kernels.cuh"

namespace dyn {

// Model helpers of the fused kernels (f', f'', f''' with FMA contraction)
template <int P, int P2>
struct Sig {
    __device__ __forceinline__ static void d12(const DModel& M, double q, double& a, double& b) {
        Sigma<P, P2>::eval(M, q, a, b);
    }
    __device__ __forceinline__ static double d1(const DModel& M, double q) {
        if constexpr (P >= 0) return fma(M.cA, ipow_c<P - 1>(q), M.cB * ipow_c<P2 - 1>(q));
        else return fma(M.cA, ipow_r(q, M.p - 1), M.cB * ipow_r(q, M.p2 - 1));
    }
    __device__ __forceinline__ static double d2(const DModel& M, double q) {
        if constexpr (P >= 0) return fma(M.cC, ipow_c<P - 2>(q), M.cD * ipow_c<P2 - 2>(q));
        else return fma(M.cC, ipow_r(q, M.p - 2), M.cD * ipow_r(q, M.p2 - 2));
    }
    __device__ __forceinline__ static double d3(const DModel& M, double q) {
        if constexpr (P >= 0) return fma(M.cE, ipow_c<P - 3>(q), M.cF * ipow_c<P2 - 3>(q));
        else return fma(M.cE, ipow_r(q, M.p - 3), M.cF * ipow_r(q, M.p2 - 3));
    }
};

// ------------------------------------------------------------------------
// FP64 gathers of the fused kernels (k_main, and the adjoint's recompute)
// sum_d w[d] * x[d] for K and R together (x interleaved)
template <int M>
__device__ __forceinline__ double2 dot2g(const double* __restrict__ w, const double2* __restrict__ x, int m) {
    double2 acc = make_double2(0.0, 0.0);
    if constexpr (M > 0 && (M % 2) == 0) {
        const double2* w2 = reinterpret_cast<const double2*>(w);
#pragma unroll
        for (int d = 0; d < M / 2; ++d) {
            const double2 ww = __ldg(w2 + d);
            const double2 xa = __ldg(x + 2 * d), xb = __ldg(x + 2 * d + 1);
            acc.x = fma(ww.x, xa.x, acc.x);
            acc.y = fma(ww.x, xa.y, acc.y);
            acc.x = fma(ww.y, xb.x, acc.x);
            acc.y = fma(ww.y, xb.y, acc.y);
        }
    } else {
        for (int d = 0; d < m; ++d) {
            const double ww = __ldg(w + d);
            const double2 xa = __ldg(x + d);
            acc.x = fma(ww, xa.x, acc.x);
            acc.y = fma(ww, xa.y, acc.y);
        }
    }
    return acc;
}

template <int M>
__device__ __forceinline__ double2 dot2s(const double* __restrict__ w, const double2* x, int m) {
    double2 acc = make_double2(0.0, 0.0);
    if constexpr (M > 0 && (M % 2) == 0) {
        const double2* w2 = reinterpret_cast<const double2*>(w);
#pragma unroll
        for (int d = 0; d < M / 2; ++d) {
            const double2 ww = __ldg(w2 + d);
            const double2 xa = x[2 * d], xb = x[2 * d + 1];
            acc.x = fma(ww.x, xa.x, acc.x);
            acc.y = fma(ww.x, xa.y, acc.y);
            acc.x = fma(ww.y, xb.x, acc.x);
            acc.y = fma(ww.y, xb.y, acc.y);
        }
    } else {
        for (int d = 0; d < m; ++d) {
            const double ww = __ldg(w + d);
            const double2 xa = x[d];
            acc.x = fma(ww, xa.x, acc.x);
            acc.y = fma(ww, xa.y, acc.y);
        }
    }
    return acc;
}

// B1 interpolation of a row at position pos (index_vec.cu:399-441 form, with the
// per-row division folded into c3); idtr(k) gives 1/delta_t_ratio of row k.  Written
// out in fused operations so that every kernel that forms it rounds alike.
template <typename InvDtr>
__device__ __forceinline__ B1Row b1_at(double pos, int maxceil, int nrows, InvDtr idtr) {
    B1Row r;
    long long F = (long long)floor(pos);
    if (F < 1) F = 1; else if (F > maxceil) F = maxceil;
    r.F = (int)F;
    const double u = __dsub_rn((double)F, pos), u2 = __dmul_rn(u, u), u3 = __dmul_rn(u2, u);
    r.cubic = F < nrows - 1;
    if (r.cubic) {
        r.c1 = fma(2.0, u3, __dmul_rn(3.0, u2));
        r.c0 = __dsub_rn(1.0, r.c1);
        r.c2 = __dadd_rn(fma(2.0, u2, u), u3);
        r.c3 = __dmul_rn(__dadd_rn(u2, u3), idtr(r.F + 1));
    } else {
        r.c0 = __dsub_rn(1.0, u2);
        r.c1 = u2;
        r.c2 = __dadd_rn(u, u2);
        r.c3 = 0.0;
    }
    return r;
}
__device__ __forceinline__ B1Row b1_row(const DevCtx& c, double pos, int maxceil, int nrows) {
    return b1_at(pos, maxceil, nrows, [&](int k) { return c.inv_dtr[k]; });
}

// What a stage needs once per target row and no target does: QK^{B1}[i,0] and rInt_i, and
// the next stage's B1 position (theta_i T_next in the list that the row this stage writes
// will end), and C(t,0) from row 0.  Not in the epilogue, whose other CTAs already overwrite
// the newest row: single contexts run these chains of dependent loads beside the gathers in
// CTAs of their own (side_row), the batch in two threads of the row's CTA (its other CTAs
// fill the gap; CTAs of their own made its gather 3 % slower).
__device__ __forceinline__ double2 row_value(const DevCtx& c, const StageDev& sp, const B1Row& r) {
    const int L = c.L;
    if (!(sp.T > 0.0)) return make_double2(c.KR[0].x, c.rvec[0]);
    const double2 x0 = c.KR[(size_t)(r.F - 1) * L], x1 = c.KR[(size_t)r.F * L];
    const double2 d1 = c.dKR[(size_t)r.F * L];
    double qb = fma(-r.c2, d1.x, fma(r.c1, x1.x, __dmul_rn(r.c0, x0.x)));
    double ri = fma(-r.c2, c.drvec[r.F], fma(r.c1, c.rvec[r.F], __dmul_rn(r.c0, c.rvec[r.F - 1])));
    if (r.cubic) {
        qb = fma(-r.c3, c.dKR[(size_t)(r.F + 1) * L].x, qb);
        ri = fma(-r.c3, c.drvec[r.F + 1], ri);
    }
    return make_double2(qb, ri);
}
__device__ __forceinline__ double next_position(const DevCtx& c, const StageDev& sp, int F, int i) {
    const ListView lv{c.t1grid, sp.nrows_next, sp.T_next};
    return search_pos_near(c.search, lv, __dmul_rn(c.theta[i], sp.T_next), F - 1);
}
__device__ __forceinline__ void side_value(const DevCtx& c, const StageDev& sp, const B1Row& r, int i) {
    c.rowval[i] = row_value(c, sp, r);
    if (i == 0) c.slots->q0 = c.KR[(size_t)(sp.nrows - 1) * c.L].x;
}
__device__ __forceinline__ void side_position(const DevCtx& c, const StageDev& sp, int F, int i) {
    if (sp.kind != KIND_RHS && sp.pos_reuse < 0) c.posB1x_next[i] = next_position(c, sp, F, i);
}
__device__ __forceinline__ void side_row(const DevCtx& c, const StageDev& sp, int i) {
    B1Row r = {};
    if (sp.T > 0.0) r = c.b1[i];
    side_value(c, sp, r, i);
    side_position(c, sp, r.F, i);
}

namespace epi {

// A warp's FP64 instruction costs 64 cycles here however few lanes or dependences it has (a
// quarter of the SM's rate: its four schedulers each feed their own unit), and the ~190 of a
// row were the time of a one-warp CTA (k_epi at L = 64 12.2 us, now 8.4; L = 512 (hi, lo)
// 14.3, now 10.4).  So EPI_ROWS rows, one per
// lane, are taken by four warps, each with its share of a row's chain:
//   warp 0: QK: right-hand side, new value, r(t) terms; warp 1: the part of QK's right-hand
//   side with theta, dr/dt terms at stage 0; warp 2: QR: right-hand side, new value;
//   warp 3: the next stage's B1 row.
constexpr int TAB_STAGES = 10;  // most stages of a tableau method
enum { EP_R0, EP_R1, EP_R2, EP_DR, EP_ERRX, EP_ERRY, EP_QK0, EP_SK0 };  // per-CTA partials
struct RowParts { double d1[EPI_ROWS], d2[EPI_ROWS], hy[EPI_ROWS], gy[EPI_ROWS]; };

// Sum over the chunks of the gather's partial k of row i, in chunk order
__device__ __forceinline__ double part_sum(const DevCtx& c, int k, int i) {
    const double* p = c.part + (size_t)k * c.L + i;
    const size_t st = (size_t)6 * c.L;
    double a = p[0];
    for (int ch = 1; ch < c.nch; ch += 4) {
        double v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = ch + q < c.nch ? p[(ch + q) * st] : 0.0;
#pragma unroll
        for (int q = 0; q < 4; ++q) if (ch + q < c.nch) a += v[q];
    }
    return a;
}

// One component (0 QK, 1 QR) of a row through the stage: begin() takes what the stages before
// this one left, value() the new value (err: the step's error term, last stage), store() writes it.
struct Comp {
    double g, ge, gf, h0;
    __device__ __forceinline__ void begin(const DevCtx& c, const StageDev& sp, const int s, const int i, const int comp) {
        const size_t L2 = (size_t)2 * c.L, e = (size_t)2 * i + comp;
        const double* h = reinterpret_cast<const double*>(c.h) + e;
        g = ge = (reinterpret_cast<const double*>(c.KR) + e)[(size_t)(sp.n0 - 1) * L2];
        gf = 0.0;
        h0 = s > 0 ? h[0] : 0.0;
        if (sp.kind == KIND_TABLEAU) {
            const bool last = sp.last;
            double hv[TAB_STAGES], cf[TAB_STAGES], ce[TAB_STAGES];
#pragma unroll
            for (int j = 0; j < TAB_STAGES - 1; ++j) {
                hv[j] = j < s ? h[j * L2] : 0.0;
                cf[j] = j < s ? sp.coef[j] : 0.0;
                ce[j] = j < s && last ? sp.coef_e[j] : 0.0;
            }
#pragma unroll
            for (int j = 0; j < TAB_STAGES - 1; ++j) {
                if (j < s) g = fma(hv[j], cf[j], g);
                if (j < s && last) ge = fma(hv[j], ce[j], ge);
            }
        } else if (sp.serk_mode != 0) {
            g = (reinterpret_cast<const double*>(c.gS))[e];
            ge = (reinterpret_cast<const double*>(c.geS))[e];
            gf = (reinterpret_cast<const double*>(c.gfS))[e];
        }
    }
    __device__ __forceinline__ double value(const DevCtx& c, const StageDev& sp, const int s, const int i, const int comp,
                                            const double hs) {
        if (s == 0) h0 = hs;
        if (sp.kind == KIND_TABLEAU) {
            g = fma(hs, sp.coef[s], g);
            if (!sp.last) return 0.0;
            ge = fma(hs, sp.coef_e[s], ge);
            return fabs(g - ge);
        }
        if (sp.serk_mode == 0) {
            gf = ge * sp.serk_b0;
            g = fma(hs, sp.serk_c, g);
        } else if (sp.serk_mode == 1) {
            g = fma(hs, sp.serk_c, g);
        } else {
            g = fma(hs, sp.serk_c2, fma(2.0, g, -ge));
            ge = g;
        }
        if (sp.serk_bnext != 0.0) gf = fma(g, sp.serk_bnext, gf);
        const size_t e = (size_t)2 * i + comp;
        (reinterpret_cast<double*>(c.gS))[e] = g;
        (reinterpret_cast<double*>(c.geS))[e] = ge;
        (reinterpret_cast<double*>(c.gfS))[e] = gf;
        return sp.last ? fabs(gf - g) : 0.0;
    }
    template <bool MIXED>
    __device__ __forceinline__ void store(const DevCtx& c, const StageDev& sp, const int s, const int i, const int comp,
                                          const double hs) const {
        const size_t L2 = (size_t)2 * c.L, e = (size_t)2 * i + comp, o = (size_t)sp.n0 * L2 + e;
        const double dk = sp.tdiff * h0;
        (reinterpret_cast<double*>(c.h))[(size_t)s * L2 + e] = hs;
        (reinterpret_cast<double*>(c.KR))[o] = g;
        (reinterpret_cast<double*>(c.dKR))[o] = dk;
        if constexpr (MIXED) {
            if (c.KRq) {
                const float2 x = hi_lo(g);
                float* q = reinterpret_cast<float*>(c.KRq + (size_t)sp.n0 * c.L + i) + comp;
                q[0] = x.x;
                q[2] = x.y;
            } else {
                (reinterpret_cast<float*>(c.KRf))[o] = (float)g;
            }
            (reinterpret_cast<float*>(c.dKRf))[o] = (float)dk;
        }
    }
};

// Rows blk*EPI_ROWS .. +EPI_ROWS of stage s.  Leaves this CTA's partials of the scalars this
// stage needs in c.epart: r(t) terms, dr/dt (stage 0), error norm, C(t,0), f'(C(t,0)) (last
// stage).  fsal: stage 0 of an RK54 step whose right-hand side is the previous step's last one
// (StageDev::fsal); no gather ran for it.  Returns the inverse that the fold of this thread's
// warp writes: of tdiff (warp 2), of delta_t_ratio (warp 3; 0 where that is 0).
template <int P, int P2, bool MIXED>
__device__ __forceinline__ double rows(const DevCtx& c, const StageDev& sp, const int s, const unsigned blk, const bool fsal) {
    __shared__ RowParts sh;
    const int L = c.L, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, i = (int)blk * EPI_ROWS + lane;
    const bool mine = i < L, step = sp.kind != KIND_RHS;
    const DModel Mo = c.M;
    const double t = sp.T;
    double inv = 0.0, d = 0.0, th = 0.0, w = 0.0, err = 0.0;
    Comp k = {};
    // stage 0, warp 1: dr/dt terms of the step's base row (drstep2, time_steps.cu:564-639)
    double2 g0 = {};
    double sk0 = 0.0, dd0 = 0.0, sr0 = 0.0, d3g = 0.0, dr = 0.0;

    if (warp == 3) {
        if (step) {
            const double dtr_new = sp.dtr_new;
            const int nrows_next = sp.nrows_next, n0 = sp.n0;
            inv = dtr_new != 0.0 ? 1.0 / dtr_new : 0.0;
            if (mine) {
                const double pos = sp.pos_reuse >= 0 ? c.posB1x_saved[(size_t)sp.pos_reuse * L + i]
                                   : fsal            ? next_position(c, sp, c.b1[i].F, i)  // no gather ran
                                                     : c.posB1x_next[i];
                c.posB1x[i] = pos;
                if (sp.pos_save >= 0) c.posB1x_saved[(size_t)sp.pos_save * L + i] = pos;
                // delta_t_ratio of the row being written is not in memory yet
                c.b1[i] = b1_at(pos, nrows_next - 1 < 1 ? 1 : nrows_next - 1, nrows_next,
                                [&](int k) { return k != n0 ? c.inv_dtr[k] : inv; });
            }
        }
    } else if (mine) {
        th = c.theta[i];
        if (step && warp != 1) k.begin(c, sp, s, i, warp >> 1);
        if (step && warp != 2) w = c.integ[i];
        // right-hand side; fused as written: every kernel that instantiates this rounds alike
        if (fsal) {
            const double2 hs = c.h[(size_t)(RK54_STAGES - 1) * L + i];
            d = warp == 2 ? hs.y : hs.x;
        } else {
            const double2 q = c.KR[(size_t)(sp.nrows - 1) * L + i], rv = c.rowval[i];
            const double rE = c.rowval[L - 1].y, q0 = c.slots->q0;
            const double aA = part_sum(c, 2 * warp + 1, i), aR = part_sum(c, 2 * warp, i);
            const double tA = t * th, tR = t * (1.0 - th);
            if (warp == 0) {
                const double fac1 = Sig<P, P2>::d1(Mo, q0) * Mo.iT0;
                d = fma(aA, tA, fma(aR, tR, fma(q.x, -rE, __dmul_rn(rv.x, fac1))));
            } else if (warp == 1) {
                const double fac2 = q0 * Mo.iT0;
                d = fma(-q.x, rv.y, fma(aA, tA, fma(aR, tR,
                    fma(q.y, 2.0 * Mo.Gamma, __dmul_rn(Sig<P, P2>::d1(Mo, rv.x), fac2)))));
            } else {
                d = fma(fma(-aA, tR, __dmul_rn(q.y, rv.y)), th, fma(aR, tR, __dmul_rn(q.y, -rE)));
            }
        }
        if (warp == 0) sh.d1[lane] = d;
        if (warp == 1) {
            sh.d2[lane] = d;
            if (step && s == 0) {
                g0 = c.KR[(size_t)(sp.n0 - 1) * L + i];
                Sig<P, P2>::d12(Mo, g0.x, sk0, dd0);
                d3g = Sig<P, P2>::d3(Mo, g0.x) * g0.y;
                sr0 = dd0 * g0.y;
                dr = fma(w * sk0, g0.y, __dmul_rn(w * sr0, g0.x));
            }
        }
        if (warp == 2) {
            sh.hy[lane] = d;
            if (step) {
                err = k.value(c, sp, s, i, 1, d);
                sh.gy[lane] = k.g;
                inv = 1.0 / sp.tdiff;
            }
        }
    }
    __syncthreads();  // and every read of the newest row is done
    double* ep = c.epart + (size_t)blk * EP_N;
    if (warp == 0) {
        double r0 = 0.0, r1 = 0.0, r2 = 0.0, sk = 0.0;
        if (mine) {
            const double hs = fsal ? d : fma(sh.d2[lane], th, d);
            if (step) {
                err = k.value(c, sp, s, i, 0, hs);
                k.store<MIXED>(c, sp, s, i, 0, hs);
                // rstep (time_steps.cpp:83-92) of the new row at its time
                const double tw = sp.T_next * w, gy = sh.gy[lane];
                double dd;
                Sig<P, P2>::d12(Mo, k.g, sk, dd);
                r0 = __dmul_rn(tw * (dd * gy), k.g);
                r1 = __dmul_rn(tw * sk, gy);
                if (i == 0) r2 = __dmul_rn(sk * k.g, Mo.iT0);
            } else {
                c.h[(size_t)s * L + i].x = hs;
                c.rhs_out[i].x = hs;
            }
        }
        if (step) {
            // both sums in five adds a lane: the lower half-warp carries r0, the upper r1
            const double mv = lane < 16 ? r0 : r1, ot = lane < 16 ? r1 : r0;
            double v = mv + __shfl_xor_sync(0xffffffffu, ot, 16);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (sp.last) err = warp_sum(err);
            if (lane == 0) {
                ep[EP_R0] = v;
                ep[EP_R2] = r2;
                if (sp.last) {
                    ep[EP_ERRX] = err;
                    ep[EP_QK0] = blk == 0 ? k.g : 0.0;
                    ep[EP_SK0] = blk == 0 ? sk : 0.0;
                }
            }
            if (lane == 16) ep[EP_R1] = v;
        }
    } else if (warp == 1) {
        if (step && s == 0) {
            if (mine) {
                const double hx = fsal ? d : fma(d, th, sh.d1[lane]), hy = sh.hy[lane];
                const double dsk = dd0 * hx, dsr = fma(dd0, hy, __dmul_rn(d3g, hx)), tw = t * w;
                dr = fma(tw * dsr, g0.x, dr);
                dr = fma(tw * dsk, g0.y, dr);
                dr = fma(tw * sr0, hx, dr);
                dr = fma(tw * sk0, hy, dr);
                if (i == 0) dr = fma(fma(sk0, hx, __dmul_rn(dsk, g0.x)), Mo.iT0, dr);
            }
            dr = warp_sum(dr);
            if (lane == 0) ep[EP_DR] = dr;
        }
    } else if (warp == 2) {
        if (mine) {
            if (step) {
                k.store<MIXED>(c, sp, s, i, 1, d);
            } else {
                c.h[(size_t)s * L + i].y = d;
                c.rhs_out[i].y = d;
            }
        }
        if (step && sp.last) {
            err = warp_sum(err);
            if (lane == 0) ep[EP_ERRY] = err;
        }
    }
    return inv;
}

// Elect the CTA of G that finishes last (atomic ticket on slots->counter, no waiting);
// true in every thread of that CTA only.
__device__ __forceinline__ bool elect_last(const DevCtx& c, const unsigned G) {
    __shared__ unsigned s_ticket;
    // releases this CTA's rows and partials, acquires the others': the barriers carry the
    // order to and from the ticket's thread
    __syncthreads();
    if (threadIdx.x == 0)
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(s_ticket) : "l"(&c.slots->counter) : "memory");
    __syncthreads();
    return s_ticket == G - 1;
}

// Fold of the G CTAs' partials (in a fixed order) and the stage's scalar writes: r of the
// written row, dr/dt, t1grid, delta_t_ratio and, at the last stage, the step result.  Ends
// with a barrier; does not reset slots->counter.
template <bool MIXED>
__device__ __forceinline__ void fold(const DevCtx& c, const StageDev& sp, const int s, const unsigned G, const double inv) {
    static_assert(EP_N == 8 && EPI_T == 128);
    __shared__ double s_tot[EPI_T / 32][EP_N];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    Slots* sl = c.slots;
    if (sp.kind != KIND_RHS) {
        const double dr_old = s == 0 ? 0.0 : sl->dr;
        double v = 0.0;
        for (unsigned b = tid / EP_N; b < G; b += EPI_T / EP_N) v += __ldcg(c.epart + (size_t)b * EP_N + tid % EP_N);
        v += __shfl_xor_sync(0xffffffffu, v, 8);
        v += __shfl_xor_sync(0xffffffffu, v, 16);
        if (lane < EP_N) s_tot[warp][lane] = v;
        __syncthreads();
        const auto tot = [&](int q) { return (s_tot[0][q] + s_tot[1][q]) + (s_tot[2][q] + s_tot[3][q]); };
        const int n0 = sp.n0;
        if (tid == 0) {
            const double r1 = tot(EP_R1), r_new = ((c.M.Gamma + tot(EP_R0)) + r1) + tot(EP_R2);
            c.rvec[n0] = r_new;
            if (sp.last) {
                sl->res_energy = -(r1 + __dmul_rn(tot(EP_SK0), c.M.iT0));
                sl->res_r = r_new;
            }
        } else if (tid == 32) {
            const double dr = s == 0 ? tot(EP_DR) : dr_old;
            if (s == 0) sl->dr = dr;
            c.drvec[n0] = sp.tdiff * dr;
            if (sp.last) sl->res_dr = dr;
        } else if (tid == 64) {
            if (c.inv_len) c.inv_len[n0 - 1] = inv;
            if constexpr (MIXED) c.inv_len_f[n0 - 1] = hi_lo(inv);
            if (sp.last) {
                sl->res_err = tot(EP_ERRX) + tot(EP_ERRY);
                sl->res_qk0 = tot(EP_QK0);
            }
        } else if (tid == 96) {
            c.t1grid[n0] = sp.T_next;
            c.dtr[n0] = sp.dtr_new;
            c.inv_dtr[n0] = inv;
            if constexpr (MIXED) c.inv_dtr_f[n0] = hi_lo(inv);
        }
    }
    __syncthreads();
}

}  // namespace epi
}  // namespace dyn
