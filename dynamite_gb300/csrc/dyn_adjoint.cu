// Discrete adjoint of the FP64 RK-stepped hot path (fixed step schedule).
//
// The two-time history is append-only: a step reads rows 0..n0-1 and writes
// row n0, so the state before any step is a prefix of the final history.
// The reverse sweep therefore needs no stored checkpoints besides the final
// history itself: for step k (last to first) the host recomputes that one
// step's stages from the prefix with the forward kernels (snapshotting the
// row-n0 state and the B1 positions each stage reads), then runs the stages
// backwards:
//
//   k_adj_enter      takes row n0's cotangents over and puts the row back into
//                    stage s's input state;
//   k_adj_rows       row n0 after stage s: r = rstep(G_s) (time_steps.cpp:83-92),
//                    dQK/dQR = tdiff_s h_0, dr = tdiff_s DR and the RK
//                    combination G_s = g0 + sum_j coef_j h_j, transposed; at
//                    stage 0 DR = drstep2(g0, h_0) (time_steps.cpp:117-125);
//                    then the RHS epilogue (QKstep/QRstep, time_steps.cpp:27-47,
//                    94-100) transposed: row cotangents of the eight memory
//                    integrals, the direct last-row terms, QK^{B1}[i,0] and
//                    rInt (index_vec.cpp:63-156) scattered to the history;
//   k_adj_targets    per target (i,j): the A1/A2/B1/B2 values that the recompute
//                    recorded, Sigma and the int.dat products differentiated, B1
//                    transposed (scatter-adds into the cotangent history), the
//                    A1/A2 cotangents stored and B2's as a packet;
//   k_adj_lastrow    the A1/A2 stencils transposed onto the last row, a partial
//                    row per target row, summed by k_adj_lastreduce;
//   k_adj_b2ser      the B2 stencils transposed, from the packets in the order of
//                    their stencil starts (k_adj_b2gen at other depths than 10).
//
// Parameter derivatives (Gamma, lambda) accumulate in device scalars.
#include <algorithm>
#include <cmath>
#include "dyn_epi.cuh"

namespace dyn {

namespace {

enum { SC_RHO = 0, SC_DELTA = 1, SC_DR = 2, SC_GAMMA = 3, SC_LAMBDA = 4 };

__device__ __forceinline__ double qpow(double q, int e) { return e < 0 ? 0.0 : ipow_r(q, e); }
__device__ __forceinline__ double falpha(int p, int k) {
    double a = 1.0;
    for (int j = 0; j < k; ++j) a *= (double)(p - j);
    return a;
}
// k-th derivative of f(q) = lam q^p + (1-lam) q^p2 and its derivative in lam
__device__ __forceinline__ void fder(const AdjModel& m, int k, double q, double& v, double& vl) {
    const double tp = falpha(m.p, k) * qpow(q, m.p - k), tp2 = falpha(m.p2, k) * qpow(q, m.p2 - k);
    v = m.lam * tp + (1.0 - m.lam) * tp2;
    vl = tp - tp2;
}

// The same with the exponents known at compile time (P < 0: runtime exponents)
template <int P, int K>
__host__ __device__ constexpr double alpha_c() {
    double a = 1.0;
    for (int j = 0; j < K; ++j) a *= (double)(P - j);
    return a;
}
template <int P, int P2, int K>
__device__ __forceinline__ void fder_t(const AdjModel& m, double q, double& v, double& vl);
template <int P, int P2, int K>
__device__ __forceinline__ double fd_t(const AdjModel& m, double q) {
    double v, vl;
    fder_t<P, P2, K>(m, q, v, vl);
    return v;
}
template <int P, int P2, int K>
__device__ __forceinline__ void fder_t(const AdjModel& m, double q, double& v, double& vl) {
    if constexpr (P < 0) {
        fder(m, K, q, v, vl);
    } else {
        constexpr double ap = alpha_c<P, K>(), ap2 = alpha_c<P2, K>();
        const double tp = (P - K >= 0 && ap != 0.0) ? ipow_c<(P - K >= 0 ? P - K : 0)>(q) : 0.0;
        const double tp2 = (P2 - K >= 0 && ap2 != 0.0) ? ipow_c<(P2 - K >= 0 ? P2 - K : 0)>(q) : 0.0;
        v = fma(m.cb[K], tp2, m.ca[K] * tp);
        vl = fma(ap, tp, -(ap2 * tp2));
    }
}

// block-wide sum (blockDim.x a multiple of 32, <= 1024); every thread gets it
__device__ double block_sum(double v) {
    __shared__ double s_w[32];
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    __syncthreads();
    if (lane == 0) s_w[w] = v;
    __syncthreads();
    double t = 0.0;
    for (int k = 0; k < nw; ++k) t += s_w[k];
    return t;
}

__device__ __forceinline__ void add2(double2* p, double x, double y) {
    atomicAdd(&p->x, x);
    atomicAdd(&p->y, y);
}

// ---------------------------------------------------------------- seeds
// J = wE * E(t_f) + sum_j cK[j] C(t_f, theta_j t_f) + wR * r(t_f) on row nl
template <int P, int P2>
__global__ void __launch_bounds__(256) k_adj_seed(const DevCtx c, const AdjDev a, const AdjModel am, const int nl, const double wE,
                           const double wR, const double wDr, const double* cK, const double* cR, const double* cdK,
                           const double* cdR) {
    const int L = c.L;
    const double tf = c.t1grid[nl];
    double lam = 0.0;
    for (int j = threadIdx.x; j < L; j += blockDim.x) {
        const double2 g = c.KR[(size_t)nl * L + j];
        const double w = c.integ[j];
        double f1, f1l, f2, f2l;
        fder_t<P, P2, 1>(am, g.x, f1, f1l);
        fder_t<P, P2, 2>(am, g.x, f2, f2l);
        // E = -(t sum_j w_j f'(K_j) R_j + f'(K_0)/T0)
        double kb = -(tf * w * f2 * g.y) - (j == 0 ? f2 / am.T0 : 0.0);
        const double rb = -(tf * w * f1);
        lam += -(tf * w * f1l * g.y) - (j == 0 ? f1l / am.T0 : 0.0);
        kb *= wE;
        if (cK) kb += cK[j];
        double2* h = a.HKR + (size_t)nl * L + j;
        h->x += kb;
        h->y += wE * rb + (cR ? cR[j] : 0.0);
        double2* hd = a.HdKR + (size_t)nl * L + j;
        hd->x += cdK ? cdK[j] : 0.0;
        hd->y += cdR ? cdR[j] : 0.0;
    }
    lam = block_sum(lam);
    if (threadIdx.x == 0) {
        a.sc[SC_LAMBDA] += wE * lam;
        a.Hr[nl] += wR;
        a.Hdr[nl] += wDr;
    }
}

// row n0 as stage k left it, and the B1 rows the next stage reads
__global__ void k_adj_save(const DevCtx c, const AdjDev a, const int k, const int n0) {
    wait_prior_grid();
    const int L = c.L, j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < L) {
        a.Gsave[(size_t)k * L + j] = c.KR[(size_t)n0 * L + j];
        a.Dsave[(size_t)k * L + j] = c.dKR[(size_t)n0 * L + j];
        if (k + 1 < SMAX) a.Bsave[(size_t)(k + 1) * L + j] = c.b1[j];
    }
    if (j < 5) a.tsave[5 * k + j] = (j == 0 ? c.rvec : j == 1 ? c.drvec : j == 2 ? c.t1grid : j == 3 ? c.dtr : c.inv_dtr)[n0];
}

// Before the reverse of stage s: the cotangents of row n0 (the state after stage s) into the
// stage buffers, and row n0 back into stage s's input state (the state after stage s-1)
__global__ void k_adj_enter(const DevCtx c, const AdjDev a, const int s, const int n0) {
    wait_prior_grid();
    const int L = c.L, j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < L) {
        const size_t o = (size_t)n0 * L + j;
        a.Gbar[j] = a.HKR[o];
        a.Dbar[j] = a.HdKR[o];
        a.HKR[o] = make_double2(0.0, 0.0);
        a.HdKR[o] = make_double2(0.0, 0.0);
        if (s >= 1) {
            c.KR[o] = a.Gsave[(size_t)(s - 1) * L + j];
            c.dKR[o] = a.Dsave[(size_t)(s - 1) * L + j];
        }
    }
    if (j == 0) {
        a.sc[SC_RHO] = a.Hr[n0];
        a.sc[SC_DELTA] = a.Hdr[n0];
        a.Hr[n0] = 0.0;
        a.Hdr[n0] = 0.0;
    }
    if (s >= 1 && j < 5)
        (j == 0 ? c.rvec : j == 1 ? c.drvec : j == 2 ? c.t1grid : j == 3 ? c.dtr : c.inv_dtr)[n0] = a.tsave[5 * (s - 1) + j];
}

// What column j's thread accumulates of the row's scalars
struct RowBars { double2 g0b, h0b; double lam; };

// ------------------------------------------------- row write of stage s
template <int P, int P2>
__device__ __forceinline__ RowBars row_write(const DevCtx& c, const AdjDev& a, const AdjModel& am, const StageDev& sp,
                                             const int s, const int j) {
    const int L = c.L;
    const double tn = sp.T_next, rb = a.sc[SC_RHO];
    const double2 G = a.Gsave[(size_t)s * L + j];
    const double w = tn * c.integ[j];
    double f1, f1l, f2, f2l;
    fder_t<P, P2, 1>(am, G.x, f1, f1l);
    fder_t<P, P2, 2>(am, G.x, f2, f2l);
    const double f3 = fd_t<P, P2, 3>(am, G.x);
    // r = Gamma + sum_j tn w (f''(K) R K + f'(K) R) + f'(K_0) K_0 / T0
    double dK = w * (f3 * G.y * G.x + 2.0 * f2 * G.y);
    const double dR = w * (f2 * G.x + f1);
    RowBars r;
    r.lam = w * (f2l * G.y * G.x + f1l * G.y);
    if (j == 0) {
        dK += (f2 * G.x + f1) / am.T0;
        r.lam += f1l * G.x / am.T0;
    }
    r.lam *= rb;
    const double2 gb0 = a.Gbar[j];
    const double2 Gb = make_double2(gb0.x + rb * dK, gb0.y + rb * dR);
    // G_s = g0 + sum_{j<=s} coef_j h_j
    r.g0b = a.g0bar[j];
    r.g0b.x += Gb.x;
    r.g0b.y += Gb.y;
    for (int q = 1; q < sp.ncoef; ++q) {
        double2 hb = a.hbar[(size_t)q * L + j];
        hb.x += sp.coef[q] * Gb.x;
        hb.y += sp.coef[q] * Gb.y;
        a.hbar[(size_t)q * L + j] = hb;
    }
    // dQK, dQR of row n0 = tdiff_s h_0
    const double2 Db = a.Dbar[j];
    r.h0b = a.hbar[j];
    r.h0b.x += sp.coef[0] * Gb.x + sp.tdiff * Db.x;
    r.h0b.y += sp.coef[0] * Gb.y + sp.tdiff * Db.y;
    return r;
}

// DR = drstep2(g0, h_0) at the step start (stage 0 time)
template <int P, int P2>
__device__ __forceinline__ void row_drstep(const DevCtx& c, const AdjModel& am, const int n0, const int j, const double T,
                                           const double DRb, RowBars& r) {
    const double2 g = c.KR[(size_t)(n0 - 1) * c.L + j];
    const double2 h = c.h[j];
    const double w = c.integ[j], tw = T * w;
    const double K = g.x, R = g.y, hK = h.x, hR = h.y;
    double f1, f1l, f2, f2l, f3, f3l;
    fder_t<P, P2, 1>(am, K, f1, f1l);
    fder_t<P, P2, 2>(am, K, f2, f2l);
    fder_t<P, P2, 3>(am, K, f3, f3l);
    const double f4 = fd_t<P, P2, 4>(am, K);
    double dK = w * (f3 * R * K + 2.0 * f2 * R) + tw * (f4 * R * hK * K + 3.0 * f3 * R * hK + f3 * hR * K + 2.0 * f2 * hR);
    const double dR = w * (f2 * K + f1) + tw * (f3 * hK * K + 2.0 * f2 * hK);
    double dhK = tw * (f3 * R * K + 2.0 * f2 * R);
    const double dhR = tw * (f2 * K + f1);
    double dl = w * (f2l * R * K + f1l * R) + tw * (f3l * R * hK * K + f2l * hR * K + 2.0 * f2l * hK * R + f1l * hR);
    if (j == 0) {
        dK += (f3 * K + 2.0 * f2) * hK / am.T0;
        dhK += (f2 * K + f1) / am.T0;
        dl += (f2l * K + f1l) * hK / am.T0;
    }
    r.g0b.x += DRb * dK;
    r.g0b.y += DRb * dR;
    r.h0b.x += DRb * dhK;
    r.h0b.y += DRb * dhR;
    r.lam += DRb * dl;
}

__device__ __forceinline__ double rint_of(const DevCtx& c, const B1Row& w) {
    double ri = w.c0 * c.rvec[w.F - 1] + w.c1 * c.rvec[w.F] - w.c2 * c.drvec[w.F];
    if (w.cubic) ri -= w.c3 * c.drvec[w.F + 1];
    return ri;
}
__device__ __forceinline__ void scatter_rint(const DevCtx& c, const AdjDev& a, const B1Row& w, double rb) {
    atomicAdd(a.Hr + w.F - 1, w.c0 * rb);
    atomicAdd(a.Hr + w.F, w.c1 * rb);
    atomicAdd(a.Hdr + w.F, -w.c2 * rb);
    if (w.cubic) atomicAdd(a.Hdr + w.F + 1, -w.c3 * rb);
}

// Row write, dr/dt (stage 0) and RHS epilogue of stage s, transposed: one column per thread,
// one-warp CTAs.  Bound by a warp's FP64 rate (one instruction in 64 cycles), so the columns
// spread over as many SMs as they fill; the sums over columns enter the history linearly, so
// each CTA adds its own share.  L = 512: 41 us as two kernels of one CTA, now 16.5.
constexpr int ADJ_ROW_T = 32;
template <int P, int P2>
__global__ void __launch_bounds__(ADJ_ROW_T) k_adj_rows(const DevCtx c, const AdjDev a, const AdjModel am, const int s, const int n0) {
    wait_prior_grid();
    const StageDev& sp = c.stages[s];
    const int L = c.L, nrows = sp.nrows, lr = nrows - 1, i = blockIdx.x * ADJ_ROW_T + threadIdx.x;
    const double t = sp.T, td = sp.tdiff;
    const bool live = t > 0.0, first = blockIdx.x == 0 && threadIdx.x == 0;
    const double q0 = c.KR[(size_t)lr * L].x;
    double rE;
    B1Row wE{};
    if (live) {
        wE = a.Bsave[(size_t)s * L + L - 1];
        rE = rint_of(c, wE);
    } else {
        rE = c.rvec[0];
    }
    double f1q0, f1lq0;
    fder_t<P, P2, 1>(am, q0, f1q0, f1lq0);
    const double fac1 = f1q0 / am.T0, fac2 = q0 / am.T0;
    double sE = 0.0, sF1 = 0.0, sF2 = 0.0, lam = 0.0, gam = 0.0;
    if (i < L) {
        RowBars rw = row_write<P, P2>(c, a, am, sp, s, i);
        // dr of row n0 = tdiff_s DR, summed over the stages
        if (s == 0) row_drstep<P, P2>(c, am, n0, i, t, a.sc[SC_DR] + td * a.sc[SC_DELTA], rw);
        a.g0bar[i] = rw.g0b;
        a.hbar[i] = rw.h0b;
        lam = rw.lam;
        const double2 hb = s == 0 ? rw.h0b : a.hbar[(size_t)s * L + i];

        const double2 q = c.KR[(size_t)lr * L + i];
        double qb, ri;
        B1Row w{};
        if (live) {
            w = a.Bsave[(size_t)s * L + i];
            qb = w.c0 * c.KR[(size_t)(w.F - 1) * L].x + w.c1 * c.KR[(size_t)w.F * L].x - w.c2 * c.dKR[(size_t)w.F * L].x;
            if (w.cubic) qb -= w.c3 * c.dKR[(size_t)(w.F + 1) * L].x;
            ri = rint_of(c, w);
        } else {
            qb = c.KR[0].x;
            ri = c.rvec[0];
        }
        const double th = c.theta[i], tA = t * th, tR = t * (1.0 - th);
        // hK = d1 + d2 th;  hR = (R (-rE) + a6 tR) + (R ri - a7 tR) th
        const double d1b = hb.x, d2b = th * hb.x;
        double* ab = a.abar + (size_t)i * 8;
        ab[0] = tR * d1b;
        ab[1] = tA * d1b;
        ab[2] = tA * d1b;
        ab[3] = tR * d2b;
        ab[4] = tA * d2b;
        ab[5] = tA * d2b;
        ab[6] = tR * hb.y;
        ab[7] = -tR * th * hb.y;
        // d1 = qb fac1 - K rE + ...;  d2 = f'(qb) fac2 + 2 Gamma R + ... - K ri
        const double Kb = -rE * d1b - ri * d2b;
        const double Rb = hb.y * (-rE + ri * th) + 2.0 * am.Gamma * d2b;
        add2(a.HKR + (size_t)lr * L + i, Kb, Rb);
        sE = -q.y * hb.y - q.x * d1b;
        const double rib = q.y * th * hb.y - q.x * d2b;
        double f1qb, f1lqb;
        fder_t<P, P2, 1>(am, qb, f1qb, f1lqb);
        const double qbb = fac1 * d1b + fd_t<P, P2, 2>(am, qb) * fac2 * d2b;
        sF1 = qb * d1b;
        sF2 = f1qb * d2b;
        lam += f1lqb * fac2 * d2b;
        gam = 2.0 * q.y * d2b;
        if (live) {
            atomicAdd(&a.HKR[(size_t)(w.F - 1) * L].x, w.c0 * qbb);
            atomicAdd(&a.HKR[(size_t)w.F * L].x, w.c1 * qbb);
            atomicAdd(&a.HdKR[(size_t)w.F * L].x, -w.c2 * qbb);
            if (w.cubic) atomicAdd(&a.HdKR[(size_t)(w.F + 1) * L].x, -w.c3 * qbb);
            scatter_rint(c, a, w, rib);
        } else {
            atomicAdd(&a.HKR[0].x, qbb);
            atomicAdd(a.Hr, rib);
        }
    }
    sE = warp_sum(sE);
    sF1 = warp_sum(sF1);
    sF2 = warp_sum(sF2);
    lam = warp_sum(lam);
    gam = warp_sum(gam);
    if (threadIdx.x == 0) {
        // rE = rInt of row L-1; q0 = QK of the last row at theta = 0
        if (live) scatter_rint(c, a, wE, sE);
        else atomicAdd(a.Hr, sE);
        const double q0b = sF1 * fd_t<P, P2, 2>(am, q0) / am.T0 + sF2 / am.T0;
        atomicAdd(&a.HKR[(size_t)lr * L].x, q0b);
        atomicAdd(a.sc + SC_LAMBDA, lam + sF1 * f1lq0 / am.T0);
        if (first) {
            gam += a.sc[SC_RHO];
            if (s > 0) a.sc[SC_DR] += td * a.sc[SC_DELTA];
        }
        atomicAdd(a.sc + SC_GAMMA, gam);
    }
}

// ------------------------------------------------------- per-target part
// One thread per target (i, j), 64-thread CTAs over (chunk, row): the
// gathered values recorded by the recompute, Sigma and the int.dat products
// differentiated, the B1 gathers transposed into the cotangent history
// (reductions), the A1/A2 cotangents of the target stored for k_adj_lastrow
// and its B2 packet for k_adj_b2ser.  Bound by the FP64 pipe (82 % busy): 150 instructions a
// target with whole derivatives and weights formed per product, 105 now (L = 512: 75 -> 57 us).
template <int P, int P2>
__global__ void __launch_bounds__(64) k_adj_targets(const DevCtx c, const AdjDev a, const AdjModel am, const int s) {
    wait_prior_grid();
    const StageDev& sp = c.stages[s];
    const int L = c.L, i = blockIdx.y, j = blockIdx.x * blockDim.x + threadIdx.x;
    const double t = sp.T;
    if (!(t > 0.0)) return;  // t = 0: the memory integrals carry a factor t, all cotangents vanish
    double lam = 0.0;
    if (j < L) {
        // row cotangents times the target's weight; rows 1, 2 and 4, 5 have the same
        const double W = c.integ[j];
        const double* ar = a.abar + (size_t)i * 8;
        const double w0 = W * ar[0], w1 = W * ar[1], w3 = W * ar[3], w4 = W * ar[4], w6 = W * ar[6], w7 = W * ar[7];
        const B1Row br = a.Bsave[(size_t)s * L + i];
        const double bc0 = br.c0, bc1 = br.c1, bc2 = br.c2, bc3 = br.c3;
        const int F = br.F, cubic1 = br.cubic;
        const size_t ij = (size_t)i * L + j;
        // ---- forward values, recorded by k_main in the recompute of this stage
        const GatherRec g = a.rec[(size_t)s * L * L + ij];
        const double2 a1 = g.a1, a2 = g.a2, b1 = g.b1, b2 = g.b2;
        const int X = g.X;
        const double x = g.x;
        // ---- Sigma and its derivatives
        double fA1[4], lA1[3], fA2[4], lA2[3], fB1[4], lB1[3], fB2[4], lB2[3];
        fder_t<P, P2, 1>(am, a1.x, fA1[1], lA1[0]);
        fder_t<P, P2, 2>(am, a1.x, fA1[2], lA1[1]);
        fder_t<P, P2, 3>(am, a1.x, fA1[3], lA1[2]);
        fder_t<P, P2, 1>(am, a2.x, fA2[1], lA2[0]);
        fder_t<P, P2, 2>(am, a2.x, fA2[2], lA2[1]);
        fder_t<P, P2, 3>(am, a2.x, fA2[3], lA2[2]);
        fder_t<P, P2, 1>(am, b1.x, fB1[1], lB1[0]);
        fder_t<P, P2, 2>(am, b1.x, fB1[2], lB1[1]);
        fder_t<P, P2, 3>(am, b1.x, fB1[3], lB1[2]);
        fder_t<P, P2, 1>(am, b2.x, fB2[1], lB2[0]);
        fder_t<P, P2, 2>(am, b2.x, fB2[2], lB2[1]);
        fder_t<P, P2, 3>(am, b2.x, fB2[3], lB2[2]);
        const double sKA1 = fA1[1], sRA1 = fA1[2] * a1.y, sRA2 = fA2[2] * a2.y;
        const double sKB1 = fB1[1], sRB1 = fB1[2] * b1.y, sKB2 = fB2[1], sRB2 = fB2[2] * b2.y;
        // ---- cotangents of the eight products P_k (row sums a_k)
        const double sRA2b = b2.x * w0 + b2.y * w6;
        double b2Kb = sRA2 * w0, b2Rb = sRA2 * w6;
        const double sRA1b = b1.x * w1;
        double b1Kb = sRA1 * w1;
        const double sKA1b = b1.y * w1;
        double b1Rb = sKA1 * w1;
        double a2Rb = sKB2 * w3 + sRB2 * w7;
        const double sKB2b = a2.y * w3, sRB2b = a2.y * w7;
        double a1Rb = sKB1 * w4;
        const double sKB1b = a1.y * w4;
        double a1Kb = sRB1 * w4;
        const double sRB1b = a1.x * w4;
        // ---- Sigma transposed: sK = f'(K), sR = f''(K) R
        a1Kb += fA1[2] * sKA1b + fA1[3] * a1.y * sRA1b;
        a1Rb += fA1[2] * sRA1b;
        const double a2Kb = fA2[3] * a2.y * sRA2b;
        a2Rb += fA2[2] * sRA2b;
        b1Kb += fB1[2] * sKB1b + fB1[3] * b1.y * sRB1b;
        b1Rb += fB1[2] * sRB1b;
        b2Kb += fB2[2] * sKB2b + fB2[3] * b2.y * sRB2b;
        b2Rb += fB2[2] * sRB2b;
        lam = lA1[0] * sKA1b + lA1[1] * a1.y * sRA1b + lA2[1] * a2.y * sRA2b + lB1[0] * sKB1b + lB1[1] * b1.y * sRB1b +
              lB2[0] * sKB2b + lB2[1] * b2.y * sRB2b;
        // ---- gathers transposed: A1/A2 through k_adj_lastrow, B1/B2 here
        a.abarA[2 * ij] = make_double2(a1Kb, a1Rb);
        a.abarA[2 * ij + 1] = make_double2(a2Kb, a2Rb);
        add2(a.HKR + (size_t)(F - 1) * L + j, bc0 * b1Kb, bc0 * b1Rb);
        add2(a.HKR + (size_t)F * L + j, bc1 * b1Kb, bc1 * b1Rb);
        add2(a.HdKR + (size_t)F * L + j, -bc2 * b1Kb, -bc2 * b1Rb);
        if (cubic1) add2(a.HdKR + (size_t)(F + 1) * L + j, -bc3 * b1Kb, -bc3 * b1Rb);
        // B2 transposed by k_adj_b2ser from the packet in static order
        a.b2pk[__ldg(a.b2rank + ij)] = AdjDev::B2Packet{(int)ij, X, x, b2Kb, b2Rb};
    }
    lam = warp_sum(lam);
    if ((threadIdx.x & 31) == 0 && lam != 0.0) atomicAdd(a.sc + SC_LAMBDA, lam);
}

// A1/A2 gathers of target row i transposed onto the last row: a sparse
// matrix-vector product with the row's static column-sorted matrix (lrW,
// lrS, lrC; 2 L m entries).  Every thread takes an equal run of entries and
// accumulates column by column in registers, adding a column's partial sum to
// shared memory when it leaves the column: two FMAs per entry whatever the
// stencil starts look like (runs of equal starts near theta = 0 or 1 only
// make long columns, split over several threads).  The row goes to
// lbar_part[i] for k_adj_lastreduce.  The entries lie as the threads take them, entry q of
// every thread side by side: read run by run they cost an L1 line per lane (L = 512: 55 us, now
// 43; the FP64 pipe is 72 % busy).
__global__ void __launch_bounds__(LR_T) k_adj_lastrow(const DevCtx c, const AdjDev a, const int s) {
    wait_prior_grid();
    const StageDev& sp = c.stages[s];
    if (!(sp.T > 0.0)) return;
    const int L = c.L, i = blockIdx.x, E = 2 * L * c.m;
    extern __shared__ double2 s_acc[];  // [L] row sums, [2L] the row's A1/A2 cotangents (2j+t), int [L+1] column starts
    double2* s_cb = s_acc + L;
    int* s_cs = (int*)(s_acc + 3 * L);
    const size_t row = (size_t)i * L;
    const int* cs = a.lrC + (size_t)i * (L + 1);
    for (int k = threadIdx.x; k < L; k += blockDim.x) s_acc[k] = make_double2(0.0, 0.0);
    for (int k = threadIdx.x; k < 2 * L; k += blockDim.x) s_cb[k] = a.abarA[2 * row + k];
    for (int k = threadIdx.x; k <= L; k += blockDim.x) s_cs[k] = __ldg(cs + k);
    __syncthreads();
    const int per = (E + LR_T - 1) / LR_T;
    const int p0 = threadIdx.x * per, p1 = min(p0 + per, E);
    if (p0 < p1) {
        const double* w = a.lrW + (size_t)i * per * LR_T + threadIdx.x;
        const unsigned short* src = a.lrS + (size_t)i * per * LR_T + threadIdx.x;
        int lo = 0, hi = L;  // column of entry p0: the last k with cs[k] <= p0
        while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (s_cs[mid] <= p0) lo = mid; else hi = mid; }
        int k = lo, kend = s_cs[k + 1];
        double ax = 0.0, ay = 0.0;
        constexpr int B = 8;  // entries loaded ahead
        for (int pb = p0, k0 = 0; pb < p1; pb += B, k0 += B) {
            double u[B];
            int si[B];
#pragma unroll
            for (int q = 0; q < B; ++q) {
                const bool in = pb + q < p1;
                u[q] = in ? __ldg(w + (size_t)(k0 + q) * LR_T) : 0.0;
                si[q] = in ? __ldg(src + (size_t)(k0 + q) * LR_T) : 0;
            }
#pragma unroll
            for (int q = 0; q < B; ++q) {
                const int p = pb + q;
                if (p >= p1) break;
                if (p >= kend) {
                    atomicAdd(&s_acc[k].x, ax);
                    atomicAdd(&s_acc[k].y, ay);
                    ax = ay = 0.0;
                    do { ++k; kend = s_cs[k + 1]; } while (p >= kend);
                }
                const double2 v = s_cb[si[q]];
                ax = fma(u[q], v.x, ax);
                ay = fma(u[q], v.y, ay);
            }
        }
        atomicAdd(&s_acc[k].x, ax);
        atomicAdd(&s_acc[k].y, ay);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < L; k += blockDim.x) a.lbar_part[row + k] = s_acc[k];
}

// B2 gathers transposed from the packets in static (iB2, phi2) order.  Each
// thread runs over `run` consecutive packets; packets with the same key
// (X, iB2) add into the same 8 m history entries (K rows X-1, X; dK rows X,
// X+1; two components), so the thread accumulates them in registers (8 m
// FMAs per packet) and adds the sums to the history when the key changes or
// the run ends.  A warp whose 32 runs all carry one key (phi2 near 0 or 1)
// sums the runs across the warp first.  No key order is assumed: a key that
// recurs non-contiguously only means more additions.  Bound by the FP64 pipe (98 instructions a
// packet), of which every SM scheduler has its own: the run is what gives each of them two
// warps (L = 512: 7; runs of 8 leave a sixth of the pipes idle at the end), and at least
// B2_RUN_MIN, for fewer additions.
constexpr int B2_RUN_MIN = 2, B2_WARPS_SM = 8;
// inv: 1 / delta_t_ratio of row X + 1 (unused where X is the last but one)
__device__ __forceinline__ void b2_coeffs(double inv, int X, double x, int nrows, double e[4]) {
    const double x2 = x * x, x3 = x2 * x;
    if (X < nrows - 1) {
        e[0] = 1.0 - 3.0 * x2 + 2.0 * x3;   // K row X-1
        e[1] = 3.0 * x2 - 2.0 * x3;         // K row X
        e[2] = x - 2.0 * x2 + x3;           // dK row X
        e[3] = (x3 - x2) * inv;           // dK row X+1
    } else {
        e[0] = 1.0 - x2;
        e[1] = x2;
        e[2] = x - x2;
        e[3] = 0.0;
    }
}
// Add the sums of the lanes in `mask` to the history, a lane's 8 M values at a time by the
// whole warp: its four rows' 2 M consecutive doubles then go out as a few sectors each.  (As
// 8 M additions of one lane each, all to different lines, they were 9 M requests a stage at
// L = 512: 84 us, now 68.)
template <int M>
__device__ __forceinline__ void b2_flush(const DevCtx& c, const AdjDev& a, unsigned mask, int X, int iB2, int nrows,
                                         const double acc[M][8], double* s_acc) {
    constexpr int N = 8 * M, STRIDE = N + 2;  // + 2: the lanes' 16-byte stores hit different banks
    const int lane = threadIdx.x & 31, L2 = 2 * c.L;
    if ((mask >> lane) & 1u) {
        double2* o = reinterpret_cast<double2*>(s_acc + lane * STRIDE);
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int d = 0; d < M; ++d) o[k * M + d] = make_double2(acc[d][2 * k], acc[d][2 * k + 1]);
    }
    __syncwarp();
    while (mask) {
        const int f = __ffs(mask) - 1;
        mask &= mask - 1;
        const int fX = __shfl_sync(0xffffffffu, X, f), fB = __shfl_sync(0xffffffffu, iB2, f);
        const size_t base = ((size_t)(fX - 1) * c.L + fB) * 2;
#pragma unroll
        for (int t0 = 0; t0 < N; t0 += 32) {
            const int t = t0 + lane, k = t / (2 * M), e = t - k * 2 * M;  // row K X-1, K X, dK X, dK X+1
            if (t < (fX < nrows - 1 ? N : N - 2 * M))
                atomicAdd(reinterpret_cast<double*>(k < 2 ? a.HKR : a.HdKR) + base + (k == 0 ? 0 : k == 3 ? 2 * L2 : L2) + e,
                          s_acc[f * STRIDE + t]);
        }
    }
    __syncwarp();
}
template <int M>
__global__ void __launch_bounds__(32, 8) k_adj_b2ser(const DevCtx c, const AdjDev a, const int s, const int run) {
    wait_prior_grid();
    const StageDev& sp = c.stages[s];
    if (!(sp.T > 0.0)) return;
    __shared__ __align__(16) double s_acc[32 * (8 * M + 2)];
    const int L = c.L, nrows = sp.nrows, lane = threadIdx.x & 31;
    const long long NP = (long long)L * L;
    const long long q0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * run;
    double acc[M][8];
#pragma unroll
    for (int d = 0; d < M; ++d)
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[d][k] = 0.0;
    long long key = -1;
    int kX = 1, kB = 0, nkeys = 0;
    // the next packet is on its way while this one's FMAs run
    const int cnt = (int)max(0ll, min((long long)run, NP - q0));
    AdjDev::B2Packet nx = {};
    int nB = 0;
    double ninv = 0.0;
    if (cnt > 0) {
        nx = a.b2pk[q0];
        nB = __ldg(c.iB2 + nx.ij);
        ninv = c.inv_dtr[min(nx.X + 1, nrows - 1)];
    }
    for (int r = 0; r < run; ++r) {
        const AdjDev::B2Packet pk = nx;
        const int iB2 = nB;
        const double inv = ninv;
        const bool in = r < cnt;
        double w[M];
#pragma unroll
        for (int d = 0; d < M; d += 2) {
            const double2 v = in ? __ldg(reinterpret_cast<const double2*>(c.wB2 + (size_t)pk.ij * M + d)) : make_double2(0.0, 0.0);
            w[d] = v.x;
            w[d + 1] = v.y;
        }
        if (r + 1 < cnt) nx = a.b2pk[q0 + r + 1];
        const long long kq = ((long long)pk.X << 32) | (unsigned)iB2;
        const bool change = in && kq != key;
        const unsigned mask = __ballot_sync(0xffffffffu, change && nkeys > 0);
        if (mask) b2_flush<M>(c, a, mask, kX, kB, nrows, acc, s_acc);
        if (change) {
#pragma unroll
            for (int d = 0; d < M; ++d)
#pragma unroll
                for (int k = 0; k < 8; ++k) acc[d][k] = 0.0;
            key = kq;
            kX = pk.X;
            kB = iB2;
            ++nkeys;
        }
        double e[4];
        b2_coeffs(inv, pk.X, pk.x, nrows, e);
        double eg[8];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            eg[2 * k] = in ? e[k] * pk.gK : 0.0;
            eg[2 * k + 1] = in ? e[k] * pk.gR : 0.0;
        }
        if (r + 1 < cnt) {
            nB = __ldg(c.iB2 + nx.ij);
            ninv = c.inv_dtr[min(nx.X + 1, nrows - 1)];
        }
#pragma unroll
        for (int d = 0; d < M; ++d)
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[d][k] = fma(eg[k], w[d], acc[d][k]);
    }
    // one key over the whole warp: reduce across the lanes, 8 lanes add
    const long long k0 = __shfl_sync(0xffffffffu, key, 0);
    if (__all_sync(0xffffffffu, nkeys == 1 && key == k0)) {
        const int vi = warp_reduce8_index(lane);
        const bool cubic2 = kX < nrows - 1;
        const size_t base = (size_t)(kX - 1) * L + kB;
        // value vi: {K row X-1, K row X, dK row X, dK row X+1} x component
        double* dst = (double*)((vi >> 1) < 2 ? a.HKR : a.HdKR) +
                      2 * (base + ((vi >> 1) == 0 ? 0 : (vi >> 1) == 3 ? 2 * (size_t)L : (size_t)L)) + (vi & 1);
        const bool writer = (lane & 3) == 0 && ((vi >> 1) != 3 || cubic2);
#pragma unroll
        for (int d = 0; d < M; ++d) {
            const double tot = warp_reduce8(acc[d], lane);
            if (writer) atomicAdd(dst + 2 * d, tot);
        }
        return;
    }
    b2_flush<M>(c, a, __ballot_sync(0xffffffffu, nkeys > 0), kX, kB, nrows, acc, s_acc);
}

// B2 transposed for a generic stencil depth: one thread per packet, m taps
// added directly.
__global__ void __launch_bounds__(256) k_adj_b2gen(const DevCtx c, const AdjDev a, const int s) {
    wait_prior_grid();
    const StageDev& sp = c.stages[s];
    if (!(sp.T > 0.0)) return;
    const int L = c.L, m = c.m, nrows = sp.nrows;
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (long long)L * L) return;
    const AdjDev::B2Packet pk = a.b2pk[q];
    const int iB2 = __ldg(c.iB2 + pk.ij);
    double e[4];
    b2_coeffs(c.inv_dtr[min(pk.X + 1, nrows - 1)], pk.X, pk.x, nrows, e);
    const bool cubic2 = pk.X < nrows - 1;
    const size_t base = (size_t)(pk.X - 1) * L + iB2;
    const double* w = c.wB2 + (size_t)pk.ij * m;
    for (int d = 0; d < m; ++d) {
        const double wd = __ldg(w + d);
        const double gK = wd * pk.gK, gR = wd * pk.gR;
        add2(a.HKR + base + d, e[0] * gK, e[0] * gR);
        add2(a.HKR + base + L + d, e[1] * gK, e[1] * gR);
        add2(a.HdKR + base + L + d, e[2] * gK, e[2] * gR);
        if (cubic2) add2(a.HdKR + base + 2 * L + d, e[3] * gK, e[3] * gR);
    }
}

// sum over target rows of the last-row stencil cotangents (none at t = 0):
// block (bx, by) sums columns bx*32.. over the row slice by, 8 row lanes
// per column, then adds its column totals to the history cotangent
constexpr int LR_COLS = 32, LR_LANES = 8, LR_SLICES = 16;
__global__ void __launch_bounds__(LR_COLS * LR_LANES) k_adj_lastreduce(const DevCtx c, const AdjDev a, const int s,
                                                                      const int lr) {
    wait_prior_grid();
    const int L = c.L;
    if (!(c.stages[s].T > 0.0)) return;
    __shared__ double2 s_acc[LR_LANES][LR_COLS];
    const int tx = threadIdx.x % LR_COLS, ty = threadIdx.x / LR_COLS;
    const int k = blockIdx.x * LR_COLS + tx;
    const int rows = (L + LR_SLICES - 1) / LR_SLICES, i0 = blockIdx.y * rows, i1 = min(L, i0 + rows);
    double2 acc = make_double2(0.0, 0.0);
    if (k < L)
        for (int i = i0 + ty; i < i1; i += LR_LANES) {
            const double2 v = a.lbar_part[(size_t)i * L + k];
            acc.x += v.x;
            acc.y += v.y;
        }
    s_acc[ty][tx] = acc;
    __syncthreads();
    if (ty == 0 && k < L) {
        for (int q = 1; q < LR_LANES; ++q) {
            acc.x += s_acc[q][tx].x;
            acc.y += s_acc[q][tx].y;
        }
        add2(a.HKR + (size_t)lr * L + k, acc.x, acc.y);
    }
}

// g0 = row n0-1: its cotangent joins the history's
__global__ void k_adj_finish(const DevCtx c, const AdjDev a, const int n0) {
    const int L = c.L;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < L; j += gridDim.x * blockDim.x) {
        double2* h = a.HKR + (size_t)(n0 - 1) * L + j;
        const double2 g = a.g0bar[j];
        h->x += g.x;
        h->y += g.y;
    }
}

// t = 0 rows: r(0) = drvec(0) = Gamma + f'(1)/T0 (initialization.cpp:217-222)
__global__ void k_adj_initial(const AdjDev a, const AdjModel am) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    double f1, f1l;
    fder(am, 1, 1.0, f1, f1l);
    const double rb = a.Hr[0] + a.Hdr[0];
    a.sc[SC_GAMMA] += rb;
    a.sc[SC_LAMBDA] += rb * f1l / am.T0;
}

// the recomputed row n0 against the forward's (snapshot): mismatching elements
__global__ void k_adj_verify(const DevCtx c, const AdjDev a, const double2* snapKR, const double2* snapdKR,
                             const double* snapr, const double* snapdr, const int n0) {
    const int L = c.L;
    int bad = 0;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < L; j += gridDim.x * blockDim.x) {
        const double2 x = c.KR[(size_t)n0 * L + j], y = snapKR[(size_t)n0 * L + j];
        const double2 dx = c.dKR[(size_t)n0 * L + j], dy = snapdKR[(size_t)n0 * L + j];
        bad += (x.x != y.x) + (x.y != y.y) + (dx.x != dy.x) + (dx.y != dy.y);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) bad += (c.rvec[n0] != snapr[n0]) + (c.drvec[n0] != snapdr[n0]);
    if (bad) atomicAdd(a.sc + 15, (double)bad);
}

}  // namespace

cudaError_t launch_adj_verify(const DevCtx& c, const AdjDev& a, const double2* snapKR, const double2* snapdKR,
                              const double* snapr, const double* snapdr, int n0, cudaStream_t st) {
    k_adj_verify<<<(c.L + 255) / 256, 256, 0, st>>>(c, a, snapKR, snapdKR, snapr, snapdr, n0);
    return cudaGetLastError();
}

// ------------------------------------------------------------- launchers
// (p, p2) pairs with compile-time exponents; anything else takes the runtime ones
#define ADJ_DISPATCH(am, CALL)                                          \
    do {                                                                \
        if ((am).p == 3 && (am).p2 == 4) { constexpr int P = 3, P2 = 4; CALL; } \
        else if ((am).p == 3 && (am).p2 == 0) { constexpr int P = 3, P2 = 0; CALL; } \
        else { constexpr int P = -1, P2 = -1; CALL; }                   \
    } while (0)

cudaError_t launch_adj_seed(const DevCtx& c, const AdjDev& a, const AdjModel& am, int nl, double wE, double wR,
                            double wDr, const double* cK, const double* cR, const double* cdK, const double* cdR,
                            cudaStream_t st) {
    ADJ_DISPATCH(am, (k_adj_seed<P, P2><<<1, 256, 0, st>>>(c, a, am, nl, wE, wR, wDr, cK, cR, cdK, cdR)));
    return cudaGetLastError();
}

// k_adj_lastrow's shared memory: row sums, the row's A1/A2 cotangents and
// the column starts
size_t lastrow_smem(int L) { return 3 * (size_t)L * sizeof(double2) + (size_t)(L + 1) * sizeof(int); }

template <int P, int P2>
cudaError_t launch_targets_pp(const DevCtx& c, const AdjDev& a, const AdjModel& am, int s,
                              cudaStream_t st) {
    const dim3 grid((c.L + 63) / 64, c.L);
    const size_t lsm = lastrow_smem(c.L);
    const size_t NP = (size_t)c.L * c.L;
    cudaError_t e = launch_pdl(k_adj_targets<P, P2>, grid, dim3(64), 0, st, c, a, am, s);
    if (e != cudaSuccess) return e;
    if ((e = launch_pdl(k_adj_lastrow, dim3(c.L), dim3(LR_T), lsm, st, c, a, s)) != cudaSuccess) return e;
    if (c.m != 10) return launch_pdl(k_adj_b2gen, dim3((unsigned)((NP + 255) / 256)), dim3(256), 0, st, c, a, s);
    int dev = 0, sms = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    const size_t lanes = (size_t)32 * B2_WARPS_SM * sms;
    const int run = (int)std::max<size_t>(B2_RUN_MIN, (NP + lanes - 1) / lanes);
    return launch_pdl(k_adj_b2ser<10>, dim3((unsigned)((NP + 32 * (size_t)run - 1) / (32 * (size_t)run))), dim3(32), 0, st, c, a, s, run);
}
cudaError_t launch_targets(const DevCtx& c, const AdjDev& a, const AdjModel& am, int s,
                           cudaStream_t st) {
    if (am.p == 3 && am.p2 == 4) return launch_targets_pp<3, 4>(c, a, am, s, st);
    if (am.p == 3 && am.p2 == 0) return launch_targets_pp<3, 0>(c, a, am, s, st);
    return launch_targets_pp<-1, -1>(c, a, am, s, st);
}

cudaError_t launch_adj_save(const DevCtx& c, const AdjDev& a, int k, int n0, cudaStream_t st) {
    return launch_pdl(k_adj_save, dim3((c.L + 63) / 64), dim3(64), 0, st, c, a, k, n0);
}

cudaError_t launch_adj_step(const DevCtx& c, const AdjDev& a, const AdjModel& am, int S, int n0, cudaStream_t st) {
    const int L = c.L;
    const int eb = (L + 255) / 256;
    cudaError_t e;
    if ((e = cudaMemsetAsync(a.hbar, 0, (size_t)SMAX * L * sizeof(double2), st)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(a.g0bar, 0, (size_t)L * sizeof(double2), st)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(a.sc + SC_DR, 0, sizeof(double), st)) != cudaSuccess) return e;
    for (int s = S - 1; s >= 0; --s) {
        if ((e = launch_pdl(k_adj_enter, dim3((L + 63) / 64), dim3(64), 0, st, c, a, s, n0)) != cudaSuccess) return e;
        const dim3 rg((L + ADJ_ROW_T - 1) / ADJ_ROW_T);
        ADJ_DISPATCH(am, (e = launch_pdl(k_adj_rows<P, P2>, rg, dim3(ADJ_ROW_T), 0, st, c, a, am, s, n0)));
        if (e != cudaSuccess) return e;
        if ((e = launch_targets(c, a, am, s, st)) != cudaSuccess) return e;
        // the last row of stage s is row n0 (s >= 1) or n0-1 (s = 0)
        if ((e = launch_pdl(k_adj_lastreduce, dim3((L + LR_COLS - 1) / LR_COLS, LR_SLICES), dim3(LR_COLS * LR_LANES), 0, st, c, a,
                            s, s >= 1 ? n0 : n0 - 1)) != cudaSuccess)
            return e;
    }
    k_adj_finish<<<eb, 256, 0, st>>>(c, a, n0);
    return cudaGetLastError();
}

cudaError_t launch_adj_initial(const AdjDev& a, const AdjModel& am, cudaStream_t st) {
    k_adj_initial<<<1, 32, 0, st>>>(a, am);
    return cudaGetLastError();
}

// The limit belongs to the kernel, which other contexts launch too: what the longest rows need
cudaError_t adj_lastrow_smem_attr() {
    return cudaFuncSetAttribute(k_adj_lastrow, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lastrow_smem(4096));
}

}  // namespace dyn
