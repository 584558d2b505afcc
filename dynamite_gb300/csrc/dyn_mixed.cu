// Mixed-precision stage kernel of the DYNAMITE hot path.
//
// Same algorithm as k_main (dyn_kernels.cu; the B2 sums kept over the stages of a call
// included: L = 512 (hi, lo) 50 -> 33 us a stage, L = 1024 177 -> 105), with the O(L^2) work
// in FP32:
//   * stencil weights are FP32 copies of the FP64 tables;
//   * the history is read from an FP32 mirror (float2 (QK,QR), (dQK,dQR))
//     that the epilogue writes next to the FP64 master rows;
//   * A1/A2/B1/B2 gathers, Sigma and the eight convolution products are FP32
//     (in the (hi, lo) form double-float, the two pairs that share their factor
//     as one sum each); each thread accumulates its products compensated (TwoSum),
//     and the cross-lane fold and everything of size L (RHS, RK combination,
//     r(t), dr/dt, C(t,t), the step-error norm, time) stay in FP64.
// The position search is the exact FP64 binary search (integer compares on
// the bit patterns); only the fractional offset inside the located interval
// is formed in FP32 (one FP64 difference scaled by a stored FP32 inverse
// interval length), so interval indices equal the FP64 form's.  FP32 copies
// of int.dat and 1/delta_t_ratio keep conversions off the (slow) FP64 pipe.
#include <cmath>
#include "dyn_mixed.cuh"

namespace dyn {

constexpr int TPB_M = 128;  // threads, and targets, of a CTA

// The register cap (48) keeps ten CTAs per SM
template <int M, int P, int P2, bool KEEP>
__global__ void __launch_bounds__(TPB_M, 10) k_main_mixed(const DevCtx c, const int s) {
    wait_prior_grid();
    const StageDev& sp = c.stages[s];
    const int nside = (c.L + TPB_M - 1) / TPB_M;
    if (blockIdx.y < nside) {
        if (blockIdx.x == 0) mixed::side_rows(c, sp, blockIdx.y);
        return;
    }
    extern __shared__ float2 s_lastf[];
    __shared__ mixed::RowShared sh;
    __shared__ mixed::B2Jobs<KEEP ? TPB_M : 0> jb;
    const int i = c.L - 1 - (blockIdx.y - nside);
    const bool keep = KEEP && sp.b2_mode == B2_KEEP;
    if (threadIdx.x == 0) jb.n[0][0] = jb.n[0][1] = 0;
    mixed::row_setup<false>(c, sp, i, s_lastf, sh, !keep);
    __syncthreads();
    mixed::chunk_sums<M, 1, P, P2, true>(c, sp, blockIdx.x, 0, s_lastf, sh, i, jb, 0, keep);
    __syncthreads();
    mixed::fold_chunks<false, false>(c, i, blockIdx.x, 1, sh);
}


// The (hi, lo) form of k_main_mixed (device functions in dyn_mixed.cuh, namespace mdf)
template <int M, int P, int P2, bool KEEP>
__global__ void __launch_bounds__(TPB_M, 8) k_main_df(const DevCtx c, const int s) {
    wait_prior_grid();
    const StageDev& sp = c.stages[s];
    const int nside = (c.L + TPB_M - 1) / TPB_M;
    if (blockIdx.y < nside) {
        if (blockIdx.x == 0) mixed::side_rows(c, sp, blockIdx.y);
        return;
    }
    extern __shared__ float4 s_row[];  // [L] the last history row (hi, hi, lo, lo)
    __shared__ mixed::RowShared sh;
    __shared__ mixed::B2Jobs<KEEP ? TPB_M : 0> jb;
    __shared__ mdf::RowConst rc;
    const int i = c.L - 1 - (blockIdx.y - nside);
    const bool keep = KEEP && sp.b2_mode == B2_KEEP;
    if (threadIdx.x == 0) jb.n[0][0] = jb.n[0][1] = 0;
    mdf::row_setup<false>(c, sp, i, s_row, sh, rc, !keep);
    __syncthreads();
    mdf::chunk_dd<M, 1, P, P2>(c, sp, blockIdx.x, 0, s_row, rc, sh, i, jb, 0, keep);
    __syncthreads();
    mixed::fold_chunks<true, false>(c, i, blockIdx.x, 1, sh);
}

namespace {

template <int M, int P, int P2, bool KEEP>
cudaError_t launch_t(const DevCtx& c, int s, cudaStream_t st) {
    const dim3 grid(c.nch, c.L + (c.L + TPB_M - 1) / TPB_M);
    if (c.mixed == 2) {
        const size_t smem = (size_t)c.L * sizeof(float4);  // with the static part > 48 KB from L = 2700 on
        static std::atomic<unsigned long long> devs{0};
        const cudaError_t e = raise_smem_limit(k_main_df<M, P, P2, KEEP>, smem, 4096 * (int)sizeof(float4), devs);
        if (e != cudaSuccess) return e;
        return launch_pdl(k_main_df<M, P, P2, KEEP>, grid, dim3(TPB_M), smem, st, c, s);
    }
    return launch_pdl(k_main_mixed<M, P, P2, KEEP>, grid, dim3(TPB_M), (size_t)(c.L + 2) * sizeof(float2), st, c, s);
}

// The depth-10 plain form reads the staged row in element pairs, which pays where whole rows
// keep one parity (RK54 step at the odd L = 257: 144 us, the generic depth 141; the (hi, lo)
// form 153 against 171 at L = 257, 281 against 321 at 513)
bool depth_ten(const DevCtx& c) { return c.m == 10 && (c.mixed == 2 || c.L % 2 == 0); }

template <int P, int P2>
cudaError_t launch_pp(const DevCtx& c, int s, cudaStream_t st) {
    const bool ten = depth_ten(c);
    if (c.b2key) return ten ? launch_t<10, P, P2, true>(c, s, st) : launch_t<0, P, P2, true>(c, s, st);
    return ten ? launch_t<10, P, P2, false>(c, s, st) : launch_t<0, P, P2, false>(c, s, st);
}

__global__ void k_mirror(const DevCtx c, size_t off, size_t count) {
    for (size_t e = off + (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < off + count; e += (size_t)gridDim.x * blockDim.x) {
        const double2 v = c.KR[e], d = c.dKR[e];
        const float2 x = hi_lo(v.x), y = hi_lo(v.y);
        if (c.KRq) c.KRq[e] = make_float4(x.x, y.x, x.y, y.y);
        else c.KRf[e] = make_float2(x.x, y.x);
        c.dKRf[e] = make_float2((float)d.x, (float)d.y);
    }
}

// FP32 pairs of the inverse interval lengths and inverse step ratios of rows [0, n)
__global__ void k_time_f32(const double* t1, const double* dtr, int n, float2* inv_len, float2* inv_dtr) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        inv_dtr[k] = hi_lo(dtr[k] != 0.0 ? 1.0 / dtr[k] : 0.0);
        inv_len[k] = k + 1 < n ? hi_lo(1.0 / (t1[k + 1] - t1[k])) : make_float2(0.f, 0.f);
    }
}

// out[p][e] = the tap pair (2p, 2p+1) of target e in FP32 (second tap 0 past the depth);
// HL: the high parts, then the low ones
template <bool HL>
__global__ void k_weights_tapmajor(const double* in, void* out, size_t targets, int m) {
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < targets; e += (size_t)gridDim.x * blockDim.x)
        for (int d = 0; d < m; d += 2) {
            const float2 a = hi_lo(in[e * m + d]), b = d + 1 < m ? hi_lo(in[e * m + d + 1]) : make_float2(0.f, 0.f);
            const size_t o = (size_t)(d >> 1) * targets + e;
            if constexpr (HL) static_cast<float4*>(out)[o] = make_float4(a.x, b.x, a.y, b.y);
            else static_cast<float2*>(out)[o] = make_float2(a.x, b.x);
        }
}

}  // namespace

// The planes pay in every form but the plain one at depth 10, whose sums are cheap beside the
// 36 bytes a target that the planes add to the 144 it reads.  Up to L = 672 all of it stays in
// L2 and keeping wins.  From there on it does not, while a short history still does, from which
// the sums are formed anew: a lone step is better off so (its first stage, which fills the planes,
// costs more than the others save), a call of four steps up to about 8 (L - 640) rows.  From 2048
// on the weights alone fill L2, and two million elements of history do.  us with planes / without,
// RK54, one step | a call of four:
//   L =  704,  300 rows  327 /  300 | 1104 /  1113     L = 1024,  3500 rows  640 /  592 |  2150 /  2142
//   L =  768,  600 rows  419 /  369 | 1377 /  1340     L = 1536,  4500 rows 1269 / 1161 |  4222 /  4205
//   L =  768, 1200 rows  419 /  382 | 1382 /  1406     L = 2048,   600 rows 2106 / 2030 |  7005 /  7290
//   L = 1024,  600 rows  628 /  532 | 2124 /  1945     L = 2048,  1100 rows 2153 / 2294 |  7078 /  8266
bool b2_planes(const DevCtx& c, size_t rows, int steps) {
    if (!c.b2key) return false;
    if (c.mixed != 1 || !depth_ten(c) || c.L <= 672) return true;
    if (c.L >= 2048) return steps >= 4 || rows * c.L >= (size_t)2 << 20;
    return steps >= 4 && rows >= 8 * (size_t)(c.L - 640);
}

cudaError_t launch_main_mixed(const DevCtx& c, int s, cudaStream_t st) {
    if (c.M.p == 3 && c.M.p2 == 4) return launch_pp<3, 4>(c, s, st);
    if (c.M.p == 3 && c.M.p2 == 0) return launch_pp<3, 0>(c, s, st);
    return launch_pp<-1, -1>(c, s, st);
}

cudaError_t launch_mirror(const DevCtx& c, size_t off, size_t count, cudaStream_t st) {
    const int blocks = (int)((count + 255) / 256 < 8192 ? (count + 255) / 256 : 8192);
    k_mirror<<<blocks > 0 ? blocks : 1, 256, 0, st>>>(c, off, count);
    return cudaGetLastError();
}

cudaError_t launch_time_f32(const double* t1, const double* dtr, int n, float2* inv_len, float2* inv_dtr,
                            cudaStream_t st) {
    k_time_f32<<<(n + 255) / 256, 256, 0, st>>>(t1, dtr, n, inv_len, inv_dtr);
    return cudaGetLastError();
}

cudaError_t launch_weights_tapmajor(const double* in, void* out, int mixed, size_t targets, int m, cudaStream_t st) {
    const int blocks = (int)((targets + 255) / 256 < 8192 ? (targets + 255) / 256 : 8192);
    if (mixed == 2) k_weights_tapmajor<true><<<blocks > 0 ? blocks : 1, 256, 0, st>>>(in, out, targets, m);
    else k_weights_tapmajor<false><<<blocks > 0 ? blocks : 1, 256, 0, st>>>(in, out, targets, m);
    return cudaGetLastError();
}

}  // namespace dyn
