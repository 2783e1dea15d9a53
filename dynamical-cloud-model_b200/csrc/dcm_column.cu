// dcm_column.cu -- the PAMM microphysics' sedimentation transport on the GPU:
// mpdata_vec_1d with first_order_upstream_1d (pamm/sfvt/advection_1d.F90:35-74,
// 463-778) for many independent columns at once, each with the caller's
// sub-stepping loop (pamm/microphysics.f90:3139-3145, 3158-3164, 3177-3183:
// n_step passes of dt/n_step, n_step from the column's largest fall speed).
//
// One warp per column.  The column's fields, a copy of the first field (the
// limiter's psi), the input and two working velocity columns, a flux buffer
// and the limiter's beta_up / beta_down sit in shared memory; every statement
// of the Fortran is a pass of the 32 lanes over the levels, separated by
// __syncwarp.  Reductions over k (minval, the positivity test's sum) are warp
// shuffles.  All arithmetic is FP64, in the reference's order of terms but for
// k_column_donor, which forms one reciprocal per level and rounds otherwise (up
// to 4e-16 of a column's largest value).
#include <algorithm>
#include <cstring>

#include "dcm_internal.h"

namespace {

constexpr double COL_SMALL = 1e-60;  // pamm/sfvt/advection_1d.F90:18
constexpr int COL_WARPS = 4;         // columns per block at most

struct ColArgs {
    int ncol, kp, nq, l_h, r_h, nw, npsi, per_warp;  // per_warp: doubles of shared memory
    int mstride, kord, monotone, neumann;
    const double *dt, *dz, *dzn, *rhoa, *rhoan, *w;
    const int* nsub;
    double* psi;
};

__device__ __forceinline__ double wmin(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ double wsum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// first_order_upstream_1d (:35-74) on one field p (level-0 pointer), the new
// values through tmp so that every lane reads the old neighbours
__device__ void col_upstream(double dt, const double* dzn, const double* rhoa,
                             const double* rhoan, int kp, const double* w, double* p,
                             int neumann, double* tmp, int lane) {
    for (int k = 1 + lane; k <= kp; k += 32) {
        const double den = 2.0 * dzn[k] * rhoan[k];
        const double wk = w[k], wm = w[k - 1];
        double fr = ((wk + fabs(wk)) * rhoa[k] * p[k] + (wk - fabs(wk)) * rhoa[k] * p[k + 1]) *
                    dt / den;
        double fl = ((wm + fabs(wm)) * rhoa[k - 1] * p[k - 1] +
                     (wm - fabs(wm)) * rhoa[k - 1] * p[k]) *
                    dt / den;
        if (neumann == 1) {  // :65-67, in the reference's order
            if (k == 1) fl = fr;
            if (k == kp) fr = fl;
        } else if (neumann == 2) {  // :68-70
            if (k == 1) fl = -fr;
            if (k == kp) fr = -fl;
        }
        tmp[k] = p[k] - (fr - fl);  // :73
    }
    __syncwarp();
    for (int k = 1 + lane; k <= kp; k += 32) p[k] = tmp[k];
    __syncwarp();
    if (lane == 0) {  // halos after each pass (:755-761)
        p[0] = 0.0;
        p[kp + 1] = 0.0;
    }
    __syncwarp();
}

// halos of a working velocity column (:656-657, :732-733)
__device__ __forceinline__ void col_w_halos(double* w, int kp, int lane) {
    if (lane == 0) {
        w[0] = w[1];
        w[kp] = w[kp - 1];
        w[kp + 1] = w[kp - 1];
    }
    __syncwarp();
}

// one call of mpdata_vec_1d (:463-778) on the column in shared memory
__device__ void col_mpdata(const ColArgs& a, double dt, const double* dz, const double* dzn,
                           const double* rhoa, const double* rhoan, const double* win,
                           double* psi, double* store, double* ws1, double* ws2, double* tmp,
                           double* bup, double* bdn, double* ming, int lane) {
    const int kp = a.kp, nq = a.nq, npsi = a.npsi, nw = a.nw;
    const int op = a.r_h - 1;
    auto P = [&](int n) { return psi + (size_t)n * npsi + op; };
    // positive definite (:507-516): minval over the interior, shift every
    // element (halos included)
    for (int n = 0; n < nq; n++) {
        double* p = P(n);
        double m = INFINITY;
        for (int k = 1 + lane; k <= kp; k += 32) m = fmin(m, p[k]);
        m = wmin(m);
        if (lane == 0) ming[n] = m;
        for (int k = -a.r_h + 1 + lane; k <= kp + a.r_h; k += 32) p[k] = p[k] - m;
    }
    __syncwarp();
    // :518-529; the interior sum is a shuffle tree here (index order in the
    // reference): it only meets the 1e-60 threshold, and the terms are >= 0
    double s = 0.0;
    for (int k = 1 + lane; k <= kp; k += 32) s += P(0)[k];
    s = wsum(s);
    if (s < COL_SMALL) {
        for (int n = 0; n < nq; n++)
            for (int k = -a.r_h + 1 + lane; k <= kp + a.r_h; k += 32) P(n)[k] += ming[n];
        __syncwarp();
        return;
    }
    const int ow = a.l_h - 1;
    const bool anti = a.kord > 1;
    double* w1 = anti ? ws1 + ow : nullptr;  // level-0 views of the working velocities
    double* w2 = anti ? ws2 + ow : nullptr;
    if (anti)
        for (int i = lane; i < nw; i += 32) ws2[i] = 0.0;  // :530 (read only when kord > 1)
    const double* wt = win + ow;                        // :534-535
    double* wt_sav = w1;
    const double* ps = anti ? store + op : nullptr;  // the limiter's psi (:542-545)
    double* po = P(0);              // psi_old (:547)
    if (a.kord > 1)
        for (int i = lane; i < npsi; i += 32) store[i] = psi[i];
    __syncwarp();
    int it2 = 0;
    for (int it = 1; it <= a.kord; it++) {
        if (it > 1) {  // antidiffusive velocities (:553-635)
            it2 = it2 + 1;
            for (int k = 1 + lane; k <= kp; k += 32) {
                const double g_bar3 = 0.5 * (rhoan[k] + rhoan[k + 1]);
                const double wk = wt[k];
                double v = (fabs(wk) * dz[k] - dt * (rhoa[k] / g_bar3) * wk * wk) *
                               (po[k + 1] - po[k]) / (po[k + 1] + po[k] + COL_SMALL) / dzn[k] -
                           0.0;
                v = v - 0.25 * dt * wk *
                            ((rhoa[k + 1] * wt[k + 1] - rhoa[k - 1] * wt[k - 1]) / dz[k - 1] +
                             0.0) /
                            g_bar3;
                wt_sav[k] = v;
            }
            __syncwarp();
            double* nwt = (it2 % 2 == 1) ? w1 : w2;  // :641-648
            wt_sav = (it2 % 2 == 1) ? w2 : w1;
            col_w_halos(nwt, kp, lane);
            wt = nwt;
        }
        if (it > 1 && a.monotone) {  // the NFT limiter (:666-745)
            it2 = it2 + 1;
            double* bu = bup + op;
            double* bd = bdn + op;
            for (int k = 1 + lane; k <= kp; k += 32) {
                const double mx = fmax(fmax(fmax(ps[k - 1], ps[k]), fmax(ps[k + 1], po[k - 1])),
                                       fmax(po[k], po[k + 1]));
                const double mn = fmin(fmin(fmin(ps[k - 1], ps[k]), fmin(ps[k + 1], po[k - 1])),
                                       fmin(po[k], po[k + 1]));
                const double denom1 = dt *
                                          (fmax(wt[k - 1], 0.0) * rhoa[k - 1] * po[k - 1] -
                                           fmin(wt[k], 0.0) * rhoa[k] * po[k + 1]) /
                                          dzn[k] +
                                      COL_SMALL;
                const double denom2 = dt *
                                          (fmax(wt[k], 0.0) * rhoa[k] * po[k] -
                                           fmin(wt[k - 1], 0.0) * rhoa[k - 1] * po[k]) /
                                          dzn[k] +
                                      COL_SMALL;
                bu[k] = rhoan[k] * (mx - po[k]) / denom1;
                bd[k] = rhoan[k] * (po[k] - mn) / denom2;
            }
            for (int k = 1 - a.r_h + lane; k <= 0; k += 32) bu[k] = bd[k] = 0.0;  // :698-701
            for (int k = kp + 1 + lane; k <= kp + a.r_h; k += 32) bu[k] = bd[k] = 0.0;
            __syncwarp();
            for (int k = 1 + lane; k <= kp; k += 32)  // :709-715
                wt_sav[k] = fmin(fmin(1.0, bd[k]), bu[k + 1]) * fmax(wt[k], 0.0) +
                            fmin(fmin(1.0, bu[k]), bd[k + 1]) * fmin(wt[k], 0.0);
            __syncwarp();
            wt_sav = w1;  // :720-721: the limited velocities are in w_store2
            col_w_halos(w2, kp, lane);
            wt = w2;
        }
        for (int n = 0; n < nq; n++)  // :748-764
            col_upstream(dt, dzn, rhoa, rhoan, kp, wt, P(n), a.neumann, tmp + op, lane);
    }
    for (int n = 0; n < nq; n++)  // :775-777
        for (int k = -a.r_h + 1 + lane; k <= kp + a.r_h; k += 32) P(n)[k] += ming[n];
    __syncwarp();
}

// 8 blocks of 4 warps per SM (64 registers): the donor-cell form (the
// sedimentation calls) took 0.237 ms for 65,536 columns of 128 levels and two
// fields at this bound, 0.267 ms at 6 blocks and 0.361 ms unbounded (126
// registers, 4 blocks)
__global__ void __launch_bounds__(32 * COL_WARPS, 8) k_column_mpdata(ColArgs a) {
    extern __shared__ double col_sm[];
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = blockIdx.x * (blockDim.x >> 5) + wib;
    if (c >= a.ncol) return;  // the whole warp: no block-wide barrier follows
    // [nq][npsi] fields, then with kord > 1 the limiter's psi, the input and
    // the two working velocities, the flux buffer, beta_up, beta_down, the
    // minima; with kord <= 1 (the donor cell alone) the flux buffer, the
    // input velocity and the minima only, so that more columns fit an SM
    double* psi = col_sm + (size_t)wib * a.per_warp;
    double* rest = psi + (size_t)a.nq * a.npsi;
    double *store = nullptr, *ws1 = nullptr, *ws2 = nullptr, *bup = nullptr, *bdn = nullptr;
    double *tmp, *win, *ming;
    if (a.kord > 1) {
        store = rest;
        win = store + a.npsi;
        ws1 = win + a.nw;
        ws2 = ws1 + a.nw;
        tmp = ws2 + a.nw;
        bup = tmp + a.npsi;
        bdn = bup + a.npsi;
        ming = bdn + a.npsi;
    } else {
        tmp = rest;
        win = tmp + a.npsi;
        ming = win + a.nw;
    }
    double* gpsi = a.psi + (size_t)c * a.nq * a.npsi;
#pragma unroll 4
    for (int i = lane; i < a.nq * a.npsi; i += 32) psi[i] = gpsi[i];
#pragma unroll 4
    for (int i = lane; i < a.nw; i += 32) win[i] = a.w[(size_t)c * a.nw + i];
    if (ws1)
        for (int i = lane; i < a.nw; i += 32) ws1[i] = 0.0;
    __syncwarp();
    const size_t mo = (size_t)c * a.mstride + (a.l_h - 1);
    const double *dz = a.dz + mo, *dzn = a.dzn + mo, *rhoa = a.rhoa + mo, *rhoan = a.rhoan + mo;
    const int ns = a.nsub ? max(a.nsub[c], 1) : 1;
    const double dt = a.dt[c] / (double)ns;
    for (int s = 0; s < ns; s++)
        col_mpdata(a, dt, dz, dzn, rhoa, rhoan, win, psi, store, ws1, ws2, tmp, bup, bdn, ming,
                   lane);
#pragma unroll 4
    for (int i = lane; i < a.nq * a.npsi; i += 32) gpsi[i] = psi[i];
}

// The sedimentation calls (kord 1, one halo level in psi): the column in
// registers, level 1 + lane + 32 m of every field, so that neither the fields
// nor the flux buffer pass through shared memory and no index arithmetic
// remains (k_column_mpdata spends 3,000 warp instructions per column on the
// same work, 77 % issue-bound).  A face's numerator
//     N(k) = ((w + |w|) rhoa p(k) + (w - |w|) rhoa p(k+1)) dt
// serves both levels it separates, and 1 / (2 dzn rhoan) is formed once per
// column instead of two divisions per level, field and pass.  65,536 columns of
// 128 levels and two fields, with a copy of the fields before each call: 272 us with
// k_column_mpdata, 158 with this kernel (the copy 40, the floor of both 73).
template <int M, int NQ>
__global__ void __launch_bounds__(32 * COL_WARPS) k_column_donor(ColArgs a) {
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int c = blockIdx.x * COL_WARPS + (threadIdx.x >> 5);
    if (c >= a.ncol) return;
    const int kp = a.kp;
    // level-0 views
    double* __restrict__ gp = a.psi + (size_t)c * NQ * a.npsi;
    const double* __restrict__ w = a.w + (size_t)c * a.nw + (a.l_h - 1);
    const size_t mo = (size_t)c * a.mstride + (a.l_h - 1);
    const double *dzn = a.dzn + mo, *rhoa = a.rhoa + mo, *rhoan = a.rhoan + mo;
    const int ns = a.nsub ? max(a.nsub[c], 1) : 1;
    const double dt = a.dt[c] / (double)ns;
    double p[NQ][M], A[M], B[M], rd[M], lo[NQ], hi[NQ];
#pragma unroll
    for (int n = 0; n < NQ; n++) {
#pragma unroll
        for (int m = 0; m < M; m++) {
            const int k = 1 + lane + 32 * m;
            p[n][m] = k <= kp ? gp[(size_t)n * a.npsi + k] : 0.0;
        }
        lo[n] = gp[(size_t)n * a.npsi];  // halo levels 0 and kp + 1
        hi[n] = gp[(size_t)n * a.npsi + kp + 1];
    }
#pragma unroll
    for (int m = 0; m < M; m++) {
        const int k = min(1 + lane + 32 * m, kp);
        const double wk = w[k], ra = rhoa[k] * dt;
        A[m] = (wk + fabs(wk)) * ra;
        B[m] = (wk - fabs(wk)) * ra;
        rd[m] = 1.0 / (2.0 * dzn[k] * rhoan[k]);
    }
    const double w0 = w[0], ra0 = rhoa[0] * dt;
    const double A0 = (w0 + fabs(w0)) * ra0, B0 = (w0 - fabs(w0)) * ra0;
    for (int s = 0; s < ns; s++) {
        // positive definite (:507-516)
        double mn[NQ];
#pragma unroll
        for (int n = 0; n < NQ; n++) {
            double v = INFINITY;
#pragma unroll
            for (int m = 0; m < M; m++)
                if (1 + lane + 32 * m <= kp) v = fmin(v, p[n][m]);
            mn[n] = wmin(v);
#pragma unroll
            for (int m = 0; m < M; m++) p[n][m] -= mn[n];
            lo[n] -= mn[n];
            hi[n] -= mn[n];
        }
        double sum = 0.0;  // :518-529
#pragma unroll
        for (int m = 0; m < M; m++)
            if (1 + lane + 32 * m <= kp) sum += p[0][m];
        if (!(wsum(sum) < COL_SMALL)) {
#pragma unroll
            for (int n = 0; n < NQ; n++) {
                // p(k+1): the next lane's, for lane 31 lane 0's next
                double up[M], N[M];
#pragma unroll
                for (int m = 0; m < M; m++) up[m] = __shfl_sync(FULL, p[n][m], lane + 1);
#pragma unroll
                for (int m = 0; m < M; m++) {
                    const int k = 1 + lane + 32 * m;
                    double x = up[m];
                    if (lane == 31) x = m + 1 < M ? up[m + 1 < M ? m + 1 : m] : hi[n];
                    if (k == kp) x = hi[n];
                    N[m] = A[m] * p[n][m] + B[m] * x;
                }
                // N(k-1): the lane below's, for lane 0 lane 31's before
                const double first = __shfl_sync(FULL, p[n][0], 0);
                double dn[M];
#pragma unroll
                for (int m = 0; m < M; m++) dn[m] = __shfl_sync(FULL, N[m], lane + 31);
                const double N0 = A0 * lo[n] + B0 * first;
#pragma unroll
                for (int m = M - 1; m >= 0; m--) {
                    const int k = 1 + lane + 32 * m;
                    double below = dn[m];
                    if (lane == 0) below = m > 0 ? dn[m > 0 ? m - 1 : 0] : N0;
                    double fr = N[m] * rd[m], fl = below * rd[m];
                    if (a.neumann == 1) {  // :65-67, in the reference's order
                        if (k == 1) fl = fr;
                        if (k == kp) fr = fl;
                    } else if (a.neumann == 2) {  // :68-70
                        if (k == 1) fl = -fr;
                        if (k == kp) fr = -fl;
                    }
                    p[n][m] -= fr - fl;  // :73
                }
                lo[n] = hi[n] = 0.0;  // :755-761
            }
        }
#pragma unroll
        for (int n = 0; n < NQ; n++) {  // :775-777
#pragma unroll
            for (int m = 0; m < M; m++) p[n][m] += mn[n];
            lo[n] += mn[n];
            hi[n] += mn[n];
        }
    }
#pragma unroll
    for (int n = 0; n < NQ; n++) {
        double* __restrict__ g = gp + (size_t)n * a.npsi;
#pragma unroll
        for (int m = 0; m < M; m++) {
            const int k = 1 + lane + 32 * m;
            if (k <= kp) g[k] = p[n][m];
        }
        if (lane == 0) {
            g[0] = lo[n];
            g[kp + 1] = hi[n];
        }
    }
}

// launches k_column_donor where it applies: up to 256 levels and three fields
// (its registers), else false
template <int M>
static bool donor_m(const ColArgs& a, cudaStream_t st) {
    const int nb = (a.ncol + COL_WARPS - 1) / COL_WARPS;
    switch (a.nq) {
        case 1: k_column_donor<M, 1><<<nb, 32 * COL_WARPS, 0, st>>>(a); return true;
        case 2: k_column_donor<M, 2><<<nb, 32 * COL_WARPS, 0, st>>>(a); return true;
        case 3: k_column_donor<M, 3><<<nb, 32 * COL_WARPS, 0, st>>>(a); return true;
        default: return false;
    }
}
static bool donor_launch(const ColArgs& a, cudaStream_t st) {
    if (a.kord != 1 || a.r_h != 1) return false;
    switch ((a.kp + 31) / 32) {
        case 1: return donor_m<1>(a, st);
        case 2: return donor_m<2>(a, st);
        case 3: return donor_m<3>(a, st);
        case 4: return donor_m<4>(a, st);
        case 5: return donor_m<5>(a, st);
        case 6: return donor_m<6>(a, st);
        case 7:
        case 8: return donor_m<8>(a, st);
        default: return false;
    }
}

}  // namespace

// shape checks shared by both entry points; fills the launch shape
static int column_shape(int ncol, int kp, int nq, int l_h, int r_h, int metric_stride,
                        int kord, int neumann, ColArgs& a, int& warps, size_t& smem) {
    if (ncol < 0 || kp < 1 || nq < 1 || l_h < 1 || r_h < 1 || kord < 0 || neumann < 0 ||
        neumann > 2)
        return DCM_E_ARG;
    const int nw = kp + l_h + r_h, npsi = kp + 2 * r_h;
    if (metric_stride != 0 && metric_stride != nw) return DCM_E_ARG;
    const int per_warp = kord > 1 ? (nq + 4) * npsi + 3 * nw + nq : (nq + 1) * npsi + nw + nq;
    const size_t warp_bytes = (size_t)per_warp * sizeof(double);
    constexpr size_t max_bytes = 200 * 1024;
    if (warp_bytes > max_bytes) return DCM_E_ARG;  // a column too tall for shared memory
    warps = std::max(1, std::min<int>(COL_WARPS, (int)(max_bytes / warp_bytes)));
    smem = (size_t)warps * warp_bytes;
    a = ColArgs{};
    a.ncol = ncol;
    a.kp = kp;
    a.nq = nq;
    a.l_h = l_h;
    a.r_h = r_h;
    a.nw = nw;
    a.npsi = npsi;
    a.per_warp = per_warp;
    a.mstride = metric_stride;
    a.kord = kord;
    a.neumann = neumann;
    return DCM_OK;
}

static bool column_launch(const ColArgs& a, int warps, size_t smem, cudaStream_t st) {
    if (donor_launch(a, st)) return cudaPeekAtLastError() == cudaSuccess;
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(k_column_mpdata, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem) != cudaSuccess)
        return false;
    k_column_mpdata<<<(a.ncol + warps - 1) / warps, 32 * warps, smem, st>>>(a);
    return cudaPeekAtLastError() == cudaSuccess;
}

extern "C" int dcm_mpdata_vec_1d_device(int ncol, int kp, int nq, int l_h, int r_h,
                                        const double* dt, const int* nsub, const double* dz,
                                        const double* dzn, const double* rhoa,
                                        const double* rhoan, int metric_stride,
                                        const double* w, double* psi, int kord, int monotone,
                                        int neumann, void* stream) {
    ColArgs a;
    int warps = 1;
    size_t smem = 0;
    const int st = column_shape(ncol, kp, nq, l_h, r_h, metric_stride, kord, neumann, a,
                                warps, smem);
    if (st != DCM_OK || ncol == 0) return st;
    if (!dt || !dz || !dzn || !rhoa || !rhoan || !w || !psi) return DCM_E_ARG;
    if (cudaPeekAtLastError() != cudaSuccess) return DCM_E_CUDA;  // not ours to clear
    a.monotone = monotone ? 1 : 0;
    a.dt = dt;
    a.nsub = nsub;
    a.dz = dz;
    a.dzn = dzn;
    a.rhoa = rhoa;
    a.rhoan = rhoan;
    a.w = w;
    a.psi = psi;
    return column_launch(a, warps, smem, (cudaStream_t)stream) ? DCM_OK : DCM_E_CUDA;
}

// Device memory of the host-array calls, kept by the thread that makes them
// (at most 32 MB, of one context) and freed when it ends: a cudaMalloc and the
// cudaFree, which waits for the device, took most of a call of a few hundred
// columns.  A thread's calls return after their last copy, so its next call
// finds the memory free.  It is used in, and given back to, the context it
// came from only: contexts are told apart by the driver's identifiers, which
// are not used twice.
namespace {
constexpr size_t COL_KEEP = 32u << 20;
constexpr size_t COL_PACK = 16u << 10;  // small arrays that go in one copy

// the current context's identifier, 0 where there is none yet (or no way to ask)
unsigned long long context_id() {
    using Ask = int (*)(void*, unsigned long long*);  // cuCtxGetId
    static const Ask ask = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &found) != cudaSuccess)
            cudaGetLastError();
        else if (found == cudaDriverEntryPointSuccess)
            return (Ask)f;
        return (Ask) nullptr;
    }();
    unsigned long long id = 0;
    return ask && ask(nullptr, &id) == 0 ? id : 0;
}

struct ColSpace {
    char* p = nullptr;
    size_t n = 0;
    unsigned long long context = 0;
    // (memory of another context is left to that context's end)
    void drop() {
        if (p && context_id() == context) cudaFree(p);
        p = nullptr;
        n = 0;
    }
    bool take(size_t want, char** out) {
        if (want > COL_KEEP) return false;
        const unsigned long long now = context_id();
        if (now == 0) return false;
        if (want > n || now != context) {
            drop();
            context = now;
            const size_t size = std::min(COL_KEEP, want + want / 2);
            if (cudaMalloc(&p, size) != cudaSuccess) {
                cudaGetLastError();
                p = nullptr;
                return false;
            }
            n = size;
        }
        *out = p;
        return true;
    }
    ~ColSpace() { drop(); }
};
thread_local ColSpace col_space;
}  // namespace

extern "C" int dcm_mpdata_vec_1d(int ncol, int kp, int nq, int l_h, int r_h, const double* dt,
                                 const int* nsub, const double* dz, const double* dzn,
                                 const double* rhoa, const double* rhoan, int metric_stride,
                                 const double* w, double* psi, int kord, int monotone,
                                 int neumann) {
    ColArgs a;
    int warps = 1;
    size_t smem = 0;
    const int st = column_shape(ncol, kp, nq, l_h, r_h, metric_stride, kord, neumann, a,
                                warps, smem);
    if (st != DCM_OK || ncol == 0) return st;
    if (!dt || !dz || !dzn || !rhoa || !rhoan || !w || !psi) return DCM_E_ARG;
    if (nsub)
        for (int c = 0; c < ncol; c++)
            if (nsub[c] < 1) return DCM_E_ARG;
    const int nw = a.nw, npsi = a.npsi;
    const size_t nmet = (size_t)(metric_stride ? ncol : 1) * nw;
    const size_t bytes_dt = (size_t)ncol * sizeof(double), bytes_ns = (size_t)ncol * sizeof(int);
    const size_t bytes_met = nmet * sizeof(double), bytes_w = (size_t)ncol * nw * sizeof(double);
    const size_t bytes_psi = (size_t)ncol * nq * npsi * sizeof(double);
    const size_t al = 256;
    auto up = [&](size_t b) { return (b + al - 1) / al * al; };
    // [dt | nsub | four metrics] in one copy, then w, then psi
    const size_t head = up(bytes_dt) + up(bytes_ns) + 4 * up(bytes_met);
    char* buf = nullptr;
    ColSpace& space = col_space;
    const size_t total = head + up(bytes_w) + up(bytes_psi);
    const bool kept = space.take(total, &buf);
    if (!kept && cudaMalloc(&buf, total) != cudaSuccess) return DCM_E_CUDA;
    size_t off = 0;
    auto take = [&](size_t b) {
        char* p = buf + off;
        off += up(b);
        return p;
    };
    double* d_dt = (double*)take(bytes_dt);
    int* d_ns = (int*)take(bytes_ns);
    double* d_met[4];
    for (double*& m : d_met) m = (double*)take(bytes_met);
    double* d_w = (double*)take(bytes_w);
    double* d_psi = (double*)take(bytes_psi);
    const double* h_met[4] = {dz, dzn, rhoa, rhoan};
    bool good = true;
    auto send = [&](void* d, const void* h, size_t n) {
        good = good && cudaMemcpyAsync(d, h, n, cudaMemcpyHostToDevice, 0) == cudaSuccess;
    };
    char packed[COL_PACK];
    if (head <= COL_PACK) {
        auto at = [&](const void* d) { return packed + ((const char*)d - buf); };
        std::memcpy(at(d_dt), dt, bytes_dt);
        if (nsub) std::memcpy(at(d_ns), nsub, bytes_ns);
        for (int q = 0; q < 4; q++) std::memcpy(at(d_met[q]), h_met[q], bytes_met);
        send(buf, packed, head);
    } else {
        send(d_dt, dt, bytes_dt);
        if (nsub) send(d_ns, nsub, bytes_ns);
        for (int q = 0; q < 4; q++) send(d_met[q], h_met[q], bytes_met);
    }
    send(d_w, w, bytes_w);
    send(d_psi, psi, bytes_psi);
    a.monotone = monotone ? 1 : 0;
    a.dt = d_dt;
    a.nsub = nsub ? d_ns : nullptr;
    a.dz = d_met[0];
    a.dzn = d_met[1];
    a.rhoa = d_met[2];
    a.rhoan = d_met[3];
    a.w = d_w;
    a.psi = d_psi;
    if (good) good = column_launch(a, warps, smem, 0);
    if (good) good = cudaMemcpy(psi, d_psi, bytes_psi, cudaMemcpyDeviceToHost) == cudaSuccess;
    if (kept) {
        // nothing of a failed call may still be reading the packed arrays
        if (!good) cudaStreamSynchronize(0);
        return good ? DCM_OK : DCM_E_CUDA;
    }
    const bool freed = cudaFree(buf) == cudaSuccess;
    return good && freed ? DCM_OK : DCM_E_CUDA;
}
