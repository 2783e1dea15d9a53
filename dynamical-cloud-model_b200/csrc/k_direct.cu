// k_direct.cu -- direct corrections of the mixed-precision pressure solve.
//
// With uniform horizontal spacings the operator of set_mat_a
// (dynamics.f90:87-95) is a sum of a periodic circulant along x, one along y
// and a tridiagonal along z, so transforms along x and y reduce the 3-D
// equation to one tridiagonal system per horizontal mode, whatever the
// vertical spacing.  A correction solves A dx = r for the FP32 residual r of
// the FP64 pressure and adds dx to the pressure:
//     x <- x + A^-1 (b - A x)
// Solved in FP32 it lowers the FP64 residual by four to five decades, so two
// or three corrections reach the 1e-10 that FP32 BiCGSTAB iterations need
// 70 to 190 for (256 x 256 x 128 warm bubble).  refine_run (k_solver.cu)
// takes the corrections and, where one does not contract the residual, goes
// on with the BiCGSTAB iterations: from the pressure as corrected, or on
// grids where that may be no better (DIRECT_SURE) from the one it started with.
//
// Kernels per correction, each one pass in and one pass out of one FP32 field:
//   k_fft      transform along y (r -> scratch)
//   k_fft      transform along x (in place)
//   k_zsolve   tridiagonal system of every mode's column (in place)
//   k_fft      inverse transform along x (in place)
//   k_fft      inverse transform along y, x += result (FP64)
//   k_dir_residual   r = b - A x, its norm, convergence and loop condition
//
// Two consecutive levels of a column make one complex number, so a real field
// transforms as complex sequences in its own layout and nothing is padded or
// repacked: Z(m) = F1(m) + i F2(m) with the spectra F1, F2 of the two levels.
// The operator's eigenvalues are even in m, and the pair Z(m), Z(-m) holds the
// complex F1(m), F2(m), which k_zsolve forms in registers: their real and
// imaginary parts are two real right-hand sides of the mode's one matrix.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <type_traits>
#include <vector>

#include "dcm_internal.h"
#include "dcm_prof.h"

namespace dcm {

// ---- small DFTs in registers -------------------------------------------------
// cos and sin of 2 pi m / n at compile time, by their Taylor series
constexpr double kTwoPi = 6.283185307179586476925286766559;
constexpr double tw_series(double x, bool sine) {
    double term = sine ? x : 1.0, sum = term;
    for (int q = sine ? 3 : 2; q < 60; q += 2) {
        term *= -x * x / ((q - 1) * q);
        sum += term;
    }
    return sum;
}
template <int N>
struct Roots {
    float c[N]{}, s[N]{};
    constexpr Roots() {
        for (int m = 0; m < N; m++) {
            // the exact values at multiples of a quarter turn
            const int q = 4 * m % N == 0 ? 4 * m / N : -1;
            c[m] = q >= 0 ? (q == 0 ? 1.0f : q == 2 ? -1.0f : 0.0f)
                          : (float)tw_series(kTwoPi * m / N, false);
            s[m] = q >= 0 ? (q == 1 ? 1.0f : q == 3 ? -1.0f : 0.0f)
                          : (float)tw_series(kTwoPi * m / N, true);
        }
    }
};

__device__ __forceinline__ float2 cadd(float2 a, float2 b) {
    return make_float2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
    return make_float2(a.x - b.x, a.y - b.y);
}
// a (c - i s), without the products by 0 and 1
__device__ __forceinline__ float2 crot(float2 a, float c, float s) {
    if (s == 0.0f) return c > 0.0f ? a : make_float2(-a.x, -a.y);
    if (c == 0.0f) return s > 0.0f ? make_float2(a.y, -a.x) : make_float2(-a.y, a.x);
    return make_float2(a.x * c + a.y * s, a.y * c - a.x * s);
}
__device__ __forceinline__ float2 cmul_conj(float2 a, float2 w) {  // w = (cos, sin)
    return make_float2(a.x * w.x + a.y * w.y, a.y * w.x - a.x * w.y);
}

template <int R>
__device__ __forceinline__ void dft(float2 (&v)[R]);

// R = R1 R2: R2 transforms of length R1, twiddles, R1 transforms of length R2
template <int R1, int R2>
__device__ __forceinline__ void dft_product(float2 (&v)[R1 * R2]) {
    constexpr Roots<R1 * R2> W;
    float2 y[R2][R1];
#pragma unroll
    for (int q = 0; q < R2; q++) {
#pragma unroll
        for (int p = 0; p < R1; p++) y[q][p] = v[R2 * p + q];
        dft<R1>(y[q]);
    }
#pragma unroll
    for (int p = 0; p < R1; p++) {
        float2 z[R2];
#pragma unroll
        for (int q = 0; q < R2; q++) z[q] = crot(y[q][p], W.c[p * q], W.s[p * q]);
        dft<R2>(z);
#pragma unroll
        for (int q = 0; q < R2; q++) v[p + R1 * q] = z[q];
    }
}

// odd R: sums and differences of the mirrored pairs
template <int R>
__device__ __forceinline__ void dft_odd(float2 (&v)[R]) {
    constexpr Roots<R> W;
    constexpr int H = (R - 1) / 2;
    float2 p[H], m[H], o[R];
    o[0] = v[0];
#pragma unroll
    for (int j = 0; j < H; j++) {
        p[j] = cadd(v[j + 1], v[R - 1 - j]);
        m[j] = csub(v[j + 1], v[R - 1 - j]);
        o[0] = cadd(o[0], p[j]);
    }
#pragma unroll
    for (int s = 1; s <= H; s++) {
        float2 a = v[0], b = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int j = 0; j < H; j++) {
            const int q = (j + 1) * s % R;
            a.x += W.c[q] * p[j].x;
            a.y += W.c[q] * p[j].y;
            b.x += W.s[q] * m[j].x;
            b.y += W.s[q] * m[j].y;
        }
        o[s] = make_float2(a.x + b.y, a.y - b.x);      // a - i b
        o[R - s] = make_float2(a.x - b.y, a.y + b.x);  // a + i b
    }
#pragma unroll
    for (int q = 0; q < R; q++) v[q] = o[q];
}

template <int R>
__device__ __forceinline__ void dft(float2 (&v)[R]) {
    if constexpr (R == 2) {
        const float2 a = v[0];
        v[0] = cadd(a, v[1]);
        v[1] = csub(a, v[1]);
    } else if constexpr (R == 4) {
        const float2 a = cadd(v[0], v[2]), b = csub(v[0], v[2]);
        const float2 c = cadd(v[1], v[3]), e = csub(v[1], v[3]);
        v[0] = cadd(a, c);
        v[2] = csub(a, c);
        v[1] = make_float2(b.x + e.y, b.y - e.x);
        v[3] = make_float2(b.x - e.y, b.y + e.x);
    } else if constexpr (R == 6) {
        dft_product<2, 3>(v);
    } else if constexpr (R == 8) {
        dft_product<2, 4>(v);
    } else if constexpr (R == 9) {
        dft_product<3, 3>(v);
    } else if constexpr (R == 10) {
        dft_product<2, 5>(v);
    } else if constexpr (R == 12) {
        dft_product<3, 4>(v);
    } else if constexpr (R == 14) {
        dft_product<2, 7>(v);
    } else if constexpr (R == 15) {
        dft_product<3, 5>(v);
    } else if constexpr (R == 16) {
        dft_product<4, 4>(v);
    } else {
        dft_odd<R>(v);
    }
}

// One Stockham pass of radix R over the C sequences of a tile: rows r0, r0 +
// rg, ... of butterflies per thread.  store(first element, stride, values).
template <int R, bool FIRST, typename L, typename St>
__device__ __forceinline__ void fft_pass(int n, int ns, const float2* __restrict__ tw, L load,
                                         St store, int r0, int rg) {
    const int nb = n / R;
    for (int b = r0; b < nb; b += rg) {
        float2 v[R];
#pragma unroll
        for (int t = 0; t < R; t++) v[t] = load(b + t * nb);
        const int kk = FIRST ? 0 : b % ns;
        if (!FIRST) {
            const int step = kk * (n / (ns * R));
#pragma unroll
            for (int t = 1; t < R; t++) v[t] = cmul_conj(v[t], __ldg(tw + t * step));
        }
        dft<R>(v);
        store((b - kk) * R + kk, ns, v);
    }
}

// a pass of any radix p (a prime factor above 13): each output is a sum of p
// products
template <typename L, typename St>
__device__ __forceinline__ void fft_pass_any(int p, int n, int ns, const float2* __restrict__ tw,
                                             L load, St store, int r0, int rg) {
    const int nb = n / p;
    for (int o = r0; o < n; o += rg) {
        const int s = o / nb, b = o - s * nb, kk = b % ns;
        const int q1 = (kk + s * ns) * (n / (ns * p));  // < n
        float2 acc = make_float2(0.0f, 0.0f);
        int q = 0;
        for (int t = 0; t < p; t++) {
            const float2 x = load(b + t * nb), w = __ldg(tw + q);
            acc.x += x.x * w.x + x.y * w.y;
            acc.y += x.y * w.x - x.x * w.y;
            q += q1;
            if (q >= n) q -= n;
        }
        const float2 v[1] = {acc};
        store((b - kk) * p + kk + s * ns, 0, v);
    }
}

// The first pass of such a radix, on the tile's elements in shared memory (x at
// [m C]), where they are first replaced by the sums and differences of mirrored
// pairs t, p - t: outputs s and p - s then share their products, a quarter of
// them in all.  An item is a pair of outputs (s = 0: one).
template <int C, typename St>
__device__ __forceinline__ void fft_first_any(int p, int n, const float2* __restrict__ tw,
                                              float2* x, St store, int r0, int rg) {
    const int nb = n / p, h = (p - 1) / 2;
    for (int e = r0; e < nb * h; e += rg) {
        const int b = e % nb, t = 1 + e / nb;
        const float2 u = x[(b + t * nb) * C], v = x[(b + (p - t) * nb) * C];
        x[(b + t * nb) * C] = cadd(u, v);
        x[(b + (p - t) * nb) * C] = csub(u, v);
    }
    __syncthreads();
    for (int e = r0; e < nb * (h + 1); e += rg) {
        const int b = e % nb, s = e / nb;
        float2 a = x[b * C], d = make_float2(0.0f, 0.0f);
        const int q1 = s * nb;  // < n
        int q = 0;
#pragma unroll 4
        for (int t = 1; t <= h; t++) {
            q += q1;
            if (q >= n) q -= n;
            const float2 u = x[(b + t * nb) * C], v = x[(b + (p - t) * nb) * C];
            const float2 w = __ldg(tw + q);
            a.x += w.x * u.x;
            a.y += w.x * u.y;
            d.x += w.y * v.x;
            d.y += w.y * v.y;
        }
        const float2 lo[1] = {make_float2(a.x + d.y, a.y - d.x)};
        const float2 hi[1] = {make_float2(a.x - d.y, a.y + d.x)};
        store(b * p + s, 0, lo);
        if (s) store(b * p + p - s, 0, hi);
    }
}

template <bool FIRST, typename L, typename St>
__device__ __forceinline__ void fft_pass_of(int radix, int n, int ns,
                                            const float2* __restrict__ tw, L load, St store,
                                            int r0, int rg) {
    switch (radix) {
#define DCM_PASS(R)                                             \
    case R:                                                     \
        fft_pass<R, FIRST>(n, ns, tw, load, store, r0, rg);     \
        break;
        DCM_PASS(2) DCM_PASS(3) DCM_PASS(4) DCM_PASS(5) DCM_PASS(6) DCM_PASS(7) DCM_PASS(8)
        DCM_PASS(9) DCM_PASS(10) DCM_PASS(11) DCM_PASS(12) DCM_PASS(13) DCM_PASS(14)
        DCM_PASS(15) DCM_PASS(16)
#undef DCM_PASS
        default: break;
    }
}

// ---- FFT along one horizontal axis -----------------------------------------------
// A block transforms C pairs of levels (2 C consecutive levels) of one row or
// column of the domain; every element of the tile is one C x 8 byte segment of
// memory.  The first pass reads memory and the last writes it, so two radices
// (n up to 256) meet in shared memory once; more take two buffers in turn.
// The inverse is the forward transform with real and imaginary parts
// exchanged.  256 x 256 x 128: 27 us a transform (67 MB, 10 us at the copy rate;
// half of the field comes from L2), bound by instruction fetch (the unrolled
// radices, a third of the stalls) and by loads in flight at 80 registers;
// FFT_ADD 44 us (168 MB, 26 us), bound by the wait for x.
enum FftMode {
    FFT_REAL = 0,  // forward, of a real field
    FFT_FWD,       // forward, of complex pairs
    FFT_INV,       // inverse, complex pairs
    FFT_ADD        // inverse into a real field: x (FP64) += it; an element that
                   // is not finite is left out, so that x stays usable
};
constexpr int FFT_THREADS = 256;

struct FftArgs {
    int n, nrad;
    int rad[DIRECT_MAX_RADICES];
    const float2* tw;  // n roots (cos, sin)(2 pi q / n)
    int line, batch;   // element strides along the axis and across rows
    int kp, base;      // levels; index of (k, j, i) = (0, 1, 1)
};

template <int C, int MODE>
__global__ void __launch_bounds__(FFT_THREADS, 3) k_fft(FftArgs a, const float* src, float* dst,
                                                     double* __restrict__ x) {
    extern __shared__ float2 fft_buf[];
    constexpr bool INV = MODE == FFT_INV || MODE == FFT_ADD;
    const int n = a.n, c = threadIdx.x % C, r0 = threadIdx.x / C;
    constexpr int RG = FFT_THREADS / C;
    float2* cur = fft_buf + c;
    float2* nxt = fft_buf + n * C + c;  // with three passes or more
    const int k0 = 1 + 2 * ((int)blockIdx.x * C + c);
    const bool one = k0 <= a.kp, both = k0 < a.kp;
    const int o0 = a.base + (int)blockIdx.y * a.batch + k0;
    auto swap = [](float2 v) { return INV ? make_float2(v.y, v.x) : v; };
    // an odd last level is paired with a zero, in the scratch with the column's
    // first padding element
    auto get = [&](int m) -> float2 {
        const float* p = src + o0 + m * a.line;
        if (both || (MODE != FFT_REAL && one)) return swap(*reinterpret_cast<const float2*>(p));
        return swap(make_float2(one ? *p : 0.0f, 0.0f));
    };
    auto put = [&](int m, int stride, const auto& v) {
        constexpr int R = sizeof(v) / sizeof(float2);
        if constexpr (MODE != FFT_ADD) {
#pragma unroll
            for (int t = 0; t < R; t++)
                if (one)
                    *reinterpret_cast<float2*>(dst + o0 + (m + t * stride) * a.line) = swap(v[t]);
        } else {
            // x's values four at a time, so that their reads overlap
            constexpr int G = R < 4 ? R : 4;
#pragma unroll
            for (int t = 0; t < R; t += G) {
                double2 y[G];
#pragma unroll
                for (int g = 0; g < G; g++)
                    if (t + g < R && one)
                        y[g] = *reinterpret_cast<const double2*>(
                            x + o0 + (m + (t + g) * stride) * a.line);
#pragma unroll
                for (int g = 0; g < G; g++) {
                    if (t + g >= R || !one) continue;
                    float2 h = swap(v[t + g < R ? t + g : 0]);
                    if (!(fabsf(h.x) <= FLT_MAX)) h.x = 0.0f;
                    if (!(fabsf(h.y) <= FLT_MAX)) h.y = 0.0f;
                    double* w = x + o0 + (m + (t + g) * stride) * a.line;
                    y[g].x += (double)h.x;
                    y[g].y += (double)h.y;
                    if (both)
                        *reinterpret_cast<double2*>(w) = y[g];
                    else
                        *w = y[g].x;
                }
            }
        }
    };
    int ns = 1, q = 0;
    const bool small0 = a.nrad > 0 && a.rad[0] <= 16;
    if (a.nrad == 1 && small0) {
        fft_pass_of<true>(a.rad[0], n, 1, a.tw, get, put, r0, RG);
        return;
    }
    if (small0) {
        float2* d = cur;
        fft_pass_of<true>(a.rad[0], n, 1, a.tw, get,
                          [&](int m, int stride, const auto& v) {
#pragma unroll
                              for (int t = 0; t < (int)(sizeof(v) / sizeof(float2)); t++)
                                  d[(m + t * stride) * C] = v[t];
                          },
                          r0, RG);
        ns = a.rad[0];
        q = 1;
    } else {
        for (int m = r0; m < n; m += RG) cur[m * C] = get(m);
        if (a.nrad == 0) {  // n = 1
            const float2 v[1] = {cur[0]};
            if (r0 == 0) put(0, 0, v);
            return;
        }
    }
    __syncthreads();
    if (q == 0) {
        const int p = a.rad[0];
        if (a.nrad == 1) {
            fft_first_any<C>(p, n, a.tw, cur, put, r0, RG);
            return;
        }
        float2* d = nxt;
        fft_first_any<C>(p, n, a.tw, cur,
                         [&](int m, int, const auto& v) { d[m * C] = v[0]; }, r0, RG);
        ns = p;
        q = 1;
        nxt = cur;
        cur = d;
        __syncthreads();
    }
    for (; q < a.nrad; q++) {
        const int r = a.rad[q];
        const float2* s = cur;
        auto load = [&](int m) { return s[m * C]; };
        if (q + 1 == a.nrad) {
            if (r <= 16)
                fft_pass_of<false>(r, n, ns, a.tw, load, put, r0, RG);
            else
                fft_pass_any(r, n, ns, a.tw, load, put, r0, RG);
            return;
        }
        float2* d = nxt;
        auto store = [&](int m, int stride, const auto& v) {
#pragma unroll
            for (int t = 0; t < (int)(sizeof(v) / sizeof(float2)); t++)
                d[(m + t * stride) * C] = v[t];
        };
        if (r <= 16)
            fft_pass_of<false>(r, n, ns, a.tw, load, store, r0, RG);
        else
            fft_pass_any(r, n, ns, a.tw, load, store, r0, RG);
        ns *= r;
        nxt = cur;
        cur = d;
        __syncthreads();
    }
}

// ---- the tridiagonal systems along z ----------------------------------------------
// One warp per pair of modes m, -m, V consecutive levels per lane.  Their two
// columns give the real and imaginary parts of the levels' spectra, two
// right-hand sides of one matrix.  Each lane eliminates its inner levels (the
// partition method), the last level of every lane then forms a 32-row
// tridiagonal system that cyclic reduction over the lanes solves in five
// shuffle steps, and the inner levels follow by substitution.  A thread per
// column (the Thomas recurrence) would be a chain of 2 kp dependent steps.
// The horizontal mean mode is singular (Neumann at both ends): it is
// integrated twice in FP64, with the additive constant that leaves the sum of
// a_p dz-weighted values unchanged, which is the constant Jacobi-preconditioned
// iterations leave unchanged too.
template <int V>
__device__ __forceinline__ void zload(const float* __restrict__ p, int nvalid, float (&v)[V]) {
#pragma unroll
    for (int e = 0; e < V; e++) v[e] = 0.0f;
    constexpr int N = V < 4 ? V : 4;
#pragma unroll
    for (int e = 0; e < V; e += N) {
        if (e < nvalid) {  // the vector ends inside the column's padding
            if constexpr (N == 4) {
                const float4 t = *reinterpret_cast<const float4*>(p + e);
                v[e] = t.x; v[e + 1] = t.y; v[e + 2] = t.z; v[e + 3] = t.w;
            } else {
                const float2 t = *reinterpret_cast<const float2*>(p + e);
                v[e] = t.x; v[e + 1] = t.y;
            }
        }
    }
#pragma unroll
    for (int e = 0; e < V; e++)
        if (e >= nvalid) v[e] = 0.0f;
}
template <int V>
__device__ __forceinline__ void zstore(float* __restrict__ p, int nvalid, const float (&v)[V]) {
    constexpr int N = V < 4 ? V : 4;
#pragma unroll
    for (int e = 0; e < V; e += N) {
        if (e + N <= nvalid) {
            if constexpr (N == 4)
                *reinterpret_cast<float4*>(p + e) = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
            else
                *reinterpret_cast<float2*>(p + e) = make_float2(v[e], v[e + 1]);
        } else {
#pragma unroll
            for (int f = 0; f < N; f++)
                if (e + f < nvalid) p[e + f] = v[e + f];
        }
    }
}

struct ZArgs {
    Dims d;
    const float *au, *ad;      // per level
    const float *lx, *ly;      // eigenvalues along x and y, scaled as au, ad
    const double *w, *g, *l;   // mean mode: row weights, 1/(w au), constant's weights / their sum
    float scale;               // 1 / (ip jp): the two inverse transforms
};

__device__ __forceinline__ double warp_scan(double v) {  // inclusive
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    return v;
}

// the mean mode's column D in place
template <int V>
__device__ __forceinline__ void mean_mode(const ZArgs& a, int k0, int nvalid, float (&D)[V]) {
    double q[V], s = 0.0;
#pragma unroll
    for (int e = 0; e < V; e++) {
        if (e < nvalid) s += a.w[k0 + e] * (double)D[e];
        q[e] = s;
    }
    double before = warp_scan(s) - s, t = 0.0;
#pragma unroll
    for (int e = 0; e < V; e++) {
        const double step = k0 + e < a.d.kp ? (q[e] + before) * a.g[k0 + e] : 0.0;
        q[e] = t;
        t += step;
    }
    before = warp_scan(t) - t;
    double m = 0.0;
#pragma unroll
    for (int e = 0; e < V; e++) {
        q[e] += before;
        if (e < nvalid) m += a.l[k0 + e] * q[e];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
#pragma unroll
    for (int e = 0; e < V; e++) D[e] = e < nvalid ? (float)(q[e] - m) : 0.0f;
}

template <int V>
__global__ void __launch_bounds__(256) k_zsolve(ZArgs a, float* __restrict__ f) {
    constexpr unsigned FULL = 0xffffffffu;
    const Dims& d = a.d;
    const int lane = threadIdx.x & 31, kp = d.kp, ip = d.ip, jp = d.jp;
    const int k0 = 1 + V * lane;
    const int nvalid = max(0, min(V, kp - k0 + 1));
    // levels of the columns in memory: an odd kp has one more (the imaginary
    // part of its last pair)
    const int nmem = max(0, min(V, kp + (kp & 1) - k0 + 1));
    float au[V], ad[V];
#pragma unroll
    for (int e = 0; e < V; e++) {
        const int k = k0 + e;
        au[e] = k < kp ? ld(a.au + k) : 0.0f;
        ad[e] = k > 1 && k <= kp ? ld(a.ad + k) : 0.0f;
    }
    // modes with 0 <= mx <= ip / 2; of the rows mx = 0 and mx = ip / 2, which
    // hold their own partners, half
    const int nmode = (ip / 2 + 1) * jp, nw = gridDim.x * 8;
    for (int mode = blockIdx.x * 8 + (threadIdx.x >> 5); mode < nmode; mode += nw) {
        const int mx = mode / jp, my = mode - mx * jp;
        const int px = mx ? ip - mx : 0, py = my ? jp - my : 0;
        if (px == mx && my > py) continue;
        const bool self = px == mx && py == my;
        float* __restrict__ p = f + d.at(k0, 1 + my, 1 + mx);
        float* __restrict__ pp = f + d.at(k0, 1 + py, 1 + px);
        float D[V], E[V];  // real and imaginary parts of the levels' spectra
        zload<V>(p, nmem, D);
        if (self) {
#pragma unroll
            for (int e = 0; e < V; e++) {
                D[e] = e < nvalid ? D[e] * a.scale : 0.0f;
                E[e] = 0.0f;
            }
        } else {
            zload<V>(pp, nmem, E);
            const float h = 0.5f * a.scale;
#pragma unroll
            for (int e = 0; e < V; e += 2) {  // (x, y) = Z(m), (z, w) = Z(-m)
                const float x = D[e], y = D[e + 1], z = E[e], w = E[e + 1];
                D[e] = h * (x + z);
                D[e + 1] = h * (y + w);
                E[e] = h * (y - w);
                E[e + 1] = h * (z - x);
            }
#pragma unroll
            for (int e = 0; e < V; e++)
                if (e >= nvalid) D[e] = E[e] = 0.0f;
        }
        if (mode == 0) {
            mean_mode<V>(a, k0, nvalid, D);
            zstore<V>(p, nmem, D);
            continue;
        }
        const float lam = -(ld(a.lx + mx) + ld(a.ly + my));
        // normalised rows u + A u(below) + C u(above) = D with A, C <= 0, and
        // S = 1 + A + C, the row's excess over its neighbours (lam / diagonal
        // at first), carried through the elimination: every diagonal is then a
        // sum of positive terms.  Formed as 1 - products it loses the excess
        // where lam is below the round-off of au + ad (flat cells: dx 50 dz and
        // 512 points made the first mode's system singular).
        float A[V], C[V], S[V];
#pragma unroll
        for (int e = 0; e < V; e++) {
            // rows beyond kp: u = 0
            float ex = e < nvalid ? lam : 1.0f;
            if (e < 2) {
                const float r = __fdividef(-1.0f, ex + ad[e] + au[e]);
                D[e] *= r;
                E[e] *= r;
                A[e] = ad[e] * r;
                C[e] = au[e] * r;
                S[e] = -r * ex;
            } else {
                ex += ad[e] * S[e - 1];
                const float r = __fdividef(-1.0f, ex - ad[e] * A[e - 1] + au[e]);
                D[e] = r * (D[e] - ad[e] * D[e - 1]);
                E[e] = r * (E[e] - ad[e] * E[e - 1]);
                A[e] = -r * ad[e] * A[e - 1];
                C[e] = r * au[e];
                S[e] = -r * ex;
            }
        }
#pragma unroll
        for (int e = V - 3; e >= 1; e--) {
            D[e] -= C[e] * D[e + 1];
            E[e] -= C[e] * E[e + 1];
            A[e] -= C[e] * A[e + 1];
            S[e] -= C[e] * S[e + 1];
            C[e] = -C[e] * C[e + 1];
        }
        if (V > 2) {
            const float ex = S[0] - C[0] * S[1];
            const float r = __fdividef(1.0f, ex - A[0] + C[0] * C[1]);
            D[0] = r * (D[0] - C[0] * D[1]);
            E[0] = r * (E[0] - C[0] * E[1]);
            A[0] = r * A[0];
            C[0] = -r * C[0] * C[1];
            S[0] = r * ex;
        }
        // the last levels: first levels of this lane and the next eliminated
        const float dn = __shfl_down_sync(FULL, D[0], 1), en = __shfl_down_sync(FULL, E[0], 1),
                    sn = __shfl_down_sync(FULL, S[0], 1), cn = __shfl_down_sync(FULL, C[0], 1);
        const float al = A[V - 1], cl = C[V - 1];
        float ex = S[V - 1] - al * S[0] - cl * sn;
        float r = __fdividef(1.0f, ex + al * A[0] + cl * cn);
        float x = r * (D[V - 1] - al * D[0] - cl * dn);
        float y = r * (E[V - 1] - al * E[0] - cl * en);
        float lo = -r * al * A[0], up = -r * cl * cn, sx = r * ex;
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
            // lo is 0 in the first s lanes and up in the last s, so what the
            // shuffles return there does not count
            const float xm = __shfl_up_sync(FULL, x, s), ym = __shfl_up_sync(FULL, y, s),
                        lm = __shfl_up_sync(FULL, lo, s), sm = __shfl_up_sync(FULL, sx, s);
            const float xp = __shfl_down_sync(FULL, x, s), yp = __shfl_down_sync(FULL, y, s),
                        sp = __shfl_down_sync(FULL, sx, s), upp = __shfl_down_sync(FULL, up, s);
            ex = sx - lo * sm - up * sp;
            r = __fdividef(1.0f, ex + lo * lm + up * upp);
            x = r * (x - lo * xm - up * xp);
            y = r * (y - lo * ym - up * yp);
            lo = -r * lo * lm;
            up = -r * up * upp;
            sx = r * ex;
        }
        float px1 = __shfl_up_sync(FULL, x, 1), py1 = __shfl_up_sync(FULL, y, 1);
        if (lane == 0) px1 = py1 = 0.0f;
        D[0] = D[0] - A[0] * px1 - C[0] * x;
        E[0] = E[0] - A[0] * py1 - C[0] * y;
#pragma unroll
        for (int e = 1; e < V - 1; e++) {
            D[e] = D[e] - A[e] * D[0] - C[e] * x;
            E[e] = E[e] - A[e] * E[0] - C[e] * y;
        }
        D[V - 1] = x;
        E[V - 1] = y;
        if (!self) {
#pragma unroll
            for (int e = 0; e < V; e += 2) {
                const float re = D[e], rf = D[e + 1], im = E[e], in = E[e + 1];
                D[e] = re - in;
                D[e + 1] = im + rf;
                E[e] = re + in;
                E[e + 1] = rf - im;
            }
            zstore<V>(pp, nmem, E);
        }
        zstore<V>(p, nmem, D);
    }
}

// ---- FP64 residual of the pressure, and the loop's decision -------------------------
// r = b - A x in FP64 (mat_ax, dynamics.f90:219-222), stored in FP32, with
// ||r|| and, at the start of a solve, ||b||.  A warp holds 64 levels (one
// 16-byte vector per lane) of one row and marches along i with the i - 1, i
// and i + 1 columns in registers.  (Loading the next plane ahead into
// registers left two blocks per SM: 75 us against
// 55 at 256 x 256 x 128; 235 MB, 36 us at the copy rate.)
struct DirResidualArgs {
    Dims d;
    Coef<double> c;
    const double *x, *b;
    double* keep;  // FIRST: a copy of x, unless null
    float* r;
    double tol;
    int itmax, max_rounds;
    int ni;  // planes per block
    cudaGraphConditionalHandle cond;
    int use_cond;
};

template <bool FIRST>
__global__ void __launch_bounds__(256, 4) k_dir_residual(DirResidualArgs a, Red2 R,
                                                      SolverScalars* S) {
    __shared__ double smem[64];
    const Dims& d = a.d;
    const int lane = threadIdx.x, ip = d.ip, jp = d.jp, kp = d.kp;
    const int k0 = 1 + 2 * ((int)blockIdx.x * 32 + lane);
    const int j = 1 + blockIdx.y * BY + threadIdx.y;
    const int i0 = 1 + blockIdx.z * a.ni, i1 = min(i0 + a.ni - 1, ip);
    double acc[2] = {0.0, 0.0};
    if (j <= jp) {  // whole warps
        const bool live = k0 <= kp, both = k0 < kp;
        const int kl = live ? k0 : 1;
        const int KJ = d.K * d.J;
        const double* __restrict__ x = a.x + kl + d.K * j;
        const double* __restrict__ bb = a.b + kl + d.K * j;
        float* __restrict__ rr = a.r + kl + d.K * j;
        const int ds = (j == 1 ? jp - 1 : -1) * d.K, dn = (j == jp ? 1 - jp : 1) * d.K;
        const double an = ld(a.c.an + j), as = ld(a.c.as + j);
        const double au0 = ld(a.c.au + kl), au1 = ld(a.c.au + kl + 1), ad0 = ld(a.c.ad + kl),
                     ad1 = ld(a.c.ad + kl + 1);
        auto at = [](const double* p) { return *reinterpret_cast<const double2*>(p); };
        double2 xw = at(x + KJ * (i0 == 1 ? ip : i0 - 1)), xc = at(x + KJ * i0);
        for (int i = i0; i <= i1; i++) {
            const int o = KJ * i;
            const double2 xe = at(x + KJ * (i == ip ? 1 : i + 1)), xs = at(x + o + ds),
                          xn = at(x + o + dn), bv = at(bb + o);
            double prev = __shfl_up_sync(0xffffffffu, xc.y, 1);
            double next = __shfl_down_sync(0xffffffffu, xc.x, 1);
            if (lane == 0 && live && k0 > 1) prev = x[o - 1];
            if (lane == 31 && k0 + 2 <= kp) next = x[o + 2];
            const double ae = ld(a.c.ae + i), aw = ld(a.c.aw + i);
            const double sij = -ae - aw - an - as;
            if (k0 == 1) prev = xc.x;  // Neumann rows, :206-211
            const double up0 = k0 == kp ? xc.x : xc.y;
            if (k0 + 1 == kp) next = xc.y;
            const double r0 = bv.x - (aw * xw.x + ae * xe.x + as * xs.x + an * xn.x + ad0 * prev +
                                      au0 * up0 + (sij - au0 - ad0) * xc.x);
            const double r1 = bv.y - (aw * xw.y + ae * xe.y + as * xs.y + an * xn.y + ad1 * xc.x +
                                      au1 * next + (sij - au1 - ad1) * xc.y);
            if (FIRST && a.keep && live) {
                double* kx = a.keep + kl + d.K * j + o;
                if (both)
                    *reinterpret_cast<double2*>(kx) = xc;
                else
                    *kx = xc.x;
            }
            if (live) {
                acc[0] += r0 * r0;
                if (FIRST) acc[1] += bv.x * bv.x;
            }
            if (both) {
                acc[0] += r1 * r1;
                if (FIRST) acc[1] += bv.y * bv.y;
                *reinterpret_cast<float2*>(rr + o) = make_float2((float)r0, (float)r1);
            } else if (live) {
                rr[o] = (float)r0;
            }
            xw = xc;
            xc = xe;
        }
    }
    block_reduce<R_SUM, 2>(acc, smem);
    double s[2];
    if (!(reduce2<2>(acc, R, smem, s) && threadIdx.x == 0 && threadIdx.y == 0)) return;
    if (FIRST) {
        double sc = sqrt(s[1]);
        sc = sc > 0.01 ? sc : 0.01;  // dynamics.f90:370-371
        S->sc_err = sc;
        S->it = 0;
        S->status = 0;
        S->done = 0;
        S->pause = 0;
        S->early = 0;
        S->updates = 0;
        S->rounds = 0;
        S->cycles = 0;
        S->ru_runs = 0;
        S->restarts = 0;
        S->restart = 0;
        S->fresh = 0;
        S->cycle_it = 0;
        S->dir_runs = 0;
    }
    const double err = sqrt(s[0]) / S->sc_err;
    int go = 0;
    if (err < a.tol) {
        S->done = 1;
        S->early = FIRST ? 1 : 0;
    } else if (FIRST && !(err == err)) {
        S->status = DCM_E_NONFINITE;
        S->done = 1;
    } else if (FIRST || err < DIRECT_CONTRACTION * S->err) {
        // another correction, within the limits of the iterations (none from
        // an infinite residual to an infinite one)
        if (S->it >= a.itmax) {
            S->status = DCM_E_NOCONV;
            S->done = 1;
        } else if (S->rounds >= a.max_rounds) {
            S->status = DCM_E_TIMEOUT;
            S->done = 1;
        } else {
            go = 1;
            S->it = S->it + 1;
            S->rounds = S->rounds + 1;
            S->updates = S->updates + 1;
            S->dir_runs = S->dir_runs + 1;
        }
    }
    S->err = err;
    S->direct = go;
    if (a.use_cond) cudaGraphSetConditional(a.cond, (unsigned)go);
}

__global__ void __launch_bounds__(256) k_dir_put_back(Dims d, const double* __restrict__ keep,
                                                      double* __restrict__ x) {
    const int k = 1 + blockIdx.x * BX + threadIdx.x;
    const int j = 1 + blockIdx.y * BY + threadIdx.y;
    const int i = 1 + blockIdx.z;
    if (k > d.kp || j > d.jp) return;
    x[d.at(k, j, i)] = keep[d.at(k, j, i)];
}

// ---- host side ----------------------------------------------------------------------
namespace {

// radices of n: as few passes as possible, then the smallest sum (fewest
// operations); prime factors above 13 go first, as passes of their own
bool best_radices(int n, std::vector<int>& cur, std::vector<int>& best) {
    if (n == 1) {
        auto cost = [](const std::vector<int>& v) {
            int s = 0;
            for (int r : v) s += r;
            return (int)v.size() * 1000 + s;
        };
        if (best.empty() || cost(cur) < cost(best)) best = cur;
        return true;
    }
    bool any = false;
    for (int r = 16; r >= 2; r--) {
        if (n % r || (!cur.empty() && r > cur.back())) continue;
        cur.push_back(r);
        any = best_radices(n / r, cur, best) || any;
        cur.pop_back();
    }
    return any;
}

std::vector<int> radices(int n) {
    std::vector<int> big, cur, best;
    for (int p = 17; p <= n; p += 2) {
        bool prime = true;
        for (int q = 3; q * q <= p; q += 2) prime = prime && p % q != 0;
        while (prime && n % p == 0) {
            big.push_back(p);
            n /= p;
        }
    }
    if (n > 1) best_radices(n, cur, best);
    big.insert(big.end(), best.begin(), best.end());
    return big;
}

bool uniform(const std::vector<double>& a, const std::vector<double>& b, int n) {
    for (int q = 1; q <= n; q++)
        if (!(std::fabs(a[q] - a[1]) <= 1e-6 * a[1]) || !(std::fabs(b[q] - a[1]) <= 1e-6 * a[1]))
            return false;
    return a[1] > 0.0;
}

// ratio of the largest eigenvalue to the smallest of the horizontal modes, or
// of the mean mode's vertical coefficients (its smallest from the column's
// height in units of the local spacing: (pi / sum of 1 / sqrt(a))^2)
double condition(const Dims& d, double ax, double ay, const std::vector<double>& au,
                 const std::vector<double>& ad) {
    double v = 0.0, height = 0.0;
    for (int k = 1; k <= d.kp; k++) {
        v = std::max(v, 2.0 * (au[k] + ad[k]));
        height += 1.0 / std::sqrt(std::sqrt(au[k] * ad[k]));
    }
    const double pi = 0.5 * kTwoPi;
    const double sx = std::sin(pi / d.ip), sy = std::sin(pi / d.jp);
    double low = HUGE_VAL;
    if (d.ip > 1) low = std::min(low, 4.0 * ax * sx * sx);
    if (d.jp > 1) low = std::min(low, 4.0 * ay * sy * sy);
    const double top = (d.ip > 1 ? 4.0 * ax : 0.0) + (d.jp > 1 ? 4.0 * ay : 0.0) + v;
    return std::max(top / low, v * (height / pi) * (height / pi));
}

// sequences per tile: 16 (128-byte segments) while two buffers of a line
// leave room for three blocks per SM, else 8
int tile_pairs(int n) { return n <= 288 ? 16 : 8; }
// shared memory of a block: a buffer between two passes, two buffers for three
// passes or more; a first pass of a large radix reads a buffer too
size_t fft_smem(int n, int nrad, int first) {
    const int meetings = nrad - 1 + (first > 16 ? 1 : 0);
    return (size_t)(meetings > 1 ? 2 : 1) * n * tile_pairs(n) * sizeof(float2);
}

}  // namespace

int direct_plan_build(const Dims& d, const std::vector<double>& ae, const std::vector<double>& aw,
                      const std::vector<double>& an, const std::vector<double>& as,
                      const std::vector<double>& au, const std::vector<double>& ad,
                      DirectPlan* plan) {
    DirectPlan& P = *plan;
    P.ok = false;
    const int n[2] = {d.ip, d.jp};
    // the rule: see DIRECT_MIN_POINTS; the longest line and column fit the
    // kernels; the horizontal spacings are uniform
    const long long points = (long long)d.ip * d.jp * d.kp;
    if (points < DIRECT_MIN_POINTS || points > DIRECT_MAX_POINTS || d.kp > 32 * 16 ||
        !uniform(ae, aw, d.ip) || !uniform(an, as, d.jp))
        return DCM_OK;
    for (int q = 0; q < 2; q++) {
        const std::vector<int> r = radices(n[q]);
        if (fft_smem(n[q], (int)r.size(), r.empty() ? 0 : r[0]) > DIRECT_MAX_SMEM) return DCM_OK;
    }
    for (int k = 1; k <= d.kp; k++)
        if (!(au[k] > 0.0 && ad[k] > 0.0)) return DCM_OK;
    const double noise = std::ldexp(condition(d, ae[1], an[1], au, ad), -24);
    if (!(noise <= DIRECT_MOST)) return DCM_OK;
    P.keep = noise > DIRECT_SURE;
    // one block: per axis n roots (float2) and n eigenvalues, then the mean
    // mode's tables (kp + 2 doubles each)
    std::vector<float> f;
    size_t off_tw[2], off_lam[2];
    for (int q = 0; q < 2; q++) {
        const double a = q == 0 ? ae[1] : an[1];
        const std::vector<int> r = radices(n[q]);
        if (r.size() > DIRECT_MAX_RADICES) return DCM_OK;
        AxisPlan& X = P.axis[q];
        X.n = n[q];
        X.nrad = (int)r.size();
        for (size_t e = 0; e < r.size(); e++) X.rad[e] = r[e];
        off_tw[q] = f.size();
        for (int m = 0; m < n[q]; m++) {
            f.push_back((float)std::cos(kTwoPi * m / n[q]));
            f.push_back((float)std::sin(kTwoPi * m / n[q]));
        }
        off_lam[q] = f.size();
        for (int m = 0; m < n[q]; m++) {
            const double s = std::sin(0.5 * kTwoPi * m / n[q]);
            f.push_back((float)(-4.0 * a * s * s));
        }
        if (f.size() % 2) f.push_back(0.0f);
    }
    const size_t K2 = d.kp + 2;
    std::vector<double> z(3 * K2, 0.0);
    double w = 1.0, sum = 0.0;
    for (int k = 1; k <= d.kp; k++) {
        z[k] = w;
        z[K2 + k] = 1.0 / (w * au[k]);
        const double ap = 2.0 * (ae[1] + an[1]) + au[k] + ad[k];
        z[2 * K2 + k] = w * ap;
        sum += w * ap;
        if (k < d.kp) w *= au[k] / ad[k + 1];  // w a symmetric: w_k au_k = w_k+1 ad_k+1
    }
    for (int k = 1; k <= d.kp; k++) z[2 * K2 + k] /= sum;
    const size_t fb = f.size() * sizeof(float), zb = z.size() * sizeof(double);
    char* dev = nullptr;
    if (cudaMalloc(&dev, fb + zb) != cudaSuccess) return DCM_E_CUDA;
    P.block = dev;
    if (cudaMemcpy(dev, f.data(), fb, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(dev + fb, z.data(), zb, cudaMemcpyHostToDevice) != cudaSuccess)
        return DCM_E_CUDA;
    for (int q = 0; q < 2; q++) {
        P.axis[q].tw = reinterpret_cast<const float2*>(dev + off_tw[q] * sizeof(float));
        P.axis[q].lam = reinterpret_cast<const float*>(dev + off_lam[q] * sizeof(float));
    }
    P.w = reinterpret_cast<const double*>(dev + fb);
    P.g = P.w + K2;
    P.l = P.g + K2;
    P.ok = true;
    return DCM_OK;
}

void direct_init() {
    const int sm = (int)DIRECT_MAX_SMEM;
    auto set = [&](auto kern) {
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    };
    set(k_fft<16, FFT_REAL>);
    set(k_fft<16, FFT_FWD>);
    set(k_fft<16, FFT_INV>);
    set(k_fft<16, FFT_ADD>);
    set(k_fft<8, FFT_REAL>);
    set(k_fft<8, FFT_FWD>);
    set(k_fft<8, FFT_INV>);
    set(k_fft<8, FFT_ADD>);
}

// the transform along axis 0 (x) or 1 (y) (x: the field that FFT_ADD adds to)
static void fft(const DirectPlan& P, const Dims& d, int axis, FftMode mode, const float* src,
                float* dst, double* x, cudaStream_t st) {
    const AxisPlan& X = P.axis[axis];
    FftArgs a;
    a.n = X.n;
    a.nrad = X.nrad;
    std::copy(X.rad, X.rad + DIRECT_MAX_RADICES, a.rad);
    a.tw = X.tw;
    a.line = axis == 0 ? d.K * d.J : d.K;
    a.batch = axis == 0 ? d.K : d.K * d.J;
    a.kp = d.kp;
    a.base = d.at(0, 1, 1);
    const int C = tile_pairs(X.n);
    const dim3 g(((d.kp + 1) / 2 + C - 1) / C, axis == 0 ? d.jp : d.ip);
    const size_t sm = fft_smem(X.n, X.nrad, X.rad[0]);
    ProfScope ps(P_JACOBI, st);
    auto go = [&](auto kern) { kern<<<g, FFT_THREADS, sm, st>>>(a, src, dst, x); };
    switch (mode) {
        case FFT_REAL: C == 16 ? go(k_fft<16, FFT_REAL>) : go(k_fft<8, FFT_REAL>); break;
        case FFT_FWD: C == 16 ? go(k_fft<16, FFT_FWD>) : go(k_fft<8, FFT_FWD>); break;
        case FFT_INV: C == 16 ? go(k_fft<16, FFT_INV>) : go(k_fft<8, FFT_INV>); break;
        case FFT_ADD: C == 16 ? go(k_fft<16, FFT_ADD>) : go(k_fft<8, FFT_ADD>); break;
    }
}

void direct_correction(const DirectPlan& P, const Dims& d, const Coef<float>& c, const float* r,
                       float* work, double* x, cudaStream_t st) {
    fft(P, d, 1, FFT_REAL, r, work, nullptr, st);
    if (d.ip > 1) fft(P, d, 0, FFT_FWD, work, work, nullptr, st);
    {
        ZArgs z;
        z.d = d;
        z.au = c.au;
        z.ad = c.ad;
        z.lx = P.axis[0].lam;
        z.ly = P.axis[1].lam;
        z.w = P.w;
        z.g = P.g;
        z.l = P.l;
        z.scale = (float)(1.0 / ((double)d.ip * d.jp));
        const int nb = ((d.ip / 2 + 1) * d.jp + 7) / 8;
        const int g = std::min(nb, 148 * 16);
        ProfScope ps(P_JACOBI, st);
        if (d.kp <= 64)
            k_zsolve<2><<<g, 256, 0, st>>>(z, work);
        else if (d.kp <= 128)
            k_zsolve<4><<<g, 256, 0, st>>>(z, work);
        else if (d.kp <= 256)
            k_zsolve<8><<<g, 256, 0, st>>>(z, work);
        else
            k_zsolve<16><<<g, 256, 0, st>>>(z, work);
    }
    if (d.ip > 1) fft(P, d, 0, FFT_INV, work, work, nullptr, st);
    fft(P, d, 1, FFT_ADD, work, nullptr, x, st);
}

void direct_put_back(const Dims& d, const double* keep, double* x, cudaStream_t st) {
    ProfScope ps(P_OTHER, st);
    k_dir_put_back<<<interior_grid(d, d.kp), dim3(BX, BY), 0, st>>>(d, keep, x);
}

void direct_residual(const Dims& d, const Coef<double>& c, const double* x, const double* b,
                     double* keep, float* r, double tol, int itmax, int max_rounds, bool first, const Red2& red,
                     int max_blocks, SolverScalars* S, const cudaGraphConditionalHandle* cond,
                     cudaStream_t st) {
    DirResidualArgs a;
    a.d = d;
    a.c = c;
    a.x = x;
    a.b = b;
    a.keep = first ? keep : nullptr;
    a.r = r;
    a.tol = tol;
    a.itmax = itmax;
    a.max_rounds = max_rounds;
    a.cond = cond ? *cond : 0;
    a.use_cond = cond ? 1 : 0;
    dim3 g((d.kp + 63) / 64, (d.jp + BY - 1) / BY, 1);
    // at most four blocks per SM (all resident), each marching over at least 4
    // planes
    const int plane = g.x * g.y;
    int want = std::max(1, std::min((d.ip + 3) / 4, 148 * 4 / plane));
    want = std::max(1, std::min(want, max_blocks / plane));
    a.ni = (d.ip + want - 1) / want;
    g.z = (d.ip + a.ni - 1) / a.ni;
    ProfScope ps(P_SETUP, st);
    if (first)
        k_dir_residual<true><<<g, dim3(BX, BY), 0, st>>>(a, red, S);
    else
        k_dir_residual<false><<<g, dim3(BX, BY), 0, st>>>(a, red, S);
}

}  // namespace dcm
