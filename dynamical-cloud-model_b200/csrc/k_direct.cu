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
// on with the BiCGSTAB iterations from there.
//
// Kernels per correction, each one pass in and one pass out of one FP32 field:
//   k_fht      transform along y (r -> scratch)
//   k_fht      transform along x (in place)
//   k_zsolve   tridiagonal system of every mode's column (in place)
//   k_fht      transform along x (in place)
//   k_fht      transform along y, x += result (FP64)
//   k_dir_residual   r = b - A x, its norm, convergence and loop condition
//
// The transform is the discrete Hartley transform, sum a_j cas(2 pi m j / n):
// real to real, its own inverse up to 1/n, and its basis vectors are
// eigenvectors of a symmetric circulant, so a mode is one real number and a
// field keeps its layout.  Two consecutive levels of a column make one
// complex sequence, whose complex FFT Z gives both Hartley transforms
// (Bracewell 1984):  H(m) = Re A - Im A with A = (Z(m) + conj Z(-m)) / 2.
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

// One Stockham pass of radix R over the C sequences of a tile (sequence c,
// element m at [m C + c]): rows r0, r0 + rg, ... of butterflies per thread.
template <int R, int C, bool FIRST, typename L>
__device__ __forceinline__ void fft_pass(int n, int ns, const float2* __restrict__ tw, L load,
                                         float2* __restrict__ dst, int c, int r0, int rg) {
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
        const int o = (b - kk) * R + kk;
#pragma unroll
        for (int t = 0; t < R; t++) dst[(o + t * ns) * C + c] = v[t];
    }
}

// a pass of any radix p (a prime factor above 13): each output is a sum of p
// products
template <int C>
__device__ __forceinline__ void fft_pass_any(int p, int n, int ns,
                                             const float2* __restrict__ tw,
                                             const float2* __restrict__ src,
                                             float2* __restrict__ dst, int c, int r0, int rg) {
    const int nb = n / p;
    for (int o = r0; o < n; o += rg) {
        const int s = o / nb, b = o - s * nb, kk = b % ns;
        const int q1 = (kk + s * ns) * (n / (ns * p));  // < n
        float2 acc = make_float2(0.0f, 0.0f);
        int q = 0;
        for (int t = 0; t < p; t++) {
            const float2 x = src[(b + t * nb) * C + c], w = __ldg(tw + q);
            acc.x += x.x * w.x + x.y * w.y;
            acc.y += x.y * w.x - x.x * w.y;
            q += q1;
            if (q >= n) q -= n;
        }
        dst[((b - kk) * p + kk + s * ns) * C + c] = acc;
    }
}

template <int C, bool FIRST, typename L>
__device__ __forceinline__ void fft_pass_of(int radix, int n, int ns,
                                            const float2* __restrict__ tw, L load,
                                            float2* __restrict__ dst, int c, int r0, int rg) {
    switch (radix) {
#define DCM_PASS(R)                                                   \
    case R:                                                           \
        fft_pass<R, C, FIRST>(n, ns, tw, load, dst, c, r0, rg);       \
        break;
        DCM_PASS(2) DCM_PASS(3) DCM_PASS(4) DCM_PASS(5) DCM_PASS(6) DCM_PASS(7) DCM_PASS(8)
        DCM_PASS(9) DCM_PASS(10) DCM_PASS(11) DCM_PASS(12) DCM_PASS(13) DCM_PASS(14)
        DCM_PASS(15) DCM_PASS(16)
#undef DCM_PASS
        default: break;
    }
}

// ---- Hartley transform along one horizontal axis --------------------------------
// A block transforms C pairs of levels (2 C consecutive levels) of one row or
// column of the domain; every element of the tile is one C x 8 byte segment of
// memory.  The first pass reads memory, the others go through two buffers in
// shared memory.  OUT = 0: to dst; OUT = 1: x (FP64) += the transform (an
// element that is not finite is left out, so that x stays usable).
constexpr int FHT_THREADS = 256;

struct FhtArgs {
    int n, nrad;
    int rad[DIRECT_MAX_RADICES];
    const float2* tw;  // n roots (cos, sin)(2 pi q / n)
    int line, batch;   // element strides along the axis and across rows
    int kp, base;      // levels; index of (k, j, i) = (0, 1, 1)
};

template <int C, int OUT>
__global__ void __launch_bounds__(FHT_THREADS) k_fht(FhtArgs a, const float* src, float* dst,
                                                     double* __restrict__ x) {
    extern __shared__ float2 fht_buf[];
    const int n = a.n, c = threadIdx.x % C, r0 = threadIdx.x / C;
    constexpr int RG = FHT_THREADS / C;
    float2* cur = fht_buf;
    float2* nxt = fht_buf + n * C;
    const int k0 = 1 + 2 * ((int)blockIdx.x * C + c);
    const bool one = k0 <= a.kp, both = k0 < a.kp;
    const int o0 = a.base + (int)blockIdx.y * a.batch + k0;
    auto global = [&](int m) -> float2 {
        const float* p = src + o0 + m * a.line;
        if (both) return *reinterpret_cast<const float2*>(p);
        return make_float2(one ? *p : 0.0f, 0.0f);
    };
    int ns = 1, q = 0;
    if (a.nrad > 0 && a.rad[0] <= 16) {
        fft_pass_of<C, true>(a.rad[0], n, 1, a.tw, global, cur, c, r0, RG);
        ns = a.rad[0];
        q = 1;
    } else {
        for (int m = r0; m < n; m += RG) cur[m * C + c] = global(m);
    }
    __syncthreads();
    for (; q < a.nrad; q++) {
        const int r = a.rad[q];
        const float2* s = cur;
        if (r <= 16)
            fft_pass_of<C, false>(r, n, ns, a.tw, [&](int m) { return s[m * C + c]; }, nxt, c, r0,
                                  RG);
        else
            fft_pass_any<C>(r, n, ns, a.tw, s, nxt, c, r0, RG);
        ns *= r;
        float2* t = cur;
        cur = nxt;
        nxt = t;
        __syncthreads();
    }
    auto put = [&](int m, float h0, float h1) {
        const int o = o0 + m * a.line;
        if (OUT == 0) {
            if (both)
                *reinterpret_cast<float2*>(dst + o) = make_float2(h0, h1);
            else if (one)
                dst[o] = h0;
        } else {
            if (!(fabsf(h0) <= FLT_MAX)) h0 = 0.0f;
            if (!(fabsf(h1) <= FLT_MAX)) h1 = 0.0f;
            if (both) {
                double2 v = *reinterpret_cast<const double2*>(x + o);
                v.x += (double)h0;
                v.y += (double)h1;
                *reinterpret_cast<double2*>(x + o) = v;
            } else if (one) {
                x[o] += (double)h0;
            }
        }
    };
    for (int m = r0; 2 * m <= n; m += RG) {
        const int m2 = m ? n - m : 0;
        const float2 z = cur[m * C + c], y = cur[m2 * C + c];
        const float sx = 0.5f * (z.x + y.x), dx = 0.5f * (z.x - y.x);
        const float sy = 0.5f * (z.y + y.y), dy = 0.5f * (z.y - y.y);
        put(m, sx - dy, sy + dx);
        if (m2 != m) put(m2, sx + dy, sy - dx);
    }
}

// ---- the tridiagonal systems along z ----------------------------------------------
// One warp per column, V consecutive levels per lane.  Each lane eliminates
// its inner levels (the partition method), the last level of every lane then
// forms a 32-row tridiagonal system that cyclic reduction over the lanes
// solves in five shuffle steps, and the inner levels follow by substitution.
// A thread per column (the Thomas recurrence) would be a chain of 2 kp
// dependent steps.  The horizontal mean mode is singular (Neumann at both
// ends): it is integrated twice in FP64, with the additive constant that
// leaves the sum of a_p dz-weighted values unchanged, which is the constant
// Jacobi-preconditioned iterations leave unchanged too.
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

template <int V>
__global__ void __launch_bounds__(256) k_zsolve(ZArgs a, float* __restrict__ f) {
    constexpr unsigned FULL = 0xffffffffu;
    const Dims& d = a.d;
    const int lane = threadIdx.x & 31, kp = d.kp;
    const int k0 = 1 + V * lane;
    const int nvalid = max(0, min(V, kp - k0 + 1));
    float au[V], ad[V], b0[V];
#pragma unroll
    for (int e = 0; e < V; e++) {
        const int k = k0 + e;
        au[e] = k < kp ? ld(a.au + k) : 0.0f;
        ad[e] = k > 1 && k <= kp ? ld(a.ad + k) : 0.0f;
        b0[e] = -au[e] - ad[e];
    }
    const int ncol = d.ip * d.jp, nw = gridDim.x * 8;
    for (int col = blockIdx.x * 8 + (threadIdx.x >> 5); col < ncol; col += nw) {
        const int i = col / d.jp, j = col - i * d.jp;
        float* __restrict__ p = f + d.at(k0, 1 + j, 1 + i);
        float D[V];
        zload<V>(p, nvalid, D);
#pragma unroll
        for (int e = 0; e < V; e++) D[e] *= a.scale;
        if (col == 0) {  // the whole warp
            double q[V], s = 0.0;
#pragma unroll
            for (int e = 0; e < V; e++) {
                if (e < nvalid) s += a.w[k0 + e] * (double)D[e];
                q[e] = s;
            }
            double before = warp_scan(s) - s, t = 0.0;
#pragma unroll
            for (int e = 0; e < V; e++) {
                const double step = k0 + e < kp ? (q[e] + before) * a.g[k0 + e] : 0.0;
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
            for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(FULL, m, o);
#pragma unroll
            for (int e = 0; e < V; e++) D[e] = (float)(q[e] - m);
            zstore<V>(p, nvalid, D);
            continue;
        }
        const float lam = ld(a.lx + i) + ld(a.ly + j);
        float A[V], C[V];
        // rows beyond kp: u = 0
#pragma unroll
        for (int e = 0; e < V; e++) {
            const float b = e < nvalid ? lam + b0[e] : 1.0f;
            if (e < 2) {
                const float r = __fdividef(1.0f, b);
                D[e] *= r;
                A[e] = ad[e] * r;
                C[e] = au[e] * r;
            } else {
                const float r = __fdividef(1.0f, b - ad[e] * C[e - 1]);
                D[e] = r * (D[e] - ad[e] * D[e - 1]);
                A[e] = -r * ad[e] * A[e - 1];
                C[e] = r * au[e];
            }
        }
#pragma unroll
        for (int e = V - 3; e >= 1; e--) {
            D[e] -= C[e] * D[e + 1];
            A[e] -= C[e] * A[e + 1];
            C[e] = -C[e] * C[e + 1];
        }
        if (V > 2) {
            const float r = __fdividef(1.0f, 1.0f - C[0] * A[1]);
            D[0] = r * (D[0] - C[0] * D[1]);
            A[0] = r * A[0];
            C[0] = -r * C[0] * C[1];
        }
        // the last levels: first levels of this lane and the next eliminated
        const float dn = __shfl_down_sync(FULL, D[0], 1), an = __shfl_down_sync(FULL, A[0], 1),
                    cn = __shfl_down_sync(FULL, C[0], 1);
        const float al = A[V - 1], cl = C[V - 1];
        float r = __fdividef(1.0f, 1.0f - al * C[0] - cl * an);
        float x = r * (D[V - 1] - al * D[0] - cl * dn);
        float lo = -r * al * A[0], up = -r * cl * cn;
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
            // lo is 0 in the first s lanes and up in the last s, so what the
            // shuffles return there does not count
            const float xm = __shfl_up_sync(FULL, x, s), lm = __shfl_up_sync(FULL, lo, s),
                        um = __shfl_up_sync(FULL, up, s);
            const float xp = __shfl_down_sync(FULL, x, s), lp = __shfl_down_sync(FULL, lo, s),
                        upp = __shfl_down_sync(FULL, up, s);
            r = __fdividef(1.0f, 1.0f - lo * um - up * lp);
            x = r * (x - lo * xm - up * xp);
            lo = -r * lo * lm;
            up = -r * up * upp;
        }
        float prev = __shfl_up_sync(FULL, x, 1);
        if (lane == 0) prev = 0.0f;
        const float u0 = D[0] - A[0] * prev - C[0] * x;
        D[0] = u0;
#pragma unroll
        for (int e = 1; e < V - 1; e++) D[e] = D[e] - A[e] * u0 - C[e] * x;
        D[V - 1] = x;
        zstore<V>(p, nvalid, D);
    }
}

// ---- FP64 residual of the pressure, and the loop's decision -------------------------
// r = b - A x in FP64 (mat_ax, dynamics.f90:219-222), stored in FP32, with
// ||r|| and, at the start of a solve, ||b||.  A warp holds 64 levels (one
// 16-byte vector per lane) of one row and marches along i with the i - 1, i
// and i + 1 columns in registers; the next plane's loads are issued before
// this plane's arithmetic.
struct DirResidualArgs {
    Dims d;
    Coef<double> c;
    const double *x, *b;
    float* r;
    double tol;
    int itmax, max_rounds;
    int ni;  // planes per block
    cudaGraphConditionalHandle cond;
    int use_cond;
};

template <bool FIRST>
__global__ void __launch_bounds__(256) k_dir_residual(DirResidualArgs a, Red2 R,
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
        double2 xw = at(x + KJ * (i0 == 1 ? ip : i0 - 1)), xc = at(x + KJ * i0),
                xe = at(x + KJ * (i0 == ip ? 1 : i0 + 1)), xs = at(x + KJ * i0 + ds),
                xn = at(x + KJ * i0 + dn), bv = at(bb + KJ * i0);
        for (int i = i0; i <= i1; i++) {
            const int o = KJ * i;
            double prev = __shfl_up_sync(0xffffffffu, xc.y, 1);
            double next = __shfl_down_sync(0xffffffffu, xc.x, 1);
            if (lane == 0 && live && k0 > 1) prev = x[o - 1];
            if (lane == 31 && k0 + 2 <= kp) next = x[o + 2];
            double2 xe2, xs2, xn2, b2;
            if (i < i1) {
                xe2 = at(x + KJ * (i + 1 == ip ? 1 : i + 2));
                xs2 = at(x + o + KJ + ds);
                xn2 = at(x + o + KJ + dn);
                b2 = at(bb + o + KJ);
            }
            const double ae = ld(a.c.ae + i), aw = ld(a.c.aw + i);
            const double sij = -ae - aw - an - as;
            if (k0 == 1) prev = xc.x;  // Neumann rows, :206-211
            const double up0 = k0 == kp ? xc.x : xc.y;
            if (k0 + 1 == kp) next = xc.y;
            const double r0 = bv.x - (aw * xw.x + ae * xe.x + as * xs.x + an * xn.x + ad0 * prev +
                                      au0 * up0 + (sij - au0 - ad0) * xc.x);
            const double r1 = bv.y - (aw * xw.y + ae * xe.y + as * xs.y + an * xn.y + ad1 * xc.x +
                                      au1 * next + (sij - au1 - ad1) * xc.y);
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
            if (i < i1) {
                xe = xe2;
                xs = xs2;
                xn = xn2;
                bv = b2;
            }
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
    } else if (FIRST || err <= DIRECT_CONTRACTION * S->err) {
        // another correction, within the limits of the iterations
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

// sequences per tile: 16 (128-byte segments) while two buffers of a line
// leave room for three blocks per SM, else 8
int tile_pairs(int n) { return n <= 288 ? 16 : 8; }
size_t fht_smem(int n) { return (size_t)2 * n * tile_pairs(n) * sizeof(float2); }

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
    for (int q = 0; q < 2; q++)
        if (fht_smem(n[q]) > DIRECT_MAX_SMEM) return DCM_OK;
    for (int k = 1; k <= d.kp; k++)
        if (!(au[k] > 0.0 && ad[k] > 0.0)) return DCM_OK;
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
    cudaFuncSetAttribute(k_fht<16, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    cudaFuncSetAttribute(k_fht<16, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    cudaFuncSetAttribute(k_fht<8, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    cudaFuncSetAttribute(k_fht<8, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
}

// the transform along axis 0 (x) or 1 (y); x non-null: added to it
static void fht(const DirectPlan& P, const Dims& d, int axis, const float* src, float* dst,
                double* x, cudaStream_t st) {
    const AxisPlan& X = P.axis[axis];
    FhtArgs a;
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
    const size_t sm = fht_smem(X.n);
    ProfScope ps(P_JACOBI, st);
    if (C == 16)
        x ? k_fht<16, 1><<<g, FHT_THREADS, sm, st>>>(a, src, dst, x)
          : k_fht<16, 0><<<g, FHT_THREADS, sm, st>>>(a, src, dst, x);
    else
        x ? k_fht<8, 1><<<g, FHT_THREADS, sm, st>>>(a, src, dst, x)
          : k_fht<8, 0><<<g, FHT_THREADS, sm, st>>>(a, src, dst, x);
}

void direct_correction(const DirectPlan& P, const Dims& d, const Coef<float>& c, const float* r,
                       float* work, double* x, cudaStream_t st) {
    fht(P, d, 1, r, work, nullptr, st);
    if (d.ip > 1) fht(P, d, 0, work, work, nullptr, st);
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
        const int nb = (d.ip * d.jp + 7) / 8;
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
    if (d.ip > 1) fht(P, d, 0, work, work, nullptr, st);
    fht(P, d, 1, work, nullptr, x, st);
}

void direct_residual(const Dims& d, const Coef<double>& c, const double* x, const double* b,
                     float* r, double tol, int itmax, int max_rounds, bool first, const Red2& red,
                     int max_blocks, SolverScalars* S, const cudaGraphConditionalHandle* cond,
                     cudaStream_t st) {
    DirResidualArgs a;
    a.d = d;
    a.c = c;
    a.x = x;
    a.b = b;
    a.r = r;
    a.tol = tol;
    a.itmax = itmax;
    a.max_rounds = max_rounds;
    a.cond = cond ? *cond : 0;
    a.use_cond = cond ? 1 : 0;
    dim3 g((d.kp + 63) / 64, (d.jp + BY - 1) / BY, 1);
    // about four blocks per SM, each marching over at least 4 planes
    const int plane = g.x * g.y;
    int want = std::max(1, std::min((d.ip + 3) / 4, (148 * 4 + plane - 1) / plane));
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
