// Eigenpairs 1..iu of the real symmetric tridiagonal T (d, e) and back-transformation
// X = Q Z, batched over k.
//
// zheevr with RANGE='I' and IU < N (LapackRoutines.f90:414-426) computes the
// eigenvalues by bisection (dstebz) and the vectors by inverse iteration (zstein);
// this file restates that route for the GPU:
//   k_gersh     : Gershgorin interval, 1-norm and pivmin per matrix;
//   k_bisect*   : eigenvalues by Sturm counts, an FP32 bracket and FP64 multisection;
//   k_clusters  : groups consecutive eigenvalues closer than ortol;
//   k_invit     : one thread per cluster: LU of T - lambda I with partial pivoting
//                 (dlagtf), perturbed back-substitution (dlagts, job=-1), modified
//                 Gram-Schmidt against the earlier members of the cluster;
//   back-transform: Q applied in compact-WY blocks (zlarft forward/columnwise) on the tensor
//                 cores (oz_fp64.cu; eig_mixed.cu for the mixed path).
// ortol is tighter than zstein's 1e-3*||T||_1 (which groups a whole dense spectrum
// into one serial cluster); with ortol = 1e-7*||T||_1 the vector error bound
// eps*||T||/gap stays below 1e-8 outside clusters.
#include <algorithm>
#include <cfloat>
#include "cvec.cuh"
#include "eig.cuh"

namespace forge {

constexpr double kEps = 1.1102230246251565e-16;    // dlamch('E')
constexpr double kSafmin = 2.2250738585072014e-308; // dlamch('S')

__global__ void k_gersh(const double* __restrict__ d, const double* __restrict__ e, int64_t n, double* __restrict__ info) {
    // one CTA (256 threads) per matrix; info[b*8 + 0..4] = gl, gu, onenrm, pivmin, tnorm
    const int64_t b = blockIdx.x;
    const double* D = d + b * n;
    const double* E = e + b * n;
    double gl = 1e300, gu = -1e300, nrm = 0.0, emax = 0.0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        double em = (i > 0) ? fabs(E[i - 1]) : 0.0;
        double ep = (i < n - 1) ? fabs(E[i]) : 0.0;
        gl = fmin(gl, D[i] - em - ep);
        gu = fmax(gu, D[i] + em + ep);
        nrm = fmax(nrm, fabs(D[i]) + em + ep);
        if (i < n - 1) emax = fmax(emax, E[i] * E[i]);
    }
    __shared__ double s[4][256];
    s[0][threadIdx.x] = gl;
    s[1][threadIdx.x] = gu;
    s[2][threadIdx.x] = nrm;
    s[3][threadIdx.x] = emax;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            s[0][threadIdx.x] = fmin(s[0][threadIdx.x], s[0][threadIdx.x + o]);
            s[1][threadIdx.x] = fmax(s[1][threadIdx.x], s[1][threadIdx.x + o]);
            s[2][threadIdx.x] = fmax(s[2][threadIdx.x], s[2][threadIdx.x + o]);
            s[3][threadIdx.x] = fmax(s[3][threadIdx.x], s[3][threadIdx.x + o]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        double pivmin = kSafmin * fmax(1.0, s[3][0]);
        double tnorm = fmax(fabs(s[0][0]), fabs(s[1][0]));
        const double fudge = 2.1, ulp = 2.0 * kEps;
        double g0 = s[0][0] - fudge * tnorm * ulp * n - fudge * 2.0 * pivmin;
        double g1 = s[1][0] + fudge * tnorm * ulp * n + fudge * 2.0 * pivmin;
        info[b * 8 + 0] = g0;
        info[b * 8 + 1] = g1;
        info[b * 8 + 2] = s[2][0];
        info[b * 8 + 3] = pivmin;
        info[b * 8 + 4] = tnorm;
    }
}

// T scaled by a power of two to |T| <= 1 for the Sturm counts: de[b][i] = (d_i, e_{i-1}^2), tf[b][i] = de
// rounded to FP32.
__device__ inline double tri_scale(const double* info) {
    // 2^-k with 2^k > max |Gershgorin bound| (both bounds are finite; k = 0 for a zero matrix)
    const double m = fmax(fabs(info[0]), fabs(info[1]));
    int k = 0;
    if (m > 0.0) frexp(m, &k);
    return ldexp(1.0, -k);
}
__global__ void k_tri_scale(const double* __restrict__ d, const double* __restrict__ e, int64_t n,
                            const double* __restrict__ info, double2* __restrict__ de, float2* __restrict__ tf) {
    const int64_t b = blockIdx.y;
    const double s = tri_scale(info + b * 8);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double di = d[b * n + i] * s, em = (i > 0) ? e[b * n + i - 1] * s : 0.0;
        de[b * n + i] = make_double2(di, em * em);
        tf[b * n + i] = make_float2((float)di, (float)(em * em));
    }
}

// Leading principal minors p_i of T - x I (Givens' recurrence; its rounding errors are those of a
// matrix with relatively perturbed d_i - x and e_i^2, as for the quotients p_i / p_{i-1}):
//   p_i = (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2}.
// One dependent FMA a step, where the quotient form has a division: on this GPU an FP64 division is
// a chain of about a thousand clocks and fourteen FP64 pipe slots, the recurrence takes three.
// A minor below 2^-THR of its predecessor is replaced by -2^-THR of it (the quotient form's
// |q| < pivmin -> -pivmin), and every fourth step both are rescaled by a power of two, so nothing
// under- or overflows: |T - x I| <= 4 grows a minor by less than 2^8 in four steps, and four
// replacements shrink it by 2^-4 THR.  Sign and exponent are handled as integers.
template <class T>
struct Minor;
template <>
struct Minor<double> {
    static constexpr int THR = 160, MB = 20, BIAS = 1023;
    __device__ static int hi(double x) { return __double2hiint(x); }
    __device__ static double add_hi(double x, int dh) { return __hiloint2double(__double2hiint(x) + dh, __double2loint(x)); }
    __device__ static double neg(double x) { return __hiloint2double(__double2hiint(x) ^ 0x80000000, __double2loint(x)); }
};
template <>
struct Minor<float> {
    static constexpr int THR = 28, MB = 23, BIAS = 127;
    __device__ static int hi(float x) { return __float_as_int(x); }
    __device__ static float add_hi(float x, int dh) { return __int_as_float(__float_as_int(x) + dh); }
    __device__ static float neg(float x) { return __int_as_float(__float_as_int(x) ^ 0x80000000); }
};
template <class T>
__device__ __forceinline__ T minor_step(T t, T e2, T p1, T p0) {
    using M = Minor<T>;
    T pn = fma(t, p1, -(e2 * p0));
    const int hn = M::hi(pn) & 0x7fffffff, h1 = M::hi(p1) & 0x7fffffff;
    if (hn + (M::THR << M::MB) < h1) pn = M::neg(M::add_hi(p1, -(M::THR << M::MB)));
    return pn;
}
template <class T>
__device__ __forceinline__ void minor_rescale(T& p1, T& p0) {
    using M = Minor<T>;
    const int h = max(M::hi(p1) & 0x7fffffff, M::hi(p0) & 0x7fffffff);
    const int dh = (M::BIAS - (h >> M::MB)) << M::MB;
    p1 = M::add_hi(p1, dh);
    p0 = M::add_hi(p0, dh);
}
// number of eigenvalues <= x: sign changes of the minors
template <class T, class T2>
__device__ inline int sturm(const T2* __restrict__ de, int n, T x) {
    using M = Minor<T>;
    T p0 = (T)1, p1 = minor_step<T>((T)de[0].x - x, (T)0, (T)1, (T)0);
    int cnt = (int)((unsigned)M::hi(p1) >> 31);
    int i = 1;
    for (; i + 4 <= n; i += 4) {
        T2 v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = de[i + q];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const T pn = minor_step<T>(v[q].x - x, v[q].y, p1, p0);
            cnt += (int)((unsigned)(M::hi(pn) ^ M::hi(p1)) >> 31);
            p0 = p1;
            p1 = pn;
        }
        minor_rescale(p1, p0);
    }
    for (; i < n; ++i) {
        const T2 v = de[i];
        const T pn = minor_step<T>(v.x - x, v.y, p1, p0);
        cnt += (int)((unsigned)(M::hi(pn) ^ M::hi(p1)) >> 31);
        p0 = p1;
        p1 = pn;
    }
    return cnt;
}

// number of eigenpairs wanted of matrix b (a padded slot of a group wants its own nUpper)
__device__ inline int64_t want_of(const int* lim, int64_t b, int64_t iu) { return lim ? (int64_t)lim[b] : iu; }

// ---------------------------------------------------------------- quotient form (mixed precision)
// number of eigenvalues <= x (dlaebz Sturm count)
__device__ inline int sturm_q(const double* __restrict__ D, const double* __restrict__ E, int n, double x,
                              double pivmin) {
    double q = D[0] - x;
    if (fabs(q) < pivmin) q = -pivmin;
    int cnt = (q <= 0.0) ? 1 : 0;
#pragma unroll 4
    for (int i = 1; i < n; ++i) {
        const double e = E[i - 1];
        q = D[i] - e * e / q - x;
        if (fabs(q) < pivmin) q = -pivmin;
        cnt += (q <= 0.0) ? 1 : 0;
    }
    return cnt;
}
// Sturm count in FP32 (the count is exact for a tridiagonal within a few FP32 ulps of T)
__device__ inline int sturm_qf(const float* __restrict__ D, const float* __restrict__ E2, int n, float x,
                               float pivmin) {
    float q = D[0] - x;
    if (fabsf(q) < pivmin) q = -pivmin;
    int cnt = (q <= 0.f) ? 1 : 0;
#pragma unroll 4
    for (int i = 1; i < n; ++i) {
        q = (D[i] - x) - __fdividef(E2[i - 1], q);
        if (fabsf(q) < pivmin) q = -pivmin;
        cnt += (q <= 0.f) ? 1 : 0;
    }
    return cnt;
}
// FP32 copies of the unscaled tridiagonal: tq[b][0..n) = d, tq[b][n..2n) = e^2
__global__ void k_tri_to_f32(const double* __restrict__ d, const double* __restrict__ e, int64_t n,
                             float* __restrict__ tq) {
    const int64_t b = blockIdx.y;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        tq[b * 2 * n + i] = (float)d[b * n + i];
        const double ei = (i < n - 1) ? e[b * n + i] : 0.0;
        tq[b * 2 * n + n + i] = (float)(ei * ei);
    }
}
// FP32 bisection of eigenvalue j in the quotient form, into w.  As in k_bisect_replay, a midpoint further
// than 64 eps_32 |T| from the eigenvalue lam is decided without a count.
__global__ void __launch_bounds__(32) k_bisect_qf(const float* __restrict__ tq, int64_t n, int64_t iu,
                                                  const int* __restrict__ lim, const double* __restrict__ info,
                                                  const double* __restrict__ lam, double* __restrict__ w) {
    const int64_t b = blockIdx.y;
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= want_of(lim, b, iu)) return;
    const float* D = tq + b * 2 * n;
    const float* E2 = D + n;
    // Gershgorin bounds widened by the FP32 rounding of the counts
    const float tn = (float)info[b * 8 + 4];
    float lo = (float)info[b * 8 + 0] - 8.f * FLT_EPSILON * tn * 64.f, hi = (float)info[b * 8 + 1] + 8.f * FLT_EPSILON * tn * 64.f;
    const float pivmin = fmaxf(1e-30f, (float)info[b * 8 + 3]);
    const double l = lam[b * iu + j], far = 64.0 * (double)FLT_EPSILON * info[b * 8 + 4];
    for (int it = 0; it < 64; ++it) {
        const float width = hi - lo;
        if (width <= 2.f * FLT_EPSILON * fmaxf(fabsf(lo), fabsf(hi)) || width <= pivmin) break;
        const float mid = 0.5f * (lo + hi);
        if (mid <= lo || mid >= hi) break;
        const bool up = mid > l + far ? true : mid < l - far ? false : sturm_qf(D, E2, (int)n, mid, pivmin) >= j + 1;
        if (up)
            hi = mid;
        else
            lo = mid;
    }
    w[b * iu + j] = 0.5 * ((double)lo + (double)hi);
}
// The FP64 bisection of the mixed path, from the bracket x -/+ 8 eps_32 |T| of the FP32 estimate x when
// the counts confirm it.  Its midpoints form a fixed dyadic sequence, and the quotient-form count decides
// each: where a midpoint lies further from the eigenvalue that k_bisect found (lam) than 64 eps |T|,
// many times the error of either count, the decision is known without a count; only the last few
// are counted, several levels of the bisection tree at once (G lanes hold the 2^LEV - 1
// midpoints of LEV levels).  Why not k_bisect's own result: the mixed path rounds the eigenvectors to
// FP32 afterwards, and that rounding noise stays in the refined density matrix to second order
// (3e-9 of its norm at N = 1324), so a last-place change of an eigenvalue would change the results by
// as much; this keeps them bit for bit.  Bound: latency of the division chain, ~1300 clocks a step.
// Measured, stage total with k_bisect: N = 5044, all eigenvalues 138 -> 51 ms; N = 1876, 9 k 46 -> 26 ms.
template <int LEV>
__global__ void __launch_bounds__(32) k_bisect_replay(const double* __restrict__ d, const double* __restrict__ e,
                                                      int64_t n, int64_t iu, const int* __restrict__ lim,
                                                      const double* __restrict__ info, const double* __restrict__ lam,
                                                      double* __restrict__ w) {
    constexpr int G = LEV == 1 ? 1 : 1 << LEV;
    const int64_t b = blockIdx.y;
    const int64_t j = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
    const int g = threadIdx.x % G, base = (threadIdx.x & 31) / G * G;
    const unsigned full = 0xffffffffu;
    const bool live = j < want_of(lim, b, iu);
    const double* D = d + b * n;
    const double* E = e + b * n;
    double lo = info[b * 8 + 0], hi = info[b * 8 + 1];
    const double pivmin = info[b * 8 + 3], tnorm = info[b * 8 + 4];
    const double l = live ? lam[b * iu + j] : 0.0, far = 64.0 * kEps * tnorm;
    if (live) {
        const double x = w[b * iu + j], delta = 8.0 * (double)FLT_EPSILON * tnorm;
        const double l2 = fmax(lo, x - delta), h2 = fmin(hi, x + delta);
        if (l2 < h2) {
            const bool lok = l2 < l - far ? true : l2 > l + far ? false : sturm_q(D, E, (int)n, l2, pivmin) < j + 1;
            const bool hok = h2 > l + far ? true : h2 < l - far ? false : sturm_q(D, E, (int)n, h2, pivmin) >= j + 1;
            if (lok && hok) {
                lo = l2;
                hi = h2;
            }
        }
    }
    const double rtol = 4.0 * kEps;
    auto open = [&](double a, double c) {
        return c - a > fmax(fmax(kSafmin, pivmin), rtol * fmax(fabs(a), fabs(c)));
    };
    int it = 0;
    for (;;) {
        // decisions that need no count
        while (live && it < 256 && open(lo, hi)) {
            const double mid = 0.5 * (lo + hi);
            if (mid > l + far)
                hi = mid;
            else if (mid < l - far)
                lo = mid;
            else
                break;
            ++it;
        }
        const bool more = live && it < 256 && open(lo, hi);
        if (!__any_sync(full, more)) break;
        // lane g holds node g of the tree (1: root; children 2g, 2g + 1 = lower, upper half)
        double a = lo, c = hi;
        if (G > 1)
            for (int bit = 30 - __clz(g > 0 ? g : 1); bit >= 0; --bit) {
                const double mid = 0.5 * (a + c);
                if ((g >> bit) & 1)
                    a = mid;
                else
                    c = mid;
            }
        bool up = false;
        if (more && (G == 1 || g > 0)) up = sturm_q(D, E, (int)n, 0.5 * (a + c), pivmin) >= j + 1;
        const unsigned ups = __ballot_sync(full, up) >> base;
        if (more) {
            int node = G == 1 ? 0 : 1;
#pragma unroll
            for (int q = 0; q < LEV; ++q) {
                if (it < 256 && open(lo, hi)) {
                    const double mid = 0.5 * (lo + hi);
                    const bool u = (ups >> node) & 1u;
                    if (u)
                        hi = mid;
                    else
                        lo = mid;
                    node = 2 * node + (u ? 0 : 1);
                    ++it;
                }
            }
        }
    }
    if (g == 0 && j < iu) w[b * iu + j] = live ? 0.5 * (lo + hi) : 0.0;
}

// ---------------------------------------------------------------- multisection (minors)
// eigenvalue j of the scaled T by bisection to FP32 accuracy, into w (scaled)
__global__ void k_bisect_f32(const float2* __restrict__ tf, int64_t n, int64_t iu, const int* __restrict__ lim,
                             const double* __restrict__ info, double* __restrict__ w) {
    const int64_t b = blockIdx.y;
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= want_of(lim, b, iu)) return;
    const double s = tri_scale(info + b * 8);
    // Gershgorin bounds widened by the FP32 rounding of the counts
    float lo = (float)(info[b * 8 + 0] * s) - 512.f * FLT_EPSILON, hi = (float)(info[b * 8 + 1] * s) + 512.f * FLT_EPSILON;
    for (int it = 0; it < 64; ++it) {
        // the counts are good to a few FP32 ulps of |T| <= 1
        if (!(hi - lo > FLT_EPSILON)) break;
        const float mid = 0.5f * (lo + hi);
        if (mid <= lo || mid >= hi) break;
        if (sturm<float>(tf + b * n, (int)n, mid) >= j + 1)
            hi = mid;
        else
            lo = mid;
    }
    w[b * iu + j] = 0.5 * ((double)lo + (double)hi);
}

// Eigenvalue j in FP64 by multisection: G lanes evaluate the Sturm counts at G equally spaced points of
// the bracket, which shrinks by G + 1 a round.  The bracket starts from the FP32 estimate in w: it is
// widened by 16 until the FP64 counts confirm it, at last to the Gershgorin interval.  Stops at the
// reference's 4 eps |lambda|.  G (launch rule in tridiag_eigvecs): a round costs the latency of n
// dependent steps as long as the FP64 pipes are not full, so few eigenvalues take many lanes each.
// Bound: FP64 pipe (three slots a step) or, below ~19000 lanes, the latency of the chain.  Measured,
// FP64 stage total (quotient-form bisection by one lane before): N = 1324, 16 k 47.9 -> 6.4 ms;
// N = 3268, one k 111 -> 8.1 ms.
template <int G>
__global__ void __launch_bounds__(32) k_bisect(const double2* __restrict__ de, int64_t n, int64_t iu,
                                                const int* __restrict__ lim, const double* __restrict__ info,
                                                double* w) {
    const int64_t b = blockIdx.y;
    const int64_t j = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
    const int g = threadIdx.x % G;
    const bool live = j < want_of(lim, b, iu);
    const double2* t = de + b * n;
    const double s = tri_scale(info + b * 8);
    const double glo = info[b * 8 + 0] * s, ghi = info[b * 8 + 1] * s;
    double lo = glo, hi = ghi;
    const unsigned full = 0xffffffffu;
    const int base = (threadIdx.x & 31) / G * G;
    const unsigned gmask = (unsigned)(((1ull << G) - 1ull) << base);
    // confirm the FP32 bracket (lane 0 of the group: lower end, last lane: upper end; G = 1: both)
    {
        const double x = live ? w[b * iu + j] : 0.0;
        double delta = 8.0 * (double)FLT_EPSILON;
        bool ok = !live;
        for (int tries = 0; tries < 3; ++tries) {
            const double l2 = fmax(glo, x - delta), h2 = fmin(ghi, x + delta);
            bool lok = true, hok = true;
            if (!ok) {
                if (g == 0) lok = sturm<double>(t, (int)n, l2) < j + 1;
                if (g == G - 1) hok = sturm<double>(t, (int)n, h2) >= j + 1;
            }
            const unsigned bad = __ballot_sync(full, !(lok && hok));
            if (!ok && (bad & gmask) == 0 && l2 < h2) {
                lo = l2;
                hi = h2;
                ok = true;
            }
            if (__all_sync(full, ok)) break;
            delta *= 16.0;
        }
    }
    const double rtol = 4.0 * kEps;
    for (int it = 0; it < 256; ++it) {
        const double width = hi - lo;
        const double tol = fmax(8.636168555094445e-78, rtol * fmax(fabs(lo), fabs(hi)));   // >= 2^-256
        const bool open = live && width > tol;
        if (!__any_sync(full, open)) break;
        const double x = lo + width * ((double)(g + 1) / (double)(G + 1));
        bool up = true;
        if (open) up = sturm<double>(t, (int)n, x) >= j + 1;
        const unsigned ups = (__ballot_sync(full, up) & gmask) >> base;
        // first point at or above eigenvalue j (the points of a closed bracket are not used)
        const int f = ups ? __ffs(ups) - 1 : G;
        const double xf = __shfl_sync(full, x, base + (f < G ? f : G - 1));
        const double xp = __shfl_sync(full, x, base + (f > 0 ? f - 1 : 0));
        if (open) {
            if (f < G) hi = fmin(hi, xf);
            if (f > 0) lo = fmax(lo, xp);
            // no representable point inside the bracket
            if (!(hi - lo < width)) lo = hi = 0.5 * (lo + hi);
        }
    }
    if (live && g == 0) w[b * iu + j] = 0.5 * (lo + hi) / s;
    if (!live && g == 0 && j < iu) w[b * iu + j] = 0.0;
}

// Work list of k_invit: clus[b*(iu+2)] = count, then in ascending order the first members of the
// clusters (runs of eigenvalues closer than ortol).
__global__ void __launch_bounds__(256) k_clusters(const double* __restrict__ w, int64_t iu, const int* __restrict__ lim,
                                                  const double* __restrict__ info, double ortol_rel,
                                                  int* __restrict__ clus) {
    const int64_t b = blockIdx.x, nw = want_of(lim, b, iu);
    const double* W = w + b * iu;
    int* C = clus + b * (iu + 2);
    const double ortol = ortol_rel * info[b * 8 + 2];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    __shared__ int cnt[8];
    int base = 0;
    for (int64_t j0 = 0; j0 < nw; j0 += 256) {
        const int64_t j = j0 + threadIdx.x;
        const bool start = j < nw && (j == 0 || W[j] - W[j - 1] > ortol);
        const unsigned m = __ballot_sync(0xffffffffu, start);
        if (lane == 0) cnt[wp] = __popc(m);
        __syncthreads();
        int off = base;
        for (int q = 0; q < wp; ++q) off += cnt[q];
        if (start) C[1 + off + __popc(m & ((1u << lane) - 1u))] = (int)j;
        for (int q = 0; q < 8; ++q) base += cnt[q];
        __syncthreads();
    }
    if (threadIdx.x == 0) C[0] = base;
}

__device__ inline uint64_t mix64(uint64_t x) {
    x ^= x >> 33;
    x *= 0xff51afd7ed558ccdULL;
    x ^= x >> 33;
    x *= 0xc4ceb9fe1a85ec53ULL;
    x ^= x >> 33;
    return x;
}

// a / b from r = RN(1 / b), correctly rounded for operands whose quotient and remainder neither over- nor
// underflow (P. W. Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34 (1990)): three dependent FMAs once r is known.
__device__ __forceinline__ double quot(double a, double b, double r) {
    const double q = a * r;
    return fma(fma(-q, b, a), r, q);
}
// exponent of |x| (biased; 0 for zero and subnormals, 2047 for Inf and NaN)
__device__ __forceinline__ int expo_of(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }

// Inverse iteration, one thread per cluster.  Scratch per thread (strided by 'stride' threads): a, b, c, dd
// (doubles), piv (bytes).  Every pass is a serial chain over the rows (a division a row in the
// factorization and the back-substitution), so the rows' loads are issued IV_U rows ahead of their use
// and the reciprocals of everything that is known before the chain gets there (the pivots of the
// back-substitution; scale and off-diagonal of the factorization) are formed off the chain.  Measured:
// N = 5044, all eigenvectors, some clusters of two 80 -> 39 ms; N = 1876, 9 k 16.9 -> 6.9 ms.
constexpr int IV_U = 8;
__global__ void __launch_bounds__(32)
    k_invit(const double* __restrict__ d, const double* __restrict__ e, int64_t n_, int64_t iu,
            const double* __restrict__ w, const int* __restrict__ lim, const double* __restrict__ info, double ortol_rel,
            const int* __restrict__ clus, double* Z /* batch x (n x iu) row-major */, double* scr, unsigned char* pivs,
            int64_t stride, int* __restrict__ fail) {
    const int64_t b = blockIdx.y;
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int* C = clus + b * (iu + 2);
    const int ncl = C[0];
    if (t >= ncl) return;
    const int n = (int)n_;
    const double* __restrict__ D = d + b * n_;
    const double* __restrict__ E = e + b * n_;
    const double* Wb = w + b * iu;
    double* Zb = Z + b * n_ * iu;
    const int64_t S = stride * gridDim.y;           // scratch row pitch
    double* ua = scr + b * stride + t;              // diag of U
    double* ub = ua + n_ * S;                       // first super-diag of U
    double* uc = ub + n_ * S;                       // multipliers
    double* ud = uc + n_ * S;                       // second super-diag of U
    unsigned char* up = pivs + b * stride + t;
    const double onenrm = info[b * 8 + 2];
    const int js = C[1 + t];
    const int64_t nw = want_of(lim, b, iu);
    int je = js + 1;
    while (je < nw && !(Wb[je] - Wb[je - 1] > ortol_rel * onenrm)) ++je;
    if (onenrm == 0.0) {
        // T = 0: any orthonormal basis (the scaled right-hand sides below would vanish)
        for (int j = js; j < je; ++j)
            for (int i = 0; i < n; ++i) Zb[i * iu + j] = (i == j) ? 1.0 : 0.0;
        return;
    }
    double xjm = 0.0;
    for (int j = js; j < je; ++j) {
        double xj = Wb[j];
        if (j > js) {
            double pertol = 10.0 * fabs(kEps * xj);
            if (xj - xjm < pertol) xj = xjm + pertol;
        }
        xjm = xj;
        double* z = Zb + j;
        // ---- dlagtf: T - xj I = P L U; tol: dlagts tolerance for job = -1
        double tol, unn;
        {
            double ak = D[0] - xj, bk = (n > 1) ? E[0] : 0.0;
            double scale1 = fabs(ak) + ((n > 1) ? fabs(E[0]) : 0.0), rs1 = 1.0 / scale1;
            tol = 0.0;
#pragma unroll 4
            for (int k = 0; k < n - 1; ++k) {
                const double ck = E[k];
                double ak1 = D[k + 1] - xj;
                double bk1 = (k < n - 2) ? E[k + 1] : 0.0;
                double scale2 = fabs(ck) + fabs(ak1);
                if (k < n - 2) scale2 += fabs(bk1);
                // off the chain: 1 / scale2, 1 / ck; the quotients by them need operands in mid-range
                const double rs2 = 1.0 / scale2, rc = 1.0 / ck;
                const int ea = expo_of(ak), ec = expo_of(ck), e1 = expo_of(scale1), e2 = expo_of(scale2);
                const bool mid = min(min(ea, ec), min(e1, e2)) > 512 && max(max(ea, ec), max(e1, e2)) < 1536;
                double qa, qc, m1;
                const double m0 = ck / ak;
                if (mid) {
                    qa = quot(fabs(ak), scale1, rs1);
                    qc = quot(fabs(ck), scale2, rs2);
                    m1 = quot(ak, ck, rc);
                } else {
                    qa = fabs(ak) / scale1;
                    qc = fabs(ck) / scale2;
                    m1 = ak / ck;
                }
                const double piv1 = (ak == 0.0) ? 0.0 : qa;
                unsigned char pv = 0;
                double dk = 0.0, a = ak, bb = bk, c = 0.0;
                if (ck == 0.0) {
                    scale1 = scale2;
                    rs1 = rs2;
                } else {
                    const double piv2 = qc;
                    if (piv2 <= piv1) {
                        scale1 = scale2;
                        rs1 = rs2;
                        const double m = m0;
                        c = m;
                        ak1 = ak1 - m * bk;
                    } else {
                        pv = 1;
                        const double mult = m1;
                        a = ck;
                        const double temp = ak1;
                        ak1 = bk - mult * temp;
                        if (k < n - 2) {
                            dk = bk1;
                            bk1 = -mult * dk;
                        }
                        bb = temp;
                        c = mult;
                    }
                }
                const int64_t o = (int64_t)k * S;
                ua[o] = a;
                ub[o] = bb;
                uc[o] = c;
                ud[o] = dk;
                up[o] = pv;
                tol = fmax(tol, fmax(fabs(a), fmax(fabs(bb), fabs(dk))));
                ak = ak1;
                bk = bk1;
            }
            unn = ak;
            ua[(int64_t)(n - 1) * S] = ak;
            tol = fmax(tol, fabs(ak));
        }
        tol *= kEps;
        if (tol == 0.0) tol = kEps;
        // ---- starting vector in Z(:, j)
        uint64_t seed = mix64(((uint64_t)b << 40) ^ ((uint64_t)j * 0x9e3779b97f4a7c15ULL) ^ 0x1234567ULL);
        double bmax = 0.0;
        for (int i = 0; i < n; ++i) {
            seed = mix64(seed + 0x9e3779b97f4a7c15ULL);
            const double v = (double)(seed >> 11) * (2.0 / 9007199254740992.0) - 1.0;
            z[i * iu] = v;
            bmax = fmax(bmax, fabs(v));
        }
        const int maxits = 5, extra = 2;
        const double dtpcrt = sqrt(0.1 / (double)n);
        int nrmchk = 0, its = 0;
        bool ok = false;
        while (its < maxits) {
            ++its;
            // scale: scl = n * onenrm * max(eps, |u_nn|) / ||b||_inf
            double scl = (double)n * onenrm * fmax(kEps, fabs(unn)) / bmax;
            // forward: apply P and L
            {
                double yprev = z[0] * scl;
                double rz[IV_U], rm[IV_U];
                unsigned char rp[IV_U];
                auto fetch = [&](int k0) {
#pragma unroll
                    for (int q = 0; q < IV_U; ++q) {
                        const int k = min(k0 + q, n - 1);
                        const int64_t o = (int64_t)(k > 0 ? k - 1 : 0) * S;
                        rz[q] = z[k * iu];
                        rm[q] = uc[o];
                        rp[q] = up[o];
                    }
                };
                fetch(1);
                for (int k0 = 1; k0 < n; k0 += IV_U) {
                    double cz[IV_U], cm[IV_U];
                    unsigned char cp[IV_U];
#pragma unroll
                    for (int q = 0; q < IV_U; ++q) {
                        cz[q] = rz[q];
                        cm[q] = rm[q];
                        cp[q] = rp[q];
                    }
                    if (k0 + IV_U < n) fetch(k0 + IV_U);
#pragma unroll
                    for (int q = 0; q < IV_U; ++q) {
                        const int k = k0 + q;
                        if (k < n) {
                            double yk = cz[q] * scl;
                            const double m = cm[q];
                            if (cp[q] == 0) {
                                yk = yk - m * yprev;
                            } else {
                                const double temp = yprev;
                                yprev = yk;
                                yk = temp - m * yk;
                            }
                            z[(k - 1) * iu] = yprev;
                            yprev = yk;
                        }
                    }
                }
                z[(n - 1) * iu] = yprev;
            }
            // backward with perturbation of tiny pivots
            double nrm = 0.0;
            {
                double y1 = 0.0, y2 = 0.0;  // y(k+1), y(k+2)
                double rz[IV_U], ra[IV_U], rb[IV_U], rd[IV_U];
                auto fetch = [&](int k0) {
#pragma unroll
                    for (int q = 0; q < IV_U; ++q) {
                        const int k = max(k0 - q, 0);
                        const int64_t o = (int64_t)k * S;
                        rz[q] = z[k * iu];
                        ra[q] = ua[o];
                        rb[q] = (k <= n - 2) ? ub[o] : 0.0;
                        rd[q] = (k <= n - 3) ? ud[o] : 0.0;
                    }
                };
                fetch(n - 1);
                for (int k0 = n - 1; k0 >= 0; k0 -= IV_U) {
                    double cz[IV_U], ca[IV_U], cb[IV_U], cd[IV_U], cr[IV_U];
#pragma unroll
                    for (int q = 0; q < IV_U; ++q) {
                        cz[q] = rz[q];
                        ca[q] = ra[q];
                        cb[q] = rb[q];
                        cd[q] = rd[q];
                        cr[q] = 1.0 / ca[q];
                    }
                    if (k0 - IV_U >= 0) fetch(k0 - IV_U);
#pragma unroll
                    for (int q = 0; q < IV_U; ++q) {
                        const int k = k0 - q;
                        if (k >= 0) {
                            double temp = cz[q];
                            if (k <= n - 3)
                                temp = temp - cb[q] * y1 - cd[q] * y2;
                            else if (k == n - 2)
                                temp = temp - cb[q] * y1;
                            double ak = ca[q], yk;
                            const int ea = expo_of(ak), et = expo_of(temp);
                            if (min(ea, et) > 512 && max(ea, et) < 1536) {
                                // mid-range operands: no scaling or perturbation applies
                                yk = quot(temp, ak, cr[q]);
                            } else {
                                double pert = copysign(tol, ak);
                                for (int guard = 0; guard < 2048; ++guard) {
                                    double absak = fabs(ak);
                                    if (absak < 1.0) {
                                        if (absak < kSafmin) {
                                            if (absak == 0.0 || fabs(temp) * kSafmin > absak) {
                                                ak += pert;
                                                pert *= 2.0;
                                                continue;
                                            }
                                            temp *= 1.0 / kSafmin;
                                            ak *= 1.0 / kSafmin;
                                        } else if (fabs(temp) > absak * (1.0 / kSafmin)) {
                                            ak += pert;
                                            pert *= 2.0;
                                            continue;
                                        }
                                    }
                                    break;
                                }
                                yk = temp / ak;
                            }
                            z[k * iu] = yk;
                            nrm = fmax(nrm, fabs(yk));
                            y2 = y1;
                            y1 = yk;
                        }
                    }
                }
            }
            // modified Gram-Schmidt against earlier cluster members
            if (j > js) {
                for (int q = js; q < j; ++q) {
                    double dot = 0.0;
                    const double* zq = Zb + q;
#pragma unroll 16
                    for (int i = 0; i < n; ++i) dot += z[i * iu] * zq[i * iu];
                    nrm = 0.0;
                    for (int i = 0; i < n; i += 16) {
                        double v[16], u[16];
#pragma unroll
                        for (int p = 0; p < 16; ++p) {
                            const int64_t o = (int64_t)min(i + p, n - 1) * iu;
                            v[p] = z[o];
                            u[p] = zq[o];
                        }
#pragma unroll
                        for (int p = 0; p < 16; ++p)
                            if (i + p < n) {
                                v[p] -= dot * u[p];
                                z[(int64_t)(i + p) * iu] = v[p];
                                nrm = fmax(nrm, fabs(v[p]));
                            }
                    }
                }
            }
            bmax = nrm;
            if (nrm < dtpcrt) continue;
            ++nrmchk;
            if (nrmchk < extra + 1) continue;
            ok = true;
            break;
        }
        if (!ok) atomicAdd(fail + b, 1);
        // normalise (2-norm), largest component positive
        double s2 = 0.0, big = 0.0, bigv = 0.0;
#pragma unroll 16
        for (int i = 0; i < n; ++i) {
            double v = z[i * iu];
            s2 += v * v;
            if (fabs(v) > big) {
                big = fabs(v);
                bigv = v;
            }
        }
        double scl = 1.0 / sqrt(s2);
        if (bigv < 0.0) scl = -scl;
        for (int i = 0; i < n; i += 16) {
            double v[16];
#pragma unroll
            for (int p = 0; p < 16; ++p) v[p] = z[(int64_t)min(i + p, n - 1) * iu] * scl;
#pragma unroll
            for (int p = 0; p < 16; ++p)
                if (i + p < n) z[(int64_t)(i + p) * iu] = v[p];
        }
    }
}

// X (n x iu complex, column-major) = Z (row-major real)
__global__ void k_z_to_x(const double* __restrict__ Z, int64_t n, int64_t iu, double2* __restrict__ X, int64_t ldx,
                         int64_t strideX) {
    const int64_t b = blockIdx.z;
    const int64_t i = blockIdx.x * 32 + threadIdx.x;
    const int64_t j0 = blockIdx.y * 32;
    __shared__ double tile[32][33];
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        int64_t ii = blockIdx.x * 32 + r, jj = j0 + threadIdx.x;
        tile[r][threadIdx.x] = (ii < n && jj < iu) ? Z[b * n * iu + ii * iu + jj] : 0.0;
    }
    __syncthreads();
    for (int c = threadIdx.y; c < 32; c += blockDim.y) {
        int64_t jj = j0 + c;
        if (i < n && jj < iu) X[b * strideX + i + jj * ldx] = make_double2(tile[threadIdx.x][c], 0.0);
    }
}

// ---------------------------------------------------------------- FP64 eigen-solver driver
int eig_fp64(cudaStream_t st, EigArgs& g) {
    const int64_t n = g.n, iu = g.iu, batch = g.batch;
    TrdArgs<double> a;
    a.A = g.A;
    a.lda = g.lda;
    a.strideA = g.strideA;
    a.n = n;
    a.d = g.d;
    a.e = g.e;
    a.tau = g.tau;
    a.W = g.Wp;
    a.Yrow = g.Yrow;
    a.Ycol = g.Ycol;
    a.ystride = g.ystride;
    a.Spart = g.Spart;
    a.sstride = g.sstride;
    a.part = g.part;
    a.pstride = g.pstride;
    a.scal = g.scal;
    a.cnt = g.cnt;
    a.w0 = g.w0;
    a.her2k = her2k_oz;
    a.her2k_user = &g;
    FORGE_CUDA(cudaMemsetAsync(g.oz_err, 0, sizeof(int), st));
    FORGE_TRY(tridiagonalize_fp64(st, a, batch));
    FORGE_TRY(tridiag_eigvecs(st, g));
    dim3 gz((unsigned)((n + 31) / 32), (unsigned)((iu + 31) / 32), (unsigned)batch);
    k_z_to_x<<<gz, dim3(32, 8), 0, st>>>(g.Z, n, iu, g.X, g.ldx, g.strideX);
    FORGE_LAUNCH_CHECK();
    prof_begin(ST_BACKTRANSFORM);
    FORGE_TRY(backtransform_oz(st, g));
    prof_end(ST_BACKTRANSFORM, batch * (double)n * iu * 16.0 * 2.0 + batch * 0.5 * n * (double)n * 16.0,
             batch * 8.0 * (double)n * n * iu);
    int herr = 0;
    FORGE_CUDA(cudaMemcpyAsync(&herr, g.oz_err, sizeof(int), cudaMemcpyDeviceToHost, st));
    FORGE_CUDA(cudaStreamSynchronize(st));
    if (herr) {
        set_error(FORGE_ERR_TIMEOUT, "tcgen05 GEMM (FP64 slices): a bounded mbarrier wait gave up");
        return FORGE_ERR_TIMEOUT;
    }
    return 0;
}

// eigenvalues 1..iu (bisection) and tridiagonal eigenvectors (inverse iteration) into g.X (real)
int tridiag_eigvecs(cudaStream_t st, EigArgs& g) {
    const int64_t n = g.n, iu = g.iu, batch = g.batch;
    k_gersh<<<(unsigned)batch, 256, 0, st>>>(g.d, g.e, n, g.info);
    FORGE_LAUNCH_CHECK();
    prof_begin(ST_BISECT);
    k_tri_scale<<<dim3((unsigned)std::min<int64_t>((n + 255) / 256, 64), (unsigned)batch), 256, 0, st>>>(
        g.d, g.e, n, g.info, g.de, g.tf);
    FORGE_LAUNCH_CHECK();
    double* lam = g.replay ? g.scr : g.w;   // the scratch of the eigenvectors is free until k_invit
    k_bisect_f32<<<dim3((unsigned)((iu + 31) / 32), (unsigned)batch), 32, 0, st>>>(g.tf, n, iu, g.iu_lim, g.info, lam);
    FORGE_LAUNCH_CHECK();
    // full FP64 accuracy in both precisions: the eigenvectors of close eigenvalues need it.  Lanes per
    // eigenvalue: four warps fill the FP64 pipes of an SM (152 x 128 lanes); beyond that more
    // points a round only add work
    const int64_t lanes = 152 * 128;
    const int G = iu * batch * 8 <= lanes ? 8 : iu * batch * 4 <= lanes + lanes / 4 ? 4 : iu * batch <= lanes ? 2 : 1;
    const dim3 gb((unsigned)((iu * G + 31) / 32), (unsigned)batch);   // one warp a CTA: spread over the SMs
    if (G == 8)
        k_bisect<8><<<gb, 32, 0, st>>>(g.de, n, iu, g.iu_lim, g.info, lam);
    else if (G == 4)
        k_bisect<4><<<gb, 32, 0, st>>>(g.de, n, iu, g.iu_lim, g.info, lam);
    else if (G == 2)
        k_bisect<2><<<gb, 32, 0, st>>>(g.de, n, iu, g.iu_lim, g.info, lam);
    else
        k_bisect<1><<<gb, 32, 0, st>>>(g.de, n, iu, g.iu_lim, g.info, lam);
    FORGE_LAUNCH_CHECK();
    if (g.replay) {
        const unsigned by = (unsigned)batch;
        k_tri_to_f32<<<dim3((unsigned)std::min<int64_t>((n + 255) / 256, 64), by), 256, 0, st>>>(g.d, g.e, n, g.tq);
        FORGE_LAUNCH_CHECK();
        k_bisect_qf<<<dim3((unsigned)((iu + 31) / 32), by), 32, 0, st>>>(g.tq, n, iu, g.iu_lim, g.info, lam, g.w);
        FORGE_LAUNCH_CHECK();
        if (G == 8)
            k_bisect_replay<3><<<dim3((unsigned)((iu * 8 + 31) / 32), by), 32, 0, st>>>(g.d, g.e, n, iu, g.iu_lim, g.info,
                                                                                        lam, g.w);
        else if (G == 4)
            k_bisect_replay<2><<<dim3((unsigned)((iu * 4 + 31) / 32), by), 32, 0, st>>>(g.d, g.e, n, iu, g.iu_lim, g.info,
                                                                                        lam, g.w);
        else
            k_bisect_replay<1><<<dim3((unsigned)((iu + 31) / 32), by), 32, 0, st>>>(g.d, g.e, n, iu, g.iu_lim, g.info,
                                                                                    lam, g.w);
        FORGE_LAUNCH_CHECK();
    }
    prof_end(ST_BISECT, batch * 16.0 * n, batch * 10.0 * 60.0 * (double)n * iu);
    FORGE_CUDA(cudaMemsetAsync(g.fail, 0, sizeof(int) * batch, st));
    prof_begin(ST_INVIT);
    // columns beyond a slot's own nUpper
    if (g.iu_lim) FORGE_CUDA(cudaMemsetAsync(g.Z, 0, sizeof(double) * (size_t)batch * n * iu, st));
    k_clusters<<<(unsigned)batch, 256, 0, st>>>(g.w, iu, g.iu_lim, g.info, g.ortol_rel, g.clus);
    FORGE_LAUNCH_CHECK();
    k_invit<<<dim3((unsigned)((g.scr_stride + 31) / 32), (unsigned)batch), 32, 0, st>>>(
        g.d, g.e, n, iu, g.w, g.iu_lim, g.info, g.ortol_rel, g.clus, g.Z, g.scr, g.pivs, g.scr_stride, g.fail);
    FORGE_LAUNCH_CHECK();
    prof_end(ST_INVIT, batch * 8.0 * (double)n * iu, 0.0);
    return 0;
}

}  // namespace forge

namespace forge {

namespace {
inline size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }
struct Carve {
    char* base;
    size_t off = 0;
    template <class T>
    T* take(size_t count) {
        size_t o = off;
        off = al256(off + count * sizeof(T));
        return base ? reinterpret_cast<T*>(base + o) : nullptr;
    }
};
void carve(EigArgs& g, Carve& c) {
    const int64_t n = g.n, iu = g.iu, B = g.batch;
    const int64_t nblk = (n + TRD_TILE - 1) / TRD_TILE;
    const int64_t nrb = (n + 127) / 128;   // slots of the panel dots
    g.ystride = nblk * n;
    g.sstride = nrb * 2 * TRD_NB;
    g.pstride = 3 * ((n + 31) / 32) + 1;  // per-CTA partials of k_col64 and k_finish64
    g.scr_stride = iu;
    g.d = c.take<double>(B * n);
    g.e = c.take<double>(B * n);
    g.tau = c.take<double2>(B * n);
    g.Wp = c.take<double2>(B * n * TRD_NB);
    g.w0 = c.take<double2>(B * n);
    g.Yrow = c.take<double2>(B * g.ystride);
    g.Ycol = c.take<double2>(B * g.ystride);
    g.Spart = c.take<double2>(B * g.sstride);
    g.part = c.take<double>(B * g.pstride);
    g.scal = c.take<double>(B * 16);
    g.cnt = c.take<unsigned>(B * 4);
    g.info = c.take<double>(B * 8);
    g.clus = c.take<int>(B * (iu + 2));
    OzSizes z;
    oz_sizes(n, iu, B, z);
    // the slices of X (and of the rank-2k update) share the scratch of the inverse iteration, those of V its
    // vectors: both are free before it, and again once Z has been copied to X
    g.Z = (double*)c.take<char>(std::max<size_t>(sizeof(double) * B * n * iu, 2 * z.vr));
    g.oz_vr = g.Z;
    g.scr = (double*)c.take<char>(std::max<size_t>(sizeof(double) * 4 * n * iu * B, 2 * std::max(z.xs, z.uz)));
    g.oz_xs = g.scr;
    g.pivs = c.take<unsigned char>(n * iu * B);
    g.fail = c.take<int>(B);
    g.oz_vh = c.take<char>(2 * z.vh);
    g.oz_ws = c.take<char>(2 * z.ws);
    g.oz_ts = c.take<char>(2 * z.ts);
    g.oz_wp = c.take<double2>(z.wp);
    g.oz_g = c.take<double2>(z.g);
    g.oz_t = c.take<double2>(z.g);
    g.oz_ex = c.take<int>(z.ex);
    g.oz_err = c.take<int>(1);
    g.tf = c.take<float2>(B * n);
    g.de = c.take<double2>(B * n);
    g.tq = c.take<float>(B * 2 * n);
}
}  // namespace

size_t eig_workspace_bytes(int64_t n, int64_t iu, int64_t batch) {
    EigArgs g{};
    g.n = n;
    g.iu = iu;
    g.batch = batch;
    Carve c{nullptr};
    carve(g, c);
    return c.off;
}

void eig_bind_workspace(EigArgs& g, void* base) {
    Carve c{static_cast<char*>(base)};
    carve(g, c);
}

}  // namespace forge
