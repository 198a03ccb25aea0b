// Eigenpairs 1..iu of the real symmetric tridiagonal T (d, e) and back-transformation
// X = Q Z, batched over k.
//
// zheevr with RANGE='I' and IU < N (LapackRoutines.f90:414-426) computes the
// eigenvalues by bisection (dstebz) and the vectors by inverse iteration (zstein);
// this file restates that route for the GPU:
//   k_gersh     : Gershgorin interval, 1-norm and pivmin per matrix;
//   k_bisect*   : eigenvalues by Sturm counts, an FP32 bracket and FP64 multisection
//                 (eigenvalues near zero by bisection with quotients);
//   k_clusters  : groups consecutive eigenvalues closer than ortol;
//   k_invit_lu  : LU of T - lambda I with partial pivoting (dlagtf), a thread an eigenvalue;
//   k_invit     : perturbed back-substitution (dlagts, job=-1): a thread an eigenvalue for the first members
//                 of the clusters and the first solve of the others, then eight lanes a cluster for the others'
//                 modified Gram-Schmidt against the earlier members and further solves;
//   back-transform: Q applied in compact-WY blocks (zlarft forward/columnwise) on the tensor
//                 cores (oz_fp64.cu; eig_mixed.cu for the mixed path).
// ortol is tighter than zstein's 1e-3*||T||_1 (which groups a whole dense spectrum
// into one serial cluster); with ortol = 1e-7*||T||_1 the vector error bound
// eps*||T||/gap stays below 1e-8 outside clusters.
#include <algorithm>
#include <cfloat>
#include <vector>

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
// replacements, with one carried over the rescale, leave it at 2^-5 THR of the larger, which has to be a normal number
// whose own predecessor is above 2^THR times the smallest (5 THR < BIAS).  In FP32 2^-25 is below the rounding of
// d_i.  Sign and exponent are handled as integers.
template <class T>
struct Minor;
template <>
struct Minor<double> {
    static constexpr int THR = 160, MB = 20, BIAS = 1023;
    static_assert(5 * THR < BIAS, "five replacements stay normal");
    __device__ static int hi(double x) { return __double2hiint(x); }
    __device__ static double add_hi(double x, int dh) { return __hiloint2double(__double2hiint(x) + dh, __double2loint(x)); }
    __device__ static double neg(double x) { return __hiloint2double(__double2hiint(x) ^ 0x80000000, __double2loint(x)); }
};
template <>
struct Minor<float> {
    static constexpr int THR = 25, MB = 23, BIAS = 127;
    static_assert(5 * THR < BIAS, "five replacements stay normal");
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

// ---------------------------------------------------------------- division by FMAs
// exponent of |x| (biased; 0 for zero and subnormals, 2047 for Inf and NaN)
__device__ __forceinline__ int expo_of(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
// operands whose quotient, remainder and products of two neither over- nor underflow
__device__ __forceinline__ bool mid_expo(double x) { return (unsigned)(expo_of(x) - 524) < 1000u; }
// Reciprocal to 2^-40: one Newton step on the hardware's approximation (2^-20).
__device__ __forceinline__ double recip(double b) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
    return fma(r, fma(-b, r, 1.0), r);
}
// a / b from r = recip(b) for operands in mid-range: the remainder of a r brings the quotient to 2^-80 before its
// one rounding (P. W. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor",
// IBM J. Res. Dev. 34 (1990)), so it is the rounded quotient but for one case in 2^27 or fewer, a
// unit in the last place then (forge_gpu_selftest_quot counts them).  Five FMAs with recip: an FP64 instruction of a warp holds its scheduler's FP64 pipe for 64 clocks on this GPU, whatever the
// number of lanes, so the count of them is what the serial chains below cost.
__device__ __forceinline__ double quot(double a, double b, double r) {
    const double q = a * r;
    return fma(fma(-q, b, a), r, q);
}

// ---------------------------------------------------------------- quotient form (mixed precision)
// number of eigenvalues <= x (dlaebz Sturm count); t[i] = (d_i, e_{i-1}^2)
__device__ inline int sturm_q(const double2* __restrict__ t, int n, double x, double pivmin) {
    constexpr int U = 8;
    double q = t[0].x - x;
    if (fabs(q) < pivmin) q = -pivmin;
    int cnt = (q <= 0.0) ? 1 : 0;
    const bool small_piv = expo_of(pivmin) < 524;
    double2 nx[U];
#pragma unroll
    for (int u = 0; u < U; ++u) nx[u] = t[min(1 + u, n - 1)];
    for (int i0 = 1; i0 < n; i0 += U) {
        double2 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = nx[u];
#pragma unroll
        for (int u = 0; u < U; ++u) nx[u] = t[min(i0 + U + u, n - 1)];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (i0 + u >= n) break;
            double f;
            if (mid_expo(q) && mid_expo(v[u].y))
                f = quot(v[u].y, q, recip(q));
            else
                f = v[u].y / q;
            q = v[u].x - f - x;
            if (!(small_piv && mid_expo(q))) {
                if (fabs(q) < pivmin) q = -pivmin;
                cnt += (q <= 0.0) ? 1 : 0;
            } else {
                cnt += (int)((unsigned)__double2hiint(q) >> 31);
            }
        }
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
// The unscaled tridiagonal for the quotient form: t[b][i] = (d_i, e_{i-1}^2), and in FP32 tq[b][0..n) = d,
// tq[b][n..2n) = e^2
__global__ void k_tri_quot(const double* __restrict__ d, const double* __restrict__ e, int64_t n, double2* __restrict__ t,
                           float* __restrict__ tq) {
    const int64_t b = blockIdx.y;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double em = (i > 0) ? e[b * n + i - 1] : 0.0;
        t[b * n + i] = make_double2(d[b * n + i], em * em);
        tq[b * 2 * n + i] = (float)d[b * n + i];
        const double ei = (i < n - 1) ? e[b * n + i] : 0.0;
        tq[b * 2 * n + n + i] = (float)(ei * ei);
    }
}
// Bisection of [lo, hi] while open(lo, hi), at most maxit halvings: where known(mid) is not 0 its sign is the decision
// (+1: the eigenvalue is not above mid), elsewhere count(mid) is.  The 2^LEV - 1 midpoints of the next LEV
// levels are counted at once by the G lanes of the eigenvalue's group.
template <int LEV, class T, class Open, class Known, class Count>
__device__ __forceinline__ void bisect_tree(T& lo, T& hi, bool live, int maxit, Open open, Known known, Count count) {
    constexpr int G = LEV == 1 ? 1 : 1 << LEV;
    const int g = threadIdx.x % G, base = (threadIdx.x & 31) / G * G;
    const unsigned full = 0xffffffffu;
    int it = 0;
    for (;;) {
        // decisions that need no count
        while (live && it < maxit && open(lo, hi)) {
            const T mid = (T)0.5 * (lo + hi);
            const int k = known(mid);
            if (k == 0) break;
            if (k > 0)
                hi = mid;
            else
                lo = mid;
            ++it;
        }
        const bool more = live && it < maxit && open(lo, hi);
        if (!__any_sync(full, more)) break;
        // lane g holds node g of the tree (1: root; children 2g, 2g + 1 = lower, upper half)
        T a = lo, c = hi;
        if (G > 1)
            for (int bit = 30 - __clz(g > 0 ? g : 1); bit >= 0; --bit) {
                const T mid = (T)0.5 * (a + c);
                if ((g >> bit) & 1)
                    a = mid;
                else
                    c = mid;
            }
        bool up = false;
        if (more && (G == 1 || g > 0)) up = count((T)0.5 * (a + c));
        const unsigned ups = __ballot_sync(full, up) >> base;
        if (more) {
            int node = G == 1 ? 0 : 1;
#pragma unroll
            for (int q = 0; q < LEV; ++q) {
                if (it < maxit && open(lo, hi)) {
                    const T mid = (T)0.5 * (lo + hi);
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
}
// FP32 bisection of eigenvalue j in the quotient form, into w.  As in k_bisect_replay, a midpoint further
// than 64 eps_32 |T| from the eigenvalue lam is decided without a count.
template <int LEV>
__global__ void __launch_bounds__(32) k_bisect_qf(const float* __restrict__ tq, int64_t n, int64_t iu,
                                                  const int* __restrict__ lim, const double* __restrict__ info,
                                                  const double* __restrict__ lam, double* __restrict__ w) {
    constexpr int G = LEV == 1 ? 1 : 1 << LEV;
    const int64_t b = blockIdx.y;
    const int64_t j = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
    const bool live = j < want_of(lim, b, iu);
    const float* D = tq + b * 2 * n;
    const float* E2 = D + n;
    // Gershgorin bounds widened by the FP32 rounding of the counts
    const float tn = (float)info[b * 8 + 4];
    float lo = (float)info[b * 8 + 0] - 8.f * FLT_EPSILON * tn * 64.f, hi = (float)info[b * 8 + 1] + 8.f * FLT_EPSILON * tn * 64.f;
    const float pivmin = fmaxf(1e-30f, (float)info[b * 8 + 3]);
    const double l = live ? lam[b * iu + j] : 0.0, far = 64.0 * (double)FLT_EPSILON * info[b * 8 + 4];
    bisect_tree<LEV>(
        lo, hi, live, 64,
        [&](float a, float c) {
            const float width = c - a, mid = 0.5f * (a + c);
            return !(width <= 2.f * FLT_EPSILON * fmaxf(fabsf(a), fabsf(c)) || width <= pivmin || mid <= a || mid >= c);
        },
        [&](float mid) { return mid > l + far ? 1 : mid < l - far ? -1 : 0; },
        [&](float mid) { return sturm_qf(D, E2, (int)n, mid, pivmin) >= j + 1; });
    if (live && threadIdx.x % G == 0) w[b * iu + j] = 0.5 * ((double)lo + (double)hi);
}
// The FP64 bisection of the mixed path, from the bracket x -/+ 8 eps_32 |T| of the FP32 estimate x when
// the counts confirm it.  Its midpoints form a fixed dyadic sequence, and the quotient-form count decides
// each: where a midpoint lies further from the eigenvalue that k_bisect found (lam) than 64 eps |T|,
// many times the error of either count, the decision is known without a count; only the last few
// are counted, several levels of the bisection tree at once.  Why not k_bisect's own result: the mixed path rounds
// the eigenvectors to FP32 afterwards, and that rounding noise stays in the refined density matrix to second order
// (3e-9 of its norm at N = 1324), so a last-place change of an eigenvalue would change the results by
// as much; this keeps them bit for bit.  Bound: the FP64 instructions of a step, seven.
// Measured, kernel alone (a library division a step before): N = 5044, all eigenvalues 31 -> 17 ms; the whole stage
// 51 -> 32 ms, N = 1324, 4 k 25 -> 16 ms, N = 1876, 9 k 26.5 -> 16 ms.
template <int LEV>
__global__ void __launch_bounds__(32) k_bisect_replay(const double2* __restrict__ de, int64_t n, int64_t iu,
                                                      const int* __restrict__ lim, const double* __restrict__ info,
                                                      const double* __restrict__ lam, double* __restrict__ w) {
    constexpr int G = LEV == 1 ? 1 : 1 << LEV;
    const int64_t b = blockIdx.y;
    const int64_t j = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
    const bool live = j < want_of(lim, b, iu);
    const double2* t = de + b * n;
    double lo = info[b * 8 + 0], hi = info[b * 8 + 1];
    const double pivmin = info[b * 8 + 3], tnorm = info[b * 8 + 4];
    const double l = live ? lam[b * iu + j] : 0.0, far = 64.0 * kEps * tnorm;
    auto known = [&](double mid) { return mid > l + far ? 1 : mid < l - far ? -1 : 0; };
    auto count = [&](double mid) { return sturm_q(t, (int)n, mid, pivmin) >= j + 1; };
    if (live) {
        const double x = w[b * iu + j], delta = 8.0 * (double)FLT_EPSILON * tnorm;
        const double l2 = fmax(lo, x - delta), h2 = fmin(hi, x + delta);
        if (l2 < h2) {
            const int kl = known(l2), kh = known(h2);
            const bool lok = kl ? kl < 0 : !count(l2);
            const bool hok = kh ? kh > 0 : count(h2);
            if (lok && hok) {
                lo = l2;
                hi = h2;
            }
        }
    }
    const double rtol = 4.0 * kEps;
    bisect_tree<LEV>(
        lo, hi, live, 256,
        [&](double a, double c) { return c - a > fmax(fmax(kSafmin, pivmin), rtol * fmax(fabs(a), fabs(c))); }, known, count);
    if (threadIdx.x % G == 0 && j < iu) w[b * iu + j] = live ? 0.5 * (lo + hi) : 0.0;
}

// ---------------------------------------------------------------- multisection (minors)
// Eigenvalue j of the scaled T to FP32 accuracy, into w (scaled): multisection by G lanes as in k_bisect.
template <int G>
__global__ void __launch_bounds__(32) k_bisect_f32(const float2* __restrict__ tf, int64_t n, int64_t iu,
                                                   const int* __restrict__ lim, const double* __restrict__ info,
                                                   double* __restrict__ w) {
    const int64_t b = blockIdx.y;
    const int64_t j = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
    const int g = threadIdx.x % G, base = (threadIdx.x & 31) / G * G;
    const bool live = j < want_of(lim, b, iu);
    const unsigned full = 0xffffffffu;
    const unsigned gmask = (unsigned)(((1ull << G) - 1ull) << base);
    const double s = tri_scale(info + b * 8);
    // Gershgorin bounds widened by the FP32 rounding of the counts
    float lo = (float)(info[b * 8 + 0] * s) - 512.f * FLT_EPSILON, hi = (float)(info[b * 8 + 1] * s) + 512.f * FLT_EPSILON;
    for (int it = 0; it < 64; ++it) {
        // the counts are good to a few FP32 ulps of |T| <= 1
        const float width = hi - lo;
        const bool open = live && width > FLT_EPSILON;
        if (!__any_sync(full, open)) break;
        const float x = lo + width * ((float)(g + 1) / (float)(G + 1));
        bool up = true;
        if (open) up = sturm<float>(tf + b * n, (int)n, x) >= j + 1;
        const unsigned ups = (__ballot_sync(full, up) & gmask) >> base;
        const int f = ups ? __ffs(ups) - 1 : G;
        const float xf = __shfl_sync(full, x, base + (f < G ? f : G - 1));
        const float xp = __shfl_sync(full, x, base + (f > 0 ? f - 1 : 0));
        if (open) {
            if (f < G) hi = fminf(hi, xf);
            if (f > 0) lo = fmaxf(lo, xp);
            // no representable point inside the bracket
            if (!(hi - lo < width)) lo = hi = 0.5f * (lo + hi);
        }
    }
    if (live && g == 0) w[b * iu + j] = 0.5 * ((double)lo + (double)hi);
}

// Eigenvalue j of the scaled T if it is below TINY: bisection with the quotients (dlaebz), whose smallest pivot is
// kSafmin for |T| <= 1.  A minor's replacement by 2^-160 of its predecessor is a change of d_i by that much, so the
// multisection's counts place an eigenvalue to 2^-159: nothing to one above 2^-106, everything to one below.
constexpr double TINY = 7.888609052210118e-31;   // 2^-100
__device__ __noinline__ double bisect_tiny(const double2* __restrict__ t, int n, int64_t j, double glo, double ghi) {
    auto count = [&](double x) {
        double q = t[0].x - x;
        if (fabs(q) < kSafmin) q = -kSafmin;
        int64_t cnt = q <= 0.0;
        for (int i = 1; i < n; ++i) {
            const double2 v = t[i];
            q = v.x - v.y / q - x;
            if (fabs(q) < kSafmin) q = -kSafmin;
            cnt += q <= 0.0;
        }
        return cnt;
    };
    double lo = fmax(glo, -2.0 * TINY), hi = fmin(ghi, 2.0 * TINY);
    if (!(lo < hi && count(lo) < j + 1 && count(hi) >= j + 1)) {
        lo = glo;
        hi = ghi;
    }
    for (int it = 0; it < 256; ++it) {
        if (!(hi - lo > fmax(kSafmin, 4.0 * kEps * fmax(fabs(lo), fabs(hi))))) break;
        const double mid = 0.5 * (lo + hi);
        if (count(mid) >= j + 1)
            hi = mid;
        else
            lo = mid;
    }
    return 0.5 * (lo + hi);
}

// Eigenvalue j in FP64 by multisection: G lanes evaluate the Sturm counts at G equally spaced points of
// the bracket, which shrinks by G + 1 a round.  The bracket starts from the FP32 estimate in w: it is
// widened by 16 until the FP64 counts confirm it, at last to the Gershgorin interval.  Stops at the
// reference's 4 eps |lambda|, or at abstol (scaled) where that is wider.  G (launch rule in tridiag_eigvecs): a round costs the latency of n
// dependent steps as long as the FP64 pipes are not full, so few eigenvalues take many lanes each.
// Bound: FP64 pipe (three slots a step) or, below ~19000 lanes, the latency of the chain.  Measured,
// FP64 stage total (quotient-form bisection by one lane before): N = 1324, 16 k 47.9 -> 6.4 ms;
// N = 3268, one k 111 -> 8.1 ms.
template <int G>
__global__ void __launch_bounds__(32) k_bisect(const double2* __restrict__ de, int64_t n, int64_t iu,
                                                const int* __restrict__ lim, const double* __restrict__ info,
                                                double abstol, double* w) {
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
        const double tol = fmax(abstol, rtol * fmax(fabs(lo), fabs(hi)));
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
    if (live && g == 0) {
        double lam = 0.5 * (lo + hi);
        // abstol is wider where k_bisect_replay follows, which has quotients of its own
        if (abstol < TINY && fabs(lam) < TINY) lam = bisect_tiny(t, (int)n, j, glo, ghi);
        w[b * iu + j] = lam / s;
    }
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

// |x| as an integer: absolute values compare as their bit patterns, off the FP64 pipe
__device__ __forceinline__ uint64_t abs_bits(double x) { return (uint64_t)__double_as_longlong(x) & 0x7fffffffffffffffULL; }

// Inverse iteration (dstein).  What bounds it is the count of FP64 instructions along the serial chains over the
// rows (see quot): twelve a row for a factorization, nine for a solve; comparisons and maxima go by bit patterns, the
// pivot is chosen by cross products unless the two quotients agree to 2^-48, and a row's one quotient is
// that of the chosen branch.  Rows are loaded IV_U ahead.  Only the orthogonalisation inside a cluster has to go
// member by member: k_invit_lu factorizes for every eigenvalue at once, k_invit<0> does the whole iteration for
// the first member of each cluster and the first solve for the others, k_invit<1> the rest of these with eight lanes a
// cluster.  Scratch (rows of pitch S = batch iu): diagonal, first and second superdiagonal
// of U, multipliers, pivots; the last row's free multiplier slot holds the tolerance of the tiny pivots.
// Measured (stage, one thread a cluster and a division a row before): N = 5044, all eigenvectors of one matrix 18.4 ->
// 12 ms without clusters, 64 -> 29 ms with one of about five; N = 1324, 4 k, some clusters 24 -> 12 ms; N = 1876, 9 k
// 6.9 -> 4.6 ms.
constexpr int IV_U = 8;

struct InvitArgs {
    const double *d, *e, *w, *info;
    const int *lim, *clus;
    int64_t n, iu;
    double ortol_rel;
    double* Z;   // batch x (n x iu) row-major
    double* scr;
    unsigned char* pivs;
    int* fail;
};
__device__ __forceinline__ bool starts_cluster(const double* W, int64_t j, double ortol) {
    return j == 0 || W[j] - W[j - 1] > ortol;
}

// dlagtf: T - xj I = P L U; tol: dlagts tolerance for job = -1
__global__ void __launch_bounds__(32) k_invit_lu(InvitArgs g) {
    const int64_t b = blockIdx.y, j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const double onenrm = g.info[b * 8 + 2];
    if (j >= want_of(g.lim, b, g.iu) || onenrm == 0.0) return;
    const int n = (int)g.n;
    const double* __restrict__ D = g.d + b * n;
    const double* __restrict__ E = g.e + b * n;
    const double* Wb = g.w + b * g.iu;
    const int64_t S = g.iu * gridDim.y;
    double* ua = g.scr + b * g.iu + j;
    double* ub = ua + n * S;
    double* uc = ub + n * S;
    double* ud = uc + n * S;
    unsigned char* up = g.pivs + b * g.iu + j;
    // close eigenvalues of a cluster are moved apart
    int64_t js = j;
    while (!starts_cluster(Wb, js, g.ortol_rel * onenrm)) --js;
    double xj = Wb[js];
    for (int64_t q = js + 1; q <= j; ++q) {
        const double xm = xj, pertol = 10.0 * fabs(kEps * Wb[q]);
        xj = Wb[q];
        if (xj - xm < pertol) xj = xm + pertol;
    }
    double ak = D[0] - xj, bk = (n > 1) ? E[0] : 0.0;
    double scale1 = fabs(ak) + ((n > 1) ? fabs(E[0]) : 0.0);
    uint64_t big = 0;
    double nd[IV_U], ne[IV_U];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int q = 0; q < IV_U; ++q) {
            nd[q] = D[min(k0 + q + 1, n - 1)];
            ne[q] = k0 + q + 1 < n - 1 ? E[k0 + q + 1] : 0.0;
        }
    };
    fetch(0);
    double ck = bk;   // E[k]
    for (int k0 = 0; k0 < n - 1; k0 += IV_U) {
        double cd[IV_U], ce[IV_U];
#pragma unroll
        for (int q = 0; q < IV_U; ++q) {
            cd[q] = nd[q];
            ce[q] = ne[q];
        }
        fetch(k0 + IV_U);
#pragma unroll
        for (int q = 0; q < IV_U; ++q) {
            const int k = k0 + q;
            if (k >= n - 1) break;
            double ak1 = cd[q] - xj, bk1 = ce[q];
            const double scale2 = k < n - 2 ? fabs(ck) + fabs(ak1) + fabs(bk1) : fabs(ck) + fabs(ak1);
            double a = ak, bb = bk, c = 0.0, dk = 0.0;
            unsigned char pv = 0;
            const bool mid = mid_expo(ak) && mid_expo(ck) && mid_expo(scale1) && mid_expo(scale2);
            const int64_t dx = mid ? __double_as_longlong(fabs(ck) * scale1) - __double_as_longlong(fabs(ak) * scale2) : 0;
            bool swap;
            if (mid && (dx > 16 || dx < -16)) {
                swap = dx > 0;
            } else {
                const double piv1 = (ak == 0.0) ? 0.0 : fabs(ak) / scale1, piv2 = fabs(ck) / scale2;
                swap = !(ck == 0.0) && !(piv2 <= piv1);
            }
            if (ck == 0.0) {
                scale1 = scale2;
            } else {
                const double num = swap ? ak : ck, den = swap ? ck : ak;
                c = mid ? quot(num, den, recip(den)) : num / den;
                // without / with exchange: ak1 - c bk and bk1, or bk - c ak1 and -c bk1
                const double x = swap ? bk : ak1, y = swap ? ak1 : bk;
                ak1 = fma(-c, y, x);
                if (swap) {
                    pv = 1;
                    a = ck;
                    bb = y;
                    if (k < n - 2) {
                        dk = bk1;
                        bk1 = -c * dk;
                    }
                } else {
                    scale1 = scale2;
                }
            }
            const int64_t o = (int64_t)k * S;
            ua[o] = a;
            ub[o] = bb;
            uc[o] = c;
            ud[o] = dk;
            up[o] = pv;
            big = max(max(big, abs_bits(a)), max(abs_bits(bb), abs_bits(dk)));
            ak = ak1;
            bk = bk1;
            ck = ce[q];
        }
    }
    ua[(int64_t)(n - 1) * S] = ak;
    big = max(big, abs_bits(ak));
    double tol = __longlong_as_double((long long)big) * kEps;
    if (tol == 0.0) tol = kEps;
    uc[(int64_t)(n - 1) * S] = tol;
}

// One pass over z by the IV_G lanes of a cluster: z -= dot u (u may be null), *dot_next = sum z un over the rows in
// order (un may be null) and the largest |z|, as bits.  The update is one instruction for IV_G rows; the sum's
// operands go round by shuffles, so that its chain of FMAs is all that a row costs.
constexpr int IV_G = 8;
__device__ __forceinline__ void mgs_pass(unsigned mask, int n, int64_t iu, double* z, const double* u, double dot,
                                         const double* un, double* dot_next, uint64_t* top) {
    const int g = threadIdx.x % IV_G;
    double acc = 0.0;
    uint64_t big = 0;
    auto at = [&](const double* x, int i) { return x && i < n ? x[(int64_t)i * iu] : 0.0; };
    constexpr int U = 4;   // IV_G U rows in flight ahead of their use
    double zv[U], uv[U], nv[U];
    auto fetch = [&](int i0) {
#pragma unroll
        for (int p = 0; p < U; ++p) {
            zv[p] = at(z, i0 + p * IV_G);
            uv[p] = at(u, i0 + p * IV_G);
            nv[p] = at(un, i0 + p * IV_G);
        }
    };
    fetch(g);
    for (int i0 = 0; i0 < n; i0 += U * IV_G) {
        double v[U], uc[U], w[U];
#pragma unroll
        for (int p = 0; p < U; ++p) {
            v[p] = zv[p];
            uc[p] = uv[p];
            w[p] = nv[p];
        }
        fetch(i0 + U * IV_G + g);
#pragma unroll
        for (int p = 0; p < U; ++p) {
            const int i = i0 + p * IV_G + g;
            if (u) {
                v[p] = fma(-dot, uc[p], v[p]);
                if (i < n) z[(int64_t)i * iu] = v[p];
            }
            if (i < n) big = max(big, abs_bits(v[p]));
        }
        if (un) {
#pragma unroll
            for (int p = 0; p < U; ++p)
#pragma unroll
                for (int q = 0; q < IV_G; ++q) {
                    const double x = __shfl_sync(mask, v[p], q, IV_G), c = __shfl_sync(mask, w[p], q, IV_G);
                    if (i0 + p * IV_G + q < n) acc = fma(x, c, acc);
                }
        }
    }
    *dot_next = acc;
#pragma unroll
    for (int o = IV_G / 2; o > 0; o >>= 1) big = max(big, (uint64_t)__shfl_xor_sync(mask, (unsigned long long)big, o, IV_G));
    *top = big;
}

// REST = 0: a thread per eigenvalue, 1: IV_G lanes per cluster (members after the first; the solves are lane 0's)
template <int REST>
__global__ void __launch_bounds__(32) k_invit(InvitArgs g) {
    const int64_t b = blockIdx.y;
    const int64_t t = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / (REST ? IV_G : 1);
    const int lane = REST ? threadIdx.x % IV_G : 0;
    const unsigned mask = ((1u << IV_G) - 1u) << (threadIdx.x & 31) / IV_G * IV_G;   // of a cluster's lanes
    const int n = (int)g.n;
    const int64_t iu = g.iu;
    const double onenrm = g.info[b * 8 + 2], ortol = g.ortol_rel * onenrm;
    const double* Wb = g.w + b * iu;
    double* Zb = g.Z + b * n * iu;
    const int64_t S = iu * gridDim.y;
    const int64_t nw = want_of(g.lim, b, iu);
    int js, je;
    bool first = true;   // the first member of its cluster
    if (REST) {
        const int* C = g.clus + b * (iu + 2);
        if (t >= C[0] || onenrm == 0.0) return;
        js = C[1 + t];
        je = js + 1;
        while (je < nw && !starts_cluster(Wb, je, ortol)) ++je;
    } else {
        if (t >= nw) return;
        js = (int)t;
        je = js + 1;
        if (onenrm == 0.0) {
            // T = 0: any orthonormal basis (the scaled right-hand sides below would vanish)
            for (int i = 0; i < n; ++i) Zb[i * iu + js] = (i == js) ? 1.0 : 0.0;
            return;
        }
        first = starts_cluster(Wb, js, ortol);
    }
    for (int j = REST ? js + 1 : js; j < je; ++j) {
        double* z = Zb + j;
        const double* ua = g.scr + b * iu + j;
        const double* ub = ua + n * S;
        const double* uc = ub + n * S;
        const double* ud = uc + n * S;
        const unsigned char* up = g.pivs + b * iu + j;
        const double unn = ua[(int64_t)(n - 1) * S], tol = uc[(int64_t)(n - 1) * S];
        double bmax = 0.0;
        if (!REST) {
            // ---- starting vector in Z(:, j)
            uint64_t seed = mix64(((uint64_t)b << 40) ^ ((uint64_t)j * 0x9e3779b97f4a7c15ULL) ^ 0x1234567ULL);
            uint64_t big = 0;
            for (int i = 0; i < n; ++i) {
                seed = mix64(seed + 0x9e3779b97f4a7c15ULL);
                const double v = (double)(seed >> 11) * (2.0 / 9007199254740992.0) - 1.0;
                z[i * iu] = v;
                big = max(big, abs_bits(v));
            }
            bmax = __longlong_as_double((long long)big);
        }
        const int maxits = 5, extra = 2;
        const double dtpcrt = sqrt(0.1 / (double)n);
        int nrmchk = 0, its = 0;
        bool ok = false;
        while (its < maxits) {
            ++its;
            double nrm = 0.0;
            if (!REST || (its > 1 && lane == 0)) {
                // scale: scl = n * onenrm * max(eps, |u_nn|) / ||b||_inf
                const double scl = (double)n * onenrm * fmax(kEps, fabs(unn)) / bmax;
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
                                const double yk = __dmul_rn(cz[q], scl);
                                const bool sw = cp[q] != 0;
                                const double top = sw ? yk : yprev;
                                yprev = fma(-cm[q], top, sw ? yprev : yk);
                                z[(k - 1) * iu] = top;
                            }
                        }
                    }
                    z[(n - 1) * iu] = yprev;
                }
                // backward with perturbation of tiny pivots
                uint64_t big = 0;
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
                        cr[q] = recip(ca[q]);   // of use for mid-range pivots only
                    }
                    if (k0 - IV_U >= 0) fetch(k0 - IV_U);
#pragma unroll
                    for (int q = 0; q < IV_U; ++q) {
                        const int k = k0 - q;
                        if (k >= 0) {
                            double temp = cz[q];
                            if (k <= n - 2) temp = fma(-cb[q], y1, temp);
                            if (k <= n - 3) temp = fma(-cd[q], y2, temp);
                            double ak = ca[q], yk;
                            if (mid_expo(ak) && mid_expo(temp)) {
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
                            big = max(big, abs_bits(yk));
                            y2 = y1;
                            y1 = yk;
                        }
                    }
                }
                nrm = __longlong_as_double((long long)big);
            }
            if (!first) break;   // the other members go on in k_invit<1>
            if (REST) {
                // modified Gram-Schmidt against earlier cluster members
                __syncwarp(mask);
                double dot = 0.0;
                uint64_t big = 0;
                mgs_pass(mask, n, iu, z, nullptr, 0.0, Zb + js, &dot, &big);
                for (int q = js; q < j; ++q) mgs_pass(mask, n, iu, z, Zb + q, dot, q + 1 < j ? Zb + q + 1 : nullptr, &dot, &big);
                __syncwarp(mask);
                nrm = __longlong_as_double((long long)big);
            }
            bmax = nrm;
            if (!(nrm >= dtpcrt)) continue;
            ++nrmchk;
            if (nrmchk < extra + 1) continue;
            ok = true;
            break;
        }
        if (!first) return;
        if (!ok && lane == 0) atomicAdd(g.fail + b, 1);
        // normalise (2-norm), largest component positive
        if (REST) {
            double s2 = 0.0;
            uint64_t big = 0;
            mgs_pass(mask, n, iu, z, nullptr, 0.0, z, &s2, &big);
            // the first row that holds the largest component
            int at = n;
            for (int i = lane; i < n && at == n; i += IV_G)
                if (abs_bits(z[(int64_t)i * iu]) == big) at = i;
#pragma unroll
            for (int o = IV_G / 2; o > 0; o >>= 1) at = min(at, __shfl_xor_sync(mask, at, o, IV_G));
            double scl = 1.0 / sqrt(s2);
            if (at < n && z[(int64_t)at * iu] < 0.0) scl = -scl;
            __syncwarp(mask);
            for (int i = lane; i < n; i += IV_G) z[(int64_t)i * iu] *= scl;
            __syncwarp(mask);
            continue;
        }
        double s2 = 0.0, bigv = 0.0;
        uint64_t big = 0;
#pragma unroll 16
        for (int i = 0; i < n; ++i) {
            const double v = z[i * iu];
            s2 += v * v;
            if (abs_bits(v) > big) {
                big = abs_bits(v);
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
    a.w0 = g.w0;
    a.limbs = g.limbs;
    a.limb_f = g.limb_f;
    a.limb_tiles = g.limb_tiles;
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
    const unsigned by = (unsigned)batch;
    auto grid = [&](int G) { return dim3((unsigned)((iu * G + 31) / 32), by); };   // one warp a CTA: spread over the SMs
    // FP32 counts are latency-bound up to four warps a scheduler
    const bool wide32 = iu * batch * 8 <= 152 * 4 * 4 * 32;
    if (wide32)
        k_bisect_f32<8><<<grid(8), 32, 0, st>>>(g.tf, n, iu, g.iu_lim, g.info, lam);
    else
        k_bisect_f32<4><<<grid(4), 32, 0, st>>>(g.tf, n, iu, g.iu_lim, g.info, lam);
    FORGE_LAUNCH_CHECK();
    // full FP64 accuracy in both precisions: the eigenvectors of close eigenvalues need it (where k_bisect_replay
    // follows, to 4 eps |T|).  Lanes per eigenvalue: four warps fill the FP64 pipes of an SM (152 x 128 lanes);
    // beyond that more points a round only add work
    const int64_t lanes = 152 * 128;
    const int G = iu * batch * 8 <= lanes ? 8 : iu * batch * 4 <= lanes + lanes / 4 ? 4 : iu * batch <= lanes ? 2 : 1;
    const double abstol = g.replay ? 4.0 * kEps : 8.636168555094445e-78;   // at least 2^-256
    if (G == 8)
        k_bisect<8><<<grid(8), 32, 0, st>>>(g.de, n, iu, g.iu_lim, g.info, abstol, lam);
    else if (G == 4)
        k_bisect<4><<<grid(4), 32, 0, st>>>(g.de, n, iu, g.iu_lim, g.info, abstol, lam);
    else if (G == 2)
        k_bisect<2><<<grid(2), 32, 0, st>>>(g.de, n, iu, g.iu_lim, g.info, abstol, lam);
    else
        k_bisect<1><<<grid(1), 32, 0, st>>>(g.de, n, iu, g.iu_lim, g.info, abstol, lam);
    FORGE_LAUNCH_CHECK();
    if (g.replay) {
        k_tri_quot<<<dim3((unsigned)std::min<int64_t>((n + 255) / 256, 64), by), 256, 0, st>>>(g.d, g.e, n, g.de, g.tq);
        FORGE_LAUNCH_CHECK();
        if (wide32)
            k_bisect_qf<3><<<grid(8), 32, 0, st>>>(g.tq, n, iu, g.iu_lim, g.info, lam, g.w);
        else
            k_bisect_qf<2><<<grid(4), 32, 0, st>>>(g.tq, n, iu, g.iu_lim, g.info, lam, g.w);
        FORGE_LAUNCH_CHECK();
        if (G == 8)
            k_bisect_replay<3><<<grid(8), 32, 0, st>>>(g.de, n, iu, g.iu_lim, g.info, lam, g.w);
        else if (G == 4)
            k_bisect_replay<2><<<grid(4), 32, 0, st>>>(g.de, n, iu, g.iu_lim, g.info, lam, g.w);
        else
            k_bisect_replay<1><<<grid(1), 32, 0, st>>>(g.de, n, iu, g.iu_lim, g.info, lam, g.w);
        FORGE_LAUNCH_CHECK();
    }
    prof_end(ST_BISECT, batch * 16.0 * n, batch * 10.0 * 60.0 * (double)n * iu);
    FORGE_CUDA(cudaMemsetAsync(g.fail, 0, sizeof(int) * batch, st));
    prof_begin(ST_INVIT);
    // columns beyond a slot's own nUpper
    if (g.iu_lim) FORGE_CUDA(cudaMemsetAsync(g.Z, 0, sizeof(double) * (size_t)batch * n * iu, st));
    k_clusters<<<(unsigned)batch, 256, 0, st>>>(g.w, iu, g.iu_lim, g.info, g.ortol_rel, g.clus);
    FORGE_LAUNCH_CHECK();
    InvitArgs v;
    v.d = g.d;
    v.e = g.e;
    v.w = g.w;
    v.info = g.info;
    v.lim = g.iu_lim;
    v.clus = g.clus;
    v.n = n;
    v.iu = iu;
    v.ortol_rel = g.ortol_rel;
    v.Z = g.Z;
    v.scr = g.scr;
    v.pivs = g.pivs;
    v.fail = g.fail;
    k_invit_lu<<<grid(1), 32, 0, st>>>(v);
    FORGE_LAUNCH_CHECK();
    k_invit<0><<<grid(1), 32, 0, st>>>(v);
    FORGE_LAUNCH_CHECK();
    k_invit<1><<<grid(IV_G), 32, 0, st>>>(v);
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
    const int64_t nrb = 4;   // slots of the panel dots
    g.ystride = nblk * n;
    g.sstride = nrb * 2 * TRD_NB;
    g.pstride = 3 * ((n + 15) / 16);  // per-CTA partials of k_col64 and k_finish64
    g.d = c.take<double>(B * n);
    g.e = c.take<double>(B * n);
    g.info = c.take<double>(B * 8);
    g.clus = c.take<int>(B * (iu + 2));
    g.pivs = c.take<unsigned char>(n * iu * B);
    g.fail = c.take<int>(B);
    g.tf = c.take<float2>(B * n);
    g.de = c.take<double2>(B * n);
    if (g.mixed) {
        // the reduction and the back-transformation have their own workspace (eig_mixed.cu)
        g.Z = c.take<double>(B * n * iu);
        g.scr = c.take<double>(4 * n * iu * B);
        g.tq = c.take<float>(B * 2 * n);
        return;
    }
    g.tau = c.take<double2>(B * n);
    g.Wp = c.take<double2>(B * n * TRD_NB);
    g.w0 = c.take<double2>(B * n);
    g.Yrow = c.take<double2>(B * g.ystride);
    g.Ycol = c.take<double2>(B * g.ystride);
    g.Spart = c.take<double2>(B * g.sstride);
    g.part = c.take<double>(B * g.pstride);
    g.scal = c.take<double>(B * 16);
    OzSizes z;
    oz_sizes(n, iu, B, g.lean, z);
    // the slices of X (and of the rank-2k update) share the scratch of the inverse iteration, those of V its
    // vectors: both are free before it, and again once Z has been copied to X
    g.Z = (double*)c.take<char>(std::max<size_t>(sizeof(double) * B * n * iu, 2 * z.vr));
    g.oz_vr = g.Z;
    g.scr = (double*)c.take<char>(std::max<size_t>(sizeof(double) * 4 * n * iu * B, 2 * std::max(z.xs, z.uz)));
    g.oz_xs = g.scr;
    // the trailing matrix in limbs (tridiagonalisation) shares the space of V^H (back-transformation)
    g.limb_tiles = nblk * (nblk + 1) / 2;
    g.oz_vh = c.take<char>(std::max<size_t>(2 * z.vh, sizeof(int4) * B * g.limb_tiles * TRD_TILE * TRD_TILE));
    g.limbs = (int4*)g.oz_vh;
    g.limb_f = c.take<int>(B * g.limb_tiles * 2 * TRD_TILE);
    g.oz_ws = c.take<char>(2 * z.ws);
    g.oz_ts = c.take<char>(2 * z.ts);
    g.oz_wp = c.take<double2>(z.wp);
    g.oz_g = c.take<double2>(z.g);
    g.oz_t = c.take<double2>(z.g);
    g.oz_ex = c.take<int>(z.ex);
    g.oz_err = c.take<int>(1);
}
}  // namespace

size_t eig_workspace_bytes(int64_t n, int64_t iu, int64_t batch, bool mixed, bool lean) {
    EigArgs g{};
    g.mixed = mixed;
    g.lean = lean;
    g.n = n;
    g.iu = iu;
    g.batch = batch;
    Carve c{nullptr};
    carve(g, c);
    return c.off;
}

int eig_bind_workspace(EigArgs& g, void* base, size_t bytes) {
    Carve c{static_cast<char*>(base)};
    carve(g, c);
    if (c.off > bytes) {
        set_error(FORGE_ERR_ARG, "eigen-solver: %zu bytes of workspace for a batch that needs %zu", bytes, c.off);
        return FORGE_ERR_ARG;
    }
    return 0;
}

}  // namespace forge

namespace forge {
namespace {
__global__ void k_selftest_sturm(const double2* de, const float2* tf, int n, int64_t nx, const double* x, int* c64, int* c32) {
    const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (q >= nx) return;
    c64[q] = sturm<double>(de, n, x[q]);
    c32[q] = sturm<float>(tf, n, (float)x[q]);
}
// counts of quot(a, b) that differ from a / b, and of those that differ by more than a unit in the last place
__global__ void k_selftest_quot(uint64_t seed, int64_t per_thread, unsigned long long* bad) {
    uint64_t s = mix64(seed ^ ((blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) * 0x9e3779b97f4a7c15ULL));
    unsigned long long off = 0, far = 0, seen = 0;
    for (int64_t i = 0; i < per_thread; ++i) {
        const uint64_t x = mix64(s += 0x9e3779b97f4a7c15ULL), y = mix64(s += 0x9e3779b97f4a7c15ULL);
        // exponents over the range that mid_expo admits, and in half of the cases close to each other
        const int ex = 524 + (int)(mix64(x ^ 1) % 1000), ey = i & 1 ? 524 + (int)(mix64(y ^ 1) % 1000) : ex;
        const double a = __longlong_as_double((long long)((x & 0x800fffffffffffffULL) | (uint64_t)ex << 52));
        const double b = __longlong_as_double((long long)((y & 0x800fffffffffffffULL) | (uint64_t)ey << 52));
        if (!mid_expo(a) || !mid_expo(b)) continue;
        ++seen;
        const long long d = __double_as_longlong(quot(a, b, recip(b))) - __double_as_longlong(a / b);
        off += d != 0;
        far += d > 1 || d < -1;
    }
    atomicAdd(bad, seen);
    atomicAdd(bad + 1, off);
    atomicAdd(bad + 2, far);
}
}  // namespace
}  // namespace forge

extern "C" int forge_gpu_selftest_sturm(int64_t n, const double* d, const double* e, int64_t nx, const double* x, int* c64,
                                        int* c32) {
    using namespace forge;
    if (n < 1 || nx < 1 || !d || !x || !c64 || !c32 || (n > 1 && !e)) {
        set_error(FORGE_ERR_ARG, "selftest_sturm: bad arguments");
        return FORGE_ERR_ARG;
    }
    std::vector<double2> de(n);
    std::vector<float2> tf(n);
    for (int64_t i = 0; i < n; ++i) {
        const double em = i > 0 ? e[i - 1] : 0.0;
        de[i] = make_double2(d[i], em * em);
        tf[i] = make_float2((float)d[i], (float)(em * em));
    }
    DevBuf a, b, p, c;
    int rc = 0;
    if (!(rc = a.ensure(n * sizeof(double2))) && !(rc = b.ensure(n * sizeof(float2))) && !(rc = p.ensure(nx * 8)) &&
        !(rc = c.ensure(nx * 8))) {
        int *g64 = c.as<int>(), *g32 = g64 + nx;
        cudaMemcpy(a.ptr, de.data(), n * sizeof(double2), cudaMemcpyHostToDevice);
        cudaMemcpy(b.ptr, tf.data(), n * sizeof(float2), cudaMemcpyHostToDevice);
        cudaMemcpy(p.ptr, x, nx * 8, cudaMemcpyHostToDevice);
        k_selftest_sturm<<<(unsigned)((nx + 63) / 64), 64>>>(a.as<double2>(), b.as<float2>(), (int)n, nx, p.as<double>(), g64, g32);
        cudaMemcpy(c64, g64, nx * 4, cudaMemcpyDeviceToHost);
        cudaMemcpy(c32, g32, nx * 4, cudaMemcpyDeviceToHost);
        const cudaError_t err = cudaGetLastError();
        if (err != cudaSuccess) {
            set_error(FORGE_ERR_CUDA, "selftest_sturm: %s", cudaGetErrorString(err));
            rc = FORGE_ERR_CUDA;
        }
    }
    for (DevBuf* q : {&a, &b, &p, &c}) q->release();
    return rc;
}

extern "C" int forge_gpu_selftest_quot(int64_t seed, int64_t count, int64_t* out) {
    using namespace forge;
    if (count < 1 || !out) {
        set_error(FORGE_ERR_ARG, "selftest_quot: bad arguments");
        return FORGE_ERR_ARG;
    }
    constexpr int64_t threads = 1216 * 128;
    DevBuf c;
    FORGE_TRY(c.ensure(3 * sizeof(int64_t)));
    cudaMemset(c.ptr, 0, 3 * sizeof(int64_t));
    k_selftest_quot<<<1216, 128>>>((uint64_t)seed, (count + threads - 1) / threads, c.as<unsigned long long>());
    const cudaError_t err = cudaMemcpy(out, c.ptr, 3 * sizeof(int64_t), cudaMemcpyDeviceToHost);
    c.release();
    if (err != cudaSuccess) {
        set_error(FORGE_ERR_CUDA, "selftest_quot: %s", cudaGetErrorString(err));
        return FORGE_ERR_CUDA;
    }
    return 0;
}

extern "C" int forge_selftest_eig_workspace(int64_t n, int64_t iu, int64_t batch, int mixed, int64_t* out) {
    using namespace forge;
    if (n < 2 || iu < 1 || iu > n || batch < 1 || !out) {
        set_error(FORGE_ERR_ARG, "selftest_eig_workspace: bad arguments");
        return FORGE_ERR_ARG;
    }
    if (mixed) {
        eig_mixed_splits(n, iu, batch, out + 1);
        out[0] = (int64_t)(eig_mixed_workspace_bytes(n, iu, batch) + eig_workspace_bytes(n, iu, batch, true));
        return 0;
    }
    OzSizes z;
    oz_sizes(n, iu, batch, false, z);
    out[0] = (int64_t)eig_workspace_bytes(n, iu, batch, false);
    out[1] = z.ks * batch;
    out[2] = z.wp / (iu * z.NB);
    out[3] = out[4] = 0;
    return 0;
}
