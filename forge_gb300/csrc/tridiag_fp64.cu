// Householder tridiagonalisation in FP64 (see tridiag.cuh for the blocked algorithm), three launches a column:
//
//   k_col64   : w_{i-1} += alpha2 v_{i-1} of the previous column, column col minus the panel's reflectors, partial
//               sums of its norm;
//   k_hemv64  : z = A22 x (strict triangles) over 64 x 64 tiles, the panel dots W^H x and V^H x, and, in one
//               CTA, the reflector's scalars (zlarfg) from the norm.  The product takes the raw column x without
//               its first element, so that it does not wait for the norm: v = e1 + s x and
//               A22 v = A22(:, 1) + s (z + D x) are formed in k_finish64;
//   k_finish64: y = A22 v - V (W^H v) - W (V^H v), w = tau y, v into A, partial sums of w^H v.
//
// k_hemv64 has eight FP64 FMAs per element to do, four clocks an element on an SM with two FP64 lanes a clock,
// where HBM delivers an element in 0.7 clocks and the integer pipe does 64 32 x 32 + 64 bit
// multiply-adds a clock.  So the product runs in integers: the tile and the two segments of x
// are block floating point (one power of two for each tile and each segment, 55 bits below it), every
// value is two 28-bit limbs and a product three multiply-adds, summed exactly in int64; only the
// 128 results of a tile are converted to FP64.  An element keeps 2^-55 of its tile's maximum (FP64
// keeps 2^-53 of its own value); the dropped low x low limb products are below 2^-56 of the two maxima
// each, of random sign.  |hi|, |lo| <= 2^27 and at most 256 products a sum stay below 2^62.  Bound: integer pipe (about 60 instructions an element) with HBM close behind.
#include <algorithm>

#include "cvec.cuh"
#include "forge_internal.cuh"
#include "tridiag.cuh"

namespace forge {

namespace {

constexpr int HT = 64;          // tile edge of k_hemv64
constexpr int FR = 32;          // rows per CTA of k_col64 / k_finish64 (8 threads a row)
// panel dots: a CTA takes 8 reflectors over 128 rows.  An FP64 instruction occupies a quarter of the SM's pipe
// for 62 clocks, so few rows per CTA keep the dots shorter than the tiles, and few slots keep their
// sum in k_finish64 short
constexpr int DOT_ROWS = 128, DOT_L = 8;

// partial sums: [0, np) norm of the column (k_col64), then np pairs w^H v (k_finish64)
__device__ inline int64_t parts_of(int64_t n) { return (n + FR - 1) / FR; }

// alpha2 = -1/2 tau (w^H v) of the last column from the nd partials of k_finish64, by one warp
__device__ inline double2 alpha2_of(const TrdArgs<double>& a, int64_t b, int64_t nd) {
    const double* part = a.part + b * a.pstride + parts_of(a.n);
    double2 s = make_double2(0.0, 0.0);
#pragma unroll 4
    for (int64_t q = threadIdx.x & 31; q < nd; q += 32) s = vadd(s, make_double2(part[2 * q], part[2 * q + 1]));
    s = warp_sum(s);
    const double tr = a.scal[b * 16 + 4], ti = a.scal[b * 16 + 5];
    return make_double2(-0.5 * (tr * s.x - ti * s.y), -0.5 * (tr * s.y + ti * s.x));
}

// 32 rows a CTA, 8 threads a row share the panel's reflectors; column ii - 1 of W is still w0
__global__ void __launch_bounds__(256) k_col64(TrdArgs<double> a, int64_t p, int ii, int64_t col) {
    const int64_t b = blockIdx.y, n = a.n, lda = a.lda;
    double2* A = a.A + b * a.strideA;
    double2* W = a.W + b * (n * TRD_NB);
    const double2* w0 = a.w0 + b * n;
    __shared__ double2 wrow[TRD_NB], arow[TRD_NB], s_al, xs[8][FR + 1];
    const int rr = threadIdx.x & 31, sl = threadIdx.x >> 5;
    const int64_t r = col + (int64_t)blockIdx.x * FR + rr;
    const double2 z = make_double2(0.0, 0.0);
    trd_chain_wait();
    // the thread's reflectors l = sl + 8 q, loaded while warp 0 forms alpha2
    double2 x = z, x2 = z, v[4], w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int l = sl + 8 * q;
        const bool ok = r < n && l < ii;
        v[q] = ok ? A[r + (p + l) * lda] : z;
        w[q] = ok ? (l == ii - 1 ? w0[r] : W[r + l * n]) : z;
    }
    if (sl == 1 && rr < ii) {
        arow[rr] = A[col + (p + rr) * lda];
        wrow[rr] = rr == ii - 1 ? w0[col] : W[col + rr * n];
    }
    if (sl == 0) {
        if (r < n) x = A[r + col * lda];
        if (ii > 0) {
            const double2 al = alpha2_of(a, b, (n - col + FR - 1) / FR);
            if (rr == 0) s_al = al;
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int l = sl + 8 * q;
        if (l < ii) {
            double2 wr = wrow[l];
            const double2 ar = arow[l];
            if (l == ii - 1) {
                const double2 al = s_al;
                wr = vadd(wr, vmul(al, ar));
                w[q] = vadd(w[q], vmul(al, v[q]));
                if (r < n) W[r + l * n] = w[q];
            }
            // x -= v conj(wr) + w conj(ar), in two chains
            x.x = fma(-v[q].x, wr.x, fma(-v[q].y, wr.y, x.x));
            x.y = fma(-v[q].y, wr.x, fma(v[q].x, wr.y, x.y));
            x2.x = fma(-w[q].x, ar.x, fma(-w[q].y, ar.y, x2.x));
            x2.y = fma(-w[q].y, ar.x, fma(w[q].x, ar.y, x2.y));
        }
    }
    xs[sl][rr] = x = vadd(x, x2);
    __syncthreads();
    if (sl != 0) return;
    double nrm = 0.0;
    if (r < n) {
        if (ii > 1)   // slices beyond ii are zero
            x = vadd(vadd(vadd(x, xs[1][rr]), vadd(xs[2][rr], xs[3][rr])),
                     vadd(vadd(xs[4][rr], xs[5][rr]), vadd(xs[6][rr], xs[7][rr])));
        if (r == col) {
            x.y = 0.0;
            a.d[b * n + col] = x.x;
        }
        A[r + col * lda] = x;
        if (r == col + 1) {
            a.scal[b * 16] = x.x;
            a.scal[b * 16 + 1] = x.y;
        }
        if (r >= col + 2) nrm = x.x * x.x + x.y * x.y;
    }
    nrm = warp_sum_d(nrm);
    if (rr == 0) a.part[b * a.pstride + blockIdx.x] = nrm;
}

// w_i += alpha2 v_i of the panel's last column (the rank-2k update reads W)
__global__ void __launch_bounds__(256) k_fix64(TrdArgs<double> a, int ii, int64_t col) {
    const int64_t b = blockIdx.y, n = a.n;
    __shared__ double2 s_al;
    trd_chain_wait();
    if (threadIdx.x < 32) {
        const double2 al = alpha2_of(a, b, (n - col - 1 + FR - 1) / FR);
        if (threadIdx.x == 0) s_al = al;
    }
    __syncthreads();
    const int64_t r = col + 1 + (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (r < n)
        a.W[b * (n * TRD_NB) + r + ii * n] = vadd(a.w0[b * n + r], vmul(s_al, a.A[b * a.strideA + r + col * a.lda]));
}

// ---------------------------------------------------------------- block floating point
__device__ inline int field_of(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
// x = (hi 2^28 + lo) 2^(fs - 1022 - 55) up to a unit, |hi| <= 2^27, |lo| <= 2^27, for field_of(x) <= fs and
// 64 <= fs (zeros and values below 2^-1022 then shift out)
__device__ __forceinline__ void limbs(double x, int fs, int& hi, int& lo) {
    const int h = __double2hiint(x), s = h >> 31;
    const unsigned long long m =
        (((unsigned long long)((h & 0xfffff) | 0x100000) << 32) | (unsigned)__double2loint(x)) << 2;
    const unsigned long long v = m >> min(fs - ((h >> 20) & 0x7ff), 63);
    const int l = (int)((unsigned)v & 0xfffffff), c = l >> 27;   // balanced low limb
    hi = (((int)(v >> 28) + c) ^ s) - s;
    lo = ((l - (c << 28)) ^ s) - s;
}
__device__ __forceinline__ void mad(long long& acc, int x, int y) { acc += (long long)x * y; }
__device__ __forceinline__ long long shfl_xor64(long long v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }

// scale 2^(fa + fv - 2 * 1022 - 82) of H 2^28 + M, a sum of limb products; NaN if an operand was not finite
__device__ inline double limb_scale(int fa, int fv) {
    if (fa == 2047 || fv == 2047) return __longlong_as_double(0x7ff8000000000000LL);
    const int k = fa + fv - 2044 - 82;
    return k > -1022 && k < 1023 ? __hiloint2double((1023 + k) << 20, 0) : ldexp(1.0, k);
}

__global__ void __launch_bounds__(256, 2) k_hemv64(TrdArgs<double> a, int64_t p, int ii, int64_t col, int64_t ndot) {
    const int64_t b = blockIdx.y, n = a.n, lda = a.lda, c0 = col + 1;
    const double2* __restrict__ A = a.A + b * a.strideA;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    trd_chain_wait();
    // the scalars' CTA and the dots (chains of FP64 instructions) go first
    const int64_t t = (int64_t)blockIdx.x - 1 - ndot;
    if (t >= 0) {
        // tile (bi, bj), bj <= bi; t = bi (bi + 1) / 2 + bj
        int64_t bi = (int64_t)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);   // corrected below
        while ((bi + 1) * (bi + 2) / 2 <= t) ++bi;
        while (bi * (bi + 1) / 2 > t) --bi;
        const int64_t bj = t - bi * (bi + 1) / 2;
        const int64_t R0 = c0 + bi * HT, C0 = c0 + bj * HT;
        __shared__ int4 vr[HT], vc[HT];              // limbs (re hi, re lo, im hi, im lo) of x
        __shared__ int redA[8], redV[4];
        __shared__ long long rs[8][HT][4], cs[HT][4];   // sums: H re, H im, M re, M im
        const int tr = tid & 15, tc = tid >> 4;
        double2 xv = make_double2(0.0, 0.0);
        if (tid < 2 * HT) {
            const int64_t r = tid < HT ? R0 + tid : C0 + tid - HT;
            if (r < n && r > c0) xv = A[r + col * lda];
        }
        double2 e[4][4];   // strict lower triangle
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int64_t r = R0 + tr + 16 * i, c = C0 + tc * 4 + j;
                e[i][j] = (r < n && c < r) ? A[r + c * lda] : make_double2(0.0, 0.0);
            }
        int f = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) f = max(f, max(field_of(e[i][j].x), field_of(e[i][j].y)));
        f = __reduce_max_sync(0xffffffffu, f);
        if (lane == 0) redA[warp] = f;
        if (warp < 4) {
            const int g = __reduce_max_sync(0xffffffffu, max(field_of(xv.x), field_of(xv.y)));
            if (lane == 0) redV[warp] = g;
        }
        __syncthreads();
        int fa = max(redA[0], 64);
#pragma unroll
        for (int q = 1; q < 8; ++q) fa = max(fa, redA[q]);
        const int fr = max(max(redV[0], redV[1]), 64), fc = max(max(redV[2], redV[3]), 64);
        if (tid < 2 * HT) {
            int4 l;
            const int fx = tid < HT ? fr : fc;
            limbs(xv.x, fx, l.x, l.y);
            limbs(xv.y, fx, l.z, l.w);
            (tid < HT ? vr[tid] : vc[tid - HT]) = l;
        }
        __syncthreads();
        // rows: a x, summed over the thread's four columns; columns: conj(a) x, over its four rows
        long long row[4][4], s[16];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int k = 0; k < 4; ++k) row[i][k] = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int4 y = vc[tc * 4 + j];
            const int nz = -y.z, nw = -y.w;
            long long hr = 0, hi = 0, mr = 0, mi = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                int4 x;
                limbs(e[i][j].x, fa, x.x, x.y);
                limbs(e[i][j].y, fa, x.z, x.w);
                long long* R = row[i];
                mad(R[0], x.x, y.x); mad(R[0], x.z, nz);
                mad(R[1], x.x, y.z); mad(R[1], x.z, y.x);
                mad(R[2], x.x, y.y); mad(R[2], x.y, y.x); mad(R[2], x.z, nw); mad(R[2], x.w, nz);
                mad(R[3], x.x, y.w); mad(R[3], x.y, y.z); mad(R[3], x.z, y.y); mad(R[3], x.w, y.x);
                const int4 u = vr[tr + 16 * i];
                x.z = -x.z;
                x.w = -x.w;
                mad(hr, x.x, u.x); mad(hr, x.z, -u.z);
                mad(hi, x.x, u.z); mad(hi, x.z, u.x);
                mad(mr, x.x, u.y); mad(mr, x.y, u.x); mad(mr, x.z, -u.w); mad(mr, x.w, -u.z);
                mad(mi, x.x, u.w); mad(mi, x.y, u.z); mad(mi, x.z, u.y); mad(mi, x.w, u.x);
            }
            s[4 * j] = hr;
            s[4 * j + 1] = hi;
            s[4 * j + 2] = mr;
            s[4 * j + 3] = mi;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const long long v = row[i][k] + shfl_xor64(row[i][k], 16);
                if (lane < 16) rs[warp][tr + 16 * i][k] = v;
            }
        // columns over the 16 lanes of the row index: at each step a lane keeps half of its values and adds the
        // partner's half
#pragma unroll
        for (int w = 8; w > 0; w >>= 1) {
            const bool up = (lane & w) != 0;
#pragma unroll
            for (int k = 0; k < w; ++k) {
                const long long send = up ? s[k] : s[k + w];
                s[k] = (up ? s[k + w] : s[k]) + shfl_xor64(send, w);
            }
        }
        cs[tc * 4 + (tr >> 2)][tr & 3] = s[0];
        __syncthreads();
        // 128 results: rows (threads 0..127) and columns, real and imaginary parts
        const int u = (tid & 127) >> 1, im = tid & 1;
        if (tid < 128) {
            long long H = 0, M = 0;
#pragma unroll
            for (int w = 0; w < 8; ++w) {
                H += rs[w][u][im];
                M += rs[w][u][2 + im];
            }
            if (R0 + u < n)
                reinterpret_cast<double*>(a.Yrow + b * a.ystride + bj * n + R0 + u)[im] =
                    fma((double)H, 268435456.0, (double)M) * limb_scale(fa, fc);
        } else if (C0 + u < n) {
            reinterpret_cast<double*>(a.Ycol + b * a.ystride + bi * n + C0 + u)[im] =
                fma((double)cs[u][im], 268435456.0, (double)cs[u][2 + im]) * limb_scale(fa, fr);
        }
    } else if (blockIdx.x > 0) {
        // panel dots: warp <-> reflector, lanes over the rows
        const int ng = (ii + DOT_L - 1) / DOT_L;
        const int64_t rb = ((int64_t)blockIdx.x - 1) / ng;
        const int lg = (int)((int64_t)blockIdx.x - 1 - rb * ng) * DOT_L, l = lg + warp;
        const double2* W = a.W + b * (n * TRD_NB);
        double2 s1 = make_double2(0.0, 0.0), s2 = s1;
        if (l < ii) {
            double2 v[DOT_ROWS / 32], w[DOT_ROWS / 32], h[DOT_ROWS / 32];
#pragma unroll
            for (int k = 0; k < DOT_ROWS / 32; ++k) {
                const int64_t r = c0 + rb * DOT_ROWS + lane + 32 * k;
                const bool ok = r < n && r > c0;
                v[k] = ok ? A[r + col * lda] : make_double2(0.0, 0.0);
                w[k] = ok ? W[r + l * n] : make_double2(0.0, 0.0);
                h[k] = ok ? A[r + (p + l) * lda] : make_double2(0.0, 0.0);
            }
#pragma unroll
            for (int k = 0; k < DOT_ROWS / 32; ++k) {
                s1.x = fma(w[k].x, v[k].x, fma(w[k].y, v[k].y, s1.x));
                s1.y = fma(w[k].x, v[k].y, fma(-w[k].y, v[k].x, s1.y));
                s2.x = fma(h[k].x, v[k].x, fma(h[k].y, v[k].y, s2.x));
                s2.y = fma(h[k].x, v[k].y, fma(-h[k].y, v[k].x, s2.y));
            }
        }
        // over the lanes: a lane keeps half of the four sums at the first two steps
        __shared__ double red[8][4][9];
        {
            const bool u1 = (lane & 16) != 0, u2 = (lane & 8) != 0;
            double a0 = u1 ? s2.x : s1.x, a1 = u1 ? s2.y : s1.y;
            a0 += __shfl_xor_sync(0xffffffffu, u1 ? s1.x : s2.x, 16);
            a1 += __shfl_xor_sync(0xffffffffu, u1 ? s1.y : s2.y, 16);
            double c = u2 ? a1 : a0;
            c += __shfl_xor_sync(0xffffffffu, u2 ? a0 : a1, 8);
            red[warp][(u1 ? 2 : 0) + (u2 ? 1 : 0)][lane & 7] = c;
        }
        __syncthreads();
        if (tid < 32) {
            // thread: reflector tid >> 2 of the group, component tid & 3
            const double* q = red[tid >> 2][tid & 3];
            const double sum = ((q[0] + q[1]) + (q[2] + q[3])) + ((q[4] + q[5]) + (q[6] + q[7]));
            const int lo = lg + (tid >> 2);
            double* S = reinterpret_cast<double*>(a.Spart + b * a.sstride + rb * 2 * TRD_NB);
            if (lo < ii) S[2 * (((tid >> 1) & 1) * TRD_NB + lo) + (tid & 1)] = sum;
        }
    } else if (warp == 0) {
        // zlarfg: beta = -sign(|(alpha, x)|, Re alpha), tau = (beta - alpha)/beta, s = 1/(alpha - beta)
        const int64_t np = (n - col + FR - 1) / FR;
        double xn2 = 0.0;
        for (int64_t q = lane; q < np; q += 32) xn2 += a.part[b * a.pstride + q];
        xn2 = warp_sum_d(xn2);
        if (lane == 0) {
            double* sc = a.scal + b * 16;
            const double ar = sc[0], ai = sc[1];
            double sr = 1.0, si = 0.0, tr = 0.0, ti = 0.0, beta = ar;
            if (!(xn2 == 0.0 && ai == 0.0)) {
                beta = -copysign(sqrt(ar * ar + ai * ai + xn2), ar);
                tr = (beta - ar) / beta;
                ti = -ai / beta;
                const double dr = ar - beta, den = dr * dr + ai * ai;
                sr = dr / den;
                si = -ai / den;
            }
            sc[2] = sr;
            sc[3] = si;
            sc[4] = tr;
            sc[5] = ti;
            a.tau[b * n + col] = make_double2(tr, ti);
            a.e[b * n + col] = beta;
        }
    }
}

// 32 rows a CTA, 8 threads a row
__global__ void __launch_bounds__(256) k_finish64(TrdArgs<double> a, int64_t p, int ii, int64_t col, int64_t nb2,
                                                  int64_t ndot) {
    const int64_t b = blockIdx.y, n = a.n, lda = a.lda, c0 = col + 1;
    double2* A = a.A + b * a.strideA;
    const double2* W = a.W + b * (n * TRD_NB);
    __shared__ double2 s1[TRD_NB], s2[TRD_NB], ys[8][FR + 1], sp[8][TRD_NB][2];
    const int rr = threadIdx.x & 31, sl = threadIdx.x >> 5;
    const int64_t r = c0 + (int64_t)blockIdx.x * FR + rr;
    const double2 z = make_double2(0.0, 0.0);
    trd_chain_wait();
    const double* sc = a.scal + b * 16;
    const double2 s = make_double2(sc[2], sc[3]), tau = make_double2(sc[4], sc[5]);
    // loads of the last steps first
    double2 xr = z, ac = z, c0w = z;
    double dg = 0.0;
    if (sl == 0 && r < n) {
        xr = A[r + col * lda];
        ac = A[r + c0 * lda];
        dg = A[r + r * lda].x;
    }
    if (threadIdx.x < 2 * TRD_NB && rr < ii) c0w = sl ? A[c0 + (p + rr) * lda] : W[c0 + rr * n];
    // W^H v = conj(W(c0, :)) + s W^H x and likewise V^H v, from the slots of the panel dots: 8 threads a reflector
    if (rr < ii) {
        double2 d1 = z, d2 = z;
        const double2* S = a.Spart + b * a.sstride + rr;
#pragma unroll 4
        for (int64_t q = sl; q < ndot; q += 8) {
            d1 = vadd(d1, S[q * 2 * TRD_NB]);
            d2 = vadd(d2, S[q * 2 * TRD_NB + TRD_NB]);
        }
        sp[sl][rr][0] = d1;
        sp[sl][rr][1] = d2;
    }
    // the row's partial products
    double2 y = z;
    if (r < n) {
        const int64_t B = (r - c0) / HT;
        const double2* Yrow = a.Yrow + b * a.ystride + r;
        const double2* Ycol = a.Ycol + b * a.ystride + r;
#pragma unroll 4
        for (int64_t q = sl; q <= B; q += 8) y = vadd(y, Yrow[q * n]);
#pragma unroll 4
        for (int64_t q = B + sl; q < nb2; q += 8) y = vadd(y, Ycol[q * n]);
        y = vmul(s, y);
    }
    double2 y2 = z, v[4], w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int l = sl + 8 * q;
        const bool ok = r < n && l < ii;
        v[q] = ok ? A[r + (p + l) * lda] : z;
        w[q] = ok ? W[r + l * n] : z;
    }
    __syncthreads();
    if (threadIdx.x < 2 * TRD_NB) {
        const int l = threadIdx.x & 31, g = threadIdx.x >> 5;
        if (l < ii) {
            double2 d = sp[0][l][g];
            if (ndot > 1)   // slots beyond ndot are zero
                d = vadd(vadd(vadd(d, sp[1][l][g]), vadd(sp[2][l][g], sp[3][l][g])),
                         vadd(vadd(sp[4][l][g], sp[5][l][g]), vadd(sp[6][l][g], sp[7][l][g])));
            (g ? s2 : s1)[l] = vadd(vconj(c0w), vmul(s, d));
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int l = sl + 8 * q;
        if (l < ii) {
            const double2 d1 = s1[l], d2 = s2[l];
            y.x = fma(-v[q].x, d1.x, fma(v[q].y, d1.y, y.x));
            y.y = fma(-v[q].x, d1.y, fma(-v[q].y, d1.x, y.y));
            y2.x = fma(-w[q].x, d2.x, fma(w[q].y, d2.y, y2.x));
            y2.y = fma(-w[q].x, d2.y, fma(-w[q].y, d2.x, y2.y));
        }
    }
    ys[sl][rr] = y = vadd(y, y2);
    __syncthreads();
    if (sl != 0) return;
    double2 dot = make_double2(0.0, 0.0);
    if (r < n) {
        y = vadd(vadd(vadd(y, ys[1][rr]), vadd(ys[2][rr], ys[3][rr])),
                 vadd(vadd(ys[4][rr], ys[5][rr]), vadd(ys[6][rr], ys[7][rr])));
        double2 u = make_double2(1.0, 0.0);
        if (r > c0) {
            // the first column of A22 and s D x
            u = vmul(s, xr);
            y = vadd(y, ac);
            y.x = fma(dg, u.x, y.x);
            y.y = fma(dg, u.y, y.y);
        } else {
            y.x += dg;
        }
        y = vmul(tau, y);
        A[r + col * lda] = u;
        a.w0[b * n + r] = y;
        dot = vcjmul(y, u);   // zdotc(w, v)
    }
    dot = warp_sum(dot);
    if (rr == 0) {
        double* part = a.part + b * a.pstride + parts_of(n) + 2 * blockIdx.x;
        part[0] = dot.x;
        part[1] = dot.y;
    }
}

}  // namespace

int tridiagonalize_fp64(cudaStream_t st, TrdArgs<double>& a, int64_t batch) {
    const int64_t n = a.n;
    const unsigned nbat = (unsigned)batch;
    for (int64_t p = 0; p < n; p += TRD_NB) {
        const int64_t w = std::min<int64_t>(n - p, TRD_NB);
        int64_t nrefl = 0;
        for (int ii = 0; ii < w; ++ii) {
            const int64_t col = p + ii, n2 = n - col - 1;
            prof_begin(ST_TRD_COL);
            FORGE_TRY(launch_chain(st, dim3((unsigned)((n - col + FR - 1) / FR), nbat), 256, k_col64, a, p, ii, col));
            prof_end(ST_TRD_COL, batch * (double)(n - col) * (2.0 * ii + 2.0) * 16.0, 0.0);
            if (n2 <= 0) {
                // the last column has no reflector
                FORGE_CUDA(cudaMemset2DAsync(a.tau + col, n * sizeof(double2), 0, sizeof(double2), batch, st));
                continue;
            }
            ++nrefl;
            const int64_t nb2 = (n2 + HT - 1) / HT, ntiles = nb2 * (nb2 + 1) / 2;
            const int64_t ndot = ii > 0 ? (n2 + DOT_ROWS - 1) / DOT_ROWS : 0;   // slots of the panel dots
            const int64_t ndc = ndot * ((ii + DOT_L - 1) / DOT_L);
            prof_begin(ST_HEMV);
            FORGE_TRY(launch_chain(st, dim3((unsigned)(ntiles + ndc + 1), nbat), 256, k_hemv64, a, p, ii, col, ndc));
            // algorithmic traffic: the trailing lower triangle read once
            prof_end(ST_HEMV, batch * 0.5 * (double)n2 * (double)(n2 + 1) * 16.0, batch * 8.0 * (double)n2 * n2);
            prof_begin(ST_TRD_FINISH);
            FORGE_TRY(launch_chain(st, dim3((unsigned)((n2 + FR - 1) / FR), nbat), 256, k_finish64, a, p, ii, col, nb2, ndot));
            if (ii == w - 1 || col == n - 2) {
                FORGE_TRY(launch_chain(st, dim3((unsigned)((n2 + 255) / 256), nbat), 256, k_fix64, a, ii, col));
            }
            prof_end(ST_TRD_FINISH, batch * (double)n2 * (2.0 * ii + 4.0) * 16.0, 0.0);
        }
        if (nrefl > 0 && p + w < n) {
            const double m2 = (double)(n - p - w);
            prof_begin(ST_HER2K);
            FORGE_TRY(a.her2k(st, a, p, nrefl, batch, a.her2k_user));
            prof_end(ST_HER2K, batch * m2 * m2 * 16.0, batch * 8.0 * m2 * m2 * (double)nrefl);
        }
    }
    return 0;
}

}  // namespace forge
