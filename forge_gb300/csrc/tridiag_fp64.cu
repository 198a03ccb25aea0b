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
// multiply-adds a clock.  So the product runs in integers: a tile is scaled by a power of two for each of its rows and
// columns, so that the largest element of every row and column is about one, a segment of x takes the
// tile's scales along, and both are block floating point (55 bits below the maximum).  Every
// value is two 28-bit limbs and a product three multiply-adds, summed exactly in int64; only the
// 128 results of a tile are converted to FP64.  A scaled element keeps 2^-55 of one (FP64
// keeps 2^-53 of its own value); the dropped low x low limb products are below 2^-56 of the two maxima
// each, of random sign.  The scales make the error of a row follow the row's size, as FP64's does: a graded matrix
// D B D keeps the relative accuracy of its small eigenvalues (with one scale a tile, 1e-10 instead of 1e-13 at a
// ratio of 1e-8, and nothing left at 1e-20).  |hi|, |lo| <= 2^27 and at most 256 products a sum stay below 2^62.  The trailing matrix does
// not change inside a panel (V and W carry its update), so k_limbs64 cuts it once for 32 columns, into as
// many bytes as it had, in the order in which k_hemv64's threads read it.  Bound: integer multiply-adds (24 an element).
// Measured (stage; cut anew in every column before): N = 1324, 16 k 57.6 -> 41 ms, N = 3268, one k 64 -> 53 ms; with an
// exponent for each row and column of a tile, not one for all, 43 and 55 ms.  What
// keeps it from the multiply-adds' rate is their latency: 16 warps an SM (registers) issue on 36% of the clocks.
// k_col64 and k_finish64, with FP64 instructions shared by more lanes and the loads of older results ahead of the
// predecessor's end: the whole reduction N = 3268, one k 103 -> 79 ms; N = 76, nine k 1.5 -> 1.3 ms.
#include <algorithm>

#include "cvec.cuh"
#include "forge_internal.cuh"
#include "tridiag.cuh"

namespace forge {

namespace {

constexpr int HT = 64;          // tile edge of k_hemv64
// k_col64 / k_finish64: eight warps a CTA, RW rows a warp, 32 / RW lanes a row
template <int RW>
constexpr int FR = 8 * RW;
// Panel dots: a warp takes one reflector over dot_rows rows, 128 at a time; at most DOT_SLOTS partial sums a reflector.
constexpr int DOT_ROWS = 128, DOT_L = 4, DOT_SLOTS = 4;

// An FP64 instruction of a warp holds its scheduler's FP64 pipe for 64 clocks, however many lanes are active, so what
// these kernels cost is the number of FP64 instructions along the longest warp (besides the round trips to memory):
// few rows a warp, sums over lanes that halve what a lane carries (re in the lower, im in the upper half
// after the first step), complex products one component a lane.

// sum over the lanes of a row (lane = slice RW + row): re in lanes 0-15, im in lanes 16-31
template <int RW>
__device__ __forceinline__ double row_sum(double2 v) {
    const bool up = threadIdx.x & 16;
    double s = (up ? v.y : v.x) + __shfl_xor_sync(0xffffffffu, up ? v.x : v.y, 16);
#pragma unroll
    for (int o = 8; o >= RW; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}
__device__ __forceinline__ double xor16(double v) { return __shfl_xor_sync(0xffffffffu, v, 16); }

// partial sums: [0, np) norm of the column (k_col64), then np pairs w^H v (k_finish64)
__device__ inline int64_t parts_of(int64_t n, int fr) { return (n + fr - 1) / fr; }

// alpha2 = -1/2 tau (w^H v) of the last column from the partials of k_finish64 (rows rows, fr a partial), by one warp;
// lanes below 16 the real part, the others the imaginary part
__device__ inline double alpha2_of(const TrdArgs<double>& a, int64_t b, int64_t rows, int fr) {
    const double* part = a.part + b * a.pstride + parts_of(a.n, fr);
    const int64_t nd = parts_of(rows, fr);
    const int lane = threadIdx.x & 31, im = lane >> 4;
    const double tr = a.scal[b * 16 + 4], ti = a.scal[b * 16 + 5];
    double s = 0.0;
    for (int64_t q0 = lane & 15; q0 < nd; q0 += 128) {
        double t[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) t[q] = q0 + 16 * q < nd ? part[2 * (q0 + 16 * q) + im] : 0.0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            if (q0 - (lane & 15) + 16 * q >= nd) break;
            s += t[q];
        }
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const double o = xor16(s);
    return -0.5 * fma(tr, s, im ? ti * o : -(ti * o));
}

// column ii - 1 of W is still w0.  The last warp forms alpha2 while the others subtract the older reflectors.
template <int RW>
__global__ void __launch_bounds__(288) k_col64(TrdArgs<double> a, int64_t p, int ii, int64_t col) {
    const int64_t b = blockIdx.y, n = a.n, lda = a.lda;
    double2* A = a.A + b * a.strideA;
    double2* W = a.W + b * (n * TRD_NB);
    const double2* w0 = a.w0 + b * n;
    __shared__ double2 wrow[TRD_NB], arow[TRD_NB], s_al;
    __shared__ double red[8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sl = lane / RW;
    const int64_t r = col + (int64_t)blockIdx.x * FR<RW> + warp * RW + lane % RW;
    const double2 z = make_double2(0.0, 0.0);
    const int lm = ii - 1;
    const bool mine = warp < 8 && r < n;
    double2 x = z, x2 = z, v[RW], w[RW];
#pragma unroll
    for (int q = 0; q < RW; ++q) {
        const int l = sl + 32 / RW * q;
        v[q] = mine && l < lm ? ld_early(A + r + (p + l) * lda) : z;
        w[q] = mine && l < lm ? ld_early(W + r + l * n) : z;
    }
    if (mine && sl == 0) x = ld_early(A + r + col * lda);
    if (warp == 8 && lane < lm) {
        arow[lane] = ld_early(A + col + (p + lane) * lda);
        wrow[lane] = ld_early(W + col + lane * n);
    }
    trd_chain_wait();
    // the last reflector: its v in lanes sl = 0, its w and v in lanes sl = 1
    double2 vl = z, wl = z;
    if (mine && sl < 2 && ii > 0) {
        vl = A[r + (p + lm) * lda];
        if (sl == 1) wl = w0[r];
    }
    __syncthreads();
    if (warp == 8 && ii > 0) {
        const double2 ar = A[col + (p + lm) * lda], wr = w0[col];
        const double al = alpha2_of(a, b, n - col, FR<RW>), ao = xor16(al);
        // w(col) += alpha2 v(col), one component a half
        const bool im = lane >> 4;
        const double t = fma(al, ar.x, im ? fma(ao, ar.y, wr.y) : fma(-ao, ar.y, wr.x));
        if ((lane & 15) == 0) {
            reinterpret_cast<double*>(&wrow[lm])[im] = t;
            reinterpret_cast<double*>(&s_al)[im] = al;
            if (!im) arow[lm] = ar;
        }
    }
#pragma unroll
    for (int q = 0; q < RW; ++q) {
        const int l = sl + 32 / RW * q;
        if (32 / RW * q < lm && warp < 8) {
            const double2 wr = l < lm ? wrow[l] : z, ar = l < lm ? arow[l] : z;
            // x -= v conj(wr) + w conj(ar), in two chains
            x.x = fma(-v[q].x, wr.x, fma(-v[q].y, wr.y, x.x));
            x.y = fma(-v[q].y, wr.x, fma(v[q].x, wr.y, x.y));
            x2.x = fma(-w[q].x, ar.x, fma(-w[q].y, ar.y, x2.x));
            x2.y = fma(-w[q].y, ar.x, fma(w[q].x, ar.y, x2.y));
        }
    }
    __syncthreads();
    if (ii > 0 && warp < 8) {
        const double2 al = s_al;
        const double2 wn = make_double2(fma(al.x, vl.x, fma(-al.y, vl.y, wl.x)), fma(al.x, vl.y, fma(al.y, vl.x, wl.y)));
        if (mine && sl == 1) W[r + lm * n] = wn;
        const double2 f = sl == 0 ? vl : sl == 1 ? wn : z, g = sl == 0 ? wrow[lm] : arow[lm];
        x2.x = fma(-f.x, g.x, fma(-f.y, g.y, x2.x));
        x2.y = fma(-f.y, g.x, fma(f.x, g.y, x2.y));
    }
    if (warp == 8) return;
    double s = row_sum<RW>(vadd(x, x2)), nrm = 0.0;
    if (mine && (lane & 15) < RW) {
        const int im = lane >> 4;
        if (r == col) {
            if (im)
                s = 0.0;
            else
                a.d[b * n + col] = s;
        }
        reinterpret_cast<double*>(A + r + col * lda)[im] = s;
        if (r == col + 1) a.scal[b * 16 + im] = s;
        if (r >= col + 2) nrm = s * s;
    }
#pragma unroll
    for (int o = RW / 2; o > 0; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
    nrm += xor16(nrm);
    if (lane == 0) red[warp] = nrm;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    if (threadIdx.x < 8) {
        nrm = red[threadIdx.x];
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) nrm += __shfl_xor_sync(0xffu, nrm, o);
        if (threadIdx.x == 0) a.part[b * a.pstride + blockIdx.x] = nrm;
    }
}

// w_i += alpha2 v_i of the panel's last column (the rank-2k update reads W)
__global__ void __launch_bounds__(256) k_fix64(TrdArgs<double> a, int ii, int64_t col, int fr) {
    const int64_t b = blockIdx.y, n = a.n;
    __shared__ double2 s_al;
    trd_chain_wait();
    if (threadIdx.x < 32) {
        const double al = alpha2_of(a, b, n - col - 1, fr);
        if ((threadIdx.x & 15) == 0) reinterpret_cast<double*>(&s_al)[threadIdx.x >> 4] = al;
    }
    __syncthreads();
    const int64_t r = col + 1 + (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (r < n)
        a.W[b * (n * TRD_NB) + r + ii * n] = vadd(a.w0[b * n + r], vmul(s_al, a.A[b * a.strideA + r + col * a.lda]));
}

// ---------------------------------------------------------------- block floating point
__device__ inline int field_of(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
// x = (hi 2^28 + lo) 2^(f - 1022 - 55) up to half a unit, |hi| <= 2^27, |lo| <= 2^27, for sh = f - field_of(x) >= 0;
// values below 2^-1022 are zero.  Nearest, ties to even: cut off towards zero, the errors of a
// row of elements of one sign add up (the lowest band of a lattice, n = 364: 1.4e-14 instead of 2e-15).
__device__ __forceinline__ void limbs(double x, int sh, int& hi, int& lo) {
    const int h = __double2hiint(x), s = h >> 31;
    const unsigned long long m =
        (((unsigned long long)((h & 0xfffff) | 0x100000) << 32) | (unsigned)__double2loint(x)) << 2;
    sh = (h >> 20) & 0x7ff ? (int)min((unsigned)sh, 63u) : 63;
    const unsigned long long v = (m + (((1ULL << sh) - 1) >> 1) + ((m >> sh) & 1)) >> sh;
    const int l = (int)((unsigned)v & 0xfffffff), c = l >> 27;   // balanced low limb
    hi = (((int)(v >> 28) + c) ^ s) - s;
    lo = ((l - (c << 28)) ^ s) - s;
}
__device__ __forceinline__ void mad(long long& acc, int x, int y) { acc += (long long)x * y; }
__device__ __forceinline__ long long shfl_xor64(long long v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }

// Exponents (as biased fields) of a tile's row or column without a nonzero element, and of operands that are not finite
constexpr int NO_EXPO = -8192, NAN_EXPO = 1 << 20;
// exponent of x 2^e
__device__ inline int scaled_field(double x, int e) {
    const int f = field_of(x);
    return f == 2047 ? NAN_EXPO : f ? f + e : 2 * NO_EXPO;
}
// scale 2^(fa + fv - 2 * 1022 - 82) of H 2^28 + M, a sum of limb products; NaN if an operand was not finite
__device__ inline double limb_scale(int fa, int fv) {
    if (max(fa, fv) >= NAN_EXPO / 2) return __longlong_as_double(0x7ff8000000000000LL);
    const int k = fa + fv - 2044 - 82;
    return k > -1022 && k < 1023 ? __hiloint2double((1023 + k) << 20, 0) : ldexp(1.0, k);
}

// The strict lower triangle of A(p:n, p:n) in limbs, 64 x 64 tiles (bi, bj), bj <= bi, t = bi (bi + 1) / 2 + bj: element
// (tr + 16 i, 8 tc + j) at (4 j + i) 128 + 16 tc + tr.  To limb_f, 128 a tile: r_i, the exponent of row i's largest
// element, and c_j <= 0, that of column j's largest once the rows are scaled; element (i, j) is in units of
// 2^(r_i + c_j - 1022 - 55).
__device__ inline int64_t tile_row(int64_t t) {
    int64_t bi = (int64_t)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);   // corrected below
    while ((bi + 1) * (bi + 2) / 2 <= t) ++bi;
    while (bi * (bi + 1) / 2 > t) --bi;
    return bi;
}
__global__ void __launch_bounds__(256) k_limbs64(TrdArgs<double> a, int64_t p) {
    const int64_t b = blockIdx.y, n = a.n, lda = a.lda, t = blockIdx.x, bi = tile_row(t), bj = t - bi * (bi + 1) / 2;
    const double2* __restrict__ A = a.A + b * a.strideA;
    const int tid = threadIdx.x, tr = tid & 15, tc = tid >> 4;
    __shared__ int red[8][HT], rexp[HT];
    // thread: rows tr + 16 i, columns tc + 16 q
    double2 e[4][4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int64_t r = p + bi * HT + tr + 16 * i, c = p + bj * HT + tc + 16 * q;
            e[i][q] = (r < n && c < r) ? A[r + c * lda] : make_double2(0.0, 0.0);
        }
    int fe[4][4], r[4], cm[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        int f = 2 * NO_EXPO;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            fe[i][q] = max(scaled_field(e[i][q].x, 0), scaled_field(e[i][q].y, 0));
            f = max(f, fe[i][q]);
        }
        f = max(f, __shfl_xor_sync(0xffffffffu, f, 16));
        if ((tid & 16) == 0) red[tid >> 5][tr + 16 * i] = f;
    }
    __syncthreads();
    if (tid < HT) {
        int f = NO_EXPO;
#pragma unroll
        for (int q = 0; q < 8; ++q) f = max(f, red[q][tid]);
        rexp[tid] = f;
    }
    // an element that is not finite spoils the tile's rows and columns
    const bool bad = __syncthreads_or(tid < HT && rexp[tid] >= NAN_EXPO);
#pragma unroll
    for (int i = 0; i < 4; ++i) r[i] = rexp[tr + 16 * i];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        int f = NO_EXPO;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (fe[i][q] > NO_EXPO) f = max(f, fe[i][q] - r[i]);
#pragma unroll
        for (int k = 8; k > 0; k >>= 1) f = max(f, __shfl_xor_sync(0xffffffffu, f, k));
        cm[q] = f;
    }
    int* ex = a.limb_f + (b * a.limb_tiles + t) * (2 * HT);
    if (tid < HT) ex[tid] = bad ? NAN_EXPO : rexp[tid];
    if (tr == 0) {
#pragma unroll
        for (int q = 0; q < 4; ++q) ex[HT + tc + 16 * q] = bad ? NAN_EXPO : cm[q];
    }
    int4* o = a.limbs + (b * a.limb_tiles + t) * (HT * HT);
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int c = tc + 16 * q;
            int4 x;
            limbs(e[i][q].x, r[i] + cm[q] - field_of(e[i][q].x), x.x, x.y);
            limbs(e[i][q].y, r[i] + cm[q] - field_of(e[i][q].y), x.z, x.w);
            o[(4 * (c & 7) + i) * 128 + 16 * (c >> 3) + tr] = x;
        }
}

constexpr int HV_T = 128;   // threads of k_hemv64
// exchange of the halving butterfly over lane bit w: the lane keeps one of the two and adds the partner's
__device__ __forceinline__ long long halve(long long lo, long long hi, bool up, int w) {
    return (up ? hi : lo) + shfl_xor64(up ? lo : hi, w);
}
__global__ void __launch_bounds__(HV_T, 4) k_hemv64(TrdArgs<double> a, int64_t p, int ii, int64_t col, int64_t ndot,
                                                  int64_t dot_rows, int fr) {
    const int64_t b = blockIdx.y, n = a.n, lda = a.lda, c0 = col + 1;
    const double2* __restrict__ A = a.A + b * a.strideA;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    extern __shared__ int4 tile[];   // a ring of four of the thread's columns, four elements each
    // the scalars' CTA and the dots (chains of FP64 instructions) go first
    const int64_t t = (int64_t)blockIdx.x - 1 - ndot;
    if (t >= 0) {
        // the thread's columns, in an order in which the butterfly's partners follow each other
        constexpr int ORD[8] = {0, 4, 2, 6, 1, 5, 3, 7};
        // The first half of the tile is under way before the column is known: the limbs are older than the
        // predecessor's start.
        const int4* L = a.limbs + (b * a.limb_tiles + t) * (HT * HT) + tid;
        const unsigned to = (unsigned)__cvta_generic_to_shared(tile + tid);
        auto fetch = [&](int q) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + (4 * (q & 3) + i) * (16 * HV_T)),
                             "l"(L + (4 * ORD[q] + i) * HV_T)
                             : "memory");
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
#pragma unroll
        for (int q = 0; q < 4; ++q) fetch(q);
        // r_i of the tile's rows (threads 0 .. 63) and c_j of its columns
        const int ex = __ldcg(a.limb_f + (b * a.limb_tiles + t) * (2 * HT) + tid);
        // tile (bi, bj), bj <= bi, from row and column p on; x vanishes up to c0
        const int64_t bi = tile_row(t), bj = t - bi * (bi + 1) / 2;
        trd_chain_wait();
        const int64_t R0 = p + bi * HT, C0 = p + bj * HT;
        __shared__ int4 vr[HT], vc[HT];              // limbs (re hi, re lo, im hi, im lo) of x
        __shared__ int redV[4], exps[2 * HT];
        __shared__ long long rs[4][4][HT], cs[4][HT];   // sums: H re, H im, M re, M im
        const int tr = tid & 15, tc = tid >> 4;
        double2 xv = make_double2(0.0, 0.0);
        {
            const int64_t r = tid < HT ? R0 + tid : C0 + tid - HT;
            if (r < n && r > c0) xv = A[r + col * lda];
        }
        // x with the scales of the rows (for the sums over them) and of the columns
        const int xs = tid < HT ? ex - 1022 : ex;
        {
            const int g = __reduce_max_sync(0xffffffffu, max(scaled_field(xv.x, xs), scaled_field(xv.y, xs)));
            if (lane == 0) redV[warp] = g;
            exps[tid] = ex;
        }
        __syncthreads();
        const int fr = max(redV[0], redV[1]), fc = max(redV[2], redV[3]);
        {
            int4 l;
            const int fx = (tid < HT ? fr : fc) - xs;
            limbs(xv.x, fx - field_of(xv.x), l.x, l.y);
            limbs(xv.y, fx - field_of(xv.y), l.z, l.w);
            (tid < HT ? vr[tid] : vc[tid - HT]) = l;
        }
        __syncthreads();
        // rows: a x, summed over the thread's eight columns; columns: conj(a) x, over its four rows, then over the 16
        // lanes of the row index: at each step a lane keeps half of its values and adds the partner's half
        long long row[4][4], lv[3][4], cur[4];
        int4 u[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            u[i] = vr[tr + 16 * i];
#pragma unroll
            for (int k = 0; k < 4; ++k) row[i][k] = 0;
        }
        const bool b8 = (lane & 8) != 0, b4 = (lane & 4) != 0, b2 = (lane & 2) != 0, b1 = (lane & 1) != 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            if (q <= 4) asm volatile("cp.async.wait_group 3;" ::: "memory");
            if (q == 5) asm volatile("cp.async.wait_group 2;" ::: "memory");
            if (q == 6) asm volatile("cp.async.wait_group 1;" ::: "memory");
            if (q == 7) asm volatile("cp.async.wait_group 0;" ::: "memory");
            const int4 y = vc[tc * 8 + ORD[q]];
            long long hr = 0, hi = 0, mr = 0, mi = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int4 x = tile[(4 * (q & 3) + i) * HV_T + tid];
                const int nz = -x.z, nw = -x.w;
                long long* R = row[i];
                mad(R[0], x.x, y.x); mad(R[1], x.x, y.z); mad(R[2], x.x, y.y); mad(R[3], x.x, y.w);
                mad(hr, x.x, u[i].x); mad(hi, x.x, u[i].z); mad(mr, x.x, u[i].y); mad(mi, x.x, u[i].w);
                mad(R[0], nz, y.z); mad(R[1], x.z, y.x); mad(R[2], nz, y.w); mad(R[3], x.z, y.y);
                mad(hr, x.z, u[i].z); mad(hi, nz, u[i].x); mad(mr, x.z, u[i].w); mad(mi, nz, u[i].y);
                mad(R[2], x.y, y.x); mad(R[3], x.y, y.z); mad(mr, x.y, u[i].x); mad(mi, x.y, u[i].z);
                mad(R[2], nw, y.z); mad(R[3], x.w, y.x); mad(mr, x.w, u[i].z); mad(mi, nw, u[i].x);
            }
            if (q < 4) fetch(q + 4);
            const long long c4[4] = {hr, hi, mr, mi};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                cur[k] = c4[k];
                if (q & 1) {
                    cur[k] = halve(lv[0][k], cur[k], b8, 8);
                    if (q & 2) {
                        cur[k] = halve(lv[1][k], cur[k], b4, 4);
                        if (q & 4)
                            cur[k] = halve(lv[2][k], cur[k], b2, 2);
                        else
                            lv[2][k] = cur[k];
                    } else {
                        lv[1][k] = cur[k];
                    }
                } else {
                    lv[0][k] = cur[k];
                }
            }
        }
        {
            // the lane's column: bits 8, 4, 2 of the lane chose bits 2, 1, 0 of its number; bit 1 the components
            const int c = tc * 8 + (b8 ? 4 : 0) + (b4 ? 2 : 0) + (b2 ? 1 : 0);
            cs[b1 ? 2 : 0][c] = halve(cur[0], cur[2], b1, 1);
            cs[b1 ? 3 : 1][c] = halve(cur[1], cur[3], b1, 1);
            const bool b16 = (lane & 16) != 0;
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int k = 0; k < 4; ++k) rs[warp][k][tr + 16 * i + (b16 ? 32 : 0)] = halve(row[i][k], row[i + 2][k], b16, 16);
        }
        __syncthreads();
        // a row's and a column's result, real or imaginary part
        const int v = tid >> 1, im = tid & 1;
        const long long H = (rs[0][im][v] + rs[1][im][v]) + (rs[2][im][v] + rs[3][im][v]);
        const long long M = (rs[0][2 + im][v] + rs[1][2 + im][v]) + (rs[2][2 + im][v] + rs[3][2 + im][v]);
        if (R0 + v < n)
            reinterpret_cast<double*>(a.Yrow + b * a.ystride + bj * n + R0 + v)[im] =
                fma((double)H, 268435456.0, (double)M) * limb_scale(exps[v], fc);
        if (C0 + v < n)
            reinterpret_cast<double*>(a.Ycol + b * a.ystride + bi * n + C0 + v)[im] =
                fma((double)cs[im][v], 268435456.0, (double)cs[2 + im][v]) * limb_scale(exps[HT + v] + 1022, fr);
    } else if (blockIdx.x > 0) {
        // panel dots: warp <-> reflector, lanes over the rows
        const int ng = (ii + DOT_L - 1) / DOT_L;
        const int64_t rb = ((int64_t)blockIdx.x - 1) / ng;
        const int lg = (int)((int64_t)blockIdx.x - 1 - rb * ng) * DOT_L, l = lg + warp;
        const double2* W = a.W + b * (n * TRD_NB);
        const double2 z = make_double2(0.0, 0.0);
        double2 s1 = z, s2 = z;
        trd_chain_wait();
        if (l < ii) {
            const int64_t rend = min(n, c0 + (rb + 1) * dot_rows);
            for (int64_t r0 = c0 + rb * dot_rows; r0 < rend; r0 += DOT_ROWS) {
                double2 v[DOT_ROWS / 32], w[DOT_ROWS / 32], h[DOT_ROWS / 32];
#pragma unroll
                for (int k = 0; k < DOT_ROWS / 32; ++k) {
                    const int64_t r = r0 + lane + 32 * k;
                    const bool ok = r < n && r > c0;
                    v[k] = ok ? A[r + col * lda] : z;
                    w[k] = ok ? W[r + l * n] : z;
                    h[k] = ok ? A[r + (p + l) * lda] : z;
                }
#pragma unroll
                for (int k = 0; k < DOT_ROWS / 32; ++k) {
                    s1.x = fma(w[k].x, v[k].x, fma(w[k].y, v[k].y, s1.x));
                    s1.y = fma(w[k].x, v[k].y, fma(-w[k].y, v[k].x, s1.y));
                    s2.x = fma(h[k].x, v[k].x, fma(h[k].y, v[k].y, s2.x));
                    s2.y = fma(h[k].x, v[k].y, fma(-h[k].y, v[k].x, s2.y));
                }
            }
        }
        // over the lanes: a lane keeps half of the four sums at the first two steps
        __shared__ double red[DOT_L][4][9];
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
        if (tid < 4 * DOT_L) {
            // thread: reflector tid >> 2 of the group, component tid & 3
            const double* q = red[tid >> 2][tid & 3];
            const double sum = ((q[0] + q[1]) + (q[2] + q[3])) + ((q[4] + q[5]) + (q[6] + q[7]));
            const int lo = lg + (tid >> 2);
            double* S = reinterpret_cast<double*>(a.Spart + b * a.sstride + rb * 2 * TRD_NB);
            if (lo < ii) S[2 * (((tid >> 1) & 1) * TRD_NB + lo) + (tid & 1)] = sum;
        }
    } else {
        // zlarfg: beta = -sign(|(alpha, x)|, Re alpha), tau = (beta - alpha)/beta, s = 1/(alpha - beta)
        __shared__ double xs[HV_T / 32];
        trd_chain_wait();
        double* sc = a.scal + b * 16;
        const double ar = sc[0], ai = sc[1];
        const int64_t np = parts_of(n - col, fr);
        double xn2 = 0.0;
        for (int64_t q = tid; q < np; q += HV_T) xn2 += a.part[b * a.pstride + q];
        xn2 = warp_sum_d(xn2);
        if (lane == 0) xs[warp] = xn2;
        __syncthreads();
        if (warp != 0) return;
        xn2 = (xs[0] + xs[1]) + (xs[2] + xs[3]);
        double q = lane == 0 ? 1.0 : 0.0, beta = ar;
        if (!(xn2 == 0.0 && ai == 0.0)) {
            beta = -copysign(sqrt(fma(ar, ar, fma(ai, ai, xn2))), ar);
            const double dr = ar - beta, den = fma(dr, dr, ai * ai);
            // lanes 0, 1: s; lanes 2, 3: tau
            q = (lane == 0 ? dr : lane == 2 ? -dr : -ai) / (lane < 2 ? den : beta);
        }
        if (lane < 4) sc[2 + lane] = q;
        if (lane == 2) a.tau[b * n + col].x = q;
        if (lane == 3) a.tau[b * n + col].y = q;
        if (lane == 0) a.e[b * n + col] = beta;
    }
}

template <int RW>
__global__ void __launch_bounds__(256) k_finish64(TrdArgs<double> a, int64_t p, int ii, int64_t col, int64_t nb2,
                                                  int64_t ndot) {
    const int64_t b = blockIdx.y, n = a.n, lda = a.lda, c0 = col + 1;
    double2* A = a.A + b * a.strideA;
    const double2* W = a.W + b * (n * TRD_NB);
    __shared__ double2 s1[TRD_NB], s2[TRD_NB];
    __shared__ double red[2][8];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, sl = lane / RW, im = lane >> 4;
    const int64_t r = c0 + (int64_t)blockIdx.x * FR<RW> + warp * RW + lane % RW;
    const double2 z = make_double2(0.0, 0.0);
    const bool mine = r < n, last = mine && (lane & 15) < RW;
    // what older kernels left: the panel, the raw column, the first column and the diagonal of A22
    double2 v[RW], w[RW], xr = z, ac = z, dg = z, c0w = z;
#pragma unroll
    for (int q = 0; q < RW; ++q) {
        const int l = sl + 32 / RW * q;
        v[q] = mine && l < ii ? ld_early(A + r + (p + l) * lda) : z;
        w[q] = mine && l < ii ? ld_early(W + r + l * n) : z;
    }
    if (last) {
        xr = ld_early(A + r + col * lda);
        if (r > c0) ac = ld_early(A + r + c0 * lda);
        dg = ld_early(A + r + r * lda);
    }
    // W^H v = conj(W(c0, :)) + s W^H x and likewise V^H v, from the slots of the panel dots: DOT_SLOTS lanes a reflector
    const int dl = (tid >> 2) & 31, dk = tid & 3, dim = dk >> 1;
    const bool dv = tid >> 7;   // V^H v
    if (dl < ii && (dk & 1) == 0) c0w = ld_early(dv ? A + c0 + (p + dl) * lda : W + c0 + dl * n);
    trd_chain_wait();
    const double* sc = a.scal + b * 16;
    const double2 s = make_double2(sc[2], sc[3]), tau = make_double2(sc[4], sc[5]);
    double2 d = z;
    if (dl < ii && dk < ndot) d = a.Spart[b * a.sstride + dk * 2 * TRD_NB + (dv ? TRD_NB : 0) + dl];
    // the row's partial products
    double2 y = z;
    {
        constexpr int LR = 32 / RW;
        const int64_t B = (r - p) / HT;
        const double2* Yrow = a.Yrow + b * a.ystride + r;
        const double2* Ycol = a.Ycol + b * a.ystride + r;
        const int64_t nr = mine && B >= sl ? (B - sl) / LR + 1 : 0;
        const int64_t nt = nr + (mine && nb2 - B > sl ? (nb2 - B - sl + LR - 1) / LR : 0);
        for (int64_t q0 = 0; q0 < nt; q0 += 4) {
            double2 t[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int64_t u = q0 + q;
                t[q] = u < nr ? Yrow[(sl + LR * u) * n] : u < nt ? Ycol[(B + sl + LR * (u - nr)) * n] : z;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (q0 + q < nt) y = vadd(y, t[q]);
        }
    }
    if (ii > 0) {
        // sum of the slots: re in lanes dk = 0, 1, im in 2, 3; then conj(c0w) + s d
        double e = (dim ? d.y : d.x) + __shfl_xor_sync(0xffffffffu, dim ? d.x : d.y, 2);
        e += __shfl_xor_sync(0xffffffffu, e, 1);
        const double o = __shfl_xor_sync(0xffffffffu, e, 2);
        const double val = dim ? fma(s.x, e, fma(s.y, o, -c0w.y)) : fma(s.x, e, fma(-s.y, o, c0w.x));
        if ((dk & 1) == 0) reinterpret_cast<double*>(dv ? &s2[dl] : &s1[dl])[dim] = val;
    }
    y = vmul(s, y);
    double2 y2 = z;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < RW; ++q) {
        const int l = sl + 32 / RW * q;
        if (32 / RW * q < ii) {
            const double2 d1 = l < ii ? s1[l] : z, d2 = l < ii ? s2[l] : z;
            y.x = fma(-v[q].x, d1.x, fma(v[q].y, d1.y, y.x));
            y.y = fma(-v[q].x, d1.y, fma(-v[q].y, d1.x, y.y));
            y2.x = fma(-w[q].x, d2.x, fma(w[q].y, d2.y, y2.x));
            y2.y = fma(-w[q].x, d2.y, fma(-w[q].y, d2.x, y2.y));
        }
    }
    // from here a lane holds one component: im = lane >> 4
    double t = row_sum<RW>(vadd(y, y2));
    // the first column of A22 and s D x
    double u = r == c0 ? (im ? 0.0 : 1.0) : fma(s.x, im ? xr.y : xr.x, im ? s.y * xr.x : -(s.y * xr.y));
    t = fma(dg.x, u, t + (im ? ac.y : ac.x));
    const double to = xor16(t), uo = xor16(u);
    t = fma(tau.x, t, im ? tau.y * to : -(tau.y * to));
    if (last) {
        reinterpret_cast<double*>(A + r + col * lda)[im] = u;
        reinterpret_cast<double*>(a.w0 + b * n + r)[im] = t;
    }
    // conj(w) v
    const double wo = xor16(t);
    double dot = im ? fma(wo, u, -(t * uo)) : fma(t, u, wo * uo);
    if (!last) dot = 0.0;
#pragma unroll
    for (int o = RW / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    if ((lane & 15) == 0) red[im][warp] = dot;
    __syncthreads();
    if (tid < 16) {
        dot = red[tid >> 3][tid & 7];
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffu, dot, o);
        if ((tid & 7) == 0) a.part[b * a.pstride + parts_of(n, FR<RW>) + 2 * blockIdx.x + (tid >> 3)] = dot;
    }
}

}  // namespace

template <int RW>
static int tridiagonalize_rows(cudaStream_t st, TrdArgs<double>& a, int64_t batch) {
    constexpr int fr = FR<RW>;
    const int64_t n = a.n;
    const unsigned nbat = (unsigned)batch;
    constexpr size_t HEMV_SMEM = sizeof(int4) * HT * HT / 2;
    FORGE_CUDA(cudaFuncSetAttribute(k_hemv64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)HEMV_SMEM));
    for (int64_t p = 0; p < n; p += TRD_NB) {
        const int64_t w = std::min<int64_t>(n - p, TRD_NB);
        int64_t nrefl = 0;
        const int64_t nb2 = (n - p + HT - 1) / HT, ntiles = nb2 * (nb2 + 1) / 2;
        prof_begin(ST_HEMV);
        k_limbs64<<<dim3((unsigned)ntiles, nbat), 256, 0, st>>>(a, p);
        FORGE_LAUNCH_CHECK();
        prof_end(ST_HEMV, batch * (double)(n - p) * (n - p) * 16.0, 0.0);
        for (int ii = 0; ii < w; ++ii) {
            const int64_t col = p + ii, n2 = n - col - 1;
            prof_begin(ST_TRD_COL);
            FORGE_TRY(launch_chain(st, dim3((unsigned)((n - col + fr - 1) / fr), nbat), 288, k_col64<RW>, a, p, ii, col));
            prof_end(ST_TRD_COL, batch * (double)(n - col) * (2.0 * ii + 2.0) * 16.0, 0.0);
            if (n2 <= 0) {
                // the last column has no reflector
                FORGE_CUDA(cudaMemset2DAsync(a.tau + col, n * sizeof(double2), 0, sizeof(double2), batch, st));
                continue;
            }
            ++nrefl;
            // slots of the panel dots and rows a slot
            const int64_t dot_rows = (n2 + DOT_SLOTS * DOT_ROWS - 1) / (DOT_SLOTS * DOT_ROWS) * DOT_ROWS;
            const int64_t ndot = ii > 0 ? (n2 + dot_rows - 1) / dot_rows : 0;
            const int64_t ndc = ndot * ((ii + DOT_L - 1) / DOT_L);
            prof_begin(ST_HEMV);
            FORGE_TRY(launch_chain_smem(st, dim3((unsigned)(ntiles + ndc + 1), nbat), HV_T, HEMV_SMEM, k_hemv64, a, p, ii, col, ndc,
                                        dot_rows, fr));
            // algorithmic traffic: the trailing lower triangle read once
            prof_end(ST_HEMV, batch * 0.5 * (double)n2 * (double)(n2 + 1) * 16.0, batch * 8.0 * (double)n2 * n2);
            prof_begin(ST_TRD_FINISH);
            FORGE_TRY(launch_chain(st, dim3((unsigned)((n2 + fr - 1) / fr), nbat), 256, k_finish64<RW>, a, p, ii, col, nb2, ndot));
            if (ii == w - 1) FORGE_TRY(launch_chain(st, dim3((unsigned)((n2 + 255) / 256), nbat), 256, k_fix64, a, ii, col, fr));
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

// Rows a warp: few of them where the rows do not fill the GPU's 608 FP64 pipes (the chain of a warp is 25 FP64
// instructions and 8 RW for a full panel), many where they do (the 25 are then shared by more rows).
int tridiagonalize_fp64(cudaStream_t st, TrdArgs<double>& a, int64_t batch) {
    const int64_t rows = a.n * batch;
    if (rows <= 2048) return tridiagonalize_rows<2>(st, a, batch);
    if (rows <= 4096) return tridiagonalize_rows<4>(st, a, batch);
    return tridiagonalize_rows<8>(st, a, batch);
}

}  // namespace forge
