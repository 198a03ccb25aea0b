// Batched Householder tridiagonalisation in FP32 (see tridiag.cuh for the structure).
//
// Bytes per column step (algorithmic): the trailing lower triangle, (n-col)^2/2
// complex elements, read once by trd_hemv; the rank-2k update is GEMM-shaped.
// What bounds a column besides trd_hemv's bytes is latency: kernel boundaries, and inside trd_col / trd_finish the
// round trips to L2.  So the three kernels are launched programmatically and load what older kernels left (the panel,
// the trailing matrix) before they wait for their predecessor, every thread's loads of a phase are in
// flight together, and no CTA adds up partials one by one.  One matrix of n = 5044 (5043 columns), whole kernels:
// trd_col 78 -> 55 ms, trd_hemv 91 -> 62 ms, trd_finish (with trd_fix, now once a panel) 116 -> 42 ms; n = 364, 36
// matrices: 5.4 -> 3.9, 4.2 -> 3.2, 5.4 -> 3.1 ms.
// The order of every FP32 sum is part of the result: refined orbitals are compared to the last place.
#include "tridiag.cuh"

namespace forge {

namespace {

// "last CTA" detection for a per-batch counter; returns true in every thread of the last CTA.
__device__ inline bool last_cta(unsigned* counter, unsigned total) {
    __shared__ bool is_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned t = atomicAdd(counter, 1u);
        is_last = (t == total - 1);
        if (is_last) *counter = 0u;
    }
    __syncthreads();
    return is_last;
}


constexpr int COL_ROWS = 64;   // rows per CTA of k_trd_col (and one warp for alpha2): the panel's columns come in over many SMs
constexpr int DOT_L = 8;       // reflectors per CTA of the panel dots

// partial sums: [0, trd_col_parts) the norms of k_trd_col, one float a warp; then pairs w^H v of k_trd_finish
__device__ inline int64_t trd_col_parts(int64_t n) { return (n + TRD_ROWS - 1) / TRD_ROWS * 4; }

__device__ inline float warp_sum_f(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// alpha2 = -1/2 tau (w^H v) of the last column from the nd partials of k_trd_finish, by one warp: lanes below 16 the real
// part, the others the imaginary part (an FP64 instruction of a warp takes 64 clocks, however many lanes are active)
__device__ inline float trd_alpha2(const TrdArgs<float>& a, int64_t b, int64_t nd) {
    const double* part = a.part + b * a.pstride + trd_col_parts(a.n);
    const int lane = threadIdx.x & 31, im = lane >> 4;
    const double tr = a.scal[b * 16 + 4], ti = a.scal[b * 16 + 5];
    double s = 0.0;
    for (int64_t q0 = lane & 15; q0 < nd; q0 += 160) {
        double t[10];
#pragma unroll
        for (int q = 0; q < 10; ++q) t[q] = q0 + 16 * q < nd ? part[2 * (q0 + 16 * q) + im] : 0.0;
#pragma unroll
        for (int q = 0; q < 10; ++q) {
            if (q0 - (lane & 15) + 16 * q >= nd) break;
            s += t[q];
        }
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const double o = __shfl_xor_sync(0xffffffffu, s, 16);
    return (float)(-0.5 * (im ? tr * s + ti * o : tr * s - ti * o));
}

// w + alpha2 v; the fused operations are spelled out because k_trd_col and k_trd_fix have to round alike
__device__ inline float2 trd_corr(float2 w, float2 al, float2 v) {
    return make_float2(__fadd_rn(w.x, fmaf(al.x, v.x, -__fmul_rn(al.y, v.y))),
                       __fadd_rn(w.y, fmaf(al.y, v.x, __fmul_rn(al.x, v.y))));
}

// ---------------------------------------------------------------- trd_col (zlatrd column update + zlarfg)
// Adds alpha2 v to the last column's w (w0), then forms column col; the last CTA forms the reflector's scalars from
// the partial norms.  The kernel is a chain of latencies (a column is a few hundred KB): all of a thread's panel
// elements are loaded at once, half a panel a time, and the last CTA's four quotients sit in four lanes.
__global__ void __launch_bounds__(COL_ROWS + 32) k_trd_col(TrdArgs<float> a, int64_t p, int ii, int64_t col, int has_refl) {
    const int64_t b = blockIdx.y, n = a.n, lda = a.lda;
    float2* A = a.A + b * a.strideA;
    float2* W = a.W + b * (n * TRD_NB);
    const float2* w0 = a.w0 + b * n;
    __shared__ float2 wrow[TRD_NB], arow[TRD_NB], s_al;
    const int lane = threadIdx.x & 31;
    const int64_t r = col + (int64_t)blockIdx.x * COL_ROWS + threadIdx.x;
    const int lm = ii - 1;
    const float2 z = make_float2(0.f, 0.f);
    const bool mine = threadIdx.x < COL_ROWS && r < n, alpha_warp = threadIdx.x >= COL_ROWS;
    // A panel's first column follows the kernel that updated the matrix.  Later ones load ahead what older kernels left:
    // the raw column, the panel but for its last reflector.
    if (ii == 0) trd_chain_wait();
    float2 x = z, wl = z, vl = z, av[16], wv[16];
    if (mine) x = ld_early(A + r + col * lda);
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        av[q] = q < lm && mine ? ld_early(A + r + (p + q) * lda) : z;
        wv[q] = q < lm && mine ? ld_early(W + r + q * n) : z;
    }
    if (alpha_warp && lane < lm) {
        wrow[lane] = ld_early(W + col + lane * n);
        arow[lane] = ld_early(A + col + (p + lane) * lda);
    }
    if (ii > 0) trd_chain_wait();
    if (mine && ii > 0) {
        wl = w0[r];
        vl = A[r + (p + lm) * lda];
    }
    __syncthreads();
    if (alpha_warp && ii > 0) {
        if (lane == 0) {
            wrow[lm] = w0[col];
            arow[lm] = A[col + (p + lm) * lda];
        }
        const float al = trd_alpha2(a, b, (n - col + 31) / 32);
        if ((lane & 15) == 0) reinterpret_cast<float*>(&s_al)[lane >> 4] = al;
    }
    if (mine) {
#pragma unroll
        for (int h = 0; h < TRD_NB; h += 16) {
            if (h >= lm) break;
            if (h > 0) {
#pragma unroll
                for (int q = 0; q < 16; ++q) {
                    av[q] = h + q < lm ? A[r + (p + h + q) * lda] : z;
                    wv[q] = h + q < lm ? W[r + (h + q) * n] : z;
                }
            }
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                if (h + q < lm) {
                    x = vsub(x, vmulcj(av[q], wrow[h + q]));
                    x = vsub(x, vmulcj(wv[q], arow[h + q]));
                }
            }
        }
    }
    __syncthreads();
    float nrm = 0.f;
    if (mine) {
        if (ii > 0) {
            // the last reflector, whose w takes its correction first
            const float2 al = s_al, ar = arow[lm];
            wl = trd_corr(wl, al, vl);
            W[r + lm * n] = wl;
            x = vsub(x, vmulcj(vl, trd_corr(wrow[lm], al, ar)));
            x = vsub(x, vmulcj(wl, ar));
        }
        if (r == col) {
            x.y = 0;
            a.d[b * n + col] = (double)x.x;
        }
        A[r + col * lda] = x;
        double* sc = a.scal + b * 16;
        if (r == col + 1) {
            sc[0] = (double)x.x;
            sc[1] = (double)x.y;
        }
        if (r >= col + 2) nrm = x.x * x.x + x.y * x.y;
    }
    nrm = warp_sum_f(nrm);
    float* part = (float*)(a.part + b * a.pstride);
    const int64_t nw = (int64_t)gridDim.x * (COL_ROWS / 32);
    if (lane == 0 && !alpha_warp) part[(int64_t)blockIdx.x * (COL_ROWS / 32) + (threadIdx.x >> 5)] = nrm;
    if (last_cta(a.cnt + b * 4, gridDim.x) && threadIdx.x < 32) {
        // 256 rows in FP32 (eight warps as a tree), beyond that in FP64
        double* sc = a.scal + b * 16;
        const double ar = ((volatile double*)sc)[0], ai = ((volatile double*)sc)[1];
        double xn2 = 0.0;   // summed in order: a last place of beta is a last place of eigenvalues
        for (int64_t g0 = 0; g0 < nw; g0 += 256) {
            const int64_t g = g0 + 8 * lane;
            float t[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) t[q] = g + q < nw ? ((volatile float*)part)[g + q] : 0.f;
            const float t8 = ((t[0] + t[4]) + (t[2] + t[6])) + ((t[1] + t[5]) + (t[3] + t[7]));
            const int m = (int)min((int64_t)32, (nw - g0 + 7) / 8);
            for (int q = 0; q < m; ++q) xn2 += (double)__shfl_sync(0xffffffffu, t8, q);
        }
        float2* tau = a.tau + b * n;
        // zlarfg: beta = -sign(|(alpha, x)|, Re alpha), tau = (beta - alpha)/beta, x *= 1/(alpha - beta)
        if (!has_refl || (xn2 == 0.0 && ai == 0.0)) {
            if (lane != 0) return;
            tau[col] = make_float2(0.f, 0.f);
            sc[2] = 1.0;
            sc[3] = 0.0;
            sc[4] = 0.0;
            sc[5] = 0.0;
            if (has_refl) a.e[b * n + col] = ar;
        } else {
            const double beta = -copysign(sqrt(ar * ar + ai * ai + xn2), ar);
            const double dr = ar - beta, di = ai, den = dr * dr + di * di;
            // lanes 0, 1: 1 / (alpha - beta); lanes 2, 3: tau
            const double num = lane == 0 ? dr : lane == 1 ? -di : lane == 2 ? beta - ar : -ai;
            const double q = num / (lane < 2 ? den : beta);
            if (lane < 4) sc[2 + lane] = q;
            if (lane == 2) tau[col].x = (float)q;
            if (lane == 3) tau[col].y = (float)q;
            if (lane == 0) a.e[b * n + col] = beta;
        }
    }
}

// ---------------------------------------------------------------- trd_hemv (+ panel dots)
// v = s x (1 in the first row); spelled out like trd_corr, so that the product and the stored v agree
__device__ inline float2 trd_scale(float2 x, bool first, float tr, float ti) {
    if (first) return make_float2(1.f, 0.f);
    return make_float2(fmaf(x.x, tr, -__fmul_rn(x.y, ti)), fmaf(x.x, ti, __fmul_rn(x.y, tr)));
}

__global__ void __launch_bounds__(256) k_trd_hemv(TrdArgs<float> a, int64_t p, int ii, int64_t col, int64_t ndc) {
    using V = float2;
    const int64_t b = blockIdx.y, n = a.n, lda = a.lda;
    const V* A = a.A + b * a.strideA;
    const double* sc = a.scal + b * 16;
    const int64_t c0 = col + 1;
    const int64_t t = (int64_t)blockIdx.x - ndc;   // the dots' CTAs, the longer chains, go first
    if (t >= 0) {
        // tile (bi, bj), bj <= bi, of the trailing matrix A(c0:n, c0:n): rows [64 bi, 64 bi + 64),
        // columns [64 bj, 64 bj + 64); t = bi (bi + 1) / 2 + bj
        int64_t bi = (int64_t)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);   // corrected below
        while ((bi + 1) * (bi + 2) / 2 <= t) ++bi;
        while (bi * (bi + 1) / 2 > t) --bi;
        const int64_t bj = t - bi * (bi + 1) / 2;
        const int64_t R0 = c0 + bi * HV_RB, C0 = c0 + bj * HV_CB;
        __shared__ V vr[HV_RB], vc[HV_CB];
        __shared__ V rsum[4][HV_RB];
        __shared__ V cs[HV_RB][HV_CB + 1];
        __shared__ V cq[4][HV_CB];
        const int tr = threadIdx.x & 63, tg = threadIdx.x >> 6;
        const int64_t r0 = R0 + tr, rv = (tg == 0 ? R0 : C0) + tr;
        // 16 loads per thread (row r0, 16 columns) before the column is known: a panel leaves A22 as it is.  Most tiles are
        // whole and below the diagonal: no bounds, no conjugates of the diagonal there (a third of the instructions).
        const bool whole = bi > bj && R0 + HV_RB <= n;
        V xv = vzero<V>(), a0[16];
        const V* pa = A + r0 + (C0 + tg * 16) * lda;
        if (whole) {
#pragma unroll
            for (int q = 0; q < 16; ++q, pa += lda) a0[q] = ld_early(pa);
        } else {
            const int cn = (int)min(n - (C0 + tg * 16), (int64_t)16), cd = (int)min(r0 - (C0 + tg * 16), (int64_t)16);
#pragma unroll
            for (int q = 0; q < 16; ++q, pa += lda) a0[q] = (r0 < n && q < cn && q <= cd) ? ld_early(pa) : vzero<V>();
        }
        trd_chain_wait();
        const float sr = (float)sc[2], si = (float)sc[3];
        if (tg < 2 && rv < n) xv = A[rv + col * lda];
        if (tg < 2) (tg == 0 ? vr : vc)[tr] = rv < n ? trd_scale(xv, rv == c0, sr, si) : vzero<V>();
        __syncthreads();
        V racc = vzero<V>();
        const V v0 = vr[tr];
        if (whole) {
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                racc = vadd(racc, vmul(a0[q], vc[tg * 16 + q]));
                cs[tr][tg * 16 + q] = vcjmul(a0[q], v0);
            }
        } else {
            const int dq = (int)max(min(r0 - (C0 + tg * 16), (int64_t)16), (int64_t)-1);   // the diagonal's column
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                V x0 = a0[q];
                const bool d0 = q == dq;
                if (d0) x0.y = 0;
                racc = vadd(racc, vmul(x0, vc[tg * 16 + q]));
                // column part: conj(A(r, c)) v_r for r > c (the diagonal belongs to the row part only)
                cs[tr][tg * 16 + q] = d0 ? vzero<V>() : vcjmul(x0, v0);
            }
        }
        rsum[tg][tr] = racc;
        __syncthreads();
        {
            // column sums: thread (col, quarter of the 64 rows)
            const int c = threadIdx.x & 63, qt = threadIdx.x >> 6;
            V acc = vzero<V>();
#pragma unroll
            for (int i = 0; i < 16; ++i) acc = vadd(acc, cs[qt * 16 + i][c]);
            cq[qt][c] = acc;
        }
        __syncthreads();
        V* Yrow = a.Yrow + b * a.ystride;
        V* Ycol = a.Ycol + b * a.ystride;
        if (threadIdx.x < HV_RB) {
            const int64_t r = R0 + threadIdx.x;
            if (r < n)
                Yrow[bj * n + r] = vadd(vadd(rsum[0][threadIdx.x], rsum[1][threadIdx.x]),
                                        vadd(rsum[2][threadIdx.x], rsum[3][threadIdx.x]));
        } else if (threadIdx.x < HV_RB + HV_CB) {
            const int q = threadIdx.x - HV_RB;
            const int64_t c = C0 + q;
            if (c < n) Ycol[bi * n + c] = vadd(vadd(cq[0][q], cq[1][q]), vadd(cq[2][q], cq[3][q]));
        }
    } else {
        // panel dots over 256 rows and DOT_L reflectors: s1 = W^H v, s2 = V^H v.  The 32 sums of a warp (8 reflectors
        // x 2 complex) are reduced together: each butterfly step halves what a lane carries, 31 shuffles, not 160.
        const int64_t nlc = (ii + DOT_L - 1) / DOT_L, rb = blockIdx.x / nlc;
        const int l0 = (int)(blockIdx.x - rb * nlc) * DOT_L;
        const int64_t r = c0 + rb * 256 + threadIdx.x;
        const V* W = a.W + b * (n * TRD_NB);
        __shared__ float sw[8][32];
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        V v = vzero<V>(), xw[DOT_L], xa[DOT_L];
#pragma unroll
        for (int q = 0; q < DOT_L; ++q) {
            // W's last column is the predecessor's
            xw[q] = r < n && l0 + q < ii - 1 ? ld_early(W + r + (l0 + q) * n) : vzero<V>();
            xa[q] = r < n && l0 + q < ii ? ld_early(A + r + (p + l0 + q) * lda) : vzero<V>();
        }
        trd_chain_wait();
        if (r < n) {
            v = A[r + col * lda];
#pragma unroll
            for (int q = 0; q < DOT_L; ++q)
                if (l0 + q == ii - 1) xw[q] = W[r + (l0 + q) * n];
        }
        v = r < n ? trd_scale(v, r == c0, (float)sc[2], (float)sc[3]) : v;
        float m[32];
#pragma unroll
        for (int q = 0; q < DOT_L; ++q) {
            const V x1 = vcjmul(xw[q], v), x2 = vcjmul(xa[q], v);
            m[4 * q] = x1.x;
            m[4 * q + 1] = x1.y;
            m[4 * q + 2] = x2.x;
            m[4 * q + 3] = x2.y;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const bool up = lane & o;
#pragma unroll
            for (int k = 0; k < o; ++k) {
                const float give = up ? m[k] : m[k + o], keep = up ? m[k + o] : m[k];
                m[k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
        }
        sw[w][lane] = m[0];   // lane = 4 q + (part)
        __syncthreads();
        const int l = l0 + (threadIdx.x >> 2), c = threadIdx.x & 3;
        if (threadIdx.x < 32 && l < ii) {
            float x = 0.f;
#pragma unroll
            for (int q = 0; q < 8; ++q) x += sw[q][threadIdx.x];
            float* S = (float*)(a.Spart + b * a.sstride + rb * 2 * TRD_NB);
            S[(c >> 1) * 2 * TRD_NB + 2 * l + (c & 1)] = x;
        }
    }
}

// ---------------------------------------------------------------- trd_finish
// y = A22 v - V (W^H v) - W (V^H v), w0 = tau y (w = w0 + alpha2 v follows in the next k_trd_col), v into A,
// partial sums of w^H v.  32 rows per CTA; 8 threads a row share the partial slots and the reflectors, and load
// theirs at once: like k_trd_col this is a chain of latencies.
__global__ void __launch_bounds__(TRD_ROWS) k_trd_finish(TrdArgs<float> a, int64_t p, int ii, int64_t col, int64_t nb2,
                                                         int64_t nrb) {
    using V = float2;
    const int64_t b = blockIdx.y, n = a.n, lda = a.lda;
    V* A = a.A + b * a.strideA;
    const V* W = a.W + b * (n * TRD_NB);
    const int64_t c0 = col + 1;
    __shared__ V s1[TRD_NB], s2[TRD_NB];
    __shared__ V ysl[8][33];
    const int rr = threadIdx.x & 31, sl = threadIdx.x >> 5;
    const int64_t r = c0 + (int64_t)blockIdx.x * 32 + rr;
    // what older kernels left: the panel, the raw column and its scalars
    V pa[4], pw[4], v = vzero<V>();
    if (r < n) {
        if (sl == 0) v = ld_early(A + r + col * lda);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int l = sl + 8 * q;
            pa[q] = l < ii ? ld_early(A + r + (p + l) * lda) : vzero<V>();
            pw[q] = l < ii ? ld_early(W + r + l * n) : vzero<V>();
        }
    }
    trd_chain_wait();
    const double* sc = a.scal + b * 16;
    const V s = make_float2((float)sc[2], (float)sc[3]), tau = make_float2((float)sc[4], (float)sc[5]);
    if (threadIdx.x >= 192 && rr < ii) {
        // warps 6 and 7 have the fewest slots: s1, s2 from the dots' partials
        const V* S = a.Spart + b * a.sstride + (sl - 6) * TRD_NB + rr;
        V x = vzero<V>();
        for (int64_t q0 = 0; q0 < nrb; q0 += 8) {
            V t[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) t[q] = q0 + q < nrb ? S[(q0 + q) * 2 * TRD_NB] : vzero<V>();
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (q0 + q < nrb) x = vadd(x, t[q]);
        }
        (sl == 6 ? s1 : s2)[rr] = x;
    }
    if (r < n) {
        // row part from the tiles (blk64(r), bj <= blk64(r)); column part from (bi >= blk64(r), blk64(r))
        const int64_t B = (r - c0) / HV_RB;
        const V* Yrow = a.Yrow + b * a.ystride + r;
        const V* Ycol = a.Ycol + b * a.ystride + r;
        const int64_t nr = B >= sl ? (B - sl) / 8 + 1 : 0, nt = nr + (nb2 - B > sl ? (nb2 - B - sl + 7) / 8 : 0);
        V y = vzero<V>();
        for (int64_t q0 = 0; q0 < nt; q0 += 12) {
            V t[12];
#pragma unroll
            for (int q = 0; q < 12; ++q) {
                const int64_t u = q0 + q;
                t[q] = u < nr ? Yrow[(sl + 8 * u) * n] : u < nt ? Ycol[(B + sl + 8 * (u - nr)) * n] : vzero<V>();
            }
#pragma unroll
            for (int q = 0; q < 12; ++q)
                if (q0 + q < nt) y = vadd(y, t[q]);
        }
        ysl[sl][rr] = y;
    }
    __syncthreads();   // s1, s2 are in shared memory
    if (r < n) {
        // the panel corrections -V s1 - W s2, split over the 8 slices
        V y = ysl[sl][rr];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int l = sl + 8 * q;
            if (l < ii) {
                y = vsub(y, vmul(pa[q], s1[l]));
                y = vsub(y, vmul(pw[q], s2[l]));
            }
        }
        ysl[sl][rr] = y;
    }
    __syncthreads();
    if (sl != 0) return;
    float dre = 0.f, dim = 0.f;
    if (r < n) {
        V y = vzero<V>();
#pragma unroll
        for (int q = 0; q < 8; ++q) y = vadd(y, ysl[q][rr]);
        y = vmul(tau, y);
        v = trd_scale(v, r == c0, s.x, s.y);
        A[r + col * lda] = v;
        a.w0[b * n + r] = y;
        // zdotc(w, v) = sum conj(w) v
        const V cv = vcjmul(y, v);
        dre = cv.x;
        dim = cv.y;
    }
    dre = warp_sum_f(dre);
    dim = warp_sum_f(dim);
    if (rr == 0) {
        double* part = a.part + b * a.pstride + trd_col_parts(n) + 2 * blockIdx.x;
        part[0] = (double)dre;
        part[1] = (double)dim;
    }
}

// w += alpha2 v of the panel's last column (the rank-2k update reads W)
__global__ void __launch_bounds__(TRD_ROWS) k_trd_fix(TrdArgs<float> a, int ii, int64_t col) {
    const int64_t b = blockIdx.y, n = a.n;
    __shared__ float2 s_al;
    trd_chain_wait();
    if (threadIdx.x < 32) {
        const float al = trd_alpha2(a, b, (n - col - 1 + 31) / 32);
        if ((threadIdx.x & 15) == 0) reinterpret_cast<float*>(&s_al)[threadIdx.x >> 4] = al;
    }
    __syncthreads();
    const int64_t r = col + 1 + (int64_t)blockIdx.x * TRD_ROWS + threadIdx.x;
    if (r < n)
        a.W[b * (n * TRD_NB) + r + ii * n] = trd_corr(a.w0[b * n + r], s_al, a.A[b * a.strideA + r + col * a.lda]);
}

}  // namespace

// ---------------------------------------------------------------- driver
int tridiagonalize_f32(cudaStream_t st, TrdArgs<float>& a, int64_t batch) {
    using T = float;
    const int64_t n = a.n;
    for (int64_t p = 0; p < n; p += TRD_NB) {
        const int64_t w = (n - p < TRD_NB) ? (n - p) : TRD_NB;
        int64_t nrefl = 0;
        for (int ii = 0; ii < w; ++ii) {
            const int64_t col = p + ii;
            const int has_refl = (col < n - 1) ? 1 : 0;
            const double esz = (double)sizeof(typename CV<T>::type);
            dim3 ga((unsigned)((n - col + COL_ROWS - 1) / COL_ROWS), (unsigned)batch);
            prof_begin(ST_TRD_COL);
            FORGE_TRY(launch_chain(st, ga, COL_ROWS + 32, k_trd_col, a, p, ii, col, has_refl));
            prof_end(ST_TRD_COL, batch * (double)(n - col) * (2.0 * ii + 2.0) * esz, 0.0);
            if (!has_refl) continue;
            ++nrefl;
            const int64_t n2 = n - col - 1;
            const int64_t nbr = (n2 + HV_RB - 1) / HV_RB;   // 64-row blocks (= 64-column blocks)
            const int64_t ntiles = nbr * (nbr + 1) / 2;     // row block bi holds bi + 1 tiles
            const int64_t nrb = ii > 0 ? (n2 + 255) / 256 : 0;
            const int64_t ndc = nrb * ((ii + DOT_L - 1) / DOT_L);
            dim3 gb((unsigned)(ntiles + ndc), (unsigned)batch);
            prof_begin(ST_HEMV);
            FORGE_TRY(launch_chain(st, gb, 256, k_trd_hemv, a, p, ii, col, ndc));
            // algorithmic traffic: the trailing lower triangle read once
            prof_end(ST_HEMV, batch * 0.5 * (double)n2 * (double)(n2 + 1) * esz, batch * 8.0 * (double)n2 * n2);
            dim3 gf((unsigned)((n2 + 31) / 32), (unsigned)batch);
            dim3 gc((unsigned)((n2 + TRD_ROWS - 1) / TRD_ROWS), (unsigned)batch);
            prof_begin(ST_TRD_FINISH);
            FORGE_TRY(launch_chain(st, gf, TRD_ROWS, k_trd_finish, a, p, ii, col, nbr, nrb));
            if (ii == w - 1) FORGE_TRY(launch_chain(st, gc, TRD_ROWS, k_trd_fix, a, ii, col));
            prof_end(ST_TRD_FINISH, batch * (double)n2 * (2.0 * ii + 4.0) * esz, 0.0);
        }
        if (nrefl > 0 && p + w < n) {
            const double m2 = (double)(n - p - w);
            prof_begin(ST_HER2K);
            FORGE_TRY(a.her2k(st, a, p, nrefl, batch, a.her2k_user));
            prof_end(ST_HER2K, batch * m2 * m2 * (double)sizeof(typename CV<T>::type),
                     batch * 8.0 * m2 * m2 * (double)nrefl);  // lower half of 2*nrefl complex MACs
        }
    }
    return 0;
}

}  // namespace forge
