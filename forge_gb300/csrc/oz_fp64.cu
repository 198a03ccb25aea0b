// The GEMM-shaped FP64 work of the plain path on the tensor cores by exact integer slices (oz_gemm.cuh):
// the back-transformation X = Q Z, the rank-2k update of the tridiagonalisation and the density-matrix
// projectors.  Inputs, outputs and everything between the products stay FP64.
//
// Measured against the FP64-pipe GEMMs they replace (stage times, ms):
//                                     N=364 36k   N=1324 16k   N=3268 1k
//   back-transformation            17.8 -> 3.4   200 -> 21.9   244 -> 21.1
//   rank-2k update                  7.1 -> 1.8    96 -> 15.4    98 -> 17.6
//   projectors                     28.9 -> 1.0    88 ->  5.9    66 ->  4.3
// The projectors also take all k points of an iteration in one launch (one k of N = 364 has 6 tiles).
// Errors against an 80-bit reference, 57 matrices H(k) and random ones of n = 76 to 364, in the mean of their
// logarithms: eigenvalues 0.84 times, occupied projector 0.88 times those of the FP64-pipe kernels.
#include <algorithm>
#include <vector>

#include "cvec.cuh"
#include "eig.cuh"
#include "oz_gemm.cuh"
#include "proj.cuh"

namespace forge {

constexpr int S7 = OZ_S;
constexpr int64_t GRID_Y = 65535;
constexpr int OZ_REF_S = 4, OZ_REF_DEPTH = 3;   // projectors of refined eigenvectors

int oz_make_tmap(CUtensorMap* map, const OzOperand& op) {
    return tc_make_tmap_bf16(map, op.ptr, op.cols, op.rows, op.nplanes, op.ld, op.plane, OZ_BK, OZ_T);
}

namespace {

inline int64_t up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }
inline unsigned cdiv(int64_t a, int64_t b) { return (unsigned)((a + b - 1) / b); }

// reflector j of A: v(j+1) = 1, v(r) = A(r, j) for r > j+1, 0 above
struct Refl {
    const double2* A;
    int64_t lda, strideA, n;
    __device__ double2 at(int64_t b, int64_t r, int64_t j) const {
        if (r < j + 1 || r >= n || j >= n - 1) return make_double2(0.0, 0.0);
        if (r == j + 1) return make_double2(1.0, 0.0);
        return A[b * strideA + r + j * lda];
    }
};
struct LdVH {  // rows l of V^H of several blocks: item z = q * batch + b is block j0 + q NB of matrix b
    Refl v;
    int64_t j0, NB, batch;
    __device__ double2 operator()(int64_t z, int64_t l, int64_t k) const {
        const int64_t q = z / batch, jb = j0 + q * NB;
        return v.at(z - q * batch, jb + k, jb + l);
    }
};
struct LdVr {  // rows r of V of one block, K = l
    Refl v;
    int64_t j0;
    __device__ int64_t extent(int64_t, int64_t K) const { return K; }
    __device__ double2 operator()(int64_t b, int64_t rr, int64_t l) const { return v.at(b, j0 + rr, j0 + l); }
};
struct LdX {  // columns c of X from row j0
    const double2* X;
    int64_t ldx, strideX, j0;
    __device__ double2 operator()(int64_t b, int64_t c, int64_t k) const { return X[b * strideX + j0 + k + c * ldx]; }
};
struct LdW {  // columns c of W (leading dimension NB), the sum of ks K-split partials (z = b ks + s)
    const double2* W;
    int64_t NB, iu, ks;
    __device__ double2 operator()(int64_t b, int64_t c, int64_t l) const {
        const double2* p = W + (b * ks * iu + c) * NB + l;
        double2 acc = p[0];
        for (int64_t s = 1; s < ks; ++s) acc = cadd(acc, p[s * iu * NB]);
        return acc;
    }
};
struct LdT {  // rows l of T (upper triangular, column-major NB x NB)
    const double2* T;
    int64_t NB;
    __device__ int64_t extent(int64_t, int64_t K) const { return K; }
    __device__ double2 operator()(int64_t z, int64_t l, int64_t q) const {
        return q < l ? make_double2(0.0, 0.0) : T[(z * NB + q) * NB + l];
    }
};

// Exponents of the largest |W| of a panel's columns (rows below the reduced one; biased), by atomicMax.  V and W share the scale
// of a row in the rank-2k update, and |v_l| <= 1 while |w_l| is of the size of what column l reduced: v_l takes
// 2^s ~ sqrt(max |w_l|) along and w_l 2^-s, so that neither loses digits to the other, nor a column to an earlier one,
// whatever unit the matrix is in and however it is graded.
__global__ void __launch_bounds__(256) k_oz_panel_max(const double2* __restrict__ W, int64_t n, int64_t p, int64_t w,
                                                      int* __restrict__ wmax) {
    const int64_t b = blockIdx.y, r = p + 1 + (int64_t)blockIdx.x * 64 + (threadIdx.x & 63);
    for (int64_t l = threadIdx.x >> 6; l < w; l += 4) {
        const double2 x = r < n && r > p + l ? W[b * n * TRD_NB + r + l * n] : make_double2(0.0, 0.0);
        const int f = __reduce_max_sync(0xffffffffu, max(oz_field(x.x), oz_field(x.y)));
        if ((threadIdx.x & 31) == 0 && f > 0) atomicMax(wmax + b * TRD_NB + l, f);
    }
}
// s of a column: 0 where w vanishes or holds a non-finite value
__device__ inline int panel_expo(int f) { return f == 0 || f == 2047 ? 0 : (f - 1023) >> 1; }

struct LdPanel {  // rows i of [2^s V  2^-s W] (swap = 0) or [2^-s W  2^s V] (swap = 1), a panel of w columns, 32 slots each
    const double2 *A, *W;
    const int* wmax;
    int64_t lda, strideA, n, r0, p, w;
    int swap;
    __device__ int64_t extent(int64_t, int64_t K) const { return K; }
    __device__ double2 operator()(int64_t b, int64_t i, int64_t k) const {
        const int64_t l = k & (TRD_NB - 1);
        if (l >= w) return make_double2(0.0, 0.0);
        const bool ofw = (k >> 5) ^ swap;
        const double2 v = ofw ? W[b * n * TRD_NB + r0 + i + l * n] : A[b * strideA + r0 + i + (p + l) * lda];
        const int e = panel_expo(wmax[b * TRD_NB + l]);
        const double s = oz_pow2(ofw ? -e : e);
        return make_double2(v.x * s, v.y * s);
    }
};

// column-major complex output, leading dimension ld, item z at z * stride; part 0: real, 1: imaginary
struct EpiStore {
    double2* C;
    int64_t ld, stride;
    const int *eA, *eB;
    int64_t seA, seB, zdiv;   // scales of item z / zdiv
    __device__ void operator()(int64_t z, int part, int64_t row, int64_t col0, const double* v, int64_t M,
                               int64_t N) const {
        if (row >= M) return;
        const int64_t b = z / zdiv;
        const int ea = eA[b * seA + row];
        double* o = reinterpret_cast<double*>(C + z * stride + row + col0 * ld) + part;
#pragma unroll
        for (int q = 0; q < 16; ++q)
            if (col0 + q < N) o[2 * q * ld] = v[q] * oz_pow2(ea + eB[b * seB + col0 + q]);
    }
};
// X(row, col) -= value
struct EpiSubX {
    double2* X;
    int64_t ld, stride;
    const int *eA, *eB;
    int64_t seA, seB;
    __device__ void operator()(int64_t b, int part, int64_t row, int64_t col0, const double* v, int64_t M,
                               int64_t N) const {
        if (row >= M) return;
        const int ea = eA[b * seA + row];
        double* o = reinterpret_cast<double*>(X + b * stride + row + col0 * ld) + part;
        double x[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) x[q] = col0 + q < N ? o[2 * q * ld] : 0.0;
#pragma unroll
        for (int q = 0; q < 16; ++q)
            if (col0 + q < N) o[2 * q * ld] = fma(-v[q], oz_pow2(ea + eB[b * seB + col0 + q]), x[q]);
    }
};
// lower triangle of A22 -= value; the diagonal stays real
struct EpiHer2k {
    double2* A;
    int64_t lda, stride;
    const int *eA, *eB;
    int64_t se;
    __device__ void operator()(int64_t b, int part, int64_t row, int64_t col0, const double* v, int64_t M,
                               int64_t N) const {
        if (row >= M || col0 > row) return;
        const int ea = eA[b * se + row];
        double* o = reinterpret_cast<double*>(A + b * stride + row + col0 * lda) + part;
        double x[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) x[q] = col0 + q <= row ? o[2 * q * lda] : 0.0;
#pragma unroll
        for (int q = 0; q < 16; ++q)
            if (col0 + q <= row)
                o[2 * q * lda] = (part && col0 + q == row) ? 0.0 : fma(-v[q], oz_pow2(ea + eB[b * se + col0 + q]), x[q]);
    }
};

// T of the compact-WY form from G = V^H V (zlarft, forward columnwise): T(0:i, i) = -tau_i T(0:i, 0:i) G(0:i, i),
// T(i, i) = tau_i.  One CTA per (block, matrix), thread l owns row l; T packed by columns in shared memory.
// FP64 pipe bound (NB^3 / 6 complex products on one SM), so all blocks of a chunk run side by side; the last block's
// chain ends with its last reflector (n = 2: 338 us for all 64 steps).
__global__ void k_oz_larft(const double2* __restrict__ G, const double2* __restrict__ tau, int64_t n, int64_t j0, int NB,
                           int64_t batch, double2* __restrict__ T) {
    extern __shared__ double2 lt_sm[];
    double2* t = lt_sm;                       // T(l, i) at i (i + 1) / 2 + l
    double2* tmp = t + NB * (NB + 1) / 2;
    const int64_t z = blockIdx.x, q = z / batch, b = z - q * batch, jb = j0 + q * NB;
    const double2* g = G + z * NB * NB;
    double2* To = T + z * NB * NB;
    const int l = threadIdx.x, nrefl = (int)min((int64_t)NB, n - 1 - jb);
    for (int i = nrefl; i < NB; ++i) To[l + i * NB] = make_double2(0.0, 0.0);
    for (int i = 0; i < nrefl; ++i) {
        const double2 ti = tau[b * n + jb + i];
        if (l < i) tmp[l] = cmul(cmake(-ti.x, -ti.y), g[l + i * NB]);
        __syncthreads();
        double2 acc = make_double2(0.0, 0.0);
        if (l < i) {
#pragma unroll 4
            for (int p = l; p < i; ++p) {
                const double2 a = t[p * (p + 1) / 2 + l], c = tmp[p];
                acc.x = fma(a.x, c.x, fma(-a.y, c.y, acc.x));
                acc.y = fma(a.x, c.y, fma(a.y, c.x, acc.y));
            }
        } else if (l == i) {
            acc = ti;
        }
        if (l <= i) t[i * (i + 1) / 2 + l] = acc;
        To[l + i * NB] = acc;
        __syncthreads();
    }
}

}  // namespace

// ---------------------------------------------------------------- workspace
// Block width of the back-transformation: 128 fills the M = 128 tile of V^H X; matrices up to 512 take
// 64 (half of the tile is padding, but T costs an eighth and the workspace half), those up to 33 32, which hold all of
// their reflectors (n = 2: 314 -> 293 us a solve, n = 12: 503 -> 480).
int oz_bt_nb(int64_t n) { return n > 512 ? 128 : n > 33 ? 64 : 32; }

void oz_sizes(int64_t n, int64_t iu, int64_t batch, bool lean, OzSizes& z) {
    z.NB = oz_bt_nb(n);
    z.nblk = (std::max<int64_t>(1, n - 1) + z.NB - 1) / z.NB;
    // blocks whose V^H and T are formed together: T is a serial chain a block, so all of them up to 512, half of them
    // (14 n^2 bytes) above; the allocation-free entry's 16 MiB array holds all up to 384 and single ones above
    const int64_t mb = n > 512 ? std::max<int64_t>(1, (z.nblk + 1) / 2) : lean && n > 384 ? 1 : z.nblk;
    // blocks x matrices in a grid's y extent; room: the most that mb x batch reaches for any batch up to this one
    z.mb = std::max<int64_t>(1, std::min<int64_t>(mb, GRID_Y / batch));
    const int64_t room = std::min(mb * batch, std::max<int64_t>(batch, GRID_Y));
    z.ldx = up(n, 8);
    // K splits of V^H X: enough CTAs for the GPU, no split shorter than 256 rows
    const int64_t t = (iu + OZ_T - 1) / OZ_T * 2, tiles = t * batch;
    const int64_t most = std::max<int64_t>(1, std::min<int64_t>(lean ? 1 : 8, n / 256));
    z.ks = std::min(most, (152 + tiles - 1) / tiles);
    const int64_t P = 2 * S7;
    z.xs = batch * P * iu * z.ldx;
    z.vr = batch * P * n * z.NB;
    z.uz = batch * 2 * P * n * 64;   // U and Z of the rank-2k update
    z.vh = room * P * z.NB * z.ldx;
    // the most that ks x batch reaches for any batch up to this one (a smaller batch takes more splits): the workspace
    // serves every batch below the one it was sized for
    z.wp = std::min(most * batch, 152 / t + batch) * iu * z.NB;
    z.ws = batch * P * iu * z.NB;
    z.g = room * z.NB * z.NB;
    z.ts = room * P * z.NB * z.NB;
    z.ex = batch * (2 * iu + 3 * n + TRD_NB) + 2 * room * z.NB;
}

// ---------------------------------------------------------------- rank-2k update
// A22 -= V W^H + W V^H for the panel [p, p + w): U = [V W], Z = [W V] (K = 64), C = U Z^H.
int her2k_oz(cudaStream_t st, TrdArgs<double>& a, int64_t p, int64_t w, int64_t batch, void* user) {
    EigArgs& g = *static_cast<EigArgs*>(user);
    const int64_t n = a.n, r0 = p + w, m = n - r0;
    if (m <= 0) return 0;
    static_assert(TRD_NB == 32, "the panel's two halves fill one K block of 64");
    const int64_t plane = n * 64, P = 2 * S7;
    unsigned short* U = reinterpret_cast<unsigned short*>(g.oz_xs);
    unsigned short* Zs = U + batch * P * plane;
    int *eU = g.oz_ex, *eZ = eU + batch * n;
    int* wmax = eZ + batch * n + p * batch;   // one a column, in the scales that the back-transformation uses later
    if (p == 0) FORGE_CUDA(cudaMemsetAsync(wmax, 0, sizeof(int) * batch * up(n, TRD_NB), st));
    k_oz_panel_max<<<dim3(cdiv(n - p - 1, 64), (unsigned)batch), 256, 0, st>>>(a.W, n, p, w, wmax);
    FORGE_LAUNCH_CHECK();
    const dim3 gs(cdiv(m, 32), (unsigned)batch), bs(32, 8);
    k_oz_rows<S7><<<gs, bs, 0, st>>>(LdPanel{a.A, a.W, wmax, a.lda, a.strideA, n, r0, p, w, 0}, m, 64, 64, U, 64, plane, eU, n, nullptr);
    FORGE_LAUNCH_CHECK();
    k_oz_rows<S7><<<gs, bs, 0, st>>>(LdPanel{a.A, a.W, wmax, a.lda, a.strideA, n, r0, p, w, 1}, m, 64, 64, Zs, 64, plane, eZ, n, nullptr);
    FORGE_LAUNCH_CHECK();
    const OzOperand A{(const __nv_bfloat16*)U, m, 64, 64, plane, batch * P, (int32_t)P};
    const OzOperand B{(const __nv_bfloat16*)Zs, m, 64, 64, plane, batch * P, (int32_t)P};
    return oz_gemm(st, A, 0, B, 0, 64, oz_plans_complex(S7, OZ_DEPTH, 64, false, true), batch, true,
                   EpiHer2k{a.A + r0 + r0 * a.lda, a.lda, a.strideA, eU, eZ, n}, g.oz_err);
}

// ---------------------------------------------------------------- back-transformation
int backtransform_oz(cudaStream_t st, EigArgs& g) {
    const int64_t n = g.n, iu = g.iu, batch = g.batch, nrefl = n - 1;
    if (nrefl <= 0) return 0;
    OzSizes z;
    oz_sizes(n, iu, batch, g.lean, z);
    const int64_t NB = z.NB, P = 2 * S7;
    const Refl v{g.A, g.lda, g.strideA, n};
    unsigned short *Xs = (unsigned short*)g.oz_xs, *Vr = (unsigned short*)g.oz_vr, *VH = (unsigned short*)g.oz_vh;
    unsigned short *Ws = (unsigned short*)g.oz_ws, *Ts = (unsigned short*)g.oz_ts;
    int* eX = g.oz_ex;
    int* eW = eX + batch * iu;
    int* eR = eW + batch * iu;
    int* eV = eR + batch * n;
    int* eT = eV + z.mb * batch * NB;
    const int64_t pX = iu * z.ldx, pV = NB * z.ldx, pR = n * NB, pW = iu * NB, pT = NB * NB;
    const size_t smem = sizeof(double2) * (size_t)(NB * (NB + 1) / 2 + NB);
    FORGE_CUDA(cudaFuncSetAttribute(k_oz_larft, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    for (int64_t hi = z.nblk; hi > 0; hi -= z.mb) {
        const int64_t lo = std::max<int64_t>(0, hi - z.mb), nb = hi - lo, zb = nb * batch;   // blocks [lo, hi)
        const int64_t j0c = lo * NB, Kc = n - j0c;
        // V^H of the chunk's blocks, their Gram matrices and T
        k_oz_cols<S7><<<dim3((unsigned)NB, (unsigned)zb), 256, 0, st>>>(LdVH{v, j0c, NB, batch}, Kc, z.ldx, VH, z.ldx, pV,
                                                                        eV, NB);
        FORGE_LAUNCH_CHECK();
        const OzOperand oV{(const __nv_bfloat16*)VH, NB, Kc, z.ldx, pV, zb * P, (int32_t)P};
        FORGE_TRY(oz_gemm(st, oV, 0, oV, 0, Kc, oz_plans_complex(S7, OZ_DEPTH, Kc, true, false), zb, false,
                          EpiStore{g.oz_g, NB, NB * NB, eV, eV, NB, NB, 1}, g.oz_err));
        k_oz_larft<<<(unsigned)zb, (unsigned)NB, smem, st>>>(g.oz_g, g.tau, n, j0c, (int)NB, batch, g.oz_t);
        FORGE_LAUNCH_CHECK();
        k_oz_rows<S7><<<dim3(cdiv(NB, 32), (unsigned)zb), dim3(32, 8), 0, st>>>(LdT{g.oz_t, NB}, NB, NB, NB, Ts, NB, pT, eT,
                                                                                NB, nullptr);
        FORGE_LAUNCH_CHECK();
        for (int64_t blk = hi - 1; blk >= lo; --blk) {
            const int64_t j0 = blk * NB, q = blk - lo, K = n - j0;
            // W = V^H X, split over K
            k_oz_cols<S7><<<dim3((unsigned)iu, (unsigned)batch), 256, 0, st>>>(LdX{g.X, g.ldx, g.strideX, j0}, K,
                                                                               std::min(z.ldx, up(K, 8)), Xs, z.ldx, pX,
                                                                               eX, iu);
            FORGE_LAUNCH_CHECK();
            const OzOperand oA{(const __nv_bfloat16*)VH + q * batch * P * pV, NB, K, z.ldx, pV, batch * P, (int32_t)P};
            const OzOperand oX{(const __nv_bfloat16*)Xs, iu, K, z.ldx, pX, batch * P, (int32_t)P};
            const int64_t ks = oz_ksplit_count((K + OZ_BK - 1) / OZ_BK, std::min<int64_t>(z.ks, std::max<int64_t>(1, K / 256)));
            FORGE_TRY(oz_gemm(st, oA, 0, oX, 0, K, oz_plans_complex(S7, OZ_DEPTH, K, true, false), batch, false,
                              EpiStore{g.oz_wp, NB, iu * NB, eV + q * batch * NB, eX, NB, iu, ks}, g.oz_err, ks));
            // W2 = T W
            k_oz_cols<S7><<<dim3((unsigned)iu, (unsigned)batch), 256, 0, st>>>(LdW{g.oz_wp, NB, iu, ks}, NB, NB, Ws, NB, pW,
                                                                               eW, iu);
            FORGE_LAUNCH_CHECK();
            const OzOperand oT{(const __nv_bfloat16*)Ts + q * batch * P * pT, NB, NB, NB, pT, batch * P, (int32_t)P};
            const OzOperand oW{(const __nv_bfloat16*)Ws, iu, NB, NB, pW, batch * P, (int32_t)P};
            FORGE_TRY(oz_gemm(st, oT, 0, oW, 0, NB, oz_plans_complex(S7, OZ_DEPTH, NB, false, false), batch, false,
                              EpiStore{g.oz_wp, NB, iu * NB, eT + q * batch * NB, eW, NB, iu, 1}, g.oz_err));
            // X(j0:, :) -= V W2
            k_oz_cols<S7><<<dim3((unsigned)iu, (unsigned)batch), 256, 0, st>>>(LdW{g.oz_wp, NB, iu, 1}, NB, NB, Ws, NB, pW,
                                                                               eW, iu);
            FORGE_LAUNCH_CHECK();
            k_oz_rows<S7><<<dim3(cdiv(K, 32), (unsigned)batch), dim3(32, 8), 0, st>>>(LdVr{v, j0}, K, NB, NB, Vr, NB, pR, eR,
                                                                                      n, nullptr);
            FORGE_LAUNCH_CHECK();
            const OzOperand oR{(const __nv_bfloat16*)Vr, K, NB, NB, pR, batch * P, (int32_t)P};
            FORGE_TRY(oz_gemm(st, oR, 0, oW, 0, NB, oz_plans_complex(S7, OZ_DEPTH, NB, false, false), batch, false,
                              EpiSubX{g.X + j0, g.ldx, g.strideX, eR, eW, n, iu}, g.oz_err));
        }
    }
    return 0;
}

// ---------------------------------------------------------------- projectors
namespace {
struct LdProj {  // rows i of X of item b, K = the occupied columns of that item
    const double2* X;
    int64_t ldx, strideX;
    const ProjItem* it;
    __device__ int64_t extent(int64_t b, int64_t) const { return it[b].K; }
    __device__ double2 operator()(int64_t b, int64_t i, int64_t k) const { return X[it[b].slot * strideX + i + k * ldx]; }
};
// lower triangle of C, real and imaginary parts apart: item z at z * 2 n^2
struct EpiProj {
    double* C;
    int64_t n;
    const int* e;
    __device__ void operator()(int64_t z, int part, int64_t row, int64_t col0, const double* v, int64_t M,
                               int64_t N) const {
        if (row >= M || col0 > row) return;
        const int er = e[z * n + row];
        double* o = C + (2 * z + part) * n * n + row + col0 * n;
#pragma unroll
        for (int q = 0; q < 16; ++q)
            if (col0 + q <= row) o[q * n] = v[q] * oz_pow2(er + e[z * n + col0 + q]);
    }
};

// P_c += sum over the items z of ph_c(z) C_z (C Hermitian, its lower triangle given): a CTA owns tile
// (bi, bj) and its mirror image (bj, bi) of all four cells and adds the items in order, so that P
// is read and written once.  HBM bound.
// diag (or null): the diagonal of the C_z (nit x n), in place of C's own.
__global__ void __launch_bounds__(256) k_proj_add(double2* __restrict__ P, const double* __restrict__ C,
                                                  const double* __restrict__ diag, const ProjItem* __restrict__ it,
                                                  int64_t nit, int64_t n) {
    const int64_t bi = blockIdx.x, bj = blockIdx.y;
    if (bi < bj) return;
    __shared__ double sr[32][33], si[32][33];
    const int64_t i0 = bi * 32, j0 = bj * 32;
    const size_t NN = (size_t)n * n;
    const int tx = threadIdx.x, ty = threadIdx.y;
    for (int mir = 0; mir < (bi == bj ? 1 : 2); ++mir) {
        // rows of the written tile: i (mir 0) or j (mir 1)
        const int64_t r0 = mir ? j0 : i0, c0 = mir ? i0 : j0;
        double2 acc[4][4];
#pragma unroll
        for (int y = 0; y < 4; ++y)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int64_t r = r0 + tx, cc = c0 + ty + 8 * y;
                acc[y][c] = (r < n && cc < n) ? P[c * NN + r + cc * n] : make_double2(0.0, 0.0);
            }
        for (int64_t z = 0; z < nit; ++z) {
            const double* Cr = C + 2 * z * NN;
            __syncthreads();
            for (int y = ty; y < 32; y += 8) {
                const int64_t i = i0 + tx, j = j0 + y;
                const bool ok = i < n && j < n && i >= j;
                sr[y][tx] = ok ? Cr[i + j * n] : 0.0;               // sr[col][row]
                si[y][tx] = ok ? Cr[NN + i + j * n] : 0.0;
            }
            __syncthreads();
            double2 ph[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) ph[c] = it[z].ph[c];
#pragma unroll
            for (int y = 0; y < 4; ++y) {
                const int col = ty + 8 * y;
                double cr, ci;
                if (mir) {                      // element (j, i) = conj C(i, j)
                    cr = sr[tx][col];
                    ci = -si[tx][col];
                } else if (bi != bj || tx >= col) {
                    cr = sr[col][tx];
                    ci = si[col][tx];
                } else {
                    cr = sr[tx][col];
                    ci = -si[tx][col];
                }
                if (diag && bi == bj && tx == col) {
                    cr = i0 + tx < n ? diag[z * n + i0 + tx] : 0.0;
                    ci = 0.0;
                }
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    acc[y][c].x += ph[c].x * cr - ph[c].y * ci;
                    acc[y][c].y += ph[c].x * ci + ph[c].y * cr;
                }
            }
        }
#pragma unroll
        for (int y = 0; y < 4; ++y)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int64_t r = r0 + tx, cc = c0 + ty + 8 * y;
                if (r < n && cc < n) P[c * NN + r + cc * n] = acc[y][c];
            }
    }
}
}  // namespace

// items per launch: as many as fit in cap bytes of slices and products and in a launch's grid, at least one
static int64_t proj_oz_chunk(int64_t n, int64_t iu, int64_t nit, int S, int64_t cap) {
    const int64_t per = 2 * S * n * up(iu, 8) * 2 + 2 * n * n * 8;
    return std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(nit, OZ_GRID_Z), cap / per));
}
size_t proj_oz_workspace_bytes(int64_t n, int64_t iu, int64_t nit, bool refined, int64_t cap) {
    const int S = refined ? OZ_REF_S : OZ_S;
    const int64_t ch = proj_oz_chunk(n, iu, nit, S, cap);
    return (size_t)ch * (2 * S * n * up(iu, 8) * 2 + 2 * n * n * 8 + up(n, 64) * 12) + (size_t)nit * sizeof(ProjItem) + 1024;
}

template <int S, int DEPTH, bool REF>
static int projectors_cut(cudaStream_t st, const double2* X, int64_t ldx, int64_t strideX, int64_t n, int64_t iu,
                          const ProjItem* items, int64_t nit, double2* P, void* ws, int* err, int64_t cap) {
    if (nit <= 0) return 0;
    prof_begin(ST_PROJECTOR);
    const int64_t ch = proj_oz_chunk(n, iu, nit, S, cap), ldk = up(iu, 8), plane = n * ldk, PL = 2 * S;
    double* C = static_cast<double*>(ws);
    unsigned short* sl = reinterpret_cast<unsigned short*>(C + ch * 2 * n * n);
    int* e = reinterpret_cast<int*>(sl + ch * PL * plane);
    double* dg = reinterpret_cast<double*>(((uintptr_t)(e + ch * n) + 255) & ~(uintptr_t)255);
    ProjItem* dit = reinterpret_cast<ProjItem*>(((uintptr_t)(dg + ch * n) + 255) & ~(uintptr_t)255);
    if (!REF) dg = nullptr;
    FORGE_CUDA(cudaMemcpyAsync(dit, items, nit * sizeof(ProjItem), cudaMemcpyHostToDevice, st));
    for (int64_t z0 = 0; z0 < nit; z0 += ch) {
        const int64_t nb = std::min(ch, nit - z0);
        int64_t K = 0;
        for (int64_t z = 0; z < nb; ++z) K = std::max(K, items[z0 + z].K);
        if (K <= 0) continue;
        k_oz_rows<S, REF><<<dim3(cdiv(n, 32), (unsigned)nb), dim3(32, 8), 0, st>>>(
            LdProj{X, ldx, strideX, dit + z0}, n, K, up(K, 8), sl, ldk, plane, e, n, dg);
        FORGE_LAUNCH_CHECK();
        const OzOperand op{(const __nv_bfloat16*)sl, n, K, ldk, plane, nb * PL, (int32_t)PL};
        FORGE_TRY(oz_gemm<REF>(st, op, 0, op, 0, K, oz_plans_complex(S, DEPTH, K, true, false), nb, true,
                               EpiProj{C, n, e}, err));
        k_proj_add<<<dim3(cdiv(n, 32), cdiv(n, 32)), dim3(32, 8), 0, st>>>(P, C, dg, dit + z0, nb, n);
        FORGE_LAUNCH_CHECK();
    }
    prof_end(ST_PROJECTOR, (double)n * iu * 16.0 * nit + 4.0 * 2.0 * n * n * 16.0, 4.0 * (double)n * n * (iu - 10) * nit);
    return 0;
}

// P_c += sum over items of ph_c conj(X) X^T over the first K columns of X at the item's slot.  refined: the
// eigenvectors come from the refined mixed solve (errors of 1e-9): four slices taken from the top, ten
// products in double-float sums (2^-48) and the diagonal (the site densities) in FP64.  Measured (TF32 slices, one
// k a launch before): N = 364, 36 k 8.7 -> 0.9 ms; N = 1324, 16 k 11.0 -> 3.8 ms; N = 5044 19.1 -> 7.2 ms
int projectors_oz(cudaStream_t st, const double2* X, int64_t ldx, int64_t strideX, int64_t n, int64_t iu,
                  const ProjItem* items, int64_t nit, double2* P, void* ws, int* err, bool refined, int64_t cap) {
    return refined ? projectors_cut<OZ_REF_S, OZ_REF_DEPTH, true>(st, X, ldx, strideX, n, iu, items, nit, P, ws, err, cap)
                   : projectors_cut<OZ_S, OZ_DEPTH, false>(st, X, ldx, strideX, n, iu, items, nit, P, ws, err, cap);
}

}  // namespace forge
