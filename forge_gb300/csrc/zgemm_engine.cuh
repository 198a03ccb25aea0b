// Tiled complex GEMM engine on the CUDA cores (FP64 for the plain path, FP32 storage
// variant for small mixed-precision helpers).
//
//   C(i, j) = sum_k a(i, k) * b(j, k)      i < M, j < N, k < K
//
// a(i,k) and b(j,k) are functors (they apply conjugation, phases, weights and
// bounds), the epilogue functor receives every computed element.  The loader
// mapping is selectable per operand so that the global reads coalesce whichever
// index is contiguous in memory: IMAJOR = consecutive threads read consecutive i
// (column-major with i the row), KMAJOR = consecutive threads read consecutive k.
//
// Tile 64 x 64, BK = 8, 256 threads, 4 x 4 complex accumulators per thread; products with few columns or few
// tiles take 32 x 32 or 16 x 16 tiles of 128 threads (four warps fill the FP64 pipes of an SM), so that no
// padding is computed and more SMs take part.  The order of a result's additions does not depend on the tile.
#pragma once
#include "cvec.cuh"
#include "forge_internal.cuh"

namespace forge {

enum LoadMajor { IMAJOR = 0, KMAJOR = 1 };

constexpr int ZG_BK = 8;

template <int T>
struct ZgTile;   // threads along the rows / columns, results per thread
template <>
struct ZgTile<64> {
    static constexpr int TX = 16, TY = 16, RX = 4, RY = 4;
};
template <>
struct ZgTile<32> {
    static constexpr int TX = 8, TY = 16, RX = 4, RY = 2;
};
template <>
struct ZgTile<16> {
    static constexpr int TX = 8, TY = 16, RX = 2, RY = 1;
};

template <int MAJOR, int BROWS, int ZG_THREADS, class V, class F>
__device__ __forceinline__ void zg_load_tile(V (*S)[BROWS + 1], const F& f, int64_t r0, int64_t k0) {
    // loads BROWS x ZG_BK elements f(r0 + r, k0 + kk) into S[kk][r]
    constexpr int TOTAL = BROWS * ZG_BK;
#pragma unroll
    for (int q = 0; q < TOTAL / ZG_THREADS; ++q) {
        int idx = threadIdx.x + q * ZG_THREADS;
        int r, kk;
        if (MAJOR == IMAJOR) {
            r = idx % BROWS;
            kk = idx / BROWS;
        } else {
            kk = idx % ZG_BK;
            r = idx / ZG_BK;
        }
        S[kk][r] = f(r0 + r, k0 + kk);
    }
}

// Grid: x = tiles along M (times K splits), y = tiles along N, z = batch (passed to the functors
// as blockIdx.z).  LOWER: skip tiles entirely above the diagonal and elements i < j.
// SPLIT: blockIdx.x = s * (M tiles) + tile; split s sums k in [s kchunk, min(K, (s+1) kchunk))
// (kchunk a multiple of ZG_BK, so no k is summed twice) and the epilogue is called as
// epi(s, i, j, c) with its partial sum.
template <class V, int AMAJOR, int BMAJOR, bool LOWER, bool SPLIT, int TILE, class FA, class FB, class EPI>
__global__ void __launch_bounds__(ZgTile<TILE>::TX * ZgTile<TILE>::TY)
    k_zgemm(int64_t M, int64_t N, int64_t K, int64_t kchunk, FA fa, FB fb, EPI epi) {
    constexpr int TX = ZgTile<TILE>::TX, TY = ZgTile<TILE>::TY, RX = ZgTile<TILE>::RX, RY = ZgTile<TILE>::RY;
    const int64_t mt = (M + TILE - 1) / TILE;
    const int64_t split = SPLIT ? blockIdx.x / mt : 0;
    const int64_t i0 = (int64_t)(blockIdx.x - split * mt) * TILE, j0 = (int64_t)blockIdx.y * TILE;
    const int64_t klo = SPLIT ? split * kchunk : 0;
    const int64_t khi = SPLIT ? (K < klo + kchunk ? K : klo + kchunk) : K;
    if (LOWER && i0 + TILE - 1 < j0) return;
    __shared__ V As[ZG_BK][TILE + 1];
    __shared__ V Bs[ZG_BK][TILE + 1];
    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
    V acc[RX][RY];
#pragma unroll
    for (int a = 0; a < RX; ++a)
#pragma unroll
        for (int b = 0; b < RY; ++b) acc[a][b] = vzero<V>();
    for (int64_t k0 = klo; k0 < khi; k0 += ZG_BK) {
        zg_load_tile<AMAJOR, TILE, TX * TY>(As, fa, i0, k0);
        zg_load_tile<BMAJOR, TILE, TX * TY>(Bs, fb, j0, k0);
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < ZG_BK; ++kk) {
            V av[RX], bv[RY];
#pragma unroll
            for (int a = 0; a < RX; ++a) av[a] = As[kk][tx + TX * a];
#pragma unroll
            for (int b = 0; b < RY; ++b) bv[b] = Bs[kk][ty + TY * b];
#pragma unroll
            for (int a = 0; a < RX; ++a)
#pragma unroll
                for (int b = 0; b < RY; ++b) {
                    acc[a][b].x = fma(av[a].x, bv[b].x, acc[a][b].x);
                    acc[a][b].x = fma(-av[a].y, bv[b].y, acc[a][b].x);
                    acc[a][b].y = fma(av[a].x, bv[b].y, acc[a][b].y);
                    acc[a][b].y = fma(av[a].y, bv[b].x, acc[a][b].y);
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < RX; ++a)
#pragma unroll
        for (int b = 0; b < RY; ++b) {
            int64_t i = i0 + tx + TX * a, j = j0 + ty + TY * b;
            if (i < M && j < N && (!LOWER || i >= j)) {
                if constexpr (SPLIT)
                    epi(split, i, j, acc[a][b]);
                else
                    epi(i, j, acc[a][b]);
            }
        }
}

template <class V, int AMAJOR, int BMAJOR, bool LOWER, int TILE = 64, class FA, class FB, class EPI>
inline int zgemm_launch(cudaStream_t st, int64_t M, int64_t N, int64_t K, int64_t batch, const FA& fa,
                        const FB& fb, const EPI& epi) {
    if (M <= 0 || N <= 0 || batch <= 0) return 0;
    dim3 grd((unsigned)((M + TILE - 1) / TILE), (unsigned)((N + TILE - 1) / TILE), (unsigned)batch);
    k_zgemm<V, AMAJOR, BMAJOR, LOWER, false, TILE><<<grd, ZgTile<TILE>::TX * ZgTile<TILE>::TY, 0, st>>>(M, N, K, K, fa, fb, epi);
    FORGE_LAUNCH_CHECK();
    return 0;
}

// Number of K splits zgemm_launch_splitk runs for a K extent when `want` are asked for (none empty).
__host__ __device__ inline int64_t zg_ksplit_count(int64_t K, int64_t want) {
    if (want <= 1 || K <= ZG_BK) return 1;
    int64_t chunk = (K + want - 1) / want;
    chunk = (chunk + ZG_BK - 1) / ZG_BK * ZG_BK;
    return (K + chunk - 1) / chunk;
}

// Split-K form: ks = zg_ksplit_count(K, want) partial products, epilogue epi(s, i, j, c).
template <class V, int AMAJOR, int BMAJOR, int TILE = 64, class FA, class FB, class EPI>
inline int zgemm_launch_splitk(cudaStream_t st, int64_t M, int64_t N, int64_t K, int64_t batch, int64_t want,
                               const FA& fa, const FB& fb, const EPI& epi) {
    if (M <= 0 || N <= 0 || batch <= 0) return 0;
    const int64_t ks = zg_ksplit_count(K, want);
    int64_t chunk = (K + ks - 1) / ks;
    chunk = (chunk + ZG_BK - 1) / ZG_BK * ZG_BK;
    const int64_t mt = (M + TILE - 1) / TILE;
    dim3 grd((unsigned)(mt * ks), (unsigned)((N + TILE - 1) / TILE), (unsigned)batch);
    k_zgemm<V, AMAJOR, BMAJOR, false, true, TILE><<<grd, ZgTile<TILE>::TX * ZgTile<TILE>::TY, 0, st>>>(M, N, K, chunk, fa, fb, epi);
    FORGE_LAUNCH_CHECK();
    return 0;
}

}  // namespace forge
