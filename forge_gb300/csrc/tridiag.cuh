// Batched Householder reduction of Hermitian matrices (lower triangle) to real
// symmetric tridiagonal form, A = Q T Q^H, restating the blocked algorithm of
// LAPACK zhetrd/zlatrd (uplo = 'L') that the reference reaches through zheevr
// (LapackRoutines.f90:414-426).
//
// Per column (all k of the batch in one launch each; names of the FP32 kernels, FP64 has its own set):
//   trd_col   : add alpha2 v to the last column's w, update column col with the
//               panel's previous reflectors, generate the reflector (zlarfg) in the
//               last CTA (deterministic partials);
//   trd_hemv  : y = A22 v over 64x64 tiles of the trailing lower triangle, every
//               element read once; row and column partials go to disjoint slots
//               (Yrow / Ycol) so the reduction order is fixed; extra CTAs form
//               the panel dots W^H v and V^H v;
//   trd_finish: y -= V s1 + W s2, w0 = tau y, v written back, partials of w^H v.
// One more launch a panel (trd_fix) adds alpha2 v to its last w.
// After each panel of NB columns, the trailing matrix gets A22 -= V W^H + W V^H
// (a rank-2k update on the tensor cores in the chosen precision).
#pragma once
#include "cvec.cuh"
#include "forge_internal.cuh"

namespace forge {

constexpr int TRD_NB = 32;      // panel width
constexpr int TRD_TILE = 64;    // column granularity of the hemv partial slots (Yrow / Ycol)
constexpr int HV_RB = 64;       // hemv tile rows
constexpr int HV_CB = 64;       // hemv tile columns
constexpr int TRD_ROWS = 256;   // rows of one FP32 norm partial; threads per CTA of trd_finish / trd_fix

template <class T>
struct TrdArgs {
    using V = typename CV<T>::type;
    V* A;
    int64_t lda, strideA, n;
    double* d;
    double* e;          // batch x n each
    V* tau;             // batch x n
    V* W;               // batch x (n x NB), ldw = n
    V* Yrow;            // batch x (nblk x n)
    V* Ycol;            // batch x (nblk x n)
    int64_t ystride;    // nblk * n
    V* Spart;           // batch x (nrb x 2NB)
    int64_t sstride;
    double* part;       // batch x pstride per-CTA partials
    int64_t pstride;
    double* scal;       // batch x 16
    unsigned* cnt;      // batch x 4
    V* w0 = nullptr;    // batch x n: the last column's w before the alpha2 correction
    // FP64: the trailing triangle as integer limbs, batch x limb_tiles tiles of 64 x 64, and the exponents of
    // their rows and columns, 128 a tile
    int4* limbs = nullptr;
    int* limb_f = nullptr;
    int64_t limb_tiles = 0;
    // trailing update on the tensor cores (her2k_oz in FP64, her2k_tc in the mixed path):
    // A(p+w:n, p+w:n) -= V W^H + W V^H for the panel [p, p+w)
    int (*her2k)(cudaStream_t st, TrdArgs<T>& a, int64_t p, int64_t w, int64_t batch, void* user) = nullptr;
    void* her2k_user = nullptr;
};

// The kernels of a column form one chain; each is launched programmatically (launch_chain) and may be scheduled
// while its predecessor still runs.  It waits here for the predecessor's results; the next kernel's CTAs are
// let in as soon as all of this grid's have started.
__device__ __forceinline__ void trd_chain_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// Loads ahead of trd_chain_wait: of what the predecessor's own predecessor, or an older kernel, wrote (the predecessor
// has started all of its CTAs past its wait by then, so those results are in memory); from L2.  The predecessor's own
// results, and those of a kernel that was not launched by launch_chain, are not: they come after the wait.
__device__ __forceinline__ double2 ld_early(const double2* p) {
    double2 v;
    asm volatile("ld.global.cg.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ float2 ld_early(const float2* p) {
    float2 v;
    asm volatile("ld.global.cg.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
template <class... P, class... Q>
int launch_chain_smem(cudaStream_t st, dim3 grid, unsigned threads, size_t smem, void (*k)(P...), Q... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.dynamicSmemBytes = smem;
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.stream = st;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k, static_cast<P>(args)...);
    FORGE_LAUNCH_CHECK();
    return 0;
}

template <class... P, class... Q>
int launch_chain(cudaStream_t st, dim3 grid, unsigned threads, void (*k)(P...), Q... args) {
    return launch_chain_smem(st, grid, threads, 0, k, args...);
}

int tridiagonalize_f32(cudaStream_t st, TrdArgs<float>& a, int64_t batch);     // tridiag.cu
int tridiagonalize_fp64(cudaStream_t st, TrdArgs<double>& a, int64_t batch);   // tridiag_fp64.cu

}  // namespace forge
