// Batched partial Hermitian eigen-solver: eigenpairs 1..iu of nb matrices
// (lower triangles, column-major), the operation of zdiagRed
// (LapackRoutines.f90:381-433) for every k point of a batch.
#pragma once
#include "forge_internal.cuh"
#include "tridiag.cuh"

namespace forge {

struct EigArgs {
    int64_t n, iu, batch;
    double2* A;                 // batch x (lda x n), overwritten by the reflectors
    int64_t lda, strideA;
    double2* X;                 // batch x (ldx x iu) eigenvectors
    int64_t ldx, strideX;
    double* w;                  // batch x iu eigenvalues (ascending)
    // workspace
    double *d, *e;              // batch x n
    double2* tau;               // batch x n
    double2* Wp;                // batch x n x NB (panel W)
    double2* w0;                // batch x n
    double2 *Yrow, *Ycol;       // batch x ystride
    int64_t ystride;
    double2* Spart;
    int64_t sstride;
    double* part;
    int64_t pstride;
    double* scal;               // batch x 16
    double* info;               // batch x 8
    int* clus;                  // batch x (iu + 2)
    double* Z;                  // batch x n x iu (row-major)
    double* scr;                // 4 x n x (iu * batch)
    unsigned char* pivs;        // n x (iu * batch)
    int* fail;                  // batch
    // FP64 products on the tensor cores (oz_fp64.cu): slices of X (and U, Z of the rank-2k update), V, V^H, W
    // and T; W and W2, the Gram matrices and T in FP64; row scales; error flag of the bounded waits
    void *oz_xs, *oz_vr, *oz_vh, *oz_ws, *oz_ts;
    double2 *oz_wp, *oz_g, *oz_t;
    int* oz_ex;
    int4* limbs;                // of the tridiagonalisation; shares oz_vh
    int* limb_f;
    int64_t limb_tiles;
    int* oz_err;
    float2* tf;                 // batch x n: T scaled to |T| <= 1, (d_i, e_{i-1}^2) in FP32 (FP32 bisection)
    double2* de;                // the same in FP64
    float* tq;                  // batch x 2n: unscaled T in FP32, d and e^2 (mixed precision)
    bool mixed = false;         // workspace of the mixed solver (set before it is bound)
    bool lean = false;          // FP64 workspace of the allocation-free entry (n <= 512, set before it is bound)
    int replay = 0;             // 1 (mixed precision): eigenvalues as the quotient-form bisection gives them
    double ortol_rel;
    const int* iu_lim = nullptr;  // device: eigenpairs wanted of each matrix (nullptr: iu of every one)
    int64_t iu_out = 0;         // mixed solver: FP64 columns written to X (0: all iu)
};

// workspace sizes (bytes) for a given problem; they serve every smaller batch as well
// (mixed: what the mixed solver shares with the FP64 one; the rest of its workspace is eig_mixed_workspace_bytes)
size_t eig_workspace_bytes(int64_t n, int64_t iu, int64_t batch, bool mixed, bool lean = false);
// carve the workspace out of one device buffer; FORGE_ERR_ARG if the batch needs more than the bytes given
int eig_bind_workspace(EigArgs& g, void* base, size_t bytes);

size_t eig_mixed_workspace_bytes(int64_t n, int64_t iu, int64_t batch);
// K-split partial products of a batch and the room for them: Gram matrices (used, room), V^H X (used, room)
void eig_mixed_splits(int64_t n, int64_t iu, int64_t batch, int64_t* out);

int eig_fp64(cudaStream_t st, EigArgs& g);
int tridiag_eigvecs(cudaStream_t st, EigArgs& g);

// workspace of the FP64 products (elements of each array)
struct OzSizes {
    int64_t NB, nblk, mb, ks, ldx;        // block width, blocks, blocks per chunk, K splits of V^H X, slice pitch
    int64_t xs, vr, vh, uz, wp, ws, g, ts, ex;
};
void oz_sizes(int64_t n, int64_t iu, int64_t batch, bool lean, OzSizes& z);
int her2k_oz(cudaStream_t st, TrdArgs<double>& a, int64_t p, int64_t w, int64_t batch, void* user);
int backtransform_oz(cudaStream_t st, EigArgs& g);

}  // namespace forge
