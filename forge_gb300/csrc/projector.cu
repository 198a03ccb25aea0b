// K6: window projector (GetFock, HartreeFock.f90:487-560) on the FP64 pipe: sorted states 1..nOcc with weight
// 1 or zdeg; the weight can be complex (reference mode of zdeg), so the full N x N product is formed,
// one GEMM per cell (grid z = cell).  The bulk projectors are in oz_fp64.cu and projector_tc.cu.
#include "proj.cuh"
#include "zgemm_engine.cuh"

namespace forge {

struct WinA {  // a(i, s) = conj(psi_s(i)) * w_s * ph_c(k_s),  c = blockIdx.z
    const WinState* st;
    const double2* X;
    int64_t ldx, strideX, N, K;
    __device__ double2 operator()(int64_t i, int64_t s) const {
        if (i >= N || s >= K) return make_double2(0.0, 0.0);
        const WinState w = st[s];
        const double2 x = X[w.k * strideX + i + w.col * ldx];
        return cmul(cconj(x), w.wph[blockIdx.z]);
    }
};
struct WinB {  // b(j, s) = psi_s(j)
    const WinState* st;
    const double2* X;
    int64_t ldx, strideX, N, K;
    __device__ double2 operator()(int64_t j, int64_t s) const {
        if (j >= N || s >= K) return make_double2(0.0, 0.0);
        const WinState w = st[s];
        return X[w.k * strideX + j + w.col * ldx];
    }
};
struct WinEpi {
    double2* P;
    int64_t N;
    __device__ void operator()(int64_t i, int64_t j, double2 v) const {
        double2* p = P + (size_t)blockIdx.z * N * N + i + (size_t)j * N;
        *p = cadd(*p, v);
    }
};

int window_projector_fp64(cudaStream_t st, const WinState* states, int64_t nstates, const double2* X, int64_t ldx,
                          int64_t strideX, int64_t N, double2* P) {
    if (nstates <= 0) return 0;
    prof_begin(ST_WINDOW);
    int rc = zgemm_launch<double2, IMAJOR, IMAJOR, false>(st, N, N, nstates, 4,
                                                          WinA{states, X, ldx, strideX, N, nstates},
                                                          WinB{states, X, ldx, strideX, N, nstates},
                                                          WinEpi{P, N});
    prof_end(ST_WINDOW, (double)N * nstates * 16.0 + 4.0 * 2.0 * N * N * 16.0, 4.0 * 8.0 * (double)N * N * nstates);
    return rc;
}

}  // namespace forge
