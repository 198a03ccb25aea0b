// FP64-accurate real GEMM on the bf16 tensor cores (tcgen05 kind::f16) by exact integer slices.
//
//   D[b](m, n) = 2^(eA(m) + eB(n)) sum_{s + t <= depth} 2^-(16 + 9 (s + t)) sum_k A_s(m, k) B_t(n, k)
//
// Every row of an operand is scaled by a power of two to |v| < 1 and cut into S integer slices of nine
// bits, v = sum_s v_s 2^-(8 + 9 s), |v_s| <= 256 (Ozaki, Ogita, Oishi, Rump, "Error-free transformations
// of matrix multiplication by using fast routines of matrix multiplication and its applications",
// Numer. Algorithms 59, 2012).  Slices are exact in bf16, a product of two is below 2^16 and a sum
// of 256 of them below 2^24, so the FP32 accumulation in TMEM is exact; every 256 products the epilogue
// warps add the block to int64 accumulators, and each level d = s + t weighs 2^9 less than the one
// before, so a level is a shift.  Nothing is rounded until the sum is converted to FP64.  With
// seven slices and depth 6 the operands keep 62 bits below their row's maximum.  A slice s is at most 2^-9s of the
// row's scale, so the neglected pairs of a real product (six with s + t = 7, the next ones 2^-9 of these) are below
// 6 x 2^-63 = 2^-60.4 of the two maxima, twice that for a component of a complex product, and about 2^-63 for digits of
// random sign: small beside the rounding of an FP64 product of the row maxima, 2^-53.  An element below 2^-9 of its
// row's maximum has fewer than FP64's 53 bits; the callers scale their operands so that a row's elements matter by
// its maximum (oz_fp64.cu).
//
// Why: this GPU's FP64 pipe does 1.2 TFLOP/s (two FMA lanes a clock and SM); 28 slice products at the
// measured bf16 rate are 1938 / 28 = 69 TFLOP/s of FP64-accurate work.
//
// One CTA of 320 threads per 128 x 128 tile, one per SM (smem ring 6 x 32 KB, 512 TMEM columns):
//   warp 0     TMA producer (3D bf16 maps {K, rows, planes}, 64 x 128 boxes, 128B swizzle)
//   warp 1     MMA issuer, M = N = 128, K = 16; allocates and frees TMEM
//   warps 2-9  accumulators: warp w reads TMEM lanes 32 (w % 4) .. +31 and column half (w - 2) / 4
// TMEM columns 0..255 are two accumulation buffers of 128, so the MMAs of one block of 256 run while
// the previous one is added up; columns 256..511 hold the FP64 value of the first levels when all
// levels together exceed 63 bits.
#pragma once
#include <algorithm>

#include <cuda_bf16.h>

#include "tc_gemm.cuh"

namespace forge {

constexpr int OZ_T = 128, OZ_BK = 64, OZ_STAGES = 6, OZ_THREADS = 320;
constexpr int OZ_TILE_BYTES = OZ_T * OZ_BK * 2;   // 16 KB per operand and stage
constexpr int OZ_SMEM = OZ_STAGES * 2 * OZ_TILE_BYTES + 1024 + 256;
constexpr int OZ_MAXSEG = 64, OZ_MAXLEV = 8;
constexpr int OZ_GRID_Z = 32767;                  // products of a batch (times K splits) per launch
constexpr int OZ_S = 7, OZ_DEPTH = 6;             // FP64-equivalent: 28 slice products
constexpr int OZ_NAN = 1 << 24;                   // exponent of a row that holds a non-finite value

struct OzOperand {
    const __nv_bfloat16* ptr;
    int64_t rows, cols;     // cols: K extent (contiguous)
    int64_t ld;             // row pitch in elements (multiple of 8)
    int64_t plane;          // elements between planes (multiple of 8)
    int64_t nplanes;        // planes in all (batch included)
    int32_t zbatch;         // planes per batch item (0: shared by the batch)
};

// The products of one output part: segments ordered by level; segment q multiplies planes pa[q] and
// pb[q] (negated if neg[q]); levels first[l] .. first[l + 1].
struct OzPlan {
    int32_t nlev, split;                 // levels below `split` are converted to FP64 apart (0: one group)
    int16_t first[OZ_MAXLEV + 1];
    uint8_t pa[OZ_MAXSEG], pb[OZ_MAXSEG], neg[OZ_MAXSEG];
};

// The output parts of one launch (the real and the imaginary part of a complex product).
struct OzPlans {
    OzPlan part[2];
};

// One term of a part: sum over slices of A part a (planes a S + s) times B part b, with a sign.
struct OzTerm {
    int a, b;
    bool neg;
};
// K: products per segment (bounds the integer sums), S slices per operand part, s + t <= depth
inline OzPlan oz_plan(int S, int depth, int64_t K, const OzTerm* terms, int nterms) {
    OzPlan p{};
    p.nlev = depth + 1;
    int q = 0;
    for (int d = 0; d <= depth; ++d) {
        p.first[d] = (int16_t)q;
        for (int s = 0; s <= d; ++s) {
            if (s >= S || d - s >= S) continue;
            for (int t = 0; t < nterms; ++t) {
                p.pa[q] = (uint8_t)(terms[t].a * S + s);
                p.pb[q] = (uint8_t)(terms[t].b * S + d - s);
                p.neg[q++] = terms[t].neg ? 1 : 0;
            }
        }
    }
    p.first[depth + 1] = (int16_t)q;
    // a level's sum is at most 2^16 K nterms (d + 1); the largest second group that an int64 holds, and
    // the first group has to fit as well (K beyond 2^17 does not: p.nlev = 0)
    auto fits = [&](int a, int b) {
        double m = 0.0;
        for (int d = a; d < b; ++d) m = m * 512.0 + 65536.0 * (double)K * nterms * (d + 1);
        return m < 4.6e18;   // 2^62
    };
    while (p.split < p.nlev && !fits(p.split, p.nlev)) ++p.split;
    if (!fits(0, p.split)) p.nlev = 0;
    return p;
}

// complex products of operands staged as (real, imaginary) planes: op(A) B^T with A conjugated or not and
// B conjugated or not
inline OzPlans oz_plans_complex(int S, int depth, int64_t K, bool conjA, bool conjB) {
    const OzTerm re[2] = {{0, 0, false}, {1, 1, conjA == conjB}};
    const OzTerm im[2] = {{0, 1, conjB}, {1, 0, conjA}};
    return OzPlans{{oz_plan(S, depth, K, re, 2), oz_plan(S, depth, K, im, 2)}};
}

int oz_make_tmap(CUtensorMap* map, const OzOperand& op);

__device__ inline void oz_mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ inline void tmem_st32(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
        "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
        "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}

// 2^k as a double; NaN for the exponent sum of a non-finite row
__device__ inline double oz_pow2(int k) {
    if (k > -1022 && k < 1023) return __hiloint2double((1023 + k) << 20, 0);
    return k > OZ_NAN / 2 ? __longlong_as_double(0x7ff8000000000000LL) : ldexp(1.0, k);
}

// lower: skip tiles whose rows all lie above the diagonal.  blockIdx.z = 2 (z - z0) + part, z = b * ksplit + s; split
// s takes K blocks [s kchunk, min(nkb, (s + 1) kchunk)) of every segment.
// EPI: epi(z, part, row, col0, v[16], M, N) with the 16 columns' values before the 2^(eA + eB) scale.
// DF: the blocks of 256 are scaled by their level's power of two (exact) and added into double-float (hi, lo)
// registers with an error-free TwoSum instead of int64; the epilogue gets hi + lo (about 48 bits) with the level scale
// applied.  The refinement of the mixed solve uses it: its residual W enters FP32 products, whose rounding
// noise reaches the refined density matrix at 1e-11 and the next iteration's at 1e-9, so its results are kept to the
// last bit by keeping this order of additions.
template <class EPI, bool DF>
__global__ void __launch_bounds__(OZ_THREADS, 1)
    k_oz_gemm(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, int64_t M, int64_t N,
              const __grid_constant__ OzPlans plans, int32_t nkb, int32_t koffA, int32_t koffB, int32_t zA, int32_t zB,
              int lower, int32_t ksplit, int32_t kchunk, int32_t z0, EPI epi, int* err) {
    const int64_t m0 = (int64_t)blockIdx.x * OZ_T, n0 = (int64_t)blockIdx.y * OZ_T;
    if (lower && m0 + OZ_T - 1 < n0) return;
    extern __shared__ __align__(1024) unsigned char oz_smem_raw[];
    unsigned char* base = (unsigned char*)(((uintptr_t)oz_smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* sA = base;
    unsigned char* sB = base + OZ_STAGES * OZ_TILE_BYTES;
    uint64_t* full = (uint64_t*)(base + 2 * OZ_STAGES * OZ_TILE_BYTES);
    uint64_t* empty = full + OZ_STAGES;
    uint64_t* tfull = empty + OZ_STAGES;
    uint64_t* tfree = tfull + 2;
    uint64_t* accum = tfree + 2;
    uint32_t* tmem_slot = (uint32_t*)(accum + 1);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    volatile int* n_issued = abort_flag + 1;
    volatile int* n_consumed = abort_flag + 2;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int part = blockIdx.z & 1, z = (int)(blockIdx.z >> 1) + z0;
    const OzPlan& plan = plans.part[part];
    const int b = z / ksplit;
    const int klo = (z - b * ksplit) * kchunk;
    const int kn = min(kchunk, nkb - klo);   // K blocks of each segment

    if (threadIdx.x == 0) {
        for (int s = 0; s < OZ_STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int t = 0; t < 2; ++t) {
            mbar_init(&tfull[t], 1);
            mbar_init(&tfree[t], 8);
        }
        mbar_init(accum, 1);
        *abort_flag = 0;
        *n_issued = 0;
        *n_consumed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(512u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            int it = 0;
            bool ok = true;
            const int nseg = plan.first[plan.nlev];
            for (int q = 0; q < nseg && ok; ++q) {
                const int za = plan.pa[q] + zA * b, zb = plan.pb[q] + zB * b;
                for (int kb = 0; kb < kn; ++kb, ++it) {
                    const int s = it % OZ_STAGES;
                    if (it >= OZ_STAGES && !mbar_wait(&empty[s], ((uint32_t)(it / OZ_STAGES) & 1u) ^ 1u, abort_flag)) {
                        *abort_flag = 1;
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(&full[s], 2 * OZ_TILE_BYTES);
                    tma_load_3d(sA + s * OZ_TILE_BYTES, &mapA, &full[s], koffA + (klo + kb) * OZ_BK, (int32_t)m0, za);
                    tma_load_3d(sB + s * OZ_TILE_BYTES, &mapB, &full[s], koffB + (klo + kb) * OZ_BK, (int32_t)n0, zb);
                    *n_issued = it + 1;
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // instruction descriptor: D F32, A = B = BF16, K-major, M = N = 128; bit 13 negates A
            const uint32_t idesc0 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(OZ_T >> 3) << 17) |
                                    ((uint32_t)(OZ_T >> 4) << 24);
            int it = 0, grp = 0;
            bool ok = true;
            for (int l = 0; l < plan.nlev && ok; ++l) {
                const int total = (plan.first[l + 1] - plan.first[l]) * kn;
                int blk = 0;
                for (int q = plan.first[l]; q < plan.first[l + 1] && ok; ++q) {
                    const uint32_t idesc = idesc0 | (plan.neg[q] ? 1u << 13 : 0u);
                    for (int kb = 0; kb < kn; ++kb, ++it, ++blk) {
                        const int s = it % OZ_STAGES, buf = grp & 1;
                        const bool first = (blk & 3) == 0, last = (blk & 3) == 3 || blk == total - 1;
                        if (!mbar_wait(&full[s], (uint32_t)(it / OZ_STAGES) & 1u, abort_flag) ||
                            (first && grp > 1 && !mbar_wait(&tfree[buf], (uint32_t)((grp >> 1) - 1) & 1u, abort_flag))) {
                            *abort_flag = 1;
                            ok = false;
                            break;
                        }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const uint32_t a0 = smem_u32(sA + s * OZ_TILE_BYTES), b0 = smem_u32(sB + s * OZ_TILE_BYTES);
#pragma unroll
                        for (int kk = 0; kk < OZ_BK / 16; ++kk)
                            oz_mma_bf16(tmem + (uint32_t)(buf * OZ_T), umma_desc_sw128(a0 + kk * 32),
                                        umma_desc_sw128(b0 + kk * 32), idesc, (!first || kk > 0) ? 1u : 0u);
                        tc_commit(&empty[s]);
                        if (last) {
                            tc_commit(&tfull[buf]);
                            ++grp;
                        }
                        *n_consumed = it + 1;
                    }
                }
            }
            // every commit's arrival lands before the CTA gives its shared memory back
            tc_commit(accum);
            if (!*abort_flag && !mbar_wait(accum, 0, abort_flag)) *abort_flag = 1;
        }
        __syncwarp();
    } else {
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        const int64_t row = m0 + quarter * 32 + lane;
        // 16-column groups of the warp's part that hold results: the conversions run on the FP64 pipe and are most of a
        // small product's time (n = 2: 65 us a product with the whole tile converted)
        const int64_t cols = m0 + quarter * 32 < M ? N - (n0 + half * 64) : 0;
        const int live = (int)min((int64_t)4, max((int64_t)0, (cols + 15) / 16));
        const uint32_t trow = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * 64);
        const uint32_t thi = tmem + ((uint32_t)(quarter * 32) << 16) + 256u + (uint32_t)(half * 128);
        long long acc[DF ? 1 : 64];
        float fh[DF ? 64 : 1], fl[DF ? 64 : 1];
        if constexpr (DF) {
#pragma unroll
            for (int q = 0; q < 64; ++q) fh[q] = fl[q] = 0.f;
        } else {
#pragma unroll
            for (int q = 0; q < 64; ++q) acc[q] = 0;
        }
        bool ok = true;
        int grp = 0;
        for (int l = 0; l < plan.nlev && ok; ++l) {
            if constexpr (!DF) {
                if (l > 0 && l == plan.split) {
                    // the first levels in FP64 (exact up to one rounding) to TMEM
#pragma unroll
                    for (int h = 0; h < 4; ++h) {
                        if (h >= live) break;
                        uint32_t r[32];
#pragma unroll
                        for (int q = 0; q < 16; ++q) {
                            const double x = (double)acc[h * 16 + q];
                            r[2 * q] = (uint32_t)__double2loint(x);
                            r[2 * q + 1] = (uint32_t)__double2hiint(x);
                            acc[h * 16 + q] = 0;
                        }
                        __syncwarp();
                        tmem_st32(thi + (uint32_t)(h * 32), r);
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                } else if (l > 0) {
#pragma unroll
                    for (int q = 0; q < 64; ++q) acc[q] = (long long)((unsigned long long)acc[q] << 9);
                }
            }
            const float scl = __int_as_float((127 - (16 + 9 * l)) << 23);   // 2^-(16 + 9 l)
            const int ng = ((plan.first[l + 1] - plan.first[l]) * kn + 3) / 4;
            for (int g = 0; g < ng; ++g, ++grp) {
                const int buf = grp & 1;
                if (!mbar_wait_warp(&tfull[buf], (uint32_t)(grp >> 1) & 1u, abort_flag)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int h = 0; h < 64; h += 32) {
                    if (h / 16 >= live) break;
                    float v[32];
                    __syncwarp();
                    tmem_ld32(trow + (uint32_t)(buf * OZ_T + h), v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if constexpr (DF) {
#pragma unroll
                        for (int q = 0; q < 32; ++q) {
                            const float x = v[q] * scl;
                            const float sm = fh[h + q] + x;
                            const float bp = sm - fh[h + q];
                            fl[h + q] += (fh[h + q] - (sm - bp)) + (x - bp);
                            fh[h + q] = sm;
                        }
                    } else {
#pragma unroll
                        for (int q = 0; q < 32; ++q) acc[h + q] += (long long)__float2int_rn(v[q]);
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&tfree[buf]);
            }
        }
        const bool failed = __shfl_sync(0xffffffffu, (!ok || *abort_flag) ? 1 : 0, 0) != 0;
        if (failed) {
            if (lane == 0) *abort_flag = 1;
        } else {
            const double c2 = oz_pow2(-(16 + 9 * (plan.nlev - 1)));
            const double c1 = plan.split ? oz_pow2(-(16 + 9 * (plan.split - 1))) : 0.0;
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                if (h >= live) break;
                double d[16];
                if constexpr (DF) {
#pragma unroll
                    for (int q = 0; q < 16; ++q) d[q] = (double)fh[h * 16 + q] + (double)fl[h * 16 + q];
                } else if (plan.split) {
                    float r[32];
                    __syncwarp();   // the epilogue functor may leave rows beyond M behind; tcgen05.ld is .aligned
                    tmem_ld32(thi + (uint32_t)(h * 32), r);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int q = 0; q < 16; ++q)
                        d[q] = fma(__hiloint2double(__float_as_int(r[2 * q + 1]), __float_as_int(r[2 * q])), c1,
                                   (double)acc[h * 16 + q] * c2);
                } else {
#pragma unroll
                    for (int q = 0; q < 16; ++q) d[q] = (double)acc[h * 16 + q] * c2;
                }
                epi((int64_t)z, part, row, n0 + half * 64 + h * 16, d, M, N);
            }
        }
    }
    __syncwarp();
    __syncthreads();
    if (*abort_flag && threadIdx.x == 0) {
        atomicExch(err, 1);
        // drain: the MMAs in flight (accum) and the TMA loads issued but not consumed
        mbar_wait(accum, 0, nullptr);
        for (int it = *n_consumed; it < *n_issued; ++it)
            mbar_wait(&full[it % OZ_STAGES], (uint32_t)(it / OZ_STAGES) & 1u, nullptr);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
    }
}

// number of K splits launched when `want` are asked for: whole K blocks, none empty
inline int oz_ksplit_count(int64_t nkb, int64_t want) {
    if (want <= 1 || nkb <= 1) return 1;
    const int64_t chunk = (nkb + want - 1) / want;
    return (int)((nkb + chunk - 1) / chunk);
}

// K: products per segment (from element koffA / koffB of the operands' rows; the offsets are multiples of
// 8 elements, the 16 bytes TMA needs)
template <bool DF = false, class EPI>
int oz_gemm(cudaStream_t st, const OzOperand& A, int64_t koffA, const OzOperand& B, int64_t koffB, int64_t K,
            const OzPlans& plans, int64_t batch, bool lower, const EPI& epi, int* err, int64_t want_split = 1) {
    if (A.rows <= 0 || B.rows <= 0 || batch <= 0 || K <= 0) return 0;
    if ((A.ld % 8) || (B.ld % 8) || (A.plane % 8) || (B.plane % 8) || (koffA % 8) || (koffB % 8) ||
        ((uintptr_t)A.ptr % 16) || ((uintptr_t)B.ptr % 16)) {
        set_error(FORGE_ERR_ARG, "oz_gemm: operands must be 16-byte aligned with pitches multiple of 8 elements");
        return FORGE_ERR_ARG;
    }
    // DF: whole blocks of 256 products per segment
    const int64_t nkb = DF ? (K + 255) / 256 * 4 : (K + OZ_BK - 1) / OZ_BK;
    if (DF && want_split != 1) {
        set_error(FORGE_ERR_ARG, "oz_gemm: the double-float mode has no K split");
        return FORGE_ERR_ARG;
    }
    const int ks = oz_ksplit_count(nkb, want_split);
    if (!plans.part[0].nlev || !plans.part[1].nlev) {
        set_error(FORGE_ERR_ARG, "oz_gemm: K = %lld exceeds the exact integer sums", (long long)K);
        return FORGE_ERR_ARG;
    }
    CUtensorMap ma, mb;
    FORGE_TRY(oz_make_tmap(&ma, A));
    FORGE_TRY(oz_make_tmap(&mb, B));
    FORGE_CUDA(cudaFuncSetAttribute(k_oz_gemm<EPI, DF>, cudaFuncAttributeMaxDynamicSharedMemorySize, OZ_SMEM));
    // the grid's z extent holds both parts of 32767 products
    for (int64_t z0 = 0; z0 < batch * ks; z0 += OZ_GRID_Z) {
        const dim3 grd((unsigned)((A.rows + OZ_T - 1) / OZ_T), (unsigned)((B.rows + OZ_T - 1) / OZ_T),
                       (unsigned)(2 * std::min<int64_t>(OZ_GRID_Z, batch * ks - z0)));
        k_oz_gemm<EPI, DF><<<grd, OZ_THREADS, OZ_SMEM, st>>>(ma, mb, A.rows, B.rows, plans, (int32_t)nkb, (int32_t)koffA,
                                                         (int32_t)koffB, A.zbatch, B.zbatch, lower ? 1 : 0, ks,
                                                         (int32_t)((nkb + ks - 1) / ks), (int32_t)z0, epi, err);
        FORGE_LAUNCH_CHECK();
    }
    return 0;
}

// ---------------------------------------------------------------- slicing
// Integer arithmetic throughout: an FP64 operation costs 32 times an integer one here.

// exponent field of |x| (2047: Inf / NaN); the power-of-two scale of a row with largest field f is
// 2^(f - 1022) > |x|
__device__ inline int oz_field(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
__device__ inline int oz_expo(int field) { return field == 2047 ? OZ_NAN : field - 1022; }

// the S slices of x 2^-e (|x| < 2^e) as bf16 bits; digits of nine bits from a fixed-point value with
// 8 + 9 (S - 1) fraction bits
template <int S>
__device__ inline void oz_cut(double x, int e, unsigned short* out) {
    constexpr int FB = 8 + 9 * (S - 1);
    const long long bits = __double_as_longlong(x);
    const int f = (int)(bits >> 52) & 0x7ff;
    long long m = f ? (bits & 0xfffffffffffffLL) | (1LL << 52) : 0;   // subnormals: below 2^-1022
    const int sh = f - 1075 + FB - e;                                   // m 2^sh = |x| 2^(FB - e)
    if (sh >= 0)
        m <<= sh;
    else
        m = sh < -54 ? 0 : (m + (1LL << (-sh - 1))) >> -sh;
    if (bits < 0) m = -m;
#pragma unroll
    for (int s = S - 1; s > 0; --s) {
        const long long d = (long long)((unsigned long long)m << 55) >> 55;   // -256 .. 255
        m = (m - d) >> 9;
        out[s] = (unsigned short)(__float_as_uint((float)(int)d) >> 16);
    }
    out[0] = (unsigned short)(__float_as_uint((float)(int)m) >> 16);
}

// The same slices taken from the top, each the nearest integer (ties to even) of what the slices before it left:
// v_0 = rint(256 a), v_1 = rint(512 (256 a - v_0)), ...  (a = x 2^-e)
template <int S>
__device__ inline void oz_cut_rint(double x, int e, unsigned short* out) {
    const long long bits = __double_as_longlong(x);
    const int f = (int)(bits >> 52) & 0x7ff;
    long long r = f ? (bits & 0xfffffffffffffLL) | (1LL << 52) : 0;
    const int sh = f - 1013 - e;   // r 2^sh = |x| 2^(62 - e)
    if (sh >= 0) {
        r <<= sh;
    } else if (sh < -54) {
        r = r != 0;
    } else {
        const long long q = r >> -sh;
        r = q | ((q << -sh) != r);   // what is cut off only breaks ties
    }
    if (bits < 0) r = -r;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int u = 54 - 9 * s;
        const long long h = r + (1LL << (u - 1));
        long long v = h >> u;
        if ((h & ((1LL << u) - 1)) == 0) v &= ~1LL;
        r -= v << u;
        out[s] = (unsigned short)(__float_as_uint((float)(int)v) >> 16);
    }
}
template <int S, bool RINT>
__device__ inline void oz_cut_as(double x, int e, unsigned short* out) {
    if constexpr (RINT)
        oz_cut_rint<S>(x, e, out);
    else
        oz_cut<S>(x, e, out);
}

// Rows of the operand = columns of a column-major source: one CTA per (row, batch item).  LD: double2
// ld(b, row, k).  Planes (0..S-1: real, S..2S-1: imaginary) of row `row` at
// out + ((blockIdx.y * 2 S + p) * plane) + row * ldo + k; its scale to expo[b * estride + row].
template <int S, bool RINT = false, class LD>
__global__ void __launch_bounds__(256) k_oz_cols(LD ld, int64_t k1, int64_t kpad, unsigned short* __restrict__ out,
                                                 int64_t ldo, int64_t plane, int* __restrict__ expo, int64_t estride) {
    const int64_t row = blockIdx.x, b = blockIdx.y;
    int f = 0;
    for (int64_t k = threadIdx.x; k < k1; k += blockDim.x) {
        const double2 v = ld(b, row, k);
        f = max(f, max(oz_field(v.x), oz_field(v.y)));
    }
    __shared__ int red[8];
    f = __reduce_max_sync(0xffffffffu, f);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = f;
    __syncthreads();
    f = red[0];
#pragma unroll
    for (int q = 1; q < 8; ++q) f = max(f, red[q]);
    const int e = oz_expo(f);
    if (threadIdx.x == 0) expo[b * estride + row] = e;
    unsigned short* o = out + b * 2 * S * plane + row * ldo;
    const int ec = e == OZ_NAN ? 1025 : e;
    for (int64_t k = threadIdx.x; k < kpad; k += blockDim.x) {
        const double2 v = k < k1 ? ld(b, row, k) : make_double2(0.0, 0.0);
        unsigned short d[S];
        oz_cut_as<S, RINT>(v.x, ec, d);
#pragma unroll
        for (int s = 0; s < S; ++s) o[s * plane + k] = d[s];
        oz_cut_as<S, RINT>(v.y, ec, d);
#pragma unroll
        for (int s = 0; s < S; ++s) o[(S + s) * plane + k] = d[s];
    }
}

// Rows of the operand = rows of a column-major source, K = its columns: a CTA (32 x 8) takes 32 rows and
// transposes 32 x 32 tiles through shared memory.  Layout of the output as in k_oz_cols.
// diag (or null): sum of |v|^2 of every row in FP64, at diag[b * estride + row].
template <int S, bool RINT = false, class LD>
__global__ void __launch_bounds__(256) k_oz_rows(LD ld, int64_t rows, int64_t K, int64_t kpad,
                                                 unsigned short* __restrict__ out, int64_t ldo, int64_t plane,
                                                 int* __restrict__ expo, int64_t estride, double* __restrict__ diag) {
    const int64_t b = blockIdx.y, i0 = (int64_t)blockIdx.x * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int64_t Kb = ld.extent(b, K);   // columns of this batch item (the rest is zero)
    __shared__ double2 tile[32][33];
    __shared__ int red[8][33];
    const int64_t i = i0 + tx;
    int f = 0;
    for (int64_t k = ty; k < Kb; k += 8)
        if (i < rows) {
            const double2 v = ld(b, i, k);
            f = max(f, max(oz_field(v.x), oz_field(v.y)));
        }
    red[ty][tx] = f;
    __syncthreads();
    if (ty == 0) {
        for (int q = 1; q < 8; ++q) f = max(f, red[q][tx]);
        const int e = oz_expo(f);
        red[0][tx] = e;
        if (i < rows) expo[b * estride + i] = e;
    }
    __syncthreads();
    unsigned short* o = out + b * 2 * S * plane;
    __shared__ double dpart[8][32];
    double dtot = 0.0;
    for (int64_t kt = 0; kt < kpad; kt += 32) {
        double dsum = 0.0;
        for (int q = ty; q < 32; q += 8) {
            const int64_t k = kt + q;
            const double2 x = (i < rows && k < Kb) ? ld(b, i, k) : make_double2(0.0, 0.0);
            tile[q][tx] = x;
            if (diag) dsum += x.x * x.x + x.y * x.y;
        }
        if (diag) dpart[ty][tx] = dsum;
        __syncthreads();
        if (diag && ty == 0) {
            double t = 0.0;
            for (int y = 0; y < 8; ++y) t += dpart[y][tx];
            dtot += t;
        }
        for (int q = ty; q < 32; q += 8) {
            const int64_t r = i0 + q, k = kt + tx;
            if (r < rows && k < kpad) {
                const int e = red[0][q], ec = e == OZ_NAN ? 1025 : e;
                const double2 v = tile[tx][q];
                unsigned short d[S];
                oz_cut_as<S, RINT>(v.x, ec, d);
#pragma unroll
                for (int s = 0; s < S; ++s) o[s * plane + r * ldo + k] = d[s];
                oz_cut_as<S, RINT>(v.y, ec, d);
#pragma unroll
                for (int s = 0; s < S; ++s) o[(S + s) * plane + r * ldo + k] = d[s];
            }
        }
        __syncthreads();
    }
    if (diag && ty == 0 && i < rows) diag[b * estride + i] = dtot;
}

}  // namespace forge
