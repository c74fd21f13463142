// Tall-skinny Gram products C = alpha A^T B for the LOBPCG pencils of small blocks
// (the reference's MakeMatrix_d_blas, lobpcg_d_multi_mpi.h:191-250, with K = the
// grid and M, N = the block's columns): A is N x ma, B is N x mb, both column-major
// with leading dimension lda / ldb (state-major blocks), ma, mb <= 64.
//
// cuBLAS spends milliseconds on these shapes (an m x m output has too few tiles to
// spread K = 64k-1.7M rows over the GPU). Here K is split over blocks and, inside a block, over
// the warps of an output part of 32 x 32: a warp loads 8 rows of 32 + 32 columns, 16 bytes per
// lane, straight into the operand layout of mma.sync.m8n8k4.f64 and issues 32 products on them;
// A^T B1 and A^T B2 of one launch share the reads of A through L1. The warps' sums are added in
// shared memory and the blocks' sums by a second kernel, both in a fixed order. Several
// problems (blockIdx.y) run in one launch. Bound: DRAM at 32 columns (the products take 0.7 of
// its time), the FP64 pipe from 64 columns on. 8 problems of 64000 x 32, two right-hand blocks: 0.09 ms
// (0.06 ms of reads).
#include "gram_ts.h"
#include "qg_internal.h"

#include <algorithm>

namespace qg {
namespace {

constexpr int kMax = 64;
constexpr int kPart = 32;      // rows and columns of a warp's part of the output
constexpr int kThreads = 256;  // 8 warps: (parts of the output) x (row groups)

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}

// Rows r, r + 1 of a column, zero past the last row. VEC: r is even and the column 16-byte aligned.
template <bool VEC>
__device__ __forceinline__ double2 load2(const double* __restrict__ col, long long r, long long r1) {
    if (VEC && r + 1 < r1) return __ldg(reinterpret_cast<const double2*>(col + r));
    return make_double2(r < r1 ? __ldg(col + r) : 0.0, r + 1 < r1 ? __ldg(col + r + 1) : 0.0);
}

// gridDim.x blocks split the rows of problem blockIdx.y; rows_per_block is a multiple of 8.
template <bool VEC>
__global__ void __launch_bounds__(kThreads, 2) k_gram_ts_partial(const double* __restrict__ A, long long lda, long long sA,
                                                                 const double* __restrict__ B1,
                                                                 const double* __restrict__ B2, long long ldb, long long sB,
                                                                 long long N, int ma, int mb, long long rows_per_block,
                                                                 double* __restrict__ part) {
    __shared__ double2 red[kThreads * 4];
    constexpr int NT = kPart / 8;
    const int prob = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
    const int nb = B2 ? 2 : 1, pa = (ma + kPart - 1) / kPart, pb = (mb + kPart - 1) / kPart;
    const int parts = pa * pb * nb, groups = kThreads / 32 / parts;  // 1, 2, 4 or 8 parts
    const int mine = warp % parts, group = warp / parts;
    const int rhs = mine / (pa * pb), i0 = mine % pa * kPart, j0 = mine / pa % pb * kPart;
    const double* a = A + prob * sA;
    const double* b = (rhs ? B2 : B1) + prob * sB;
    const long long r0 = (long long)blockIdx.x * rows_per_block, r1 = min(N, r0 + rows_per_block);
    // columns past the last repeat an earlier one; their products are not stored
    const double* ca = a + min(i0 + r, ma - 1) * lda;
    const double* cb = b + min(j0 + r, mb - 1) * ldb;
    const int na8 = (ma - i0 - r + 7) / 8, nb8 = (mb - j0 - r + 7) / 8;  // tiles with this lane's column
    double acc[NT][NT][2] = {};
    for (long long p = r0 + 8 * group; p < r1; p += 8 * groups) {
        double2 va[NT], vb[NT];
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            va[t] = load2<VEC>(ca + (t < na8 ? 8 * t * lda : 0), p + 2 * q, r1);
            vb[t] = load2<VEC>(cb + (t < nb8 ? 8 * t * ldb : 0), p + 2 * q, r1);
        }
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j) dmma(acc[i][j], va[i].x, vb[j].x);
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j) dmma(acc[i][j], va[i].y, vb[j].y);
    }
    // the row groups of a part are added in order, one row of tiles at a time; compact result
    // part[((prob * nblocks + block) * nb + rhs) * ma * mb + i * mb + j]
    double* out = part + (((long long)prob * gridDim.x + blockIdx.x) * nb + rhs) * ma * mb;
#pragma unroll
    for (int i = 0; i < NT; ++i) {
        __syncthreads();
#pragma unroll
        for (int j = 0; j < NT; ++j) red[(warp * NT + j) * 32 + lane] = make_double2(acc[i][j][0], acc[i][j][1]);
        __syncthreads();
        if (group == 0) {
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                double2 s = red[(warp * NT + j) * 32 + lane];
                for (int g = 1; g < groups; ++g) {
                    const double2 v = red[((warp + g * parts) * NT + j) * 32 + lane];
                    s.x += v.x;
                    s.y += v.y;
                }
                const int ii = i0 + 8 * i + r, jj = j0 + 8 * j + 2 * q;
                if (ii < ma && jj < mb) out[ii * mb + jj] = s.x;
                if (ii < ma && jj + 1 < mb) out[ii * mb + jj + 1] = s.y;
            }
        }
    }
}

// 32 output elements per block, 8 threads per element: each adds every 8th block's partial sum, then
// the eight are added in order (the same order every call).
__global__ void __launch_bounds__(256) k_gram_ts_reduce(const double* __restrict__ part, int nblocks, int nb, int ma, int mb,
                                                        double alpha, double* __restrict__ C1, double* __restrict__ C2,
                                                        int ldc, long long sC) {
    __shared__ double sm[8][32];
    const int prob = blockIdx.y, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int e = blockIdx.x * 32 + lane, msz = ma * mb;
    double s = 0.0;
    if (e < nb * msz) {
        const double* p = part + (long long)prob * nblocks * nb * msz + e;
#pragma unroll 4
        for (int b = w; b < nblocks; b += 8) s += p[(long long)b * nb * msz];
    }
    sm[w][lane] = s;
    __syncthreads();
    if (w == 0 && e < nb * msz) {
        for (int i = 1; i < 8; ++i) s += sm[i][lane];
        const int ij = e % msz, i = ij / mb, j = ij % mb;
        double* C = (e < msz ? C1 : C2) + prob * sC;
        C[i + (long long)j * ldc] = alpha * s;
    }
}

}  // namespace

size_t gram_ts_scratch_doubles(long long N, int nprob, bool two) {
    const int nblocks = gram_ts_blocks(N, nprob);
    return (size_t)nprob * nblocks * (two ? 2 : 1) * kMax * kMax;
}

int gram_ts_blocks(long long N, int nprob) {
    // about 2 blocks per SM over all problems, at least 256 rows each
    const long long per = (2 * 148 + nprob - 1) / nprob;
    const long long b = std::min<long long>(per, (N + 255) / 256);
    return (int)std::max<long long>(1, b);
}

int gram_ts(const double* A, long long lda, long long sA, const double* B1, const double* B2, long long ldb,
            long long sB, long long N, int ma, int mb, double alpha, double* C1, double* C2, int ldc, long long sC,
            int nprob, double* scratch, cudaStream_t st) {
    if (ma <= 0 || mb <= 0 || ma > kMax || mb > kMax || N <= 0 || nprob <= 0) return QG_ERR_UNSUPPORTED;
    const int nblocks = gram_ts_blocks(N, nprob);
    const long long rows = ((N + nblocks - 1) / nblocks + 7) / 8 * 8;
    const uintptr_t al = (uintptr_t)A | (uintptr_t)B1 | (uintptr_t)B2;
    const bool vec = al % 16 == 0 && (lda | ldb | sA | sB) % 2 == 0;
    (vec ? k_gram_ts_partial<true> : k_gram_ts_partial<false>)<<<dim3(nblocks, nprob), kThreads, 0, st>>>(
        A, lda, sA, B1, B2, ldb, sB, N, ma, mb, rows, scratch);
    const int nb = B2 ? 2 : 1;
    k_gram_ts_reduce<<<dim3((nb * ma * mb + 31) / 32, nprob), 256, 0, st>>>(scratch, nblocks, nb, ma, mb, alpha, C1, C2, ldc,
                                                                            sC);
    QG_CUDA_TRY(cudaGetLastError());
    return QG_OK;
}

int gram_ts_tiled(const double* A, long long lda, long long sA, const double* B1, const double* B2, long long ldb,
                  long long sB, long long N, int ma, int mb, double alpha, double* C1, double* C2, int ldc,
                  long long sC, int nprob, double* scratch, cudaStream_t st) {
    for (int i0 = 0; i0 < ma; i0 += kMax)
        for (int j0 = 0; j0 < mb; j0 += kMax) {
            const int ta = std::min(kMax, ma - i0), tb = std::min(kMax, mb - j0);
            const int rc = gram_ts(A + (long long)i0 * lda, lda, sA, B1 + (long long)j0 * ldb,
                                   B2 ? B2 + (long long)j0 * ldb : nullptr, ldb, sB, N, ta, tb, alpha,
                                   C1 + i0 + (long long)j0 * ldc, C2 ? C2 + i0 + (long long)j0 * ldc : nullptr, ldc,
                                   sC, nprob, scratch, st);
            if (rc != QG_OK) return rc;
        }
    return QG_OK;
}

}  // namespace qg

extern "C" int qg_gram_small_d(qg_context ctx, long long N, int ma, int mb, const double* A, const double* B,
                               double alpha, double* C) {
    if (!ctx || N <= 0 || ma <= 0 || mb <= 0 || !A || !B || !C) return QG_ERR_INVALID;
    QG_CUDA_TRY(cudaSetDevice(ctx->device));
    double* scratch = nullptr;
    const size_t bytes = qg::gram_ts_scratch_doubles(N, 1, false) * sizeof(double);
    QG_CUDA_TRY(cudaMallocAsync(reinterpret_cast<void**>(&scratch), bytes, ctx->stream));
    const int rc = qg::gram_ts_tiled(A, N, 0, B, nullptr, N, 0, N, ma, mb, alpha, C, nullptr, ma, 0, 1, scratch,
                                     ctx->stream);
    cudaFreeAsync(scratch, ctx->stream);
    if (rc != QG_OK) return rc;
    QG_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    return QG_OK;
}
