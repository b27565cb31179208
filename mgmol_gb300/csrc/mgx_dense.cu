// Gram / H-matrix contractions and the small dense FP64 algebra of the
// orbital hot path on sm_103a:
//  - S = Psi^T Psi * vel and H = Psi^T (H Psi) * vel as split-K tall-skinny
//    products on CUDA cores (FP64 data with FP64 FMA, or FP32 data with FP32
//    FMA in a three-level summation ending in double-float within the
//    K-slice),
//    FP64 atomics across slices, then the finishing pass
//    (scale by vel, the |x| > 1e-14 filter of
//    src/LocalMatrices2DistMatrix.cc:16,60, symmetric fill of S);
//  - GramMatrix::updateLS / computeInverse (src/GramMatrix.cc:75-191):
//    blocked right-looking Cholesky with inverted diagonal blocks, the
//    inverse factor, and S^-1 = L^-T L^-1, all FP64;
//  - ProjectedMatrices::getEigSum (src/ProjectedMatrices.cc:550-566):
//    tr(H S^-1) as a device reduction.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "mgx_internal.cuh"
#include "mgx_slice.cuh"
#include "mgx_stencil.cuh"

namespace mgx
{

/* ------------------------------------------------------------------ */
/* split-K Gram kernel: C[i][j] += sum_p A[i][p] B[j][p]                 */
/* A, B orbital-major (row i at A + i*ld), 64x64 output tiles.            */
/* ------------------------------------------------------------------ */
constexpr int GT  = 64; // output tile
constexpr int GKC = 32; // k chunk
// FP32 data: three-level summation.  FMAs chain over 8 k values; every 8
// k values that chain's sum is added to a second FP32 sum; every
// GKC * GRAM_F32_CHAIN = 128 k values the second sum goes into a
// double-float (hi + lo, two FP32) accumulator by an error-free two-sum.
// The rounding error then grows like 8 + 16 terms of FP32 rounding instead
// of the whole K slice's length, for one FP32 add per 8 FMAs and a two-sum
// per 128.
constexpr int GRAM_F32_CHAIN = 4;
constexpr int GRAM_F32_INNER = 8;

/* s + e = a + b exactly (Knuth's two-sum; no reassociation, no multiply to
 * contract) */
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e)
{
    s              = a + b;
    const float bb = s - a;
    e              = (a - (s - bb)) + (b - bb);
}

/* tiles of a launch: column tile by column tile; with lower only those that
 * reach an entry i >= j + col0 */
__host__ __device__ inline int gram_first_row(int j, int lower, int col0, int nti)
{
    const int f = lower ? col0 / GT + j : 0;
    return f < nti ? f : nti;
}

/* only_if: nothing is done unless *only_if is set (the FP64 products that the
 * tensor cores took over run here when an operand is not finite) */
template <typename T>
__global__ void __launch_bounds__(256) gram_splitk_kernel(const T* __restrict__ A,
    const T* __restrict__ B, size_t ld, int n, int ncols, size_t K, size_t kslice,
    int lower, int col0, const int* __restrict__ only_if, double* __restrict__ C)
{
    __shared__ T As[GKC][GT + 1];
    __shared__ T Bs[GKC][GT + 1];
    if (only_if && *only_if == 0) return;
    const int nti = (n + GT - 1) / GT;
    int ti = blockIdx.x, tj = 0;
    for (int f; (f = gram_first_row(tj, lower, col0, nti), ti >= nti - f); tj++)
        ti -= nti - f;
    const int i0 = (gram_first_row(tj, lower, col0, nti) + ti) * GT, j0 = tj * GT;
    const size_t k0 = (size_t)blockIdx.y * kslice;
    const size_t k1 = min(K, k0 + kslice);
    const int tid   = threadIdx.x;
    const int tx = tid % 16, ty = tid / 16; // 16 x 16 threads, 4x4 outputs each
    T acc[4][4];
    float mid[4][4];          // FP32 data: the sum of the 8-term chains
    float hi[4][4], lo[4][4]; // FP32 data: the double-float sum of the chains
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 4; b++)
        {
            acc[a][b] = (T)0;
            mid[a][b] = 0.f;
            hi[a][b]  = 0.f;
            lo[a][b]  = 0.f;
        }
    int chain = 0;
    for (size_t kc = k0; kc < k1; kc += GKC)
    {
        // 64 rows x 32 k for each operand: 2048 elements, 8 per thread
#pragma unroll
        for (int r = 0; r < 8; r++)
        {
            const int e   = tid + r * 256;
            const int row = e / GKC;
            const int kk  = e % GKC;
            const size_t k = kc + kk;
            T av = (T)0, bv = (T)0;
            if (k < k1)
            {
                if (i0 + row < n) av = A[(size_t)(i0 + row) * ld + k];
                if (j0 + row < ncols) bv = B[(size_t)(j0 + row) * ld + k];
            }
            As[kk][row] = av;
            Bs[kk][row] = bv;
        }
        __syncthreads();
#pragma unroll 8
        for (int kk = 0; kk < GKC; kk++)
        {
            T a[4], b[4];
#pragma unroll
            for (int q = 0; q < 4; q++)
            {
                a[q] = As[kk][ty + 16 * q];
                b[q] = Bs[kk][tx + 16 * q];
            }
#pragma unroll
            for (int p = 0; p < 4; p++)
#pragma unroll
                for (int q = 0; q < 4; q++)
                    acc[p][q] += a[p] * b[q];
            if constexpr (sizeof(T) == 4)
            {
                if (kk % GRAM_F32_INNER == GRAM_F32_INNER - 1)
                {
#pragma unroll
                    for (int p = 0; p < 4; p++)
#pragma unroll
                        for (int q = 0; q < 4; q++)
                        {
                            mid[p][q] += (float)acc[p][q];
                            acc[p][q] = (T)0;
                        }
                }
            }
        }
        __syncthreads();
        if constexpr (sizeof(T) == 4)
        {
            if (++chain == GRAM_F32_CHAIN || kc + GKC >= k1)
            {
                chain = 0;
#pragma unroll
                for (int p = 0; p < 4; p++)
#pragma unroll
                    for (int q = 0; q < 4; q++)
                    {
                        float sum, err;
                        two_sum(hi[p][q], mid[p][q], sum, err);
                        hi[p][q] = sum;
                        lo[p][q] += err;
                        mid[p][q] = 0.f;
                    }
            }
        }
    }
#pragma unroll
    for (int p = 0; p < 4; p++)
#pragma unroll
        for (int q = 0; q < 4; q++)
        {
            const int i = i0 + ty + 16 * p, j = j0 + tx + 16 * q;
            double v;
            if constexpr (sizeof(T) == 4)
                v = (double)hi[p][q] + (double)lo[p][q];
            else
                v = (double)acc[p][q];
            if (i < n && j < ncols) atomicAdd(&C[(size_t)j * n + i], v);
        }
}

/* S or H finishing: scale, filter, (S) mirror the lower triangle */
__global__ void gram_finish_kernel(double* C, int n, double vel, int symmetric)
{
    const size_t nn = (size_t)n * n;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < nn;
         t += (size_t)gridDim.x * blockDim.x)
    {
        const int i = (int)(t % n), j = (int)(t / n);
        if (symmetric && i < j) continue;
        double x = C[t] * vel;
        if (!(fabs(x) > 1.e-14)) x = 0.;
        C[t] = x;
        if (symmetric && i != j) C[(size_t)i * n + j] = x;
    }
}

/* C += A B^T of n x ncols functions of K points (with lower, at least the
 * entries i >= j + col0) for each of nf products with the same A.  FP64
 * products of some size are formed from slices on the tensor cores; the
 * CUDA-core kernels behind them run only when an operand is not finite. */
static int gram_add(mgx_ctx* ctx, int dtype, const void* A, size_t ld, size_t K, int n,
    const sl::Factor* f, int nf, cudaStream_t s)
{
    int* only_if = nullptr;
    if (dtype == MGX_F64 && sl::pays(ctx, n, f[0].ncols, K))
    {
        const int st = sl::accumulate(ctx, (const double*)A, ld, K, n, f, nf, &only_if, s);
        if (st == MGX_NO_MEMORY)
            only_if = nullptr; // no room for the planes: the CUDA cores do it
        else if (st != MGX_OK)
            return st;
    }
    const int nti = (n + GT - 1) / GT;
    for (int q = 0; q < nf; q++)
    {
        const int ncols = f[q].ncols, lower = f[q].lower, col0 = f[q].col0;
        const int ntj = (ncols + GT - 1) / GT;
        int ntiles    = 0;
        for (int j = 0; j < ntj; j++)
            ntiles += nti - gram_first_row(j, lower, col0, nti);
        int ksplit    = std::max(1, (8 * ctx->sm_count + ntiles - 1) / ntiles);
        size_t kslice = (K + ksplit - 1) / ksplit;
        kslice        = ((kslice + GKC - 1) / GKC) * GKC;
        ksplit        = (int)((K + kslice - 1) / kslice);
        if (ksplit > 65535) return fail(MGX_UNSUPPORTED, "K too large for split");
        dim3 grid(ntiles, ksplit);
        if (dtype == MGX_F64)
            gram_splitk_kernel<double><<<grid, 256, 0, s>>>((const double*)A, f[q].B, ld, n, ncols,
                K, kslice, lower, col0, only_if, f[q].C);
        else
            gram_splitk_kernel<float><<<grid, 256, 0, s>>>((const float*)A, (const float*)f[q].B,
                ld, n, ncols, K, kslice, lower, col0, only_if, f[q].C);
        MGX_LAUNCH_CHECK("gram_splitk_kernel");
    }
    return MGX_OK;
}

static int gram_begin(double* C, int n, cudaStream_t s)
{
    return cuda_check(cudaMemsetAsync(C, 0, (size_t)n * n * sizeof(double), s), "gram zero");
}

static int gram_finish(double* C, int n, double vel, int symmetric, cudaStream_t s)
{
    const int nb = (int)std::min<size_t>(((size_t)n * n + 255) / 256, 4096);
    gram_finish_kernel<<<nb, 256, 0, s>>>(C, n, vel, symmetric);
    MGX_LAUNCH_CHECK("gram_finish_kernel");
    return MGX_OK;
}

int gram_cuda_cores(mgx_ctx* ctx, int dtype, const void* A, const void* B,
    size_t ld, size_t K, int n, double vel, int symmetric, double* C,
    cudaStream_t s)
{
    MGX_TRY(gram_begin(C, n, s));
    const sl::Factor f = { (const double*)B, n, symmetric, 0, C };
    MGX_TRY(gram_add(ctx, dtype, A, ld, K, n, &f, 1, s));
    return gram_finish(C, n, vel, symmetric, s);
}

/* S, H and B of FP64 blocks in one go, B Psi whole in `work`: Psi is sliced
 * once for the three products */
int gram_hmat_matb_f64(mgx_ctx* ctx, const double* psi, const double* hpsi, size_t ld, size_t K,
    int n, double vel, double* S, double* H, double* Bm, double* work, cudaStream_t s)
{
    MGX_TRY(rhs_block(ctx->grid, MGX_F64, psi, ld, work, ld, n, s));
    double* C[3]         = { S, H, Bm };
    const sl::Factor f[] = { { psi, n, 1, 0, S }, { hpsi, n, 0, 0, H }, { work, n, 1, 0, Bm } };
    for (double* c : C)
        MGX_TRY(gram_begin(c, n, s));
    MGX_TRY(gram_add(ctx, MGX_F64, psi, ld, K, n, f, 3, s));
    for (int i = 0; i < 3; i++)
        MGX_TRY(gram_finish(C[i], n, vel, f[i].lower, s));
    return MGX_OK;
}

/* B = Psi^T (B Psi) * vel (LocGridOrbitals::computeMatB,
 * src/LocGridOrbitals.cc:1428-1487) on CUDA cores: B Psi is formed `wf`
 * functions at a time in `work` (leading dimension ld) by the Mehrstellen
 * right-hand-side stencil, and only output tiles that reach the lower
 * triangle are computed; the finishing pass mirrors the lower triangle. */
int matb_cuda_cores(mgx_ctx* ctx, int dtype, const void* psi, size_t ld, size_t K, int n,
    double vel, double* C, void* work, int wf, cudaStream_t s)
{
    if (wf <= 0) return fail(MGX_BAD_ARG, "matB: empty work block");
    const size_t es = dtype_size(dtype);
    MGX_TRY(gram_begin(C, n, s));
    for (int c0 = 0; c0 < n; c0 += wf)
    {
        const int nc = std::min(wf, n - c0);
        MGX_TRY(rhs_block(ctx->grid, dtype, (const char*)psi + (size_t)c0 * ld * es, ld, work,
            ld, nc, s));
        const sl::Factor f = { (const double*)work, nc, 1, c0, C + (size_t)c0 * n };
        MGX_TRY(gram_add(ctx, dtype, psi, ld, K, n, &f, 1, s));
    }
    return gram_finish(C, n, vel, 1, s);
}

/* ------------------------------------------------------------------ */
/* generic FP64 GEMM, column-major: C = alpha op(A) op(B) + beta C        */
/* ------------------------------------------------------------------ */
// On the FP64 units, 2 multiply-adds per SM and clock: a tile of TS x TS x k
// takes TS^2 k / 2 clocks of its SM, so the tile is the largest one that
// still spreads over all SMs (64^3: 69 us on one SM, 5 us in 16 x 16 tiles).
// lower_only: entries i + roff >= j; blockIdx.z: a batch of equal products at
// strides sA, sB, sC; only_if as in gram_splitk_kernel, and where it says
// sl::LOST the result is NaN.
template <bool TA, bool TB, int TS>
__global__ void __launch_bounds__(256) dgemm_kernel(int m, int n, int k,
    double alpha, const double* __restrict__ A, int lda,
    const double* __restrict__ B, int ldb, double beta, double* C, int ldc,
    int lower_only, int roff, size_t sA, size_t sB, size_t sC, const int* __restrict__ only_if)
{
    constexpr int R = TS / 16;
    __shared__ double As[16][TS + 1];
    __shared__ double Bs[16][TS + 1];
    const int take = only_if ? *only_if : 1;
    if (take == 0) return;
    A += blockIdx.z * sA;
    B += blockIdx.z * sB;
    C += blockIdx.z * sC;
    const int i0 = blockIdx.x * TS, j0 = blockIdx.y * TS;
    if (lower_only && i0 + TS - 1 + roff < j0) return;
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    double acc[R][R] = {};
    for (int kc = 0; kc < k; kc += 16)
    {
#pragma unroll
        for (int r = 0; r < R; r++)
        {
            // the 16 x TS elements of each operand along the direction in
            // which it is contiguous
            const int e = tid + r * 256;
            {
                const int mm = TA ? e / 16 : e % TS, kk = TA ? e % 16 : e / TS;
                const int i = i0 + mm, kq = kc + kk;
                As[kk][mm] = (i < m && kq < k) ? (TA ? A[(size_t)i * lda + kq] : A[(size_t)kq * lda + i])
                                               : 0.;
            }
            {
                const int mm = TB ? e % TS : e / 16, kk = TB ? e / TS : e % 16;
                const int j = j0 + mm, kq = kc + kk;
                Bs[kk][mm] = (j < n && kq < k) ? (TB ? B[(size_t)kq * ldb + j] : B[(size_t)j * ldb + kq])
                                               : 0.;
            }
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < 16; kk++)
        {
            double a[R], b[R];
#pragma unroll
            for (int q = 0; q < R; q++)
            {
                a[q] = As[kk][tx + 16 * q];
                b[q] = Bs[kk][ty + 16 * q];
            }
#pragma unroll
            for (int p = 0; p < R; p++)
#pragma unroll
                for (int q = 0; q < R; q++)
                    acc[p][q] = fma(a[p], b[q], acc[p][q]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int p = 0; p < R; p++)
#pragma unroll
        for (int q = 0; q < R; q++)
        {
            const int i = i0 + tx + 16 * p, j = j0 + ty + 16 * q;
            if (i < m && j < n && (!lower_only || i + roff >= j))
            {
                double* c = C + (size_t)j * ldc + i;
                *c        = take == sl::LOST
                                ? __longlong_as_double(0x7ff8000000000000ll)
                                : alpha * acc[p][q] + (beta == 0. ? 0. : beta * *c);
            }
        }
}

/* C = alpha op(A) op(B) + beta C on the FP64 units */
struct Gemm
{
    bool ta, tb;
    int m, n, k;
    double alpha;
    const double* A;
    int lda;
    const double* B;
    int ldb;
    double beta;
    double* C;
    int ldc;
    int lower = 0;
    int batch = 1;
    size_t sA = 0, sB = 0, sC = 0;
};

template <bool TA, bool TB>
static int dgemm_t(const Gemm& g, int roff, const int* only_if, int sms, cudaStream_t s)
{
    auto tiles = [&](int ts) {
        return (long)((g.m + ts - 1) / ts) * ((g.n + ts - 1) / ts) * g.batch;
    };
    const int ts = tiles(64) >= sms ? 64 : tiles(32) >= sms ? 32 : 16;
    const dim3 grid((g.m + ts - 1) / ts, (g.n + ts - 1) / ts, g.batch);
    auto kern = ts == 64 ? dgemm_kernel<TA, TB, 64>
                         : ts == 32 ? dgemm_kernel<TA, TB, 32> : dgemm_kernel<TA, TB, 16>;
    kern<<<grid, 256, 0, s>>>(g.m, g.n, g.k, g.alpha, g.A, g.lda, g.B, g.ldb, g.beta, g.C, g.ldc,
        g.lower, roff, g.sA, g.sB, g.sC, only_if);
    MGX_LAUNCH_CHECK("dgemm_kernel");
    return MGX_OK;
}

static int dgemm(const Gemm& g, int sms, cudaStream_t s, int roff = 0, const int* only_if = nullptr)
{
    if (g.m <= 0 || g.n <= 0) return MGX_OK;
    if (!g.ta && !g.tb) return dgemm_t<false, false>(g, roff, only_if, sms, s);
    if (!g.ta && g.tb) return dgemm_t<false, true>(g, roff, only_if, sms, s);
    if (g.ta && !g.tb) return dgemm_t<true, false>(g, roff, only_if, sms, s);
    return dgemm_t<true, true>(g, roff, only_if, sms, s);
}

/* C = alpha op(A) op(B) + beta C, from slices on the tensor cores where they
 * pay (C may then alias A or B only as far as it may for the kernel above,
 * which takes over when an operand is not finite) */
static int gemm(mgx_ctx* ctx, const Gemm& g, cudaStream_t s)
{
    if (g.m <= 0 || g.n <= 0) return MGX_OK;
    if (g.batch == 1 && sl::pays(ctx, g.m, g.n, g.k))
    {
        const sl::View a = { g.A, (size_t)g.lda, (size_t)g.m, (size_t)g.k, g.ta };
        const sl::View b = { g.B, (size_t)g.ldb, (size_t)g.n, (size_t)g.k, !g.tb };
        const sl::Target t
            = { g.C, (size_t)g.ldc, nullptr, g.alpha, g.beta, g.C, (size_t)g.ldc, g.lower, 0 };
        const int st = sl::store(ctx, a, b, t, s, [&](size_t r0, size_t rows, const int* bad) {
            Gemm c = g;
            c.m    = (int)rows;
            c.A += g.ta ? r0 * g.lda : r0;
            c.C += r0;
            return dgemm(c, ctx->sm_count, s, (int)r0, bad);
        });
        if (st != MGX_NO_MEMORY) return st;
    }
    return dgemm(g, ctx->sm_count, s);
}

/* ------------------------------------------------------------------ */
/* orbital block times a small FP64 matrix on CUDA cores (MPgemmNN,      */
/* src/linear_algebra/mputils.cc:719-760):                               */
/*   out_j[p] = sum_i psi_i[p] theta(i, j) + beta cin_j[p], j < ncols,   */
/*   theta column j at theta + j * ldt                                   */
/* ACC double: FP64 accumulation as the reference does for both orbital  */
/* types; ACC float: theta rounded to FP32 and FP32 FMA.  Tiles of 128   */
/* points x 64 functions, 8 x 4 results per thread.  cin may alias out.  */
/* only_if as in dgemm_kernel.                                          */
/* ------------------------------------------------------------------ */
template <typename T, typename ACC>
__global__ void __launch_bounds__(256) psi_theta_kernel(size_t npts, int n,
    const T* __restrict__ psi, size_t ld, const double* __restrict__ theta, int ldt,
    int ncols, double beta, const T* cin, T* out, const int* __restrict__ only_if)
{
    __shared__ ACC As[16][128];
    __shared__ ACC Bs[16][65];
    const int take = only_if ? *only_if : 1;
    if (take == 0) return;
    const size_t p0 = (size_t)blockIdx.x * 128;
    const int j0 = blockIdx.y * 64;
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    ACC acc[8][4];
#pragma unroll
    for (int a = 0; a < 8; a++)
#pragma unroll
        for (int b = 0; b < 4; b++)
            acc[a][b] = ACC(0);
    for (int kc = 0; kc < n; kc += 16)
    {
#pragma unroll
        for (int r = 0; r < 8; r++)
        {
            const int e = tid + r * 256;
            const int mm = e % 128, kk = e / 128;
            const size_t p = p0 + mm;
            const int i = kc + kk;
            As[kk][mm] = (p < npts && i < n) ? (ACC)psi[(size_t)i * ld + p] : ACC(0);
        }
#pragma unroll
        for (int r = 0; r < 4; r++)
        {
            const int e = tid + r * 256;
            const int kk = e % 16, jj = e / 16;
            const int i = kc + kk, j = j0 + jj;
            Bs[kk][jj] = (i < n && j < ncols) ? (ACC)theta[(size_t)j * ldt + i] : ACC(0);
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < 16; kk++)
        {
            ACC a[8], b[4];
#pragma unroll
            for (int q = 0; q < 8; q++) a[q] = As[kk][tx + 16 * q];
#pragma unroll
            for (int q = 0; q < 4; q++) b[q] = Bs[kk][ty + 16 * q];
#pragma unroll
            for (int u = 0; u < 8; u++)
#pragma unroll
                for (int v = 0; v < 4; v++)
                    acc[u][v] = fma(a[u], b[v], acc[u][v]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int v = 0; v < 4; v++)
    {
        const int j = j0 + ty + 16 * v;
        if (j >= ncols) continue;
#pragma unroll
        for (int u = 0; u < 8; u++)
        {
            const size_t p = p0 + tx + 16 * u;
            if (p >= npts) continue;
            const size_t o = (size_t)j * ld + p;
            double r = (double)acc[u][v];
            if (beta != 0.) r += beta * (double)cin[o];
            if (take == sl::LOST) r = __longlong_as_double(0x7ff8000000000000ll);
            out[o] = (T)r;
        }
    }
}

/* kind 0: FP64 orbitals (from slices on the tensor cores where they pay, the
 * CUDA-core kernel then only for operands that are not finite); 1: FP32
 * orbitals, FP64 accumulation; 2: FP32 orbitals, FP32 accumulation */
int psi_theta_cuda_cores(mgx_ctx* ctx, int kind, const void* psi, size_t ld, size_t npts, int n,
    const double* theta, int ldt, int ncols, double beta, const void* cin, void* out,
    cudaStream_t s)
{
    if (n <= 0 || ncols <= 0 || npts == 0) return MGX_OK;
    const unsigned gy = (unsigned)((ncols + 63) / 64);
    if (gy > 65535) return fail(MGX_UNSUPPORTED, "too many functions");
    auto cores = [&](size_t p0, size_t np, const int* only_if) -> int {
        const dim3 grid((unsigned)((np + 127) / 128), gy);
        if (kind == 0)
            psi_theta_kernel<double, double><<<grid, 256, 0, s>>>(np, n, (const double*)psi + p0,
                ld, theta, ldt, ncols, beta, cin ? (const double*)cin + p0 : nullptr,
                (double*)out + p0, only_if);
        else if (kind == 1)
            psi_theta_kernel<float, double><<<grid, 256, 0, s>>>(np, n, (const float*)psi + p0, ld,
                theta, ldt, ncols, beta, cin ? (const float*)cin + p0 : nullptr, (float*)out + p0,
                only_if);
        else
            psi_theta_kernel<float, float><<<grid, 256, 0, s>>>(np, n, (const float*)psi + p0, ld,
                theta, ldt, ncols, beta, cin ? (const float*)cin + p0 : nullptr, (float*)out + p0,
                only_if);
        MGX_LAUNCH_CHECK("psi_theta_kernel");
        return MGX_OK;
    };
    if (kind == 0 && sl::pays(ctx, npts, ncols, n))
    {
        const sl::View a = { (const double*)psi, ld, npts, (size_t)n, false };
        const sl::View b = { theta, (size_t)ldt, (size_t)ncols, (size_t)n, true };
        const sl::Target t
            = { (double*)out, ld, nullptr, 1., beta, (const double*)cin, ld, 0, 0 };
        const int st = sl::store(ctx, a, b, t, s, cores);
        if (st != MGX_NO_MEMORY) return st;
    }
    return cores(0, npts, nullptr);
}

/* ------------------------------------------------------------------ */
/* Cholesky                                                             */
/* ------------------------------------------------------------------ */
constexpr int NB        = 64;  // diagonal blocks, factored and inverted by one CTA
constexpr int OB        = 256; // blocks of the products between them
constexpr int DIAG_SMEM = 2 * NB * (NB + 1) * sizeof(double);

/* 1 / d to the last bit or two for d of exponent -1020 .. 1020: an FP32
 * reciprocal of the leading mantissa bits and one cubic Newton step.  Three
 * FP64 operations: each occupies its SM's FP64 unit for 16 clocks per warp, and
 * the division this replaces stood on the critical path of every column. */
__device__ __forceinline__ bool reciprocal_ok(double d)
{
    const int hi = __double2hiint(d); // positive, no extreme exponent
    return hi >= 0x00300000 && hi < 0x7fb00000;
}
__device__ __forceinline__ double reciprocal(double d)
{
    const int hi   = __double2hiint(d), lo = __double2loint(d);
    const double m = __hiloint2double((hi & 0x000fffff) | 0x3ff00000, lo); // [1, 2)
    const unsigned t
        = __float_as_uint(__frcp_rn(__uint_as_float(0x3f800000u | ((hi & 0xfffff) << 3) | ((unsigned)lo >> 29))));
    const double r = __hiloint2double((int)(t >> 3) + ((1023 - 127) << 20), (int)(t << 29));
    const double e = fma(-m, r, 1.);
    const double q = fma(r, fma(e, e, e), r); // in (1/2, 1]
    return __hiloint2double(__double2hiint(q) - (((hi >> 20) - 1023) << 20), __double2loint(q));
}

/* Factor the diagonal block A[k0:k0+nb, k0:k0+nb] (lower), write L_kk in
 * place (upper part zeroed) and its inverse W (nb x nb, column-major, ld
 * NB) to `winv`.  Sets *info to the 1-based global pivot index on failure.
 *
 * One sweep over the columns factors and inverts: with A = G D G^T, G unit
 * lower, column j takes G(i, j) = u_i / d_j times row j of [G^-1 | A] from
 * each row i > j, in one array whose columns before j already hold G^-1 and
 * the others what is left of A (in-place Gauss-Jordan).  L = G D^1/2 and W =
 * D^-1/2 G^-1 are scaled at the end, all columns at once.  1 / d_j itself stands
 * in the array, so where the block's diagonal leaves 2^-500 .. 2^500, row and
 * column i are taken times a power of two that brings A(i, i) between 1 and 4
 * (the bits of L and W do not depend on it): pivots of any exponent, subnormal
 * ones too, are factored.  (Done always, it took 2 of 73 us.)  Eight warps: two
 * column halves x four row groups, a lane per column, so that all four FP64
 * units work; the warp that updates the next pivot forms its reciprocal
 * before its other rows, so that the others need not wait for it.  Bound by
 * the FP64 units of its SM (175 k multiply-adds at 2 per clock would be 23 us
 * at 64). */
__global__ void __launch_bounds__(256) potrf_diag_kernel(double* A, int n, int k0,
    int nb, double* winv, int* info)
{
    extern __shared__ double dsm[];
    double(*X)[NB + 1] = reinterpret_cast<double(*)[NB + 1]>(dsm);
    double(*U)[NB + 1] = reinterpret_cast<double(*)[NB + 1]>(dsm + NB * (NB + 1)); // u columns
    __shared__ double inv[NB], sq[NB], up[NB], down[NB]; // up: the powers of two of the rows
    __shared__ int bad;
    if (*info != 0) return;
    const int tid = threadIdx.x;
    for (int e = tid; e < NB * NB; e += blockDim.x)
    {
        const int i = e % NB, j = e / NB;
        X[i][j]     = (i >= j && i < nb && j < nb) ? A[(size_t)(k0 + j) * n + k0 + i] : 0.;
    }
    if (tid == 0) bad = 0;
    __syncthreads();
    int k = 0; // the exponent of row tid over two, -537 .. 511
    if (tid < nb && X[tid][tid] > 0. && isfinite(X[tid][tid])) k = ilogb(X[tid][tid]) >> 1;
    const bool far = __syncthreads_or(k < -250 || k >= 250);
    if (far)
    {
        if (tid < NB)
        {
            up[tid]   = scalbn(1., -k);
            down[tid] = scalbn(1., k);
        }
        __syncthreads();
        for (int e = tid; e < NB * NB; e += blockDim.x)
            X[e % NB][e / NB] = X[e % NB][e / NB] * up[e % NB] * up[e / NB];
        __syncthreads();
    }
    if (tid < NB) U[tid][0] = X[tid][0];
    __syncthreads();
    // the pivot d of column j: its reciprocal, or -1 for a failure
    auto pivot = [&](int j, double d) {
        if (reciprocal_ok(d))
            inv[j] = reciprocal(d);
        else if (d > 0. && isfinite(d))
            inv[j] = 1. / d;
        else
        {
            inv[j] = -1.;
            bad    = k0 + j + 1;
        }
    };
    if (tid == 0) pivot(0, X[0][0]);
    __syncthreads();
    const int warp = tid / 32, lane = tid & 31;
    const int half = warp >> 2, wr = warp & 3;
    const int c = 32 * half + lane;
    for (int j = 0; j < nb; j++)
    {
        if (__double2hiint(inv[j]) < 0) break;
        // row j of [G^-1 | A] over d_j at this lane's column
        const double v = (c < j ? X[j][c] : c == j ? 1. : U[c][j]) * inv[j];
        // its rows from the diagonal down, the first of all with the pivot, the
        // others four at a time (the loads of four before the first store)
        int i = j + 1 + wr;
        if (wr == 0 && i < nb)
        {
            if (i >= 32 * half)
            {
                const double x = (c == j ? 0. : X[i][c]) - U[i][j] * v;
                if (c <= i) X[i][c] = x;
                if (c == j + 1) U[i][j + 1] = x;
                if (half == (i >> 5))
                {
                    const double d = __shfl_sync(0xffffffffu, x, i & 31);
                    if (lane == 0) pivot(i, d);
                }
            }
            i += 4;
        }
        if (i < 32 * half) i += (32 * half - i + 3) / 4 * 4; // columns past the diagonal
        for (; i < nb; i += 16)
        {
            double x[4], u[4];
#pragma unroll
            for (int q = 0; q < 4; q++)
            {
                const int r = min(i + 4 * q, nb - 1);
                x[q]        = X[r][c];
                u[q]        = U[r][j];
            }
#pragma unroll
            for (int q = 0; q < 4; q++)
            {
                const int r = i + 4 * q;
                if (r >= nb) break;
                const double y = (c == j ? 0. : x[q]) - u[q] * v;
                if (c <= r) X[r][c] = y;
                if (c == j + 1) U[r][j + 1] = y;
            }
        }
        __syncthreads();
    }
    if (bad) // set before the last barrier that every thread has passed
    {
        if (tid == 0) atomicCAS(info, 0, bad);
        return;
    }
    for (int i = tid; i < nb; i += blockDim.x)
    {
        const double r = sqrt(U[i][i]);
        sq[i]          = r;
        inv[i]         = 1. / r;
    }
    __syncthreads();
    for (int e = tid; e < nb * nb; e += blockDim.x)
    {
        const int i = e % nb, j = e / nb;
        double l = i > j ? U[i][j] * inv[j] : i == j ? sq[i] : 0.;
        double w = i > j ? X[i][j] * inv[i] : i == j ? inv[i] : 0.;
        if (far)
        {
            l *= down[i];
            w *= up[j];
        }
        A[(size_t)(k0 + j) * n + k0 + i] = l;
        winv[(size_t)j * NB + i]         = w;
    }
}

/* The panel of a Cholesky step in place: rows [k0 + nb, rend) of columns
 * k0 .. k0+nb of A (column-major, leading dimension n) become
 * A_panel W^T, W = L_kk^-1 (lower, column-major, leading dimension NB):
 * the L_ik = A_ik L_kk^-T of the blocked algorithm.  16 rows per CTA. */
constexpr int PANEL_ROWS = 16;

__global__ void __launch_bounds__(256) panel_trsm_kernel(double* A, int n, int k0, int nb, int rend,
    const double* __restrict__ winv)
{
    __shared__ double Ws[NB][NB + 1];
    __shared__ double As[PANEL_ROWS][NB + 1];
    const int tid = threadIdx.x;
    const int r0  = k0 + nb + blockIdx.x * PANEL_ROWS;
    for (int e = tid; e < NB * NB; e += blockDim.x)
    {
        const int i = e % NB, j = e / NB;
        Ws[i][j]    = (i >= j && i < nb) ? winv[(size_t)j * NB + i] : 0.;
    }
    for (int e = tid; e < PANEL_ROWS * NB; e += blockDim.x)
    {
        const int rr = e % PANEL_ROWS, q = e / PANEL_ROWS;
        As[rr][q]    = (q < nb && r0 + rr < rend) ? A[(size_t)(k0 + q) * n + r0 + rr] : 0.;
    }
    __syncthreads();
    const int rr = tid % PANEL_ROWS;
    for (int c = tid / PANEL_ROWS; c < nb; c += blockDim.x / PANEL_ROWS)
    {
        double acc = 0.;
        for (int q = 0; q <= c; q++)
            acc += As[rr][q] * Ws[c][q];
        if (r0 + rr < rend) A[(size_t)(k0 + c) * n + r0 + rr] = acc;
    }
}

__global__ void copy_panel_kernel(const double* src, int lds, double* dst,
    int ldd, int m, int nb)
{
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < m * nb;
         e += gridDim.x * blockDim.x)
    {
        const int i = e % m, j = e / m;
        dst[(size_t)j * ldd + i] = src[(size_t)j * lds + i];
    }
}

static int copy_panel(const double* src, int lds, double* dst, int ldd, int m, int n, cudaStream_t s)
{
    copy_panel_kernel<<<std::min(1024, (m * n + 255) / 256), 256, 0, s>>>(src, lds, dst, ldd, m, n);
    MGX_LAUNCH_CHECK("copy_panel_kernel");
    return MGX_OK;
}

__global__ void zero_upper_kernel(double* A, int n)
{
    const size_t nn = (size_t)n * n;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < nn;
         t += (size_t)gridDim.x * blockDim.x)
    {
        const int i = (int)(t % n), j = (int)(t / n);
        if (i < j) A[t] = 0.;
    }
}

/* copies the NB x NB inverses of a block's diagonal (packed, leading
 * dimension NB) to the diagonal of W (leading dimension OB) */
__global__ void place_diag_kernel(const double* __restrict__ winv, double* __restrict__ W, int kb)
{
    const int k0 = blockIdx.x * NB, nb = min(NB, kb - k0);
    for (int e = threadIdx.x; e < nb * nb; e += blockDim.x)
    {
        const int i = e % nb, j = e / nb;
        W[(size_t)(k0 + j) * OB + k0 + i] = winv[(size_t)k0 * NB + (size_t)j * NB + i];
    }
}

/* workspace: diagonal inverses (nblocks x NB x NB), OB x OB inverses, a panel
 * (n x OB) and an n x n matrix */
struct DenseWs
{
    double *winv, *wob, *panel, *X;
    int* info;
};

static int dense_ws(mgx_ctx* ctx, int n, DenseWs* w)
{
    const size_t nbk = (n + NB - 1) / NB, nob = (n + OB - 1) / OB;
    const size_t b_w = nbk * NB * NB * 8, b_o = nob * OB * OB * 8, b_p = (size_t)n * OB * 8,
                 b_x = (size_t)n * n * 8;
    MGX_TRY(ctx->dense_ws.ensure(b_w + b_o + b_p + b_x + 256));
    char* base = (char*)ctx->dense_ws.ptr;
    w->winv    = (double*)base;
    w->wob     = (double*)(base + b_w);
    w->panel   = (double*)(base + b_w + b_o);
    w->X       = (double*)(base + b_w + b_o + b_p);
    w->info    = (int*)(base + b_w + b_o + b_p + b_x);
    return MGX_OK;
}

/* W (leading dimension ldw, lower) holds the inverses of L's diagonal blocks
 * of `step` rows; on return those of 2 step, for `batch` matrices of kb rows
 * at strides sL and sW: the block below the first inverse W1 of a pair is
 * -W2 (L21 W1), T a scratch of (step x step) per product at stride sT */
static int merge_inverses(mgx_ctx* ctx, int kb, int step, const double* L, int ldl, double* W,
    int ldw, double* T, int batch, size_t sL, size_t sW, size_t sT, cudaStream_t s)
{
    for (int o = 0; o + step < kb; o += 2 * step)
    {
        const int m = std::min(step, kb - o - step);
        Gemm g{ false, false, m, step, step, 1., L + (size_t)o * ldl + o + step, ldl,
            W + (size_t)o * ldw + o, ldw, 0., T, m };
        g.batch = batch;
        g.sA    = sL;
        g.sB    = sW;
        g.sC    = sT;
        MGX_TRY(gemm(ctx, g, s));
        Gemm h{ false, false, m, step, m, -1., W + (size_t)(o + step) * ldw + o + step, ldw, T, m,
            0., W + (size_t)o * ldw + o + step, ldw };
        h.batch = batch;
        h.sA    = sW;
        h.sB    = sT;
        h.sC    = sW;
        MGX_TRY(gemm(ctx, h, s));
    }
    return MGX_OK;
}

/* the OB x OB inverse of one diagonal block of kb rows from its NB x NB ones */
static int block_inverse(mgx_ctx* ctx, int kb, const double* L, int n, const double* winv,
    double* W, double* T, cudaStream_t s)
{
    MGX_TRY(cuda_check(cudaMemsetAsync(W, 0, sizeof(double) * OB * OB, s), "block inverse reset"));
    place_diag_kernel<<<(kb + NB - 1) / NB, 256, 0, s>>>(winv, W, kb);
    MGX_LAUNCH_CHECK("place_diag_kernel");
    for (int step = NB; step < kb; step *= 2)
        MGX_TRY(merge_inverses(ctx, kb, step, L, n, W, OB, T, 1, 0, 0, 0, s));
    return MGX_OK;
}

/* info_host set: synchronous, *info_host receives the pivot index; else
 * info_dev (device) receives it and nothing waits for the factorization.
 * Blocks of OB columns: their diagonal block by NB columns on the FP64 units,
 * then the panel below it, A W^T with the block's inverse W, and the trailing
 * update, both products of OB values that the tensor cores form from slices */
int cholesky(mgx_ctx* ctx, int n, double* A, int* info_host, cudaStream_t s,
    int* info_dev = nullptr)
{
    if (n <= 0 || !A || (!info_host && !info_dev))
        return fail(MGX_BAD_ARG, "cholesky: bad arguments");
    DenseWs w;
    MGX_TRY(dense_ws(ctx, n, &w));
    int* dinfo = info_dev ? info_dev : w.info;
    MGX_TRY(cuda_check(cudaMemsetAsync(dinfo, 0, sizeof(int), s), "info reset"));
    MGX_TRY(cuda_check(cudaFuncSetAttribute(potrf_diag_kernel,
                           cudaFuncAttributeMaxDynamicSharedMemorySize, DIAG_SMEM),
        "potrf smem attribute"));
    for (int o = 0; o < n; o += OB)
    {
        const int kb = std::min(OB, n - o), end = o + kb;
        for (int k0 = o; k0 < end; k0 += NB)
        {
            const int nb = std::min(NB, end - k0);
            double* wk   = w.winv + (size_t)k0 * NB;
            potrf_diag_kernel<<<1, 256, DIAG_SMEM, s>>>(A, n, k0, nb, wk, dinfo);
            MGX_LAUNCH_CHECK("potrf_diag_kernel");
            const int m = end - k0 - nb; // rows below, in this block
            if (m <= 0) continue;
            panel_trsm_kernel<<<(m + PANEL_ROWS - 1) / PANEL_ROWS, 256, 0, s>>>(A, n, k0, nb, end, wk);
            MGX_LAUNCH_CHECK("panel_trsm_kernel");
            const double* P = A + (size_t)k0 * n + k0 + nb;
            Gemm g{ false, true, m, m, nb, -1., P, n, P, n, 1.,
                A + (size_t)(k0 + nb) * n + k0 + nb, n };
            g.lower = 1;
            MGX_TRY(gemm(ctx, g, s));
        }
        const int m = n - end;
        if (m <= 0) continue;
        double* P = A + (size_t)o * n + end;
        double* W = w.wob;
        MGX_TRY(block_inverse(ctx, kb, A + (size_t)o * n + o, n, w.winv + (size_t)o * NB, W, w.X, s));
        MGX_TRY(gemm(ctx, Gemm{ false, true, m, kb, kb, 1., P, n, W, OB, 0., w.panel, m }, s));
        MGX_TRY(copy_panel(w.panel, m, P, n, m, kb, s));
        Gemm g{ false, true, m, m, kb, -1., P, n, P, n, 1., A + (size_t)end * n + end, n };
        g.lower = 1;
        MGX_TRY(gemm(ctx, g, s));
    }
    zero_upper_kernel<<<std::min<size_t>(((size_t)n * n + 255) / 256, 4096), 256, 0, s>>>(A, n);
    MGX_LAUNCH_CHECK("zero_upper_kernel");
    if (!info_host) return MGX_OK;
    int hinfo = 0;
    MGX_TRY(cuda_check(cudaMemcpyAsync(&hinfo, dinfo, sizeof(int), cudaMemcpyDeviceToHost, s),
        "info download"));
    MGX_TRY(cuda_check(cudaStreamSynchronize(s), "cholesky sync"));
    *info_host = hinfo;
    if (hinfo != 0) return fail(MGX_NOT_SPD, "Cholesky: leading minor %d not positive", hinfo);
    return MGX_OK;
}

/* inverses of the NB x NB diagonal blocks of a lower-triangular factor, one
 * CTA each, into the diagonal of X (leading dimension ldx; with stride > 0 the
 * blocks of each OB rows go to X + stride * (row / OB)).  Column by column on
 * all rows below, a lane per column (as potrf_diag_kernel does). */
__global__ void __launch_bounds__(256) trinv_diag_kernel(const double* L, int n,
    double* X, int ldx, size_t stride)
{
    extern __shared__ double dsm[];
    double(*T)[NB + 1] = reinterpret_cast<double(*)[NB + 1]>(dsm);
    double(*W)[NB + 1] = reinterpret_cast<double(*)[NB + 1]>(dsm + NB * (NB + 1));
    __shared__ double inv[NB];
    const int k0 = blockIdx.x * NB, nb = min(NB, n - k0);
    const int tid = threadIdx.x;
    for (int e = tid; e < nb * nb; e += blockDim.x)
    {
        const int i = e % nb, j = e / nb;
        T[i][j]     = (i >= j) ? L[(size_t)(k0 + j) * n + k0 + i] : 0.;
        W[i][j]     = i == j ? 1. : 0.;
    }
    __syncthreads();
    for (int i = tid; i < nb; i += blockDim.x)
        inv[i] = 1. / T[i][i];
    __syncthreads();
    const int warp = tid / 32, lane = tid & 31;
    const int half = warp >> 2, wr = warp & 3;
    const int c = 32 * half + lane;
    for (int j = 0; j < nb; j++)
    {
        // row j is final but for its factor; the rows below lose T(i, j) of it
        if (32 * half <= j && c < nb)
        {
            const double v = W[j][c] * inv[j];
            for (int i = j + 1 + wr; i < nb; i += 16)
            {
                double x[4], t[4];
#pragma unroll
                for (int q = 0; q < 4; q++)
                {
                    const int r = min(i + 4 * q, nb - 1);
                    x[q]        = W[r][c];
                    t[q]        = T[r][j];
                }
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (i + 4 * q < nb && c <= j) W[i + 4 * q][c] = x[q] - t[q] * v;
            }
        }
        __syncthreads();
    }
    double* out = X + (stride ? stride * (k0 / OB) : 0);
    const int q = stride ? k0 % OB : k0;
    for (int e = tid; e < nb * nb; e += blockDim.x)
    {
        const int i = e % nb, j = e / nb;
        out[(size_t)(q + j) * ldx + q + i] = i >= j ? W[i][j] * inv[i] : 0.;
    }
}

static int diag_inverses(int n, const double* L, double* X, int ldx, size_t stride, cudaStream_t s)
{
    MGX_TRY(cuda_check(cudaFuncSetAttribute(trinv_diag_kernel,
                           cudaFuncAttributeMaxDynamicSharedMemorySize, DIAG_SMEM),
        "trinv smem attribute"));
    trinv_diag_kernel<<<(n + NB - 1) / NB, 256, DIAG_SMEM, s>>>(L, n, X, ldx, stride);
    MGX_LAUNCH_CHECK("trinv_diag_kernel");
    return MGX_OK;
}

/* the inverses of L's OB x OB diagonal blocks into w.wob (leading dimension
 * OB), all full blocks in batches */
static int ob_inverses(mgx_ctx* ctx, int n, const double* L, const DenseWs& w, cudaStream_t s)
{
    const size_t so = (size_t)OB * OB;
    const int full = n / OB, rest = n - full * OB, nob = full + (rest ? 1 : 0);
    MGX_TRY(cuda_check(cudaMemsetAsync(w.wob, 0, nob * so * sizeof(double), s), "inverses reset"));
    MGX_TRY(diag_inverses(n, L, w.wob, OB, so, s));
    for (int step = NB; step < OB; step *= 2)
    {
        if (full)
            MGX_TRY(merge_inverses(ctx, OB, step, L, n, w.wob, OB, w.panel, full,
                (size_t)OB * n + OB, so, (size_t)step * step, s));
        if (step < rest)
            MGX_TRY(merge_inverses(ctx, rest, step, L + (size_t)full * OB * (n + 1), n,
                w.wob + full * so, OB, w.panel, 1, 0, 0, 0, s));
    }
    return MGX_OK;
}

// upper triangle <- lower triangle (of src, into dst; they may be the same)
__global__ void mirror_lower_kernel(const double* src, double* dst, int n)
{
    const size_t nn = (size_t)n * n;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < nn;
         t += (size_t)gridDim.x * blockDim.x)
    {
        const size_t i = t % n, j = t / n;
        if (i < j)
            dst[t] = src[i * n + j];
        else if (src != dst)
            dst[t] = src[t];
    }
}

static int mirror_lower(const double* src, double* dst, int n, cudaStream_t s)
{
    const int nb = (int)std::min<size_t>(((size_t)n * n + 255) / 256, 4096);
    mirror_lower_kernel<<<nb, 256, 0, s>>>(src, dst, n);
    MGX_LAUNCH_CHECK("mirror_lower_kernel");
    return MGX_OK;
}

/* S M for a symmetric S of which the lower triangle is read (BLAS symm 'l',
 * 'l') */
static int symm(mgx_ctx* ctx, int n, const double* S, const double* M, double* out, cudaStream_t s)
{
    DenseWs w;
    MGX_TRY(dense_ws(ctx, n, &w));
    MGX_TRY(mirror_lower(S, w.X, n, s));
    // S = S^T: read along the columns, the values of k
    return gemm(ctx, Gemm{ true, false, n, n, n, 1., w.X, n, M, n, 0., out, n }, s);
}

/* ProjectedMatrices::updateTheta (src/ProjectedMatrices.h:218-225):
 * theta = Sinv H with Sinv symmetric, read from its lower triangle. */
int theta_product(mgx_ctx* ctx, int n, const double* Sinv, const double* H, double* theta,
    cudaStream_t s)
{
    if (n <= 0 || !Sinv || !H || !theta) return fail(MGX_BAD_ARG, "theta: bad arguments");
    return symm(ctx, n, Sinv, H, theta, s);
}

/* Sinv = (L L^T)^-1 = X^T X with X = L^-1, whose diagonal blocks are inverted
 * and merged in pairs until one is left. */
int inverse_from_cholesky(mgx_ctx* ctx, int n, const double* L, double* Sinv,
    cudaStream_t s)
{
    if (n <= 0 || !L || !Sinv) return fail(MGX_BAD_ARG, "inverse: bad arguments");
    if (Sinv == L) return fail(MGX_BAD_ARG, "inverse: Sinv aliases L");
    DenseWs w;
    MGX_TRY(dense_ws(ctx, n, &w));
    MGX_TRY(cuda_check(cudaMemsetAsync(w.X, 0, (size_t)n * n * 8, s), "inverse reset"));
    MGX_TRY(diag_inverses(n, L, w.X, n, 0, s));
    for (int step = NB; step < n; step *= 2)
    {
        // the full pairs of small blocks in one batch each
        const int pairs = step < OB ? n / (2 * step) : 0, done = pairs * 2 * step;
        if (pairs)
            MGX_TRY(merge_inverses(ctx, 2 * step, step, L, n, w.X, n, Sinv, pairs,
                (size_t)2 * step * (n + 1), (size_t)2 * step * (n + 1), (size_t)step * step, s));
        MGX_TRY(merge_inverses(ctx, n - done, step, L + (size_t)done * (n + 1), n,
            w.X + (size_t)done * (n + 1), n, Sinv, 1, 0, 0, 0, s));
    }
    // the lower triangle of S^-1 = X^T X, mirrored
    Gemm g{ true, false, n, n, n, 1., w.X, n, w.X, n, 0., Sinv, n };
    g.lower = 1;
    MGX_TRY(gemm(ctx, g, s));
    return mirror_lower(Sinv, Sinv, n, s);
}

/* theta = S^-1 H = L^-T (L^-1 H) from the Cholesky factor L, without
 * forming S^-1: blocked forward substitution L Y = H and back substitution
 * L^T theta = Y with the n columns of H as right-hand sides.  The OB x OB
 * diagonal blocks are applied through their inverses; the off-diagonal
 * updates are (n - k) x n x OB products, from slices on the tensor cores.
 * 2 n^3 flop instead of the n^3 / 3 + 2 n^3 + 2 n^3 of
 * computeInverse followed by updateTheta (src/GramMatrix.cc:75-91,
 * src/ProjectedMatrices.h:218-225).  trace (device, may be NULL) receives
 * tr(theta) = tr(S^-1 H). */
__global__ void diag_sum_kernel(const double* __restrict__ A, int n, double* __restrict__ out)
{
    __shared__ double red[256];
    double acc = 0.;
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        acc += A[(size_t)i * n + i];
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1)
    {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = red[0];
}

int theta_from_cholesky(mgx_ctx* ctx, int n, const double* L, const double* H,
    double* theta, double* trace, cudaStream_t s)
{
    if (n <= 0 || !L || !H || !theta) return fail(MGX_BAD_ARG, "theta: bad arguments");
    if (theta == H || theta == L) return fail(MGX_BAD_ARG, "theta aliases an input");
    DenseWs w;
    MGX_TRY(dense_ws(ctx, n, &w));
    MGX_TRY(ob_inverses(ctx, n, L, w, s));
    MGX_TRY(cuda_check(cudaMemcpyAsync(theta, H, (size_t)n * n * 8, cudaMemcpyDeviceToDevice, s),
        "theta init"));
    // rows o .. o + kb of theta <- W^(T) times them, through the panel
    auto apply_diag = [&](int o, int kb, bool transpose) -> int {
        MGX_TRY(gemm(ctx, Gemm{ transpose, false, kb, n, kb, 1., w.wob + (size_t)(o / OB) * OB * OB,
                              OB, theta + o, n, 0., w.panel, kb }, s));
        return copy_panel(w.panel, kb, theta + o, n, kb, n, s);
    };
    const int nob = (n + OB - 1) / OB;
    // forward: L Y = H
    for (int b = 0; b < nob; b++)
    {
        const int o = b * OB, kb = std::min(OB, n - o), m = n - o - kb;
        MGX_TRY(apply_diag(o, kb, false));
        if (m > 0)
            MGX_TRY(gemm(ctx, Gemm{ false, false, m, n, kb, -1., L + (size_t)o * n + o + kb, n,
                                  theta + o, n, 1., theta + o + kb, n }, s));
    }
    // backward: L^T theta = Y
    for (int b = nob - 1; b >= 0; b--)
    {
        const int o = b * OB, kb = std::min(OB, n - o);
        MGX_TRY(apply_diag(o, kb, true));
        if (o > 0)
            MGX_TRY(gemm(ctx, Gemm{ true, false, o, n, kb, -1., L + o, n, theta + o, n, 1., theta, n },
                s));
    }
    if (trace)
    {
        diag_sum_kernel<<<1, 256, 0, s>>>(theta, n, trace);
        MGX_LAUNCH_CHECK("diag_sum_kernel");
    }
    return MGX_OK;
}

/* tr(H Sinv) with both matrices symmetric and read from their lower
 * triangles: sum_k [H(k,k) S(k,k) + 2 sum_{i>k} H(i,k) S(i,k)], columns
 * spread over the blocks (coalesced column reads), one partial per block,
 * then a fixed-order sum of the partials. */
constexpr int TRACE_BLOCKS = 256;

__global__ void __launch_bounds__(256) trace_partial_kernel(const double* __restrict__ H,
    const double* __restrict__ Sinv, int n, double* __restrict__ part)
{
    __shared__ double red[256];
    double acc = 0.;
    for (int k = blockIdx.x; k < n; k += gridDim.x)
    {
        const double* h = H + (size_t)k * n;
        const double* q = Sinv + (size_t)k * n;
        for (int i = k + threadIdx.x; i < n; i += blockDim.x)
            acc += (i == k ? 1. : 2.) * h[i] * q[i];
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1)
    {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

__global__ void __launch_bounds__(256) trace_sum_kernel(const double* __restrict__ part, int n,
    double* __restrict__ out)
{
    __shared__ double red[256];
    double acc = 0.;
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        acc += part[i];
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1)
    {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = red[0];
}

int trace_prod(mgx_ctx* ctx, int n, const double* H, const double* Sinv, double* out,
    cudaStream_t s)
{
    if (n <= 0 || !H || !Sinv || !out) return fail(MGX_BAD_ARG, "trace: bad arguments");
    MGX_TRY(ctx->red.ensure(TRACE_BLOCKS * sizeof(double)));
    double* part = (double*)ctx->red.ptr;
    trace_partial_kernel<<<TRACE_BLOCKS, 256, 0, s>>>(H, Sinv, n, part);
    MGX_LAUNCH_CHECK("trace_partial_kernel");
    trace_sum_kernel<<<1, 256, 0, s>>>(part, TRACE_BLOCKS, out);
    MGX_LAUNCH_CHECK("trace_sum_kernel");
    return MGX_OK;
}

/* ProjectedMatricesMehrstellen::updateHB
 * (src/ProjectedMatricesMehrstellen.h:55-62): HB = S theta with S read as
 * symmetric from its lower triangle (symm 'l', 'l'), then
 * HB = 0.5 HB + 0.5 HB^T (the transpose(0.5, copy, 0.5) of the reference);
 * element (i, j) and (j, i) receive the same sum 0.5 a_ij + 0.5 a_ji. */
__global__ void sym_average_kernel(double* A, int n)
{
    const size_t nn = (size_t)n * n;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < nn;
         t += (size_t)gridDim.x * blockDim.x)
    {
        const int i = (int)(t % n), j = (int)(t / n);
        if (i <= j) continue;
        const double x = 0.5 * A[(size_t)j * n + i] + 0.5 * A[(size_t)i * n + j];
        A[(size_t)j * n + i] = x;
        A[(size_t)i * n + j] = x;
    }
}

int update_hb(mgx_ctx* ctx, int n, const double* S, const double* theta, double* HB, cudaStream_t s)
{
    if (n <= 0 || !S || !theta || !HB) return fail(MGX_BAD_ARG, "updateHB: bad arguments");
    if (HB == S || HB == theta) return fail(MGX_BAD_ARG, "HB aliases an input");
    MGX_TRY(symm(ctx, n, S, theta, HB, s));
    const int nb = (int)std::min<size_t>(((size_t)n * n + 255) / 256, 4096);
    sym_average_kernel<<<nb, 256, 0, s>>>(HB, n);
    MGX_LAUNCH_CHECK("sym_average_kernel");
    return MGX_OK;
}

/* LocGridOrbitals::normalize (src/LocGridOrbitals.cc:2230-2311, the branch
 * without short-sighted matrices): diagS_i = vel * psi_i . psi_i with FP64
 * accumulation (BlockVector::dot -> MPdot, src/linear_algebra/mputils.cc:
 * 145-166), then psi_i <- (T)(diagS_i^-1/2 * (double)psi_i) (MPscal,
 * mputils.cc:61-80).  The dot products are deterministic: NORM_BLOCKS
 * partial sums per function, then a fixed-order sum. */
constexpr int NORM_BLOCKS = 64;

template <typename T>
__global__ void __launch_bounds__(256) sumsq_partial_kernel(const T* __restrict__ psi,
    size_t ld, size_t npts, double* __restrict__ part)
{
    __shared__ double red[256];
    const int f    = blockIdx.y;
    const T* p     = psi + (size_t)f * ld;
    double acc     = 0.;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < npts;
         i += (size_t)gridDim.x * blockDim.x)
    {
        const double v = (double)p[i];
        acc += v * v;
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1)
    {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[(size_t)f * gridDim.x + blockIdx.x] = red[0];
}

// one thread per function: diagS = vel * sum of the partials; alpha =
// 1 / sqrt(diagS); a diagS <= 1e-15 (the reference asserts) raises *bad
__global__ void norm_finish_kernel(const double* __restrict__ part, int nblk, int nfunc,
    double vel, double* __restrict__ diag, double* __restrict__ alpha, int* bad)
{
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nfunc) return;
    double acc = 0.;
    for (int b = 0; b < nblk; b++)
        acc += part[(size_t)f * nblk + b];
    const double d = vel * acc;
    if (diag) diag[f] = d;
    if (!(d > 1.e-15))
    {
        atomicExch(bad, 1);
        alpha[f] = 1.;
    }
    else
        alpha[f] = 1. / sqrt(d);
}

// psi_f <- (T)(alpha_f * (double)psi_f), skipped entirely when *bad is set
template <typename T>
__global__ void __launch_bounds__(256) scale_columns_kernel(T* __restrict__ psi, size_t ld,
    size_t npts, const double* __restrict__ alpha, const int* __restrict__ bad)
{
    if (bad && *bad) return;
    const int f    = blockIdx.y;
    const double a = alpha[f];
    T* p           = psi + (size_t)f * ld;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < npts;
         i += (size_t)gridDim.x * blockDim.x)
        p[i] = (T)(a * (double)p[i]);
}

int normalize(mgx_ctx* ctx, int dtype, void* psi, size_t ld, size_t npts, int nfunc,
    double vel, double* diag, cudaStream_t s)
{
    if (nfunc <= 0) return MGX_OK;
    if (nfunc > 65535) return fail(MGX_UNSUPPORTED, "normalize: more than 65535 functions");
    const size_t part_bytes = (size_t)nfunc * NORM_BLOCKS * sizeof(double);
    MGX_TRY(ctx->red.ensure(part_bytes + (size_t)nfunc * sizeof(double) + 256));
    double* part  = (double*)ctx->red.ptr;
    double* alpha = part + (size_t)nfunc * NORM_BLOCKS;
    int* bad      = (int*)(alpha + nfunc);
    MGX_TRY(cuda_check(cudaMemsetAsync(bad, 0, sizeof(int), s), "normalize flag"));
    dim3 grid(NORM_BLOCKS, nfunc);
    if (dtype == MGX_F64)
        sumsq_partial_kernel<double><<<grid, 256, 0, s>>>((const double*)psi, ld, npts, part);
    else
        sumsq_partial_kernel<float><<<grid, 256, 0, s>>>((const float*)psi, ld, npts, part);
    MGX_LAUNCH_CHECK("sumsq_partial_kernel");
    norm_finish_kernel<<<(nfunc + 127) / 128, 128, 0, s>>>(part, NORM_BLOCKS, nfunc, vel, diag,
        alpha, bad);
    MGX_LAUNCH_CHECK("norm_finish_kernel");
    const int sblk = (int)std::min<size_t>((npts + 255) / 256, 256);
    dim3 sgrid(sblk, nfunc);
    if (dtype == MGX_F64)
        scale_columns_kernel<double><<<sgrid, 256, 0, s>>>((double*)psi, ld, npts, alpha, bad);
    else
        scale_columns_kernel<float><<<sgrid, 256, 0, s>>>((float*)psi, ld, npts, alpha, bad);
    MGX_LAUNCH_CHECK("scale_columns_kernel");
    int hbad = 0;
    MGX_TRY(cuda_check(cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, s),
        "normalize flag read"));
    MGX_TRY(cuda_check(cudaStreamSynchronize(s), "normalize sync"));
    if (hbad) return fail(MGX_NOT_SPD, "normalize: a function with vel * |psi|^2 <= 1e-15");
    return MGX_OK;
}

/* d_i = 1 / sqrt(S(i, i)): the normalization factors of the functions
 * whose Gram matrix is S (LocGridOrbitals::normalize takes the same
 * diagonal from its own dot products) */
__global__ void diag_rsqrt_kernel(const double* __restrict__ S, int n, double* __restrict__ d)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) d[i] = 1. / sqrt(S[(size_t)i * n + i]);
}

int diag_rsqrt(mgx_ctx*, int n, const double* S, double* d, cudaStream_t s)
{
    if (n <= 0 || !S || !d) return fail(MGX_BAD_ARG, "diag_rsqrt: bad arguments");
    diag_rsqrt_kernel<<<(n + 255) / 256, 256, 0, s>>>(S, n, d);
    MGX_LAUNCH_CHECK("diag_rsqrt_kernel");
    return MGX_OK;
}

} // namespace mgx
