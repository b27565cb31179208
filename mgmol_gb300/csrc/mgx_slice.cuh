// FP64 products on the tensor cores from bf16 slices (mgx_slice.cu).
#pragma once

#include "mgx_internal.cuh"

namespace mgx
{
namespace sl
{
/* An FP64 operand of a product C = A B^T: `rows` rows of K values, element
 * (r, k) at x[r * ld + k] (kmajor) or x[k * ld + r]. */
struct View
{
    const double* x;
    size_t ld;
    size_t rows;
    size_t K;
    bool kmajor;
};

/* What becomes of the product P = A B^T (m x n):
 *   sum given: P(i, j) is added to an integer in units of 2^-SUM_W of a digit
 *     product, sum[j * m + i] 2^32 + sum[(n + j) * m + i], both signed; K is
 *     split over CTAs that add atomically, and the order does not matter
 *   else: C[j * ldc + i] = alpha P(i, j) + beta cin[j * ldcin + i]
 * lower: only entries i >= j + col0 (the others are left as they are). */
struct Target
{
    double* C;
    size_t ldc;
    unsigned long long* sum;
    double alpha;
    double beta;
    const double* cin;
    size_t ldcin;
    int lower;
    int col0;
};

/* digits per value: of the sums over grid points, and of the other products */
constexpr int NS_SUM = 7, NS_STORE = 8;

/* bytes of the ns planes of `rows` rows of K values */
size_t plane_bytes(size_t rows, size_t K, int ns);

/* resets the keys of the view's rows and takes the row maxima into them; *bad
 * is set by a NaN or an infinity (and never reset here) */
int row_keys(const View& v, int* keys, int* bad, cudaStream_t s);
/* planes of columns [k0, k0 + kc) of the view */
int make_planes(const View& v, size_t k0, size_t kc, const int* keys, void* planes, int ns,
    cudaStream_t s);
/* the product of two sets of planes (NS_SUM with Target::sum, else NS_STORE) of
 * kc values of K; does nothing when *bad is set, and sets it when a bounded wait
 * gives up: to 1, or to LOST where Target::cin == C with beta != 0, an operand
 * that is overwritten in part by then */
constexpr int LOST = 2;
int product(int sms, size_t m, const void* pa, const int* ka, size_t n, const void* pb,
    const int* kb, size_t kc, const Target& t, int* bad, cudaStream_t s);

/* whether a product of this size is formed from slices: from 2^24
 * multiply-adds on, where the context allows it */
bool pays(const mgx_ctx* ctx, size_t m, size_t n, size_t K);

/* One product with a shared left operand: C(i, j) += sum_k A(i, k) B(j, k),
 * j < ncols, C of leading dimension n; with lower, entries i >= j + col0. */
struct Factor
{
    const double* B;
    int ncols;
    int lower;
    int col0;
    double* C;
};

/* The products of K-contiguous blocks of leading dimension ld (n rows of A),
 * in chunks of K that bound the planes to PLANE_CAP bytes, or less where there
 * is no memory for them; the planes of A serve all of them.  *bad (device) tells whether an operand was not finite
 * and nothing was added.  MGX_NO_MEMORY: no workspace, or K too large for the integers; nothing was added. */
constexpr size_t PLANE_CAP = size_t(1) << 30, PLANE_CAP_LEAST = size_t(1) << 24;
int accumulate(mgx_ctx* ctx, const double* A, size_t ld, size_t K, int n, const Factor* f, int nf,
    int** bad, cudaStream_t s);

/* C = alpha A B^T + beta cin of FP64 operands of any layout, the rows of A
 * in chunks that bound the planes as above.  After each chunk
 * fallback(r0, rows, bad) enqueues the CUDA-core kernel of these rows, which
 * does nothing unless *bad is set, and for LOST writes NaN.  MGX_NO_MEMORY: no
 * workspace, nothing was written. */
template <typename F>
int store(mgx_ctx* ctx, const View& A, const View& B, const Target& t, cudaStream_t s, F fallback);

/* the parts of store() */
struct StorePlan
{
    size_t chunk;
    int *ka, *kb, *bad;
    char *pa, *pb;
};
int store_begin(mgx_ctx* ctx, const View& A, const View& B, StorePlan* plan, cudaStream_t s);
int store_chunk(mgx_ctx* ctx, const View& A, const View& B, const Target& t, const StorePlan& plan,
    size_t r0, size_t rows, cudaStream_t s);

template <typename F>
int store(mgx_ctx* ctx, const View& A, const View& B, const Target& t, cudaStream_t s, F fallback)
{
    StorePlan p;
    MGX_TRY(store_begin(ctx, A, B, &p, s));
    for (size_t r0 = 0; r0 < A.rows; r0 += p.chunk)
    {
        const size_t rows = p.chunk < A.rows - r0 ? p.chunk : A.rows - r0;
        MGX_TRY(store_chunk(ctx, A, B, t, p, r0, rows, s));
        MGX_TRY(fallback(r0, rows, (const int*)p.bad));
    }
    return MGX_OK;
}
} // namespace sl
} // namespace mgx
