// FP64 products C = A B^T on the tcgen05 tensor cores of sm_103a, from exact
// slices of the operands (the scheme of Ozaki, Ogita, Oishi and Rump,
// "Error-free transformations of matrix multiplication", 2012).
//
// GB300 runs two FP64 multiply-adds per SM and clock, 1.18 TFLOP/s, and
// 1.87 PFLOP/s of bf16 on the tensor cores.  So a product of FP64 operands is
// formed from bf16 products whose sums are exact:
//   - every row r of an operand is scaled by 2^-e_r, |x| < 2^e_r, and written
//     as a 56-bit fixed-point number of seven balanced base-256 digits,
//     x 2^(7 - e_r) = d_0 + d_1 2^-8 + ... + d_6 2^-48, |d| <= 128, each digit
//     (with its power of 256) one bf16 value.  Seven digits serve the sums
//     over grid points; the products of N x N matrices and Psi Theta, where one
//     entry of a row may be far larger than the rest, take an eighth (with
//     seven S theta and the residual were off 5 to 10 times as far as with FP64
//     multiply-adds, with eight no further);
//   - digit s of A times digit t of B are integers of at most 2^14 at weight
//     2^(-8 (s + t)).  The products of one s + t add up in an FP32 accumulator
//     of their own, which rounds nothing while |sum| <= 2^24: after 192 values
//     of K (256 where only s + t <= 3 are summed) it is read and added to a
//     64-bit integer.  (All of s + t <= 4 are
//     exact for any input; of the 6 or 7 x 192 products of s + t = 5 and 6, at
//     2^-40 and 2^-48, the last bit could round if all digits were extreme.)
//     The sums have to be exact and not only FP32: the tensor cores truncate
//     when they add, which biases a sum of squares by 2^-24 per addition;
//   - products of s + t > 6 (7), 2^-56 (2^-64) of |row scale| |column scale|
//     and less, are left out.
// 28 (36) bf16 products stand for one FP64 product.  An entry is off by about
// 2^-54 sqrt(K) (2^-60 sqrt(K)) of row maximum x column maximum: the digits left
// out are six (seven) products of 0.33 2^14 rms, and a row scale is up to twice (four
// times) its maximum.  Against the norms of the rows that is what FP64
// multiply-adds give or less, as long as a row's values of some size are not a
// few of its K; against sum |a b|, which FP64 multiply-adds are relative to, it is not:
// entries far below the norms lose digits, and for them the context can turn the
// slices off.
//
// A NaN or an infinity in an operand has no digits: it raises a flag, on
// which the kernels here do nothing and the caller's CUDA-core kernel,
// launched behind them, does the work instead of returning at once.  A bounded
// wait that gives up raises the same flag, or, when the product is added to its
// own target and cannot be formed again, the flag that fills the target with NaN.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <type_traits>
#include <vector>

#include "mgx_slice.cuh"
#include "mgx_tcgen05.cuh"

namespace mgx
{
namespace sl
{
constexpr int BM      = 128; // rows of a tile (A)
constexpr int BN      = 128; // most columns of a tile (B)
constexpr int BN1     = 64;  // most columns with all NS accumulators in TMEM at once
constexpr int BK      = 32;  // K values of a stage (64 bytes, SWIZZLE_64B)
constexpr int STAGES  = 2;
constexpr int DRAIN   = 6;   // stages between reads of the accumulators
constexpr int DRAIN2  = 8;   // the same for the walk of s + t = 0 .. 3 alone
constexpr int A_SLICE = BM * BK * 2;
constexpr int EPI     = 16;  // epilogue warps: four per scheduler hide the TMEM reads
constexpr int SUM_W   = 48;  // sums over items are kept in units of 2^-SUM_W
// the most values of K of a sum and of a stored product: a digit product is at
// most 2^14 and five of them share s + t = 4, so that the lower words of a sum
// reach 5.1 K 2^30, and L of a stored product 5.1 K 2^38
constexpr size_t MAX_K_SUM = size_t(1) << 30, MAX_K_STORE = size_t(1) << 22;
constexpr int THREADS = 32 * (2 + EPI);

/* the kernel's two forms: NP 1, all s + t in one walk over K, at most 64
 * columns; NP 2, two walks, at most 128 */
template <int NP, int NS>
struct Form
{
    static constexpr int W       = NP == 1 ? BN1 : BN;
    static constexpr int B_SLICE = W * BK * 2;
    static constexpr int STAGE   = NS * (A_SLICE + B_SLICE);
    static constexpr size_t SMEM
        = (size_t)STAGES * STAGE + (2 * STAGES + 1 + NS) * 8 + 16 + 1024;
    static_assert(SMEM <= 227 * 1024, "two stages fit one SM");
    static_assert((NP == 1 ? NS : 4) * W <= 512, "the accumulators of a walk fit TMEM");
};

/* The key of a row: the upper half of the bits of max |x|.  Exponent e with
 * |x| < 2^e for every x of the row (one more with eight digits, whose first
 * then fits the upper byte of 64 bits). */
template <int NS>
__device__ __forceinline__ int key_exponent(int key)
{
    return max(key >> 20, 1) - 1022 + (NS == 8);
}

constexpr int KEY_NONFINITE = 0x7ff00000;

__device__ __forceinline__ int abs_hi(double x) { return __double2hiint(x) & 0x7fffffff; }

/* row maxima, K contiguous: blockIdx.y = row (grid-stride), blockIdx.x = a
 * part of K */
__global__ void __launch_bounds__(256) keys_kmajor_kernel(const double* __restrict__ x, size_t ld,
    size_t rows, size_t K, int* __restrict__ keys, int* __restrict__ bad)
{
    const size_t part = ((K + gridDim.x - 1) / gridDim.x + 255) & ~size_t(255);
    const size_t k0 = blockIdx.x * part, k1 = min(K, k0 + part);
    for (size_t r = blockIdx.y; r < rows; r += gridDim.y)
    {
        int m             = 0;
        const double* row = x + r * ld;
        size_t k          = k0 + threadIdx.x;
        for (; k + 3 * 256 < k1; k += 4 * 256)
        {
            const double a = row[k], b = row[k + 256], c = row[k + 512], d = row[k + 768];
            m = max(m, max(max(abs_hi(a), abs_hi(b)), max(abs_hi(c), abs_hi(d))));
        }
        for (; k < k1; k += 256)
            m = max(m, abs_hi(row[k]));
        m = __reduce_max_sync(0xffffffffu, m);
        if ((threadIdx.x & 31) == 0 && m > 0)
        {
            atomicMax(keys + r, m);
            if (m >= KEY_NONFINITE) *bad = 1;
        }
    }
}

/* row maxima, rows contiguous: a thread owns a row, blockIdx.y a part of K */
__global__ void __launch_bounds__(128) keys_rmajor_kernel(const double* __restrict__ x, size_t ld,
    size_t rows, size_t K, int* __restrict__ keys, int* __restrict__ bad)
{
    const size_t part = (K + gridDim.y - 1) / gridDim.y;
    const size_t k0 = blockIdx.y * part, k1 = min(K, k0 + part);
    for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < rows;
         r += (size_t)gridDim.x * blockDim.x)
    {
        int m = 0;
#pragma unroll 8
        for (size_t k = k0; k < k1; k++)
            m = max(m, abs_hi(x[k * ld + r]));
        if (m > 0)
        {
            atomicMax(keys + r, m);
            if (m >= KEY_NONFINITE) *bad = 1;
        }
    }
}

/* x 2^(8 NS - 1 - e) rounded to an integer (half away from zero), |x| < 2^e, in
 * integer arithmetic: the FP64 units are the scarce ones here */
template <int NS>
__device__ __forceinline__ long long to_fixed(double x, int e)
{
    const long long b = __double_as_longlong(x);
    const int ex      = (int)(b >> 52) & 0x7ff;
    long long m       = b & 0xfffffffffffffll;
    if (ex) m |= 0x10000000000000ll;
    // |x| = m 2^(max(ex, 1) - 1075)
    const int sh = min(e + 1076 - 8 * NS - max(ex, 1), 62);
    m            = sh <= 0 ? m << (-sh) : (m + (1ll << (sh - 1))) >> sh;
    return b < 0 ? -m : m;
}

/* the NS digits of q, most significant first, each times 2^(-8 s), as the
 * upper halves of FP32 values (exact in bf16) */
template <int NS>
__device__ __forceinline__ void digits(long long q, uint32_t (&f)[NS])
{
    // with 128 added at the place of every digit but the first, the bytes of
    // q are the balanced digits plus 128
    const long long b = q + (NS == 8 ? 0x0080808080808080ll : 0x0000808080808080ll);
    const uint32_t lo = (uint32_t)b, hi = (uint32_t)((unsigned long long)b >> 32);
    f[0] = __float_as_uint((float)((int)hi >> (NS == 8 ? 24 : 16)));
#pragma unroll
    for (int s = 1; s < NS; s++)
    {
        const int by         = NS - 1 - s; // byte of b
        const uint32_t byte  = ((by >= 4 ? hi : lo) >> (8 * (by & 3))) & 0xffu;
        const uint32_t magic = (uint32_t)(150 - 8 * s) << 23; // 2^(23 - 8 s)
        // (2^(23 - 8 s) + byte 2^(-8 s)) - (2^(23 - 8 s) + 128 2^(-8 s))
        f[s] = __float_as_uint(
            __uint_as_float(magic | byte) - __uint_as_float(magic | 128u));
    }
}

/* stores the digits of 8 consecutive K values: 16 bytes in each plane.  The
 * planes are K-blocked: element (row, k) of slice s at
 * ((s * kblocks + k / 64) * rows + row) * 64 + k % 64. */
template <int NS>
__device__ __forceinline__ void store8(const long long (&q)[8], __nv_bfloat16* planes, size_t rows,
    size_t kblocks, size_t kb, size_t r, int g)
{
    uint32_t w[NS][4];
#pragma unroll
    for (int p = 0; p < 4; p++)
    {
        uint32_t a[NS], b[NS];
        digits<NS>(q[2 * p], a);
        digits<NS>(q[2 * p + 1], b);
#pragma unroll
        for (int s = 0; s < NS; s++)
            w[s][p] = __byte_perm(a[s], b[s], 0x7632);
    }
#pragma unroll
    for (int s = 0; s < NS; s++)
        *reinterpret_cast<uint4*>(planes + ((s * kblocks + kb) * rows + r) * 64 + g)
            = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
}

/* planes of a K-contiguous operand, 8 values of K per thread; HBM bound (8
 * bytes read, 14 written per value) */
template <int NS>
__global__ void __launch_bounds__(256) planes_kmajor_kernel(const double* __restrict__ x, size_t ld,
    size_t rows, size_t K, const int* __restrict__ keys, size_t kblocks,
    __nv_bfloat16* __restrict__ planes)
{
    const size_t total = rows * kblocks * 8;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (size_t)gridDim.x * blockDim.x)
    {
        const int g     = 8 * (int)(t % 8);
        const size_t rk = t / 8;
        const size_t kb = rk % kblocks, r = rk / kblocks;
        const size_t k  = kb * 64 + g;
        const int e     = key_exponent<NS>(keys[r]);
        const double* p = x + r * ld + k;
        long long q[8];
#pragma unroll
        for (int i = 0; i < 8; i++)
            q[i] = (k + i < K) ? to_fixed<NS>(p[i], e) : 0;
        store8<NS>(q, planes, rows, kblocks, kb, r, g);
    }
}

/* planes of a row-contiguous operand: a block takes 64 rows x 64 values of K
 * through shared memory (73 values between rows: conflict-free stores along
 * rows, two-way reads of the values k = 8 q + g in the order that puts g
 * next to each other) */
constexpr int TP = 73;

template <int NS>
__global__ void __launch_bounds__(256) planes_rmajor_kernel(const double* __restrict__ x, size_t ld,
    size_t rows, size_t K, const int* __restrict__ keys, size_t kblocks,
    __nv_bfloat16* __restrict__ planes)
{
    __shared__ long long t[64 * TP];
    const size_t r0 = (size_t)blockIdx.x * 64, kb = blockIdx.y;
    const int rr    = threadIdx.x % 64;
    const size_t r  = r0 + rr;
    const int e     = r < rows ? key_exponent<NS>(keys[r]) : 0;
#pragma unroll 4
    for (int kk = threadIdx.x / 64; kk < 64; kk += 4)
    {
        const size_t k = kb * 64 + kk;
        // value k = 8 a + b of the block at place 8 b + a
        t[rr * TP + (kk % 8) * 8 + kk / 8]
            = (r < rows && k < K) ? to_fixed<NS>(x[k * ld + r], e) : 0;
    }
    __syncthreads();
    for (int it = threadIdx.x; it < 64 * 8; it += 256)
    {
        const int a = it % 8, row = it / 8;
        if (r0 + row >= rows) continue;
        long long q[8];
#pragma unroll
        for (int b = 0; b < 8; b++)
            q[b] = t[row * TP + 8 * b + a];
        store8<NS>(q, planes, rows, kblocks, kb, r0 + row, 8 * a);
    }
}

struct Params
{
    int nti, ntj;    // tiles
    int bn;          // columns of a tile, a multiple of 32
    int ntiles;      // tiles formed (with lower: those that reach i >= j + col0)
    int nst;         // stages of K
    int st_per_item; // stages of one item
    int nitems;
    int kblocks;     // 64-value blocks of K in each plane
    size_t m, n;
    const int* ka;
    const int* kb;
    Target t;
    int* bad;
    uint32_t polls; // after which a wait gives up
};

/* the first row tile that reaches an entry i >= c */
__host__ __device__ inline int first_tile(int c, int nti)
{
    const int f = c > 0 ? c / BM : 0;
    return f < nti ? f : nti;
}

/* item w: its tile and stages.  The tiles of one K range sit side by side in
 * the list, so that CTAs that run together read the same planes. */
__device__ __forceinline__ void decode(const Params& p, int w, int& ti, int& tj, int& st0, int& nst)
{
    int tile = w % p.ntiles;
    st0      = (w / p.ntiles) * p.st_per_item;
    nst      = min(p.nst - st0, p.st_per_item);
    if (!p.t.lower)
    {
        ti = tile % p.nti;
        tj = tile / p.nti;
        return;
    }
    for (tj = 0; tj < p.ntj; tj++)
    {
        const int first = first_tile(p.t.col0 + tj * p.bn, p.nti);
        if (tile < p.nti - first)
        {
            ti = first + tile;
            return;
        }
        tile -= p.nti - first;
    }
    ti = 0; // not reached
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]),
                 "=f"(v[6]), "=f"(v[7])
                 : "r"(taddr));
}

/* waits for the loads in flight; the values of v are used only behind it */
__device__ __forceinline__ void tmem_wait_ld(float (&v)[8])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]),
                 "+f"(v[6]), "+f"(v[7])
                 :
                 : "memory");
}

/* V 2^E rounded to FP64, in integer arithmetic (a conversion would take the
 * FP64 unit, which the conversions of a tile of few values of K kept busy four
 * times as long as its MMAs ran); scalbn where the result is not normal */
__device__ __forceinline__ double scaled(__int128 V, int E)
{
    if (V == 0) return 0.;
    const bool neg               = V < 0;
    const unsigned __int128 a    = neg ? (unsigned __int128)0 - (unsigned __int128)V
                                       : (unsigned __int128)V;
    const unsigned long long hi  = (unsigned long long)(a >> 64), lo = (unsigned long long)a;
    const int lz                 = hi ? __clzll(hi) : 64 + __clzll(lo);
    const unsigned long long u   = (unsigned long long)((a << lz) >> 64); // leading bit at 63
    // 53 bits, the leading one of which adds 1 to the exponent field
    const unsigned long long m = (u >> 11) + ((u >> 10) & 1);
    const int field            = 1023 + 126 - lz + E;
    if ((unsigned)(field - 1) >= 2044u)
    {
        const double v = scalbn((double)u, E + 64 - lz);
        return neg ? -v : v;
    }
    return __longlong_as_double(
        (long long)(m + ((unsigned long long)field << 52) + (neg ? 1ull << 63 : 0ull)));
}

/* One CTA per SM walks the items.  Warp 0 streams the slices of both operands
 * (two stages of up to 114 KB), warp 1 issues the MMAs, one accumulator per
 * s + t, and warps 2 .. 17 add the accumulators into 64-bit integers in
 * registers (32 per thread) and finish the tile.  A tile has 128 columns,
 * for which TMEM holds four accumulators: K is walked twice, for s + t = 4 .. 6
 * (18 products of 7 slices) and 0 .. 3 (10 products of 4).  An MMA of 128 x 128
 * x 16 reads 8 KB of shared memory in 64 clocks, just what the SM delivers; one
 * of 128 x 64 would wait for it, so narrow tiles, which take all of s + t in
 * one walk (NP = 1), serve only products of at most 64 columns.  The accumulators
 * are handed over one by one: those of the next 192 values start while the
 * epilogue warps still empty the later ones. */
template <int NP, int NS>
__global__ void __launch_bounds__(THREADS, 1) slice_product_kernel(
    const __grid_constant__ CUtensorMap mA, const __grid_constant__ CUtensorMap mB, const Params p)
{
    using namespace tc;
    constexpr int B_SLICE = Form<NP, NS>::B_SLICE, STAGE = Form<NP, NS>::STAGE;
    // (one decision for the CTA: another one that gives up may set it just now)
    if (__syncthreads_or(*(volatile const int*)p.bad)) return;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full  = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE);
    uint64_t* empty = full + STAGES;
    uint64_t* accf  = empty + STAGES; // the MMAs up to a drain are done
    uint64_t* acce  = accf + 1;       // [NS] the epilogue warps have read accumulator a
    uint32_t* tslot = reinterpret_cast<uint32_t*>(acce + NS);
    __shared__ volatile int abort_all; // a wait gave up
    __shared__ uint64_t mma_done;

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    // diagonals s + t of walk ps: [pass_lo, pass_hi), which read slices < pass_hi
    auto pass_lo = [](int ps) { return NP == 1 || ps == 1 ? 0 : 4; };
    auto pass_hi = [](int ps) { return NP == 1 || ps == 0 ? NS : 4; };
    auto drain   = [](int ps) { return ps == 0 ? DRAIN : DRAIN2; };
    if (threadIdx.x == 0)
    {
        for (int s = 0; s < STAGES; s++)
        {
            mbar_init(full + s, 1);
            mbar_init(empty + s, 1);
        }
        mbar_init(accf, 1);
        mbar_init(&mma_done, 1);
        for (int a = 0; a < NS; a++)
            mbar_init(acce + a, EPI);
        abort_all = 0;
        fence_mbar_init();
    }
    if (warp == 1)
    {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tslot)),
            "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = *tslot;

    if (warp == 0 && lane == 0)
    {
        prefetch_map(&mA);
        prefetch_map(&mB);
        const uint32_t bytes = (uint32_t)(A_SLICE + p.bn * BK * 2); // of one slice
        int g                = 0; // stages issued so far
        for (int w = blockIdx.x; w < p.nitems && !abort_all; w += gridDim.x)
        {
            int ti, tj, st0, nst;
            decode(p, w, ti, tj, st0, nst);
            for (int ps = 0; ps < NP && !abort_all; ps++)
            {
                const int ns = pass_hi(ps);
                for (int it = 0; it < nst; it++, g++)
                {
                    const int b = g % STAGES;
                    if (!mbar_wait(empty + b, (uint32_t)(((g / STAGES) & 1) ^ 1), p.polls))
                    {
                        abort_all = 1;
                        break;
                    }
                    unsigned char* st = smem + b * STAGE;
                    mbar_arrive_expect_tx(full + b, ns * bytes);
                    const int k = (st0 + it) * BK, e0 = k % 64, kb = k / 64;
#pragma unroll 1
                    for (int s = 0; s < ns; s++)
                    {
                        tma_load_3d(st + s * A_SLICE, &mA, e0, ti * BM, s * p.kblocks + kb,
                            full + b);
                        tma_load_3d(st + NS * A_SLICE + s * B_SLICE, &mB, e0, tj * p.bn,
                            s * p.kblocks + kb, full + b);
                    }
                }
            }
        }
        drain_loads<STAGES>(full, g);
    }
    else if (warp == 1 && lane == 0)
    {
        const uint32_t id = instr_desc<1>(BM, 0) | ((uint32_t)(p.bn >> 3) << 17);
        int g = 0, drains = 0; // drains committed so far
        for (int w = blockIdx.x; w < p.nitems && !abort_all; w += gridDim.x)
        {
            int ti, tj, st0, nst;
            decode(p, w, ti, tj, st0, nst);
            bool ok = true;
            for (int ps = 0; ps < NP && ok; ps++)
            {
                const int lo = pass_lo(ps), hi = pass_hi(ps);
                for (int it = 0; it < nst && ok; it++, g++)
                {
                    const int b = g % STAGES;
                    ok          = mbar_wait(full + b, (uint32_t)((g / STAGES) & 1), p.polls);
                    if (!ok) break;
                    fence_after_sync();
                    const uint64_t ad = desc_sw<64>(smem_u32(smem + b * STAGE));
                    const uint64_t bd = desc_sw<64>(smem_u32(smem + b * STAGE) + NS * A_SLICE);
                    const bool fresh  = it % drain(ps) == 0;
                    // one descriptor addition per operand and MMA: the issuing
                    // thread has 64 clocks for each
                    auto diagonal = [&](auto dc) {
                        constexpr int d = decltype(dc)::value;
                        if (d < lo || d >= hi || !ok) return;
                        if (fresh && drains > 0)
                        {
                            ok = mbar_wait(acce + (d - lo), (uint32_t)((drains - 1) & 1), p.polls);
                            if (!ok) return;
                            fence_after_sync();
                        }
                        const uint32_t acc = tmem + (uint32_t)((d - lo) * p.bn);
#pragma unroll
                        for (int kk = 0; kk < BK / 16; kk++)
#pragma unroll
                            for (int s = 0; s <= d; s++)
                                mma<1>(acc, ad + ((s * A_SLICE + kk * 32) >> 4),
                                    bd + (((d - s) * B_SLICE + kk * 32) >> 4), id,
                                    (!fresh || kk > 0 || s > 0) ? 1u : 0u);
                    };
                    diagonal(std::integral_constant<int, 0>());
                    diagonal(std::integral_constant<int, 1>());
                    diagonal(std::integral_constant<int, 2>());
                    diagonal(std::integral_constant<int, 3>());
                    diagonal(std::integral_constant<int, 4>());
                    diagonal(std::integral_constant<int, 5>());
                    diagonal(std::integral_constant<int, 6>());
                    if (NS == 8) diagonal(std::integral_constant<int, NS - 1>());
                    if (!ok) break;
                    mma_commit(empty + b);
                    if (it % drain(ps) == drain(ps) - 1 || it == nst - 1)
                    {
                        mma_commit(accf);
                        drains++;
                    }
                }
            }
            if (!ok)
            {
                abort_all = 1;
                mma_commit(accf);
                break;
            }
        }
        drain_mma(&mma_done);
    }
    else if (warp >= 2)
    {
        const int q    = warp & 3; // TMEM lane quarter of this warp
        const int nc   = p.bn / 4, c0 = (warp - 2) / 4 * nc; // its columns
        const uint32_t tw = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c0;
        int drains        = 0;
        for (int w = blockIdx.x; w < p.nitems; w += gridDim.x)
        {
            int ti, tj, st0, nst;
            decode(p, w, ti, tj, st0, nst);
            // the exponents of this thread's row and of column j0 + lane, fetched
            // while the MMAs run
            const size_t i     = (size_t)ti * BM + q * 32 + lane;
            const long long j0 = (long long)tj * p.bn + c0;
            const int ei = i < p.m ? key_exponent<NS>(p.ka[i]) - 14 : 0;
            const int ej
                = lane < nc && j0 + lane < (long long)p.n ? key_exponent<NS>(p.kb[j0 + lane]) : 0;
            // s + t >= 4 in units of 2^-LOW of a digit product, in L (NP 1) or, until
            // the second walk begins, in T; s + t <= 3 in units of 2^-24
            constexpr int EL = Form<NP, NS>::W / 4, LOW = 8 * (NS - 1);
            long long T[EL], L[NP == 1 ? EL : 1];
#pragma unroll
            for (int c = 0; c < EL; c++)
            {
                T[c] = 0;
                if (NP == 1) L[NP == 1 ? c : 0] = 0;
            }
            // entries of this thread: row i, columns j0 .. j0 + nc - 1 that exist
            // (lower: from the diagonal down)
            const int cols = i < p.m ? (int)min((long long)nc, (long long)p.n - j0) : 0;
            const int last = p.t.lower ? (int)min((long long)cols, (long long)i + 1 - j0 - p.t.col0)
                                       : cols;
            const int nd = (nst + DRAIN - 1) / DRAIN; // of the first walk
            const int na = NP == 1 ? nd : nd + (nst + DRAIN2 - 1) / DRAIN2;
            bool ok      = true;
            for (int d = 0; d < na; d++, drains++)
            {
                // (one decision for the warp, which reads TMEM together)
                ok = __all_sync(0xffffffffu,
                    !abort_all && mbar_wait(accf, (uint32_t)(drains & 1), p.polls) && !abort_all);
                if (!ok) break;
                fence_after_sync();
                const int ps = d < nd ? 0 : 1, lo = pass_lo(ps), hi = pass_hi(ps);
                if (NP == 2 && d == nd)
                {
                    // s + t >= 4 goes to the lower words of the sum as it is
#pragma unroll
                    for (int c = 0; c < EL; c++)
                    {
                        if (c < last)
                            atomicAdd(p.t.sum + (p.n + j0 + c) * p.m + i, (unsigned long long)T[c]);
                        T[c] = 0;
                    }
                }
#pragma unroll 1
                for (int a = 0; a < NS; a++)
                {
                    if (lo + a < hi)
                    {
                        const int dg = lo + a;
                        // the accumulator holds integers times 2^(-8 dg): they
                        // join the sum shifted left by at most 24 bits
                        const float up = __uint_as_float((uint32_t)(127 + 8 * dg) << 23);
                        const int mul  = 1 << ((dg >= 4 ? LOW : 24) - 8 * dg);
#pragma unroll
                        for (int c = 0; c < EL; c += 8)
                        {
                            if (c >= nc) break;
                            float x[8];
                            tmem_ld8(tw + a * p.bn + c, x);
                            tmem_wait_ld(x);
#pragma unroll
                            for (int i = 0; i < 8; i++)
                            {
                                const long long y = (long long)__float2int_rn(x[i] * up) * mul;
                                if (NP == 1 && dg >= 4)
                                    L[NP == 1 ? c + i : 0] += y;
                                else
                                    T[c + i] += y;
                            }
                        }
                    }
                    fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(acce + a);
                }
            }
            if (!ok)
            {
                abort_all = 1;
                break;
            }
#pragma unroll
            for (int c = 0; c < EL; c += 8)
            {
                if (c >= nc) break;
                if (p.t.sum)
                {
                    // in units of 2^-SUM_W: upper 2^32 + lower
#pragma unroll
                    for (int x = 0; x < 8; x++)
                        if (c + x < last)
                        {
                            const long long v     = T[c + x];
                            unsigned long long* o = p.t.sum + (j0 + c + x) * p.m + i;
                            atomicAdd(o, (unsigned long long)(v >> 8));
                            atomicAdd(o + p.n * p.m,
                                (unsigned long long)(((v & 255) << 24)
                                                     + (NP == 1 ? L[NP == 1 ? c + x : 0] : 0)));
                        }
                    continue;
                }
                double v[8];
#pragma unroll
                for (int x = 0; x < 8; x++)
                    v[x] = scaled(((__int128)T[c + x] << (LOW - 24)) + L[NP == 1 ? c + x : 0],
                        ei - LOW + __shfl_sync(0xffffffffu, ej, c + x));
                if (p.t.beta != 0.)
                {
                    double y[8];
#pragma unroll
                    for (int x = 0; x < 8; x++)
                        y[x] = c + x < last ? p.t.cin[(j0 + c + x) * p.t.ldcin + i] : 0.;
#pragma unroll
                    for (int x = 0; x < 8; x++)
                        v[x] = p.t.alpha * v[x] + p.t.beta * y[x];
                }
                else if (p.t.alpha != 1.)
                {
#pragma unroll
                    for (int x = 0; x < 8; x++)
                        v[x] *= p.t.alpha;
                }
#pragma unroll
                for (int x = 0; x < 8; x++)
                    if (c + x < last) p.t.C[(j0 + c + x) * p.t.ldc + i] = v[x];
            }
        }
    }
    fence_before_sync();
    __syncthreads(); // every role is done: abort_all is final
    fence_after_sync();
    if (abort_all && threadIdx.x == 0)
    {
        // a wait gave up: the CUDA-core kernels form the product instead, or, where
        // C held an operand that is overwritten in part by now, fill it with NaN
        const bool lost = p.t.sum == nullptr && p.t.beta != 0. && p.t.cin == p.t.C;
        atomicExch(p.bad, lost ? LOST : 1);
    }
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512)
                     : "memory");
}

/* C(i, j) += the integer sums of Target::sum */
__global__ void __launch_bounds__(256) add_sums_kernel(const unsigned long long* __restrict__ sum,
    int m, int n, const int* __restrict__ ka, const int* __restrict__ kb, int lower, int col0,
    double* __restrict__ C, size_t ldc, const int* __restrict__ bad)
{
    if (*bad) return;
    const size_t total = (size_t)m * n;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (size_t)gridDim.x * blockDim.x)
    {
        const int i = (int)(t % m), j = (int)(t / m);
        if (lower && i < j + col0) continue;
        const long long lo = (long long)sum[total + t];
        const long long hi = (long long)sum[t] + (lo >> 32);
        const double v = (double)hi * 4294967296. + (double)(unsigned)lo;
        C[j * ldc + i] += scalbn(v, key_exponent<7>(ka[i]) + key_exponent<7>(kb[j]) - 14 - SUM_W);
    }
}

size_t plane_bytes(size_t rows, size_t K, int ns)
{
    return ns * rows * ((K + 63) / 64) * 128;
}

int row_keys(const View& v, int* keys, int* bad, cudaStream_t s)
{
    MGX_TRY(cuda_check(cudaMemsetAsync(keys, 0, v.rows * sizeof(int), s), "keys reset"));
    if (v.kmajor)
    {
        const unsigned gy = (unsigned)std::min<size_t>(v.rows, 32768);
        const unsigned gx = (unsigned)std::max<size_t>(1,
            std::min<size_t>((v.K + 4095) / 4096, (4096 + gy - 1) / gy));
        keys_kmajor_kernel<<<dim3(gx, gy), 256, 0, s>>>(v.x, v.ld, v.rows, v.K, keys, bad);
    }
    else
    {
        const unsigned gx = (unsigned)std::min<size_t>((v.rows + 127) / 128, 65536);
        const unsigned gy = (unsigned)std::max<size_t>(1,
            std::min<size_t>((v.K + 31) / 32, (1024 + gx - 1) / gx));
        keys_rmajor_kernel<<<dim3(gx, gy), 128, 0, s>>>(v.x, v.ld, v.rows, v.K, keys, bad);
    }
    MGX_LAUNCH_CHECK("slice keys kernel");
    return MGX_OK;
}

int make_planes(const View& v, size_t k0, size_t kc, const int* keys, void* planes, int ns,
    cudaStream_t s)
{
    const size_t kblocks = (kc + 63) / 64;
    if (v.kmajor)
    {
        const size_t total = v.rows * kblocks * 8;
        auto kern = ns == 8 ? planes_kmajor_kernel<8> : planes_kmajor_kernel<7>;
        kern<<<(unsigned)std::min<size_t>((total + 255) / 256, 1u << 20), 256, 0, s>>>(v.x + k0, v.ld, v.rows, kc, keys, kblocks, (__nv_bfloat16*)planes);
    }
    else
    {
        const dim3 grid((unsigned)((v.rows + 63) / 64), (unsigned)kblocks);
        if (grid.y > 65535) return fail(MGX_UNSUPPORTED, "slices: K too large");
        auto kern = ns == 8 ? planes_rmajor_kernel<8> : planes_rmajor_kernel<7>;
        kern<<<grid, 256, 0, s>>>(v.x + k0 * v.ld, v.ld, v.rows, kc, keys, kblocks,
            (__nv_bfloat16*)planes);
    }
    MGX_LAUNCH_CHECK("slice planes kernel");
    return MGX_OK;
}

int product(int sms, size_t m, const void* pa, const int* ka, size_t n, const void* pb,
    const int* kb, size_t kc, const Target& t, int* bad, cudaStream_t s)
{
    const int ns = t.sum ? NS_SUM : NS_STORE;
    if (m == 0 || n == 0 || kc == 0) return MGX_OK;
    Params p;
    p.m = m;
    p.n = n;
    p.nti = (int)((m + BM - 1) / BM);
    // equal column tiles of at most `width`: BN where K is split over the SMs;
    // else the width whose tiles are done first (an MMA of bn columns takes
    // about 64 + bn / 4 clocks, a tile some 12000 besides)
    // (an eighth digit leaves room for one walk over 64 columns only)
    const int most = ns == 8 ? BN1 : BN;
    int width      = most;
    if (!t.sum)
    {
        double best = 0.;
        for (int c = most; c >= 32; c -= 32)
        {
            const long tiles = (long)p.nti * ((n + c - 1) / c);
            const double cost = (double)((tiles + sms - 1) / sms)
                                * (ns * (ns + 1) / 2. * (kc + 15) / 16 * (64 + c / 4) + 12000.);
            if (c == most || cost < best)
            {
                best  = cost;
                width = c;
            }
        }
    }
    p.ntj = (int)((n + width - 1) / width);
    p.bn  = (int)(((n + p.ntj - 1) / p.ntj + 31) / 32 * 32);
    p.ntiles = p.nti * p.ntj;
    if (t.lower)
    {
        p.ntiles = 0;
        for (int j = 0; j < p.ntj; j++)
            p.ntiles += p.nti - first_tile(t.col0 + j * p.bn, p.nti);
        if (p.ntiles == 0) return MGX_OK;
    }
    p.kblocks = (int)((kc + 63) / 64);
    p.nst     = (int)((kc + BK - 1) / BK);
    p.st_per_item = p.nst;
    if (t.sum)
    {
        // K split into items of whole drains: the split whose busiest SM has
        // the least to do (a drain's worth of work for the end of each item),
        // of at most 2^17 values each (T then reaches 2^55)
        const int nd = (p.nst + DRAIN - 1) / DRAIN;
        long best    = -1;
        for (int ks = 1; ks <= std::min(nd, std::max(1, 4 * sms / p.ntiles + 1)); ks++)
        {
            const int per    = (nd + ks - 1) / ks;
            const long items = (long)p.ntiles * ((nd + per - 1) / per);
            const long cost  = ((items + sms - 1) / sms) * (per + 1);
            if (best < 0 || cost < best)
            {
                best          = cost;
                p.st_per_item = per * DRAIN;
            }
        }
        p.st_per_item = std::min(p.st_per_item, (1 << 17) / BK);
    }
    const int ks     = (p.nst + p.st_per_item - 1) / p.st_per_item;
    const long items = (long)p.ntiles * ks;
    if (items > (1L << 30)) return fail(MGX_UNSUPPORTED, "too many work items");
    p.nitems = (int)items;
    p.ka  = ka;
    p.kb  = kb;
    p.t   = t;
    p.bad = bad;
    p.polls = tc::wait_polls();
    CUtensorMap mA, mB;
    MGX_TRY(tc::make_map_blocked(&mA, pa, m, (size_t)ns * p.kblocks, BM, 64));
    MGX_TRY(tc::make_map_blocked(&mB, pb, n, (size_t)ns * p.kblocks, p.bn, 64));
    const bool two    = p.bn > BN1;
    auto kern         = ns == 8 ? slice_product_kernel<1, 8>
                        : two   ? slice_product_kernel<2, 7> : slice_product_kernel<1, 7>;
    const size_t smem = ns == 8 ? Form<1, 8>::SMEM : two ? Form<2, 7>::SMEM : Form<1, 7>::SMEM;
    MGX_TRY(cuda_check(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)smem),
        "slice_product_kernel smem attribute"));
    kern<<<(int)std::min<long>(items, sms), THREADS, smem, s>>>(mA, mB, p);
    MGX_LAUNCH_CHECK("slice_product_kernel");
    return MGX_OK;
}

bool pays(const mgx_ctx* ctx, size_t m, size_t n, size_t K)
{
    return ctx->fp64_slices && (double)m * (double)n * (double)K >= 16. * 1024. * 1024.;
}

namespace
{
size_t up256(size_t b) { return (b + 255) / 256 * 256; }

/* keys of na + nb rows, the flag and the planes of `planes`
 * bytes in ctx's workspace */
int workspace(mgx_ctx* ctx, size_t na, size_t nb, size_t planes, int** ka, int** kb, int** bad,
    char** pl)
{
    const size_t head = up256((na + nb + 2) * sizeof(int));
    if (const char* e = getenv("MGX_SLICE_ROOM")) // bytes, for tests: no memory for more
        if (head + planes > (size_t)atoll(e)) return MGX_NO_MEMORY;
    MGX_TRY(ctx->slices.ensure(head + planes));
    *bad = (int*)ctx->slices.ptr;
    *ka  = *bad + 2;
    *kb  = *ka + na;
    *pl  = (char*)ctx->slices.ptr + head;
    return MGX_OK;
}

/* The bytes that planes may take at first: PLANE_CAP, MGX_SLICE_CAP for tests, or
 * what a former call had memory for. */
size_t plane_cap(const mgx_ctx* ctx)
{
    size_t cap = PLANE_CAP;
    if (const char* e = getenv("MGX_SLICE_CAP"))
        if (atoll(e) > 0) cap = (size_t)atoll(e);
    return ctx->slice_cap ? std::min(cap, ctx->slice_cap) : cap;
}

/* take(cap) with half the planes each time that there is no memory for them,
 * which the context keeps in mind: smaller chunks cost a few launches, the CUDA
 * cores ten times the time */
template <typename F> int with_room(mgx_ctx* ctx, F take)
{
    for (size_t cap = plane_cap(ctx);; cap /= 2)
    {
        const int st = take(cap);
        if (st != MGX_NO_MEMORY || cap / 2 < PLANE_CAP_LEAST) return st;
        ctx->slice_cap = cap / 2;
    }
}
} // namespace

int accumulate(mgx_ctx* ctx, const double* A, size_t ld, size_t K, int n, const Factor* f, int nf,
    int** bad, cudaStream_t s)
{
    if (K > MAX_K_SUM) return MGX_NO_MEMORY;
    // the planes of A and, in turn, those of each B that is not A; a sum and
    // the keys of each
    size_t brows = 0, bkeys = 0, sums = 0;
    for (int i = 0; i < nf; i++)
    {
        if (f[i].B != A || f[i].ncols != n)
        {
            brows = std::max<size_t>(brows, f[i].ncols);
            bkeys += f[i].ncols;
        }
        sums += 2 * (size_t)n * f[i].ncols;
    }
    size_t kc, pa_bytes, pb_bytes;
    int *ka, *kb;
    char* pl;
    MGX_TRY(with_room(ctx, [&](size_t cap) {
        const size_t fit = std::max<size_t>(1, cap / plane_bytes(n + brows, 64, NS_SUM));
        kc       = std::min((K + 63) / 64, fit) * 64;
        pa_bytes = up256(plane_bytes(n, kc, NS_SUM));
        pb_bytes = up256(plane_bytes(brows, kc, NS_SUM));
        return workspace(ctx, n, bkeys, pa_bytes + pb_bytes + sums * sizeof(unsigned long long),
            &ka, &kb, bad, &pl);
    }));
    char* pb  = pl + pa_bytes;
    auto* sum = (unsigned long long*)(pb + pb_bytes);
    MGX_TRY(cuda_check(cudaMemsetAsync(*bad, 0, sizeof(int), s), "slice flag"));
    MGX_TRY(cuda_check(cudaMemsetAsync(sum, 0, sums * sizeof(unsigned long long), s), "slice sums"));
    const View va = { A, ld, (size_t)n, K, true };
    MGX_TRY(row_keys(va, ka, *bad, s));
    struct Part
    {
        bool same;
        View v;
        int* keys;
        Target t;
    };
    std::vector<Part> parts;
    for (int i = 0; i < nf; i++)
    {
        Part q;
        q.same = f[i].B == A && f[i].ncols == n;
        q.v    = { f[i].B, ld, (size_t)f[i].ncols, K, true };
        q.keys = q.same ? ka : kb;
        q.t    = { nullptr, 0, sum, 1., 0., nullptr, 0, f[i].lower, f[i].col0 };
        sum += 2 * (size_t)n * f[i].ncols;
        if (!q.same)
        {
            MGX_TRY(row_keys(q.v, kb, *bad, s));
            kb += f[i].ncols;
        }
        parts.push_back(q);
    }
    for (size_t k0 = 0; k0 < K; k0 += kc)
    {
        const size_t k = std::min(kc, K - k0);
        MGX_TRY(make_planes(va, k0, k, ka, pl, NS_SUM, s));
        for (const Part& q : parts)
        {
            if (!q.same) MGX_TRY(make_planes(q.v, k0, k, q.keys, pb, NS_SUM, s));
            MGX_TRY(product(ctx->sm_count, n, pl, ka, q.v.rows, q.same ? pl : pb, q.keys, k, q.t,
                *bad, s));
        }
    }
    for (int i = 0; i < nf; i++)
    {
        const unsigned blocks
            = (unsigned)std::min<size_t>(((size_t)n * f[i].ncols + 255) / 256, 2048);
        add_sums_kernel<<<blocks, 256, 0, s>>>(parts[i].t.sum, n, f[i].ncols, ka, parts[i].keys,
            f[i].lower, f[i].col0, f[i].C, n, *bad);
        MGX_LAUNCH_CHECK("add_sums_kernel");
    }
    return MGX_OK;
}

int store_begin(mgx_ctx* ctx, const View& A, const View& B, StorePlan* p, cudaStream_t s)
{
    constexpr int ns = NS_STORE;
    const size_t K  = A.K;
    if (K > MAX_K_STORE) return MGX_NO_MEMORY;
    const size_t b1 = up256(plane_bytes(B.rows, K, ns));
    char* pl;
    MGX_TRY(with_room(ctx, [&](size_t cap) {
        const size_t fit = std::max<size_t>(1, cap / plane_bytes(BM, K, ns));
        p->chunk = std::min((A.rows + BM - 1) / BM, fit) * BM;
        const size_t rows = std::min(p->chunk, A.rows);
        return workspace(ctx, rows, B.rows, b1 + plane_bytes(rows, K, ns), &p->ka, &p->kb, &p->bad,
            &pl);
    }));
    p->pb = pl;
    p->pa = pl + b1;
    MGX_TRY(cuda_check(cudaMemsetAsync(p->bad, 0, sizeof(int), s), "slice flag"));
    MGX_TRY(row_keys(B, p->kb, p->bad, s));
    return make_planes(B, 0, K, p->kb, p->pb, ns, s);
}

int store_chunk(mgx_ctx* ctx, const View& A, const View& B, const Target& t, const StorePlan& p,
    size_t r0, size_t rows, cudaStream_t s)
{
    View a = A;
    a.x += A.kmajor ? r0 * A.ld : r0;
    a.rows   = rows;
    Target c = t;
    c.C += r0;
    if (c.cin) c.cin += r0;
    c.col0 -= (int)r0;
    MGX_TRY(row_keys(a, p.ka, p.bad, s));
    MGX_TRY(make_planes(a, 0, A.K, p.ka, p.pa, NS_STORE, s));
    return product(ctx->sm_count, rows, p.pa, p.ka, B.rows, p.pb, p.kb, A.K, c, p.bad, s);
}
} // namespace sl
} // namespace mgx
