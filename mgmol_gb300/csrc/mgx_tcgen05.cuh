// tcgen05 / TMA helpers shared by the tensor-core kernels: shared-memory and
// instruction descriptors, tiled bulk loads, MMA issue and commit, TMEM reads,
// and the tensor maps of K-blocked operands.
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <cstdlib>

#include "mgx_internal.cuh"

namespace mgx
{
namespace tc
{
// Shared-memory operand descriptor of a K-major tile whose rows are one
// swizzle atom of SW bytes (128 or 64): stride between 8-row groups 8 * SW,
// layout SWIZZLE_128B (2) or SWIZZLE_64B (4).
template <int SW>
__device__ __forceinline__ uint64_t desc_sw(uint32_t saddr)
{
    static_assert(SW == 128 || SW == 64, "swizzle atom");
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;                 // leading byte offset (unused, K-major swizzled)
    d |= (uint64_t)((8 * SW) >> 4) << 32;   // stride byte offset: 8 rows x SW bytes
    d |= (uint64_t)1 << 46;                 // descriptor version for tcgen05
    d |= (uint64_t)(SW == 128 ? 2 : 4) << 61;
    return d;
}

// Shared-memory descriptor of an MN-major tile (bf16) under SWIZZLE_128B:
// rows of 128 bytes hold 64 consecutive MN elements (one K index each),
// 8-row groups (K) are 1024 bytes apart (stride byte offset) and the next
// 64 MN elements start lbo bytes further (leading byte offset).
__device__ __forceinline__ uint64_t desc_mn128(uint32_t saddr, uint32_t lbo)
{
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// kind::tf32 (KIND 0, operand format 2), kind::f16 with bf16 operands
// (KIND 1, format 1) or with fp16 operands (KIND 2, format 0); FP32 D, both
// operands K-major
template <int KIND>
__host__ __device__ constexpr uint32_t instr_desc(int M, int N)
{
    return (1u << 4) | ((KIND == 0 ? 2u : KIND == 1 ? 1u : 0u) << 7)
           | ((KIND == 0 ? 2u : KIND == 1 ? 1u : 0u) << 10) | ((uint32_t)(N >> 3) << 17)
           | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map,
    int c0, int c1, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(smem_u32(bar))
        : "memory");
}

// 3-D box of a K-blocked operand: (element within the 64-element K block,
// row, K block)
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map,
    int c0, int c1, int c2, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void prefetch_map(const CUtensorMap* map)
{
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map))
                 : "memory");
}

template <int KIND>
__device__ __forceinline__ void mma(uint32_t tmem, uint64_t ad, uint64_t bd,
    uint32_t idesc, uint32_t acc)
{
    if (KIND == 0)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
            "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
            : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
            "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
            : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t* bar)
{
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_u32(bar))
        : "memory");
}

/* What a role owes before its CTA ends, however it got there: the bulk loads
 * that it has started into shared memory (the last ones of a ring of STAGES, g
 * in all) have landed, and the MMAs that it has issued are done (bar: an
 * mbarrier of one arrival that nothing else uses).  Bounded, like every wait. */
template <int STAGES>
__device__ __forceinline__ void drain_loads(uint64_t* full, int g)
{
    for (int k = g > STAGES ? g - STAGES : 0; k < g; k++)
        mbar_wait(full + k % STAGES, (uint32_t)((k / STAGES) & 1));
}
__device__ __forceinline__ void drain_mma(uint64_t* bar)
{
    mma_commit(bar);
    mbar_wait(bar, 0);
}

__device__ __forceinline__ void fence_after_sync()
{
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_before_sync()
{
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32])
{
    uint32_t r[32];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                 "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
                 "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
                 "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
                 "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]),
                 "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; i++)
        v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

/* Polls after which a wait of a product's pipeline gives up; MGX_WAIT_POLLS
 * lowers it (0: every wait gives up), for the tests of what happens then. */
constexpr uint32_t WAIT_POLLS = 1u << 26;
inline uint32_t wait_polls()
{
    const char* e = getenv("MGX_WAIT_POLLS");
    const long v  = e ? atol(e) : (long)WAIT_POLLS;
    return v >= 0 && v < (long)WAIT_POLLS ? (uint32_t)v : WAIT_POLLS;
}

inline PFN_cuTensorMapEncodeTiled_v12000 encoder()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn)
    {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000,
                cudaEnableDefault, &q)
                == cudaSuccess
            && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }
    return fn;
}

// 3-D map over a K-blocked bf16 operand (rows x kblocks * 64): dims
// (64, rows, kblocks), box (sw / 2, box_rows, 1), SWIZZLE_128B / _64B.
inline int make_map_blocked(CUtensorMap* m, const void* base, size_t rows, size_t kblocks,
    int box_rows, int sw = 128, bool half = false)
{
    auto enc = encoder();
    if (!enc) return fail(MGX_CUDA_ERROR, "cuTensorMapEncodeTiled unavailable");
    if ((uintptr_t)base % 16) return fail(MGX_BAD_ARG, "tensor-core operands need 16-byte alignment");
    cuuint64_t dims[3]    = { 64, (cuuint64_t)rows, (cuuint64_t)kblocks };
    cuuint64_t strides[2] = { 128, (cuuint64_t)(rows * 128) };
    cuuint32_t box[3]     = { (cuuint32_t)(sw / 2), (cuuint32_t)box_rows, 1 };
    cuuint32_t estr[3]    = { 1, 1, 1 };
    CUresult r = enc(m, half ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16,
        3, const_cast<void*>(base), dims,
        strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
        sw == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(MGX_CUDA_ERROR, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return MGX_OK;
}

} // namespace tc
} // namespace mgx
