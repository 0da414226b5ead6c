// tma_ring.cuh -- operand staging by TMA for products of 64-column tiles whose
// inner index runs along the columns: boxes of eight complex rows (128 bytes)
// through a ring of mbarrier stages, shared by the persistent LDL^H and the
// candidates' GEMM.  Every wait is bounded.
#pragma once
#include <cuda.h>  // CUtensorMap
#include "ecg_internal.h"

namespace ecg {

constexpr int TMA_KC = 8;           // k rows per TMA stage of an update: 128 bytes, the width of the swizzle
constexpr int TMA_ST = 6;           // stages

// ---------------------------------------------------------------------------
// mbarriers and boxes.
// ---------------------------------------------------------------------------
constexpr int TMA_LIMIT = 1 << 21;  // bound on the polls for a copy or a stage (tens of ms)

__device__ __forceinline__ unsigned smem32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(unsigned bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(unsigned bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Wait for the phase of the given parity to end; false when the limit runs out.
__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned parity)
{
    for (int i = 0; i < TMA_LIMIT; i++) {
        unsigned done;
        asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n"
            "}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
// Box of 8 complex rows from row k0 (16 doubles, x = 2 k0: 16-byte aligned)
// and the map's columns from column c.
__device__ __forceinline__ void tma_box(unsigned dst, const CUtensorMap* map, int k0, int c, unsigned bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            dst),
        "l"(map), "r"(2 * k0), "r"(c), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void fence_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// The stages' ring as it goes on from one tile to the next: the next
// stage and the parity of its current use.
struct TmaRing {
    unsigned full, empty;  // shared addresses of TMA_ST mbarriers each
    int st = 0;
    unsigned ph = 0;
    // full: one arrival and the bytes; empty: eight warps
    __device__ __forceinline__ void init(unsigned at, int tid)
    {
        full = at;
        empty = at + 8u * TMA_ST;
        if (tid == 0) {
            for (int i = 0; i < TMA_ST; i++) {
                bar_init(full + 8u * i, 1);
                bar_init(empty + 8u * i, 8);
            }
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    }
    __device__ __forceinline__ void step(int& i, unsigned& p) const
    {
        if (++i == TMA_ST) {
            i = 0;
            p ^= 1u;
        }
    }
};
// Stages refilled before chunk ch of n, one a chunk from the third on.
__device__ __forceinline__ int ring_refilled(int ch, int n) { return max(0, min(ch, n - TMA_ST + 2) - 2); }
// Thread 0, after a wait that ran out: a CTA does not leave while a copy may
// still write its shared memory.  `uses` are to come from the one of stage i
// and parity p on, the oldest not known to have arrived; of them those of the
// next TMA_ST stages, on either side of the ring's end, may be in flight (one
// that was not asked for runs into the limit).  A call, because its code
// inside the candidates' GEMM costs that 1 %.
static __device__ __noinline__ void ring_drain(unsigned full, int i, unsigned p, int uses)
{
    for (int u = 0; u < min(uses, TMA_ST); u++) {
        bar_wait(full + 8u * i, p);
        if (++i == TMA_ST) {
            i = 0;
            p ^= 1u;
        }
    }
}

// Tensor map of the rows x cols matrix at A (column-major complex) as doubles
// by columns, boxes of TMA_KC complex rows x `box_cols` columns, 128-byte
// swizzle; beyond the matrix a box holds zeros.
inline bool tma_map(CUtensorMap* map, void* A, int ld, int rows, int cols, int box_cols)
{
    typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                               const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                               CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &found) != cudaSuccess || !fn) {
        cudaGetLastError();
        return false;
    }
    const cuuint64_t dim[2] = {2 * (cuuint64_t)rows, (cuuint64_t)cols}, stride[1] = {(cuuint64_t)ld * sizeof(cd)};
    const cuuint32_t box[2] = {2 * TMA_KC, (cuuint32_t)box_cols}, one[2] = {1, 1};
    return reinterpret_cast<Encode>(fn)(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, A, dim, stride, box, one,
                                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                        CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace ecg
