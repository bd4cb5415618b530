// Host-side construction of TMA tensor maps (cuTensorMapEncodeTiled through the runtime's
// driver entry point, so the library needs no link-time dependency on libcuda) and the
// device-side tiled load.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace ak {

enum TmaSwizzle { TMA_SWIZZLE_NONE = 0, TMA_SWIZZLE_128B = 3 };

// 2-D row-major tensor [rows, cols] of `elem_bytes`-byte elements (2 = bf16, 4 = f32), row pitch
// `row_stride_bytes` (multiple of 16). Box = [box_rows, box_cols]; out-of-range elements read 0.
int make_tmap_2d(CUtensorMap* out, const void* base, uint32_t elem_bytes, uint64_t cols, uint64_t rows,
                 uint64_t row_stride_bytes, uint32_t box_cols, uint32_t box_rows, TmaSwizzle swizzle);

// bf16 [rows, cols] seen as [rows, cols / inner, inner], so that one box may hold more than 256 columns of its rows: box_pieces * inner of
// them, row after row. What lies outside reads 0.
int make_tmap_rows(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint32_t inner, uint32_t box_pieces, uint32_t box_rows);

#ifdef __CUDACC__
// Tiled 2-D load, completion counted in bytes on `bar`. x (the innermost coordinate) times the
// element size must be a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* tmap, int32_t x, int32_t y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
            smem_u32(smem_dst)),
        "l"(tmap), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}
// A box of make_tmap_rows(): pieces from `piece` on of the rows from `row` on. `pol`: L2 cache policy.
__device__ __forceinline__ void tma_load_rows(void* smem_dst, const CUtensorMap* tmap, int32_t piece, int32_t row, uint64_t* bar, uint64_t pol) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4, %5}], [%2], %6;" ::"r"(
            smem_u32(smem_dst)),
        "l"(tmap), "r"(smem_u32(bar)), "r"(0), "r"(piece), "r"(row), "l"(pol)
        : "memory");
}
// The same box brought into L2
__device__ __forceinline__ void tma_prefetch_rows(const CUtensorMap* tmap, int32_t piece, int32_t row) {
    asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global [%0, {%1, %2, %3}];" ::"l"(tmap), "r"(0), "r"(piece), "r"(row) : "memory");
}
// Tiled 2-D store from shared memory (elements outside the tensor are not written), and the same adding into f32. The
// shared-memory writes must be ordered before it with tma_store_fence() in the writing threads and a barrier.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* tmap, const void* smem_src, int32_t x, int32_t y) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(tmap), "r"(smem_u32(smem_src)), "r"(x), "r"(y)
                 : "memory");
}
__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap* tmap, const void* smem_src, int32_t x, int32_t y) {
    asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(tmap), "r"(smem_u32(smem_src)),
                 "r"(x), "r"(y)
                 : "memory");
}
__device__ __forceinline__ void tma_store_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// at most N of this thread's store groups still read their shared-memory source / are still under way
template <int N> __device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
template <int N> __device__ __forceinline__ void tma_store_wait() { asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* tmap) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(tmap) : "memory");
}
#endif

}  // namespace ak
