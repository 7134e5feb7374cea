// TMA (tensor-map) support: host-side descriptor builder and device-side issue wrappers.
// Only plain per-CTA tiled loads are used (the K / V key blocks of the attention kernels),
// completion through an mbarrier's transaction count.  No multicast.
#pragma once
#include <cuda.h>

#include "fmb_tc.cuh"

namespace fmb {

// 3-D tensor map over a (tokens, heads, d) tensor with arbitrary (16-byte aligned) token and head
// strides: box = 64 elements of d x 1 head x box_rows tokens, 128-byte swizzle; elements past d and
// tokens past `rows` read as zero.
int make_tmap_3d(CUtensorMap* map, const void* base, int dtype, uint64_t d, uint64_t heads, uint64_t rows,
                 uint64_t head_stride_bytes, uint64_t row_stride_bytes, uint32_t box_rows);

namespace tc {

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

// box whose first element is (x, head, row) -> shared memory
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int head, int row, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      :
      : "r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(head), "r"(row)
      : "memory");
}

// shared memory -> box at (x, head, row); joins the thread's open bulk group.  The box must lie inside the tensor.
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, const void* src, int x, int head, int row) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];"
               :
               : "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(src)), "r"(x), "r"(head), "r"(row)
               : "memory");
}

__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

}  // namespace tc
}  // namespace fmb
