// Inline PTX and the tile order shared by the tensor-core GEMM kernels.
#pragma once
#include <cuda.h>

#include "mbarrier.cuh"

namespace mnpbem {

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"((unsigned long long)map), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void mma_f16(uint32_t dtmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
      ::"r"(dtmem), "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}
// Tile order of the persistent kernels: groups of TC_GROUP_M row tiles, and
// within a group the column tiles one after another (the group's row tiles
// fastest).  The CTAs in flight then share a few A row panels (TC_GROUP_M x
// 128 rows) and a few B' tiles, which stay in L2; with the plain row-fastest
// order every column of tiles sweeps the whole A panel, which at n = 24 000
// and K = 512 (98 MB) does not stay in L2 next to the streamed C tiles and is
// read again from HBM for every column.
constexpr int TC_GROUP_M = 32;
__device__ __forceinline__ void tile_coords(int t, int MT, int NT, int& mt, int& nt) {
  const int per_group = TC_GROUP_M * NT;
  const int g = t / per_group;
  const int m_first = g * TC_GROUP_M;
  const int gm = min(TC_GROUP_M, MT - m_first);
  const int r = t - g * per_group;
  mt = m_first + r % gm;
  nt = r / gm;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

}  // namespace mnpbem
