// What the matmul kernels on the 5th-generation tensor cores share: mbarriers with bounded waits, TMA loads, matrix
// descriptors, the walk over output tiles, tensor maps, and the flag that a wait that gave up leaves behind.
#pragma once
#include <cuda.h>

#include <cstdint>

#include "common.h"

namespace lapis_b200 {

// Device word that a kernel sets when a bounded wait gives up (lapis_b200_bgemm_status reads it); null on failure, with
// the error recorded.
int *bgemm_error_flag(int dev);

namespace tc {

constexpr int BM = 128;  // rows of an output tile of one CTA: the lanes of tensor memory
constexpr uint32_t WAIT_LIMIT = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Bounded wait: false when the phase did not complete within WAIT_LIMIT polls.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
  const uint32_t addr = smem_u32(bar);
  for (uint32_t i = 0; i < WAIT_LIMIT; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
// The same for a barrier that threads of the other CTA of a pair arrive at.
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t *bar, uint32_t parity) {
  const uint32_t addr = smem_u32(bar);
  for (uint32_t i = 0; i < WAIT_LIMIT; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, uint64_t *bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}

// Tile t of the persistent schedule -> (batch, m block, n block).  Within a batch entry the tiles
// are walked in groups of 8 m-blocks so that the blocks running at the same time share A and B
// panels in L2.
struct TileCoord {
  int batch, m0, n0;
};
__device__ __forceinline__ TileCoord tile_coord(int t, int tm, int tn, int bm, int bn) {
  constexpr int GROUP = 8;
  const int per = tm * tn;
  const int batch = t / per, r = t - batch * per;
  const int g = r / (GROUP * tn), first_m = g * GROUP;
  const int gsize = tm - first_m < GROUP ? tm - first_m : GROUP;
  const int q = r - g * GROUP * tn;
  return TileCoord{batch, (first_m + q % gsize) * bm, (q / gsize) * bn};
}

// Row-major [batch][rows][cols] tensor with rows row_bytes apart, box = box_rows x box_cols, swizzled.
int make_map(CUtensorMap *map, CUtensorMapDataType type, const void *base, int64_t batch, int64_t rows, int64_t cols,
             int64_t row_bytes, int box_rows, int box_cols, CUtensorMapSwizzle swizzle);

}  // namespace tc

// Which operand panels of a product that is computed from split operands (gemm_split.cu) the split does not cover: a word
// for every 128 rows of A and every 128 columns of B, for each of the stretches of `kc` that K is cut into (whole tiles: that a
// launch takes).  Null: the kernel computes everything.
struct PanelFlags {
  const unsigned long long *a, *b;  // [batch][stretches][panels_a], [batch][stretches][panels_b]
  int panels_a, panels_b;
  int stretches, kc;
  __device__ __forceinline__ const unsigned long long *row(int64_t batch, int s) const { return a + (batch * stretches + s) * panels_a; }
  __device__ __forceinline__ const unsigned long long *col(int64_t batch, int s) const { return b + (batch * stretches + s) * panels_b; }
};

}  // namespace lapis_b200
