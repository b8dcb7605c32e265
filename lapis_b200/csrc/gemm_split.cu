// fp32 matmul on the 5th-generation tensor cores from operands that are split once:  C[b] = C_in[b] + A[b] B[b]  for any M,
// N, K and any alignment.
//
// Whole tiles, two parts in fp16:  x 2^e = hi + 2^-11 lo (11 bits each, lo rounded), e one exponent for each row of A and each
// column of B; the product is hi hi + 2^-11 (hi lo + lo hi), three fp16 products at twice the rate of the three TF32 products of
// gemm_tcgen05.cu.  What is left out (lo lo, the rounding of lo) is at most 2^-21 of a product as long as hi is a normal fp16
// number, where the TF32 split, whose parts the tensor core truncates, leaves up to 2^-19.
//
// Other shapes, three parts in bf16:  x = b1 + b2 + b3, 8 bits each and signed, which is all 24 bits of x; six products, b1 b1 in
// one accumulator, the others down to 2^-16 of it (b2 b2, b1 b3) in the second.  What is left out is at most 2^-24 of a product,
// less than its rounding in the kernel for such shapes, and nothing where one factor has 8 bits: products with a permutation or
// a selection are exact, as they are there.  With two parts they were not (a quarter of the elements off by a bit).
//
//   split_kernel       reads A and B once, writes the parts as 16-bit matrices with 16-byte rows (so that TMA can load shapes
//                      and pointers of any alignment), and the scales of two parts.  K is cut into stretches of at most 1024,
//                      each with scales of its own.
//   gemm_split_kernel  a persistent GEMM over the parts: TMA -> tcgen05.mma.kind::f16 -> two accumulators in tensor memory
//                      (the large product, and the mixed ones) -> scaled, joined, added to C: two parts once a stretch, three
//                      parts once, after all of K.
//
// 8192^3: 5.05 -> 2.70 ms where the clock holds (407 TFLOP/s, three products at 75 % of cuBLAS's bf16 rate), 5.91 -> 3.33 where
// power caps it, with an error of 1.25e-6 against 64 bits (2-norm; TF32 split 8.0e-6).  Three parts cost 5 to 65 % more time
// than two: 1000 x 1501 x 777 142 us in the kernel for general shapes, 30.6 with two parts, 36.7 with three; 5000 x 3000 x 1999
// 2270, 260 and 319; 8191^3 46, 4.3 and 5.8 ms.  Their errors, that kernel's first: 1000 x 1501 x 777 uniform in [-1, 1) 5.0e-7,
// 3.9e-7 and 1.2e-7, in [0, 1) 4.2e-7, 1.4e-6 and 1.5e-7, A with 1 % nonzeros 6.3e-8, 7.5e-8 and 5.2e-8, 100 x 200^3 2.6e-7,
// 1.8e-7 and 7.7e-8.
//
// fp16 has 5 bits of exponent: the hi of an element below 2^-14 after scaling (2^-29 of the largest of its row or column)
// would be subnormal and lo lo up to 2^-17 of a product of two such, and an infinity or NaN has no scale.  split_kernel marks
// the 128-row and 128-column panels that hold such an element (three parts: below 2^-31); the products of those panels are left to
// the kernels on unsplit operands (PanelFlags), which run behind this one and return at once where there are none.  Three
// parts: with all of K, in the loop's order and bits.  In 8192 x 8192 normally distributed numbers one is expected in every
// second matrix, in uniformly distributed ones (multiples of 2^-24) none.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "tcgen05.h"

namespace lapis_b200 {

namespace split {

constexpr int KC = 1024;  // longest stretch of K: one scale for each row or column and stretch, one chain in tensor memory
constexpr int GROUP_ROWS = 16, GROUP_COLS = 16;  // rows of A, columns of B that a block of split_kernel takes
constexpr int SPLIT_THREADS = 512;
constexpr float LO_SCALE = 2048.0f, LO_UNSCALE = 1.0f / 2048.0f;

struct Shape {
  int M, N, Np, K;          // Np: columns of the split B, a multiple of GROUP_COLS
  int ldn;                   // elements between rows of B and C
  int chain;                 // elements of K that are added in tensor memory, a multiple of 64
  int kc, first, stretches;  // stretches first .. first + stretches - 1, of kc (a multiple of 64) each, the last one shorter
  int panels_a, panels_b;
  // Three parts, where the launches of several groups of stretches make one product: the sums of the groups in front (null: one
  // group), element by element as the epilogue's threads hold them, whether there are any, and whether this is the last.
  float *sums;
  bool fresh, last;
  __host__ __device__ int length(int s) const { return K - (first + s) * kc < kc ? K - (first + s) * kc : kc; }
};

struct Scratch {
  uint16_t *a, *b;           // [batch][stretch][part][M][kc], [batch][stretch][part][kc][Np]: fp16 or bf16
  float *scale_a, *scale_b;  // [batch][stretch][M], [batch][stretch][Np]: 2^-e
  unsigned char *flag_a, *flag_b;  // a byte for every 16 rows or columns: [batch][stretch][panel][8], strides and place of
  int flag_stretches, flag_first, flag_panels_a, flag_panels_b;  // the first stretch of the launch
};

// Exponent of the scale for a row or column whose largest magnitude has these bits: the largest power of two that keeps it
// below 65504.  False: it has none (infinity, NaN) or one so far out that two scales might leave fp32's range together.
__device__ __forceinline__ bool scale_exponent(uint32_t max_bits, int &e) {
  const int ex = (int)(max_bits >> 23) - 127;
  e = max_bits == 0 ? 0 : (max_bits & 0x7fffffu) < 0x7fe000u ? 15 - ex : 14 - ex;
  return max_bits == 0 || (ex >= -48 && ex <= 48);
}
__device__ __forceinline__ float pow2(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }

// The parts of four elements, scaled by s where there are two; true if one of them is too small beside the largest of its row
// or column.  Two parts: its hi would be subnormal.  Three parts hold it, but rows graded like that keep the loop's order.
template <int PARTS>
__device__ __forceinline__ bool split4(const float (&x)[4], float s, uint2 (&part)[PARTS]) {
  uint16_t h[PARTS][4];
  bool small = false;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float v = __fmul_rn(x[i], s);
    if (PARTS == 2) {
      small |= x[i] != 0.0f && fabsf(v) < 1.0f / 16384.0f;
      const __half hi = __float2half_rn(v);
      h[0][i] = __half_as_ushort(hi);
      h[1][i] = __half_as_ushort(__float2half_rn(__fmul_rn(__fsub_rn(v, __half2float(hi)), LO_SCALE)));
    } else {
      small |= x[i] != 0.0f && fabsf(v) < 1.0f / 65536.0f;
      float rest = x[i];
#pragma unroll
      for (int q = 0; q < PARTS; ++q) {
        const __nv_bfloat16 b = __float2bfloat16_rn(rest);
        h[q][i] = __bfloat16_as_ushort(b);
        rest = __fsub_rn(rest, __bfloat162float(b));
      }
    }
  }
#pragma unroll
  for (int q = 0; q < PARTS; ++q) part[q] = make_uint2(h[q][0] | (uint32_t)h[q][1] << 16, h[q][2] | (uint32_t)h[q][3] << 16);
  return small;
}
// A or B may be what the launch in front has written.
__device__ __forceinline__ float load_now(const float *p) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float4 load_now4(const float *p) {
  float4 v;
  asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t magnitude(float x) { return __float_as_uint(x) & 0x7fffffffu; }

// Bound by memory: reads an element once, writes two halves.  Blocks 0 .. 8 panels_a - 1 take 16 rows of A, a warp each;
// the others 16 columns of B: four threads a row, 128 rows at a time.  A thread keeps its elements in registers between
// the search for the largest and the split.
template <int PARTS, bool VEC_A, bool VEC_B>
__global__ void __launch_bounds__(SPLIT_THREADS, 2)
split_kernel(const float *A, const float *B, Shape sh, Scratch w) {
  __shared__ uint32_t s_max[SPLIT_THREADS / 32][4][4];
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int s = blockIdx.y, kc = sh.length(s);
  const int64_t batch = blockIdx.z, at = batch * sh.stretches + s, k0 = (int64_t)(sh.first + s) * sh.kc;
  const int64_t flags_at = batch * w.flag_stretches + w.flag_first + s;
  const int kpad = (kc + 63) & ~63;
  constexpr int STEPS = KC / 128;
  if ((int)blockIdx.x < 8 * sh.panels_a) {
    const int row = blockIdx.x * GROUP_ROWS + warp;
    bool bad = false;
    if (row < sh.M) {
      const float *src = A + (batch * sh.M + row) * sh.K + k0;
      float v[STEPS][4];
      uint32_t m = 0;
#pragma unroll
      for (int i = 0; i < STEPS; ++i) {
        const int k = 128 * i + 4 * lane;
        if (VEC_A) {
          const float4 q = k < kc ? load_now4(src + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          v[i][0] = q.x, v[i][1] = q.y, v[i][2] = q.z, v[i][3] = q.w;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) v[i][j] = k + j < kc ? load_now(src + k + j) : 0.0f;
        }
      }
#pragma unroll
      for (int i = 0; i < STEPS; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) m = max(m, magnitude(v[i][j]));
      m = __reduce_max_sync(0xffffffffu, m);
      int e;
      bad = !scale_exponent(m, e);
      const float sc = pow2(bad ? 0 : e);
      uint16_t *dst = w.a + ((PARTS * at) * sh.M + row) * sh.kc;
#pragma unroll
      for (int i = 0; i < STEPS; ++i) {
        const int k = 128 * i + 4 * lane;
        uint2 part[PARTS];
        bad |= split4<PARTS>(v[i], sc, part);
        if (k < kpad) {
#pragma unroll
          for (int q = 0; q < PARTS; ++q) *reinterpret_cast<uint2 *>(dst + (int64_t)q * sh.M * sh.kc + k) = part[q];
        }
      }
      if (PARTS == 2 && lane == 0) w.scale_a[at * sh.M + row] = pow2(bad ? 0 : -e);
    }
    pdl_release();
    const int any = __syncthreads_or(bad);
    if (tid == 0) w.flag_a[flags_at * 8 * w.flag_panels_a + blockIdx.x] = any ? 1 : 0;
  } else {
    const int group = blockIdx.x - 8 * sh.panels_a, col = group * GROUP_COLS + 4 * (tid & 3), r0 = tid >> 2;
    bool bad = false;
    if (group * GROUP_COLS < sh.Np) {
      const float *src = B + (batch * sh.K + k0) * sh.ldn + col;
      float v[STEPS][4];
      uint32_t m[4] = {0, 0, 0, 0};
#pragma unroll
      for (int i = 0; i < STEPS; ++i) {
        const int k = r0 + 128 * i;
        if (VEC_B) {
          const float4 q = k < kc && col < sh.N ? load_now4(src + (int64_t)k * sh.ldn) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          v[i][0] = q.x, v[i][1] = q.y, v[i][2] = q.z, v[i][3] = q.w;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) v[i][j] = k < kc && col + j < sh.N ? load_now(src + (int64_t)k * sh.ldn + j) : 0.0f;
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int i = 0; i < STEPS; ++i) m[j] = max(m[j], magnitude(v[i][j]));
        m[j] = max(m[j], __shfl_xor_sync(0xffffffffu, m[j], 4));
        m[j] = max(m[j], __shfl_xor_sync(0xffffffffu, m[j], 8));
        m[j] = max(m[j], __shfl_xor_sync(0xffffffffu, m[j], 16));
      }
      if (lane < 4) {
#pragma unroll
        for (int j = 0; j < 4; ++j) s_max[warp][lane][j] = m[j];
      }
      __syncthreads();
      float sc[4];
      int e[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int q = 0; q < SPLIT_THREADS / 32; ++q) m[j] = max(m[j], s_max[q][tid & 3][j]);
        const bool no = !scale_exponent(m[j], e[j]);
        bad |= no;
        e[j] = no ? 0 : e[j];
        sc[j] = pow2(e[j]);
      }
      if (PARTS == 2 && tid < 4) {
#pragma unroll
        for (int j = 0; j < 4; ++j) w.scale_b[at * sh.Np + col + j] = pow2(-e[j]);
      }
      uint16_t *dst = w.b + (PARTS * at) * sh.kc * sh.Np + col;
#pragma unroll
      for (int i = 0; i < STEPS; ++i) {
        const int k = r0 + 128 * i;
        float x[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          x[j] = PARTS == 2 ? __fmul_rn(v[i][j], sc[j]) : v[i][j];
          bad |= v[i][j] != 0.0f && (PARTS == 2 ? x[j] == 0.0f : fabsf(__fmul_rn(v[i][j], sc[j])) < 1.0f / 65536.0f);
        }
        uint2 part[PARTS];
        const bool small = split4<PARTS>(x, 1.0f, part);  // three parts: seen above
        bad |= PARTS == 2 && small;
        if (k < kpad) {
#pragma unroll
          for (int q = 0; q < PARTS; ++q) *reinterpret_cast<uint2 *>(dst + ((int64_t)q * sh.kc + k) * sh.Np) = part[q];
        }
      }
    }
    pdl_release();
    const int any = __syncthreads_or(bad);
    if (tid == 0) w.flag_b[flags_at * 8 * w.flag_panels_b + group] = any ? 1 : 0;
  }
}

// ---- the product of the parts ------------------------------------------------------------------------------------
constexpr int BK = 64;                       // k block: rows of 128 B, 128-byte swizzle
constexpr int BOX_BYTES = 64 * BK * 2;       // one TMA box of B: 64 k-rows x 64 columns
constexpr int THREADS = 384;                 // producer, MMA issuer, two idle warps, eight epilogue warps
constexpr int TILE_BYTES = 32 * 32 * 4;      // an epilogue warp's staging tile

// CTAS CTAs own a tile of 128 CTAS x BN: each loads its 128 rows of A and its share of B's columns, the first one issues the
// MMAs for all.  In tensor memory: hi hi and mixed products of a tile, 2 BN columns, once or twice.
template <int PARTS_, int CTAS_, int BN_, bool SUMS_ = false>
struct Config {
  static constexpr bool SUMS = SUMS_;  // in several launches, the sums kept in between
  static constexpr int PARTS = PARTS_, CTAS = CTAS_, BN = BN_, BUFS = 256 / BN, NB = BN / CTAS;
  static constexpr int A_BYTES = tc::BM * BK * 2, B_BYTES = NB * BK * 2;  // of a part
  static constexpr int STAGE_BYTES = PARTS * (A_BYTES + B_BYTES), STAGES = 196608 / STAGE_BYTES;
  static constexpr int SMEM_BYTES = 1024 + STAGES * STAGE_BYTES + 8 * TILE_BYTES + 256;
  static constexpr uint32_t TYPE = PARTS == 2 ? 0 : 1;  // f16, bf16
  // D = f32, A and B of TYPE, A K-major, B MN-major
  static constexpr uint32_t IDESC = (1u << 4) | (TYPE << 7) | (TYPE << 10) | (1u << 16) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(tc::BM * CTAS >> 4) << 24);
  static_assert(NB % 64 == 0 && 4 * BN * BUFS == 1024 && SMEM_BYTES <= 232448, "tile");
};

template <int CTAS>
__device__ __forceinline__ uint32_t leader_addr(const void *p) {  // the same place in the shared memory of the pair's first CTA
  uint32_t a = tc::smem_u32(p);
  if (CTAS == 2) asm("mapa.shared::cluster.u32 %0, %0, 0;" : "+r"(a));
  return a;
}
// Load into this CTA's shared memory; the bytes are counted by the barrier at `bar`, the leader's.
template <int CTAS>
__device__ __forceinline__ void load(void *dst, const CUtensorMap *map, uint32_t bar, int x, int y, int z) {
  if (CTAS == 2)
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(tc::smem_u32(dst)), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z)
        : "memory");
  else
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(tc::smem_u32(dst)), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z)
        : "memory");
}
template <int CTAS>
__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
  if (CTAS == 2)
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
                 "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate)
                 : "memory");
  else
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
                 "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate)
                 : "memory");
}
// Arrives at `bar` of every CTA of the pair once the MMAs issued so far have finished.
template <int CTAS>
__device__ __forceinline__ void commit(uint64_t *bar) {
  if (CTAS == 2)
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                     tc::smem_u32(bar)),
                 "h"((uint16_t)3)
                 : "memory");
  else
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tc::smem_u32(bar)) : "memory");
}
template <int CTAS>
__device__ __forceinline__ void arrive_leader(uint64_t *bar) {
  if (CTAS == 2)
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(leader_addr<2>(bar)) : "memory");
  else
    tc::mbar_arrive(bar);
}
template <int CTAS>
__device__ __forceinline__ void all_ctas_barrier() {
  if (CTAS == 2) {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  } else {
    __syncthreads();
  }
}
// K-major rows of 128 B (A): 8-row groups 1024 B apart.  MN-major (B): 64-column boxes BOX_BYTES apart, groups of 8 k-rows
// 1024 B apart.  Both with the 128-byte swizzle (layout type 2).
__device__ __forceinline__ uint64_t desc_a(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ uint64_t desc_b(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(BOX_BYTES >> 4) << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
// What the kernel in front wrote is read by ordinary loads (it may still run when this one starts), at this place.
__device__ __forceinline__ unsigned long long load_flag(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ float load_scale(const float *p) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void tmem_load16(uint32_t addr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(addr));
}
// Waits for this thread's loads from tensor memory; r is not touched before.
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                 "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])::"memory");
}

// Two parts, in shared memory, of 128 bytes a cycle: <2, 256> 43 written by TMA and 64 read by the tensor core, <2, 128> 64 and 96,
// <1, 128> 85 and 128.  The first is for many tiles; its accumulators fill tensor memory, so the sums are drained to registers
// (eight warps, 128 columns a thread) before the epilogue touches C, the mixed products first, because the next chain
// starts with those.  The others hold two tiles and give a small product more of them.  Three parts: <1, 128>, whose 24 MMAs a
// k block (32 cycles each) wait for 96 KB from L2.
//
// The tensor core truncates when it adds to its accumulator, an error that grows with the length of the chain (chain / 16
// additions, 2^-25 of the partial sum each on average); sh.chain of K are added there, the rest in registers, rounded.  For
// operands of one sign, or of so wide a range that few products make the sum, that is the largest error.  Chains of about 4.5 sqrt(K)
// keep it below the sequential sum's: in [0, 1) K = 777 1.5e-7 and 4.2e-7, 8351 5.9e-7 and 1.23e-6; lognormal entries (sigma 2) 0.4 of
// it in the median of 76 shapes, up to 1.5 where one element is the norm.  With 9 sqrt(K) 2.4e-7, 1.26e-6, 0.65 and up to 2.8; it
// costs 2 to 5 % more time (1000 x 1501 x 777 35.9 -> 36.7 us, 8191^3 5.6 -> 5.7 to 5.9 ms).
template <typename C_>
__global__ void __launch_bounds__(THREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, float *__restrict__ C, Shape sh,
                  Scratch w, PanelFlags flags, int tiles, bool vec, int *__restrict__ error_flag) {
  constexpr int PARTS = C_::PARTS, CTAS = C_::CTAS, BN = C_::BN, BUFS = C_::BUFS, NB = C_::NB, A_BYTES = C_::A_BYTES, B_BYTES = C_::B_BYTES,
                STAGE_BYTES = C_::STAGE_BYTES, STAGES = C_::STAGES, COLS = BN / 2;  // COLS: of an epilogue thread
  constexpr uint32_t IDESC = C_::IDESC;
  constexpr bool SUMS = C_::SUMS;
  const int chain = sh.chain / BK;  // k blocks
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + STAGES * STAGE_BYTES + 8 * TILE_BYTES);
  uint64_t *full = bars, *empty = bars + STAGES, *acc_full = bars + 2 * STAGES, *mixed_empty = acc_full + BUFS, *main_empty = mixed_empty + BUFS;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(main_empty + BUFS);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t rank = 0;
  if (CTAS == 2) asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int tm = (sh.M + tc::BM * CTAS - 1) / (tc::BM * CTAS), tn = (sh.N + BN - 1) / BN;
  const int unit0 = blockIdx.x / CTAS, units = gridDim.x / CTAS;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < BUFS; ++i) {
      tc::mbar_init(&acc_full[i], 1);
      tc::mbar_init(&mixed_empty[i], 8 * CTAS);
      tc::mbar_init(&main_empty[i], 8 * CTAS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    if (CTAS == 2) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(tc::smem_u32(tmem_slot)) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(tc::smem_u32(tmem_slot)) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  all_ctas_barrier<CTAS>();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  pdl_wait();

  // Nothing of the tile is computed here: every row panel or every column panel of it is left to the other kernel.
  auto skipped = [&](const tc::TileCoord &t, int s) {
    bool row_in = false, col_in = false;
#pragma unroll
    for (int i = 0; i < CTAS; ++i) {
      const int pa = t.m0 / 128 + i;
      if (pa < sh.panels_a) row_in |= load_flag(flags.row(t.batch, s) + pa) == 0;
    }
#pragma unroll
    for (int i = 0; i < BN / 128; ++i) {
      const int pb = t.n0 / 128 + i;
      if (pb < sh.panels_b) col_in |= load_flag(flags.col(t.batch, s) + pb) == 0;
    }
    return !(row_in && col_in);
  };
  // Three parts: the whole tile is left to the other kernel, which then adds all of K in the loop's order.  A mark of a later
  // group of stretches is met by the launch for that group.
  const int marks = w.flag_first + sh.stretches;
  auto left_out = [&](const tc::TileCoord &t) {
    unsigned long long any = 0;
#pragma unroll 4
    for (int s = 0; s < marks; ++s) any |= load_flag(flags.row(t.batch, s) + t.m0 / 128) | load_flag(flags.col(t.batch, s) + t.n0 / 128);
    return any != 0;
  };
  auto coord = [&](int t) { return tc::tile_coord(t, tm, tn, tc::BM * CTAS, BN); };
  bool ok = true;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      uint32_t g = 0;
      for (int t = unit0; t < tiles && ok; t += units) {
        const tc::TileCoord c = coord(t);
        if (PARTS == 3 && left_out(c)) continue;
        for (int s = 0; s < sh.stretches && ok; ++s) {
          if (PARTS == 2 && skipped(c, s)) continue;
          const int z = PARTS * (c.batch * sh.stretches + s), nk = (sh.length(s) + BK - 1) / BK;
          for (int kb = 0; kb < nk; ++kb, ++g) {
            const int st = g % STAGES;
            ok = tc::mbar_wait(&empty[st], ((g / STAGES) & 1) ^ 1);
            if (!ok) break;
            if (rank == 0) tc::mbar_expect_tx(&full[st], CTAS * STAGE_BYTES);
            const uint32_t bar = leader_addr<CTAS>(&full[st]);
            uint8_t *p = smem + st * STAGE_BYTES;
#pragma unroll
            for (int part = 0; part < PARTS; ++part) {
              load<CTAS>(p + part * A_BYTES, &map_a, bar, kb * BK, c.m0 + 128 * rank, z + part);
#pragma unroll
              for (int j = 0; j < NB / 64; ++j)
                load<CTAS>(p + PARTS * A_BYTES + part * B_BYTES + j * BOX_BYTES, &map_b, bar, c.n0 + NB * rank + 64 * j, kb * BK, z + part);
            }
          }
        }
      }
      if (!ok) atomicExch(error_flag, 5);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer: one thread of the pair ----------------
    if (lane == 0 && rank == 0) {
      uint32_t g = 0, it = 0;
      for (int t = unit0; t < tiles && ok; t += units) {
        const tc::TileCoord c = coord(t);
        if (PARTS == 3 && left_out(c)) continue;
        for (int s = 0; s < sh.stretches && ok; ++s) {
          if (PARTS == 2 && skipped(c, s)) continue;
          const int nk = (sh.length(s) + BK - 1) / BK;
          for (int kb = 0; kb < nk && ok; ++it) {  // chains
            const int end = nk - kb < chain ? nk : kb + chain;
            const uint32_t buf = it % BUFS, phase = (it / BUFS) & 1;
            const uint32_t d_main = tmem + buf * 2 * BN, d_mixed = d_main + BN;
            ok = tc::mbar_wait_cluster(&mixed_empty[buf], phase ^ 1);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (bool first = true; kb < end; ++kb, ++g, first = false) {
              const int st = g % STAGES;
              ok = tc::mbar_wait_cluster(&full[st], (g / STAGES) & 1);
              if (!ok) break;
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              const uint32_t p = tc::smem_u32(smem + st * STAGE_BYTES);
              uint64_t a[PARTS], b[PARTS];
#pragma unroll
              for (int q = 0; q < PARTS; ++q) {
                a[q] = desc_a(p + q * A_BYTES);
                b[q] = desc_b(p + PARTS * A_BYTES + q * B_BYTES);
              }
#pragma unroll
              for (int ks = 0; ks < BK / 16; ++ks) {  // 32 bytes of a row of A, two groups of 8 k-rows of B
                if (PARTS == 3) {
                  mma<CTAS>(d_mixed, a[0] + 2 * ks, b[PARTS - 1] + 128 * ks, IDESC, !first || ks > 0);
                  mma<CTAS>(d_mixed, a[PARTS - 1] + 2 * ks, b[0] + 128 * ks, IDESC, true);
                  mma<CTAS>(d_mixed, a[1] + 2 * ks, b[1] + 128 * ks, IDESC, true);
                }
                mma<CTAS>(d_mixed, a[0] + 2 * ks, b[1] + 128 * ks, IDESC, PARTS == 3 || !first || ks > 0);
                mma<CTAS>(d_mixed, a[1] + 2 * ks, b[0] + 128 * ks, IDESC, true);
              }
              if (first) {
                ok = tc::mbar_wait_cluster(&main_empty[buf], phase ^ 1);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              }
#pragma unroll
              for (int ks = 0; ks < BK / 16; ++ks) mma<CTAS>(d_main, a[0] + 2 * ks, b[0] + 128 * ks, IDESC, !first || ks > 0);
              commit<CTAS>(&empty[st]);
            }
            if (ok) commit<CTAS>(&acc_full[buf]);
          }
        }
      }
      if (!ok) atomicExch(error_flag, 6);
    }
  } else if (warp == 2) {
    // The kernel for the marked panels may start: at once where this CTA's tiles have no mark, so that it looks at the marks
    // beside this kernel; otherwise at the end, because blocks that come while SMs are taken are spread unevenly over them
    // (1000 x 1501 x 777, all panels marked: 180 us, 147 now).
    bool any = false;
    for (int t = unit0; t < tiles && !any; t += units) {
      const tc::TileCoord c = coord(t);
      for (int s = lane; s < marks; s += 32) {
        unsigned long long m = 0;
#pragma unroll
        for (int i = 0; i < CTAS; ++i)
          if (c.m0 / 128 + i < sh.panels_a) m |= load_flag(flags.row(c.batch, s) + c.m0 / 128 + i);
#pragma unroll
        for (int i = 0; i < BN / 128; ++i)
          if (c.n0 / 128 + i < sh.panels_b) m |= load_flag(flags.col(c.batch, s) + c.n0 / 128 + i);
        any |= m != 0;
      }
      any = __any_sync(0xffffffffu, any);
    }
    if (!any) pdl_release();
  } else if (warp >= 4) {
    // ---------------- epilogue ----------------
    constexpr float MIXED = PARTS == 2 ? LO_UNSCALE : 1.0f;  // weight of the mixed products
    constexpr int DEPTH = COLS == 128 ? 4 : 8;  // requests for C in flight: what the registers beside the sums allow
    const int q = warp & 3, half = (warp - 4) >> 2;  // lanes 32 q .. of tensor memory, columns COLS * half ..
    float *stile = reinterpret_cast<float *>(smem + STAGES * STAGE_BYTES) + (warp - 4) * 32 * 32;
    uint32_t it = 0;
    for (int t = unit0; t < tiles && ok; t += units) {
      const tc::TileCoord c = coord(t);
      const int m0 = c.m0 + 128 * rank, row0 = m0 + 32 * q, col0 = c.n0 + COLS * half;
      if (PARTS == 3) {
        bool any = false;
        for (int s = lane; s < marks; s += 32)
          any |= (load_flag(flags.row(c.batch, s) + m0 / 128) | load_flag(flags.col(c.batch, s) + c.n0 / 128)) != 0;
        if (__any_sync(0xffffffffu, any)) continue;
      }
      float4 *sums = SUMS ? reinterpret_cast<float4 *>(sh.sums) + ((int64_t)t * 8 + warp - 4) * COLS / 4 * 32 + lane : nullptr;
      uint32_t acc[COLS / 16][16];
      for (int s = 0; s < sh.stretches; ++s) {
        float fa = 1.0f, fb[COLS / 32];  // scales of this thread's row, of the columns 32 ch + lane
        bool mine = true;
        if (PARTS == 2) {
          // every load of this stretch at once: the marks, then the scales of this thread's row and columns
          const bool row_in = m0 / 128 < sh.panels_a, col_in = col0 / 128 < sh.panels_b;
          const int64_t at = (int64_t)c.batch * sh.stretches + s;
          const float *scale_a = w.scale_a + at * sh.M, *scale_b = w.scale_b + at * sh.Np;
          const unsigned long long mark_a = row_in ? load_flag(flags.row(c.batch, s) + m0 / 128) : 1;
          const unsigned long long mark_b = col_in ? load_flag(flags.col(c.batch, s) + col0 / 128) : 1;
          fa = row0 + lane < sh.M ? load_scale(scale_a + row0 + lane) : 0.0f;
#pragma unroll
          for (int ch = 0; ch < COLS / 32; ++ch) fb[ch] = col0 + 32 * ch + lane < sh.N ? load_scale(scale_b + col0 + 32 * ch + lane) : 0.0f;
          if (skipped(c, s)) continue;
          mine = (mark_a | mark_b) == 0;
        } else {
#pragma unroll
          for (int ch = 0; ch < COLS / 32; ++ch) fb[ch] = 1.0f;
        }
        if (SUMS && s == 0 && !sh.fresh)
          for (int i = lane & 7; i < COLS / 4; i += 8) asm volatile("prefetch.global.L2 [%0];" ::"l"(sums + 32 * i - lane + (lane & 24)));
        if (s == 0 && mine && (!SUMS || sh.last) && row0 + lane < sh.M) {  // C into L2 while the product is computed
          const float *p = C + ((int64_t)c.batch * sh.M + row0 + lane) * sh.ldn + col0;
          const int cols = sh.N - col0 < COLS ? sh.N - col0 : COLS;
          for (int i = 0; i < cols; i += 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + i));
          if (cols > 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + cols - 1));
        }
        for (int kb = 0, nk = (sh.length(s) + BK - 1) / BK; kb < nk; kb += chain, ++it) {
          const uint32_t buf = it % BUFS;
          ok = tc::mbar_wait(&acc_full[buf], (it / BUFS) & 1);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t addr = tmem + buf * 2 * BN + ((uint32_t)(32 * q) << 16) + COLS * half;
          if (kb == 0 && (PARTS == 2 || s == 0)) {
#pragma unroll
            for (int i = 0; i < COLS / 16; ++i) tmem_load16(addr + BN + 16 * i, acc[i]);
#pragma unroll
            for (int i = 0; i < COLS / 16; ++i) {
              tmem_wait(acc[i]);
#pragma unroll
              for (int j = 0; j < 16; ++j) acc[i][j] = __float_as_uint(__fmul_rn(__uint_as_float(acc[i][j]), MIXED));
            }
          } else {
#pragma unroll
            for (int i = 0; i < COLS / 16; ++i) {
              uint32_t r[16];
              tmem_load16(addr + BN + 16 * i, r);
              tmem_wait(r);
#pragma unroll
              for (int j = 0; j < 16; ++j)
                acc[i][j] = __float_as_uint(__fmaf_rn(__uint_as_float(r[j]), MIXED, __uint_as_float(acc[i][j])));
            }
          }
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) arrive_leader<CTAS>(&mixed_empty[buf]);
#pragma unroll
          for (int i = 0; i < COLS / 16; ++i) {
            uint32_t r[16];
            tmem_load16(addr + 16 * i, r);
            tmem_wait(r);
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[i][j] = __float_as_uint(__fadd_rn(__uint_as_float(acc[i][j]), __uint_as_float(r[j])));
          }
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) arrive_leader<CTAS>(&main_empty[buf]);
        }
        if (!ok) break;
        if (!mine) continue;
        if (PARTS == 3) {  // C is joined last and once
          if (s + 1 < sh.stretches) continue;
          if (SUMS && !sh.fresh) {
#pragma unroll
            for (int i = 0; i < COLS / 4; ++i) {
              const float4 v = sums[32 * i];
              uint32_t *a = &acc[i / 4][4 * (i & 3)];
              a[0] = __float_as_uint(__fadd_rn(v.x, __uint_as_float(a[0])));
              a[1] = __float_as_uint(__fadd_rn(v.y, __uint_as_float(a[1])));
              a[2] = __float_as_uint(__fadd_rn(v.z, __uint_as_float(a[2])));
              a[3] = __float_as_uint(__fadd_rn(v.w, __uint_as_float(a[3])));
            }
          }
          if (SUMS && !sh.last) {
#pragma unroll
            for (int i = 0; i < COLS / 4; ++i) {
              const uint32_t *a = &acc[i / 4][4 * (i & 3)];
              sums[32 * i] = make_float4(__uint_as_float(a[0]), __uint_as_float(a[1]), __uint_as_float(a[2]), __uint_as_float(a[3]));
            }
            continue;
          }
        }
        const int rows = sh.M - row0 < 32 ? sh.M - row0 : 32;
        const int64_t row4 = 4 * (int64_t)sh.ldn;
        // 32 columns at a time through shared memory (float4 slots rotated by the row: no bank conflicts), so that C is
        // accessed by rows
#pragma unroll
        for (int ch = 0; ch < COLS / 32; ++ch) {
          const int c0 = col0 + 32 * ch;
          float *cp = C + ((int64_t)c.batch * sh.M + row0) * sh.ldn + c0;
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint32_t *a = &acc[2 * ch + i / 4][4 * (i & 3)];
            *reinterpret_cast<float4 *>(stile + lane * 32 + 4 * (i ^ (lane & 7))) =
                make_float4(__fmul_rn(__uint_as_float(a[0]), fa), __fmul_rn(__uint_as_float(a[1]), fa), __fmul_rn(__uint_as_float(a[2]), fa),
                            __fmul_rn(__uint_as_float(a[3]), fa));
          }
          __syncwarp();
          if (vec) {
            const int qc = lane & 7, col = c0 + 4 * qc;
            const float4 f = make_float4(__shfl_sync(0xffffffffu, fb[ch], 4 * qc), __shfl_sync(0xffffffffu, fb[ch], 4 * qc + 1),
                                         __shfl_sync(0xffffffffu, fb[ch], 4 * qc + 2), __shfl_sync(0xffffffffu, fb[ch], 4 * qc + 3));
            if (col < sh.N) {
              int row = lane >> 3;
              float *p = cp + (int64_t)row * sh.ldn + 4 * qc;
#pragma unroll 1
              for (int pass = 0; pass < 8; pass += DEPTH) {
                float4 cin[DEPTH];
#pragma unroll
                for (int i = 0; i < DEPTH; ++i)
                  if (row + 4 * i < rows) cin[i] = *reinterpret_cast<const float4 *>(p + i * row4);
#pragma unroll
                for (int i = 0; i < DEPTH; ++i) {
                  const float4 a = *reinterpret_cast<const float4 *>(stile + (row + 4 * i) * 32 + 4 * (qc ^ ((row + 4 * i) & 7)));
                  if (row + 4 * i < rows)
                    *reinterpret_cast<float4 *>(p + i * row4) =
                        make_float4(__fadd_rn(__fmul_rn(a.x, f.x), cin[i].x), __fadd_rn(__fmul_rn(a.y, f.y), cin[i].y),
                                    __fadd_rn(__fmul_rn(a.z, f.z), cin[i].z), __fadd_rn(__fmul_rn(a.w, f.w), cin[i].w));
                }
                row += 4 * DEPTH;
                p += DEPTH * row4;
              }
            }
          } else if (c0 + lane < sh.N) {
            const float f = fb[ch];
            float *p = cp + lane;
#pragma unroll 1
            for (int row = 0; row < rows; row += 2 * DEPTH) {
              float cin[2 * DEPTH];
#pragma unroll
              for (int i = 0; i < 2 * DEPTH; ++i)
                if (row + i < rows) cin[i] = p[(int64_t)i * sh.ldn];
#pragma unroll
              for (int i = 0; i < 2 * DEPTH; ++i) {
                const float a = stile[(row + i) * 32 + 4 * ((lane >> 2) ^ (i & 7)) + (lane & 3)];  // row is a multiple of 8
                if (row + i < rows) p[(int64_t)i * sh.ldn] = __fadd_rn(__fmul_rn(a, f), cin[i]);
              }
              p += 2 * DEPTH * (int64_t)sh.ldn;
            }
          }
        }
      }
    }
    if (!ok) atomicExch(error_flag, 7);
  }

  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  all_ctas_barrier<CTAS>();  // neither CTA frees or leaves what the other still uses
  if (warp == 1) {
    if (CTAS == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
}

template <typename C_>
static int launch_gemm(const CUtensorMap &map_a, const CUtensorMap &map_b, float *C, const Shape &sh, const Scratch &w, const PanelFlags &flags,
                       int64_t tiles, bool vec, int *error_flag, int dev, cudaStream_t st) {
  static std::atomic<uint64_t> allowed{0};  // devices on which this kernel may use its shared memory
  if ((allowed.load(std::memory_order_relaxed) >> dev & 1) == 0) {
    LAPIS_CUDA_TRY(cudaFuncSetAttribute(gemm_split_kernel<C_>, cudaFuncAttributeMaxDynamicSharedMemorySize, C_::SMEM_BYTES));
    allowed.fetch_or(uint64_t(1) << dev, std::memory_order_relaxed);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(C_::CTAS * std::min<int64_t>(tiles, sm_count() / C_::CTAS)));
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = C_::SMEM_BYTES;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = C_::CTAS;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = C_::CTAS == 2 ? 2 : 1;
  LAPIS_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemm_split_kernel<C_>, map_a, map_b, C, sh, w, flags, (int)tiles, vec, error_flag));
  return LAPIS_OK;
}

// With PARTS = 2 or 3.
template <int PARTS>
static int launch_tiles(int64_t group_b, int64_t nb, const float *A, const float *B, float *C, const Shape &sh,
                        const Scratch &w, const PanelFlags &flags, int *error_flag, int dev, cudaStream_t st) {
  const int64_t M = sh.M, N = sh.N;
  const bool vec_a = sh.K % 4 == 0 && reinterpret_cast<uintptr_t>(A) % 16 == 0, vec_b = sh.ldn % 4 == 0 && reinterpret_cast<uintptr_t>(B) % 16 == 0;
  const bool vec_c = sh.ldn % 4 == 0 && reinterpret_cast<uintptr_t>(C) % 16 == 0;
  const dim3 grid((unsigned)(8 * (sh.panels_a + sh.panels_b)), (unsigned)sh.stretches, (unsigned)nb);
  auto kernel = vec_a ? (vec_b ? split_kernel<PARTS, true, true> : split_kernel<PARTS, true, false>)
                      : (vec_b ? split_kernel<PARTS, false, true> : split_kernel<PARTS, false, false>);
  LAPIS_CUDA_TRY(launch_pdl(kernel, grid, SPLIT_THREADS, 0, st, A, B, sh, w));
  CUtensorMap map_a, map_b;
  const int64_t parts = PARTS * nb * sh.stretches;
  const CUtensorMapDataType type = PARTS == 2 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  LAPIS_TRY(tc::make_map(&map_a, type, w.a, parts, M, sh.kc, 2 * (int64_t)sh.kc, tc::BM, BK, CU_TENSOR_MAP_SWIZZLE_128B));
  LAPIS_TRY(tc::make_map(&map_b, type, w.b, parts, sh.kc, sh.Np, 2 * (int64_t)sh.Np, BK, 64, CU_TENSOR_MAP_SWIZZLE_128B));
  auto count = [&](int64_t rows, int64_t cols) { return ((M + rows - 1) / rows) * ((N + cols - 1) / cols); };
  if (PARTS == 3)  // six products of what a CTA loads: pairs, which load half of B each, are no faster (1000 x 1501 x 777 36.8, single 35.7 us)
    return sh.sums != nullptr ? launch_gemm<Config<3, 1, 128, true>>(map_a, map_b, C, sh, w, flags, nb * count(128, 128), vec_c, error_flag, dev, st)
                              : launch_gemm<Config<3, 1, 128>>(map_a, map_b, C, sh, w, flags, nb * count(128, 128), vec_c, error_flag, dev, st);
  // rounds of tiles that the busiest SM works through, by what one takes
  const int64_t sms = sm_count();
  auto cost = [&](int64_t n, int64_t at_once, int64_t each) { return (n * group_b + at_once - 1) / at_once * each; };
  const int64_t wide = cost(count(256, 256), sms / 2, 128), pair = cost(count(256, 128), sms / 2, 80), single = cost(count(128, 128), sms, 107);
  if (wide < pair && wide < single)
    return launch_gemm<Config<2, 2, 256>>(map_a, map_b, C, sh, w, flags, nb * count(256, 256), vec_c, error_flag, dev, st);
  if (pair < single) return launch_gemm<Config<2, 2, 128>>(map_a, map_b, C, sh, w, flags, nb * count(256, 128), vec_c, error_flag, dev, st);
  return launch_gemm<Config<2, 1, 128>>(map_a, map_b, C, sh, w, flags, nb * count(128, 128), vec_c, error_flag, dev, st);
}

}  // namespace split

int bgemm_unsplit_stretches(int64_t batch, int64_t M, int64_t N, int64_t K, const float *A, const float *B, float *C, const PanelFlags &flags,
                            int first, cudaStream_t st);
int bgemm_unsplit_panels(int64_t batch, int64_t M, int64_t N, int64_t K, const float *A, const float *B, float *C, const PanelFlags &flags,
                         cudaStream_t st);

constexpr size_t SPLIT_BYTES = size_t(160) << 20;

// *done: false where the caller has to use another kernel (no memory for the split operands).
//
// What does not fit into SPLIT_BYTES is worked on in groups of stretches of K.  Whole tiles add each group to C, as the kernel
// that they replaced adds its segments.  Three parts keep the sums of the groups aside, so that C is joined last and once, as
// in the loop (with |C| near 1000 and K = 8000 an addition for every 1024 of K had 2.8 times the loop's error), and take C in
// blocks whose sums leave at least a third of SPLIT_BYTES to the operands, which are split again for every block beside theirs:
// 8191^3 5.38 -> 5.59 ms, in four blocks; 2100 x 2099 x 8000 425 -> 407 us; 70,000 x 321 x 1300 1165 -> 643, where shorter
// stretches had made room before.
int bgemm_split_launch(int64_t batch, int64_t M, int64_t N, int64_t K, const float *A, const float *B, float *C, bool exact_order,
                       bool *done, cudaStream_t st) {
  using namespace split;
  *done = false;
  int dev = 0;
  LAPIS_CUDA_TRY(cudaGetDevice(&dev));
  int *error_flag = bgemm_error_flag(dev);
  if (error_flag == nullptr) return LAPIS_ECUDA;

  auto panels = [](int64_t extent) { return (extent + 127) / 128; };
  auto padded = [](int64_t cols) { return (cols + GROUP_COLS - 1) / GROUP_COLS * GROUP_COLS; };
  const int parts = exact_order ? 3 : 2;
  Shape sh = {};
  sh.K = (int)K;
  sh.ldn = (int)N;
  sh.chain = exact_order ? std::min(KC, 64 * std::max(1, (int)(std::sqrt((double)K) / 14 + 0.5))) : KC;
  int64_t all = 0;  // stretches of K
  int64_t block_m = M, block_n = N;
  size_t sums = 0;  // bytes
  auto per = [&] {  // bytes of a stretch: parts, scales, flags
    return 2 * (size_t)parts * sh.kc * (block_m + padded(block_n)) + 4 * (size_t)(block_m + padded(block_n)) + 8 * (size_t)(panels(block_m) + panels(block_n));
  };
  for (int longest = KC; longest >= 64; longest /= 2) {
    all = (K + longest - 1) / longest;
    sh.kc = (int)(((K + all - 1) / all + 63) / 64 * 64);
    all = (K + sh.kc - 1) / sh.kc;
    if (parts == 3 || per() <= SPLIT_BYTES) break;
  }
  if (parts == 3 && per() * all > SPLIT_BYTES) {
    for (int64_t cm = 1, cn = 1;;) {
      block_m = cm == 1 ? M : 128 * panels((M + cm - 1) / cm);
      block_n = cn == 1 ? N : 128 * panels((N + cn - 1) / cn);
      sums = 4 * (size_t)(128 * panels(block_m)) * (size_t)(128 * panels(block_n));
      if (per() <= SPLIT_BYTES && sums <= SPLIT_BYTES - std::max(per(), SPLIT_BYTES / 3)) break;
      ++(block_m >= block_n ? cm : cn);
    }
  }
  if (per() > SPLIT_BYTES) return LAPIS_OK;
  const bool aside = sums != 0;
  const int64_t group_s = std::min<int64_t>({all, (int64_t)((SPLIT_BYTES - sums) / per()), 65535});
  const int64_t group_b = aside ? 1 : std::min<int64_t>({batch, std::max<int64_t>(1, SPLIT_BYTES / (per() * group_s)), 65535});
  const int64_t marks = parts == 3 ? all : group_s;  // stretches whose marks are kept
  size_t total = 0;
  auto take = [&](size_t bytes) {
    const size_t at = total;
    total = (total + bytes + 255) & ~size_t(255);
    return at;
  };
  const size_t n = (size_t)(group_s * group_b);
  const size_t off_a = take(n * 2 * parts * block_m * sh.kc), off_b = take(n * 2 * parts * sh.kc * padded(block_n)), off_sa = take(n * block_m * 4),
               off_sb = take(n * padded(block_n) * 4), off_fa = take((size_t)(marks * group_b) * 8 * panels(M)),
               off_fb = take((size_t)(marks * group_b) * 8 * panels(N)), off_sums = take(sums);
  // The pool is made by the first allocation, which belongs to no stream and may come while one is being captured.
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  LAPIS_CUDA_TRY(cudaThreadExchangeStreamCaptureMode(&mode));
  PoolBuf buf;
  const int allocated = buf.alloc(total, st);
  cudaThreadExchangeStreamCaptureMode(&mode);
  if (allocated != LAPIS_OK) {
    clear_error();
    return LAPIS_OK;
  }
  uint8_t *p = static_cast<uint8_t *>(buf.p);
  Scratch w = {reinterpret_cast<uint16_t *>(p + off_a), reinterpret_cast<uint16_t *>(p + off_b), reinterpret_cast<float *>(p + off_sa),
               reinterpret_cast<float *>(p + off_sb)};
  w.flag_panels_a = (int)panels(M);
  w.flag_panels_b = (int)panels(N);
  sh.sums = aside ? reinterpret_cast<float *>(p + off_sums) : nullptr;
  PanelFlags flags = {nullptr, nullptr, w.flag_panels_a, w.flag_panels_b, 0, sh.kc};
  for (int64_t b0 = 0; b0 < batch; b0 += group_b) {
    const int64_t nb = std::min(group_b, batch - b0);
    const float *Ab = A + b0 * M * K, *Bb = B + b0 * K * N;
    float *Cb = C + b0 * M * N;
    for (int64_t m0 = 0; m0 < M; m0 += block_m) {
      for (int64_t n0 = 0; n0 < N; n0 += block_n) {
        sh.M = (int)std::min(block_m, M - m0);
        sh.N = (int)std::min(block_n, N - n0);
        sh.Np = (int)padded(sh.N);
        sh.panels_a = (int)panels(sh.M);
        sh.panels_b = (int)panels(sh.N);
        for (int64_t s0 = 0; s0 < all; s0 += group_s) {
          sh.first = (int)s0;
          sh.stretches = (int)std::min(group_s, all - s0);
          sh.fresh = s0 == 0;
          sh.last = parts == 2 || s0 + group_s >= all;
          w.flag_a = p + off_fa + 8 * (m0 / 128);
          w.flag_b = p + off_fb + 8 * (n0 / 128);
          w.flag_stretches = flags.stretches = parts == 3 ? (int)all : sh.stretches;
          w.flag_first = parts == 3 ? (int)s0 : 0;
          flags.a = reinterpret_cast<const unsigned long long *>(w.flag_a);
          flags.b = reinterpret_cast<const unsigned long long *>(w.flag_b);
          const float *As = Ab + m0 * K, *Bs = Bb + n0;
          float *Cs = Cb + m0 * N + n0;
          LAPIS_TRY(parts == 2 ? launch_tiles<2>(group_b, nb, As, Bs, Cs, sh, w, flags, error_flag, dev, st)
                               : launch_tiles<3>(group_b, nb, As, Bs, Cs, sh, w, flags, error_flag, dev, st));
          if (parts == 2) LAPIS_TRY(bgemm_unsplit_stretches(nb, M, N, K, Ab, Bb, Cb, flags, (int)s0, st));
        }
      }
    }
    if (parts == 3) {
      flags.a = reinterpret_cast<const unsigned long long *>(p + off_fa);
      flags.b = reinterpret_cast<const unsigned long long *>(p + off_fb);
      LAPIS_TRY(bgemm_unsplit_panels(nb, M, N, K, Ab, Bb, Cb, flags, st));
    }
  }
  *done = true;
  return LAPIS_OK;
}

}  // namespace lapis_b200
