// Dense and batched fp32 matmul for sm_100a:  C[b] = C_in[b] + A[b] B[b].
//
// Replaces the loop nest the LAPIS pipeline makes of linalg.matmul /
// linalg.batch_matmul (tests/Dialect/Kokkos/linalg_to_loops_3.mlir.gold:6-20, from
// mlir/lib/Dialect/Kokkos/Transforms/DenseLinalgToParallelLoops.cpp:309-348): one
// output element per Kokkos thread, each reading a row of A and a strided column
// of B from global memory, no reuse.
//
// Three paths, chosen by shape and alignment:
//   * general shapes: a register-tiled kernel on the fp32 pipes that keeps the reference's arithmetic exactly -- k
//     ascending, separate multiply and add, C_in joined last -- so small and ragged problems (the 8x7x9 and 64x5x5
//     cases of examples/gemm_no_alloc.py and examples/batched_gemm_no_alloc.py) are bit-identical to the sequential
//     loop.
//   * tile-aligned shapes (M, N multiples of 128, K of 32): the tcgen05 kernel in gemm_tcgen05.cu, fp32 emulated with three
//     TF32 products.
//   * products of either kind that are large enough to pay for a pass over their operands first (split_pays): gemm_split.cu,
//     fp32 from three fp16 or six bf16 products.  What that split does not cover (infinities, NaN, elements 2^29 times smaller
//     than the largest of their row or column) is left to the other two, panel by panel.
#include <algorithm>
#include <cmath>

#include "tcgen05.h"

namespace lapis_b200 {

int bgemm_tcgen05_supported(int64_t batch, int64_t M, int64_t N, int64_t K);
int bgemm_tcgen05_launch(int64_t batch, int64_t M, int64_t N, int64_t K, const float *A, const float *B, float *C,
                         const PanelFlags &flags, int first, cudaStream_t st);
int bgemm_split_launch(int64_t batch, int64_t M, int64_t N, int64_t K, const float *A, const float *B, float *C, bool exact_order,
                       bool *done, cudaStream_t st);

// Two fp32 products / sums per instruction (sm_100), each rounded to nearest on its own: the bits of __fmul_rn and
// __fadd_rn.  The product is a fused multiply-add of -0, which changes no product, zeros included; the -0 pair comes
// from the host because the assembler turns a packed mul followed by a packed add into one fused operation.
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b, uint64_t minus_zero) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(minus_zero));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t pack2(float x, float y) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
  return d;
}
__device__ __forceinline__ void unpack2(uint64_t v, float &x, float &y) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}
// Copies 4 or 16 bytes to shared memory without passing through registers; `in` false: zeros, nothing is read.
template <int BYTES>
__device__ __forceinline__ void copy_async(float *dst, const float *src, bool in) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int n = in ? BYTES : 0;
  if (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

constexpr int SG_K = 16;      // k-slab per pipeline stage
constexpr int SG_STAGES = 3;  // slabs in shared memory

// Bound by the fp32 pipes: two instructions per two products, 36 TFLOP/s if nothing else issued.  The kernel before this
// one gave a thread 2 x 2 outputs, one shared-memory read for every product; 4 x 8 need three 16-byte reads for 32, slabs
// arrive by cp.async while the one before is used, and products and sums are packed in pairs.  Measured, before and
// now: 1000 x 1501 x 777 210 -> 142 us, 5000 x 3000 x 1999 4.62 -> 2.28 ms, 8191 x 8192 x 2047 20.8 -> 10.0 ms
// (27 TFLOP/s), 2000 problems of 60 x 70 x 33 106 -> 68 us, 4000 of 4 x 5 x 6 18.5 -> 12.4 us.  Where rows do not start on
// 16-byte boundaries the slabs travel in 4-byte copies (2000 x 2001 x 2002: 21 TFLOP/s).
//
// One block owns a BM x BN tile of C, a thread TM rows (BM / TM apart) by TN columns (groups of four, 4 BN / TN apart).
template <int BM, int BN, int TM, int TN, int MINB, bool MARKED>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), MINB)
bgemm_simt_kernel(int64_t batch, int64_t M, int64_t N, int64_t K, const float *__restrict__ A0,
                  const float *__restrict__ B0, float *__restrict__ C0, bool vec_a, bool vec_b, uint64_t minus_zero, PanelFlags flags) {
  constexpr int TX = BN / TN, TY = BM / TM, THREADS = TX * TY, PITCH = SG_K + 4;
  static_assert(TN % 4 == 0 && THREADS % 32 == 0 && THREADS >= BN / 4, "tile");
  __shared__ __align__(16) float sA[SG_STAGES][BM][PITCH];
  __shared__ __align__(16) float sB[SG_STAGES][SG_K][BN];
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const int64_t row0 = (int64_t)blockIdx.y * BM, col0 = (int64_t)blockIdx.x * BN;
  const int nslab = (int)((K + SG_K - 1) / SG_K);
  static_assert(128 % BM == 0 && 128 % BN == 0, "a tile lies in one panel of rows and one of columns");
  if (!MARKED) pdl_wait();
  for (int64_t b = blockIdx.z; b < batch; b += gridDim.z) {
    // MARKED: only what is marked in any stretch of K, over all of K.  The inputs and the marks were there before the kernel in
    // front let this one start, and that kernel leaves the marked elements of C alone.
    if (MARKED) {
      bool any = false;
      for (int s = tid; s < flags.stretches; s += THREADS) any |= (flags.row(b, s)[row0 / 128] | flags.col(b, s)[col0 / 128]) != 0;
      if (!__syncthreads_or(any)) continue;
    }
    const float *A = A0 + b * M * K;
    const float *B = B0 + b * K * N;
    float *C = C0 + b * M * N;
    auto load = [&](int slab) {
      if (slab < nslab) {
        const int st = slab % SG_STAGES;
        const int64_t k0 = (int64_t)slab * SG_K;
        if (vec_a) {
          constexpr int Q = SG_K / 4;
          const int c = 4 * (tid % Q);
#pragma unroll
          for (int i = 0; i < (BM * Q + THREADS - 1) / THREADS; ++i) {
            const int r = tid / Q + i * (THREADS / Q);
            const bool in = row0 + r < M && k0 + c < K;
            if (BM * Q % THREADS == 0 || r < BM) copy_async<16>(&sA[st][r][c], in ? A + (row0 + r) * K + k0 + c : A, in);
          }
        } else {
          const int c = tid % SG_K;
#pragma unroll
          for (int i = 0; i < BM * SG_K / THREADS; ++i) {
            const int r = tid / SG_K + i * (THREADS / SG_K);
            const bool in = row0 + r < M && k0 + c < K;
            copy_async<4>(&sA[st][r][c], in ? A + (row0 + r) * K + k0 + c : A, in);
          }
        }
        if (vec_b) {
          constexpr int Q = BN / 4;
          const int c = 4 * (tid % Q);
#pragma unroll
          for (int i = 0; i < (SG_K * Q + THREADS - 1) / THREADS; ++i) {
            const int r = tid / Q + i * (THREADS / Q);
            const bool in = k0 + r < K && col0 + c < N;
            if (SG_K * Q % THREADS == 0 || r < SG_K) copy_async<16>(&sB[st][r][c], in ? B + (k0 + r) * N + col0 + c : B, in);
          }
        } else {
#pragma unroll
          for (int i = 0; i < SG_K * BN / THREADS; ++i) {
            const int e = tid + i * THREADS, r = e / BN, c = e % BN;
            const bool in = k0 + r < K && col0 + c < N;
            copy_async<4>(&sB[st][r][c], in ? B + (k0 + r) * N + col0 + c : B, in);
          }
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    uint64_t acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0;
#pragma unroll
    for (int s = 0; s < SG_STAGES - 1; ++s) load(s);
    for (int slab = 0; slab < nslab; ++slab) {
      asm volatile("cp.async.wait_group %0;" ::"n"(SG_STAGES - 2) : "memory");
      __syncthreads();
      load(slab + SG_STAGES - 1);  // into the stage that every thread has left
      const int st = slab % SG_STAGES;
#pragma unroll
      for (int k4 = 0; k4 < SG_K; k4 += 4) {
        float4 a[TM];
#pragma unroll
        for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4 *>(&sA[st][ty + i * TY][k4]);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          ulonglong2 bb[TN / 4];
#pragma unroll
          for (int j = 0; j < TN / 4; ++j)
            bb[j] = *reinterpret_cast<const ulonglong2 *>(&sB[st][k4 + kk][4 * tx + 4 * TX * j]);
#pragma unroll
          for (int i = 0; i < TM; ++i) {
            const float av = kk == 0 ? a[i].x : kk == 1 ? a[i].y : kk == 2 ? a[i].z : a[i].w;
            const uint64_t aa = pack2(av, av);
#pragma unroll
            for (int j = 0; j < TN / 4; ++j) {
              acc[i][2 * j] = add2(acc[i][2 * j], mul2(aa, bb[j].x, minus_zero));
              acc[i][2 * j + 1] = add2(acc[i][2 * j + 1], mul2(aa, bb[j].y, minus_zero));
            }
          }
        }
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // the stages are free for the next problem
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int64_t gr = row0 + ty + i * TY;
      if (gr >= M) break;
#pragma unroll
      for (int j = 0; j < TN / 4; ++j) {
        const int64_t gc = col0 + 4 * tx + 4 * TX * j;
        float o[4];
        unpack2(acc[i][2 * j], o[0], o[1]);
        unpack2(acc[i][2 * j + 1], o[2], o[3]);
        float *c = C + gr * N + gc;
        if (vec_b) {
          if (gc < N) {
            const float4 cin = *reinterpret_cast<const float4 *>(c);
            *reinterpret_cast<float4 *>(c) =
                make_float4(__fadd_rn(o[0], cin.x), __fadd_rn(o[1], cin.y), __fadd_rn(o[2], cin.z), __fadd_rn(o[3], cin.w));
          }
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (gc + q < N) c[q] = __fadd_rn(o[q], c[q]);
        }
      }
    }
  }
  if (MARKED && (blockIdx.x | blockIdx.y | blockIdx.z) == 0) pdl_wait();  // what follows in the stream waits for both
}

template <int BM, int BN, int TM, int TN, int MINB>
static cudaError_t launch_simt(int64_t batch, int64_t M, int64_t N, int64_t K, const float *A, const float *B, float *C,
                               const PanelFlags &flags, cudaStream_t st) {
  const dim3 grid((unsigned)((N + BN - 1) / BN), (unsigned)((M + BM - 1) / BM), (unsigned)(batch < 65535 ? batch : 65535));
  const bool vec_a = K % 4 == 0 && reinterpret_cast<uintptr_t>(A) % 16 == 0;
  const bool vec_b = N % 4 == 0 && (reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C)) % 16 == 0;
  if (flags.a != nullptr)
    return launch_pdl(bgemm_simt_kernel<BM, BN, TM, TN, MINB, true>, grid, (BM / TM) * (BN / TN), 0, st, batch, M, N, K, A, B, C, vec_a, vec_b,
                      0x8000000080000000ull, flags);
  return launch_pdl(bgemm_simt_kernel<BM, BN, TM, TN, MINB, false>, grid, (BM / TM) * (BN / TN), 0, st, batch, M, N, K, A, B, C, vec_a, vec_b,
                    0x8000000080000000ull, flags);
}

// Tile by the time the busiest SM needs for a k-slab of its tiles: `slab` us each when it has several to overlap,
// `alone` us when it is bound by the latency of one (measured on 8191 x 8192 x 2047 and 35 x 37 x 8000).
struct GeneralTile {
  int bm, bn;
  float slab, alone;
  cudaError_t (*launch)(int64_t, int64_t, int64_t, int64_t, const float *, const float *, float *, const PanelFlags &, cudaStream_t);
};
static constexpr GeneralTile general_tiles[] = {{64, 64, 0.706f, 0.92f, launch_simt<64, 64, 4, 8, 4>},
                                                {64, 32, 0.403f, 0.55f, launch_simt<64, 32, 4, 4, 5>},
                                                {32, 64, 0.360f, 0.86f, launch_simt<32, 64, 4, 8, 8>},
                                                {32, 32, 0.220f, 0.60f, launch_simt<32, 32, 4, 4, 8>},
                                                {32, 32, 0.255f, 0.46f, launch_simt<32, 32, 2, 4, 6>}};
struct TileChoice {
  const GeneralTile *tile;
  float us, all;  // a k-slab: what the choice goes by; what the busiest SM takes, a few tiles overlapping only in part
};
static TileChoice general_tile(int64_t batch, int64_t M, int64_t N) {
  TileChoice best = {nullptr, 0.0f, 0.0f};
  for (const GeneralTile &t : general_tiles) {
    const int64_t count = batch * ((M + t.bm - 1) / t.bm) * ((N + t.bn - 1) / t.bn);
    const float most = (float)((count + sm_count() - 1) / sm_count()), us = std::max(t.alone, t.slab * most);
    if (best.tile == nullptr || us < best.us) best = {&t, us, t.alone + t.slab * (most - 1.0f)};
  }
  return best;
}

static int launch_general(int64_t batch, int64_t M, int64_t N, int64_t K, const float *A, const float *B, float *C, const PanelFlags &flags,
                          cudaStream_t st) {
  LAPIS_CUDA_TRY(general_tile(batch, M, N).tile->launch(batch, M, N, K, A, B, C, flags, st));
  return LAPIS_OK;
}

// the tensor-core kernel on fp32 operands moves them with TMA, which needs 16-byte aligned bases
static bool whole_tiles(int64_t batch, int64_t M, int64_t N, int64_t K, const float *A, const float *B, const float *C) {
  return (reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C)) % 16 == 0 &&
         bgemm_tcgen05_supported(batch, M, N, K);
}

// What a product from split operands leaves out.  Whole tiles: the marked panels of the group of stretches of K from `first`.
int bgemm_unsplit_stretches(int64_t batch, int64_t M, int64_t N, int64_t K, const float *A, const float *B, float *C, const PanelFlags &flags,
                            int first, cudaStream_t st) {
  return bgemm_tcgen05_launch(batch, M, N, K, A, B, C, flags, first, st);
}
// Other shapes: the panels that are marked in any stretch.
int bgemm_unsplit_panels(int64_t batch, int64_t M, int64_t N, int64_t K, const float *A, const float *B, float *C, const PanelFlags &flags,
                         cudaStream_t st) {
  return launch_general(batch, M, N, K, A, B, C, flags, st);
}

// Whether the product is left to gemm_split.cu: estimates of the time of both, in us, measured on one machine (split / other
// kernel).  Whole tiles, two parts: 8192^3 2700 / 5055, 2048^3 67 / 126, 1024^3 25 / 38, 128 x 128 x 1024 24 / 35; not for 512^3
// 20 / 21, 2048 x 2048 x 256 28 / 22, 64 of 256^3 60 / 22.  Other shapes, three parts: 1000 x 1501 x 777 36 / 142, 5000 x 3000 x
// 1999 310 / 2272, 129 x 4000 x 1000 35 / 100, 8191 x 8190 x 130 430 / 947, 100 problems of 200^3 74 / 97; not for 255 x 296 x
// 719 24.7 / 23.1, 227 x 96 x 1016 28.4 / 27.0, 291 x 247 x 968 34.8 / 32.9, 400 of 100 x 100 x 128 111 / 68, 300^3 19 / 12.
// Below K = 128 the chains in tensor memory would cost more precision than the sequential sum of the kernel for general shapes
// loses, and with fewer than 64 rows or columns most of a tile is padding.
//
// What the estimates cannot see are the values: operands of which the split covers nothing (a range above 2^29 in every 128
// rows or columns: graded matrices, exponentials) pay for the pass over them and for two more launches, 1000 x 1501 x 777 146.5
// us, which it takes alone as well, 1024^3 44.5 for 36.9, 4096^3 786 for 705, 100 of 200^3 153 for 103.
static bool split_pays(int64_t batch, int64_t M, int64_t N, int64_t K, bool tiles, bool vec_c) {
  if (M > (1 << 30) || N > (1 << 30) || K > (1 << 30) || batch * ((M + 127) / 128) * ((N + 127) / 128) >= (1ll << 31)) return false;
  if (M < 64 || N < 64 || (!tiles && K < 128)) return false;
  const double sms = sm_count(), depth = (double)K, problems = (double)batch;
  auto rounds = [&](int64_t rows, int64_t cols, double at_once) {
    return std::ceil(problems * (double)((M + rows - 1) / rows) * (double)((N + cols - 1) / cols) / at_once);
  };
  const double c = vec_c ? 1.0 : 2.0, operands = 8.0 * problems * depth * (double)(M + N);  // bytes of the parts, about
  if (!tiles) {
    // Launches; the pass over the operands, by bytes and by blocks of 16 rows or columns, two on an SM; rounds of tiles, by the
    // products or, where K is short, by the accesses to C.  Fitted to 700 shapes of 3e6 to 6e9 products: with it 4 of them take
    // the kernel that is slower by more than 3 % (at most 11 %), with the estimate for two parts 51 (up to 62 %).
    const double before = 4.0 + general_tile(batch, M, N).all * std::ceil(depth / SG_K);
    const double blocks = 8.0 * problems * (double)((M + 127) / 128 + (N + 127) / 128) * std::ceil(depth / 1024.0);
    const double now = 12.0 + 4.0 * (c - 1.0) + operands / 5.2e6 + 3.4 * blocks / (2.0 * sms) + rounds(128, 128, sms) * std::max(0.0163 * depth, 3.4 * c);
    return 1.1 * now < before;
  }
  const double wide = N % 256 == 0 ? rounds(128, 256, sms) : 1e30;
  double before = wide > 1 && wide < 1e30 ? wide * 0.0441 * depth : rounds(128, 128, sms) * 0.030 * depth;
  before = 5.0 + std::max(before, 4.0 * problems * (depth * (double)(M + N) + 2.0 * (double)M * (double)N) / 5.3e6);
  // a round of tiles: the MMAs, or the accesses to C where K is short
  const double product = std::min({rounds(256, 256, sms / 2) * std::max(0.0213 * depth, 12.0 * c), rounds(256, 128, sms / 2) * std::max(0.0133 * depth, 6.0 * c),
                                   rounds(128, 128, sms) * std::max(0.0178 * depth, 6.0 * c)});
  const double now = std::max(16.0, 8.0 + operands / 4.5e6 + product);
  return before > 20.0 && 1.15 * now < before;
}

}  // namespace lapis_b200

using namespace lapis_b200;

extern "C" int lapis_b200_bgemm_f32(int64_t batch, int64_t M, int64_t N, int64_t K, const float *d_A, const float *d_B,
                                    float *d_C, void *stream) {
  clear_error();
  if (batch < 0 || M < 0 || N < 0 || K < 0) return fail(LAPIS_EBADSHAPE, "bgemm: negative dimension");
  if (batch == 0 || M == 0 || N == 0) return LAPIS_OK;
  if (d_C == nullptr || (K > 0 && (d_A == nullptr || d_B == nullptr))) return fail(LAPIS_EBADARG, "bgemm: null operand");
  cudaStream_t st = as_stream(stream);
  const bool tiles = whole_tiles(batch, M, N, K, d_A, d_B, d_C);
  if (!tiles && (M + 31) / 32 > 65535) return fail(LAPIS_ETOOBIG, "bgemm: M too large for the general-shape kernel");
  if (split_pays(batch, M, N, K, tiles, N % 4 == 0 && reinterpret_cast<uintptr_t>(d_C) % 16 == 0)) {
    bool done = false;
    LAPIS_TRY(bgemm_split_launch(batch, M, N, K, d_A, d_B, d_C, !tiles, &done, st));
    if (done) return LAPIS_OK;
  }
  if (tiles) return bgemm_tcgen05_launch(batch, M, N, K, d_A, d_B, d_C, PanelFlags(), 0, st);
  return launch_general(batch, M, N, K, d_A, d_B, d_C, PanelFlags(), st);
}
