// Dense and batched fp32 matmul for sm_100a:  C[b] = C_in[b] + A[b] B[b].
//
// Replaces the loop nest the LAPIS pipeline makes of linalg.matmul /
// linalg.batch_matmul (tests/Dialect/Kokkos/linalg_to_loops_3.mlir.gold:6-20, from
// mlir/lib/Dialect/Kokkos/Transforms/DenseLinalgToParallelLoops.cpp:309-348): one
// output element per Kokkos thread, each reading a row of A and a strided column
// of B from global memory, no reuse.
//
// Two paths, chosen by shape only (no fallback between them at run time):
//   * general shapes: a register-tiled kernel on the fp32 pipes that keeps the reference's arithmetic exactly -- k
//     ascending, separate multiply and add, C_in joined last -- so small and ragged problems (the 8x7x9 and 64x5x5
//     cases of examples/gemm_no_alloc.py and examples/batched_gemm_no_alloc.py) are bit-identical to the sequential
//     loop.
//   * tile-aligned shapes (M, N multiples of 128, K of 32): the tcgen05 kernel in
//     gemm_tcgen05.cu, fp32 emulated with three TF32 products.
#include <algorithm>

#include "common.h"

namespace lapis_b200 {

int bgemm_tcgen05_supported(int64_t batch, int64_t M, int64_t N, int64_t K);
int bgemm_tcgen05_launch(int64_t batch, int64_t M, int64_t N, int64_t K, const float *A, const float *B, float *C,
                         cudaStream_t st);

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
template <int BM, int BN, int TM, int TN, int MINB>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), MINB)
bgemm_simt_kernel(int64_t batch, int64_t M, int64_t N, int64_t K, const float *__restrict__ A0,
                  const float *__restrict__ B0, float *__restrict__ C0, bool vec_a, bool vec_b, uint64_t minus_zero) {
  constexpr int TX = BN / TN, TY = BM / TM, THREADS = TX * TY, PITCH = SG_K + 4;
  static_assert(TN % 4 == 0 && THREADS % 32 == 0 && THREADS >= BN / 4, "tile");
  __shared__ __align__(16) float sA[SG_STAGES][BM][PITCH];
  __shared__ __align__(16) float sB[SG_STAGES][SG_K][BN];
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const int64_t row0 = (int64_t)blockIdx.y * BM, col0 = (int64_t)blockIdx.x * BN;
  const int nslab = (int)((K + SG_K - 1) / SG_K);
  for (int64_t b = blockIdx.z; b < batch; b += gridDim.z) {
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
}

template <int BM, int BN, int TM, int TN, int MINB>
static void launch_simt(int64_t batch, int64_t M, int64_t N, int64_t K, const float *A, const float *B, float *C, cudaStream_t st) {
  const dim3 grid((unsigned)((N + BN - 1) / BN), (unsigned)((M + BM - 1) / BM), (unsigned)(batch < 65535 ? batch : 65535));
  const bool vec_a = K % 4 == 0 && reinterpret_cast<uintptr_t>(A) % 16 == 0;
  const bool vec_b = N % 4 == 0 && (reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C)) % 16 == 0;
  bgemm_simt_kernel<BM, BN, TM, TN, MINB><<<grid, (BM / TM) * (BN / TN), 0, st>>>(batch, M, N, K, A, B, C, vec_a, vec_b,
                                                                                   0x8000000080000000ull);
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
  // the tensor-core kernel moves its operands with TMA, which needs 16-byte aligned bases; other pointers (a
  // slice of a larger tensor, say) take the general-shape kernel, which has no alignment rule
  const bool aligned = ((reinterpret_cast<uintptr_t>(d_A) | reinterpret_cast<uintptr_t>(d_B) | reinterpret_cast<uintptr_t>(d_C)) % 16) == 0;
  if (aligned && bgemm_tcgen05_supported(batch, M, N, K)) return bgemm_tcgen05_launch(batch, M, N, K, d_A, d_B, d_C, st);
  if ((M + 31) / 32 > 65535) return fail(LAPIS_ETOOBIG, "bgemm: M too large for the general-shape kernel");
  // Tile by the time the busiest SM needs for a k-slab of its tiles: `slab` us each when it has several to overlap,
  // `alone` us when it is bound by the latency of one (measured on 8191 x 8192 x 2047 and 35 x 37 x 8000).
  static constexpr struct {
    int bm, bn;
    float slab, alone;
    void (*launch)(int64_t, int64_t, int64_t, int64_t, const float *, const float *, float *, cudaStream_t);
  } tiles[] = {{64, 64, 0.706f, 0.92f, launch_simt<64, 64, 4, 8, 4>},
               {64, 32, 0.403f, 0.55f, launch_simt<64, 32, 4, 4, 5>},
               {32, 64, 0.360f, 0.86f, launch_simt<32, 64, 4, 8, 8>},
               {32, 32, 0.220f, 0.60f, launch_simt<32, 32, 4, 4, 8>},
               {32, 32, 0.255f, 0.46f, launch_simt<32, 32, 2, 4, 6>}};
  int best = 0;
  float best_us = 0.0f;
  for (int i = 0; i < 5; ++i) {
    const int64_t count = batch * ((M + tiles[i].bm - 1) / tiles[i].bm) * ((N + tiles[i].bn - 1) / tiles[i].bn);
    const float us = std::max(tiles[i].alone, tiles[i].slab * (float)((count + sm_count() - 1) / sm_count()));
    if (i == 0 || us < best_us) {
      best = i;
      best_us = us;
    }
  }
  tiles[best].launch(batch, M, N, K, d_A, d_B, d_C, st);
  LAPIS_CUDA_TRY(cudaGetLastError());
  return LAPIS_OK;
}
