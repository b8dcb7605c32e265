// Neighbouring sparse formats of the same front end: batched SpMM over a CSRV tensor and SpMM over a DCSR
// matrix.
//
// CSRV (examples/bspmm.py:14-52 in the LAPIS project): a 3-D tensor A[n1, n2, nh] stored as
// (dense, compressed, dense) -- a CSR pattern (pos, crd) whose stored entry j carries a fiber of nh values
// val[j*nh .. j*nh+nh).  out[n1, dh, nh] = sum_n2 A[n1, n2, nh] * B[n2, dh, nh], fp32, all batches share the
// pattern.  The emitted loop nest is rows -> stored entries -> dh -> nh with the two inner loops dense and
// parallel, so every output element is updated in place once per stored entry, in ascending entry order:
// out = a*b + out.  One thread owns an output element for the whole row here, which keeps that order.
//
// DCSR (examples/spmm_dcsr_opdsl.py:46-101, 137-160): the entry point is here, the kernel in spmm.cu.
#include <cstdint>

#include "common.h"

namespace lapis_b200 {

constexpr int BSPMM_THREADS = 128;

// Rows of more than 128 elements that no 16-byte access fits: GROUP threads share one row; each thread owns EPT output
// elements per pass, GROUP apart, so that B rows and C rows are read and written coalesced.
template <typename I, int GROUP, int EPT>
__global__ void __launch_bounds__(BSPMM_THREADS)
bspmm_csrv_kernel(const I *__restrict__ pos, const I *__restrict__ crd, const float *__restrict__ val, int64_t nrows,
                  int64_t nh, int64_t E, const float *__restrict__ B, float *__restrict__ C, int accumulate) {
  const int g = threadIdx.x % GROUP;
  const int64_t row = (int64_t)blockIdx.x * (BSPMM_THREADS / GROUP) + threadIdx.x / GROUP;
  if (row >= nrows) return;
  const int64_t lo = (int64_t)pos[row], hi = (int64_t)pos[row + 1];
  float *crow = C + row * E;
  for (int64_t e0 = 0; e0 < E; e0 += (int64_t)GROUP * EPT) {
    int64_t e[EPT];
    int fiber[EPT];
    float acc[EPT];
#pragma unroll
    for (int q = 0; q < EPT; ++q) {
      e[q] = e0 + g + (int64_t)q * GROUP;
      fiber[q] = (int)(e[q] % nh);
      acc[q] = (accumulate && e[q] < E) ? crow[e[q]] : 0.0f;
    }
    int64_t j = lo;
    for (; j + 1 < hi; j += 2) {  // two stored entries in flight; the adds stay in entry order
      const int64_t c0 = (int64_t)crd[j], c1 = (int64_t)crd[j + 1];
      float a0[EPT], b0[EPT], a1[EPT], b1[EPT];
#pragma unroll
      for (int q = 0; q < EPT; ++q) {
        const bool in = e[q] < E;
        a0[q] = in ? val[j * nh + fiber[q]] : 0.0f;
        b0[q] = in ? __ldg(B + c0 * E + e[q]) : 0.0f;
        a1[q] = in ? val[(j + 1) * nh + fiber[q]] : 0.0f;
        b1[q] = in ? __ldg(B + c1 * E + e[q]) : 0.0f;
      }
#pragma unroll
      for (int q = 0; q < EPT; ++q) {
        acc[q] = __fadd_rn(__fmul_rn(a0[q], b0[q]), acc[q]);
        acc[q] = __fadd_rn(__fmul_rn(a1[q], b1[q]), acc[q]);
      }
    }
    if (j < hi) {
      const int64_t c0 = (int64_t)crd[j];
#pragma unroll
      for (int q = 0; q < EPT; ++q)
        if (e[q] < E) acc[q] = __fadd_rn(__fmul_rn(val[j * nh + fiber[q]], __ldg(B + c0 * E + e[q])), acc[q]);
    }
#pragma unroll
    for (int q = 0; q < EPT; ++q)
      if (e[q] < E) crow[e[q]] = acc[q];
  }
}

// Rows of up to 256 elements with 16-byte accesses, for fibers whose length is a multiple of four (and 16-byte aligned
// arrays): a
// thread owns four consecutive output elements, which lie in one fiber, so one float4 of the entry's values
// meets one float4 of the B row.  Four stored entries are in flight per thread; the adds stay in entry order.
template <typename I, int GROUP>
__global__ void __launch_bounds__(BSPMM_THREADS)
bspmm_csrv_vec4_kernel(const I *__restrict__ pos, const I *__restrict__ crd, const float4 *__restrict__ val4,
                       int64_t nrows, int nh4, int64_t E4, const float4 *__restrict__ B4, float4 *__restrict__ C4,
                       int accumulate) {
  const int g = threadIdx.x % GROUP;
  const int64_t row = (int64_t)blockIdx.x * (BSPMM_THREADS / GROUP) + threadIdx.x / GROUP;
  if (row >= nrows) return;
  const int64_t lo = (int64_t)pos[row], hi = (int64_t)pos[row + 1];
  float4 *crow = C4 + row * E4;
  for (int64_t f = g; f < E4; f += GROUP) {  // f: index of this thread's float4 inside the row
    const float4 *vcol = val4 + (f % nh4);   // + j * nh4 selects the entry
    const float4 *bcol = B4 + f;             // + crd[j] * E4 selects the row of B
    float4 acc = accumulate ? crow[f] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    int64_t j = lo;
    for (; j + 3 < hi; j += 4) {
      float4 a[4], b[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t c = (int64_t)crd[j + u];
        a[u] = __ldg(vcol + (j + u) * nh4);
        b[u] = __ldg(bcol + c * E4);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        acc.x = __fadd_rn(__fmul_rn(a[u].x, b[u].x), acc.x);
        acc.y = __fadd_rn(__fmul_rn(a[u].y, b[u].y), acc.y);
        acc.z = __fadd_rn(__fmul_rn(a[u].z, b[u].z), acc.z);
        acc.w = __fadd_rn(__fmul_rn(a[u].w, b[u].w), acc.w);
      }
    }
    for (; j < hi; ++j) {
      const float4 a = __ldg(vcol + j * nh4), b = __ldg(bcol + (int64_t)crd[j] * E4);
      acc.x = __fadd_rn(__fmul_rn(a.x, b.x), acc.x);
      acc.y = __fadd_rn(__fmul_rn(a.y, b.y), acc.y);
      acc.z = __fadd_rn(__fmul_rn(a.z, b.z), acc.z);
      acc.w = __fadd_rn(__fmul_rn(a.w, b.w), acc.w);
    }
    crow[f] = acc;
  }
}

__device__ __forceinline__ float madd(float a, float b, float c) { return __fadd_rn(__fmul_rn(a, b), c); }

// The same for short rows and for fibers that are no multiple of four: G threads share one row; a thread owns Q groups of V
// neighbouring output elements, G groups apart, with U stored entries in flight; the adds stay in entry order.  V = 4:
// 16-byte accesses to B and C, the values of the elements' fibers one by one, or with FIBER4 (nh a multiple of four) also by
// 16 bytes: taken for rows of more than 256 elements, where 40 registers and twelve blocks an SM keep more gathers in
// flight than bspmm_csrv_vec4_kernel's 48 (131,072 rows of 32, 8 x 64: 1.29 -> 1.15 ms; 20,000 of 30, 16 x 128: 558 -> 487 us).  Bound by the gathers of
// rows of B; G follows the row's length, so that short rows do not leave most of a warp idle (50,000 rows of 20, 4 elements
// each: 84 -> 17 us; 200,000 rows of 8, 2 x 4: 155 -> 28), and wide accesses halve the requests (50,000 rows of 20, 1 x 64:
// 85 -> 48; 30,000 of 30, 11 x 40: 269 -> 235; 20,000 of 30, 15 x 128: 718 -> 676).
template <typename I, int V, bool FIBER4, int G, int Q>
__global__ void __launch_bounds__(BSPMM_THREADS, FIBER4 ? 12 : 6)
bspmm_csrv_group_kernel(const I *__restrict__ pos, const I *__restrict__ crd, const float *__restrict__ val, int64_t nrows,
                  int64_t nh, int64_t E, const float *__restrict__ B, float *__restrict__ C, int accumulate) {
  constexpr int U = V == 4 ? 4 : 8 / Q;
  const int g = threadIdx.x % G;
  const int64_t row = (int64_t)blockIdx.x * (BSPMM_THREADS / G) + threadIdx.x / G;
  if (row >= nrows) return;
  const int64_t lo = (int64_t)pos[row], hi = (int64_t)pos[row + 1];
  float *crow = C + row * E;
  for (int64_t e0 = (int64_t)g * V; e0 < E; e0 += G * Q * V) {
    bool in[Q];
    int64_t fiber[Q][FIBER4 ? 1 : V];
    alignas(16) float acc[Q][V];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int64_t e = e0 + q * G * V;
      in[q] = q == 0 || e < E;
      fiber[q][0] = e % nh;
#pragma unroll
      for (int i = 1; i < (FIBER4 ? 1 : V); ++i) fiber[q][i] = fiber[q][i - 1] + 1 == nh ? 0 : fiber[q][i - 1] + 1;
#pragma unroll
      for (int i = 0; i < V; ++i) acc[q][i] = 0.0f;
      if (accumulate && in[q]) {
        if (V == 4) *reinterpret_cast<float4 *>(acc[q]) = *reinterpret_cast<const float4 *>(crow + e);
        else acc[q][0] = crow[e];
      }
    }
    auto fetch = [&](int64_t j, int64_t c, float(&a)[Q][V], float(&b)[Q][V]) {
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const float *v = val + j * nh, *brow = B + c * E + e0 + q * G * V;
        if (FIBER4) *reinterpret_cast<float4 *>(a[q]) = __ldg(reinterpret_cast<const float4 *>(v + fiber[q][0]));
#pragma unroll
        for (int i = 0; i < V; ++i)
          if (!FIBER4) a[q][i] = Q == 1 || in[q] ? __ldg(v + fiber[q][i]) : 0.0f;
        if (V == 4) *reinterpret_cast<float4 *>(b[q]) = __ldg(reinterpret_cast<const float4 *>(brow));
        else b[q][0] = Q == 1 || in[q] ? __ldg(brow) : 0.0f;
      }
    };
    int64_t j = lo;
    for (; j + U <= hi; j += U) {
      alignas(16) float a[U][Q][V], b[U][Q][V];
#pragma unroll
      for (int u = 0; u < U; ++u) fetch(j + u, (int64_t)crd[j + u], a[u], b[u]);
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
          for (int i = 0; i < V; ++i) acc[q][i] = madd(a[u][q][i], b[u][q][i], acc[q][i]);
    }
    for (; j < hi; ++j) {
      alignas(16) float a[Q][V], b[Q][V];
      fetch(j, (int64_t)crd[j], a, b);
#pragma unroll
      for (int q = 0; q < Q; ++q)
#pragma unroll
        for (int i = 0; i < V; ++i) acc[q][i] = madd(a[q][i], b[q][i], acc[q][i]);
    }
#pragma unroll
    for (int q = 0; q < Q; ++q)
      if (in[q]) {
        float *c = crow + e0 + q * G * V;
        if (V == 4) *reinterpret_cast<float4 *>(c) = *reinterpret_cast<const float4 *>(acc[q]);
        else c[0] = acc[q][0];
      }
  }
}

template <typename I>
struct BspmmArgs {
  const I *pos, *crd;
  const float *val;
  int64_t nrows, nh, E;
  const float *B;
  float *C;
  int accumulate;
};

template <typename I, int G>
static void launch_bspmm_vec4(const BspmmArgs<I> &m, cudaStream_t st) {
  constexpr int ROWS = BSPMM_THREADS / G;
  bspmm_csrv_vec4_kernel<I, G><<<(unsigned)((m.nrows + ROWS - 1) / ROWS), BSPMM_THREADS, 0, st>>>(
      m.pos, m.crd, reinterpret_cast<const float4 *>(m.val), m.nrows, (int)(m.nh / 4), m.E / 4, reinterpret_cast<const float4 *>(m.B),
      reinterpret_cast<float4 *>(m.C), m.accumulate);
}

template <typename I, int V, bool FIBER4, int G, int Q>
static void launch_bspmm_group(const BspmmArgs<I> &m, cudaStream_t st) {
  constexpr int ROWS = BSPMM_THREADS / G;
  bspmm_csrv_group_kernel<I, V, FIBER4, G, Q><<<(unsigned)((m.nrows + ROWS - 1) / ROWS), BSPMM_THREADS, 0, st>>>(
      m.pos, m.crd, m.val, m.nrows, m.nh, m.E, m.B, m.C, m.accumulate);
}

template <typename I>
static void launch_bspmm(const BspmmArgs<I> &m, cudaStream_t st) {
  const bool aligned = (reinterpret_cast<uintptr_t>(m.B) | reinterpret_cast<uintptr_t>(m.C)) % 16 == 0;
  const int64_t E = m.E, E4 = m.E / 4;
  if (aligned && m.nh % 4 == 0 && m.nh / 4 <= 0x7fffffff && reinterpret_cast<uintptr_t>(m.val) % 16 == 0) {
    if (E4 <= 4) launch_bspmm_vec4<I, 4>(m, st);
    else if (E4 <= 8) launch_bspmm_vec4<I, 8>(m, st);
    else if (E4 <= 16) launch_bspmm_vec4<I, 16>(m, st);
    else if (E4 <= 32) launch_bspmm_vec4<I, 32>(m, st);
    else if (E4 <= 64) launch_bspmm_vec4<I, 64>(m, st);
    else launch_bspmm_group<I, 4, true, 128, 1>(m, st);
  } else if (aligned && E % 4 == 0) {
    if (E4 <= 4) launch_bspmm_group<I, 4, false, 4, 1>(m, st);
    else if (E4 <= 8) launch_bspmm_group<I, 4, false, 8, 1>(m, st);
    else if (E4 <= 16) launch_bspmm_group<I, 4, false, 16, 1>(m, st);
    else if (E4 <= 32) launch_bspmm_group<I, 4, false, 32, 1>(m, st);
    else if (E4 <= 64) launch_bspmm_group<I, 4, false, 64, 1>(m, st);
    else launch_bspmm_group<I, 4, false, 128, 1>(m, st);
  } else if (E <= 8) launch_bspmm_group<I, 1, false, 8, 1>(m, st);
  else if (E <= 16) launch_bspmm_group<I, 1, false, 16, 1>(m, st);
  else if (E <= 32) launch_bspmm_group<I, 1, false, 32, 1>(m, st);
  else if (E <= 64) launch_bspmm_group<I, 1, false, 32, 2>(m, st);
  else if (E <= 128) launch_bspmm_group<I, 1, false, 32, 4>(m, st);
  else
    bspmm_csrv_kernel<I, 128, 4><<<(unsigned)m.nrows, BSPMM_THREADS, 0, st>>>(m.pos, m.crd, m.val, m.nrows, m.nh, E, m.B, m.C, m.accumulate);
}

}  // namespace lapis_b200

using namespace lapis_b200;

extern "C" int lapis_b200_bspmm_csrv_f32(int idx_bytes, int64_t n1, int64_t n2, int64_t nh, int64_t dh, const void *d_pos,
                                         const void *d_crd, const float *d_val, const float *d_B, float *d_C,
                                         int accumulate, void *stream) {
  clear_error();
  if (idx_bytes != 4 && idx_bytes != 8) return fail(LAPIS_EBADARG, "bspmm: idx_bytes must be 4 or 8");
  if (n1 < 0 || n2 < 0 || nh < 0 || dh < 0) return fail(LAPIS_EBADSHAPE, "bspmm: negative dimension");
  if (n1 > 0x7fffffffLL * 4) return fail(LAPIS_ETOOBIG, "bspmm: too many rows for one launch");
  const int64_t E = dh * nh;
  if (n1 == 0 || E == 0) return LAPIS_OK;
  if (d_pos == nullptr || d_C == nullptr) return fail(LAPIS_EBADARG, "bspmm: null operand");
  cudaStream_t st = as_stream(stream);
  auto run = [&](auto index) {
    using I = decltype(index);
    launch_bspmm<I>({static_cast<const I *>(d_pos), static_cast<const I *>(d_crd), d_val, n1, nh, E, d_B, d_C, accumulate}, st);
  };
  if (idx_bytes == 4) run(int32_t());
  else run(int64_t());
  LAPIS_CUDA_TRY(cudaGetLastError());
  return LAPIS_OK;
}

extern "C" int lapis_b200_spmm_dcsr_f64(int idx_bytes, int64_t nrows, int64_t ncols, int64_t nstored, int64_t k,
                                        const void *d_i1, const void *d_p2, const void *d_i2, const double *d_val,
                                        const double *d_B, double *d_C, void *stream) {
  clear_error();
  if (idx_bytes != 4 && idx_bytes != 8) return fail(LAPIS_EBADARG, "spmm_dcsr: idx_bytes must be 4 or 8");
  if (nrows < 0 || ncols < 0 || nstored < 0 || k < 0)
    return fail(LAPIS_EBADSHAPE, "spmm_dcsr: bad dimensions");
  if (nstored == 0 || k == 0) return LAPIS_OK;
  if (d_i1 == nullptr || d_p2 == nullptr || d_C == nullptr) return fail(LAPIS_EBADARG, "spmm_dcsr: null operand");
  return spmm_launch(idx_bytes, d_i1, d_p2, d_i2, d_val, nstored, k, 0, -1, d_B, d_C, 1, as_stream(stream));
}
