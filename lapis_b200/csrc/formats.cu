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
#include <algorithm>
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

// Rows with 16-byte accesses, for fibers whose length is a multiple of four (and 16-byte aligned arrays): a thread owns Q times
// four consecutive output elements, which lie in one fiber, so one float4 of the entry's values meets one float4 of the B row;
// with SAME the Q fours stand at the same place of their fibers and share the values.  Four stored entries are in flight per
// thread; the adds stay in entry order.  Where the rows of B come from L2 (bspmm_slice) the trips to L2 and the instructions
// bound it, about 25 for each entry and Q = 1, which is what Q = 2 is for; it also asks for the columns of the next entries
// while the current ones are added, without which a long row, a chain of trips, took longer than with Q = 1.  us with B whole
// and Q = 1, and now: 131,072 columns, rows of 32, 8 x 64 1136 -> 735 (DRAM 6.5 -> 1.9 GB); 40,000 of 20, 16 x 128 393 -> 293;
// 200,000 of 20, 4 x 40 477 -> 244; B in L2, 20,000 of 20, 8 x 32 97 -> 76, with rows of up to 4096 490 -> 420.
// Passing the columns of 32 entries round by shuffles, one trip to memory for them all, took 1.52 ms of the first, Q = 4 0.95.
template <typename I, int GROUP, int Q, bool SAME, bool SLICED>
__global__ void __launch_bounds__(BSPMM_THREADS, Q == 1 ? 10 : 8)
bspmm_csrv_vec4_kernel(const I *__restrict__ pos, const I *__restrict__ crd, const float4 *__restrict__ val4,
                       int64_t nrows, int nh4, int64_t E4, int64_t width4, const float4 *__restrict__ B4, float4 *__restrict__ C4,
                       int accumulate) {
  constexpr int QA = SAME ? 1 : Q;
  const int g = threadIdx.x % GROUP;
  const int64_t row = (int64_t)blockIdx.x * (BSPMM_THREADS / GROUP) + threadIdx.x / GROUP;
  if (row >= nrows) return;
  const int64_t lo = (int64_t)pos[row], hi = (int64_t)pos[row + 1];
  float4 *crow = C4 + row * E4;
  const int64_t first = SLICED ? (int64_t)blockIdx.y * width4 : 0, last = SLICED && first + width4 < E4 ? first + width4 : E4;
  for (int64_t f = first + g; f < last; f += GROUP * Q) {  // f: index of this thread's first float4 inside the row
    const float4 *vcol[QA];                // + j * nh4 selects the entry
    const float4 *bcol = B4 + f;           // + crd[j] * E4 selects the row of B
    bool in[Q];
    float4 acc[Q];
#pragma unroll
    for (int q = 0; q < QA; ++q) vcol[q] = val4 + ((f + q * GROUP) % nh4);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      in[q] = q == 0 || f + q * GROUP < last;
      acc[q] = accumulate && in[q] ? crow[f + q * GROUP] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    auto add = [&](const float4(&a)[QA], const float4(&b)[Q]) {
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const float4 &v = a[SAME ? 0 : q];
        acc[q].x = __fadd_rn(__fmul_rn(v.x, b[q].x), acc[q].x);
        acc[q].y = __fadd_rn(__fmul_rn(v.y, b[q].y), acc[q].y);
        acc[q].z = __fadd_rn(__fmul_rn(v.z, b[q].z), acc[q].z);
        acc[q].w = __fadd_rn(__fmul_rn(v.w, b[q].w), acc[q].w);
      }
    };
    auto fetch = [&](int64_t j, I c, float4(&a)[QA], float4(&b)[Q]) {
      const float4 *brow = bcol + (int64_t)c * E4;
#pragma unroll
      for (int q = 0; q < QA; ++q) a[q] = __ldg(vcol[q] + j * nh4);
#pragma unroll
      for (int q = 0; q < Q; ++q) b[q] = in[q] ? __ldg(brow + q * GROUP) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    };
    int64_t j = lo;
    if (Q == 1) {
      for (; j + 3 < hi; j += 4) {
        float4 a[4][QA], b[4][Q];
#pragma unroll
        for (int u = 0; u < 4; ++u) fetch(j + u, crd[j + u], a[u], b[u]);
#pragma unroll
        for (int u = 0; u < 4; ++u) add(a[u], b[u]);
      }
    } else {
      int c[4];  // a row of B has more than 48 floats here: its columns fit 31 bits
#pragma unroll
      for (int u = 0; u < 4; ++u) c[u] = j + 3 < hi ? (int)crd[j + u] : 0;
      for (; j + 3 < hi; j += 4) {
        float4 a[4][QA], b[4][Q];
#pragma unroll
        for (int u = 0; u < 4; ++u) fetch(j + u, c[u], a[u], b[u]);
#pragma unroll
        for (int u = 0; u < 4; ++u) c[u] = j + 7 < hi ? (int)crd[j + 4 + u] : 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) add(a[u], b[u]);
      }
    }
    for (; j < hi; ++j) {
      float4 a[QA], b[Q];
      fetch(j, crd[j], a, b);
      add(a, b);
    }
#pragma unroll
    for (int q = 0; q < Q; ++q)
      if (in[q]) crow[f + q * GROUP] = acc[q];
  }
}

__device__ __forceinline__ float madd(float a, float b, float c) { return __fadd_rn(__fmul_rn(a, b), c); }

// The same for fibers that are no multiple of four: G threads share one row; a thread owns Q groups of V neighbouring output
// elements, G groups apart, with U stored entries in flight; the adds stay in entry order.  V = 4: 16-byte accesses to B and
// C, the values of the elements' fibers one by one, or with FIBER4 (nh a multiple of four) also by 16 bytes: taken for rows of
// more than 256 elements whose fours share no values, where 40 registers and twelve blocks an SM keep more gathers in flight
// than bspmm_csrv_vec4_kernel (20,000 columns, rows of 20, 12 x 32: 100 us, 115 there).  Bound by the gathers of rows of B; G
// follows the row's length, so that short rows do not leave most of a warp idle (50,000 rows of 20, 4 elements each: 84 -> 17
// us; 200,000 rows of 8, 2 x 4: 155 -> 28), and wide accesses halve the requests (50,000 rows of 20, 1 x 64: 85 -> 48; 30,000 of
// 30, 11 x 40: 269 -> 235; 20,000 of 30, 15 x 128: 718 -> 676).  Whole rows have kernels without the bounds of a slice, which cost
// up to 10 % (130,000 columns, 7 x 32: 613 and 672 us).
template <typename I, int V, bool FIBER4, int G, int Q, bool SLICED>
__global__ void __launch_bounds__(BSPMM_THREADS, FIBER4 ? 12 : 6)
bspmm_csrv_group_kernel(const I *__restrict__ pos, const I *__restrict__ crd, const float *__restrict__ val, int64_t nrows,
                  int64_t nh, int64_t E, int64_t width, const float *__restrict__ B, float *__restrict__ C, int accumulate) {
  constexpr int U = V == 4 ? 4 : 8 / Q;
  const int g = threadIdx.x % G;
  const int64_t row = (int64_t)blockIdx.x * (BSPMM_THREADS / G) + threadIdx.x / G;
  if (row >= nrows) return;
  const int64_t lo = (int64_t)pos[row], hi = (int64_t)pos[row + 1];
  float *crow = C + row * E;
  const int64_t first = SLICED ? (int64_t)blockIdx.y * width : 0, last = SLICED && first + width < E ? first + width : E;
  for (int64_t e0 = first + (int64_t)g * V; e0 < last; e0 += G * Q * V) {
    bool in[Q];
    int64_t fiber[Q][FIBER4 ? 1 : V];
    alignas(16) float acc[Q][V];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int64_t e = e0 + q * G * V;
      in[q] = q == 0 || e < last;
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
    int c[U];  // sliced (fewer than 10^6 columns): of the next entries
    if (SLICED) {
#pragma unroll
      for (int u = 0; u < U; ++u) c[u] = j + U <= hi ? (int)crd[j + u] : 0;
    }
    for (; j + U <= hi; j += U) {
      alignas(16) float a[U][Q][V], b[U][Q][V];
#pragma unroll
      for (int u = 0; u < U; ++u) fetch(j + u, (int64_t)(SLICED ? c[u] : crd[j + u]), a[u], b[u]);
      if (SLICED) {
#pragma unroll
        for (int u = 0; u < U; ++u) c[u] = j + 2 * U <= hi ? (int)crd[j + U + u] : 0;
      }
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
  int64_t nrows, nh, E, width;  // width: elements of a row that one pass over the matrix takes
  const float *B;
  float *C;
  int accumulate;
};

// Elements of a row of B (E floats, n2 rows) that one pass over the matrix gathers: E, or 256, 128 and so on, not less than
// `least`.  A gather from L2 runs at 20 TB/s as long as what is gathered from stays under about 70 MB, from DRAM at 7 (measured
// with random rows of 256 and 512 bytes), so a larger B is taken in slices of at most 72 MB, the slice slowest: every slice is
// read from DRAM once, and only the entries of the matrix are read once a slice.  Wider slices gain nothing (16,000 columns, 8 x
// 192, which would allow 768: 131 us in slices of 256, 134 of 512, 131 of 384 with twice the passes).
static int64_t bspmm_slice(int64_t n2, int64_t E, int64_t least) {
  if (4.0 * (double)n2 * (double)E <= 96e6) return E;
  for (int64_t width = 256; width >= least; width /= 2)
    if (4.0 * (double)n2 * (double)width <= 72e6) return width < E && (E + width - 1) / width <= 65535 ? width : E;
  return E;
}
// Fibers of nh = 4 << i elements, by vec4 kernels; others always whole (their fours share no values, and the passes are bound by
// instructions: 27,000 columns, 12 x 75, whole 208 us, in slices 211 to 219).  Slices of 32 elements lose to B whole (400,000
// columns, 4 x 24, 318 and 273 us; 1,000,000, 8 x 8, which would need narrower ones still, 625 and 420), and so do slices
// that a fiber fills for more than a quarter, whose values are read again (150,000, 64 x 4, 438 and 274).  At most three slices of
// 64: the rows of the last one begin late, which shows where a row is long (262,144 columns, 4 x 64, rows of 10 and of up to 4096
// entries: whole 383 and 1437 us, in four slices 346 and 1830).
static int64_t bspmm_slice_fours(int64_t n2, int64_t E, int64_t nh) {
  const int64_t nh4 = nh / 4, width = bspmm_slice(n2, E, std::max<int64_t>(64, 4 * nh));
  return (nh4 & (nh4 - 1)) != 0 || (width == 64 && E > 192) ? E : width;
}
// Other fibers, values one by one: rows of up to 256 elements (60,000 columns, 11 x 80: 0.67 ms whole, 0.69 in two slices), that fill
// five sixths of their slices (500,000 columns, 2 x 26: 454 us whole, 516 in slices of 32), and with 64-bit indices fibers
// of three and more (400,000, 1 x 64: 243 whole, 260 in slices).  180,000 of 5 x 32 816 -> 585, 150,000 of 3 x 64 653 -> 440, 160,000
// of 11 x 16 763 -> 616, 300,000 of 6 x 16 545 -> 387; with rows of up to 4096 entries 0.97 to 1.17 times as fast as whole.
static int64_t bspmm_slice_ones(int64_t n2, int64_t E, int64_t nh, int idx_bytes) {
  if (E > 256 || (idx_bytes == 8 && nh < 3)) return E;
  const int64_t width = bspmm_slice(n2, E, 32);
  return 6 * E >= 5 * width * ((E + width - 1) / width) ? width : E;
}

template <typename I>
static dim3 bspmm_grid(const BspmmArgs<I> &m, int rows) {
  return dim3((unsigned)((m.nrows + rows - 1) / rows), (unsigned)((m.E + m.width - 1) / m.width));
}

template <typename I, int G, int Q, bool SAME, bool SLICED>
static void launch_bspmm_vec4(const BspmmArgs<I> &m, cudaStream_t st) {
  bspmm_csrv_vec4_kernel<I, G, Q, SAME, SLICED><<<bspmm_grid(m, BSPMM_THREADS / G), BSPMM_THREADS, 0, st>>>(
      m.pos, m.crd, reinterpret_cast<const float4 *>(m.val), m.nrows, (int)(m.nh / 4), m.E / 4, m.width / 4, reinterpret_cast<const float4 *>(m.B),
      reinterpret_cast<float4 *>(m.C), m.accumulate);
}
// Two fours a thread, for rows that fill the group twice.
template <typename I, int G>
static void launch_bspmm_vec4_twice(const BspmmArgs<I> &m, cudaStream_t st) {
  if (m.width < m.E) launch_bspmm_vec4<I, G, 2, true, true>(m, st);
  else launch_bspmm_vec4<I, G, 2, true, false>(m, st);
}

template <typename I, int V, bool FIBER4, int G, int Q>
static void launch_bspmm_group(const BspmmArgs<I> &m, cudaStream_t st) {
  const dim3 grid = bspmm_grid(m, BSPMM_THREADS / G);
  if constexpr (V == 4 && G <= 64)
    if (m.width < m.E) {
      bspmm_csrv_group_kernel<I, V, false, G, Q, true><<<grid, BSPMM_THREADS, 0, st>>>(m.pos, m.crd, m.val, m.nrows, m.nh, m.E, m.width, m.B, m.C, m.accumulate);
      return;
    }
  bspmm_csrv_group_kernel<I, V, FIBER4, G, Q, false><<<grid, BSPMM_THREADS, 0, st>>>(m.pos, m.crd, m.val, m.nrows, m.nh, m.E, m.width, m.B, m.C, m.accumulate);
}

template <typename I>
static void launch_bspmm(const BspmmArgs<I> &m, int64_t n2, cudaStream_t st) {
  const bool aligned = (reinterpret_cast<uintptr_t>(m.B) | reinterpret_cast<uintptr_t>(m.C)) % 16 == 0;
  if (aligned && m.nh % 4 == 0 && m.nh / 4 <= 0x7fffffff && reinterpret_cast<uintptr_t>(m.val) % 16 == 0) {
    const int64_t nh4 = m.nh / 4, E4 = m.E / 4;
    BspmmArgs<I> s = m;
    s.width = bspmm_slice_fours(n2, m.E, m.nh);
    const int64_t w4 = s.width / 4;
    auto same = [&](int64_t group) { return group % nh4 == 0; };
    if (E4 <= 4) launch_bspmm_vec4<I, 4, 1, true, false>(s, st);
    else if (E4 <= 8) launch_bspmm_vec4<I, 8, 1, true, false>(s, st);
    else if (w4 > 12 && w4 <= 16 && same(8)) launch_bspmm_vec4_twice<I, 8>(s, st);
    else if (w4 <= 16) launch_bspmm_vec4<I, 16, 1, true, false>(s, st);
    else if (w4 <= 32 && same(16)) launch_bspmm_vec4_twice<I, 16>(s, st);
    else if (w4 <= 32) launch_bspmm_vec4<I, 32, 1, true, false>(s, st);
    else if (w4 <= 64 && same(32)) launch_bspmm_vec4_twice<I, 32>(s, st);
    else if (w4 <= 64) launch_bspmm_vec4<I, 32, 2, false, false>(s, st);
    else if (same(64)) launch_bspmm_vec4_twice<I, 64>(s, st);
    else launch_bspmm_group<I, 4, true, 128, 1>(s, st);
    return;
  }
  const int64_t E = m.E;
  if (aligned && E % 4 == 0) {
    BspmmArgs<I> s = m;
    s.width = bspmm_slice_ones(n2, E, m.nh, sizeof(I));
    const int64_t w4 = s.width / 4;
    if (w4 <= 4) launch_bspmm_group<I, 4, false, 4, 1>(s, st);
    else if (w4 <= 8) launch_bspmm_group<I, 4, false, 8, 1>(s, st);
    else if (w4 <= 16) launch_bspmm_group<I, 4, false, 16, 1>(s, st);
    else if (w4 <= 32) launch_bspmm_group<I, 4, false, 32, 1>(s, st);
    else if (w4 <= 64) launch_bspmm_group<I, 4, false, 64, 1>(s, st);
    else launch_bspmm_group<I, 4, false, 128, 1>(s, st);
  } else if (E <= 8) launch_bspmm_group<I, 1, false, 8, 1>(m, st);
  else if (E <= 16) launch_bspmm_group<I, 1, false, 16, 1>(m, st);
  else if (E <= 32) launch_bspmm_group<I, 1, false, 32, 1>(m, st);
  else if (E <= 64) launch_bspmm_group<I, 1, false, 32, 2>(m, st);
  else if (E <= 128) launch_bspmm_group<I, 1, false, 32, 4>(m, st);
  else bspmm_csrv_kernel<I, 128, 4><<<(unsigned)m.nrows, BSPMM_THREADS, 0, st>>>(m.pos, m.crd, m.val, m.nrows, m.nh, m.E, m.B, m.C, m.accumulate);
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
    launch_bspmm<I>({static_cast<const I *>(d_pos), static_cast<const I *>(d_crd), d_val, n1, nh, E, E, d_B, d_C, accumulate}, n2, st);
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
