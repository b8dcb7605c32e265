// SpMM with fp64 values for sm_100a: CSR  C = (accumulate ? C : 0) + A B,  DCSR  C[i1[r], :] += A[r, :] B.
//
// Every output element is summed by one lane in ascending entry order: the bits of the sequential row loop
// (examples/bspmm.py:15-23, spmm_dcsr_opdsl.py:132-135: only the row loop is parallel).  CSR sums from zero and joins
// C last; DCSR updates C in place (examples/spmm_dcsr_opdsl.py:46-101).
//
// A group of G lanes owns a row, each lane Q columns (of V doubles), with U entries of the row in flight.  Bound by the
// gathers of rows of B (DRAM where B is larger than L2, L2 otherwise); G follows k so that a narrow B does not leave
// most of a warp idle, and Q follows an odd k so that the entries of a row are read once for up to 128 columns.  With a
// whole warp per row and one entry in flight per lane at odd k, before: 142,060 rows of 21, k = 3, 172 us (DCSR 136),
// now 25; k = 6, 104 -> 32; 63,642 rows of 24, k = 33, 87 -> 63.  2^21 rows of 32, k = 64, is at DRAM bandwidth as it
// was: 5.1 to 5.3 ms before and now (33.9 GB).
//
// A row of 4096 entries walked U at a time is a chain of 4096 / U trips to memory, which outlasts everything else in a
// skewed matrix.  Such rows go to a kernel of their own that runs beside this one (spmm_long_kernel): 50,021 rows with
// a mean of 16 and rows up to 4096, k = 37, DCSR: 884 -> 218 to 283 us with the matrix drawn; 10,000 rows, mean 30,
// k = 128: 839 -> 235.
#include <algorithm>
#include <cstdint>

#include "common.h"

namespace lapis_b200 {

constexpr int SPMM_THREADS = 256;
constexpr int SPMM_LONG = 256;  // shorter rows never leave their group (a few dozen trips to memory)
constexpr int SPMM_LONG_THREADS = 512;
constexpr int SPMM_TILE = 2048;  // products per tile of a long row

template <int V>
struct Columns;
template <>
struct Columns<1> {
  using type = double;
};
template <>
struct Columns<2> {
  using type = double2;
};
// Loads that keep their place: the compiler otherwise mixes the gathers of a batch with the sums before them.
__device__ __forceinline__ double cols_load(const double *p) {
  double v;
  asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double2 cols_load(const double2 *p) {
  double2 v;
  asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ double cols_zero(double) { return 0.0; }
__device__ __forceinline__ double2 cols_zero(double2) { return make_double2(0.0, 0.0); }
__device__ __forceinline__ double cols_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double2 cols_add(double2 a, double2 b) { return make_double2(__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y)); }
__device__ __forceinline__ double cols_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double2 cols_mul(double a, double2 b) { return make_double2(__dmul_rn(a, b.x), __dmul_rn(a, b.y)); }

// Whether a row of len entries is left to spmm_long_kernel.  A group of lanes walks it in a chain of trips to memory, about
// 0.15 us an entry and 64 columns; it may last half as long as the whole product of nnz entries does (8 (k + 8) bytes an
// entry at 5 TB/s), and is then hidden by it.
__host__ __device__ __forceinline__ bool spmm_is_long(int64_t len, int64_t nnz, int64_t k) {
  return len > SPMM_LONG && len > nnz * (k + 8) / ((k + 63) / 64) >> 17;
}
template <typename I>
__device__ __forceinline__ bool spmm_is_long(int64_t len, const I *__restrict__ pos, int64_t nrows, int64_t k) {
  return len > SPMM_LONG && spmm_is_long(len, (int64_t)pos[nrows] - (int64_t)pos[0], k);
}

// The stored entries [lo, hi) of row r and the row of C it belongs to; false: nothing to do for r.
template <typename I, bool DCSR>
__device__ __forceinline__ bool spmm_row(const I *__restrict__ rowno, const I *__restrict__ pos, int64_t nrows, int64_t r,
                                         int64_t &lo, int64_t &hi, int64_t &out) {
  if (r >= nrows) return false;
  int64_t rend = r + 1;
  out = r;
  if (DCSR) {
    // a row number may be listed more than once; equal numbers are adjacent, the first of a run takes all of it
    const I no = rowno[r];
    if (r > 0 && rowno[r - 1] == no) return false;
    while (rend < nrows && rowno[rend] == no) ++rend;
    out = (int64_t)no;
  }
  lo = (int64_t)pos[r];
  hi = (int64_t)pos[rend];
  return true;
}

// rowno: null for CSR; the stored rows' numbers for DCSR.  kv: columns in units of V.  With LONG_ROWS the long rows are
// left to spmm_long_kernel, which this kernel overlaps: an extra block at its end waits for that kernel.
// Blocks per SM: 32-bit indices fit 40 registers without the compiler pulling the gathers of a batch apart (six blocks:
// 2^20 rows of 32, k = 64, 2.50 ms, without the bound 2.67); 64-bit ones need 48 (2^21 rows: 2 % slower with six).
template <typename I, bool DCSR, bool LONG_ROWS, int V, int G, int Q>
__global__ void __launch_bounds__(SPMM_THREADS, sizeof(I) == 8 ? 1 : 6)
spmm_kernel(const I *__restrict__ rowno, const I *__restrict__ pos, const I *__restrict__ crd, const double *__restrict__ val,
            int64_t nrows, int64_t kv, const typename Columns<V>::type *__restrict__ B, typename Columns<V>::type *__restrict__ C,
            int accumulate) {
  using T = typename Columns<V>::type;
  constexpr int U = (V == 1 ? 8 : 4) / Q < 2 ? 2 : (V == 1 ? 8 : 4) / Q;
  if (LONG_ROWS && blockIdx.x == gridDim.x - 1) {
    pdl_wait();
    return;
  }
  const int g = threadIdx.x % G;
  int64_t lo, hi, out;
  if (!spmm_row<I, DCSR>(rowno, pos, nrows, (int64_t)blockIdx.x * (SPMM_THREADS / G) + threadIdx.x / G, lo, hi, out)) return;
  if (LONG_ROWS && spmm_is_long(hi - lo, pos, nrows, kv * V)) return;
  T *crow = C + out * kv;
  for (int64_t c0 = g; c0 < kv; c0 += G * Q) {
    T acc[Q];
    bool in[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      in[q] = q == 0 || c0 + q * G < kv;
      acc[q] = cols_zero(T());
      if (DCSR && in[q]) acc[q] = crow[c0 + q * G];
    }
    int64_t j = lo;
#pragma unroll 1
    for (; j + U <= hi; j += U) {
      I ci[U];
      double a[U];
      T b[U][Q];
#pragma unroll
      for (int u = 0; u < U; ++u) ci[u] = crd[j + u];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        a[u] = __ldg(val + j + u);
        const T *brow = B + (int64_t)ci[u] * kv + c0;
#pragma unroll
        for (int q = 0; q < Q; ++q) b[u][q] = in[q] ? cols_load(brow + q * G) : cols_zero(T());
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int q = 0; q < Q; ++q) acc[q] = cols_add(acc[q], cols_mul(a[u], b[u][q]));
    }
#pragma unroll 1
    for (; j < hi; ++j) {
      const double a = __ldg(val + j);
      const T *brow = B + (int64_t)crd[j] * kv + c0;
#pragma unroll
      for (int q = 0; q < Q; ++q)
        if (in[q]) acc[q] = cols_add(acc[q], cols_mul(a, __ldg(brow + q * G)));
    }
#pragma unroll
    for (int q = 0; q < Q; ++q)
      if (in[q]) {
        if (!DCSR) {
          T cin = cols_zero(T());
          if (accumulate) cin = crow[c0 + q * G];
          acc[q] = cols_add(acc[q], cin);
        }
        crow[c0 + q * G] = acc[q];
      }
  }
}

// The long rows.  A block looks for them among its rows (eight neighbours, then the eight gridDim.x * 8 further on, so
// that neighbouring long rows meet different blocks) and walks each in tiles of SPMM_TILE products: all threads gather and
// multiply the next tile while the first `width` add the current one, a column each, in entry order out of shared
// memory.  Bound by one trip to memory per tile; at most one block per SM, so that half of the registers and most of L1
// stay with the kernel beside it.  blockIdx.y: panel of `width` <= 32 columns.
template <typename I, bool DCSR>
__global__ void __launch_bounds__(SPMM_LONG_THREADS, 2)
spmm_long_kernel(const I *__restrict__ rowno, const I *__restrict__ pos, const I *__restrict__ crd, const double *__restrict__ val,
                 int64_t nrows, int64_t k, int width, const double *__restrict__ B, double *__restrict__ C, int accumulate) {
  constexpr int PER = SPMM_TILE / SPMM_LONG_THREADS;
  __shared__ double s_prod[2][SPMM_TILE];
  __shared__ int64_t s_lo[SPMM_LONG_THREADS], s_hi[SPMM_LONG_THREADS], s_out[SPMM_LONG_THREADS];
  __shared__ int s_n;
  pdl_release();  // the kernel for the other rows shares nothing with this one but inputs
  const int tid = threadIdx.x;
  const int entries = SPMM_TILE / width;  // per tile
  int je[PER], ce[PER];  // this thread's products in a tile: entry and column
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    je[i] = (tid + i * SPMM_LONG_THREADS) / width;
    ce[i] = (tid + i * SPMM_LONG_THREADS) % width;
  }
  if (tid == 0) s_n = 0;
  __syncthreads();
  const int64_t turn = (int64_t)gridDim.x * SPMM_LONG_THREADS;
  for (int64_t r0 = 0; r0 < nrows; r0 += turn) {
    int64_t lo = 0, hi = 0, out = 0;
    const int64_t r = r0 + ((int64_t)(tid / 8) * gridDim.x + blockIdx.x) * 8 + tid % 8;
    const bool found = spmm_row<I, DCSR>(rowno, pos, nrows, r, lo, hi, out) && spmm_is_long(hi - lo, pos, nrows, k);
    if (found) {
      const int at = atomicAdd(&s_n, 1);  // the order of the list does not matter: rows are independent
      s_lo[at] = lo;
      s_hi[at] = hi;
      s_out[at] = out;
    }
    if (!__syncthreads_or(found)) continue;
    const int n = s_n;
    for (int q = 0; q < n; ++q) {
      const int64_t first = s_lo[q], last = s_hi[q];
      for (int64_t c0 = (int64_t)blockIdx.y * width; c0 < k; c0 += (int64_t)gridDim.y * width) {
        const int cols = k - c0 < width ? (int)(k - c0) : width;
        double *c = C + s_out[q] * k + c0 + tid;
        double acc = DCSR && tid < cols ? *c : 0.0;
        I ci[PER];
        double b[PER], a[PER];
        auto columns = [&](int64_t j0) {
#pragma unroll
          for (int i = 0; i < PER; ++i) ci[i] = je[i] < entries && ce[i] < cols && j0 + je[i] < last ? crd[j0 + je[i]] : (I)-1;
        };
        auto gather = [&](int64_t j0) {
#pragma unroll
          for (int i = 0; i < PER; ++i) {
            const bool there = ci[i] >= 0;
            a[i] = there ? __ldg(val + j0 + je[i]) : 0.0;
            b[i] = there ? __ldg(B + (int64_t)ci[i] * k + c0 + ce[i]) : 0.0;
          }
        };
        columns(first);
        gather(first);
        columns(first + entries);
        int buf = 0;
        for (int64_t j0 = first; j0 < last; j0 += entries, buf ^= 1) {
#pragma unroll
          for (int i = 0; i < PER; ++i) s_prod[buf][tid + i * SPMM_LONG_THREADS] = __dmul_rn(a[i], b[i]);
          __syncthreads();
          gather(j0 + entries);
          columns(j0 + 2 * entries);
          if (tid < cols) {
            const double *p = s_prod[buf] + tid;
            const int m = last - j0 < entries ? (int)(last - j0) : entries;
#pragma unroll 8
            for (int t = 0; t < m; ++t) acc = __dadd_rn(acc, p[t * width]);
          }
        }
        if (tid < cols) {
          if (!DCSR) acc = __dadd_rn(acc, accumulate ? *c : 0.0);
          *c = acc;
        }
        __syncthreads();  // the buffers are free
      }
    }
    if (tid == 0) s_n = 0;
    __syncthreads();
  }
}

template <typename I>
struct SpmmArgs {
  const I *rowno, *pos, *crd;
  const double *val;
  int64_t nrows, k;
  const double *B;
  double *C;
  int accumulate;
  bool long_rows;
};

template <typename I, bool DCSR, int V, int G, int Q>
static cudaError_t launch_spmm_as(const SpmmArgs<I> &m, cudaStream_t st) {
  using T = typename Columns<V>::type;
  constexpr int ROWS = SPMM_THREADS / G;
  const unsigned grid = (unsigned)((m.nrows + ROWS - 1) / ROWS);
  const T *B = reinterpret_cast<const T *>(m.B);
  T *C = reinterpret_cast<T *>(m.C);
  if constexpr (!DCSR)
    if (!m.long_rows) {
      spmm_kernel<I, false, false, V, G, Q><<<grid, SPMM_THREADS, 0, st>>>(m.rowno, m.pos, m.crd, m.val, m.nrows, m.k / V, B, C,
                                                                           m.accumulate);
      return cudaGetLastError();
    }
  return launch_pdl(spmm_kernel<I, DCSR, true, V, G, Q>, grid + 1, SPMM_THREADS, 0, st, m.rowno, m.pos, m.crd, m.val, m.nrows, m.k / V, B,
                    C, m.accumulate);
}

// Pairs keep one pair per lane and pass (Q = 2 and 3 measured 10 to 17 % slower at k = 66 and 96); single columns, which move
// half as much per request, take up to four.
template <typename I, bool DCSR, int V>
static cudaError_t launch_spmm_width(const SpmmArgs<I> &m, cudaStream_t st) {
  const int64_t kv = m.k / V;
  if (kv <= 2) return launch_spmm_as<I, DCSR, V, 2, 1>(m, st);
  if (kv <= 4) return launch_spmm_as<I, DCSR, V, 4, 1>(m, st);
  if (kv <= 8) return launch_spmm_as<I, DCSR, V, 8, 1>(m, st);
  if (kv <= 16) return launch_spmm_as<I, DCSR, V, 16, 1>(m, st);
  if (kv <= 32 || V == 2) return launch_spmm_as<I, DCSR, V, 32, 1>(m, st);
  if (kv <= 64) return launch_spmm_as<I, DCSR, 1, 32, 2>(m, st);
  return launch_spmm_as<I, DCSR, 1, 32, 4>(m, st);
}

template <typename I, bool DCSR>
static cudaError_t launch_spmm(const SpmmArgs<I> &m, cudaStream_t st) {
  if (m.long_rows) {
    const int64_t panels = (m.k + 31) / 32, chunks = (m.nrows + 7) / 8, py = std::min<int64_t>(panels, 8);
    const dim3 grid((unsigned)std::min<int64_t>(chunks, sm_count() / py), (unsigned)py);
    spmm_long_kernel<I, DCSR><<<grid, SPMM_LONG_THREADS, 0, st>>>(m.rowno, m.pos, m.crd, m.val, m.nrows, m.k,
                                                                  (int)((m.k + panels - 1) / panels), m.B, m.C, m.accumulate);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  // pairs of columns travel as 16-byte accesses when k is even and B and C are aligned for it
  const bool pairs = m.k % 2 == 0 && (reinterpret_cast<uintptr_t>(m.B) | reinterpret_cast<uintptr_t>(m.C)) % 16 == 0;
  return pairs ? launch_spmm_width<I, DCSR, 2>(m, st) : launch_spmm_width<I, DCSR, 1>(m, st);
}

int spmm_launch(int idx_bytes, const void *rowno, const void *pos, const void *crd, const double *val, int64_t nrows, int64_t k,
                int64_t nnz, int64_t max_row_len, const double *B, double *C, int accumulate, cudaStream_t st) {
  // nothing is known of the stored rows of a DCSR matrix
  const bool long_rows = rowno != nullptr || max_row_len < 0 || spmm_is_long(max_row_len, nnz, k);
  auto run = [&](auto index) {
    using I = decltype(index);
    const SpmmArgs<I> m = {static_cast<const I *>(rowno), static_cast<const I *>(pos), static_cast<const I *>(crd), val, nrows, k, B, C,
                           accumulate, long_rows};
    return rowno == nullptr ? launch_spmm<I, false>(m, st) : launch_spmm<I, true>(m, st);
  };
  LAPIS_CUDA_TRY(idx_bytes == 4 ? run(int32_t()) : run(int64_t()));
  return LAPIS_OK;
}

}  // namespace lapis_b200
