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
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdint>

#include "common.h"

namespace lapis_b200 {

constexpr int SPMM_THREADS = 256;
constexpr int SPMM_LONG = 256;  // shorter rows never leave their group (a few dozen trips to memory)
constexpr int SPMM_PANEL = 64;                     // columns of a row that a block takes at once
constexpr int SPMM_ADDERS = 2, SPMM_FEEDERS = 10;  // warps that add and warps that gather and multiply
constexpr int SPMM_LONG_THREADS = 32 * (SPMM_ADDERS + SPMM_FEEDERS);
constexpr int SPMM_PER = 4, SPMM_TILE = 32 * SPMM_FEEDERS * SPMM_PER;  // products of a feeder, of a tile
constexpr int SPMM_CLUSTER = 4;                       // blocks that share their long rows
constexpr int SPMM_LIST = SPMM_LONG_THREADS + 64;     // long rows that a block notes before it works on them
constexpr int SPMM_SHARED = 768;                      // pieces that a cluster divides among its blocks

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
// 0.15 us an entry and 64 columns; it may last a quarter as long as the whole product of nnz entries does (8 (k + 8) bytes an
// entry at 5 TB/s), and is then hidden by it, also where it comes late.
__host__ __device__ __forceinline__ bool spmm_is_long(int64_t len, int64_t nnz, int64_t k) {
  return len > SPMM_LONG && len < (1 << 30) && k < (1 << 30) && len > nnz * (k + 8) / ((k + 63) / 64) >> 18;
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

// Between the warps that feed and those that add, which meet at different places of the code, once a tile each: barrier 1 with a
// count, because __syncthreads() in one branch of an if is undefined even where the other branch has as many.
__device__ __forceinline__ void tile_barrier() { asm volatile("barrier.sync 1, %0;" ::"n"(SPMM_LONG_THREADS) : "memory"); }

// The long rows.  A block notes those among its rows (eight neighbours, then the eight gridDim.x * 8 further on, so that
// neighbouring long rows meet different blocks); at the end the blocks of a cluster divide what they noted, a piece being a row
// and up to 64 columns: by length, the longest first, 0 1 2 3 3 2 1 0 0 1 .. (too many pieces: each block keeps its own).
// A block works through its pieces in tiles of SPMM_TILE products: ten warps gather and multiply, two tiles ahead of the one
// they store, across the ends of pieces, and two warps add, a lane one column, in entry order out of shared memory.
// One tile ahead, one row on an SM, a barrier for both, and now: 50,021 rows, k = 37 264 -> 104 us; 40,000, k = 130 374 -> 252;
// 30,000 of 39, k = 100 476 -> 363; 200,000 of 30, k = 16 566 -> 274.
template <typename I, bool DCSR>
__global__ void __launch_bounds__(SPMM_LONG_THREADS, 2)  // registers: the kernel beside this one needs half of them
spmm_long_kernel(const I *__restrict__ rowno, const I *__restrict__ pos, const I *__restrict__ crd, const double *__restrict__ val,
                 int64_t nrows, int64_t k, const double *__restrict__ B, double *__restrict__ C, int accumulate) {
  namespace cg = cooperative_groups;
  __shared__ double s_prod[2][SPMM_TILE];
  __shared__ int64_t s_lo[SPMM_LIST], s_out[SPMM_LIST];  // noted rows
  __shared__ int s_len[SPMM_LIST];
  __shared__ int64_t w_lo[SPMM_LIST], w_out[SPMM_LIST];  // pieces of work
  __shared__ int w_len[SPMM_LIST], w_c0[SPMM_LIST], w_c1[SPMM_LIST];
  __shared__ int s_all[SPMM_SHARED];
  __shared__ int s_n, s_count;
  pdl_release();  // the kernel for the other rows shares nothing with this one but inputs
  cg::cluster_group cluster = cg::this_cluster();
  const int tid = threadIdx.x, feeder = tid - 32 * SPMM_ADDERS;  // negative: an adder
  const int64_t panels = (k + SPMM_PANEL - 1) / SPMM_PANEL;
  const int width = (int)((k + panels - 1) / panels), entries = SPMM_TILE / width;  // of a tile
  int je[SPMM_PER], ce[SPMM_PER];  // this feeder's products in a tile: entry (beyond any row: none) and column
#pragma unroll
  for (int i = 0; i < SPMM_PER; ++i) {
    const int at = feeder + 32 * SPMM_FEEDERS * i;
    je[i] = feeder >= 0 && at < entries * width ? at / width : 0x40000000;
    ce[i] = at - at / width * width;
  }
  if (tid == 0) s_n = 0;
  __syncthreads();
  const int64_t turn = (int64_t)gridDim.x * SPMM_LONG_THREADS;
  for (int64_t r0 = 0;;) {
    int noted = 0;
    for (; r0 < nrows && noted <= SPMM_LIST - SPMM_LONG_THREADS; r0 += turn) {
      int64_t lo = 0, hi = 0, out = 0;
      const int64_t r = r0 + ((int64_t)(tid / 8) * gridDim.x + blockIdx.x) * 8 + tid % 8;
      const bool found = spmm_row<I, DCSR>(rowno, pos, nrows, r, lo, hi, out) && spmm_is_long(hi - lo, pos, nrows, k);
      if (found) {
        const int at = atomicAdd(&s_n, 1);  // the order of the list does not matter: rows are independent
        s_lo[at] = lo;
        s_len[at] = (int)(hi - lo);
        s_out[at] = out;
      }
      noted += __syncthreads_count(found);
    }
    const bool end = r0 >= nrows;
    int n = 0;  // pieces
    bool shared = false;
    if (end) {
      if (tid == 0) s_count = 0;
      cluster.sync();
      int all = 0, begin[SPMM_CLUSTER + 1];
#pragma unroll
      for (int c = 0; c < SPMM_CLUSTER; ++c) {
        begin[c] = all;
        all += *cluster.map_shared_rank(&s_n, c);
      }
      begin[SPMM_CLUSTER] = all;
      shared = all * panels <= SPMM_SHARED;
      if (shared) {
        const int np = (int)panels, pieces = all * np;
        for (int u = tid; u < pieces; u += SPMM_LONG_THREADS) {
          const int row = u / np;
          int c = 0;
          while (row >= begin[c + 1]) ++c;
          s_all[u] = cluster.map_shared_rank(s_len, c)[row - begin[c]];
        }
        __syncthreads();
        for (int u = tid; u < pieces; u += SPMM_LONG_THREADS) {
          const int mine = s_all[u];
          int rank = 0;  // longer ones, and equal ones in front
          for (int v = 0; v < pieces; ++v) rank += s_all[v] > mine || (s_all[v] == mine && v < u);
          const int place = rank % (2 * SPMM_CLUSTER);
          if ((place < SPMM_CLUSTER ? place : 2 * SPMM_CLUSTER - 1 - place) != (int)cluster.block_rank()) continue;
          const int row = u / np, at = rank / SPMM_CLUSTER;  // its turn in this block
          int c = 0;
          while (row >= begin[c + 1]) ++c;
          w_lo[at] = cluster.map_shared_rank(s_lo, c)[row - begin[c]];
          w_out[at] = cluster.map_shared_rank(s_out, c)[row - begin[c]];
          w_len[at] = mine;
          w_c0[at] = (u - row * np) * width;
          w_c1[at] = min(w_c0[at] + width, (int)k);
          atomicAdd(&s_count, 1);
        }
      }
      cluster.sync();  // nobody reads another block's list any more
      n = shared ? s_count : 0;
    }
    if (!shared) {
      n = noted;
      for (int u = tid; u < n; u += SPMM_LONG_THREADS) {
        w_lo[u] = s_lo[u];
        w_out[u] = s_out[u];
        w_len[u] = s_len[u];
        w_c0[u] = 0;
        w_c1[u] = (int)k;
      }
      __syncthreads();
    }
    // a place in the sequence of tiles: piece, first column of the panel, first entry of the tile
    struct Place {
      int q, c0, j;
    };
    auto start = [&](int q) { return Place{q, q < n ? w_c0[q] : 0, 0}; };
    auto step = [&](Place &p) {  // true: the next tile belongs to another piece or panel
      p.j += entries;
      if (p.j < w_len[p.q]) return false;
      p.j = 0;
      p.c0 += width;
      if (p.c0 >= w_c1[p.q]) p = start(p.q + 1);
      return true;
    };
    if (feeder >= 0) {
      I ci[SPMM_PER];                                                 // columns of the tile that is gathered next
      double b0[SPMM_PER], a0[SPMM_PER], b1[SPMM_PER], a1[SPMM_PER];  // operands of the next two tiles
      Place cols = start(0), rows = start(0);
      auto columns = [&] {
        if (cols.q < n) {
          const int left = w_len[cols.q] - cols.j, wide = w_c1[cols.q] - cols.c0;
          const I *c = crd + w_lo[cols.q] + cols.j;
#pragma unroll
          for (int i = 0; i < SPMM_PER; ++i) ci[i] = je[i] < left && ce[i] < wide ? c[je[i]] : (I)-1;
          step(cols);
        } else {
#pragma unroll
          for (int i = 0; i < SPMM_PER; ++i) ci[i] = (I)-1;
        }
      };
      auto gather = [&](double(&b)[SPMM_PER], double(&a)[SPMM_PER]) {
        const bool more = rows.q < n;
        const double *v = val + (more ? w_lo[rows.q] + rows.j : 0), *Bc = B + rows.c0;
#pragma unroll
        for (int i = 0; i < SPMM_PER; ++i) {
          const bool there = ci[i] >= 0;
          a[i] = there ? __ldg(v + je[i]) : 0.0;
          b[i] = there ? cols_load(Bc + (int64_t)ci[i] * k + ce[i]) : 0.0;
        }
        if (more) step(rows);
      };
      auto store = [&](int buf, const double(&b)[SPMM_PER], const double(&a)[SPMM_PER]) {
#pragma unroll
        for (int i = 0; i < SPMM_PER; ++i) s_prod[buf][feeder + 32 * SPMM_FEEDERS * i] = __dmul_rn(a[i], b[i]);
      };
      columns();
      gather(b0, a0);
      columns();
      gather(b1, a1);
      columns();
      // a tile is stored while the one before is added; its buffer was left at the barrier behind that one's store
      for (Place p = start(0); p.q < n;) {
        store(0, b0, a0);
        gather(b0, a0);
        columns();
        tile_barrier();
        step(p);
        if (p.q >= n) break;
        store(1, b1, a1);
        gather(b1, a1);
        columns();
        tile_barrier();
        step(p);
      }
    } else {
      auto element = [&](const Place &p) { return C + w_out[p.q] * k + p.c0 + tid; };
      auto mine = [&](const Place &p) { return p.q < n && tid < width && p.c0 + tid < w_c1[p.q]; };
      const bool read = DCSR || accumulate;
      Place p = start(0);
      double next = mine(p) && read ? *element(p) : 0.0;  // of C, fetched a piece or panel ahead
      int buf = 0;
      while (p.q < n) {
        const bool in = mine(p);
        const double cin = next;
        double *c = in ? element(p) : nullptr;
        Place after = p;
        after.j = w_len[p.q];
        step(after);
        next = mine(after) && read ? *element(after) : 0.0;
        double acc = DCSR ? cin : 0.0;
        bool ended = false;
        while (!ended) {
          tile_barrier();
          const double *s = s_prod[buf] + (in ? tid : 0);
          const int left = w_len[p.q] - p.j, m = left < entries ? left : entries;
#pragma unroll 16
          for (int e = 0; e < m; ++e) acc = __dadd_rn(acc, s[e * width]);
          buf ^= 1;
          ended = step(p);
        }
        if (in) *c = DCSR ? acc : __dadd_rn(acc, cin);
      }
    }
    if (end) break;
    __syncthreads();
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
    const int64_t clusters = std::min<int64_t>((m.nrows + 8 * SPMM_CLUSTER - 1) / (8 * SPMM_CLUSTER), sm_count() / SPMM_CLUSTER);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(clusters * SPMM_CLUSTER));
    cfg.blockDim = dim3(SPMM_LONG_THREADS);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = SPMM_CLUSTER;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, spmm_long_kernel<I, DCSR>, m.rowno, m.pos, m.crd, m.val, m.nrows, m.k, m.B, m.C, m.accumulate);
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
