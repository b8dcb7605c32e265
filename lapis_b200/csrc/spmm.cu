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
// a mean of 16 and rows up to 4096, k = 37, DCSR: 884 -> 102 us.
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
constexpr int SPMM_TEAM = 4;                          // blocks that share their long rows
constexpr int SPMM_LOOK = 4;                          // neighbouring rows that a thread looks at together
constexpr int64_t SPMM_TEAM_BYTES = 450000;           // offsets that a team looks through, for every eight columns
constexpr int SPMM_LIST = SPMM_LONG_THREADS + 64;     // long rows that a block notes before it works on them
constexpr int SPMM_SHARED = 768;                      // pieces that a team divides by length; a block alone: SPMM_LIST

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

// Which of the rows r .. r + 3 are long: what spmm_row finds, but with loads that do not wait for each other.
template <typename I, bool DCSR>
__device__ __forceinline__ unsigned spmm_long_among(const I *__restrict__ rowno, const I *__restrict__ pos, int64_t nrows, int64_t k, int64_t r) {
  I at[SPMM_LOOK + 1], no[SPMM_LOOK + 2];
#pragma unroll
  for (int i = 0; i <= SPMM_LOOK; ++i) at[i] = r + i <= nrows ? pos[r + i] : (I)0;
  if (DCSR) {
#pragma unroll
    for (int i = 0; i <= SPMM_LOOK + 1; ++i) no[i] = r + i > 0 && r + i <= nrows ? rowno[r + i - 1] : (I)-1;
  }
  unsigned found = 0;
#pragma unroll
  for (int i = 0; i < SPMM_LOOK; ++i) {
    if (r + i >= nrows || (DCSR && no[i] == no[i + 1])) continue;  // beyond the last, or not the first of its run
    int64_t lo = (int64_t)at[i], hi = (int64_t)at[i + 1], out;
    if (DCSR && no[i + 1] == no[i + 2]) spmm_row<I, DCSR>(rowno, pos, nrows, r + i, lo, hi, out);
    if (spmm_is_long(hi - lo, pos, nrows, k)) found |= 1u << i;
  }
  return found;
}

// The long rows.  The blocks of a team note those among the team's rows (eight neighbours, then the eight further on by eight
// for every team, so that neighbouring long rows meet different teams), all four alike, and divide them, a piece being a row
// and up to 64 columns: by length, the longest first, 0 1 2 3 3 2 1 0 0 1 .. (too many pieces: whole rows in turn).  That each
// block looks through four times as many rows costs less than an exchange: with one share of the rows for each block of a
// cluster, passed round through shared memory, products without long rows took 2 to 4 us longer, the launch of clusters and its
// barriers (10,844 stored rows of 25, k = 3, 12.3 us, now 8.3; 50,021 of 4, k = 37, 20.9 and 19.0).  It does so while a
// team's offsets are few beside the product's columns; otherwise blocks look at their own rows and share nothing: there are enough
// long rows for each (1,000,000 rows of 4, k = 2, 64 us in teams, 47 alone, 54 in clusters; with skewed lengths 1,500,000 of 8,
// k = 8, 722, 684 and 697; but 100,000 of 16, k = 8, 81, 117 and 79, 91,623 of 25, 64-bit, k = 153, 1103 and 1715).  Where a team has
// fewer pieces than blocks they are of 32 or 16 columns (3465 rows, five of them long, k = 64, 14.4 us once, 16.4, 12.3 now).
// A block works through its pieces in tiles of SPMM_TILE products: ten warps gather and multiply, two tiles ahead of the one
// they store, across the ends of pieces, and two warps add, a lane one column, in entry order out of shared memory.
// One tile ahead, one row on an SM, a barrier for both, and now: 50,021 rows of 16, k = 37 276 -> 102 us; 40,000 of 30, k = 130
// 635 -> 438; 30,000 of 39, k = 100 426 -> 267; 200,000 of 30, k = 16 400 -> 273; 20,000 of 10, k = 3 94 -> 33.
template <typename I, bool DCSR>
__global__ void __launch_bounds__(SPMM_LONG_THREADS, 2)  // registers: the kernel beside this one needs half of them
spmm_long_kernel(const I *__restrict__ rowno, const I *__restrict__ pos, const I *__restrict__ crd, const double *__restrict__ val,
                 int64_t nrows, int64_t k, int team, const double *__restrict__ B, double *__restrict__ C, int accumulate) {
  __shared__ double s_prod[2][SPMM_TILE];
  __shared__ int64_t s_lo[SPMM_LIST], s_out[SPMM_LIST];  // noted rows
  __shared__ int s_len[SPMM_LIST];
  __shared__ int64_t w_lo[SPMM_LIST], w_out[SPMM_LIST];  // pieces of work
  __shared__ int w_len[SPMM_LIST], w_c0[SPMM_LIST], w_c1[SPMM_LIST];
  __shared__ int s_before[SPMM_LONG_THREADS / 32 + 1];
  pdl_release();  // the kernel for the other rows shares nothing with this one but inputs
  const int tid = threadIdx.x, feeder = tid - 32 * SPMM_ADDERS;  // negative: an adder
  const int member = blockIdx.x % team;
  const int64_t teams = gridDim.x / team, turn = teams * SPMM_LONG_THREADS * SPMM_LOOK;
  const int64_t mine = ((int64_t)(tid / (8 / SPMM_LOOK)) * teams + blockIdx.x / team) * 8 + tid % (8 / SPMM_LOOK) * SPMM_LOOK;
  int seen = 0;  // rows of each thread's in this turn that are noted or worked on
  for (int64_t r0 = 0;;) {
    int noted = 0;
    for (bool room = true; room && r0 < nrows;) {
      const unsigned found = spmm_long_among<I, DCSR>(rowno, pos, nrows, k, r0 + mine);
      if (__syncthreads_or(found != 0)) {
        for (; seen < SPMM_LOOK; ++seen) {
          const bool one = found >> seen & 1;
          const int more = __syncthreads_count(one);
          room = noted + more <= SPMM_LIST;
          if (!room) break;
          if (more == 0) continue;
          // in the order of the threads, which is the same in every block of the team
          const unsigned votes = __ballot_sync(0xffffffffu, one);
          if (tid % 32 == 0) s_before[tid / 32] = __popc(votes);
          __syncthreads();
          if (one) {
            int at = noted + __popc(votes & ((1u << tid % 32) - 1));
            for (int q = 0; q < tid / 32; ++q) at += s_before[q];
            int64_t lo, hi, out;
            spmm_row<I, DCSR>(rowno, pos, nrows, r0 + mine + seen, lo, hi, out);
            s_lo[at] = lo;
            s_len[at] = (int)(hi - lo);
            s_out[at] = out;
          }
          noted += more;
        }
        if (!room) break;
      }
      seen = 0;
      r0 += turn;
    }
    const bool end = r0 >= nrows;
    if (end && noted == 0) return;
    __syncthreads();
    // pieces of this block: of up to 64 columns, or of up to 16 where the team has few rows, so that each block has one
    int64_t panels = (k + SPMM_PANEL - 1) / SPMM_PANEL;
    for (int most = SPMM_PANEL / 2; most >= 16 && noted * panels < team; most /= 2) panels = (k + most - 1) / most;
    const int width = (int)((k + panels - 1) / panels), entries = SPMM_TILE / width;  // of a tile
    int je[SPMM_PER], ce[SPMM_PER];  // this feeder's products in a tile: entry (beyond any row: none) and column
#pragma unroll
    for (int i = 0; i < SPMM_PER; ++i) {
      const int at = feeder + 32 * SPMM_FEEDERS * i;
      je[i] = feeder >= 0 && at < entries * width ? at / width : 0x40000000;
      ce[i] = at - at / width * width;
    }
    const bool by_length = noted * panels <= (team == 1 ? SPMM_LIST : SPMM_SHARED);
    const int np = by_length ? (int)panels : 1, pieces = noted * np;
    const int rounds = pieces / team, turned = by_length && rounds % 2 != 0 ? team - 1 - member : member;
    const int n = rounds + (turned < pieces % team ? 1 : 0);
    for (int u = tid; u < pieces; u += SPMM_LONG_THREADS) {
      const int row = u / np, len = s_len[row];
      int at;
      if (by_length) {
        int rank = 0;  // longer ones, and equal ones in front
        for (int v = 0; v < noted; ++v) rank += s_len[v] > len ? np : s_len[v] == len && v < row ? np : 0;
        rank += u - row * np;
        const int place = rank % (2 * team);
        if ((place < team ? place : 2 * team - 1 - place) != member) continue;
        at = rank / team;  // its turn in this block
      } else {
        if (u % team != member) continue;
        at = u / team;
      }
      w_lo[at] = s_lo[row];
      w_out[at] = s_out[row];
      w_len[at] = len;
      w_c0[at] = by_length ? (u - row * np) * width : 0;
      w_c1[at] = by_length ? min(w_c0[at] + width, (int)k) : (int)k;
    }
    __syncthreads();
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
    __syncthreads();  // the lists are free
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
    const int team = m.nrows * (int64_t)sizeof(I) <= SPMM_TEAM_BYTES * std::max<int64_t>(1, m.k / 8) ? SPMM_TEAM : 1;
    const int64_t teams = std::min<int64_t>((m.nrows + 8 * team - 1) / (8 * team), std::max(1, sm_count() / team));
    spmm_long_kernel<I, DCSR><<<(unsigned)(teams * team), SPMM_LONG_THREADS, 0, st>>>(m.rowno, m.pos, m.crd, m.val, m.nrows, m.k, team, m.B, m.C,
                                                                                     m.accumulate);
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
