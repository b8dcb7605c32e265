// Jacobi-PCG on systems that fit one thread-block cluster: the whole solve in one launch.
//
// With two or three launches an iteration a system of a few thousand rows is bound by the launches, by the chain of a
// last-block tail in each, and by the tuner that picks the SpMV kernel first.  Here every thread keeps its rows of x, r and
// dinv in registers, p lives in the shared memory of the CTAs, a slice each, and the SpMV gathers it from there; the
// partial sums of a dot product are stored into every CTA's shared memory by the warps that made them and added in one
// fixed order by every warp after the cluster's barrier, so that all derive the same alpha, beta and stop test.  Three
// barriers of the cluster an iteration, no global memory but the matrix, which the L1 caches of the SMs in use hold up to
// about 200 KB each and L2 beyond.
//
// Bound by the chains of dependent additions and shuffles between the barriers.  5-point stencils, us an iteration, with
// 512 to 1024 threads a CTA and the totals left to one warp, and now, 32-bit indices (64-bit): 1024 rows 2.96 and 1.86 (2.25),
// 4096 rows 3.50 and 3.28 (3.32), 6400 rows 4.6 and 4.0 (4.2), 16,384 rows 6.1 and 5.4 (6.3); the passes of pcg.cu 18.
// With scattered columns by the gathers from the other CTAs' memory: 8000 rows of 9, 56,000 such gathers, 17.1 and 16.1 (15.5), of
// 11, 70,000, 20.9, passes 20 to 21.5.  The solve therefore counts them first.  Where there are more than one in eight a thread
// takes its rows one behind the other: side by side all wait for the longest of them, and rows of scattered matrices differ in
// length (8000 rows of 9 20.0 (22.9), 16,000 of 5 19.5 (20.6) instead of 15.2 (15.3)), where those of a stencil gain by the
// loads that are under way together (6400 rows 5.3 one behind the other); rows of up to four entries on average do, too, as long
// as a CTA has no more than 1024.  Where there are too many the system is left to the passes.
//
// One CTA on an SM is said to the compiler: without that it keeps to half of the registers, and the loads of a step wait for each
// other (3000 rows of 9 10.7 and 9.3, 900 of 9 4.3 and 3.9).
//
// The recurrences are those of pcg.cu (examples/pcg_solve.py:65-98 in the LAPIS project), element by element; a row of A p
// is added in entry order.  Results are identical from run to run; against the other passes they differ by the order of the
// dot products' sums.
#include <cstdint>

#include "common.h"
#include "pcg_fuse.h"

namespace lapis_b200 {

constexpr int SMALL_FAR = 60000;  // gathers from other CTAs' memory in an iteration, beyond which the passes are faster
constexpr int SMALL_SHARE = 8;    // one in so many entries far: a system with scattered columns
constexpr int SMALL_LEFT = 2;     // FL_DONE of a system that was left to the passes
constexpr int SMALL_BUDGET = 4096;  // iterations per launch (a few milliseconds): the host looks at the outcome in between

struct SmallSolve {
  const double *b, *dinv;
  double *x, *r, *p;  // r and p: kept from one launch of a solve to the next
  double *sc;
  long long *fl;
  double tol;
  unsigned long long maxiter;
  int n, nnz;
  bool first, count_far;
};

template <int CTAS>
__device__ __forceinline__ void small_barrier() {
  if (CTAS == 1) {
    __syncthreads();
  } else {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  }
}
__device__ __forceinline__ uint32_t small_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t small_remote(const double *p, uint32_t rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ double warp_total(double v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = __dadd_rn(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}

// CTAS x THREADS threads, R rows each.  Eight warps a CTA: with 32 the shuffles of the partial sums took longer than the work
// between them, and a total had to be formed by one warp and handed out behind another barrier, where eight can each form it
// (the same additions, so the same bits) together with alpha, beta and the stop test.
template <typename I, int CTAS, int THREADS, int R>
__global__ void __launch_bounds__(THREADS, 1)
pcg_small_kernel(const I *__restrict__ pos, const I *__restrict__ crd, const double *__restrict__ val, SmallSolve s) {
  constexpr int SLICE = THREADS * R, WARPS = THREADS / 32, PARTS = CTAS * WARPS;
  constexpr int STEP = R >= 4 && sizeof(I) == 4 ? 2 : 4;  // entries of each row requested together
  constexpr bool TWO_FORMS = CTAS > 1 && R >= 4;           // scattered columns: the rows one behind the other
  constexpr bool AHEAD = THREADS < 512 || sizeof(I) == 8;  // their columns asked for while the entries before are gathered
  static_assert(PARTS % 32 == 0 || 32 % PARTS == 0, "a warp adds whole rounds of parts, or has each of them in several lanes");
  __shared__ double s_p[SLICE];
  __shared__ double s_part[3][PARTS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t rank = CTAS == 1 ? 0 : small_rank();

  // this warp's part of a sum goes to every CTA; total() adds the parts after the barrier, in every warp alike
  auto send = [&](int which, double v) {
    const double t = warp_total(v);
    double *slot = &s_part[which][rank * WARPS + warp];
    if (CTAS == 1) {
      if (lane == 0) *slot = t;
    } else if (lane < CTAS) {
      asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(small_remote(slot, lane)), "d"(t) : "memory");
    }
  };
  auto total = [&](int which) {
    double t = 0.0;
    if (PARTS >= 32) {
#pragma unroll
      for (int q = 0; q < PARTS / 32; ++q) t = __dadd_rn(t, s_part[which][lane + 32 * q]);
    } else {
      t = s_part[which][lane % PARTS];
    }
#pragma unroll
    for (int off = (PARTS < 32 ? PARTS : 32) / 2; off > 0; off >>= 1) t = __dadd_rn(t, __shfl_xor_sync(0xffffffffu, t, off));
    return t;
  };
  auto gather = [&](I col) {
    const uint32_t c = min((uint32_t)col, (uint32_t)s.n - 1);  // a bad index stays inside the cluster's memory
    if (CTAS == 1) return s_p[c];
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(small_remote(s_p, c / SLICE) + 8 * (c % SLICE)));
    return v;
  };

  const I *c[R];
  const double *v[R];
  int len[R], longest = 0;
  double x[R], r[R], z[R], d[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int row = (int)rank * SLICE + tid + i * THREADS;
    const bool in = row < s.n;
    const int64_t lo = in ? (int64_t)pos[row] : 0;
    c[i] = crd + lo;
    v[i] = val + lo;
    len[i] = in ? (int)((int64_t)pos[row + 1] - lo) : 0;
    longest = max(longest, len[i]);
    d[i] = in ? s.dinv[row] : 0.0;
    r[i] = in ? (s.first ? s.b[row] : s.r[row]) : 0.0;
    x[i] = in && !s.first ? s.x[row] : 0.0;
    z[i] = __dmul_rn(r[i], d[i]);
    s_p[tid + i * THREADS] = in ? (s.first ? z[i] : s.p[row]) : 0.0;
  }
  bool scattered = false;
  if (TWO_FORMS || (CTAS > 1 && s.count_far)) {
    int far = 0;
#pragma unroll
    for (int i = 0; i < R; ++i)
      for (int j = 0; j < len[i]; ++j) far += (uint32_t)__ldg(c[i] + j) / SLICE != rank;
    small_barrier<CTAS>();  // every CTA of the cluster runs before its shared memory is written
    send(0, (double)far);
    small_barrier<CTAS>();
    const double all = total(0);
    if (s.count_far && all > SMALL_FAR) {  // in all CTAs alike; nothing of theirs is read or written any more
      if (rank == 0 && tid == 0) s.fl[FL_DONE] = SMALL_LEFT;
      return;
    }
    scattered = TWO_FORMS && SMALL_SHARE * all > (double)s.nnz && (SLICE > 1024 || s.nnz > 4 * s.n);
  }
  double initres = 0.0, rz = 0.0, relres = 0.0;
  unsigned long long iters = 0;
  bool done = false;
  if (s.first) {
    double rr = 0.0, rzp = 0.0;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      rr = __dadd_rn(rr, __dmul_rn(r[i], r[i]));
      rzp = __dadd_rn(rzp, __dmul_rn(r[i], z[i]));
    }
    small_barrier<CTAS>();  // every CTA of the cluster runs before its shared memory is written
    send(1, rr);
    send(2, rzp);
    small_barrier<CTAS>();
    initres = sqrt(total(1));
    rz = total(2);
  } else {
    initres = s.sc[SC_INITRES];
    rz = s.sc[SC_RZ];
    iters = (unsigned long long)s.fl[FL_ITERS];
  }
  small_barrier<CTAS>();

  for (int left = SMALL_BUDGET; left > 0 && !done; --left) {
    double ap[R], pap = 0.0;
#pragma unroll
    for (int i = 0; i < R; ++i) ap[i] = 0.0;
    if (TWO_FORMS && scattered) {
#pragma unroll
      for (int i = 0; i < R; ++i) {
        int col[4];
        if (AHEAD) {
#pragma unroll
          for (int u = 0; u < 4; ++u) col[u] = u < len[i] ? (int)__ldg(c[i] + u) : 0;
        }
        for (int j = 0; j < len[i]; j += 4) {
          double a[4], g[4];
          int next[4];
          if (!AHEAD) {
#pragma unroll
            for (int u = 0; u < 4; ++u) col[u] = j + u < len[i] ? (int)__ldg(c[i] + j + u) : 0;
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) a[u] = j + u < len[i] ? __ldg(v[i] + j + u) : 0.0;
#pragma unroll
          for (int u = 0; u < 4; ++u) g[u] = j + u < len[i] ? gather((I)col[u]) : 0.0;
          if (AHEAD) {
#pragma unroll
            for (int u = 0; u < 4; ++u) next[u] = j + 4 + u < len[i] ? (int)__ldg(c[i] + j + 4 + u) : 0;
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (j + u < len[i]) ap[i] = __dadd_rn(ap[i], __dmul_rn(a[u], g[u]));
            if (AHEAD) col[u] = next[u];
          }
        }
      }
    } else {
      for (int j = 0; j < longest; j += STEP) {  // the rows side by side, each in entry order
        double a[R][STEP], g[R][STEP];
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
          for (int u = 0; u < STEP; ++u) {
            const bool in = j + u < len[i];
            a[i][u] = in ? __ldg(v[i] + j + u) : 0.0;
            g[i][u] = in ? gather(__ldg(c[i] + j + u)) : 0.0;
          }
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
          for (int u = 0; u < STEP; ++u)
            if (j + u < len[i]) ap[i] = __dadd_rn(ap[i], __dmul_rn(a[i][u], g[i][u]));
      }
    }
#pragma unroll
    for (int i = 0; i < R; ++i)
      if ((int)rank * SLICE + tid + i * THREADS < s.n) pap = __dadd_rn(pap, __dmul_rn(ap[i], s_p[tid + i * THREADS]));
    send(0, pap);
    small_barrier<CTAS>();
    const double alpha = rz / total(0), malpha = -alpha;
    double rr = 0.0, rzp = 0.0;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      x[i] = __dadd_rn(__dmul_rn(x[i], 1.0), __dmul_rn(s_p[tid + i * THREADS], alpha));
      r[i] = __dadd_rn(__dmul_rn(r[i], 1.0), __dmul_rn(ap[i], malpha));
      z[i] = __dmul_rn(r[i], d[i]);
      if ((int)rank * SLICE + tid + i * THREADS < s.n) {  // a thread without a row adds nothing, not 0 * inf either
        rr = __dadd_rn(rr, __dmul_rn(r[i], r[i]));
        rzp = __dadd_rn(rzp, __dmul_rn(r[i], z[i]));
      }
    }
    send(1, rr);
    send(2, rzp);
    small_barrier<CTAS>();
    ++iters;
    const double rznew = total(2);
    const double beta = rznew / rz;
    relres = sqrt(total(1)) / initres;
    done = !(relres > s.tol && iters != s.maxiter);  // ordered compare: NaN stops the loop
    if (!done) {
      rz = rznew;
#pragma unroll
      for (int i = 0; i < R; ++i) {
        double *p = s_p + tid + i * THREADS;
        *p = __dadd_rn(__dmul_rn(z[i], 1.0), __dmul_rn(*p, beta));
      }
      small_barrier<CTAS>();
    }
  }
  if (CTAS > 1) small_barrier<CTAS>();  // no CTA leaves while its parts may still be read or written
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int row = (int)rank * SLICE + tid + i * THREADS;
    if (row < s.n) {
      s.x[row] = x[i];
      if (!done) {
        s.r[row] = r[i];
        s.p[row] = s_p[tid + i * THREADS];
      }
    }
  }
  if (rank == 0 && tid == 0) {
    s.sc[SC_INITRES] = initres;
    s.sc[SC_RZ] = rz;
    s.sc[SC_RELRES] = relres;
    s.fl[FL_ITERS] = (long long)iters;
    s.fl[FL_DONE] = done ? 1 : 0;
  }
}

template <typename I, int CTAS, int THREADS, int R>
static cudaError_t launch_small(const lapis_b200_csr *h, const SmallSolve &s, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CTAS);
  cfg.blockDim = dim3(THREADS);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CTAS;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = CTAS > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, pcg_small_kernel<I, CTAS, THREADS, R>, static_cast<const I *>(h->pos), static_cast<const I *>(h->crd),
                            h->val, s);
}

template <typename I>
static cudaError_t launch_small_size(const lapis_b200_csr *h, const SmallSolve &s, cudaStream_t st) {
  if (s.n <= 1024) return launch_small<I, 1, 256, 4>(h, s, st);
  if (s.n <= 4096) return launch_small<I, 8, 256, 2>(h, s, st);
  if (s.n <= 8192) return launch_small<I, 8, 256, 4>(h, s, st);
  return launch_small<I, 8, 512, 4>(h, s, st);  // 256 x 8: 6.9 us an iteration where this takes 5.3
}

// Only for handles on which spmv_fits_small_pcg() is true (at most 16384 rows).  *solved: false where the system is left
// to the passes.
int pcg_small(const lapis_b200_csr *h, const double *d_b, const double *d_dinv, double tol, uint64_t maxiter, double *d_x,
              uint64_t *iters, double *relres, bool *solved, cudaStream_t st) {
  const int64_t n = h->nrows;
  PoolBuf buf;
  LAPIS_TRY(buf.alloc((size_t)(16 + 2 * n) * sizeof(double), st));
  SmallSolve s = {};
  s.sc = static_cast<double *>(buf.p);
  s.fl = reinterpret_cast<long long *>(s.sc + SC_COUNT);
  s.r = s.sc + 16;
  s.p = s.r + n;
  s.b = d_b;
  s.dinv = d_dinv;
  s.x = d_x;
  s.tol = tol;
  s.maxiter = maxiter;
  s.n = (int)n;
  s.nnz = (int)h->nnz;  // at most 131,072 (spmv_fits_small_pcg)
  s.first = true;
  s.count_far = h->nnz > SMALL_FAR;
  const uint64_t limit = maxiter == 0 ? (1ull << 31) : maxiter;
  int done = 0;
  uint64_t it = 0;
  do {
    LAPIS_CUDA_TRY(h->idx_bytes == 4 ? launch_small_size<int32_t>(h, s, st) : launch_small_size<int64_t>(h, s, st));
    s.first = s.count_far = false;
    LAPIS_TRY(lapis_b200_pcg_status(s.sc, &done, &it, relres, st));
    *solved = done != SMALL_LEFT;
    if (!*solved) return LAPIS_OK;
  } while (!done && it < limit);
  if (iters) *iters = it;
  return LAPIS_OK;
}

}  // namespace lapis_b200
