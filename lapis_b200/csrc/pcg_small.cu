// Jacobi-PCG on systems that fit one thread-block cluster: the whole solve in one launch.
//
// With two or three launches an iteration a system of a few thousand rows is bound by the launches, by the chain of a
// last-block tail in each, and by the tuner that picks the SpMV kernel first.  Here every thread keeps its rows of x, r and
// dinv in registers, p lives in the shared memory of the CTAs, a slice each, and the SpMV gathers it from there; the
// partial sums of a dot product are stored into every CTA's shared memory by the warps that made them and added in one
// fixed order by the first warp of every CTA after the cluster's barrier, so that all CTAs derive the same alpha, beta and
// stop test (one warp, not all: the divisions of 32 warps take longer than the barrier they save).  Three barriers of the
// cluster an iteration, no global memory but the matrix, which the L1 caches of the SMs in use hold up to about 200 KB each
// and L2 beyond (1000 rows of 29, 64-bit indices, 460 KB on one SM: 17 us an iteration, 12.5 with 32-bit ones).
//
// Bound by the barriers (5-point stencils: 3.0 us an iteration at 1024 rows, 6.2 at 16,384; the passes of pcg.cu take 17 to
// 19) and, with scattered columns, by the gathers from the other CTAs' memory: 8000 rows of 11, 70,000 such
// gathers, 20.9 us, passes 21.5; 8000 of 15, 98,000 gathers, 29.2 and 22.5, where a band of the same size takes 8.1.  The
// solve therefore counts them first where there may be too many, and leaves the system to the passes.
//
// The recurrences are those of pcg.cu (examples/pcg_solve.py:65-98 in the LAPIS project), element by element; a row of A p
// is added in entry order.  Results are identical from run to run; against the other passes they differ by the order of the
// dot products' sums.
#include <cstdint>

#include "common.h"
#include "pcg_fuse.h"

namespace lapis_b200 {

constexpr int SMALL_FAR = 75000;  // gathers from other CTAs' memory in an iteration, beyond which the passes are faster
constexpr int SMALL_LEFT = 2;     // FL_DONE of a system that was left to the passes
constexpr int SMALL_BUDGET = 4096;  // iterations per launch (a few milliseconds): the host looks at the outcome in between

struct SmallSolve {
  const double *b, *dinv;
  double *x, *r, *p;  // r and p: kept from one launch of a solve to the next
  double *sc;
  long long *fl;
  double tol;
  unsigned long long maxiter;
  int n;
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

// CTAS x THREADS threads, R rows each.
template <typename I, int CTAS, int THREADS, int R>
__global__ void __launch_bounds__(THREADS)
pcg_small_kernel(const I *__restrict__ pos, const I *__restrict__ crd, const double *__restrict__ val, SmallSolve s) {
  constexpr int SLICE = THREADS * R, WARPS = THREADS / 32, PARTS = CTAS * WARPS;
  static_assert(PARTS % 32 == 0, "a warp adds whole rounds of parts");
  __shared__ double s_p[SLICE];
  __shared__ double s_part[3][PARTS];
  __shared__ double s_alpha, s_beta;
  __shared__ int s_done;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t rank = CTAS == 1 ? 0 : small_rank();

  // this warp's part of a sum goes to every CTA; total() adds the parts after the barrier
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
#pragma unroll
    for (int q = 0; q < PARTS / 32; ++q) t = __dadd_rn(t, s_part[which][lane + 32 * q]);
    return warp_total(t);
  };
  auto gather = [&](I col) {
    const uint32_t c = min((uint32_t)col, (uint32_t)s.n - 1);  // a bad index stays inside the cluster's memory
    if (CTAS == 1) return s_p[c];
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(small_remote(s_p, c / SLICE) + 8 * (c % SLICE)));
    return v;
  };

  int64_t lo[R];
  int len[R];
  double x[R], r[R], z[R], d[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int row = (int)rank * SLICE + tid + i * THREADS;
    const bool in = row < s.n;
    lo[i] = in ? (int64_t)pos[row] : 0;
    len[i] = in ? (int)((int64_t)pos[row + 1] - lo[i]) : 0;
    d[i] = in ? s.dinv[row] : 0.0;
    r[i] = in ? (s.first ? s.b[row] : s.r[row]) : 0.0;
    x[i] = in && !s.first ? s.x[row] : 0.0;
    z[i] = __dmul_rn(r[i], d[i]);
    s_p[tid + i * THREADS] = in ? (s.first ? z[i] : s.p[row]) : 0.0;
  }
  if (CTAS > 1 && s.count_far) {
    int far = 0;
#pragma unroll
    for (int i = 0; i < R; ++i)
      for (int j = 0; j < len[i]; ++j) far += (uint32_t)__ldg(crd + lo[i] + j) / SLICE != rank;
    small_barrier<CTAS>();  // every CTA of the cluster runs before its shared memory is written
    send(0, (double)far);
    small_barrier<CTAS>();
    if (warp == 0) s_done = total(0) > SMALL_FAR ? 1 : 0;
    __syncthreads();
    if (s_done != 0) {  // in all CTAs alike; nothing of theirs is read or written any more
      if (rank == 0 && tid == 0) s.fl[FL_DONE] = SMALL_LEFT;
      return;
    }
  }
  double initres = 0.0, rz = 0.0, relres = 0.0;  // of warp 0, as the sums are
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
    if (warp == 0) {
      initres = sqrt(total(1));
      rz = total(2);
    }
  } else {
    initres = s.sc[SC_INITRES];
    rz = s.sc[SC_RZ];
    iters = (unsigned long long)s.fl[FL_ITERS];
  }
  small_barrier<CTAS>();

  for (int left = SMALL_BUDGET; left > 0 && !done; --left) {
    double ap[R], pap = 0.0;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const I *c = crd + lo[i];
      const double *v = val + lo[i];
      double sum = 0.0;
      for (int j = 0; j < len[i]; j += 4) {
        double a[4], g[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const bool in = j + u < len[i];
          a[u] = in ? __ldg(v + j + u) : 0.0;
          g[u] = in ? gather(__ldg(c + j + u)) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (j + u < len[i]) sum = __dadd_rn(sum, __dmul_rn(a[u], g[u]));
      }
      ap[i] = sum;
      if ((int)rank * SLICE + tid + i * THREADS < s.n) pap = __dadd_rn(pap, __dmul_rn(sum, s_p[tid + i * THREADS]));
    }
    send(0, pap);
    small_barrier<CTAS>();
    if (warp == 0) s_alpha = rz / total(0);
    __syncthreads();
    const double alpha = s_alpha, malpha = -alpha;
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
    if (warp == 0) {
      relres = sqrt(total(1)) / initres;
      const double rznew = total(2);
      const bool stop = !(relres > s.tol && iters != s.maxiter);  // ordered compare: NaN stops the loop
      if (!stop) {
        s_beta = rznew / rz;
        rz = rznew;
      }
      s_done = stop ? 1 : 0;
    }
    __syncthreads();
    done = s_done != 0;
    if (!done) {
      const double beta = s_beta;
#pragma unroll
      for (int i = 0; i < R; ++i) {
        double *p = s_p + tid + i * THREADS;
        *p = __dadd_rn(__dmul_rn(z[i], 1.0), __dmul_rn(*p, beta));
      }
      small_barrier<CTAS>();
    }
  }
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
  if (s.n <= 1024) return launch_small<I, 1, 1024, 1>(h, s, st);
  if (s.n <= 4096) return launch_small<I, 8, 512, 1>(h, s, st);
  if (s.n <= 8192) return launch_small<I, 8, 512, 2>(h, s, st);
  return launch_small<I, 8, 1024, 2>(h, s, st);
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
