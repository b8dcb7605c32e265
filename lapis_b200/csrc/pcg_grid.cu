// Jacobi-PCG on systems of up to a few rows per thread of the GPU: the whole solve in one cooperative launch.
//
// With two launches an iteration such a system is bound by the launches and by the tail of each, in which one block adds
// the partial sums of all (17 to 22 us an iteration at 20,000 to 300,000 rows), and by the tuning of the SpMV kernels in
// front of the solve.  Here a thread keeps up to four rows of x, r, z, p and dinv in registers for the whole solve; z and p are
// in global memory as well, where the other blocks gather them (from L2), and the matrix stays in L1 and L2.
//
// Two meetings of all blocks an iteration.  A block stores its partial sums and the number of the meeting into a slot of
// its own; every block polls the slots of all, a thread each, and adds the sums in one fixed order, so that all derive the
// same alpha, beta and stop test.  The direction p = z + beta p is formed by whoever gathers it (pcg_fuse.h, two-pass form),
// so it needs no meeting; the p buffers alternate.  Between the stores of z and p and their gathers lies a meeting:
//   gathers of z, p_old | sums of p.Ap | stores of z | sums of r.r, r.z | gathers ...
// A slot is written again only behind a meeting that needed every block's reading of it.
//
// The launch is cooperative: all blocks are resident, so every wait ends; each is bounded all the same, and a block whose
// wait runs out sets a flag that ends the others' waits, and the host leaves the system to the passes of pcg.cu.  So it does
// where the driver refuses the launch, because the context has fewer SMs than the device.
//
// us an iteration, in passes and now: 25,600 rows of a 5-point stencil 18.4 and 9.5, 62,500 20 and 11, 160,000 25 and 13.4,
// 291,600 30 and 15.5; scattered columns, 30,000 rows of 12 21.4 and 16.5, 100,000 of 12 31 and 26, 300,000 of 10 56 and
// 35, but 100,000 of 30 39 and 50 (a thread a row reads the entries uncoalesced): at most 16 entries a row on average.  Bound
// by trips to L2, about eight an iteration: columns, gathers, stores, slots, twice.
//
// The recurrences are those of pcg.cu (examples/pcg_solve.py:65-98 in the LAPIS project), element by element; a row of A p
// is added in entry order.  Results are identical from run to run.
#include <algorithm>
#include <cstdint>

#include "common.h"
#include "pcg_fuse.h"

namespace lapis_b200 {

constexpr int GRID_THREADS = 512, GRID_ROWS = 4;  // rows of a thread at most
constexpr int GRID_BUDGET = 4096;                 // iterations per launch (tens of milliseconds)
constexpr unsigned GRID_POLLS = 1u << 20;         // of a wait (about half a second)
constexpr int GRID_GAVE_UP = 3;                   // FL_DONE of a solve in which a wait ran out

struct alignas(16) GridSlot {  // written and read as one
  double sum;
  unsigned long long meeting;
};
struct GridSolve {
  const double *b, *dinv;
  double *x, *r, *z, *p0, *p1;
  GridSlot *slots;  // three for each block: p.Ap, r.r, r.z
  double *sc;
  long long *fl;
  int *gave_up;
  double tol;
  unsigned long long maxiter;
  int n;
  bool first;
};

__device__ __forceinline__ void slot_store(GridSlot *slot, double sum, unsigned long long meeting) {
  asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(slot), "l"(__double_as_longlong(sum)), "l"(meeting)
               : "memory");
}
__device__ __forceinline__ void slot_load(const GridSlot *slot, double &sum, unsigned long long &meeting) {
  unsigned long long s;
  asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}" : "=l"(s), "=l"(meeting) : "l"(slot) : "memory");
  sum = __longlong_as_double(s);
}
// Loads of what other blocks write while this kernel runs.
__device__ __forceinline__ double load_l2(const double *p) {
  double v;
  asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
  return v;
}

template <typename I, int R>
__global__ void __launch_bounds__(GRID_THREADS, 1)
pcg_grid_kernel(const I *__restrict__ pos, const I *__restrict__ crd, const double *__restrict__ val, GridSolve s) {
  constexpr int WARPS = GRID_THREADS / 32;
  __shared__ double s_part[2][WARPS], s_sum[2][WARPS];
  __shared__ int s_ok;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, blocks = gridDim.x;
  unsigned long long meeting = s.first ? 0 : (unsigned long long)s.fl[FL_COUNT];
  if (tid == 0) s_ok = 1;

  auto warp_sum = [&](double v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v = __dadd_rn(v, __shfl_xor_sync(0xffffffffu, v, off));
    return v;
  };
  // Sums of v0 and, with which == 1, of v1 over all threads of all blocks; what any block stored before such a meeting of
  // two sums is visible to all behind it.  False: a wait ran out, here or elsewhere.
  auto meet = [&](int which, double &v0, double &v1) {
    ++meeting;
    const double w0 = warp_sum(v0), w1 = which == 1 ? warp_sum(v1) : 0.0;
    if (lane == 0) {
      s_part[0][warp] = w0;
      s_part[1][warp] = w1;
    }
    __syncthreads();
    if (warp == 0) {
      double t0 = lane < WARPS ? s_part[0][lane] : 0.0, t1 = lane < WARPS ? s_part[1][lane] : 0.0;
      t0 = warp_sum(t0);
      if (which == 1) t1 = warp_sum(t1);
      if (lane == 0) {
        GridSlot *slot = s.slots + 3 * blockIdx.x;
        if (which == 0) {
          slot_store(slot, t0, meeting);
        } else {
          asm volatile("fence.acq_rel.gpu;" ::: "memory");  // this block's z and p, ordered in front by the barrier above, before the number
          slot_store(slot + 1, t0, meeting);
          slot_store(slot + 2, t1, meeting);
        }
      }
    }
    double a0 = 0.0, a1 = 0.0;
    for (int q = tid; q < blocks; q += GRID_THREADS) {
      const GridSlot *slot = s.slots + 3 * q + which;
      double v0 = 0.0, v1 = 0.0;
      bool there = false;
      for (unsigned poll = 0; poll < GRID_POLLS && !there; ++poll) {
        unsigned long long m0, m1 = meeting;
        slot_load(slot, v0, m0);
        if (which == 1) slot_load(slot + 1, v1, m1);
        there = m0 == meeting && m1 == meeting;
        if (!there && (poll & 1023) == 1023 && *reinterpret_cast<volatile int *>(s.gave_up) != 0) break;
      }
      if (!there) {
        *reinterpret_cast<volatile int *>(s.gave_up) = 1;
        s_ok = 0;
      }
      a0 = __dadd_rn(a0, v0);
      if (which == 1) a1 = __dadd_rn(a1, v1);
    }
    if (which == 1) asm volatile("fence.acq_rel.gpu;" ::: "memory");  // the others' z and p behind their numbers
    a0 = warp_sum(a0);
    if (which == 1) a1 = warp_sum(a1);
    if (lane == 0) {
      s_sum[0][warp] = a0;
      s_sum[1][warp] = a1;
    }
    __syncthreads();
    v0 = v1 = 0.0;
    const int used = (blocks + 31) / 32 < WARPS ? (blocks + 31) / 32 : WARPS;
    for (int q = 0; q < used; ++q) {
      v0 = __dadd_rn(v0, s_sum[0][q]);
      v1 = __dadd_rn(v1, s_sum[1][q]);
    }
    return s_ok != 0;
  };

  const I *c[R];
  const double *v[R];
  int row[R], len[R];
  double x[R], r[R], z[R], d[R], p[R];
  double rr = 0.0, rzp = 0.0;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    row[i] = (i * blocks + (int)blockIdx.x) * GRID_THREADS + tid;
    const bool in = row[i] < s.n;
    const int64_t lo = in ? (int64_t)pos[row[i]] : 0;
    c[i] = crd + lo;
    v[i] = val + lo;
    len[i] = in ? (int)((int64_t)pos[row[i] + 1] - lo) : -1;  // -1: no row
    d[i] = in ? s.dinv[row[i]] : 0.0;
    r[i] = in ? (s.first ? s.b[row[i]] : s.r[row[i]]) : 0.0;
    x[i] = in && !s.first ? s.x[row[i]] : 0.0;
    z[i] = __dmul_rn(r[i], d[i]);
    p[i] = in && !s.first ? s.p0[row[i]] : z[i];
    if (in && s.first) {
      s.z[row[i]] = z[i];
      s.p0[row[i]] = z[i];
      rr = __dadd_rn(rr, __dmul_rn(r[i], r[i]));
      rzp = __dadd_rn(rzp, __dmul_rn(r[i], z[i]));
    }
  }
  double initres, rz, relres = 0.0, beta = 0.0;
  unsigned long long iters = 0;
  bool done = false, fresh = s.first, ok = true;  // fresh: p is the one to use, no direction update yet
  if (s.first) {
    ok = meet(1, rr, rzp);
    initres = sqrt(rr);
    rz = rzp;
  } else {
    initres = s.sc[SC_INITRES];
    rz = s.sc[SC_RZ];
    beta = s.sc[SC_BETA];
    iters = (unsigned long long)s.fl[FL_ITERS];
  }
  double *pold = s.p0, *pnew = s.p1;
  for (int left = GRID_BUDGET; left > 0 && !done && ok; --left) {
    double ap[R], pap = 0.0;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      ap[i] = 0.0;
      if (!fresh) {
        p[i] = __dadd_rn(__dmul_rn(z[i], 1.0), __dmul_rn(p[i], beta));
        if (len[i] >= 0) pnew[row[i]] = p[i];
      }
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
      // Five at a time, us an iteration with 4, 5 and 8: 250,000 rows of a 9-point stencil 18.7, 17.2, 18.9, 291,600 of a 5-point one
      // 15.7, 14.3, 15.1, 30,000 scattered rows of 5 13.0, 11.6, 12.2, 100,000 of 11 28.3, 27.3, 27.8; but 300,000 of 9 42.9, 42.0, 37.3.
      for (int j = 0; j < len[i]; j += 5) {
        double a[5], zv[5], pv[5];
#pragma unroll
        for (int u = 0; u < 5; ++u) {
          const bool in = j + u < len[i];
          const uint32_t at = in ? min((uint32_t)__ldg(c[i] + j + u), (uint32_t)s.n - 1) : 0;  // a bad index stays inside
          a[u] = in ? __ldg(v[i] + j + u) : 0.0;
          pv[u] = in ? load_l2(pold + at) : 0.0;
          zv[u] = in && !fresh ? load_l2(s.z + at) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 5; ++u) {
          const double pc = fresh ? pv[u] : __dadd_rn(__dmul_rn(zv[u], 1.0), __dmul_rn(pv[u], beta));
          if (j + u < len[i]) ap[i] = __dadd_rn(ap[i], __dmul_rn(a[u], pc));
        }
      }
      if (len[i] >= 0) pap = __dadd_rn(pap, __dmul_rn(ap[i], p[i]));
    }
    if (!fresh) {
      double *swap = pold;
      pold = pnew;
      pnew = swap;
    }
    fresh = false;
    double unused = 0.0;
    ok = meet(0, pap, unused);
    if (!ok) break;
    const double alpha = rz / pap, malpha = -alpha;
    rr = rzp = 0.0;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      x[i] = __dadd_rn(__dmul_rn(x[i], 1.0), __dmul_rn(p[i], alpha));
      r[i] = __dadd_rn(__dmul_rn(r[i], 1.0), __dmul_rn(ap[i], malpha));
      z[i] = __dmul_rn(r[i], d[i]);
      if (len[i] >= 0) {
        s.z[row[i]] = z[i];
        rr = __dadd_rn(rr, __dmul_rn(r[i], r[i]));
        rzp = __dadd_rn(rzp, __dmul_rn(r[i], z[i]));
      }
    }
    ok = meet(1, rr, rzp);
    if (!ok) break;
    ++iters;
    relres = sqrt(rr) / initres;
    done = !(relres > s.tol && iters != s.maxiter);  // ordered compare: NaN stops the loop
    if (!done) {
      beta = rzp / rz;
      rz = rzp;
    }
  }
  // p0 is read by other blocks until the last meeting, which all have passed
#pragma unroll
  for (int i = 0; i < R; ++i) {
    if (len[i] < 0) continue;
    s.x[row[i]] = x[i];
    if (!done) {
      s.r[row[i]] = r[i];
      s.p0[row[i]] = p[i];
    }
  }
  if (blockIdx.x == 0 && tid == 0) {
    s.sc[SC_INITRES] = initres;
    s.sc[SC_RZ] = rz;
    s.sc[SC_BETA] = beta;
    s.sc[SC_RELRES] = relres;
    s.fl[FL_ITERS] = (long long)iters;
    s.fl[FL_COUNT] = (long long)meeting;
    s.fl[FL_DONE] = !ok ? GRID_GAVE_UP : done ? 1 : 0;
  }
}

template <typename I>
static cudaError_t launch_grid(const lapis_b200_csr *h, GridSolve &s, cudaStream_t st) {
  const int64_t blocks = std::min<int64_t>((s.n + GRID_THREADS - 1) / GRID_THREADS, sm_count());
  const int64_t rows = (s.n + blocks * GRID_THREADS - 1) / (blocks * GRID_THREADS);
  const I *pos = static_cast<const I *>(h->pos), *crd = static_cast<const I *>(h->crd);
  const double *val = h->val;
  void *args[] = {&pos, &crd, &val, &s};
  const void *kernel = rows <= 1 ? reinterpret_cast<const void *>(pcg_grid_kernel<I, 1>) : rows <= 2 ? reinterpret_cast<const void *>(pcg_grid_kernel<I, 2>)
                                                                                       : reinterpret_cast<const void *>(pcg_grid_kernel<I, GRID_ROWS>);
  return cudaLaunchCooperativeKernel(kernel, dim3((unsigned)blocks), dim3(GRID_THREADS), args, 0, st);
}

// Whether a system of rows that a thread each can work on, no more than 32 entries long, is solved here.
bool pcg_grid_fits(int64_t nrows, int64_t nnz) {
  int dev = 0, can = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&can, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || can == 0) return false;
  return nrows <= (int64_t)GRID_ROWS * GRID_THREADS * sm_count() && nnz <= 16 * nrows;
}

// *solved: false where the launch was refused or a wait ran out and the system is left to the passes.
int pcg_grid(const lapis_b200_csr *h, const double *d_b, const double *d_dinv, double tol, uint64_t maxiter, double *d_x, uint64_t *iters,
             double *relres, bool *solved, cudaStream_t st) {
  const int64_t n = h->nrows, slots = 3 * (int64_t)sm_count();
  const size_t head = 32 * sizeof(double) + slots * sizeof(GridSlot);
  PoolBuf buf;
  LAPIS_TRY(buf.alloc(head + (size_t)(4 * n) * sizeof(double), st));
  LAPIS_CUDA_TRY(cudaMemsetAsync(buf.p, 0, head, st));
  GridSolve s = {};
  s.sc = static_cast<double *>(buf.p);
  s.fl = reinterpret_cast<long long *>(s.sc + SC_COUNT);
  s.gave_up = reinterpret_cast<int *>(s.sc + 16);
  s.slots = reinterpret_cast<GridSlot *>(s.sc + 32);
  s.r = reinterpret_cast<double *>(s.slots + slots);
  s.z = s.r + n;
  s.p0 = s.z + n;
  s.p1 = s.p0 + n;
  s.b = d_b;
  s.dinv = d_dinv;
  s.x = d_x;
  s.tol = tol;
  s.maxiter = maxiter;
  s.n = (int)n;
  s.first = true;
  const uint64_t limit = maxiter == 0 ? (1ull << 31) : maxiter;
  int done = 0;
  uint64_t it = 0;
  do {
    const cudaError_t e = h->idx_bytes == 4 ? launch_grid<int32_t>(h, s, st) : launch_grid<int64_t>(h, s, st);
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorLaunchOutOfResources || e == cudaErrorNotSupported) {
      cudaGetLastError();
      *solved = false;
      return LAPIS_OK;
    }
    LAPIS_CUDA_TRY(e);
    s.first = false;
    LAPIS_TRY(lapis_b200_pcg_status(s.sc, &done, &it, relres, st));
    *solved = done != GRID_GAVE_UP;
    if (!*solved) return LAPIS_OK;
  } while (!done && it < limit);
  if (iters) *iters = it;
  return LAPIS_OK;
}

}  // namespace lapis_b200
