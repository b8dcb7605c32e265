// Shared host-side helpers: status recording, CUDA error checks, the CSR handle.
#pragma once
#include <cuda_runtime.h>
#include <cstdarg>
#include <cstdint>
#include <cstdio>

#include "../../include/lapis_b200.h"

namespace lapis_b200 {

// Records status + message for lapis_last_error(); returns `code` so callers can
// `return fail(...)`.
int fail(int code, const char *fmt, ...);
void clear_error();

#define LAPIS_CUDA_TRY(expr)                                                              \
  do {                                                                                    \
    cudaError_t _e = (expr);                                                              \
    if (_e != cudaSuccess)                                                                \
      return ::lapis_b200::fail(LAPIS_ECUDA, "%s failed: %s (%s:%d)", #expr,              \
                                cudaGetErrorString(_e), __FILE__, __LINE__);              \
  } while (0)

#define LAPIS_TRY(expr)          \
  do {                           \
    int _s = (expr);             \
    if (_s != LAPIS_OK) return _s; \
  } while (0)

inline cudaStream_t as_stream(void *s) { return reinterpret_cast<cudaStream_t>(s); }

// Number of SMs of the current device (cached per device).
int sm_count();

// Stream-ordered device memory from a pool of this library, one per device (cudaMalloc and cudaFree cost 330 and
// 265 us each where they were measured, an allocation from the pool about 1 us).  Safe with several threads and
// streams: the driver orders reuse by stream.  The pool keeps at most POOL_KEEP_BYTES of freed memory, which is the
// largest block that it serves, and gives the rest back at the next synchronisation; pool_trim returns all of it
// (lapis_finalize, and an allocation that fails).
constexpr size_t POOL_LARGEST = size_t(256) << 20;
constexpr size_t POOL_KEEP_BYTES = POOL_LARGEST;
int pool_alloc(void **p, size_t bytes, cudaStream_t st);
void pool_free(void *p, cudaStream_t st);
void pool_trim();
int large_alloc(void **p, size_t bytes);  // cudaMalloc

// Scoped device memory.  Large blocks come from cudaMalloc: mapping memory into the pool and out again costs 25 ms each
// way for 850 MB, cudaMalloc and cudaFree 1 to 4 ms.
struct PoolBuf {
  void *p = nullptr;
  cudaStream_t st = nullptr;
  bool pooled = true;
  PoolBuf() = default;
  PoolBuf(const PoolBuf &) = delete;
  PoolBuf &operator=(const PoolBuf &) = delete;
  ~PoolBuf() {
    if (pooled) pool_free(p, st);
    else cudaFree(p);
  }
  int alloc(size_t bytes, cudaStream_t stream) {
    st = stream;
    pooled = bytes <= POOL_LARGEST;
    return pooled ? pool_alloc(&p, bytes, stream) : large_alloc(&p, bytes);
  }
};

// Launch that may start while the kernel in front of it drains (programmatic stream serialization): the blocks become
// resident early and stop at pdl_wait().  Only for kernels that call pdl_wait() before their first access to memory that
// the kernel in front writes (the main SpMM kernel shares nothing but inputs with the one for long rows in front of it);
// what that kernel may still be writing is read by ordinary loads, not by the read-only path.  Back-to-back small launches
// then follow each other without the gap of about 1.5 us.
template <typename... P, typename... A>
inline cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
#ifdef __CUDACC__
// Waits until everything in front of this kernel has completed and its writes are visible.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The next launch_pdl kernel may become resident.  Called late in a block's work: blocks that come in while this
// kernel still fills some SMs are placed on the others, and a grid that does not fill the GPU ends up unevenly spread
// (measured: 1e6 entries, 11 -> 16 us with the call at the top).
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;"); }
// Ordinary load, for what the launch in front may still have been writing when this kernel became resident (launch_pdl).
// The read-only path (ld.global.nc, which __ldg and reads through const __restrict__ compile to) asks that data stays as it
// is for the kernel's whole lifetime, which begins in front of pdl_wait().
__device__ __forceinline__ double load_now(const double *p) {
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
#endif

}  // namespace lapis_b200

// The CSR handle: borrowed matrix arrays + the streaming plan owned by the handle.
struct lapis_b200_csr {
  int idx_bytes;
  int64_t nrows, ncols, nnz, base;  // base = pos[0]
  const void *pos, *crd;
  const double *val;
  // Streaming plan: thread block b of the SpMV kernel processes the stored entries
  // [abase + b*TILE, abase + (b+1)*TILE), abase = base & ~1; blk_row[b] is the first row
  // that ends inside that chunk (nblk+1 entries).  carry[b] receives the partial sum of
  // the row that runs past chunk b.
  int64_t nblk;
  int64_t *blk_row;
  double *carry;
  // Scratch for the fused dot product of the PCG SpMV pass (one double per block).
  double *blk_partial;
  // Kernel variant chosen by lapis_b200_csr_tune (tuned_threads == 0: not tuned).
  int tuned_threads, tuned_minb, tuned_hint;
  // The fastest of the candidates that the passes of a solver run as they are timed (with a dot product fused, rows one
  // thread each are spmv_rowthread_kernel whatever short-row kernel wins a plain product).
  int fused_threads, fused_minb, fused_hint;
  // Longest row (-1: not known).  The kernels for short rows are only used when no row has more than 32 entries: up
  // to there they return the same bits as the chunk kernels.
  int64_t max_row_len;
  int device;
  // Second plan for the warp-walk kernel on small matrices: ranges of walk_tile entries (null: it uses blk_row).
  int64_t *walk_plan;
  double *walk_carry;
  int64_t walk_nblk;
  int walk_tile;
};

namespace lapis_b200 {
// SpMM over a CSR matrix (rowno null) or the stored rows of a DCSR matrix (their numbers in rowno), spmm.cu.
// nnz, max_row_len (-1: not known): of a CSR matrix only.
int spmm_launch(int idx_bytes, const void *rowno, const void *pos, const void *crd, const double *val, int64_t nrows, int64_t k,
                int64_t nnz, int64_t max_row_len, const double *B, double *C, int accumulate, cudaStream_t st);
// Fills a handle over arrays whose first offset, entry count and longest row are known, allocates its scratch and
// enqueues the planning kernels.  plan_on_demand: no scratch and no plan when SpMV will run on the kernels for short
// rows, which need none (for a handle that serves one product).
int csr_setup(lapis_b200_csr *h, int idx_bytes, int64_t nrows, int64_t ncols, int64_t base, int64_t nnz, int64_t max_row_len,
              const void *d_pos, const void *d_crd, const double *d_val, bool plan_on_demand, PoolBuf *scratch, cudaStream_t st);
}  // namespace lapis_b200
