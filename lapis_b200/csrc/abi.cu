// Emitted-module ABI: lapis_initialize / lapis_finalize and the py_<func> wrappers.
//
// Mirrors what mlir/lib/Target/KokkosCpp/TranslateToKokkosCpp.cpp:2541-2684 prints
// for every public function: descriptors in (host memory), results out through
// `ret` slots, device work fenced before returning.  Where the emitted wrapper
// wraps host pointers in unmanaged Kokkos views and lets LAPIS::DualView copy them
// to the device (LAPISSupport.hpp:193-282), this file stages the operands in device
// buffers (stage.h), runs the kernels and copies the result back.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "common.h"
#include "stage.h"

extern "C" int64_t lapis_b200_pcg_workspace_bytes(int64_t n, int64_t n_p);

namespace lapis_b200 {

static thread_local int g_status = LAPIS_OK;
static thread_local char g_message[512] = "";

int fail(int code, const char *fmt, ...) {
  g_status = code;
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_message, sizeof(g_message), fmt, ap);
  va_end(ap);
  return code;
}

void clear_error() {
  g_status = LAPIS_OK;
  g_message[0] = '\0';
}

int sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (cached[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev] = n;
  }
  return cached[dev];
}

// ---- device memory pool -----------------------------------------------------
static std::mutex g_pool_mutex;
static cudaMemPool_t g_pools[64] = {nullptr};

static int pool_of_device(cudaMemPool_t *out) {
  int dev = 0;
  LAPIS_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return fail(LAPIS_EBADARG, "device index %d not supported", dev);
  std::lock_guard<std::mutex> lock(g_pool_mutex);
  if (g_pools[dev] == nullptr) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool;
    LAPIS_CUDA_TRY(cudaMemPoolCreate(&pool, &props));
    uint64_t keep = POOL_KEEP_BYTES;
    LAPIS_CUDA_TRY(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    g_pools[dev] = pool;
  }
  *out = g_pools[dev];
  return LAPIS_OK;
}

// Where the device is full, the memory that the pools hold idle goes back to it and the allocation is tried again.
template <typename F>
static cudaError_t alloc_or_trim(F &&alloc) {
  cudaError_t e = alloc();
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    cudaDeviceSynchronize();  // what was freed behind work still running
    pool_trim();
    e = alloc();
  }
  return e;
}

static int alloc_status(cudaError_t e, void **p, size_t bytes) {
  if (e == cudaSuccess) return LAPIS_OK;
  *p = nullptr;
  return fail(LAPIS_ECUDA, "device allocation of %zu bytes failed: %s", bytes, cudaGetErrorString(e));
}

int pool_alloc(void **p, size_t bytes, cudaStream_t st) {
  cudaMemPool_t pool = nullptr;
  LAPIS_TRY(pool_of_device(&pool));
  return alloc_status(alloc_or_trim([&] { return cudaMallocFromPoolAsync(p, bytes > 0 ? bytes : 16, pool, st); }), p, bytes);
}

int large_alloc(void **p, size_t bytes) {
  return alloc_status(alloc_or_trim([&] { return cudaMalloc(p, bytes); }), p, bytes);
}

void pool_free(void *p, cudaStream_t st) {
  if (p != nullptr) cudaFreeAsync(p, st);
}

void pool_trim() {
  std::lock_guard<std::mutex> lock(g_pool_mutex);
  for (cudaMemPool_t pool : g_pools)
    if (pool != nullptr) cudaMemPoolTrimTo(pool, 0);
}

// ---- module state -----------------------------------------------------------
static int g_init_count = 0;
static std::vector<void *> g_alive_host;  // result buffers handed to the caller (LAPISSupport.hpp:93-120)

static int require_init() {
  if (g_init_count <= 0) return fail(LAPIS_ENOTINIT, "lapis_initialize has not been called");
  return LAPIS_OK;
}

// C-contiguity check of LAPISSupport.hpp:80-89 (LayoutRight).
template <typename M, int R>
static int check_contig(const M *m, const char *what) {
  if (m == nullptr) return fail(LAPIS_EBADARG, "%s: null descriptor", what);
  int64_t expect = 1;
  for (int i = R - 1; i >= 0; --i) {
    if (m->sizes[i] < 0) return fail(LAPIS_EBADSHAPE, "%s: negative extent", what);
    if (m->sizes[i] > 1 && m->strides[i] != expect)
      return fail(LAPIS_ELAYOUT, "%s: descriptor is not contiguous row-major", what);
    expect *= m->sizes[i];
  }
  if (expect > 0 && m->data == nullptr) return fail(LAPIS_EBADARG, "%s: null data pointer", what);
  return LAPIS_OK;
}

template <typename T, typename M>
static T *elem_ptr(const M *m) {
  return static_cast<T *>(m->data) + m->offset;
}

struct CsrArgs {
  int64_t nrows, ncols, npos, nnz;
};

static int check_csr(const lapis_memref1 *pos, const lapis_memref1 *crd, const lapis_memref1 *val,
                     const lapis_csr_spec *spec, CsrArgs *out) {
  LAPIS_TRY((check_contig<lapis_memref1, 1>(pos, "pos")));
  LAPIS_TRY((check_contig<lapis_memref1, 1>(crd, "crd")));
  LAPIS_TRY((check_contig<lapis_memref1, 1>(val, "val")));
  if (spec == nullptr) return fail(LAPIS_EBADARG, "null storage specifier");
  out->nrows = spec->dims[0];
  out->ncols = spec->dims[1];
  out->npos = spec->mem_sizes[0];
  out->nnz = spec->mem_sizes[2];
  if (out->nrows < 0 || out->ncols < 0) return fail(LAPIS_EBADSHAPE, "negative matrix dimension");
  if (out->npos != out->nrows + 1 || pos->sizes[0] < out->npos)
    return fail(LAPIS_EBADSHAPE, "pos must have rows+1 entries");
  if (spec->mem_sizes[1] != out->nnz || crd->sizes[0] < out->nnz || val->sizes[0] < out->nnz)
    return fail(LAPIS_EBADSHAPE, "crd/val shorter than the specifier says");
  return LAPIS_OK;
}

// Validates pos on the host (non-decreasing, ends at nnz) before any kernel trusts it.
template <typename I>
static int check_pos_host(const I *pos, int64_t nrows, int64_t nnz) {
  if (pos[0] != 0) return fail(LAPIS_EBADSHAPE, "pos[0] must be 0");
  for (int64_t r = 0; r < nrows; ++r)
    if (pos[r + 1] < pos[r]) return fail(LAPIS_EBADSHAPE, "pos is not non-decreasing at row %lld", (long long)r);
  if ((int64_t)pos[nrows] != nnz) return fail(LAPIS_EBADSHAPE, "pos[rows] != number of stored entries");
  return LAPIS_OK;
}

// Validates the column indices on the host: 0 <= crd[j] < ncols for every stored entry.  The emitted code
// indexes x with them unchecked (a bad index is undefined behaviour there); here a bad index must not
// reach a gather on the device.  Min and max over slices of the array on a few host threads.
template <typename I>
static int check_crd_host(const I *crd, int64_t nnz, int64_t ncols) {
  if (nnz <= 0) return LAPIS_OK;
  const int nthreads = nnz < (1 << 20) ? 1 : (int)std::min<int64_t>(8, std::max(1u, std::thread::hardware_concurrency()));
  std::vector<I> lo(nthreads), hi(nthreads);
  auto scan = [&](int t) {
    const int64_t b = nnz * t / nthreads, e = nnz * (t + 1) / nthreads;
    I mn = crd[b], mx = crd[b];
    for (int64_t j = b; j < e; ++j) {
      mn = crd[j] < mn ? crd[j] : mn;
      mx = crd[j] > mx ? crd[j] : mx;
    }
    lo[t] = mn;
    hi[t] = mx;
  };
  if (nthreads == 1) {
    scan(0);
  } else {
    std::vector<std::thread> pool;
    for (int t = 0; t < nthreads; ++t) pool.emplace_back(scan, t);
    for (auto &th : pool) th.join();
  }
  I mn = lo[0], mx = hi[0];
  for (int t = 1; t < nthreads; ++t) {
    mn = lo[t] < mn ? lo[t] : mn;
    mx = hi[t] > mx ? hi[t] : mx;
  }
  if ((int64_t)mn < 0 || (int64_t)mx >= ncols)
    return fail(LAPIS_EBADSHAPE, "column index out of range: crd holds values in [%lld, %lld], the matrix has %lld columns",
                (long long)mn, (long long)mx, (long long)ncols);
  return LAPIS_OK;
}

// A result vector owned by the module until lapis_finalize (LAPISSupport.hpp:93-120), filled from the device.
static int result_vector(const void *d_src, int64_t n, lapis_memref1 *out, cudaStream_t st) {
  double *hx = static_cast<double *>(std::malloc(n > 0 ? (size_t)n * 8 : 8));
  if (hx == nullptr) return fail(LAPIS_ECUDA, "host allocation failed");
  g_alive_host.push_back(hx);
  LAPIS_TRY(stage_download(hx, d_src, (size_t)n * 8, st));
  out->basePtr = hx;
  out->data = hx;
  out->offset = 0;
  out->sizes[0] = n;
  out->strides[0] = 1;
  return LAPIS_OK;
}

// Operands of a call: laid out in one device allocation and sent there.  Page-locked arrays are copied in place, so a call
// that fails after the upload waits for the stream before the caller has its arrays back; one that succeeds has waited
// for its result.
struct Operands {
  Upload up;
  PoolBuf dev;
  bool in_flight = false;
  ~Operands() {
    if (in_flight) cudaStreamSynchronize(dev.st);
  }
  int send(cudaStream_t st, Upload::Facts *facts, size_t extra = 0) {
    const size_t bytes = up.layout();
    extra_at = bytes;
    LAPIS_TRY(dev.alloc(bytes + extra, st));
    in_flight = true;
    return up.run(dev.p, st, facts);
  }
  // The last download's status goes through here.
  int finish(int status) {
    if (status == LAPIS_OK) in_flight = false;
    return status;
  }
  template <typename T>
  T *at(int part) const {
    return up.at<T>(dev.p, part);
  }
  template <typename T>
  T *extra(size_t offset = 0) const {
    return reinterpret_cast<T *>(static_cast<char *>(dev.p) + extra_at + offset);
  }
  size_t extra_at = 0;
};

// What the upload found out about the index arrays, as a status.
template <typename I>
static int check_facts(const Upload::Facts &f, const I *pos, const I *crd, int64_t nrows, int64_t nnz, int64_t ncols) {
  if (pos[0] != 0) return fail(LAPIS_EBADSHAPE, "pos[0] must be 0");
  if (f.bad_row >= 0) return fail(LAPIS_EBADSHAPE, "pos is not non-decreasing at row %lld", (long long)f.bad_row);
  if ((int64_t)pos[nrows] != nnz) return fail(LAPIS_EBADSHAPE, "pos[rows] != number of stored entries");
  if (!f.crd_in_range) return check_crd_host<I>(crd, nnz, ncols);  // finds the values for the message
  return LAPIS_OK;
}

// A CSR operand of a call: its three arrays among the uploaded parts, and the handle over them.
struct CsrOperand {
  int pos = 0, crd = 0, val = 0;
  lapis_b200_csr h;
  PoolBuf scratch;
  template <typename I>
  void add(Upload &up, const lapis_memref1 *mpos, const lapis_memref1 *mcrd, const lapis_memref1 *mval, const CsrArgs &a) {
    pos = up.add_pos(elem_ptr<I>(mpos), a.npos);
    crd = up.add_crd(elem_ptr<I>(mcrd), a.nnz, a.ncols);
    val = up.add(elem_ptr<double>(mval), (size_t)a.nnz * 8);
  }
  template <typename I>
  int setup(const Operands &ops, const Upload::Facts &f, const lapis_memref1 *mpos, const lapis_memref1 *mcrd, const CsrArgs &a,
            bool plan_on_demand, cudaStream_t st) {
    LAPIS_TRY((check_facts<I>(f, elem_ptr<I>(mpos), elem_ptr<I>(mcrd), a.nrows, a.nnz, a.ncols)));
    return csr_setup(&h, (int)sizeof(I), a.nrows, a.ncols, 0, a.nnz, f.max_row_len, ops.at<void>(pos), ops.at<void>(crd),
                     ops.at<double>(val), plan_on_demand, &scratch, st);
  }
};

template <typename I>
static int spmv_host(lapis_memref1 **ret0, lapis_memref1 *pos, lapis_memref1 *crd, lapis_memref1 *val,
                     const lapis_csr_spec *spec, lapis_memref1 *x, lapis_memref1 *y) {
  clear_error();
  LAPIS_TRY(require_init());
  CsrArgs a;
  LAPIS_TRY(check_csr(pos, crd, val, spec, &a));
  LAPIS_TRY((check_contig<lapis_memref1, 1>(x, "x")));
  LAPIS_TRY((check_contig<lapis_memref1, 1>(y, "y")));
  if (x->sizes[0] != a.ncols || y->sizes[0] != a.nrows) return fail(LAPIS_EBADSHAPE, "spmv: x/y length mismatch");
  cudaStream_t st = nullptr;
  Operands ops;
  CsrOperand A;
  A.add<I>(ops.up, pos, crd, val, a);
  const int px = ops.up.add(elem_ptr<double>(x), (size_t)a.ncols * 8), py = ops.up.add(elem_ptr<double>(y), (size_t)a.nrows * 8);
  Upload::Facts facts;
  LAPIS_TRY(ops.send(st, &facts));
  LAPIS_TRY(A.setup<I>(ops, facts, pos, crd, a, true, st));
  LAPIS_TRY(lapis_b200_spmv_f64(&A.h, ops.at<double>(px), ops.at<double>(py), 1, st));
  LAPIS_TRY(ops.finish(stage_download(elem_ptr<double>(y), ops.at<double>(py), (size_t)a.nrows * 8, st)));  // emitted fence, :2682
  if (ret0 != nullptr && *ret0 != nullptr) **ret0 = *y;  // the function returns its outs argument
  return LAPIS_OK;
}

template <typename I>
static int spmm_host(lapis_memref2 **ret0, lapis_memref1 *pos, lapis_memref1 *crd, lapis_memref1 *val,
                     const lapis_csr_spec *spec, lapis_memref2 *B, lapis_memref2 *C) {
  clear_error();
  LAPIS_TRY(require_init());
  CsrArgs a;
  LAPIS_TRY(check_csr(pos, crd, val, spec, &a));
  LAPIS_TRY((check_contig<lapis_memref2, 2>(B, "B")));
  LAPIS_TRY((check_contig<lapis_memref2, 2>(C, "C")));
  const int64_t k = B->sizes[1];
  if (B->sizes[0] != a.ncols || C->sizes[0] != a.nrows || C->sizes[1] != k)
    return fail(LAPIS_EBADSHAPE, "spmm: B/C shape mismatch");
  cudaStream_t st = nullptr;
  Operands ops;
  CsrOperand A;
  A.add<I>(ops.up, pos, crd, val, a);
  const size_t bC = (size_t)a.nrows * k * 8;
  const int pB = ops.up.add(elem_ptr<double>(B), (size_t)a.ncols * k * 8), pC = ops.up.add(elem_ptr<double>(C), bC);
  Upload::Facts facts;
  LAPIS_TRY(ops.send(st, &facts));
  LAPIS_TRY(A.setup<I>(ops, facts, pos, crd, a, true, st));
  LAPIS_TRY(lapis_b200_spmm_f64(&A.h, k, ops.at<double>(pB), ops.at<double>(pC), 1, st));
  LAPIS_TRY(ops.finish(stage_download(elem_ptr<double>(C), ops.at<double>(pC), bC, st)));
  if (ret0 != nullptr && *ret0 != nullptr) **ret0 = *C;
  return LAPIS_OK;
}

static int gemm_host(int64_t batch, int64_t M, int64_t N, int64_t K, const float *A, const float *B, float *C) {
  cudaStream_t st = nullptr;
  Operands ops;
  const size_t bC = (size_t)batch * M * N * 4;
  const int pA = ops.up.add(A, (size_t)batch * M * K * 4), pB = ops.up.add(B, (size_t)batch * K * N * 4), pC = ops.up.add(C, bC);
  Upload::Facts facts;
  LAPIS_TRY(ops.send(st, &facts));
  LAPIS_TRY(lapis_b200_bgemm_f32(batch, M, N, K, ops.at<float>(pA), ops.at<float>(pB), ops.at<float>(pC), st));
  LAPIS_TRY(lapis_b200_bgemm_status(st));
  return ops.finish(stage_download(C, ops.at<float>(pC), bC, st));
}

template <typename I>
static int pcg_host(lapis_memref1 **ret0, size_t *ret1, double *ret2, lapis_memref1 *pos, lapis_memref1 *crd,
                    lapis_memref1 *val, const lapis_csr_spec *spec, lapis_memref1 *b, lapis_memref1 *dinv, double tol,
                    size_t maxiter) {
  clear_error();
  LAPIS_TRY(require_init());
  CsrArgs a;
  LAPIS_TRY(check_csr(pos, crd, val, spec, &a));
  LAPIS_TRY((check_contig<lapis_memref1, 1>(b, "b")));
  LAPIS_TRY((check_contig<lapis_memref1, 1>(dinv, "dinv")));
  const int64_t n = b->sizes[0];
  if (a.nrows != n || a.ncols != n || dinv->sizes[0] != n) return fail(LAPIS_EBADSHAPE, "pcg: A, b, dinv sizes differ");
  if (ret0 == nullptr || *ret0 == nullptr) return fail(LAPIS_EBADARG, "pcg: null result slot");
  cudaStream_t st = nullptr;
  Operands ops;
  CsrOperand A;
  A.add<I>(ops.up, pos, crd, val, a);
  const int pb = ops.up.add(elem_ptr<double>(b), (size_t)n * 8), pd = ops.up.add(elem_ptr<double>(dinv), (size_t)n * 8);
  Upload::Facts facts;
  LAPIS_TRY(ops.send(st, &facts, (size_t)n * 8));
  LAPIS_TRY(A.setup<I>(ops, facts, pos, crd, a, false, st));
  double *dx = ops.extra<double>();
  uint64_t iters = 0;
  double relres = 0.0;
  LAPIS_TRY(lapis_b200_pcg_f64(&A.h, ops.at<double>(pb), ops.at<double>(pd), tol, (uint64_t)maxiter, dx, &iters, &relres, st));
  LAPIS_TRY(ops.finish(result_vector(dx, n, *ret0, st)));
  if (ret1) *ret1 = (size_t)iters;
  if (ret2) *ret2 = relres;
  return LAPIS_OK;
}

// examples/hitting_times.py:151-194 (@mht), call at :216
template <typename I>
static int mht_host(lapis_memref1 **ret0, lapis_memref1 **ret1, lapis_memref1 *pos, lapis_memref1 *crd, lapis_memref1 *val,
                    const lapis_csr_spec *spec, lapis_memref1 *mask, lapis_memref1 *dvec, double alpha, double tol,
                    size_t maxiter) {
  clear_error();
  LAPIS_TRY(require_init());
  CsrArgs a;
  LAPIS_TRY(check_csr(pos, crd, val, spec, &a));
  LAPIS_TRY((check_contig<lapis_memref1, 1>(mask, "mask")));
  LAPIS_TRY((check_contig<lapis_memref1, 1>(dvec, "d")));
  const int64_t n = dvec->sizes[0];
  if (a.nrows != n || a.ncols != n || mask->sizes[0] != n) return fail(LAPIS_EBADSHAPE, "mht: A, mask, d sizes differ");
  if (ret0 == nullptr || *ret0 == nullptr || ret1 == nullptr || *ret1 == nullptr)
    return fail(LAPIS_EBADARG, "mht: null result slot");
  cudaStream_t st = nullptr;
  Operands ops;
  CsrOperand A;
  A.add<I>(ops.up, pos, crd, val, a);
  const int pm = ops.up.add(elem_ptr<double>(mask), (size_t)n * 8), pd = ops.up.add(elem_ptr<double>(dvec), (size_t)n * 8);
  Upload::Facts facts;
  LAPIS_TRY(ops.send(st, &facts, 2 * (size_t)n * 8));
  LAPIS_TRY(A.setup<I>(ops, facts, pos, crd, a, false, st));
  double *m1 = ops.extra<double>(), *m2 = m1 + n;
  LAPIS_TRY(lapis_b200_mht_f64(&A.h, ops.at<double>(pm), ops.at<double>(pd), alpha, tol, (uint64_t)maxiter, m1, m2, nullptr, nullptr, st));
  LAPIS_TRY(result_vector(m1, n, *ret0, st));
  return ops.finish(result_vector(m2, n, *ret1, st));
}

// examples/hitting_times.py:196-218 (@normalize_mom2), call at :218
static int normalize_mom2_host(lapis_memref1 **ret0, lapis_memref1 *mom1, lapis_memref1 *mom2) {
  clear_error();
  LAPIS_TRY(require_init());
  LAPIS_TRY((check_contig<lapis_memref1, 1>(mom1, "mom1")));
  LAPIS_TRY((check_contig<lapis_memref1, 1>(mom2, "mom2")));
  const int64_t n = mom1->sizes[0];
  if (mom2->sizes[0] != n) return fail(LAPIS_EBADSHAPE, "normalize_mom2: lengths differ");
  if (ret0 == nullptr || *ret0 == nullptr) return fail(LAPIS_EBADARG, "normalize_mom2: null result slot");
  cudaStream_t st = nullptr;
  Operands ops;
  const int p1 = ops.up.add(elem_ptr<double>(mom1), (size_t)n * 8), p2 = ops.up.add(elem_ptr<double>(mom2), (size_t)n * 8);
  Upload::Facts facts;
  LAPIS_TRY(ops.send(st, &facts, (size_t)n * 8));
  LAPIS_TRY(lapis_b200_normalize_mom2_f64(n, ops.at<double>(p1), ops.at<double>(p2), ops.extra<double>(), st));
  return ops.finish(result_vector(ops.extra<double>(), n, *ret0, st));
}

// examples/bspmm.py:26-52, call at :103
template <typename I>
static int bspmm_host(lapis_memref3 **ret0, lapis_memref1 *pos, lapis_memref1 *crd, lapis_memref1 *val,
                      const lapis_csrv_spec *spec, lapis_memref3 *B) {
  clear_error();
  LAPIS_TRY(require_init());
  LAPIS_TRY((check_contig<lapis_memref1, 1>(pos, "pos")));
  LAPIS_TRY((check_contig<lapis_memref1, 1>(crd, "crd")));
  LAPIS_TRY((check_contig<lapis_memref1, 1>(val, "val")));
  LAPIS_TRY((check_contig<lapis_memref3, 3>(B, "B")));
  if (spec == nullptr) return fail(LAPIS_EBADARG, "null storage specifier");
  if (ret0 == nullptr || *ret0 == nullptr) return fail(LAPIS_EBADARG, "bspmm: null result slot");
  const int64_t n1 = spec->dims[0], n2 = spec->dims[1], nh = spec->dims[2];
  const int64_t npos = spec->mem_sizes[0], nnz = spec->mem_sizes[1], nval = spec->mem_sizes[2];
  if (n1 < 0 || n2 < 0 || nh < 0) return fail(LAPIS_EBADSHAPE, "negative tensor dimension");
  if (npos != n1 + 1 || pos->sizes[0] < npos) return fail(LAPIS_EBADSHAPE, "pos must have rows+1 entries");
  if (nval != nnz * nh || crd->sizes[0] < nnz || val->sizes[0] < nval)
    return fail(LAPIS_EBADSHAPE, "crd/val shorter than the specifier says");
  if (B->sizes[0] != n2 || B->sizes[2] != nh) return fail(LAPIS_EBADSHAPE, "bspmm: B must be [n2, dh, nh]");
  const int64_t dh = B->sizes[1];
  const I *hpos = elem_ptr<I>(pos), *hcrd = elem_ptr<I>(crd);
  cudaStream_t st = nullptr;
  Operands ops;
  const size_t bC = (size_t)n1 * dh * nh * 4;
  const int ppos = ops.up.add_pos(hpos, npos), pcrd = ops.up.add_crd(hcrd, nnz, n2);
  const int pval = ops.up.add(elem_ptr<float>(val), (size_t)nval * 4), pB = ops.up.add(elem_ptr<float>(B), (size_t)n2 * dh * nh * 4);
  Upload::Facts facts;
  LAPIS_TRY(ops.send(st, &facts, bC));
  LAPIS_TRY(check_facts<I>(facts, hpos, hcrd, n1, nnz, n2));
  LAPIS_TRY(lapis_b200_bspmm_csrv_f32((int)sizeof(I), n1, n2, nh, dh, ops.at<void>(ppos), ops.at<void>(pcrd), ops.at<float>(pval),
                                      ops.at<float>(pB), ops.extra<float>(), 0, st));
  float *hc = static_cast<float *>(std::malloc(bC > 0 ? bC : 8));
  if (hc == nullptr) return fail(LAPIS_ECUDA, "bspmm: host allocation failed");
  g_alive_host.push_back(hc);
  LAPIS_TRY(ops.finish(stage_download(hc, ops.extra<float>(), bC, st)));
  lapis_memref3 out;
  out.basePtr = hc;
  out.data = hc;
  out.offset = 0;
  out.sizes[0] = n1;
  out.sizes[1] = dh;
  out.sizes[2] = nh;
  out.strides[0] = dh * nh;
  out.strides[1] = nh;
  out.strides[2] = 1;
  **ret0 = out;
  return LAPIS_OK;
}

// examples/spmm_dcsr_opdsl.py:59-101, call at :160 (decomposed arguments)
template <typename I>
static int spmm_dcsr_host(lapis_memref2 **ret0, lapis_memref1 *p1, lapis_memref1 *i1, lapis_memref1 *p2, lapis_memref1 *i2,
                          lapis_memref1 *val, const lapis_dcsr_spec *spec, lapis_memref2 *B, lapis_memref2 *C) {
  clear_error();
  LAPIS_TRY(require_init());
  LAPIS_TRY((check_contig<lapis_memref1, 1>(p1, "p1")));
  LAPIS_TRY((check_contig<lapis_memref1, 1>(i1, "i1")));
  LAPIS_TRY((check_contig<lapis_memref1, 1>(p2, "p2")));
  LAPIS_TRY((check_contig<lapis_memref1, 1>(i2, "i2")));
  LAPIS_TRY((check_contig<lapis_memref1, 1>(val, "val")));
  LAPIS_TRY((check_contig<lapis_memref2, 2>(B, "B")));
  LAPIS_TRY((check_contig<lapis_memref2, 2>(C, "C")));
  if (spec == nullptr) return fail(LAPIS_EBADARG, "null storage specifier");
  const int64_t nrows = spec->dims[0], ncols = spec->dims[1];
  const int64_t nstored = spec->mem_sizes[1], nnz = spec->mem_sizes[4];
  if (nrows < 0 || ncols < 0) return fail(LAPIS_EBADSHAPE, "negative matrix dimension");
  if (spec->mem_sizes[0] != 2 || p1->sizes[0] < 2 || spec->mem_sizes[2] != nstored + 1 || p2->sizes[0] < nstored + 1 ||
      i1->sizes[0] < nstored || spec->mem_sizes[3] != nnz || i2->sizes[0] < nnz || val->sizes[0] < nnz)
    return fail(LAPIS_EBADSHAPE, "spmm_dcsr: buffers do not match the specifier");
  const int64_t k = B->sizes[1];
  if (B->sizes[0] != ncols || C->sizes[0] != nrows || C->sizes[1] != k) return fail(LAPIS_EBADSHAPE, "spmm_dcsr: B/C shape mismatch");
  const I *hp1 = elem_ptr<I>(p1), *hi1 = elem_ptr<I>(i1), *hp2 = elem_ptr<I>(p2), *hi2 = elem_ptr<I>(i2);
  if (hp1[0] != 0 || (int64_t)hp1[1] != nstored) return fail(LAPIS_EBADSHAPE, "spmm_dcsr: p1 must be {0, stored rows}");
  for (int64_t r = 0; r < nstored; ++r)  // ascending row numbers: equal ones are adjacent and one warp takes the run
    if (hi1[r] < 0 || (int64_t)hi1[r] >= nrows || (r > 0 && hi1[r] < hi1[r - 1]))
      return fail(LAPIS_EBADSHAPE, "spmm_dcsr: stored row numbers must ascend within [0, rows)");
  cudaStream_t st = nullptr;
  Operands ops;
  const size_t bC = (size_t)nrows * k * 8;
  const int pi1 = ops.up.add(hi1, (size_t)nstored * sizeof(I)), pp2 = ops.up.add_pos(hp2, nstored + 1);
  const int pi2 = ops.up.add_crd(hi2, nnz, ncols), pval = ops.up.add(elem_ptr<double>(val), (size_t)nnz * 8);
  const int pB = ops.up.add(elem_ptr<double>(B), (size_t)ncols * k * 8), pC = ops.up.add(elem_ptr<double>(C), bC);
  Upload::Facts facts;
  LAPIS_TRY(ops.send(st, &facts));
  LAPIS_TRY(check_facts<I>(facts, hp2, hi2, nstored, nnz, ncols));
  LAPIS_TRY(lapis_b200_spmm_dcsr_f64((int)sizeof(I), nrows, ncols, nstored, k, ops.at<void>(pi1), ops.at<void>(pp2), ops.at<void>(pi2),
                                     ops.at<double>(pval), ops.at<double>(pB), ops.at<double>(pC), st));
  LAPIS_TRY(ops.finish(stage_download(elem_ptr<double>(C), ops.at<double>(pC), bC, st)));
  if (ret0 != nullptr && *ret0 != nullptr) **ret0 = *C;
  return LAPIS_OK;
}

}  // namespace lapis_b200

using namespace lapis_b200;

extern "C" int lapis_last_error(void) { return g_status; }
extern "C" const char *lapis_last_error_message(void) { return g_message; }

extern "C" void lapis_initialize(void) {
  clear_error();
  int ndev = 0;
  cudaError_t e = cudaGetDeviceCount(&ndev);
  if (e != cudaSuccess || ndev <= 0) {
    fail(LAPIS_ECUDA, "lapis_initialize: no usable CUDA device (%s); this library has no CPU path",
         e != cudaSuccess ? cudaGetErrorString(e) : "device count is 0");
    return;
  }
  e = cudaFree(nullptr);  // brings the primary context up, as Kokkos::initialize does (:4289)
  if (e != cudaSuccess) {
    fail(LAPIS_ECUDA, "lapis_initialize: %s", cudaGetErrorString(e));
    return;
  }
  ++g_init_count;
}

extern "C" void lapis_finalize(void) {
  clear_error();
  if (g_init_count <= 0) {
    pool_trim();  // a program that holds matrix handles only gives idle memory back this way
    return;
  }
  if (--g_init_count == 0) {
    for (void *p : g_alive_host) std::free(p);
    g_alive_host.clear();
    cudaDeviceSynchronize();
    pool_trim();
  }
}

extern "C" void py_spmv_f64_i32(lapis_memref1 **ret0, lapis_memref1 *pos, lapis_memref1 *crd, lapis_memref1 *val,
                                const lapis_csr_spec *spec, lapis_memref1 *x, lapis_memref1 *y) {
  spmv_host<int32_t>(ret0, pos, crd, val, spec, x, y);
}
extern "C" void py_spmv_f64_i64(lapis_memref1 **ret0, lapis_memref1 *pos, lapis_memref1 *crd, lapis_memref1 *val,
                                const lapis_csr_spec *spec, lapis_memref1 *x, lapis_memref1 *y) {
  spmv_host<int64_t>(ret0, pos, crd, val, spec, x, y);
}
extern "C" void py_spmm_f64_i32(lapis_memref2 **ret0, lapis_memref1 *pos, lapis_memref1 *crd, lapis_memref1 *val,
                                const lapis_csr_spec *spec, lapis_memref2 *B, lapis_memref2 *C) {
  spmm_host<int32_t>(ret0, pos, crd, val, spec, B, C);
}
extern "C" void py_spmm_f64_i64(lapis_memref2 **ret0, lapis_memref1 *pos, lapis_memref1 *crd, lapis_memref1 *val,
                                const lapis_csr_spec *spec, lapis_memref2 *B, lapis_memref2 *C) {
  spmm_host<int64_t>(ret0, pos, crd, val, spec, B, C);
}

extern "C" void py_matmul_f32(lapis_memref2 **ret0, lapis_memref2 *A, lapis_memref2 *B, lapis_memref2 *C) {
  clear_error();
  if (require_init() != LAPIS_OK) return;
  if (check_contig<lapis_memref2, 2>(A, "A") || check_contig<lapis_memref2, 2>(B, "B") ||
      check_contig<lapis_memref2, 2>(C, "C"))
    return;
  // cf.assert of benchmarks/gemm/gemm.mlir:10-11
  if (A->sizes[1] != B->sizes[0]) {
    fail(LAPIS_EBADSHAPE, "mismatching contracting dimension for torch.aten.mm");
    return;
  }
  if (C->sizes[0] != A->sizes[0] || C->sizes[1] != B->sizes[1]) {
    fail(LAPIS_EBADSHAPE, "matmul: output shape mismatch");
    return;
  }
  if (gemm_host(1, A->sizes[0], B->sizes[1], A->sizes[1], elem_ptr<float>(A), elem_ptr<float>(B), elem_ptr<float>(C)))
    return;
  if (ret0 != nullptr && *ret0 != nullptr) **ret0 = *C;
}

extern "C" void py_batch_matmul_f32(lapis_memref3 **ret0, lapis_memref3 *A, lapis_memref3 *B, lapis_memref3 *C) {
  clear_error();
  if (require_init() != LAPIS_OK) return;
  if (check_contig<lapis_memref3, 3>(A, "A") || check_contig<lapis_memref3, 3>(B, "B") ||
      check_contig<lapis_memref3, 3>(C, "C"))
    return;
  // cf.assert pair of benchmarks/batched_gemm/batched_gemm.mlir:14-20
  if (A->sizes[0] != B->sizes[0] || A->sizes[2] != B->sizes[1]) {
    fail(LAPIS_EBADSHAPE, "mismatching contracting dimension");
    return;
  }
  if (C->sizes[0] != A->sizes[0] || C->sizes[1] != A->sizes[1] || C->sizes[2] != B->sizes[2]) {
    fail(LAPIS_EBADSHAPE, "batch_matmul: output shape mismatch");
    return;
  }
  if (gemm_host(A->sizes[0], A->sizes[1], B->sizes[2], A->sizes[2], elem_ptr<float>(A), elem_ptr<float>(B),
                elem_ptr<float>(C)))
    return;
  if (ret0 != nullptr && *ret0 != nullptr) **ret0 = *C;
}

extern "C" void py_pcg_f64_i32(lapis_memref1 **ret0, size_t *ret1, double *ret2, lapis_memref1 *pos,
                               lapis_memref1 *crd, lapis_memref1 *val, const lapis_csr_spec *spec, lapis_memref1 *b,
                               lapis_memref1 *dinv, double tol, size_t maxiter) {
  pcg_host<int32_t>(ret0, ret1, ret2, pos, crd, val, spec, b, dinv, tol, maxiter);
}
extern "C" void py_pcg_f64_i64(lapis_memref1 **ret0, size_t *ret1, double *ret2, lapis_memref1 *pos,
                               lapis_memref1 *crd, lapis_memref1 *val, const lapis_csr_spec *spec, lapis_memref1 *b,
                               lapis_memref1 *dinv, double tol, size_t maxiter) {
  pcg_host<int64_t>(ret0, ret1, ret2, pos, crd, val, spec, b, dinv, tol, maxiter);
}

extern "C" void py_mht_f64_i32(lapis_memref1 **ret0, lapis_memref1 **ret1, lapis_memref1 *pos, lapis_memref1 *crd,
                               lapis_memref1 *val, const lapis_csr_spec *spec, lapis_memref1 *mask, lapis_memref1 *d,
                               double alpha, double tol, size_t maxiter) {
  mht_host<int32_t>(ret0, ret1, pos, crd, val, spec, mask, d, alpha, tol, maxiter);
}
extern "C" void py_mht_f64_i64(lapis_memref1 **ret0, lapis_memref1 **ret1, lapis_memref1 *pos, lapis_memref1 *crd,
                               lapis_memref1 *val, const lapis_csr_spec *spec, lapis_memref1 *mask, lapis_memref1 *d,
                               double alpha, double tol, size_t maxiter) {
  mht_host<int64_t>(ret0, ret1, pos, crd, val, spec, mask, d, alpha, tol, maxiter);
}
extern "C" void py_normalize_mom2_f64(lapis_memref1 **ret0, lapis_memref1 *mom1, lapis_memref1 *mom2) {
  normalize_mom2_host(ret0, mom1, mom2);
}

extern "C" void py_bspmm_f32_i32(lapis_memref3 **ret0, lapis_memref1 *pos, lapis_memref1 *crd, lapis_memref1 *val,
                                 const lapis_csrv_spec *spec, lapis_memref3 *B) {
  bspmm_host<int32_t>(ret0, pos, crd, val, spec, B);
}
extern "C" void py_bspmm_f32_i64(lapis_memref3 **ret0, lapis_memref1 *pos, lapis_memref1 *crd, lapis_memref1 *val,
                                 const lapis_csrv_spec *spec, lapis_memref3 *B) {
  bspmm_host<int64_t>(ret0, pos, crd, val, spec, B);
}
extern "C" void py_spmm_dcsr_f64_i32(lapis_memref2 **ret0, lapis_memref1 *p1, lapis_memref1 *i1, lapis_memref1 *p2,
                                     lapis_memref1 *i2, lapis_memref1 *val, const lapis_dcsr_spec *spec,
                                     lapis_memref2 *B, lapis_memref2 *C) {
  spmm_dcsr_host<int32_t>(ret0, p1, i1, p2, i2, val, spec, B, C);
}
extern "C" void py_spmm_dcsr_f64_i64(lapis_memref2 **ret0, lapis_memref1 *p1, lapis_memref1 *i1, lapis_memref1 *p2,
                                     lapis_memref1 *i2, lapis_memref1 *val, const lapis_dcsr_spec *spec,
                                     lapis_memref2 *B, lapis_memref2 *C) {
  spmm_dcsr_host<int64_t>(ret0, p1, i1, p2, i2, val, spec, B, C);
}

// ---- host-side partition rule ------------------------------------------------
template <typename I>
static void partition_rows(int64_t nrows, const I *pos, int G, int64_t *bounds) {
  const int64_t base = (int64_t)pos[0];
  const int64_t nnz = (int64_t)pos[nrows] - base;
  for (int g = 0; g <= G; ++g) {
    if (g == G) {
      bounds[g] = nrows;
      continue;
    }
    const int64_t target = base + (int64_t)(((__int128)nnz * g) / G);
    int64_t lo = 0, hi = nrows;
    while (lo < hi) {
      const int64_t mid = lo + (hi - lo) / 2;
      if ((int64_t)pos[mid] < target)
        lo = mid + 1;
      else
        hi = mid;
    }
    bounds[g] = lo;
  }
}

extern "C" int lapis_b200_validate_csr_host(int idx_bytes, int64_t nrows, int64_t ncols, int64_t nnz, const void *pos,
                                           const void *crd) {
  clear_error();
  if ((idx_bytes != 4 && idx_bytes != 8) || nrows < 0 || ncols < 0 || nnz < 0 || pos == nullptr || (nnz > 0 && crd == nullptr))
    return fail(LAPIS_EBADARG, "validate_csr_host: bad arguments");
  if (idx_bytes == 4) {
    LAPIS_TRY(check_pos_host<int32_t>(static_cast<const int32_t *>(pos), nrows, nnz));
    return check_crd_host<int32_t>(static_cast<const int32_t *>(crd), nnz, ncols);
  }
  LAPIS_TRY(check_pos_host<int64_t>(static_cast<const int64_t *>(pos), nrows, nnz));
  return check_crd_host<int64_t>(static_cast<const int64_t *>(crd), nnz, ncols);
}

extern "C" int lapis_b200_partition_rows(int idx_bytes, int64_t nrows, const void *pos, int G, int64_t *bounds) {
  clear_error();
  if (pos == nullptr || bounds == nullptr || G < 1 || nrows < 0) return fail(LAPIS_EBADARG, "partition_rows: bad arguments");
  if (idx_bytes == 4)
    partition_rows<int32_t>(nrows, static_cast<const int32_t *>(pos), G, bounds);
  else if (idx_bytes == 8)
    partition_rows<int64_t>(nrows, static_cast<const int64_t *>(pos), G, bounds);
  else
    return fail(LAPIS_EBADARG, "partition_rows: idx_bytes must be 4 or 8");
  return LAPIS_OK;
}
