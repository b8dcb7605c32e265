// The calls on host arrays (abi.cu, stage.cu) over a stand-in CUDA runtime in which device memory is host memory, and
// stand-ins for the kernels: what they do before a launch and after one, on a machine without a GPU.
//
//   host_calls <scenario>     prints "ok" and returns 0, or names what did not hold
#include <csignal>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <mutex>
#include <new>
#include <set>
#include <string>
#include <vector>

#include <dlfcn.h>
#include <pthread.h>
#include <sys/wait.h>
#include <unistd.h>

#include "../../lapis_b200/csrc/abi.cu"
#include "../../lapis_b200/csrc/stage.cu"

#define EXPECT(cond)                                                              \
  do {                                                                            \
    if (!(cond)) {                                                                \
      std::printf("%s:%d: %s does not hold (last error: %d %s)\n", __FILE__, __LINE__, #cond, lapis_last_error(), \
                  lapis_last_error_message());                                    \
      std::exit(1);                                                               \
    }                                                                             \
  } while (0)

// ---- the stand-in runtime ----------------------------------------------------------------------------------------
static std::mutex g_fake;
static std::set<void *> g_device, g_locked;  // live device allocations, page-locked host blocks
static int g_copies = 0, g_waited = 0;       // copies from page-locked memory so far; how many of them were waited for
static int g_launches = 0;                   // calls into the kernels
static int g_kernel_status = LAPIS_OK;       // what the kernels return
static size_t g_idle = 0, g_keep = 0;        // what the pool holds freed, what it may hold
static bool g_full = false;                  // the device has no room but what the pool holds idle
static std::vector<char *> g_page_locked;    // blocks of a caller, LOCKED_BYTES each
constexpr size_t LOCKED_BYTES = size_t(4) << 20;

// The allocation in so many allocations of this thread fails (0: none), and so does every start of a thread.
static thread_local int g_fail_alloc = 0;
static bool g_no_threads = false;
void *operator new(size_t n) {
  if (g_fail_alloc > 0 && --g_fail_alloc == 0) throw std::bad_alloc();
  return std::malloc(n);
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }
extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *arg) {
  if (g_no_threads) return EAGAIN;
  return reinterpret_cast<decltype(&pthread_create)>(dlsym(RTLD_NEXT, "pthread_create"))(t, a, f, arg);
}
struct NoFailure {  // the stand-ins themselves keep their memory
  int saved = g_fail_alloc;
  NoFailure() { g_fail_alloc = 0; }
  ~NoFailure() { g_fail_alloc = saved; }
};

static bool of_caller(const void *p) {
  for (char *b : g_page_locked)
    if (p >= b && p < b + LOCKED_BYTES) return true;
  return false;
}

extern "C" {
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 148, cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "stand-in error"; }
cudaError_t cudaMalloc(void **p, size_t n) {
  NoFailure keep;
  std::lock_guard<std::mutex> l(g_fake);
  if (g_full && g_idle > 0) return cudaErrorMemoryAllocation;
  *p = std::malloc(n);
  g_device.insert(*p);
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  std::lock_guard<std::mutex> l(g_fake);
  if (p != nullptr) EXPECT(g_device.erase(p) == 1);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t *pool, const cudaMemPoolProps *) { return *pool = (cudaMemPool_t)1, cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *v) { return g_keep = *static_cast<uint64_t *>(v), cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return g_idle = 0, cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
  NoFailure keep;
  std::lock_guard<std::mutex> l(g_fake);
  *p = std::aligned_alloc(4096, n);
  g_locked.insert(*p);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
  std::lock_guard<std::mutex> l(g_fake);
  EXPECT(g_locked.erase(p) == 1);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
  NoFailure keep;
  *e = reinterpret_cast<cudaEvent_t>(new int(0));  // an event: the copies in front of it
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete reinterpret_cast<int *>(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
  std::lock_guard<std::mutex> l(g_fake);
  *reinterpret_cast<int *>(e) = g_copies;
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  std::lock_guard<std::mutex> l(g_fake);
  g_waited = std::max(g_waited, *reinterpret_cast<int *>(e));
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
  a->type = of_caller(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *to, const void *from, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(to, from, n);
  std::lock_guard<std::mutex> l(g_fake);
  if (of_caller(from)) ++g_copies;
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
  std::lock_guard<std::mutex> l(g_fake);
  g_waited = g_copies;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) { return cudaStreamSynchronize(nullptr); }

// ---- the stand-in kernels: y = A x and C = A B on the host, the others only count ---------------------------------
static int launched() {
  __atomic_add_fetch(&g_launches, 1, __ATOMIC_SEQ_CST);
  return g_kernel_status == LAPIS_OK ? LAPIS_OK : lapis_b200::fail(g_kernel_status, "as asked");
}
int lapis_b200_spmv_f64(lapis_b200_csr_t h, const double *x, double *y, int, void *) {
  for (int64_t r = 0; h->idx_bytes == 8 && g_kernel_status == LAPIS_OK && r < h->nrows; ++r) {
    const int64_t *pos = static_cast<const int64_t *>(h->pos), *crd = static_cast<const int64_t *>(h->crd);
    for (int64_t j = pos[r]; j < pos[r + 1]; ++j) y[r] += h->val[j] * x[crd[j]];
  }
  return launched();
}
int lapis_b200_spmm_f64(lapis_b200_csr_t, int64_t, const double *, double *, int, void *) { return launched(); }
int lapis_b200_bgemm_f32(int64_t, int64_t, int64_t, int64_t, const float *, const float *, float *, void *) { return launched(); }
int lapis_b200_bgemm_status(void *) { return LAPIS_OK; }
int lapis_b200_pcg_f64(lapis_b200_csr_t, const double *, const double *, double, uint64_t, double *, uint64_t *, double *, void *) {
  return launched();
}
int lapis_b200_mht_f64(lapis_b200_csr_t, const double *, const double *, double, double, uint64_t, double *, double *, uint64_t *,
                       double *, void *) {
  return launched();
}
int lapis_b200_normalize_mom2_f64(int64_t, const double *, const double *, double *, void *) { return launched(); }
int lapis_b200_bspmm_csrv_f32(int, int64_t, int64_t, int64_t, int64_t, const void *, const void *, const float *, const float *, float *,
                              int, void *) {
  return launched();
}
int lapis_b200_spmm_dcsr_f64(int, int64_t, int64_t, int64_t, int64_t, const void *, const void *, const void *, const double *,
                             const double *, double *, void *) {
  return launched();
}
}  // extern "C"

namespace lapis_b200 {
int csr_setup(lapis_b200_csr *h, int idx_bytes, int64_t nrows, int64_t ncols, int64_t base, int64_t nnz, int64_t max_row_len,
              const void *pos, const void *crd, const double *val, bool, PoolBuf *, cudaStream_t) {
  *h = lapis_b200_csr{};
  h->idx_bytes = idx_bytes;
  h->nrows = nrows;
  h->ncols = ncols;
  h->base = base;
  h->nnz = nnz;
  h->max_row_len = max_row_len;
  h->pos = pos;
  h->crd = crd;
  h->val = val;
  return LAPIS_OK;
}
}  // namespace lapis_b200

// ---- scenarios ---------------------------------------------------------------------------------------------------
template <typename T>
static lapis_memref1 ref(std::vector<T> &v) {
  return {v.data(), v.data(), 0, {(int64_t)v.size()}, {1}};
}
static lapis_memref2 ref2(std::vector<double> &v, int64_t rows, int64_t cols) {
  return {v.data(), v.data(), 0, {rows, cols}, {cols, 1}};
}

// Offsets whose differences leave the index type: refused before any kernel, wherever in the array they are.
template <typename I>
static void offsets(void (*spmm)(lapis_memref2 **, lapis_memref1 *, lapis_memref1 *, lapis_memref1 *, const lapis_csr_spec *, lapis_memref2 *,
                                 lapis_memref2 *)) {
  const I top = std::numeric_limits<I>::max(), low = std::numeric_limits<I>::min();
  const std::vector<std::vector<I>> middles = {{top, -2}, {top, low, -5}, {low}, {-1}, {top, low + 1, low}, {7, 3}, {top}, {11}, {top, low, low + 1, -1}};
  const int64_t nnz = 10, per_block = 65536 / sizeof(I);
  for (int64_t at : {(int64_t)1, (int64_t)5, per_block - 1, per_block, 9 * per_block - 1, 20 * per_block})
    for (const auto &m : middles) {
      std::vector<I> pos(at, 0), crd(nnz, 0);
      pos.insert(pos.end(), m.begin(), m.end());
      pos.push_back((I)nnz);
      const int64_t rows = (int64_t)pos.size() - 1;
      std::vector<double> val(nnz, 1.0), B(3, 1.0), C(rows, 0.0);
      lapis_memref1 p = ref(pos), c = ref(crd), v = ref(val);
      lapis_memref2 b = ref2(B, 3, 1), out = ref2(C, rows, 1);
      const lapis_csr_spec spec = {{rows, 3}, {rows + 1, nnz, nnz}};
      spmm(nullptr, &p, &c, &v, &spec, &b, &out);
      EXPECT(lapis_last_error() == LAPIS_EBADSHAPE && g_launches == 0);
      for (size_t i = 0; i < m.size(); ++i) pos[at + i] = 4;  // the same array, mended
      spmm(nullptr, &p, &c, &v, &spec, &b, &out);
      EXPECT(lapis_last_error() == LAPIS_OK && g_launches == 1);
      g_launches = 0;
    }
}

// A call that fails behind the upload: page-locked operands, which are copied in place, are no longer being read when it
// returns.
template <typename T>
static T *page_locked_block() {
  g_page_locked.push_back(static_cast<char *>(std::aligned_alloc(4096, LOCKED_BYTES)));
  std::memset(g_page_locked.back(), 0, LOCKED_BYTES);
  return reinterpret_cast<T *>(g_page_locked.back());
}
static void in_flight() {
  const int64_t n = 200000;  // 1.6 MB a vector
  int64_t *pos = page_locked_block<int64_t>(), *crd = page_locked_block<int64_t>();
  double *val = page_locked_block<double>(), *x = page_locked_block<double>(), *y = page_locked_block<double>();
  for (int64_t i = 0; i <= n; ++i) pos[i] = i;
  int64_t two[2] = {0, n};
  lapis_memref1 p = {pos, pos, 0, {n + 1}, {1}}, c = {crd, crd, 0, {n}, {1}}, v = {val, val, 0, {n}, {1}}, p1 = {two, two, 0, {2}, {1}};
  lapis_memref1 xv = {x, x, 0, {n}, {1}}, yv = {y, y, 0, {n}, {1}}, i1 = {pos, pos, 0, {n}, {1}};
  lapis_memref2 xm = {x, x, 0, {n, 1}, {1, 1}}, ym = {y, y, 0, {n, 1}, {1, 1}}, one = {val, val, 0, {1, 1}, {1, 1}};
  lapis_memref3 xb = {x, x, 0, {n, 1, 1}, {1, 1, 1}}, ob;
  lapis_memref1 o1, o2, *r1 = &o1, *r2 = &o2;
  lapis_memref3 *r3 = &ob;
  const lapis_csr_spec spec = {{n, n}, {n + 1, n, n}};
  const lapis_csrv_spec vspec = {{n, n, 1}, {n + 1, n, n}};
  const lapis_dcsr_spec dspec = {{n, n}, {2, n, n + 1, n, n}};
  for (int status : {LAPIS_ECUDA, LAPIS_OK}) {
    g_kernel_status = status;
    auto after = [&](const char *call) {
      const bool quiet = g_copies > 0 && g_waited == g_copies;
      if (!quiet || lapis_last_error() != status) std::printf("%s: status %d\n", call, status);
      EXPECT(quiet && lapis_last_error() == status && g_launches == 1);
      g_launches = 0;
    };
    py_spmv_f64_i64(nullptr, &p, &c, &v, &spec, &xv, &yv), after("spmv");
    py_spmm_f64_i64(nullptr, &p, &c, &v, &spec, &xm, &ym), after("spmm");
    py_matmul_f32(nullptr, &xm, &one, &ym), after("matmul");
    py_pcg_f64_i64(&r1, nullptr, nullptr, &p, &c, &v, &spec, &xv, &yv, 0.0, 1), after("pcg");
    py_mht_f64_i64(&r1, &r2, &p, &c, &v, &spec, &xv, &yv, 0.5, 0.0, 1), after("mht");
    py_normalize_mom2_f64(&r1, &xv, &yv), after("normalize_mom2");
    py_bspmm_f32_i64(&r3, &p, &c, &v, &vspec, &xb), after("bspmm");
    py_spmm_dcsr_f64_i64(nullptr, &p1, &i1, &p, &c, &v, &dspec, &xm, &ym), after("spmm_dcsr");
  }
}

// y = A x with one entry a row, large enough for the helper threads.
struct Product {
  int64_t n;
  std::vector<int64_t> pos, crd;
  std::vector<double> val, x, y;
  explicit Product(int64_t rows) : n(rows), pos(rows + 1), crd(rows), val(rows), x(rows), y(rows) {
    for (int64_t i = 0; i < n; ++i) pos[i + 1] = i + 1, crd[i] = n - 1 - i, val[i] = 2.0, x[i] = (double)i;
  }
  int run() {
    std::fill(y.begin(), y.end(), 1.0);
    lapis_memref1 p = ref(pos), c = ref(crd), v = ref(val), xv = ref(x), yv = ref(y);
    const lapis_csr_spec spec = {{n, n}, {n + 1, n, n}};
    py_spmv_f64_i64(nullptr, &p, &c, &v, &spec, &xv, &yv);
    return lapis_last_error();
  }
  bool right() const {
    for (int64_t i = 0; i < n; ++i)
      if (y[i] != 1.0 + 2.0 * (double)(n - 1 - i)) return false;
    return true;
  }
};

// Memory and threads that cannot be had end a call with a status or slow it down; no exception leaves the C entry point.
static void exhausted() {
  Product a(300000);
  g_no_threads = true;
  EXPECT(a.run() == LAPIS_OK && a.right());
  g_no_threads = false;
  int failures = 0;
  for (int at = 1;; ++at) {
    g_fail_alloc = at;
    const int status = a.run();
    const bool reached = g_fail_alloc == 0;
    g_fail_alloc = 0;
    EXPECT(status == (reached ? LAPIS_ECUDA : LAPIS_OK));
    if (!reached) break;
    ++failures;
  }
  EXPECT(failures >= 4);
  EXPECT(a.run() == LAPIS_OK && a.right());
}

// A child process forked behind a large call exits.
static void fork_exit() {
  Product a(300000);
  EXPECT(a.run() == LAPIS_OK && a.right());
  const pid_t child = fork();
  if (child == 0) std::exit(0);
  int status = -1;
  for (int i = 0; i < 200 && waitpid(child, &status, WNOHANG) == 0; ++i) usleep(50000);
  if (status == -1) kill(child, SIGKILL);
  EXPECT(status == 0);
}

// Several threads in calls at once share one ring and one set of helpers.
static void threads() {
  std::vector<std::thread> pool;
  for (int t = 0; t < 4; ++t)
    pool.emplace_back([t] {
      Product a(1000 + 90000 * t);
      for (int i = 0; i < 25; ++i) EXPECT(a.run() == LAPIS_OK && a.right());
    });
  for (std::thread &t : pool) t.join();
}

// A device that is full but for what the pool holds idle: the call gets that memory, from the pool and beside it.
static void full_device() {
  Product small(1000), large(9000000);  // 300 MB of operands
  EXPECT(small.run() == LAPIS_OK && small.right());
  EXPECT(0 < g_keep && g_keep <= POOL_LARGEST);
  g_full = true;
  for (Product *a : {&small, &large}) {
    g_idle = g_keep;
    EXPECT(a->run() == LAPIS_OK && a->right() && g_idle == 0);
  }
  g_full = false;
  g_idle = g_keep;
  lapis_finalize();
  EXPECT(g_idle == 0);
  g_idle = g_keep;
  lapis_finalize();  // no module is alive: idle memory is given back all the same
  EXPECT(g_idle == 0);
  lapis_initialize();
}

int main(int argc, char **argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  lapis_initialize();
  if (what == "offsets") {
    offsets<int32_t>(py_spmm_f64_i32);
    offsets<int64_t>(py_spmm_f64_i64);
  } else if (what == "in_flight") {
    in_flight();
  } else if (what == "exhausted") {
    exhausted();
  } else if (what == "fork_exit") {
    fork_exit();
  } else if (what == "full_device") {
    full_device();
  } else if (what == "threads") {
    threads();
  } else {
    std::printf("unknown scenario '%s'\n", what.c_str());
    return 1;
  }
  lapis_finalize();
  EXPECT(g_device.empty());
  std::printf("ok\n");
  return 0;
}
