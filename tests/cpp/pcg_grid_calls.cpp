// The host side of pcg_grid.cu over a stand-in CUDA runtime that refuses the cooperative launch.  Prints "ok" and returns 0.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "../../lapis_b200/csrc/common.h"

static cudaError_t g_answer = cudaSuccess, g_last = cudaSuccess;
static int g_launches = 0, g_done = 1;

extern "C" {
void **__cudaRegisterFatBinary(void *) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st *) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *, dim3 *, size_t *, void *) { return cudaSuccess; }
cudaError_t __cudaGetKernel(cudaKernel_t *, const void *) { return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void **, size_t, cudaStream_t) { return cudaSuccess; }
char __cudaInitModule(void **) { return 0; }
cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaLaunchCooperativeKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t) {
  ++g_launches;
  return g_last = g_answer;
}
cudaError_t cudaGetLastError(void) {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
const char *cudaGetErrorString(cudaError_t) { return "stand-in error"; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 1, cudaSuccess; }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { return std::memset(p, v, n), cudaSuccess; }
cudaError_t cudaFree(void *p) { return std::free(p), cudaSuccess; }
int lapis_b200_pcg_status(void *, int *done, uint64_t *iters, double *relres, void *) {
  *done = g_done;
  *iters = 7;
  *relres = 0.5;
  return LAPIS_OK;
}
}

namespace lapis_b200 {
int fail(int code, const char *, ...) { return code; }
int sm_count() { return 148; }
int pool_alloc(void **p, size_t bytes, cudaStream_t) { return *p = std::malloc(bytes), LAPIS_OK; }
void pool_free(void *p, cudaStream_t) { std::free(p); }
int large_alloc(void **p, size_t bytes) { return *p = std::malloc(bytes), LAPIS_OK; }
int pcg_grid(const lapis_b200_csr *h, const double *d_b, const double *d_dinv, double tol, uint64_t maxiter, double *d_x, uint64_t *iters,
             double *relres, bool *solved, cudaStream_t st);
}  // namespace lapis_b200

#define EXPECT(cond)                                                        \
  do {                                                                      \
    if (!(cond)) return std::printf("line %d: %s\n", __LINE__, #cond), 1; \
  } while (0)

int main() {
  lapis_b200_csr h = {};
  h.nrows = h.ncols = 20000;
  h.nnz = 100000;
  uint64_t iters = 0;
  double relres = 0.0;
  bool solved = false;
  for (const int idx_bytes : {4, 8}) {
    h.idx_bytes = idx_bytes;
    g_answer = cudaSuccess;
    g_done = 1;
    EXPECT(lapis_b200::pcg_grid(&h, nullptr, nullptr, 0.0, 10, nullptr, &iters, &relres, &solved, nullptr) == LAPIS_OK);
    EXPECT(solved && iters == 7 && relres == 0.5);
    for (const cudaError_t refusal : {cudaErrorCooperativeLaunchTooLarge, cudaErrorLaunchOutOfResources, cudaErrorNotSupported}) {
      g_answer = refusal;
      g_launches = 0;
      solved = true;
      EXPECT(lapis_b200::pcg_grid(&h, nullptr, nullptr, 0.0, 10, nullptr, &iters, &relres, &solved, nullptr) == LAPIS_OK);
      EXPECT(!solved && g_launches == 1 && g_last == cudaSuccess);
    }
    g_answer = cudaErrorInvalidValue;  // any other error is one
    EXPECT(lapis_b200::pcg_grid(&h, nullptr, nullptr, 0.0, 10, nullptr, &iters, &relres, &solved, nullptr) == LAPIS_ECUDA);
  }
  std::puts("ok");
  return 0;
}
