// A CUDA runtime that has no device, for tests of the host side on a machine without a GPU: loaded
// in front of libcudart (LD_PRELOAD), it answers the calls below as a healthy device would, makes
// the ones that a test asks for fail, counts the streams and events that are alive, and keeps the
// "last error" as the runtime does (set by a failing call, read and cleared by cudaGetLastError).
// Nothing is launched and no device memory exists.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <unistd.h>

static thread_local cudaError_t last = cudaSuccess;
static int fail_create = 0, fail_launch = 0, fail_malloc = 0;  // the n-th such call from now fails
static long live = 0;                                          // streams and events alive
static dim3 cfg_grid, cfg_block;
static size_t cfg_smem;
static cudaStream_t cfg_stream;

static cudaError_t answer(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
static bool fails(int &counter) { return counter > 0 && --counter == 0; }
static cudaError_t make(void **p) {
  if (fails(fail_create)) return answer(cudaErrorMemoryAllocation);
  *p = malloc(1);
  ++live;
  return cudaSuccess;
}
static cudaError_t drop(void *p) {
  if (!p) return answer(cudaErrorInvalidResourceHandle);
  free(p);
  --live;
  return cudaSuccess;
}

// kernel_fit of the library, called once more when the process is past the static destructors
typedef int (*Fit)(const void *, int, size_t, int *, int *, const char *);
static Fit fit;
static void late() {
  int sms = 0, per_sm = 0;
  const int st = fit(reinterpret_cast<const void *>(&late), 128, 1024, &sms, &per_sm, "late");
  const char ok[] = "fit after exit: ok\n", bad[] = "fit after exit: wrong\n";
  const bool good = st == 0 && sms == 152 && per_sm == 4;
  if (write(1, good ? ok : bad, (good ? sizeof ok : sizeof bad) - 1) < 0) _exit(9);
}

extern "C" {

void fake_fail(int create, int launch, int mallocs) {
  fail_create = create;
  fail_launch = launch;
  fail_malloc = mallocs;
}
long fake_live() { return live; }
int fake_fit_at_exit(Fit f) {
  fit = f;
  atexit(late);  // before the library's first use of its tables, so it runs after they are destroyed
  int sms = 0, per_sm = 0;
  return f(reinterpret_cast<const void *>(&late), 128, 1024, &sms, &per_sm, "first");
}

cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
cudaError_t cudaPeekAtLastError() { return last; }
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int, size_t) { return *n = 4, cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
  return *n = 4, cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) {
  if (fails(fail_malloc)) return answer(cudaErrorMemoryAllocation);
  return *p = calloc(1, n), cudaSuccess;
}
cudaError_t cudaFree(void *) { return cudaSuccess; }
cudaError_t cudaMemset(void *, int, size_t) { return cudaSuccess; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *, int) { return answer(cudaErrorNotSupported); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return make(reinterpret_cast<void **>(s)); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return drop(s); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return make(reinterpret_cast<void **>(e)); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return drop(e); }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) {
  return *s = cudaStreamCaptureStatusNone, cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) {
  cfg_grid = g;
  cfg_block = b;
  cfg_smem = smem;
  cfg_stream = s;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *s) {
  *g = cfg_grid;
  *b = cfg_block;
  *smem = cfg_smem;
  memcpy(s, &cfg_stream, sizeof cfg_stream);
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t) {
  return answer(fails(fail_launch) ? cudaErrorInvalidValue : cudaSuccess);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *, void **) {
  return answer(fails(fail_launch) ? cudaErrorInvalidValue : cudaSuccess);
}

}  // extern "C"
