// Shared helpers of libbrick_gb300: status handling, element types, layout math.
#pragma once

#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include <string>

#include "bricklib_gb300.h"

namespace bk {

// ---------------------------------------------------------------- status

void set_error(const std::string &msg);
int fail(int status, const std::string &msg);
int cuda_fail(cudaError_t e, const char *what);

#define BK_CUDA(call)                                   \
  do {                                                  \
    cudaError_t e_ = (call);                            \
    if (e_ != cudaSuccess) return bk::cuda_fail(e_, #call); \
  } while (0)

inline cudaStream_t as_stream(void *s) { return reinterpret_cast<cudaStream_t>(s); }

// Device word of error flags, one per device, set by kernels with atomicOr.
int *device_error_word();
constexpr int FLAG_BOUNDS = 1;
constexpr int FLAG_TIMEOUT = 2;

// Launch of a kernel that begins with grid_begin(): it is brought up, as far as it needs no global
// memory, while the stream's previous kernel ends (programmatic dependent launch).  Sweeps in a row,
// us each, without / with it: 7-point Laplacian 128^3 32.0 / 29.8, heat step 128^3 15.9 / 13.7 and 256^3
// 77.2 / 74.8.  Inside a stream capture, where the previous node need not be a kernel, an ordinary
// launch.
template <class... P, class... A>
cudaError_t launch_overlapped(void (*kern)(P...), unsigned grid, unsigned threads, size_t smem, cudaStream_t s, const A &...args) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  const cudaError_t asked = cudaStreamIsCapturing(s, &cap);
  const bool eager = asked == cudaSuccess && cap == cudaStreamCaptureStatusNone;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = eager ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, P(args)...);
  // the caller has the error: it is not left as the thread's last one, by which plain launches are checked
  if (asked != cudaSuccess || e != cudaSuccess) (void)cudaGetLastError();
  return e;
}

// The CTAs of `threads` threads and `smem` bytes of dynamic shared memory that the current device
// holds at a time: `sms` and resident CTAs per SM of a kernel.  Asked of the runtime once per
// kernel, device and size (the queries took about as long as a launch); lets the kernel use that
// much shared memory.
int kernel_fit(const void *kern, int threads, size_t smem, int *sms, int *per_sm, const char *what);

inline size_t dtype_size(int dt) { return dt == BK_F64 ? 8 : dt == BK_F32 ? 4 : 2; }
inline bool dtype_ok(int dt) { return dt == BK_F64 || dt == BK_F32 || dt == BK_BF16; }

// ---------------------------------------------------------------- element types

// First in a kernel, before any access to global memory: waits until the stream's previous kernel is
// through and its writes are visible.  Every thread calls it, so a grid never ends before the one it
// waits for.  (No early trigger, griddepcontrol.launch_dependents: with it the next grid's CTAs
// took the places of the first ones to end and the 7-point Laplacian at 128^3 went from 29.8 to
// 32.7 us a sweep, the 125-point cube at 512^3 from 2272 to 2329.)
__device__ __forceinline__ void grid_begin() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

template <typename T> struct Elem;
template <> struct Elem<double> {
  typedef double acc;
  static __device__ __forceinline__ double load(const double *p) { return __ldg(p); }
  static __device__ __forceinline__ void store(double *p, double v) { *p = v; }
};
template <> struct Elem<float> {
  typedef float acc;
  static __device__ __forceinline__ float load(const float *p) { return __ldg(p); }
  static __device__ __forceinline__ void store(float *p, float v) { *p = v; }
};
template <> struct Elem<__nv_bfloat16> {
  typedef float acc;
  static __device__ __forceinline__ float load(const __nv_bfloat16 *p) { return __bfloat162float(*p); }
  static __device__ __forceinline__ void store(__nv_bfloat16 *p, float v) { *p = __float2bfloat16_rn(v); }
};

// ---------------------------------------------------------------- layout

// In-brick offset of element (k,j,i) for brick dims B and fold F (all (k,j,i)).
struct Layout {
  int bk, bj, bi, fk, fj, fi;
  __host__ __device__ __forceinline__ int offset(int k, int j, int i) const {
    const int vl = fk * fj * fi;
    const int vec = ((k / fk) * (bj / fj) + j / fj) * (bi / fi) + i / fi;
    const int lane = ((k % fk) * fj + j % fj) * fi + i % fi;
    return vec * vl + lane;
  }
  __host__ __device__ __forceinline__ int size() const { return bk * bj * bi; }
  // true when offset(k,j,i) == (k*bj + j)*bi + i for every element: along i the fold spans the brick
  // or is the only one with more than one element, along j likewise for what remains
  __host__ bool row_major() const { return fi == bi ? fj == bj || fk == 1 : fj == 1 && fk == 1; }
};

int check_layout(const bk_layout *lay, Layout *out);
int check_field(const bk_field *f, const Layout &L, const char *name);
int check_disjoint(const bk_field *in, const bk_field *out, size_t brick_elems);

}  // namespace bk
