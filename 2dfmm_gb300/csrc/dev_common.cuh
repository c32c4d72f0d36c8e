// Device helpers shared by the kernels.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "internal.h"

#define T2D_CUDA_TRY(expr)                            \
  do {                                                \
    cudaError_t e_ = (expr);                          \
    if (e_ != cudaSuccess) {                          \
      ::t2d::note_cuda_error(e_, #expr);              \
      return TREE2D_ERR_CUDA;                         \
    }                                                 \
  } while (0)

namespace t2d {

// The kernels of a solve follow one another on a stream, each short in a small
// solve, and a plain launch begins 2.7 us later than it needs to: it waits for
// the kernel before it to be finished and flushed before its own blocks are
// set up (200 launches in a row: 4.1 us each, so launched 1.4 us).  chained()
// lets a kernel's blocks start once those of the kernel before have ended
// (programmatic stream serialization); chain_wait(), the first statement of
// every such kernel, then waits until that kernel is complete and its writes
// are visible.  As every kernel of the chain waits, completion carries over
// from kernel to kernel.  A kernel launched without the attribute passes
// chain_wait() at once.  Whole solves: static plain of 4,096 blobs 299 -> 261
// us, mixed of 50,000 516 -> 424 us, learned of 1M 1.82 -> 1.73 ms, 20 training
// steps 1.56 -> 1.43 ms.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P>
struct Chained {
  void (*kernel)(P...);
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
  // an error stays for cudaGetLastError, as after a plain launch
  template <class... A>
  void operator()(A &&...args) const {
    cudaLaunchConfig_t c{};
    c.gridDim = grid, c.blockDim = block, c.dynamicSmemBytes = smem, c.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    c.attrs = attr, c.numAttrs = 1;
    (void)cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
  }
};
template <class... P>
Chained<P...> chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
  return {kernel, grid, block, smem, stream};
}

__device__ __forceinline__ void set_err(DevStatus *st, int code) { atomicCAS(&st->err, 0, code); }

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }

__device__ __forceinline__ double2 shfl_d2(double2 v, int src) {
  return make_double2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

// 1/x for a positive normal x: the SFU's approximate reciprocal refined by
// two Newton-Raphson steps for f(y) = 1/y - x, y <- y + y (1 - x y), each
// with the residual 1 - x y formed by one FMA.
__device__ __forceinline__ double rcp_nr(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(y, fma(-x, y, 1.0), y);
  y = fma(y, fma(-x, y, 1.0), y);
  return y;
}

// Tests on a double's bits: FP64 comparisons run at 1/64 of the integer rate.
__device__ __forceinline__ bool finite_bits(double v) {
  return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000;
}
__device__ __forceinline__ bool nan_bits(double v) {
  return (unsigned long long)(__double_as_longlong(v) & 0x7fffffffffffffffll) > 0x7ff0000000000000ull;
}

// Number of leading base-4 digits shared by two keys (32 if equal).
__device__ __forceinline__ int common_levels(uint64_t a, uint64_t b) {
  uint64_t d = a ^ b;
  return d == 0 ? kKeyLevels : (__clzll(d) >> 1);
}

}  // namespace t2d
