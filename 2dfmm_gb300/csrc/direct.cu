// FP64 direct O(N*M) sum of the regularised Biot-Savart kernel: the yardstick
// of the approximate modes.  The pair kernel is direct_evaluate's
// (ver-c/src/fmm.c:121-142, r > 1e-10) applied to every source, in 64-bit
// fixed point (fix64.cuh).  Sources are staged through shared memory in tiles,
// decoded once; one thread per target.
#include "dev_common.cuh"
#include "fix64.cuh"
#include "position_hash.h"
#include "tc_ptx.cuh"

namespace t2d {
namespace {

constexpr int kThreads = 256;
constexpr double kPi = 3.14159265358979323846;

__device__ const fix::ExpTables g_exp = fix::make_exp_tables();

// A source as the pairs need it: |G| and 1/sigma^2 as mantissas and exponent
// fields (fix::mantissa), the upper word of G for its sign.  `odd`: a NaN or
// an infinity among its numbers (not a core radius of 0 or infinity), whose
// pairs run in FP64 so that they come out as they always did.
struct Source {
  double x, y;
  uint64_t gm, cm;
  int ge, ce;
  uint32_t gh;
  int odd;
};

// The pair in FP64: (r/sigma)^2 as r2 / sigma^2 and 1/r2 by a Newton-refined
// reciprocal; r > 1e-10 <=> r2 > 1e-20.
__device__ __noinline__ void pair64(double rx, double ry, double g, double rc, double &ax, double &ay) {
  const double ic = 1.0 / (rc * rc);
  const double r2 = rx * rx + ry * ry;
  if (r2 > 1.0e-20) {
    const double x2 = r2 * ic;
    const double e1 = x2 > 40.0 ? 1.0 : 1.0 - exp(-x2);
    const double rv = g * e1 * rcp_nr(r2);
    ax -= rv * ry;
    ay += rv * rx;
  }
}

// grid.y splits the sources into chunks; each block adds its partial sums
// into uv (zeroed by the caller) with FP64 atomics.  Bound by the dispatch of
// integer instructions (two cycles each, 117 per 32 pairs): 16,384 targets x
// 262,144 two-patch sources take 26.2 ms, 24.7 of them for that, and took 125 ms
// with the pairs in FP64.
__global__ void __launch_bounds__(kThreads) k_direct(int ntgt, const double *__restrict__ txy, int nsrc,
                                                     const double *__restrict__ sxy, const double *__restrict__ cir,
                                                     const double *__restrict__ cor, double *__restrict__ uv, int chunk,
                                                     fix::One one) {
  __shared__ Source src[kThreads];
  __shared__ uint64_t s_exp_int[fix::kExpInts], s_exp_frac[fix::kExpFracs];
  for (int j = threadIdx.x; j < fix::kExpFracs; j += kThreads) s_exp_frac[j] = g_exp.fracs[j];
  for (int j = threadIdx.x; j < fix::kExpInts; j += kThreads) s_exp_int[j] = g_exp.ints[j];
  const long i = blockIdx.x * (long)kThreads + threadIdx.x;
  const bool valid = i < ntgt;
  const double x = valid ? txy[2 * i] : 0.0, y = valid ? txy[2 * i + 1] : 0.0;
  int odd_target = !isfinite(x) || !isfinite(y);
  asm volatile("" : "+r"(odd_target));  // once: not as two FP64 comparisons per pair
  fix::SumXY sum;
  double ax = 0.0, ay = 0.0;  // the FP64 pairs
  const int s0 = blockIdx.y * chunk;
  const int s1 = min(nsrc, s0 + chunk);
  for (int base = s0; base < s1; base += kThreads) {
    const int j = base + threadIdx.x;
    __syncthreads();
    if (j < s1) {
      const double sx = sxy[2 * (long)j], sy = sxy[2 * (long)j + 1], g = cir[j], rc = cor[j];
      const double ic = 1.0 / (rc * rc);
      Source q;
      q.x = sx;
      q.y = sy;
      q.gm = fix::mantissa(g, q.ge);
      q.cm = fix::mantissa(ic, q.ce);
      q.gh = fix::hi32(fix::bits(g));
      q.odd = !isfinite(sx) || !isfinite(sy) || !isfinite(g) || isnan(rc);
      src[threadIdx.x] = q;
    }
    __syncthreads();
    const int cnt = min(kThreads, s1 - base);
    for (int k0 = 0; k0 < cnt; k0 += 32) {
      fix::settle(sum);
      const int k1 = min(cnt, k0 + 32);
      for (int k = k0; k < k1; k++) {
        const Source &q = src[k];
        const double rx = fix::minus(x, q.x);
        const double ry = fix::minus(y, q.y);
        const fix::Vec v = fix::vec(rx, ry);
        if (q.odd || odd_target || v.e == 0x7ff) {
          pair64(rx, ry, cir[base + k], cor[base + k], ax, ay);
          continue;
        }
        if (fix::apart(v, rx, ry))
          fix::add_pair(sum, v, fix::hi32(fix::bits(rx)), fix::hi32(fix::bits(ry)), q.gm, q.ge, q.gh, q.cm, q.ce,
                        s_exp_int, s_exp_frac, one);
      }
    }
  }
  if (valid) {
    ax += fix::to_double(sum.x.v, sum.x.l, sum.x.e);
    ay += fix::to_double(sum.y.v, sum.y.l, sum.y.e);
    atomicAdd(&uv[2 * i], 0.5 * ax / kPi);
    atomicAdd(&uv[2 * i + 1], 0.5 * ay / kPi);
  }
}

// FP32 pipe throughput probe: 8 independent FMA chains per thread.
__global__ void __launch_bounds__(256) k_ffma_probe(float *out, int iters, float b, float c) {
  float a0 = threadIdx.x * 1e-9f, a1 = a0 + 1e-3f, a2 = a0 + 2e-3f, a3 = a0 + 3e-3f;
  float a4 = a0 + 4e-3f, a5 = a0 + 5e-3f, a6 = a0 + 6e-3f, a7 = a0 + 7e-3f;
  for (int i = 0; i < iters; i++) {
    a0 = fmaf(a0, b, c);
    a1 = fmaf(a1, b, c);
    a2 = fmaf(a2, b, c);
    a3 = fmaf(a3, b, c);
    a4 = fmaf(a4, b, c);
    a5 = fmaf(a5, b, c);
    a6 = fmaf(a6, b, c);
    a7 = fmaf(a7, b, c);
  }
  float s = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
  if (s == 12345.678f) out[0] = s;
}

// FP64 pipe throughput probe: 8 independent FMA chains per thread.
__global__ void __launch_bounds__(256) k_dfma_probe(double *out, int iters, double b, double c) {
  double a0 = threadIdx.x * 1e-9, a1 = a0 + 1e-3, a2 = a0 + 2e-3, a3 = a0 + 3e-3;
  double a4 = a0 + 4e-3, a5 = a0 + 5e-3, a6 = a0 + 6e-3, a7 = a0 + 7e-3;
  for (int i = 0; i < iters; i++) {
    a0 = fma(a0, b, c);
    a1 = fma(a1, b, c);
    a2 = fma(a2, b, c);
    a3 = fma(a3, b, c);
    a4 = fma(a4, b, c);
    a5 = fma(a5, b, c);
    a6 = fma(a6, b, c);
    a7 = fma(a7, b, c);
  }
  double s = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
  if (s == 12345.678) out[0] = s;  // never true in practice; keeps the chains live
}

}  // namespace

// Bounded-wait check: lane 0 waits on a shared-memory mbarrier that nothing
// arrives on, with the same bounded poll the tensor-core kernels use, and
// records TREE2D_ERR_TIMEOUT when the wait gives up (1 = the wait ended,
// which no arrival can cause here).  The kernel always returns, so the
// context stays usable.
__global__ void k_wait_probe(long polls, int *out) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) *out = mbar_wait(&bar, 0, polls) ? 1 : TREE2D_ERR_TIMEOUT;
}

cudaError_t wait_probe(long polls, int *out, cudaStream_t s) {
  k_wait_probe<<<1, 32, 0, s>>>(polls, out);
  ::t2d::g_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

cudaError_t dfma_probe(double *out, int blocks, int iters, cudaStream_t s) {
  k_dfma_probe<<<blocks, 256, 0, s>>>(out, iters, 0.999999, 1e-7);
  ::t2d::g_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

// Forward Euler step of the blob positions, x += dt * u (the solver's drift,
// e_drift.f90:17-59), on the device: xy and uv interleaved.  The product
// and the sum are rounded separately (no FMA contraction), as the host
// expression x + dt*u evaluates without fused multiply-add.
__global__ void k_advect(long n, double *xy, const double *uv, double dt) {
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < 2 * n) xy[i] = __dadd_rn(xy[i], __dmul_rn(dt, uv[i]));
}

// Image blobs for a mirror wall at y = d: (x, 2d - y), circulation -G, core
// radius 0 (a point vortex, as the solver's image term d_biot.f90:39-53).
__global__ void k_mirror(long n, const double *xy, const double *cir, const double *cor, double d, double *oxy,
                         double *ocir, double *ocor) {
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  oxy[2 * i] = xy[2 * i];
  oxy[2 * i + 1] = xy[2 * i + 1];
  ocir[i] = cir[i];
  ocor[i] = cor[i];
  oxy[2 * (n + i)] = xy[2 * i];
  oxy[2 * (n + i) + 1] = 2.0 * d - xy[2 * i + 1];
  ocir[n + i] = -cir[i];
  ocor[n + i] = 0.0;
}

// Velocities of query points [b, e) at the blob positions: query i takes
// blob i's velocity when the two positions have the same bit patterns (a
// sweep over the blobs in order, the common case); any other query gets NaN
// here and its index appended to `miss` (in no particular order) for the
// host to resolve.
__global__ void k_lookup(long b, long e, const double2 *__restrict__ q, long nb, const double2 *__restrict__ bxy,
                         const double2 *__restrict__ buv, double2 *__restrict__ out, int *__restrict__ miss,
                         int *__restrict__ nmiss) {
  const long i = b + blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= e) return;
  const double2 p = q[i];
  bool hit = false;
  if (i < nb) {
    const double2 c = bxy[i];
    hit = __double_as_longlong(p.x) == __double_as_longlong(c.x) && __double_as_longlong(p.y) == __double_as_longlong(c.y);
  }
  if (hit) {
    out[i] = buv[i];
  } else {
    out[i] = make_double2(__longlong_as_double(0x7ff8000000000000ll), __longlong_as_double(0x7ff8000000000000ll));
    miss[atomicAdd(nmiss, 1)] = (int)i;
  }
}

cudaError_t lookup_blobs(long b, long e, const double *q, long nb, const double *bxy, const double *buv, double *out,
                         int *miss, int *nmiss, cudaStream_t s) {
  if (e <= b) return cudaSuccess;
  k_lookup<<<(unsigned)((e - b + 255) / 256), 256, 0, s>>>(b, e, reinterpret_cast<const double2 *>(q), nb,
                                                         reinterpret_cast<const double2 *>(bxy),
                                                         reinterpret_cast<const double2 *>(buv),
                                                         reinterpret_cast<double2 *>(out), miss, nmiss);
  ::t2d::g_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

// ------------------------------------------------ blobs by their position

namespace {

__device__ __forceinline__ unsigned position_slot(double2 p, unsigned mask) {
  return (unsigned)position_hash((uint64_t)__double_as_longlong(p.x), (uint64_t)__double_as_longlong(p.y)) & mask;
}
__device__ __forceinline__ bool same_position(double2 a, double2 b) {
  return __double_as_longlong(a.x) == __double_as_longlong(b.x) && __double_as_longlong(a.y) == __double_as_longlong(b.y);
}

// Open addressing, at most half full: slot = blob index + 1, the smallest of
// the blobs that share a position bit for bit.
__global__ void __launch_bounds__(256) k_position_insert(long n, const double2 *__restrict__ bxy, int *slot, unsigned mask) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double2 p = bxy[i];
  unsigned h = position_slot(p, mask);
  for (unsigned probe = 0; probe <= mask; probe++, h = (h + 1) & mask) {
    const int cur = atomicCAS(&slot[h], 0, (int)i + 1);
    if (cur == 0) return;
    if (same_position(bxy[cur - 1], p)) {
      atomicMin(&slot[h], (int)i + 1);
      return;
    }
  }
}

// The missed queries miss[0..n): res[j] = the velocity of the blob at query
// miss[j]'s position, else NaN and j appended to `off` (count in *noff).
__global__ void __launch_bounds__(256) k_position_find(int n, const int *__restrict__ miss, const double2 *__restrict__ q,
                                                       const double2 *__restrict__ bxy, const double2 *__restrict__ buv,
                                                       const int *__restrict__ slot, unsigned mask, double2 *res,
                                                       int *off, int *noff) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const double2 p = q[miss[j]];
  unsigned h = position_slot(p, mask);
  for (unsigned probe = 0; probe <= mask; probe++, h = (h + 1) & mask) {
    const int cur = slot[h];
    if (cur == 0) break;
    if (same_position(bxy[cur - 1], p)) {
      res[j] = buv[cur - 1];
      return;
    }
  }
  res[j] = make_double2(NAN, NAN);
  off[atomicAdd(noff, 1)] = j;
}

__global__ void __launch_bounds__(256) k_off_points(int n, const int *__restrict__ off, const int *__restrict__ miss,
                                                    const double2 *__restrict__ q, double2 *pts) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) pts[k] = q[miss[off[k]]];
}
__global__ void __launch_bounds__(256) k_off_results(int n, const int *__restrict__ off, const double2 *__restrict__ uv,
                                                     double2 *res) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) res[off[k]] = uv[k];
}

cudaError_t launched() {
  ::t2d::g_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

}  // namespace

cudaError_t position_table(long n, const double *bxy, int *slot, unsigned mask, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(slot, 0, sizeof(int) * ((size_t)mask + 1), s);
  if (e != cudaSuccess || n <= 0) return e;
  k_position_insert<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, reinterpret_cast<const double2 *>(bxy), slot, mask);
  return launched();
}

cudaError_t position_find(int n, const int *miss, const double *q, const double *bxy, const double *buv, const int *slot,
                          unsigned mask, double *res, int *off, int *noff, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(noff, 0, sizeof(int), s);
  if (e != cudaSuccess || n <= 0) return e;
  k_position_find<<<(n + 255) / 256, 256, 0, s>>>(n, miss, reinterpret_cast<const double2 *>(q),
                                                  reinterpret_cast<const double2 *>(bxy),
                                                  reinterpret_cast<const double2 *>(buv), slot, mask,
                                                  reinterpret_cast<double2 *>(res), off, noff);
  return launched();
}

cudaError_t off_points(int n, const int *off, const int *miss, const double *q, double *pts, cudaStream_t s) {
  k_off_points<<<(n + 255) / 256, 256, 0, s>>>(n, off, miss, reinterpret_cast<const double2 *>(q),
                                               reinterpret_cast<double2 *>(pts));
  return launched();
}

cudaError_t off_results(int n, const int *off, const double *uv, double *res, cudaStream_t s) {
  k_off_results<<<(n + 255) / 256, 256, 0, s>>>(n, off, reinterpret_cast<const double2 *>(uv),
                                                reinterpret_cast<double2 *>(res));
  return launched();
}

cudaError_t advect(long n, double *xy, const double *uv, double dt, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_advect<<<(int)((2 * n + 255) / 256), 256, 0, s>>>(n, xy, uv, dt);
  ::t2d::g_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

cudaError_t mirror_images(long n, const double *xy, const double *cir, const double *cor, double d, double *oxy,
                          double *ocir, double *ocor, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_mirror<<<(int)((n + 255) / 256), 256, 0, s>>>(n, xy, cir, cor, d, oxy, ocir, ocor);
  ::t2d::g_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

cudaError_t ffma_probe(float *out, int blocks, int iters, cudaStream_t s) {
  k_ffma_probe<<<blocks, 256, 0, s>>>(out, iters, 0.999999f, 1e-7f);
  ::t2d::g_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

cudaError_t direct_sum(int ntgt, const double *txy, int nsrc, const double *sxy, const double *cir,
                       const double *cor, double *uv, cudaStream_t s) {
  if (ntgt <= 0) return cudaSuccess;
  cudaError_t e = cudaMemsetAsync(uv, 0, sizeof(double) * 2 * (size_t)ntgt, s);
  if (e != cudaSuccess) return e;
  const int tblocks = (ntgt + kThreads - 1) / kThreads;
  int chunks = max(1, (152 * 8) / tblocks);
  int chunk = (nsrc + chunks - 1) / chunks;
  chunk = ((chunk + kThreads - 1) / kThreads) * kThreads;
  if (chunk < kThreads) chunk = kThreads;
  chunks = (nsrc + chunk - 1) / chunk;
  if (chunks < 1) chunks = 1;
  k_direct<<<dim3(tblocks, chunks), kThreads, 0, s>>>(ntgt, txy, nsrc, sxy, cir, cor, uv, chunk, fix::One());
  ::t2d::g_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

}  // namespace t2d
