// Learned order selection: features, labels, and the training kernels of
// the MLP (BF16 weights and layer inputs, FP32 accumulation).
//
// What the network decides.  In the mixed FMM the near field of a leaf B is
// its U list (adjacent leaves, exact regularised P2P) and its K list (leaves
// within the cutoff, Gaussian correction).  For each such interaction the
// network picks the cheapest treatment whose error stays under a budget:
// direct evaluation (class 0), or the source leaf's multipole at order
// p = 4..16 (classes 1..13; for a K interaction this means the correction
// is skipped because the far field already covers the point-vortex part).
// The fixed form (all interactions direct) is the fallback when no trained
// weights are loaded.
//
// Labels come from the FMM itself against the FP64 exact contribution of
// the interaction (the direct sum restricted to it): `k_labels`.  Training
// runs on the GPU in FP32 over BF16-rounded operands: per step one kernel for
// the forward pass, the softmax cross-entropy and the layers' gradients, and
// one for the weight gradients and Adam; gradients are checked against the
// CPU oracle (oracle/mlp_oracle.py).
#include <cuda_bf16.h>

#include <cmath>
#include <cstring>

#include "dev_common.cuh"
#include "learn.h"

namespace t2d {

namespace {

__global__ void k_leaf_stats(MixedView m, LeafStats *out) {
  chain_wait();
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= m.nleaf) return;
  const int c = m.leaf_cell[w];
  const float ih = m.inv_h[c];
  float ga = 0.f, mx = 0.f, my = 0.f, m2 = 0.f, sg = 0.f;
  for (int j = m.begin[c] + lane; j < m.end[c]; j += 32) {
    const float4 s = m.src4[j];
    const float g = fabsf(s.z);
    const float zx = s.x * ih, zy = s.y * ih;
    ga += g;
    mx += s.z * zx;
    my += s.z * zy;
    m2 += g * (zx * zx + zy * zy);
    sg = fmaxf(sg, rsqrtf(fmaxf(-s.w * 0.69314718f, 1e-30f)));  // s.w = -log2(e)/sigma^2
  }
  for (int o = 16; o; o >>= 1) {
    ga += __shfl_xor_sync(0xffffffffu, ga, o);
    mx += __shfl_xor_sync(0xffffffffu, mx, o);
    my += __shfl_xor_sync(0xffffffffu, my, o);
    m2 += __shfl_xor_sync(0xffffffffu, m2, o);
    sg = fmaxf(sg, __shfl_xor_sync(0xffffffffu, sg, o));
  }
  if (lane == 0) {
    LeafStats r;
    r.g_abs = ga;
    r.m1 = ga > 0.f ? sqrtf(mx * mx + my * my) / ga : 0.f;
    r.m2 = ga > 0.f ? m2 / ga : 0.f;
    r.sig = sg;
    out[c] = r;
  }
}

__device__ __forceinline__ float2 cmulf(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// One warp per sampled interaction.  samples[3*i] = leaf ordinal,
// [3*i+1] = kind (0 U, 1 K), [3*i+2] = entry index in that list.
__global__ void k_labels(MixedView m, const LeafStats *st, const float *u_ref_ptr, double tol, int ns,
                         const int *samples, float *features, int *labels) {
  chain_wait();
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= ns) return;
  const int l = samples[3 * w], kind = samples[3 * w + 1], e = samples[3 * w + 2];
  const int B = m.leaf_cell[l];
  const int A = kind == 0 ? m.u_idx[e] : m.k_idx[e];
  const float u_ref = *u_ref_ptr;
  const int P = m.P;
  const double ox = m.cx[B] - m.cx[A], oy = m.cy[B] - m.cy[A];
  const float oxf = centre_offset(m.cxf, m.cxl, B, A), oyf = centre_offset(m.cyf, m.cyl, B, A);
  const float ihA = m.inv_h[A];
  const float *MA = m.M + (size_t)A * 2 * P;
  double err[14];
  // orders beyond the stored expansion cannot be used
  for (int c = 0; c < 14; c++) err[c] = (kind == 0 && class_order(c) > P) ? 1e300 : 0.0;
  for (int t0 = m.begin[B]; t0 < m.end[B]; t0 += 32) {
    const int t = t0 + lane;
    const bool valid = t < m.end[B];
    const float2 zt = valid ? m.loc[t] : make_float2(0.f, 0.f);
    // exact contribution in FP64
    double ex = 0.0, ey = 0.0;
    for (int j = m.begin[A]; j < m.end[A]; j++) {
      const float4 s = m.src4[j];
      const double rx = ((double)zt.x - (double)s.x) + ox, ry = ((double)zt.y - (double)s.y) + oy;
      const double r2 = rx * rx + ry * ry;
      const double r = sqrt(r2);
      // s.w = -log2(e)/sigma^2, so exp(-r^2/sigma^2) = 2^(r^2 s.w)
      if (kind == 0) {
        if (r > 1e-10) {
          const double f = (double)s.z * (1.0 - exp2(r2 * (double)s.w)) / r2;
          ex -= f * ry;
          ey += f * rx;
        }
      } else if (r > 1e-10) {
        const double f = -(double)s.z * exp2(r2 * (double)s.w) / r2;
        ex -= f * ry;
        ey += f * rx;
      }
    }
    if (kind == 1) {
      // skipping the correction leaves exactly this out
      const double em = valid ? sqrt(ex * ex + ey * ey) : 0.0;
      for (int c = 1; c < 14; c++) err[c] = fmax(err[c], em);
    } else {
      // the source leaf's multipole at order p (FP32, as the evaluation does)
      const float zx = (zt.x + oxf) * ihA, zy = (zt.y + oyf) * ihA;
      const float ir2 = 1.f / (zx * zx + zy * zy);
      const float2 wv = make_float2(zx * ir2, -zy * ir2);
      float2 pw = wv;       // w^(k+1)
      float2 phi = make_float2(0.f, 0.f);
      for (int k = 0; k < 16 && k < P; k++) {
        const float2 a = make_float2(MA[k], MA[P + k]);
        const float2 t2 = cmulf(a, pw);
        phi.x += t2.x * ihA;
        phi.y += t2.y * ihA;
        pw = cmulf(pw, wv);
        const int p = k + 1;  // terms 0..k used
        if (p >= 4) {
          const double dx = (double)phi.y - ex, dy = (double)phi.x - ey;
          const double em = (valid && isfinite(dx) && isfinite(dy)) ? sqrt(dx * dx + dy * dy) : (valid ? 1e300 : 0.0);
          err[p - 3] = fmax(err[p - 3], em);
        }
      }
      if (A == B) for (int c = 1; c < 14; c++) err[c] = valid ? 1e300 : err[c];
    }
  }
  for (int c = 1; c < 14; c++)
    for (int o = 16; o; o >>= 1) err[c] = fmax(err[c], __shfl_xor_sync(0xffffffffu, err[c], o));
  if (lane == 0) {
    int label = 0;
    if (kind == 1) {
      label = err[1] <= tol ? 1 : 0;
    } else {
      for (int c = 1; c < 14; c++)
        if (err[c] <= tol) {
          label = c;
          break;
        }
    }
    labels[w] = label;
    float f[kMlpIn];
    interaction_features(m, st, B, A, kind, u_ref, f);
    for (int k = 0; k < kMlpIn; k++) features[(size_t)w * kMlpIn + k] = f[k];
  }
}

// ------------------------------------------------------------ training

__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

__device__ __forceinline__ float gelu_f(float z) {
  const float c = 0.7978845608028654f;
  return 0.5f * z * (1.f + tanhf(c * (z + 0.044715f * z * z * z)));
}
__device__ __forceinline__ float gelu_grad_f(float z) {
  const float c = 0.7978845608028654f;
  const float t = tanhf(c * (z + 0.044715f * z * z * z));
  return 0.5f * (1.f + t) + 0.5f * z * (1.f - t * t) * c * (1.f + 3.f * 0.044715f * z * z);
}

__device__ __forceinline__ uint32_t hash32(uint32_t x) {
  x ^= x >> 16;
  x *= 0x7feb352du;
  x ^= x >> 15;
  x *= 0x846ca68bu;
  x ^= x >> 16;
  return x;
}

constexpr int kH = kMlpHidden;
struct Offs {
  int W1, b1, W2, b2, W3, b3, W4, b4;
};
constexpr Offs kOff{0, 1024, 1088, 5184, 5248, 9344, 9408, 10432};
static_assert(kMlpIn == 16 && kMlpHidden == 64 && kMlpOut == 16, "the tiles below are for 16 -> 64 -> 64 -> 64 -> 16");

// A mini-batch's layer inputs A (BF16-rounded) and the loss's gradients D by
// the layers' sums, row-major, for the weight gradients.
struct Pass {
  float *A0, *A1, *A2, *A3, *D1, *D2, *D3, *D4;
};

// Rows of the batch and how they are drawn: row i is X's row i, or with
// `draw` one drawn by `seed` and i.
struct Rows {
  const float *X;
  const int *y;  // null: forward only
  int n, bt, draw;
  unsigned seed;
};
__device__ __forceinline__ int row_of(const Rows &r, int i) {
  return r.draw ? (int)(hash32(r.seed * 2654435761u + (unsigned)i) % (unsigned)r.n) : i;
}

constexpr int kRowsPerBlock = 32;
constexpr int kPadH = kH + 4, kPadIn = kMlpIn + 4;  // row strides in shared memory (16-byte loads of 8 rows: 32 banks)
struct RowsShared {
  float W1[kH][kPadIn], W2[kH][kPadH], W3[kH][kPadH], W4[kMlpOut][kPadH];
  float A0[kRowsPerBlock][kPadIn];
  float A[kRowsPerBlock][kPadH], Z1[kRowsPerBlock][kPadH], Z2[kRowsPerBlock][kPadH], Z3[kRowsPerBlock][kPadH];
  float Z4[kRowsPerBlock][kPadIn], D4[kRowsPerBlock][kPadIn], Da[kRowsPerBlock][kPadH], Db[kRowsPerBlock][kPadH];
};

// Z[r][o] = sum_k A[r][k] W[o][k] + bias[o] (k ascending, one FMA per term),
// for 16 O outputs; a thread forms 2 rows x O outputs.
template <int K, int O, int SA, int SW, int SZ>
__device__ __forceinline__ void layer(const float (*A)[SA], const float (*W)[SW], const float *bias, float (*Z)[SZ]) {
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float acc[2][O];
#pragma unroll
  for (int r = 0; r < 2; r++)
#pragma unroll
    for (int o = 0; o < O; o++) acc[r][o] = 0.f;
#pragma unroll 4
  for (int k = 0; k < K; k += 4) {
    float4 a[2], w[O];
#pragma unroll
    for (int r = 0; r < 2; r++) a[r] = *reinterpret_cast<const float4 *>(&A[ty + 16 * r][k]);
#pragma unroll
    for (int o = 0; o < O; o++) w[o] = *reinterpret_cast<const float4 *>(&W[tx + 16 * o][k]);
#pragma unroll
    for (int r = 0; r < 2; r++)
#pragma unroll
      for (int o = 0; o < O; o++) {
        acc[r][o] = fmaf(a[r].x, w[o].x, acc[r][o]);
        acc[r][o] = fmaf(a[r].y, w[o].y, acc[r][o]);
        acc[r][o] = fmaf(a[r].z, w[o].z, acc[r][o]);
        acc[r][o] = fmaf(a[r].w, w[o].w, acc[r][o]);
      }
  }
#pragma unroll
  for (int r = 0; r < 2; r++)
#pragma unroll
    for (int o = 0; o < O; o++) Z[ty + 16 * r][tx + 16 * o] = acc[r][o] + bias[tx + 16 * o];
}

// out[r][h] = (sum_o D[r][o] W[o][h]) gelu'(Z[r][h]), o ascending; also to the
// row-major global array g (rows below `rows`).
template <int O, int SD>
__device__ __forceinline__ void back(const float (*D)[SD], const float (*W)[kPadH], const float (*Z)[kPadH],
                                     float (*out)[kPadH], float *g, int rows) {
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float acc[2][4] = {};
#pragma unroll 2
  for (int o = 0; o < O; o += 4) {
    float4 d[2];
#pragma unroll
    for (int r = 0; r < 2; r++) d[r] = *reinterpret_cast<const float4 *>(&D[ty + 16 * r][o]);
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const float w = W[o + q][tx + 16 * j];
        acc[0][j] = fmaf((&d[0].x)[q], w, acc[0][j]);
        acc[1][j] = fmaf((&d[1].x)[q], w, acc[1][j]);
      }
  }
#pragma unroll
  for (int r = 0; r < 2; r++)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int i = ty + 16 * r, h = tx + 16 * j;
      float v = acc[r][j] + 0.f;
      v *= gelu_grad_f(Z[i][h]);
      out[i][h] = v;
      if (i < rows) g[(size_t)i * kH + h] = v;
    }
}

// A = bf16(gelu(Z)), also to the row-major global array g (if any).
__device__ __forceinline__ void activate(const float (*Z)[kPadH], float (*A)[kPadH], float *g, int rows) {
  for (int e = threadIdx.x; e < kRowsPerBlock * kH; e += blockDim.x) {
    const int i = e / kH, h = e & (kH - 1);
    const float v = bf16r(gelu_f(Z[i][h]));
    A[i][h] = v;
    if (g && i < rows) g[(size_t)i * kH + h] = v;
  }
}

template <int K, int O, int S>
__device__ __forceinline__ void load_weights(const float *theta, float (*W)[S]) {
#pragma unroll
  for (int e = 4 * threadIdx.x; e < K * O; e += 4 * 256) {
    const float4 v = *reinterpret_cast<const float4 *>(theta + e);
    *reinterpret_cast<float4 *>(&W[e / K][e % K]) = make_float4(bf16r(v.x), bf16r(v.y), bf16r(v.z), bf16r(v.w));
  }
}

// Forward pass, loss and the gradients by the layers' sums for 32 rows per
// block, everything between the layers in shared memory.  Each sum runs in
// the order of a plain loop, so the values do not depend on the tiling.
__global__ void __launch_bounds__(256) k_rows(Rows rows, const float *__restrict__ theta, Pass p, float *logits,
                                              float *loss) {
  chain_wait();
  extern __shared__ float4 shared_rows[];
  RowsShared &s = *reinterpret_cast<RowsShared *>(shared_rows);
  const int i0 = blockIdx.x * kRowsPerBlock, left = min(kRowsPerBlock, rows.bt - i0);
  const bool train = rows.y != nullptr;
  load_weights<kMlpIn, kH>(theta + kOff.W1, s.W1);
  load_weights<kH, kH>(theta + kOff.W2, s.W2);
  load_weights<kH, kH>(theta + kOff.W3, s.W3);
  load_weights<kH, kMlpOut>(theta + kOff.W4, s.W4);
  for (int e = threadIdx.x; e < kRowsPerBlock * kMlpIn; e += blockDim.x) {
    const int i = e / kMlpIn, k = e & (kMlpIn - 1);
    float v = 0.f;
    if (i < left) v = bf16r(rows.X[(size_t)row_of(rows, i0 + i) * kMlpIn + k]);
    s.A0[i][k] = v;
    if (train && i < left) p.A0[(size_t)(i0 + i) * kMlpIn + k] = v;
  }
  const size_t at = (size_t)i0 * kH;
  __syncthreads();
  layer<kMlpIn, 4>(s.A0, s.W1, theta + kOff.b1, s.Z1);
  __syncthreads();
  activate(s.Z1, s.A, train ? p.A1 + at : nullptr, left);
  __syncthreads();
  layer<kH, 4>(s.A, s.W2, theta + kOff.b2, s.Z2);
  __syncthreads();
  activate(s.Z2, s.A, train ? p.A2 + at : nullptr, left);
  __syncthreads();
  layer<kH, 4>(s.A, s.W3, theta + kOff.b3, s.Z3);
  __syncthreads();
  activate(s.Z3, s.A, train ? p.A3 + at : nullptr, left);
  __syncthreads();
  layer<kH, 1>(s.A, s.W4, theta + kOff.b4, s.Z4);
  __syncthreads();
  if (!train) {
    for (int e = threadIdx.x; e < left * kMlpOut; e += blockDim.x)
      logits[(size_t)i0 * kMlpOut + e] = s.Z4[e / kMlpOut][e & (kMlpOut - 1)];
    return;
  }
  // D4 = (softmax(Z4[:14]) - onehot) / bt, loss summed into *loss
  if (threadIdx.x < kRowsPerBlock) {
    const int i = threadIdx.x;
    const float *z = s.Z4[i];
    float mx = z[0];
    for (int c = 1; c < kMlpClasses; c++) mx = fmaxf(mx, z[c]);
    float q[kMlpClasses], sum = 0.f;
    for (int c = 0; c < kMlpClasses; c++) {
      q[c] = expf(z[c] - mx);
      sum += q[c];
    }
    const int y = i < left ? rows.y[row_of(rows, i0 + i)] : 0;
    float py = 1.f;
    for (int c = 0; c < kMlpOut; c++) {
      float d = c < kMlpClasses ? q[c < kMlpClasses ? c : 0] / sum : 0.f;
      if (c == y) {
        if (c < kMlpClasses) py = d;
        d -= 1.f;
      }
      d /= (float)rows.bt;
      s.D4[i][c] = i < left ? d : 0.f;
      if (i < left) p.D4[(size_t)(i0 + i) * kMlpOut + c] = d;
    }
    float l = i < left ? -logf(fmaxf(py, 1e-30f)) / (float)rows.bt : 0.f;
    for (int o = 16; o; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if (i == 0) atomicAdd(loss, l);
  }
  __syncthreads();
  back<kMlpOut>(s.D4, s.W4, s.Z3, s.Da, p.D3 + at, left);
  __syncthreads();
  back<kH>(s.Da, s.W3, s.Z2, s.Db, p.D2 + at, left);
  __syncthreads();
  back<kH>(s.Db, s.W2, s.Z1, s.Da, p.D1 + at, left);
}

// Weight gradients g[o][h] = sum_i D[i][o] A[i][h], i ascending: 16 x 16 of
// them per block, 2 x 2 per thread of the first two warps; the other two copy
// the rows' columns asynchronously, three stages of 64 rows ahead (more change
// nothing).  The last blocks sum the columns of D (biases).  Bound by the one
// chain of multiply-adds per weight that the sums' order leaves: 33 us for
// 4,096 rows.  A step takes 54 us with k_rows, where one tiled product per
// layer and direction (4 blocks walking the rows for each weight gradient)
// and one block per bias took 1,440.
constexpr int kStage = 64, kStages = 4;
constexpr int kWTiles2 = (kH / 16) * (kH / 16), kWTiles1 = kH / 16;
constexpr int kWeightBlocks = 2 * kWTiles2 + 2 * kWTiles1 + 7;
struct Adam {
  float *theta, *m1, *v1;  // null theta: gradients only
  float lr, b1c, b2c;
};
__device__ __forceinline__ void adam(const Adam &a, int i, float g) {
  const float b1 = 0.9f, b2 = 0.999f;
  const float mi = b1 * a.m1[i] + (1.f - b1) * g;
  const float vi = b2 * a.v1[i] + (1.f - b2) * g * g;
  a.m1[i] = mi;
  a.v1[i] = vi;
  a.theta[i] -= a.lr * (mi / a.b1c) / (sqrtf(vi / a.b2c) + 1e-8f);
}

__global__ void __launch_bounds__(128) k_weights(int bt, Pass p, float *grad, Adam a) {
  chain_wait();
  __shared__ __align__(16) float cols[kStages][kStage][32];  // [buffer][row][16 columns of D, 16 of A, or 32 of D]
  const bool copier = threadIdx.x >= 64;
  const int t = threadIdx.x & 63;
  auto put = [&](int i, float g) {
    if (grad) grad[i] = g;
    if (a.theta) adam(a, i, g);
  };
  // nd columns of D from dc and, for a weight tile, 16 of A from ac
  const float *D, *A = nullptr;
  int ld, la = 0, dc = 0, ac = 0, nd = 16, out, so = 0;
  int b = blockIdx.x;
  if (b < 2 * kWTiles2) {
    const bool second = b >= kWTiles2;
    b -= second ? kWTiles2 : 0;
    D = second ? p.D3 : p.D2, A = second ? p.A2 : p.A1;
    ld = la = kH, dc = 16 * (b / 4), ac = 16 * (b & 3), out = second ? kOff.W3 : kOff.W2, so = kH;
  } else if ((b -= 2 * kWTiles2) < kWTiles1) {
    D = p.D4, A = p.A3, ld = kMlpOut, la = kH, ac = 16 * b, out = kOff.W4, so = kH;
  } else if ((b -= kWTiles1) < kWTiles1) {
    D = p.D1, A = p.A0, ld = kH, la = kMlpIn, dc = 16 * b, out = kOff.W1, so = kMlpIn;
  } else {
    b -= kWTiles1;  // 32 columns of D1, D1, D2, D2, D3, D3, D4
    const int l = b >> 1;
    D = l == 0 ? p.D1 : l == 1 ? p.D2 : l == 2 ? p.D3 : p.D4;
    ld = l == 3 ? kMlpOut : kH;
    nd = min(ld, 32);
    dc = 32 * (b & 1);
    out = (l == 0 ? kOff.b1 : l == 1 ? kOff.b2 : l == 2 ? kOff.b3 : kOff.b4) + dc;
  }
  // a copying thread takes 4 columns (of 32, or 16 of D4) of every 8th row
  const int col = 4 * (t & 7);
  const float *from = col < nd ? D + dc + col : A ? A + ac + (col - nd) : nullptr;
  const int stride = col < nd ? ld : la;
  auto stage = [&](int k) {
    const int r0 = k * kStage;
    if (r0 < bt && from) {
      unsigned dst = (unsigned)__cvta_generic_to_shared(&cols[k % kStages][t >> 3][col]);
      const float *src = from + (size_t)(r0 + (t >> 3)) * stride;
#pragma unroll
      for (int r = t >> 3; r < kStage; r += 8, dst += 8 * 32 * 4, src += (size_t)8 * stride) {
        const bool in = r0 + r < bt;  // rows past the batch: zeros
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(in ? src : from), "r"(in ? 16 : 0));
      }
    }
    asm volatile("cp.async.commit_group;");
  };
  const int h = 2 * (t & 7), o = 2 * (t >> 3);
  float g00 = 0.f, g01 = 0.f, g10 = 0.f, g11 = 0.f;  // [o][h]
  const int nk = (bt + kStage - 1) / kStage;
  if (copier) {
    for (int k = 0; k < kStages - 1; k++) stage(k);
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2));
  }
  for (int k = 0; k < nk; k++) {
    __syncthreads();  // stage k is in, and stage k - 1 done with
    if (copier) {
      stage(k + kStages - 1);
      asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2));  // stage k + 1
      continue;
    }
    const int buf = k % kStages;
    if (A) {
#pragma unroll 16
      for (int r = 0; r < kStage; r++) {
        const float2 x = *reinterpret_cast<const float2 *>(&cols[buf][r][16 + h]);
        const float2 d = *reinterpret_cast<const float2 *>(&cols[buf][r][o]);
        g00 = fmaf(d.x, x.x, g00);
        g01 = fmaf(d.x, x.y, g01);
        g10 = fmaf(d.y, x.x, g10);
        g11 = fmaf(d.y, x.y, g11);
      }
    } else if (t < nd) {
#pragma unroll 16
      for (int r = 0; r < kStage; r++) g00 += cols[buf][r][t];
    }
  }
  if (copier) {
    asm volatile("cp.async.wait_all;");
    return;
  }
  if (A) {
    const int i = out + (dc + o) * so + ac + h;
    put(i, g00 + 0.f);
    put(i + 1, g01 + 0.f);
    put(i + so, g10 + 0.f);
    put(i + so + 1, g11 + 0.f);
  } else if (t < nd) {
    put(out + t, g00);
  }
}

cudaError_t run_weights(int bt, const Pass &p, float *grad, const Adam &a, cudaStream_t s) {
  chained(k_weights, kWeightBlocks, 128, 0, s)(bt, p, grad, a);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

size_t pass_floats(int bt) { return (size_t)bt * (2 * kMlpIn + 6 * kH); }

void carve(float *base, int bt, Pass &p) {
  const size_t H = (size_t)bt * kH, I = (size_t)bt * kMlpIn;
  float *q = base;
  for (float **a : {&p.A1, &p.A2, &p.A3, &p.D1, &p.D2, &p.D3}) *a = q, q += H;
  for (float **a : {&p.A0, &p.D4}) *a = q, q += I;
}

cudaError_t run_rows(const Rows &rows, const float *theta, const Pass &p, float *logits, float *loss, cudaStream_t s) {
  const int bytes = (int)sizeof(RowsShared);
  cudaError_t e = cudaFuncSetAttribute(k_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return e;
  chained(k_rows, (rows.bt + kRowsPerBlock - 1) / kRowsPerBlock, 256, bytes, s)(rows, theta, p, logits, loss);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

}  // namespace

// u_ref = sum |G| / R0 (deterministic: fixed per-thread ranges, tree sum).
__global__ void __launch_bounds__(1024) k_uref(MixedView m, const LeafStats *st, const RootBox *root, float *out) {
  chain_wait();
  __shared__ float part[1024];
  const int t = threadIdx.x;
  const int per = (m.nleaf + 1023) / 1024;
  float s = 0.f;
  for (int l = t * per; l < min(m.nleaf, (t + 1) * per); l++) s += st[m.leaf_cell[l]].g_abs;
  part[t] = s;
  __syncthreads();
  for (int o = 512; o; o >>= 1) {
    if (t < o) part[t] += part[t + o];
    __syncthreads();
  }
  if (t == 0) *out = part[0] / (float)root->region;
}

// The leaves of each set of a batched tree: one contiguous range of the
// leaf order (a set's cells are the subtree of its root), [lo[k], hi[k]).
__global__ void k_set_leaf_ranges(MixedView m, int *lo, int *hi) {
  chain_wait();
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= m.nleaf) return;
  const int k = set_of_cell(m, m.leaf_cell[l]);
  if (l == 0 || set_of_cell(m, m.leaf_cell[l - 1]) != k) lo[k] = l;
  if (l == m.nleaf - 1 || set_of_cell(m, m.leaf_cell[l + 1]) != k) hi[k] = l + 1;
}

// k_uref for each set of a batched tree, one block per set: the set's leaves
// in order, split over the threads as k_uref splits a single tree's, so that
// a set's u_ref is the one it gets alone, bit for bit.
__global__ void __launch_bounds__(1024) k_uref_sets(MixedView m, const LeafStats *st, const RootBox *root,
                                                    const int *lo, const int *hi, float *out) {
  chain_wait();
  __shared__ float part[1024];
  const int k = blockIdx.x, t = threadIdx.x;
  const int l0 = lo[k], cnt = max(hi[k] - l0, 0);
  const int per = (cnt + 1023) / 1024;
  float s = 0.f;
  for (int l = t * per; l < min(cnt, (t + 1) * per); l++) s += st[m.leaf_cell[l0 + l]].g_abs;
  part[t] = s;
  __syncthreads();
  for (int o = 512; o; o >>= 1) {
    if (t < o) part[t] += part[t + o];
    __syncthreads();
  }
  if (t == 0) out[k] = part[0] / (float)root[k].region;
}

int learned_uref_sets(MixedView &m, const LeafStats *stats, const RootBox *roots, int nsets, int *leaf_lo,
                      int *leaf_hi, float *out, cudaStream_t s) {
  if (nsets <= 0) return TREE2D_OK;
  T2D_CUDA_TRY(cudaMemsetAsync(leaf_lo, 0, sizeof(int) * (size_t)nsets, s));
  T2D_CUDA_TRY(cudaMemsetAsync(leaf_hi, 0, sizeof(int) * (size_t)nsets, s));
  if (m.nleaf > 0) chained(k_set_leaf_ranges, (m.nleaf + 255) / 256, 256, 0, s)(m, leaf_lo, leaf_hi);
  chained(k_uref_sets, nsets, 1024, 0, s)(m, stats, roots, leaf_lo, leaf_hi, out);
  g_launches.fetch_add(2, std::memory_order_relaxed);
  T2D_CUDA_TRY(cudaGetLastError());
  return TREE2D_OK;
}

int learned_uref(MixedView &m, const LeafStats *stats, const RootBox *root, float *out, cudaStream_t s) {
  chained(k_uref, 1, 1024, 0, s)(m, stats, root, out);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  T2D_CUDA_TRY(cudaGetLastError());
  return TREE2D_OK;
}

int learned_leaf_stats(MixedView &m, LeafStats *stats, cudaStream_t s) {
  chained(k_leaf_stats, (int)(((long)m.nleaf * 32 + 255) / 256), 256, 0, s)(m, stats);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  T2D_CUDA_TRY(cudaGetLastError());
  return TREE2D_OK;
}

int learned_labels(MixedView &m, const LeafStats *stats, const float *u_ref_ptr, double tol, int ns,
                   const int *samples, float *features, int *labels, cudaStream_t s) {
  if (ns <= 0) return TREE2D_OK;
  chained(k_labels, (int)(((long)ns * 32 + 255) / 256), 256, 0, s)(m, stats, u_ref_ptr, tol, ns, samples, features,
                                                               labels);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  T2D_CUDA_TRY(cudaGetLastError());
  return TREE2D_OK;
}

int mlp_train(int n, const float *X, const int *y, float *theta, float *m1, float *v1, int steps, int batch,
              float lr, unsigned seed, float *loss_out, cudaStream_t s) {
  if (n <= 0 || steps <= 0 || batch <= 0) return TREE2D_ERR_BAD_INPUT;
  float *buf = nullptr;
  T2D_CUDA_TRY(cudaMalloc(reinterpret_cast<void **>(&buf), (pass_floats(batch) + 1) * sizeof(float)));
  Pass p;
  carve(buf, batch, p);
  float *loss = buf + pass_floats(batch);
  cudaError_t e = cudaSuccess;
  for (int it = 0; it < steps && e == cudaSuccess; it++) {
    if (it == steps - 1) e = cudaMemsetAsync(loss, 0, sizeof(float), s);  // only the last step's is reported
    if (e == cudaSuccess) e = run_rows(Rows{X, y, n, batch, 1, seed + (unsigned)it * 7919u}, theta, p, nullptr, loss, s);
    const float b1c = 1.f - powf(0.9f, (float)(it + 1)), b2c = 1.f - powf(0.999f, (float)(it + 1));
    if (e == cudaSuccess) e = run_weights(batch, p, nullptr, Adam{theta, m1, v1, lr, b1c, b2c}, s);
  }
  if (e == cudaSuccess && loss_out) e = cudaMemcpyAsync(loss_out, loss, sizeof(float), cudaMemcpyDeviceToHost, s);
  const cudaError_t es = cudaStreamSynchronize(s);
  cudaFree(buf);
  T2D_CUDA_TRY(e);
  T2D_CUDA_TRY(es);
  return TREE2D_OK;
}

int mlp_grad(int n, const float *X, const int *y, const float *theta, float *grad, float *loss_out, cudaStream_t s) {
  if (n <= 0) return TREE2D_ERR_BAD_INPUT;
  float *buf = nullptr;
  T2D_CUDA_TRY(cudaMalloc(reinterpret_cast<void **>(&buf), (pass_floats(n) + 1) * sizeof(float)));
  Pass p;
  carve(buf, n, p);
  float *loss = buf + pass_floats(n);
  cudaError_t e = cudaMemsetAsync(loss, 0, sizeof(float), s);
  if (e == cudaSuccess) e = run_rows(Rows{X, y, n, n, 0, 0u}, theta, p, nullptr, loss, s);
  if (e == cudaSuccess) e = run_weights(n, p, grad, Adam{}, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(loss_out, loss, sizeof(float), cudaMemcpyDeviceToHost, s);
  const cudaError_t es = cudaStreamSynchronize(s);
  cudaFree(buf);
  T2D_CUDA_TRY(e);
  T2D_CUDA_TRY(es);
  return TREE2D_OK;
}

int mlp_forward_cc(int n, const float *X, const float *theta, float *logits, cudaStream_t s) {
  if (n <= 0) return TREE2D_OK;
  T2D_CUDA_TRY(run_rows(Rows{X, nullptr, n, n, 0, 0u}, theta, Pass{}, logits, nullptr, s));
  T2D_CUDA_TRY(cudaStreamSynchronize(s));
  return TREE2D_OK;
}

}  // namespace t2d
