// Plain FP64 treecode on the device: the reference's numerics
// (ver-c/src/fmm.c) with GPU-shaped control flow.
//
//  k_upward    S2M (fmm.c:18-33) and M2M (fmm.c:35-58) in one launch: one
//              warp per leaf sums its blobs' powers, then climbs; the warp
//              that completes a cell's last child forms that cell (children
//              in quadrant order 3,2,1,0).  The level-1 -> root shift is
//              skipped as in the reference.
//  k_eval      one warp per 8, 4 or 2 consecutive targets (tree order, so the
//              targets are neighbours), 4, 8 or 16 lanes per target.  The warp walks
//              the UNION of its targets' traversals with a shared LIFO of
//              (cell, lane mask): restricted to one target, the visit order
//              is that target's own LIFO order in fmm.c:90-112.  The opening
//              test uses round-to-nearest FP64 operations without contraction
//              (r = sqrt(dx*dx + dy*dy); region > theta*r), so each target
//              takes exactly the reference's branch.  The lanes of a
//              target share its accepted cells (M2S, fmm.c:60-67, by Horner in
//              w = 1/(z - zc)) and its direct pairs (fmm.c:121-142); their
//              partial sums are added in a fixed order at the end.  Both
//              in 64-bit fixed point (fix64.cuh): FP64 runs at 1/64 of the
//              FP32 rate here.
#include "dev_common.cuh"
#include "fix64.cuh"

namespace t2d {
namespace {

// a b + c for complex values as FMAs only: Re = a.x b.x + (c.x - a.y b.y),
// Im = a.x b.y + (c.y + a.y b.x), each inner term one FMA and each outer one
// another (explicit, so the rounding does not depend on how the compiler
// contracts the code around it).
__device__ __forceinline__ double2 cfma(double2 a, double2 b, double2 c) {
  return make_double2(__fma_rn(a.x, b.x, __fma_rn(-a.y, b.y, c.x)), __fma_rn(a.x, b.y, __fma_rn(a.y, b.x, c.y)));
}

__device__ const fix::ExpTables g_exp = fix::make_exp_tables();

constexpr double kPi = 3.14159265358979323846;

// Climbing state per cell, in the memory of Tree::mac (whose bounds are
// formed after the upward pass).
struct Climb {
  int parent, arrived, children, pad;
};
static_assert(sizeof(Climb) == sizeof(double2), "the climbing state replaces the opening bounds");

__global__ void __launch_bounds__(256) k_climb_init(Tree t, int nt) {
  chain_wait();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < t.n) t.icor2[c] = 1.0 / (t.cor[c] * t.cor[c]);  // here, not in the build: mixed solves do not use it
  if (c >= t.ncell) return;
  Climb *climb = reinterpret_cast<Climb *>(t.mac);
  const int4 ch = reinterpret_cast<const int4 *>(t.child)[c];
  int n = 0;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int k = (&ch.x)[q];
    if (k < 0) continue;
    climb[k].parent = c;
    n++;
  }
  climb[c].arrived = 0;
  climb[c].children = n;
  if (c == 0) {
    climb[0].parent = -1;
    for (int k = 0; k < nt; k++) t.coef[k] = make_double2(0.0, 0.0);  // the root has no expansion
  }
}

// The sum over the warp of v[k] (k < 16), in lanes k and k + 16: halves of
// the values change lanes at every step, 32 additions instead of 160.
__device__ __forceinline__ double2 warp_sum16(double2 (&v)[16], int lane) {
#pragma unroll
  for (int o = 8; o; o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int k = 0; k < o; k++) {
      const double2 keep = up ? v[k + o] : v[k], give = up ? v[k] : v[k + o];
      v[k] = make_double2(keep.x + __shfl_xor_sync(0xffffffffu, give.x, o),
                          keep.y + __shfl_xor_sync(0xffffffffu, give.y, o));
    }
  }
  return make_double2(v[0].x + __shfl_xor_sync(0xffffffffu, v[0].x, 16),
                      v[0].y + __shfl_xor_sync(0xffffffffu, v[0].y, 16));
}

// Coefficient k of a leaf in lane k: a lane takes every 32nd blob and runs
// through its powers, 16 coefficients at a time.
__device__ __forceinline__ double2 leaf_coef(const Tree &t, int b, int e, double cx, double cy, int nt, int lane) {
  double2 mine = make_double2(0.0, 0.0);
  for (int k0 = 0; k0 < nt; k0 += 16) {
    double2 acc[16];
#pragma unroll
    for (int k = 0; k < 16; k++) acc[k] = make_double2(0.0, 0.0);
    for (int j = b + lane; j < e; j += 32) {
      const double2 z = make_double2(t.x[j] - cx, t.y[j] - cy);
      double2 p = make_double2(t.cir[j], 0.0);
      for (int k = 0; k < k0; k++) p = cmul(p, z);
#pragma unroll
      for (int k = 0; k < 16; k++) {
        if (k0 + k >= nt) break;
        acc[k].x += p.x;
        acc[k].y += p.y;
        p = cmul(p, z);
      }
    }
    const double2 s = warp_sum16(acc, lane);
    if (lane >= k0 && lane < k0 + 16) mine = s;
  }
  return mine;
}

// The shift of an expansion by d (fmm.c:50: d = z_child - z_parent), lane l
// of each group of `width` lanes holding coefficient l: a_l <- sum_{k<=l}
// C(l,k) a_k d^(l-k), as nt - 1 sweeps a_l <- a_l + d a_(l-1) over l >= j, j =
// 1, 2, ... (a Taylor shift by repeated Horner steps).
__device__ __forceinline__ double2 shift_coef(double2 a, double2 d, int nt, int l, int width) {
  for (int j = 1; j < nt; j++) {
    const double2 below = make_double2(__shfl_up_sync(0xffffffffu, a.x, 1, width), __shfl_up_sync(0xffffffffu, a.y, 1, width));
    if (l >= j) a = cfma(d, below, a);
  }
  return a;
}

// Bound by FP64 (S2M: 4 instructions per coefficient for 32 blobs and 32 for
// their sum; M2M: 4 per sweep for two children) and, in small sets, by the
// climb's depth.  One launch per level, with a warp per cell and lane k of it
// multiplying out coefficient k, took 2.87 ms at 1M Lamb-Oseen blobs and 0.46
// ms at 20,000 uniform ones; this takes 0.42 and 0.05 (solves 21.5 -> 19.0
// and 1.03 -> 0.63 ms).
__global__ void __launch_bounds__(128) k_upward(Tree t, int nt) {
  chain_wait();
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= t.nleaf) return;
  Climb *climb = reinterpret_cast<Climb *>(t.mac);
  int c = t.leaf_cell[wid];
  double2 a = leaf_coef(t, t.begin[c], t.end[c], t.cx[c], t.cy[c], nt, lane);
  const int width = nt <= 16 ? 16 : 32, groups = 32 / width;
  const int l = lane & (width - 1), group = lane / width;
  while (true) {
    if (lane < nt) t.coef[(size_t)c * nt + lane] = a;
    const int p = climb[c].parent;
    if (p <= 0) return;  // children of the root: done
    // the last of the parent's children to arrive goes on with the parent;
    // the fences order every child's coefficients before its arrival
    __threadfence();
    __syncwarp();
    int last = 0;
    if (lane == 0) last = atomicAdd(&climb[p].arrived, 1) + 1 == climb[p].children;
    if (!__shfl_sync(0xffffffffu, last, 0)) return;
    __threadfence();
    const double px = t.cx[p], py = t.cy[p];
    const int4 ch = reinterpret_cast<const int4 *>(t.child)[p];
    a = make_double2(0.0, 0.0);
    for (int q0 = 3; q0 >= 0; q0 -= groups) {
      const int k = (&ch.x)[q0 - group];
      double2 v = make_double2(0.0, 0.0), d = make_double2(0.0, 0.0);
      if (k >= 0) {
        d = make_double2(t.cx[k] - px, t.cy[k] - py);
        if (l < nt) v = __ldcg(t.coef + (size_t)k * nt + l);  // other SMs wrote it: not through L1
      }
      if (!__any_sync(0xffffffffu, k >= 0)) continue;
      v = shift_coef(v, d, nt, l, width);
      a = cadd(a, shfl_d2(v, l));
      if (groups == 2) a = cadd(a, shfl_d2(v, l + 16));
    }
    c = p;
  }
}

constexpr int kEvalWarps = 4;
constexpr int kStackCap = 160;
constexpr int kQueue = 64;  // deferred M2S cells per target
static_assert((kQueue & (kQueue - 1)) == 0, "the M2S queues are rings indexed by a mask");

struct EvalArgs {
  Tree t;
  int nt;
  double theta;
  int ntgt;
  const double *tx, *ty;
  const int *out_idx;
  double *uv;
  DevStatus *st;
  const longlong2 *fix;  // the coefficients in fixed point (kFormFp64: null)
  int k0;        // first term of the sums in FP32 pairs (fix::first_pair_term)
  bool keep64;   // t.coef holds every cell's FP64 coefficients (else only those left to FP64: the rest in place of them)
  fix::One one;
};

// The multipole sums: in FP64 (theta above kFixTheta), or in fixed point with |w| 2^es < 1 or < 1/2.
enum EvalForm { kFormFp64, kFormFull, kFormHalf };

// Bound: instruction dispatch.  Integer instructions take two dispatch cycles
// each (ALU and multiplier pipes alike; FP32 one): 15.0 ms for the 9.4 G of
// them at 1M Lamb-Oseen blobs (2.4 ms' worth in the traversal, 8 in the 250
// M2S, 9 in the 500 pairs per target), of 18.35 ms, against 67.5 with both sums
// in FP64, whose pipe was 89% busy; 0.27 against 0.90 ms at 20,000 uniform
// blobs.  Four lanes per target at least, not one: 8 targets' traversals
// overlap more than 32 targets', the four children of a cell are tested at
// once, a leaf's pairs need no queue, and a small set fills more warps (20,000
// blobs, one lane against four: 1.43 -> 1.07 ms per solve; eval_share has 8 and
// 16).  80 registers, 24 warps per SM: 64 registers spill (24.0 against 21.4
// ms per solve), 2 or 8 warps per block are slower (23.6, 22.2).
template <int kForm, int kShare>
__global__ void __launch_bounds__(kEvalWarps * 32, 6) k_eval(EvalArgs a) {
  chain_wait();
  constexpr int kEvalTargets = 32 / kShare;  // per warp
  constexpr unsigned kLanes = 0xffffffffu >> (32 - kShare), kEachTarget = 0xffffffffu / kLanes;  // a target's; each's first
  static_assert(kShare >= 4 && (kShare & (kShare - 1)) == 0, "a target's first four lanes test a cell's four children");
  __shared__ int s_cell[kEvalWarps][kStackCap];
  __shared__ unsigned s_mask[kEvalWarps][kStackCap];
  __shared__ int s_queue[kEvalWarps][kEvalTargets][kQueue];
  __shared__ double2 s_far64[kForm == kFormFp64 ? 1 : kEvalWarps * 32];
  __shared__ uint64_t s_exp_int[fix::kExpInts], s_exp_frac[fix::kExpFracs];
  for (int j = threadIdx.x; j < fix::kExpFracs; j += kEvalWarps * 32) s_exp_frac[j] = g_exp.fracs[j];
  for (int j = threadIdx.x; j < fix::kExpInts; j += kEvalWarps * 32) s_exp_int[j] = g_exp.ints[j];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane & (kShare - 1), tgt = lane / kShare;
  const long i = ((long)blockIdx.x * kEvalWarps + warp) * kEvalTargets + tgt;
  const bool valid = i < a.ntgt;
  const unsigned vmask = __ballot_sync(0xffffffffu, valid);
  if (vmask == 0) return;
  const Tree &t = a.t;
  const int nt = a.nt;
  const double x = valid ? a.tx[i] : 0.0, y = valid ? a.ty[i] : 0.0;
  const double theta = a.theta;
  // the target as FP32 pairs, for the opening pre-test (x - xh is exact)
  const float xh = __double2float_rn(x), yh = __double2float_rn(y);
  const float xl = __double2float_rn(x - (double)xh), yl = __double2float_rn(y - (double)yh);
  const float sxy = __fadd_rn(fabsf(xh), fabsf(yh));
  fix::Sum2 far;                                // this lane's share of the target's sums
  fix::SumXY near;
  // The FP64 multipole sums: all in kFormFp64, else few (cells and targets left
  // to FP64), in shared memory to leave the registers to the pairs.
  double2 far64_reg = make_double2(0.0, 0.0);
  double2 &far64 = kForm == kFormFp64 ? far64_reg : s_far64[kForm == kFormFp64 ? 0 : threadIdx.x];
  if (kForm != kFormFp64) far64 = make_double2(0.0, 0.0);
  unsigned n_m2s = 0;
  unsigned long long n_pairs = 0;
  bool overflow = false;

  // The targets accept cells at different depths, so an M2S evaluated where
  // it is accepted runs with the warp's other lanes idle.  Each target
  // instead queues its accepted cells (a ring: head qh, count nq, the same in
  // its lanes) and the warp evaluates the queues together, an entry per lane
  // and round.  Entry k of a target (counted over the whole
  // traversal) is lane k mod kShare's, so the partial sums do not depend on when
  // the queues are emptied, nor on the warp's other targets.  A flush when
  // some queue could overflow evaluates only as many rounds as every target
  // can fill, or as the fullest one needs to make room for four entries, if
  // that is more; the end of the traversal empties them all.
  unsigned qh = 0;
  int nq = 0;
  auto flush = [&](bool all) {
    int hi = nq, lo = nq;
    for (int o = 16; o >= kShare; o >>= 1) {
      hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    }
    const int rounds = (all ? hi + kShare - 1 : max(lo, hi - (kQueue - 4) + kShare - 1)) / kShare;
    const int first = (int)((unsigned)(sub - (int)qh) & (kShare - 1));
    fix::settle(far);  // at most kQueue / kShare terms follow
    for (int r = 0; r < rounds; r++) {
      const int k = first + r * kShare;
      if (k < nq) {
        // M2S, fmm.c:60-67: sum_{k<nt-1} a_k w^{k+1}, w = 1/(z - zc)
        const int cc = s_queue[warp][tgt][(qh + k) & (kQueue - 1)];
        const double dx = fix::minus(x, t.cx[cc]);
        const double dy = fix::minus(y, t.cy[cc]);
        bool done = false;
        if constexpr (kForm != kFormFp64) {
          const longlong2 *cf = a.fix + (size_t)cc * nt;
          const longlong2 sc = __ldg(cf + (nt - 1));
          done = fix::add_multipole<kForm == kFormHalf>(
              far, dx, dy, fix::CellScale{(int)sc.x, (int)sc.y}, nt - 1, a.k0,
              [&](int k) {
                const longlong2 v = __ldg(cf + k);
                return fix::Coef{v.x, v.y};
              },
              [&](int k) {
                const float4 v = __ldg(reinterpret_cast<const float4 *>(cf + k));
                return fix::PairCoef{v.x, v.y, v.z, v.w};
              },
              a.keep64, a.one);
        }
        if (!done) {
          const double d2 = __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
          const double inv = rcp_nr(d2);
          const double2 w = make_double2(__dmul_rn(dx, inv), -__dmul_rn(dy, inv));
          const double2 *cf = t.coef + (size_t)cc * nt;
          // Horner, each step acc <- acc w + a_k as two FMAs per component
          double2 acc = cf[nt - 2];
          for (int k = nt - 3; k >= 0; k--) acc = cfma(acc, w, cf[k]);
          far64 = cfma(acc, w, far64);
        }
      }
    }
    const int out = min(rounds * kShare, nq);
    qh += (unsigned)out;
    nq -= out;
  };

  int top = 0;
  if (lane == 0) {
    s_cell[warp][0] = 0;
    s_mask[warp][0] = vmask;
  }
  __syncwarp();
  while (top >= 0) {
    const int c = s_cell[warp][top];
    const unsigned m = s_mask[warp][top];
    __syncwarp();
    top--;
    const bool act = (m >> lane) & 1u;
    if (t.leaf[c]) {
      // direct_evaluate, fmm.c:121-142: the leaf's blobs dealt to the kShare
      // lanes of each target that opened it
      const int b = t.begin[c], e = t.end[c];
      if (act) {
        for (int j0 = b; j0 < e; j0 += 32 * kShare) {
          fix::settle(near);
          const int j1 = min(e, j0 + 32 * kShare);
          for (int j = j0 + sub; j < j1; j += kShare) {
            const double rx = fix::minus(x, t.x[j]);
            const double ry = fix::minus(y, t.y[j]);
            // The reference forms r = sqrt(r2), (r/sigma)^2 and 1/(r*r); r2 and
            // r2/sigma^2 (1/sigma^2 precomputed per blob) give the same
            // quantities.
            const fix::Vec v = fix::vec(rx, ry);
            if (fix::apart(v, rx, ry)) {
              int ge;
              const double g = t.cir[j], ic = t.icor2[j];
              const uint64_t gm = fix::mantissa(g, ge);
              // 1/sigma^2 of zero or below the normal range makes x = 0 with any mantissa
              const int ce = (int)(fix::bits(ic) >> 52);
              const uint64_t cm = ((fix::bits(ic) << 10) & 0x3fffffffffffffffull) | 0x4000000000000000ull;
              fix::add_pair(near, v, fix::hi32(fix::bits(rx)), fix::hi32(fix::bits(ry)), gm, ge,
                            fix::hi32(fix::bits(g)), cm, ce, s_exp_int, s_exp_frac, a.one);
            }
          }
        }
        if (sub == 0) n_pairs += (unsigned)(e - b);
      }
      __syncwarp();
    } else {
      // a cell's four children can add four entries to a target's queue
      if (__any_sync(0xffffffffu, nq > kQueue - 4)) flush(false);
      // each of a target's first four lanes tests one child
      const int cc = sub < 4 ? t.child[4 * (long)c + sub] : -1;
      bool desc = false;
      if (act && cc >= 0) {
        // The reference's test is region > theta * sqrt(d2), each step
        // rounded.  Squared, region^2 > theta^2 d2, it needs no square
        // root: below the cell's bound mb.x (region^2 / (theta^2 (1 +
        // 2e-13))) it surely descends, above mb.y (the same with 1 -
        // 2e-13) it surely accepts (the roundings of either side and of
        // the bounds are below 1e-15 relative); only a d2 between the two
        // takes the exact rounded path.
        //
        // An FP64 instruction costs this GPU's SM sub-partition about 64
        // issue cycles, an FP32 one 1, so d2 is first formed in FP32 from
        // the hi/lo pairs: dxf = (xh - cxh) + (xl - cxl).  Its error is at
        // most 2^-23 |dx| + 2^-46 (|x| + |cx|), and so
        //   |d2f - d2| <= 3 2^-23 d2 + 2^-45 S (|dxf| + |dyf|) + (...)^2,
        // S = |x| + |y| + |cx| + |cy|.  err below takes 2^-20 d2f and
        // 2^-44 S, over twice that, so d2f + err < the FP32 lower bound
        // (rounded down from mb.x) means d2 < mb.x, and d2f - err > the
        // upper one (rounded up from mb.y) d2 > mb.y: the FP64 test would
        // decide the same.  Anything else (and any infinity or NaN on the
        // way, where a comparison fails) takes the FP64 test as before.
        const float4 cf = t.cf32[cc];
        const float2 mf = t.macf[cc];
        const float dxf = __fadd_rn(__fsub_rn(xh, cf.x), __fsub_rn(xl, cf.y));
        const float dyf = __fadd_rn(__fsub_rn(yh, cf.z), __fsub_rn(yl, cf.w));
        const float d2f = __fmaf_rn(dxf, dxf, __fmul_rn(dyf, dyf));
        const float ef = __fmul_rn(0x1p-44f, __fadd_rn(sxy, __fadd_rn(fabsf(cf.x), fabsf(cf.z))));
        const float err = __fmaf_rn(0x1p-20f, d2f, __fmul_rn(ef, __fadd_rn(__fadd_rn(fabsf(dxf), fabsf(dyf)), ef)));
        if (__fadd_ru(d2f, err) < mf.x) {
          desc = true;
        } else if (__fsub_rd(d2f, err) > mf.y && d2f <= 3.0e38f) {
          desc = false;
        } else {
          const double2 mb = t.mac[cc];
          const double dx = __dsub_rn(x, t.cx[cc]);
          const double dy = __dsub_rn(y, t.cy[cc]);
          const double d2 = __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
          if (d2 < mb.x) {
            desc = true;
          } else if (d2 > mb.y) {
            desc = false;
          } else {
            desc = t.region[cc] > __dmul_rn(theta, __dsqrt_rn(d2));
          }
        }
      }
      const unsigned dmask = __ballot_sync(0xffffffffu, desc);
      const unsigned amask = __ballot_sync(0xffffffffu, act && cc >= 0 && !desc);
      const unsigned mine = (amask >> (lane & ~(kShare - 1))) & 0xfu;  // children this target accepts
      if (nt >= 2) {
        if ((mine >> sub) & 1u)
          s_queue[warp][tgt][(qh + (unsigned)(nq + __popc(mine & ((1u << sub) - 1u)))) & (kQueue - 1)] = cc;
        nq += __popc(mine);
      }
      n_m2s += __popc(mine);
      // lane q < 4 pushes child q with the lanes of the targets that open it
      const unsigned open = (dmask >> sub) & kEachTarget;
      const unsigned some = __ballot_sync(0xffffffffu, open != 0) & 0xfu;
      const int cnt = __popc(some);
      if (top + cnt >= kStackCap) {
        overflow = true;
        break;
      }
      if (lane < 4 && open) {
        const int at = top + 1 + __popc(some & ((1u << lane) - 1u));
        s_cell[warp][at] = cc;
        s_mask[warp][at] = open * kLanes;
      }
      top += cnt;
      __syncwarp();
    }
  }
  flush(true);
  if (overflow && lane == 0) set_err(a.st, TREE2D_ERR_TIMEOUT);
  // the lanes' sums
  double2 phi = kForm != kFormFp64 ? make_double2(fix::to_double(far.x, far.xl, far.e), fix::to_double(far.y, far.yl, far.e))
                                   : make_double2(0.0, 0.0);
  phi.x = __dadd_rn(phi.x, far64.x);
  phi.y = __dadd_rn(phi.y, far64.y);
  double2 dir = make_double2(fix::to_double(near.x.v, near.x.l, near.x.e), fix::to_double(near.y.v, near.y.l, near.y.e));
  for (int o = 1; o < kShare; o <<= 1) {
    phi.x = __dadd_rn(phi.x, __shfl_xor_sync(0xffffffffu, phi.x, o));
    phi.y = __dadd_rn(phi.y, __shfl_xor_sync(0xffffffffu, phi.y, o));
    dir.x = __dadd_rn(dir.x, __shfl_xor_sync(0xffffffffu, dir.x, o));
    dir.y = __dadd_rn(dir.y, __shfl_xor_sync(0xffffffffu, dir.y, o));
  }
  if (valid && sub == 0) {
    // fmm.c:115-117 with its direct part 0.5 a / pi
    double u = (0.5 * (phi.y + dir.x)) / kPi;
    double v = (0.5 * (phi.x + dir.y)) / kPi;
    // the fixed-point terms do not carry an infinity or a NaN of the target
    if (!isfinite(x) || !isfinite(y)) {
      if ((nt >= 2 && n_m2s > 0) || (n_pairs > 0 && !isnan(x) && !isnan(y))) u = v = NAN;
    }
    const long o = a.out_idx ? a.out_idx[i] : i;
    a.uv[2 * o] = overflow ? NAN : u;
    a.uv[2 * o + 1] = overflow ? NAN : v;
  }
  unsigned long long m2s = valid && sub == 0 ? n_m2s : 0;
  for (int o = 16; o; o >>= 1) {
    m2s += __shfl_xor_sync(0xffffffffu, m2s, o);
    n_pairs += __shfl_xor_sync(0xffffffffu, n_pairs, o);
  }
  if (lane == 0) {
    atomicAdd(&a.st->n_m2s, m2s);
    atomicAdd(&a.st->n_pairs, n_pairs);
  }
}

// The opening test's bounds per cell for a given theta: squared distances
// d2 with d2 < lo surely have region > theta sqrt(d2) (the cell is opened),
// d2 > hi surely not (it is accepted), with a relative margin of 2e-13 that
// covers the roundings of the reference's test and of the bounds.  With
// theta <= 0 the reference's test opens every cell (region > 0 >= theta r):
// both bounds are +inf.
//
// For the FP32 pre-test of k_eval: the centre as two FP32 pairs (hi = the
// nearest float, lo = the rest, rounded) and the bounds rounded outwards to
// FP32; a lower bound below 1e-30 becomes -1 and an upper one below 1e-30
// +inf (no sure answer: the FP32 error bound does not cover subnormals).
__global__ void k_mac_bounds(Tree t, double theta, int nt, longlong2 *fixed) {
  chain_wait();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= t.ncell) return;
  const double r2 = t.region[c] * t.region[c], th2 = theta * theta;
  const double2 mb = theta > 0.0 ? make_double2(r2 / (th2 * (1.0 + 2e-13)), r2 / (th2 * (1.0 - 2e-13)))
                                 : make_double2(INFINITY, INFINITY);
  t.mac[c] = mb;
  const double cx = t.cx[c], cy = t.cy[c];
  const float cxh = __double2float_rn(cx), cyh = __double2float_rn(cy);
  t.cf32[c] = make_float4(cxh, __double2float_rn(cx - (double)cxh), cyh, __double2float_rn(cy - (double)cyh));
  t.macf[c] = make_float2(mb.x >= 1e-30 ? __double2float_rd(mb.x) : -1.0f,
                          mb.y >= 1e-30 ? __double2float_ru(mb.y) : INFINITY);
  if (fixed) {
    // The coefficients in fixed point, the cell's scale in the last entry
    // (whose a_k the sums do not use).  `fixed` may be t.coef: a thread has
    // read what it needs of its cell before it writes entry k.
    const double2 *src = t.coef + (size_t)c * nt;
    longlong2 *dst = fixed + (size_t)c * nt;
    const fix::CellScale sc = fix::cell_scale(nt - 1, t.region[c], theta, [&](int k, double &re, double &im) {
      const double2 a = src[k];
      re = a.x;
      im = a.y;
    });
    const int k0 = fix::first_pair_term(theta);
    for (int k = 0; k < nt - 1 && sc.es != fix::kLeave; k++) {  // else the FP64 ones stay
      const double2 a = src[k];
      if (nt - 1 > k0 && k >= k0) {
        float4 v;
        fix::pair_coef(a.x, k, sc, v.x, v.y);
        fix::pair_coef(a.y, k, sc, v.z, v.w);
        reinterpret_cast<float4 *>(dst)[k] = v;
      } else {
        dst[k] = make_longlong2(fix::fix_coef(a.x, k, sc), fix::fix_coef(a.y, k, sc));
      }
    }
    dst[nt - 1] = make_longlong2(sc.es, sc.eb);
  }
}

// Opening angle up to which the multipole sums run in fixed point: es can
// reach log2(0.71 R), the farthest blob's, so that the coefficients do not
// grow with k (fix::cell_scale).  Above it FP64, as before.
constexpr double kFixTheta = 2.0 * fix::kHalfTheta;

// Once per upward pass: the coefficients may be converted in place.
cudaError_t mac_bounds(Workspace &ws, const Tree &t, cudaStream_t s) {
  if (ws.mac_ready || t.ncell <= 0) return cudaSuccess;
  const Params &p = t.params;
  ws.fix = nullptr;
  if (p.theta <= kFixTheta && p.nterms >= 2) {
    if (ws.cell_arena.fixed()) {
      ws.fix = reinterpret_cast<long long *>(t.coef);
    } else {
      const size_t entries = 2 * (size_t)t.ncell * p.nterms;
      const cudaError_t e = ws.fix_arena.reserve(Arena::bytes_for(entries, 8));
      if (e != cudaSuccess) return e;
      ws.fix_arena.reset();
      ws.fix = ws.fix_arena.take<long long>(entries);
    }
  }
  chained(k_mac_bounds, (t.ncell + 63) / 64, 64, 0, s)(t, p.theta, p.nterms, reinterpret_cast<longlong2 *>(ws.fix));
  ::t2d::g_launches.fetch_add(1, std::memory_order_relaxed);
  const cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) ws.mac_ready = true;
  return e;
}

}  // namespace

int plain_upward(Workspace &ws, const Tree &t, cudaStream_t s) {
  const int nt = t.params.nterms;
  if (t.ncell <= 0) return TREE2D_OK;
  ws.mac_ready = false;  // the climb uses the bounds' memory
  chained(k_climb_init, ((t.n > t.ncell ? t.n : t.ncell) + 255) / 256, 256, 0, s)(t, nt);
  if (t.nleaf > 0 && nt > 0) chained(k_upward, (t.nleaf + 3) / 4, 128, 0, s)(t, nt);
  ::t2d::g_launches.fetch_add(2, std::memory_order_relaxed);
  T2D_CUDA_TRY(cudaGetLastError());
  return TREE2D_OK;
}

// Lanes per target.  A small tree's evaluation has few warps and waits on
// latencies: more lanes leave fewer targets to a warp, for more warps; a large
// one's fills the chip anyway, and sharing a target costs.  The lines grow with
// the leaf size, as a target's work does.  Measured evaluation, us, with 4 / 8
// / 16 lanes, Lamb-Oseen blobs:
//    num_p        33                65                250                500
//    4,096   247 / 157 / 114   296 / 183 / 112   593 / 318 / 179    699 / 368 / 206
//    8,192   286 / 181 / 169   337 / 218 / 169   808 / 429 / 296   1017 / 540 / 357
//   12,288   307 / 223 / 244   371 / 268 / 262   855 / 524 / 440   1536 / 870 / 670
//   32,768   531 / 507 / 589   620 / 558 / 607  1136 / 953 / 943   2258 / 1844 / 1644
//   65,536   963 / 985 / 1169 1122 / 1092 / 1233 2346 / 2032 / 2043 3971 / 3333 / 3205
//  131,072  1797 / 1938 / -   2070 / 2138 / -   3608 / 3423 / 3690 6871 / 6301 / 6465
// The lines lie where the sums of a row change hands, to within 3% (65,536
// blobs with num_p 33 take eight lanes although four are 2% ahead), and hold
// for other distributions as far as their targets' work is alike.  By the tree,
// not the targets' number: a point's sums do not depend on how many points are
// asked for.
int eval_share(int n, int num_p) {
  if (n <= 8192 || (n <= 65536 && n <= 200l * num_p)) return 16;
  if (n <= 65536 || (n <= 131072 && n <= 1024l * num_p)) return 8;
  return 4;
}

template <int kShare>
auto eval_kernel(double theta) {
  return theta > kFixTheta         ? k_eval<kFormFp64, kShare>
         : theta > fix::kHalfTheta ? k_eval<kFormFull, kShare>
                                   : k_eval<kFormHalf, kShare>;
}

int plain_evaluate(Workspace &ws, const Tree &t, int ntgt, const double *tx, const double *ty, const int *out_idx,
                   double *uv, cudaStream_t s) {
  if (ntgt <= 0) return TREE2D_OK;
  const Params &p = t.params;
  T2D_CUDA_TRY(mac_bounds(ws, t, s));
  EvalArgs a{t, p.nterms, p.theta, ntgt, tx, ty, out_idx, uv, ws.status, reinterpret_cast<const longlong2 *>(ws.fix),
             fix::first_pair_term(p.theta),
             reinterpret_cast<const void *>(ws.fix) != reinterpret_cast<const void *>(t.coef), fix::One()};
  const int share = eval_share(t.n, p.num_p);
  const int warps = (int)(((long)ntgt * share + 31) / 32);
  const int blocks = (warps + kEvalWarps - 1) / kEvalWarps;
  auto kernel = share == 16 ? eval_kernel<16>(p.theta) : share == 8 ? eval_kernel<8>(p.theta) : eval_kernel<4>(p.theta);
  chained(kernel, blocks, kEvalWarps * 32, 0, s)(a);
  ::t2d::g_launches.fetch_add(1, std::memory_order_relaxed);
  T2D_CUDA_TRY(cudaGetLastError());
  return TREE2D_OK;
}

}  // namespace t2d
