// extern "C" view of csrc/fix64.cuh for test_fix64.py (host build).
#include "../2dfmm_gb300/csrc/fix64.cuh"
using namespace t2d::fix;

// one term per call: the pair's two components, over n pairs
extern "C" void pair_terms(int n, const double *dx, const double *dy, const double *g, const double *ic,
                           const uint64_t *ints, const uint64_t *fracs, double *out) {
  for (int i = 0; i < n; i++) {
    Sum2 s;
    int ge, ce;
    const uint64_t gm = mantissa(g[i], ge), cm = mantissa(ic[i], ce);
    add_pair(s, vec(dx[i], dy[i]), hi32(bits(dx[i])), hi32(bits(dy[i])), gm, ge, hi32(bits(g[i])), cm, ce, ints, fracs,
             One());
    out[2 * i] = to_double(s.x, s.xl, s.e);
    out[2 * i + 1] = to_double(s.y, s.yl, s.e);
  }
}

// one cell of K coefficients (re, im interleaved) at n offsets, each alone
extern "C" void cell_terms(int K, const double *a, double R, double theta, int n, const double *dx, const double *dy,
                           double *out) {
  const CellScale sc = cell_scale(K, R, theta, [&](int k, double &re, double &im) {
    re = a[2 * k];
    im = a[2 * k + 1];
  });
  auto load = [&](int k) { return Coef{fix_coef(a[2 * k], k, sc), fix_coef(a[2 * k + 1], k, sc)}; };
  auto pair = [&](int k) {
    PairCoef c;
    pair_coef(a[2 * k], k, sc, c.re, c.rl);
    pair_coef(a[2 * k + 1], k, sc, c.im, c.il);
    return c;
  };
  const int k0 = first_pair_term(theta);
  for (int i = 0; i < n; i++) {
    Sum2 s;
    const bool done = theta <= kHalfTheta ? add_multipole<true>(s, dx[i], dy[i], sc, K, k0, load, pair, true, One())
                                          : add_multipole<false>(s, dx[i], dy[i], sc, K, k0, load, pair, true, One());
    if (!done) {  // left to FP64
      out[2 * i] = out[2 * i + 1] = NAN;
      continue;
    }
    out[2 * i] = to_double(s.x, s.xl, s.e);
    out[2 * i + 1] = to_double(s.y, s.yl, s.e);
  }
}

// running sum of n terms m 2^e, settled every 32
extern "C" void sum_terms(int n, const long long *mx, const long long *my, const int *e, double *out) {
  Sum2 s;
  for (int i = 0; i < n; i++) {
    if (i % 32 == 0) settle(s);
    add(s, mx[i], my[i], e[i]);
  }
  out[0] = to_double(s.x, s.xl, s.e);
  out[1] = to_double(s.y, s.yl, s.e);
}
