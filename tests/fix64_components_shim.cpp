// extern "C" view of csrc/fix64.cuh for test_fix64_components.py (host build):
// the pairs of n offsets summed as the kernels do.
#include "../2dfmm_gb300/csrc/fix64.cuh"
using namespace t2d::fix;

extern "C" void pair_sum(int n, const double *dx, const double *dy, const double *g, const double *ic,
                         const uint64_t *ints, const uint64_t *fracs, double *out) {
  SumXY s;
  for (int i = 0; i < n; i++) {
    if (i % 32 == 0) settle(s);
    int ge, ce;
    const uint64_t gm = mantissa(g[i], ge), cm = mantissa(ic[i], ce);
    add_pair(s, vec(dx[i], dy[i]), hi32(bits(dx[i])), hi32(bits(dy[i])), gm, ge, hi32(bits(g[i])), cm, ce, ints, fracs,
             One());
  }
  out[0] = to_double(s.x.v, s.x.l, s.x.e);
  out[1] = to_double(s.y.v, s.y.l, s.y.e);
}
