// extern "C" view of csrc/position_hash.h for test_position_table.py (host build).
#include "../2dfmm_gb300/csrc/position_hash.h"

extern "C" void position_hashes(int n, const uint64_t *xy, uint64_t *out) {
  for (int i = 0; i < n; i++) out[i] = t2d::position_hash(xy[2 * i], xy[2 * i + 1]);
}
