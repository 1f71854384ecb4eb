// p2_consts.cpp — host generation of Poseidon2 constants (see p2_consts.h).
#include "p2_consts.h"

#include "field.cuh"

namespace zkb {

uint64_t sample_goldilocks(SmallRng &r) {
  for (;;) {
    uint64_t v = r.next_u64();
    if (v < Goldilocks::P) return v;
  }
}

uint32_t sample_babybear(SmallRng &r) {
  for (;;) {
    uint32_t v = r.next_u32() >> 1;
    if (v < BabyBear::P) return BabyBear::from_mont(v);
  }
}

bool p2_round_numbers(int field, int width, int *rf, int *rp) {
  if (field == FIELD_BABYBEAR) {
    if (width == 16) { *rf = 8; *rp = 13; return true; }
    if (width == 24) { *rf = 8; *rp = 21; return true; }
    return false;
  }
  if (field == FIELD_GOLDILOCKS && (width == 8 || width == 12 || width == 16 || width == 20)) {
    *rf = 8;
    *rp = 22;
    return true;
  }
  return false;
}

std::vector<uint64_t> p2_flat_constants(int field, int width, uint64_t seed) {
  int rf, rp;
  if (!p2_round_numbers(field, width, &rf, &rp)) return {};
  SmallRng r(seed);
  auto draw = [&]() -> uint64_t {
    return field == FIELD_BABYBEAR ? (uint64_t)sample_babybear(r) : sample_goldilocks(r);
  };
  std::vector<uint64_t> ext((size_t)rf * width);
  for (auto &v : ext) v = draw();
  std::vector<uint64_t> flat;
  size_t half = (size_t)(rf / 2) * width;
  flat.insert(flat.end(), ext.begin(), ext.begin() + half);
  for (int i = 0; i < rp; i++) flat.push_back(draw());
  flat.insert(flat.end(), ext.begin() + half, ext.end());
  return flat;
}

static std::vector<uint64_t> babybear_diagonal() {
  // V = [-2, 1, 2, 1/2, 3, 4, -1/2, -3, -4, 1/2^8, 1/4, 1/8, 1/2^27, -1/2^8, -1/16, -1/2^27]
  // (zkf-metal/src/poseidon2/babybear.rs:14-58)
  const uint32_t P = BabyBear::P;
  uint32_t inv2 = inv_host<BabyBear>(2);
  auto ip = [&](int e) { return pow_host<BabyBear>(inv2, e); };
  return {P - 2, 1, 2, inv2, 3, 4, P - inv2, P - 3, P - 4, ip(8), ip(2), ip(3), ip(27),
          P - ip(8), P - ip(4), P - ip(27)};
}

static std::vector<uint64_t> goldilocks_diagonal(int width) {
  const GoldilocksDiag g = goldilocks_diag(width);
  return std::vector<uint64_t>(g.d, g.d + width);
}

// Made once: a batch permutation asks for it twice per call.
const std::vector<uint64_t> &p2_diagonal(int field, int width) {
  static const std::vector<uint64_t> bb16 = babybear_diagonal(), gl12 = goldilocks_diagonal(12),
                                     gl16 = goldilocks_diagonal(16), none;
  if (field == FIELD_BABYBEAR && width == 16) return bb16;
  if (field == FIELD_GOLDILOCKS && width == 16) return gl16;
  if (field == FIELD_GOLDILOCKS && width == 12) return gl12;
  return none;
}

bool make_hasher_spec(int field, int width, uint64_t seed, HasherSpec *out) {
  HasherSpec h;
  h.field = field;
  h.width = width;
  h.rate = 8;
  h.out = width == 16 ? 8 : (width == 12 ? 4 : 0);
  if (!h.out) return false;
  if (!p2_round_numbers(field, width, &h.rounds_f, &h.rounds_p)) return false;
  h.rc = p2_flat_constants(field, width, seed);
  h.diag = p2_diagonal(field, width);
  if (h.rc.empty() || h.diag.empty()) return false;
  *out = std::move(h);
  return true;
}

}  // namespace zkb
