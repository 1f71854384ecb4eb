// p2_consts.h — Poseidon2 instance parameters on the host.
//
// Constants follow the reference's flatten_round_constants(seed)
// (zkf-metal/src/poseidon2/babybear.rs:76-111, goldilocks.rs:42-83): rand 0.9
// SmallRng::seed_from_u64(seed) (xoshiro256++ expanded by SplitMix64), then
// ExternalLayerConstants::new_from_rng(R_F) (R_F/2 initial then R_F/2 terminal
// width-arrays) and R_P internal draws.  Flat layout [initial | internal | terminal].
#pragma once
#include <cstddef>
#include <cstdint>
#include <vector>

namespace zkb {

enum FieldId : int { FIELD_BABYBEAR = 0, FIELD_GOLDILOCKS = 1 };

struct SmallRng {
  uint64_t s[4] = {};
  // SplitMix64 expansion of a u64 seed into the xoshiro256++ state.
  constexpr explicit SmallRng(uint64_t seed) {
    uint64_t state = seed;
    for (int i = 0; i < 4; i++) {
      state += 0x9e3779b97f4a7c15ull;
      uint64_t z = state;
      z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
      z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
      s[i] = z ^ (z >> 31);
    }
  }
  static constexpr uint64_t rotl(uint64_t x, int k) { return (x << k) | (x >> (64 - k)); }
  // xoshiro256++ (Blackman & Vigna).
  constexpr uint64_t next_u64() {
    const uint64_t res = rotl(s[0] + s[3], 23) + s[0], t = s[1] << 17;
    s[2] ^= s[0];
    s[3] ^= s[1];
    s[1] ^= s[2];
    s[0] ^= s[3];
    s[2] ^= t;
    s[3] = rotl(s[3], 45);
    return res;
  }
  constexpr uint32_t next_u32() { return (uint32_t)(next_u64() >> 32); }
};

// Internal diagonals of the Goldilocks instances (widths 16 and 12).
struct GoldilocksDiag {
  uint64_t d[16];
};
constexpr GoldilocksDiag goldilocks_diag(int width) {
  // MATRIX_DIAG_16_GOLDILOCKS (zkf-metal/src/poseidon2/goldilocks.rs:21-38)
  if (width == 16)
    return {{0xde9b91a467d6afc0ull, 0xc5f16b9c76a9be17ull, 0x0ab0fef2d540ac55ull, 0x3001d27009d05773ull,
             0xed23b1f906d3d9ebull, 0x5ce73743cba97054ull, 0x1c3bab944af4ba24ull, 0x2faa105854dbafaeull,
             0x53ffb3ae6d421a10ull, 0xbcda9df8884ba396ull, 0xfc1273e4a31807bbull, 0xc77952573d5142c0ull,
             0x56683339a819b85eull, 0x328fcbd8f0ddc8ebull, 0xb5101e303fce9cb7ull, 0x774487b8c40089bbull}};
  // The reference ships no width-12 instance.  This diagonal is self-generated: twelve distinct
  // Goldilocks draws, each > 1, from SmallRng seeded with the ASCII bytes "W12DIAG".  It is a
  // parity-unpinned stand-in, not p3's constant.
  GoldilocksDiag g{};
  SmallRng r(0x57313244494147ull);
  for (int n = 0; n < 12;) {
    const uint64_t v = r.next_u64();
    bool ok = v < 0xFFFFFFFF00000001ull && v > 1;
    for (int i = 0; i < n; i++) ok = ok && g.d[i] != v;
    if (ok) g.d[n++] = v;
  }
  return g;
}

// Canonical draws matching p3's StandardUniform samplers.
uint64_t sample_goldilocks(SmallRng &r);
uint32_t sample_babybear(SmallRng &r);  // 31-bit draw taken as Montgomery form

// poseidon2_round_numbers_128 (D = 7).  Returns false when unsupported.
bool p2_round_numbers(int field, int width, int *rounds_f, int *rounds_p);

// Canonical flat constants; empty on unsupported configuration.
std::vector<uint64_t> p2_flat_constants(int field, int width, uint64_t seed);
// Canonical internal diagonal (BabyBear W16 V, Goldilocks W16 MATRIX_DIAG_16, the
// self-generated Goldilocks W12 one).  Empty on unsupported configuration.
const std::vector<uint64_t> &p2_diagonal(int field, int width);

// A fully described Poseidon2 hash configuration: permutation + sponge geometry
// (PaddingFreeSponge<Perm, W, 8, OUT>, TruncatedPermutation<Perm, 2, OUT, W>).
struct HasherSpec {
  int field = 0;
  int width = 16;
  int rate = 8;
  int out = 8;
  int rounds_f = 0, rounds_p = 0;
  std::vector<uint64_t> rc;    // canonical
  std::vector<uint64_t> diag;  // canonical
};
bool make_hasher_spec(int field, int width, uint64_t seed, HasherSpec *out);

}  // namespace zkb
