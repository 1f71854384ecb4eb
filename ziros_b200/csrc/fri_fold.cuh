// fri_fold.cuh — one output of the FRI fold over the BabyBear quartic extension.
#pragma once
#include "field.cuh"

namespace zkb {

// ---------------------------------------------------------- quartic extension
struct Ext4 {
  uint32_t c[4];
};

// a * b with b encoded (Montgomery) coefficientwise; x^4 = 11.
__device__ __forceinline__ Ext4 ext4_mul_enc(const Ext4 &a, const Ext4 &b_enc) {
  using B = BabyBear;
  uint32_t p[7];
#pragma unroll
  for (int k = 0; k < 7; k++) p[k] = 0;
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) p[i + j] = B::add(p[i + j], B::mont(a.c[i], b_enc.c[j]));
  Ext4 r;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const uint32_t h = p[k + 4];
    const uint32_t h2 = B::add(h, h), h4 = B::add(h2, h2), h8 = B::add(h4, h4);
    r.c[k] = B::add(p[k], B::add(B::add(h8, h2), h));  // + 11 h
  }
  r.c[3] = p[3];
  return r;
}

struct Ext4Params {
  Ext4 half_beta_enc;  // beta / 2, Montgomery-encoded coefficients
  uint32_t inv2_enc;
};

// Output i of the fold from the rows r0 = e[2i], r1 = e[2i+1] (n_out = 2^log_n outputs).
__device__ __forceinline__ uint4 fold_ext4_one(uint4 r0, uint4 r1, uint64_t i, int log_n, const Ext4Params &prm,
                                               const uint32_t *__restrict__ itw) {
  using B = BabyBear;
  uint64_t r = log_n ? (__brevll(i) >> (64 - log_n)) : 0;
  const uint32_t w = itw[r];
  Ext4 d;
  d.c[0] = B::mul_tw(B::sub(r0.x, r1.x), w);
  d.c[1] = B::mul_tw(B::sub(r0.y, r1.y), w);
  d.c[2] = B::mul_tw(B::sub(r0.z, r1.z), w);
  d.c[3] = B::mul_tw(B::sub(r0.w, r1.w), w);
  Ext4 t = ext4_mul_enc(d, prm.half_beta_enc);
  uint4 o;
  o.x = B::add(B::mul_tw(B::add(r0.x, r1.x), prm.inv2_enc), t.c[0]);
  o.y = B::add(B::mul_tw(B::add(r0.y, r1.y), prm.inv2_enc), t.c[1]);
  o.z = B::add(B::mul_tw(B::add(r0.z, r1.z), prm.inv2_enc), t.c[2]);
  o.w = B::add(B::mul_tw(B::add(r0.w, r1.w), prm.inv2_enc), t.c[3]);
  return o;
}

}  // namespace zkb
