// p2_tensor.cuh — BabyBear width-16 Poseidon2 with its linear layers on the tensor cores.
//
// The permutation's linear layers are 16 x 16 matrices over F_p and its S-boxes are
// element-wise, so the layers run as integer matrix products on the tensor cores
// (tcgen05.mma kind::i8, 128 x N x 32 steps, exact s32 accumulation in TMEM) while the
// integer pipes do the S-boxes.  One thread owns one permutation, and a group of 128
// threads (four warps, the 128 TMEM lanes) shares one product per layer:
//   A (TMEM): row = thread; the thread's u32 words, written by tcgen05.st.  The four bytes of a
//      word ARE four consecutive 8-bit operands, so no limb is ever split off.
//   B (shared memory): the layer's matrix.  Entry c of the layer, against byte l' of an input
//      word, contributes c * 2^(8 l') mod p; byte l of that constant goes to column (output, l).
//      (A small entry c <= 255 simply puts c in column (output, l').)
//   D (TMEM): four s32 accumulators per output word, weights 2^0, 2^8, 2^16, 2^24.
// A thread reads its accumulators back (tcgen05.ld), recombines each output with six integer
// operations and a Barrett quotient instead of the additions mod p of the layer, and goes on with
// the next S-box.  Round constants ride on a constant-one operand byte.  The thirteen
// partial rounds have one S-box each and are linear otherwise: the S-box inputs y_k are
// functionals of the state that entered them plus known multiples of the S-box outputs
// w_j (j < k), so three products (blocks of 4, 4 and 5 rounds) and a few scalar products
// replace thirteen dense rounds.  The last layer of a permutation and the first layer of the
// next absorb step are one product.
#pragma once
#include "field.cuh"
#include "limbs.cuh"
#include "poseidon2.cuh"
#include "tcgen05.cuh"

namespace zkb {
namespace p2t {
using namespace tc;

constexpr int NF = 8, NP = 13;   // rounds this form is built for (R_F, R_P)
constexpr int GROUP = 128;       // threads (= permutations) of one product
constexpr int MAX_GROUPS = 5;    // per block: 5 * 96 columns <= 512
constexpr int COLS = 96;         // TMEM columns of a group: D 64, Z 16, W 16
constexpr int COL_D = 0, COL_Z = 64, COL_W = 80;
constexpr int W_ONE = 13;        // word of the W region holding the constant 1
constexpr uint32_t P = BabyBear::P;
constexpr uint32_t SMALL_BIAS = 0x4B400000u;  // see recombine_small

// ------------------------------------------------------------- coefficients (host)
// Each coefficient is stored as its four limb multiples c * 2^(8 l) mod p.
struct Coefs {
  uint32_t in[16][16][4];    // M * R: canonical input word -> state (Montgomery)
  uint32_t y[13][16][4];     // state that entered the last initial full round's layer -> y_k
  uint32_t oz[16][16][4];    // ... -> state after the partial rounds
  uint32_t ow[16][13][4];    // w_j -> state after the partial rounds
  uint32_t c[13][4];         // y_k += c[k-1-j] * w_j
  uint32_t fin[16][16][4];   // M * R^-1: last S-box outputs -> canonical state
  uint32_t cm[13];           // c[i] as the centred Montgomery multiplier of a scalar product, negated
  uint8_t m[16][16];         // external matrix
};

constexpr uint32_t mulp(uint32_t a, uint32_t b) { return (uint32_t)((uint64_t)a * b % P); }
constexpr uint32_t addp(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a + b) % P); }
constexpr uint32_t powp(uint32_t a, uint32_t e) {
  uint32_t r = 1;
  while (e) {
    if (e & 1) r = mulp(r, a);
    a = mulp(a, a);
    e >>= 1;
  }
  return r;
}
constexpr void limbs(uint32_t (&o)[4], uint32_t c) {
  for (int l = 0; l < 4; l++) {
    o[l] = c;
    c = mulp(c, 256);
  }
}

constexpr Coefs make_coefs() {
  Coefs k{};
  const uint32_t R = (uint32_t)((1ull << 32) % P), Ri = powp(R, P - 2);
  const uint8_t m4[4][4] = {{2, 3, 1, 1}, {1, 2, 3, 1}, {1, 1, 2, 3}, {3, 1, 1, 2}};
  for (int i = 0; i < 16; i++)
    for (int j = 0; j < 16; j++) k.m[i][j] = (uint8_t)(m4[i % 4][j % 4] * (i / 4 == j / 4 ? 2 : 1));
  // internal diagonal V (poseidon2.cuh: bb16::internal_round)
  const uint32_t i2 = powp(2, P - 2), i8 = powp(256, P - 2), i27 = powp(1u << 27, P - 2);
  const uint32_t d[16] = {P - 2, 1, 2, i2, 3, 4, P - i2, P - 3, P - 4, i8, mulp(i2, i2), mulp(i2, mulp(i2, i2)),
                          i27, P - i8, P - powp(16, P - 2), P - i27};
  // a = A e0, Abar = A with column 0 cleared; Abar v = d_i v_i + sum_{j>=1} v_j (lane 0 in: 0)
  uint32_t a[16] = {};
  for (int i = 0; i < 16; i++) a[i] = i == 0 ? addp(d[0], 1) : 1;
  // functionals f_k = e0^T Abar^k M and c_k = e0^T Abar^k a
  uint32_t f[16] = {};
  f[0] = 1;
  for (int t = 0; t < 13; t++) {
    for (int j = 0; j < 16; j++) {
      uint32_t s = 0;
      for (int i = 0; i < 16; i++) s = addp(s, mulp(f[i], k.m[i][j]));
      limbs(k.y[t][j], s);
    }
    uint32_t c = 0;
    for (int i = 0; i < 16; i++) c = addp(c, mulp(f[i], a[i]));
    limbs(k.c[t], c);
    const uint32_t neg = mulp(c ? P - c : 0, R);
    k.cm[t] = neg > P / 2 ? neg - P : neg;  // centred (two's complement)
    uint32_t sum = 0;
    for (int i = 0; i < 16; i++) sum = addp(sum, f[i]);
    uint32_t g[16] = {};
    for (int j = 1; j < 16; j++) g[j] = addp(sum, mulp(d[j], f[j]));
    for (int j = 0; j < 16; j++) f[j] = g[j];
  }
  // columns after the partial rounds
  for (int j = 0; j < 16 + 13; j++) {
    uint32_t v[16] = {};
    int steps = 13;
    if (j < 16) {
      for (int i = 0; i < 16; i++) v[i] = k.m[i][j];
    } else {
      for (int i = 0; i < 16; i++) v[i] = a[i];
      steps = 12 - (j - 16);
    }
    for (int t = 0; t < steps; t++) {
      uint32_t sum = 0;
      for (int i = 1; i < 16; i++) sum = addp(sum, v[i]);
      for (int i = 1; i < 16; i++) v[i] = addp(sum, mulp(d[i], v[i]));
      v[0] = sum;
    }
    // the next full round adds its constants and applies x^7 to this state directly
    for (int i = 0; i < 16; i++) {
      if (j < 16)
        limbs(k.oz[i][j], v[i]);
      else
        limbs(k.ow[i][j - 16], v[i]);
    }
  }
  for (int i = 0; i < 16; i++)
    for (int j = 0; j < 16; j++) {
      limbs(k.in[i][j], mulp(k.m[i][j], R));
      limbs(k.fin[i][j], mulp(k.m[i][j], Ri));
    }
  return k;
}

// True when these parameters are the instance the tables above describe.
inline bool usable(const P2Params<BabyBear, 16> &p) {
  return p.diag_kind == 1 && p.rounds_f == NF && p.rounds_p == NP;
}


// ------------------------------------------------------------------ layer matrices
// A slab is one 32-byte K step: N rows x 32 bytes in 8 x 16-byte core matrices,
// [k / 16][n / 8][n % 8][k % 16].  Image offsets (bytes); the first five are copied as they lie.
constexpr int SLAB64 = 2048;
constexpr int I_EXT = 0;                      // M against Z: 2 slabs
constexpr int I_Y = I_EXT + 2 * SLAB64;       // 2 slabs
constexpr int I_O = I_Y + 2 * SLAB64;         // Z 2 slabs, W 2
constexpr int I_B2 = I_O + 4 * SLAB64;        // N = 48
constexpr int I_B3 = I_B2 + 48 * 32;          // N = 32
constexpr int COMMON = I_B3 + 32 * 32;
constexpr int I_FIN8 = COMMON;                // N = 32: 2 slabs of 1024
constexpr int I_FIN16 = I_FIN8 + SLAB64;      // N = 64: 2 slabs
constexpr int I_IN16 = I_FIN16 + 2 * SLAB64;  // 16 canonical words in: 2 slabs
constexpr int I_ABS = I_IN16 + 2 * SLAB64;    // absorb chunks of 8, 1, 2, ... 7 words: Z 2 slabs, input 1
constexpr int ABS_BYTES = 3 * SLAB64;
constexpr int IMAGE = I_ABS + 8 * ABS_BYTES;

// Column of an output's weight-2^(8 l) accumulator among its four: 0, 2, 1, 3, so that the low
// halves of adjacent columns pack into a0 + a2 2^16 and a1 + a3 2^16.
__host__ __device__ constexpr int acc_col(int l) { return l == 1 ? 2 : l == 2 ? 1 : l; }
__host__ __device__ constexpr int slot(int N, int n, int k) {
  return ((k >> 4) * (N >> 3) + (n >> 3)) * 128 + (n & 7) * 16 + (k & 15);
}

struct alignas(16) Image {
  uint8_t b[IMAGE];
  constexpr void gen(int base, int N, int i, int j, const uint32_t (&c)[4]) {
    for (int lp = 0; lp < 4; lp++)
      for (int l = 0; l < 4; l++) b[base + slot(N, 4 * i + acc_col(l), 4 * j + lp)] = (uint8_t)(c[lp] >> (8 * l));
  }
  constexpr void small(int base, int N, int i, int j, uint32_t c) {
    for (int l = 0; l < 4; l++) b[base + slot(N, 4 * i + acc_col(l), 4 * j + l)] = (uint8_t)c;
  }
};

constexpr Image make_image() {
  Image m{};
  const Coefs k = make_coefs();
  for (int i = 0; i < 16; i++)
    for (int j = 0; j < 16; j++) {
      m.small(I_EXT, 64, i, j, k.m[i][j]);
      m.gen(I_O, 64, i, j, k.oz[i][j]);
      if (i < 13) m.gen(I_Y, 64, i, j, k.y[i][j]);
      if (j < 13) m.gen(I_O + 2 * SLAB64, 64, i, j, k.ow[i][j]);
      if (i < 8) m.gen(I_FIN8, 32, i, j, k.fin[i][j]);
      m.gen(I_FIN16, 64, i, j, k.fin[i][j]);
      m.gen(I_IN16, 64, i, j, k.in[i][j]);
      // y_k += c[k-1-j] w_j: block 2 (j 0..3 -> k 4..12) and block 3 (j 4..7 -> k 8..12)
      if (i < 9 && j < 4) m.gen(I_B2, 48, i, j, k.c[i + 3 - j]);
      if (i < 5 && j >= 4 && j < 8) m.gen(I_B3, 32, i, j, k.c[i + 7 - j]);
    }
  // Absorbing `rem` words: lane l < rem takes its input word, the others keep the last
  // permutation's state M z; the first layer of the next is M again.
  for (int rem = 1; rem <= 8; rem++) {
    const int base = I_ABS + (rem % 8) * ABS_BYTES;
    for (int i = 0; i < 16; i++) {
      for (int j = 0; j < 16; j++) {
        uint32_t s = 0;
        for (int l = rem; l < 16; l++) s += (uint32_t)k.m[i][l] * k.m[l][j];
        m.small(base, 64, i, j, s);  // at most 255: checked below
      }
      for (int j = 0; j < rem; j++) m.gen(base + 2 * SLAB64, 64, i, j, k.in[i][j]);
    }
  }
  return m;
}
constexpr bool absorb_fits() {
  const Coefs k = make_coefs();
  for (int i = 0; i < 16; i++)
    for (int j = 0; j < 16; j++) {
      int s = 0;
      for (int l = 1; l < 16; l++) s += k.m[i][l] * k.m[l][j];
      if (s > 255) return false;
    }
  return true;
}
static_assert(absorb_fits(), "the fused absorb layer needs entries below 256");

// The largest a0 + a1 2^8 or a2 + a3 2^8 that any output of a layer recombined by limbs::babybear can have:
// operand bytes of 255 throughout, and the largest constant (0.489 p).
constexpr uint64_t max_half() {
  const Image m = make_image();
  struct Part {
    int base, N, steps, col0;  // matrix rows of accumulator columns col0 .. col0 + N
  };
  // the products that add up in one accumulator
  const Part layers[6][3] = {{{I_IN16, 64, 2, 0}},
                             {{I_ABS, 64, 3, 0}},  // every absorb matrix in turn, below
                             {{I_Y, 64, 2, 0}, {I_B2, 48, 1, 16}, {I_B3, 32, 1, 32}},
                             {{I_O, 64, 4, 0}},
                             {{I_FIN8, 32, 2, 0}},
                             {{I_FIN16, 64, 2, 0}}};
  uint64_t best = 0;
  for (int layer = 0; layer < 6; layer++)
    for (int a = 0; a < (layer == 1 ? 8 : 1); a++) {
      uint64_t sum[64] = {};
      for (const Part &p : layers[layer])
        for (int n = 0; n < p.N; n++)
          for (int k = 0; k < 32 * p.steps; k++)
            sum[p.col0 + n] += m.b[p.base + a * ABS_BYTES + (k / 32) * p.N * 32 + slot(p.N, n, k % 32)];
      for (int i = 0; i < 16; i++)
        for (int h = 0; h < 4; h += 2) {
          const uint64_t v = 255 * (sum[4 * i + acc_col(h)] + 256 * sum[4 * i + acc_col(h + 1)]) + 65535;
          best = v > best ? v : best;
        }
    }
  return best;
}
static_assert(max_half() <= limbs::BABYBEAR_MAX_HALF, "accumulators exceed the recombination's range");

#ifdef __CUDACC__
static __device__ constexpr Coefs kCoefs = make_coefs();
static __device__ const Image kImage = make_image();

// ------------------------------------------------------------------- shared memory
enum Mode { SPONGE = 0, SPONGE_ANY = 1, STATE16 = 2, PERM16 = 3 };
constexpr int S_C = COMMON;                  // constants: first layer, rounds 1-3, y, terminal 1-3
constexpr int S_FIN = S_C + 8 * SLAB64;      // last layer: 2 slabs of N = 32, or of N = 64 (PERM16)
constexpr int S_IN = S_FIN + 2 * SLAB64;     // 16-word input (2 slabs), or absorb matrices: full chunk,
                                             // then the partial one (SPONGE) or those of 1..7 words (SPONGE_ANY)
constexpr int S_LAST = S_IN + ABS_BYTES;
__host__ __device__ constexpr int smem_tables(Mode m) {
  return m == SPONGE ? S_LAST + ABS_BYTES : m == SPONGE_ANY ? S_LAST + 7 * ABS_BYTES : S_IN + 2 * SLAB64;
}
// TMEM address, the image's mbarrier and one per group follow the tables.
__host__ __device__ constexpr int smem_bytes(Mode m) { return smem_tables(m) + 16 + 8 * MAX_GROUPS; }

// The matrices a kernel needs: issued by one thread, completed on mbar.
__device__ __forceinline__ void copy_image(uint32_t sm, Mode mode, int last_rem, uint32_t mbar) {
  const bool sponge = mode == SPONGE || mode == SPONGE_ANY;
  const int fin = mode == PERM16 ? 2 * SLAB64 : SLAB64, in = sponge ? ABS_BYTES : 2 * SLAB64;
  const int last = mode == SPONGE_ANY ? 7 * ABS_BYTES : mode == SPONGE && last_rem != 8 ? ABS_BYTES : 0;
  expect_bytes(mbar, COMMON + fin + in + last);
  bulk_copy(sm, kImage.b, COMMON, mbar);
  bulk_copy(sm + S_FIN, kImage.b + (mode == PERM16 ? I_FIN16 : I_FIN8), fin, mbar);
  bulk_copy(sm + S_IN, kImage.b + (sponge ? I_ABS : I_IN16), in, mbar);
  if (last) bulk_copy(sm + S_LAST, kImage.b + I_ABS + (mode == SPONGE_ANY ? 1 : last_rem) * ABS_BYTES, last, mbar);
}
// The round constants: byte 4 * (W_ONE - 8) of the second W slab meets the constant one.
__device__ __forceinline__ void put_constants(uint8_t *sm, const P2Params<BabyBear, 16> &p) {
  constexpr int kb = 4 * (W_ONE - 8);
  for (int t = threadIdx.x; t < 9 * 16; t += blockDim.x) {
    const int r = t >> 4, i = t & 15;
    uint32_t v;
    int base = S_C + r * SLAB64;
    if (r < 4)
      v = p.rc[r * 16 + i] + (r ? SMALL_BIAS : 0);  // first layer, rounds 1..3
    else if (r == 4)
      v = i < NP ? p.rc[64 + i] : 0;
    else {
      v = p.rc[64 + NP + (r - 5) * 16 + i] + (r > 5 ? SMALL_BIAS : 0);  // terminal rounds 0..3
      base = r == 5 ? I_O + 3 * SLAB64 : S_C + (r - 1) * SLAB64;
    }
#pragma unroll
    for (int l = 0; l < 4; l++) sm[base + slot(64, 4 * i + acc_col(l), kb)] = (uint8_t)(v >> (8 * l));
  }
}

// --------------------------------------------------------------------- arithmetic
__device__ __forceinline__ int smul(int a, int b) { return BabyBear::smul(a, b); }
__device__ __forceinline__ uint32_t lift(int x) { return BabyBear::lift(x); }
__device__ __forceinline__ int smul2(int a0, int b0, int a1, int b1) {
  const int64_t t = (int64_t)a0 * b0 + (int64_t)a1 * b1;
  const int m = (int)((uint32_t)t * BabyBear::PINV);
  return (int)(t >> 32) - __mulhi(m, (int)P);
}
// x^7 of any int32 input, in (-p, p).  A product a b gives |a b| / 2^32 + p / 2 at most in absolute value:
// 1.0334 p for x2, 1.0167 p for x3, 1.0006 p for x4, and the last product's |x3 x4| <= 1.0173 p^2 = 4.124e18 is
// below the 2^31 p = 4.323e18 that keeps its result in (-p, p).
__device__ __forceinline__ int sbox(int x) {
  const int x2 = smul(x, x);
  const int x3 = smul(x2, x);
  const int x4 = smul(x2, x2);
  return smul(x3, x4);
}
__device__ __forceinline__ int recombine(uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3) {
  return limbs::babybear(a0, a1, a2, a3);
}
// An output of the external matrix alone, whose accumulators stay below 2^14 (35 * 255 + 255), read
// in pairs as p02 = a0 + a2 2^16 and p13 = a1 + a3 2^16.  The quotient comes from a3 as a float:
// f = 2^15 + a3 exactly, k = (1 - 0.00146) 2^24 / p, so f k - 273 lies between 0.33 and 0.45 below
// a3 2^24 / p and the fma rounds it to q in the low mantissa bits, 0x4B400000 + q.  The rest of the
// accumulators is worth at most 0.3 p, so t - q p lies in [-0.17 p, 1.25 p]; the 0x4B400000 p that
// is subtracted with it equals 0x4B400000 mod 2^32 (0.627 p), which the round constants carry
// (SMALL_BIAS), leaving [-0.8 p, 0.63 p].
__device__ __forceinline__ int recombine_small(uint32_t p02, uint32_t p13) {
  const uint32_t t = p02 + (p13 << 8);
  const float f = __uint_as_float(__byte_perm(p13, 0x47000000u, 0x7324));
  const float k = (float)(16777216.0 / 2013265921.0 * (1.0 - 0.00146));
  const float q = __fmaf_rn(f, k, 12582912.0f - 273.0f);
  return (int)(t - __float_as_uint(q) * P);
}

// One layer's outputs to S-box outputs: 16 words, each x^7 + p in (0, 2p), stored as the next
// operand.
template <bool SMALL>
__device__ __forceinline__ void full_sbox(const Group &g) {
  uint32_t z[16];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    if constexpr (SMALL) {
      uint32_t a[16];
      ld16_pack(a, g.tw + COL_D + 32 * h);
      ld_wait(a);
#pragma unroll
      for (int e = 0; e < 8; e++) z[8 * h + e] = (uint32_t)sbox(recombine_small(a[2 * e], a[2 * e + 1])) + P;
    } else {
      uint32_t a[16], b[16];
      ld16(a, g.tw + COL_D + 32 * h);
      ld16(b, g.tw + COL_D + 32 * h + 16);
      ld_wait(a);
      ld_wait(b);
#pragma unroll
      for (int e = 0; e < 4; e++) {
        z[8 * h + e] = (uint32_t)sbox(recombine(a[4 * e], a[4 * e + 2], a[4 * e + 1], a[4 * e + 3])) + P;
        z[8 * h + 4 + e] = (uint32_t)sbox(recombine(b[4 * e], b[4 * e + 2], b[4 * e + 1], b[4 * e + 3])) + P;
      }
    }
  }
  st8(g.tw + COL_Z, z);
  st8(g.tw + COL_Z + 8, z + 8);
}

// y_k of a block of partial rounds starting at k0: base (its accumulators) plus the known
// multiples of the block's earlier w: c_0 = -1 exactly, the others as scalar products.
template <int K0, int CNT>
__device__ __forceinline__ void partial_block(const Group &g, int (&w)[13]) {
  int b[CNT];
  {
    uint32_t a[16];
    ld16(a, g.tw + COL_D + 4 * K0);
    ld_wait(a);
#pragma unroll
    for (int e = 0; e < 4; e++) b[e] = recombine(a[4 * e], a[4 * e + 2], a[4 * e + 1], a[4 * e + 3]);
  }
  if constexpr (CNT == 5) {
    uint32_t a[4];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];\n\ttcgen05.wait::ld.sync.aligned;"
                 : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3])
                 : "r"(g.tw + COL_D + 4 * (K0 + 4))
                 : "memory");
    b[4] = recombine(a[0], a[2], a[1], a[3]);
  }
#pragma unroll
  for (int e = 0; e < CNT; e++) {
    int y = b[e];
    if (e > 0) y = (int)(lift(y) - lift(w[K0 + e - 1]));  // - w_{k-1}
#pragma unroll
    for (int q = 2; q <= e; q += 2) {
      // minus (the negated coefficient) products of w_{k-1-i}, i = q-1 and q
      const int t = q + 1 <= e ? smul2(w[K0 + e - q], (int)kCoefs.cm[q - 1], w[K0 + e - q - 1], (int)kCoefs.cm[q])
                               : smul(w[K0 + e - q], (int)kCoefs.cm[q - 1]);
      y = (int)(lift(y) - lift(t));
    }
    w[K0 + e] = sbox(y);
  }
}

// The rounds of one permutation after its first layer's products: leaves the last
// S-box outputs in the Z columns (their layer belongs to the next product).
__device__ __forceinline__ void rounds(Group &g) {
#pragma unroll 1
  for (int r = 0; r < 4; r++) {
    if (r == 0)
      full_sbox<false>(g);
    else
      full_sbox<true>(g);
    arrive(g);
    if (g.lead) {
      const int off = r < 3 ? I_EXT : I_Y;
      mma_slab(g, COL_D, COL_Z, off, 64, false);
      mma_slab(g, COL_D, COL_Z + 8, off + SLAB64, 64, true);
      mma_slab(g, COL_D, COL_W + 8, S_C + (r + 1) * SLAB64, 64, true);
    }
    finish(g);
  }
  {
    int w[13];
    uint32_t o[5];
    partial_block<0, 4>(g, w);
#pragma unroll
    for (int e = 0; e < 4; e++) o[e] = (uint32_t)w[e] + P;
    st4(g.tw + COL_W, o);
    arrive(g);
    if (g.lead) mma_slab(g, COL_D + 16, COL_W, I_B2, 48, true);
    finish(g);
    partial_block<4, 4>(g, w);
#pragma unroll
    for (int e = 0; e < 4; e++) o[e] = (uint32_t)w[4 + e] + P;
    st4(g.tw + COL_W + 4, o);
    arrive(g);
    if (g.lead) mma_slab(g, COL_D + 32, COL_W, I_B3, 32, true);
    finish(g);
    partial_block<8, 5>(g, w);
#pragma unroll
    for (int e = 0; e < 5; e++) o[e] = (uint32_t)w[8 + e] + P;
    st4(g.tw + COL_W + 8, o);
    st1(g.tw + COL_W + 12, o[4]);
    arrive(g);
    if (g.lead) {
      mma_slab(g, COL_D, COL_Z, I_O, 64, false);
      mma_slab(g, COL_D, COL_Z + 8, I_O + SLAB64, 64, true);
      mma_slab(g, COL_D, COL_W, I_O + 2 * SLAB64, 64, true);
      mma_slab(g, COL_D, COL_W + 8, I_O + 3 * SLAB64, 64, true);
    }
    finish(g);
  }
#pragma unroll 1
  for (int r = 0; r < 4; r++) {
    if (r == 0)
      full_sbox<false>(g);
    else
      full_sbox<true>(g);
    if (r == 3) break;
    arrive(g);
    if (g.lead) {
      mma_slab(g, COL_D, COL_Z, I_EXT, 64, false);
      mma_slab(g, COL_D, COL_Z + 8, I_EXT + SLAB64, 64, true);
      mma_slab(g, COL_D, COL_W + 8, S_C + (r + 5) * SLAB64, 64, true);
    }
    finish(g);
  }
}

// The last S-box outputs, as `rounds` left them.
__device__ __forceinline__ void load_z(const Group &g, uint32_t (&z)[16]) {
  st_wait();
  ld16(z, g.tw + COL_Z);
  ld_wait(z);
}

// First layer of an absorb step whose (canonical) input words are in x: `fresh` when the
// state before it is zero, `off` the absorb matrices (S_IN or S_LAST).
__device__ __forceinline__ void absorb(Group &g, const uint32_t (&x)[8], bool fresh, int off) {
  st8(g.tw + COL_W, x);
  arrive(g);
  if (g.lead) {
    mma_slab(g, COL_D, COL_W, off + 2 * SLAB64, 64, false);
    mma_slab(g, COL_D, COL_W + 8, S_C, 64, true);
    if (!fresh) {
      mma_slab(g, COL_D, COL_Z, off, 64, true);
      mma_slab(g, COL_D, COL_Z + 8, off + SLAB64, 64, true);
    }
  }
  finish(g);
}
// First layer of a permutation of 16 canonical words.
__device__ __forceinline__ void enter16(Group &g, const uint32_t (&x)[16]) {
  st8(g.tw + COL_Z, x);
  st8(g.tw + COL_Z + 8, x + 8);
  arrive(g);
  if (g.lead) {
    mma_slab(g, COL_D, COL_Z, S_IN, 64, false);
    mma_slab(g, COL_D, COL_Z + 8, S_IN + SLAB64, 64, true);
    mma_slab(g, COL_D, COL_W + 8, S_C, 64, true);
  }
  finish(g);
}
// The last layer: the first OUT state words, canonical.
template <int OUT>
__device__ __forceinline__ void leave(Group &g, uint32_t (&o)[OUT]) {
  arrive(g);
  if (g.lead) {
    mma_slab(g, COL_D, COL_Z, S_FIN, 4 * OUT, false);
    mma_slab(g, COL_D, COL_Z + 8, S_FIN + 32 * 4 * OUT, 4 * OUT, true);
  }
  finish(g);
#pragma unroll
  for (int q = 0; q < OUT / 4; q++) {
    uint32_t a[16];
    ld16(a, g.tw + COL_D + 16 * q);
    ld_wait(a);
#pragma unroll
    for (int e = 0; e < 4; e++)
      o[4 * q + e] = BabyBear::red(lift(recombine(a[4 * e], a[4 * e + 2], a[4 * e + 1], a[4 * e + 3])));
  }
}

// TMEM columns of a block of `groups` groups (a power of two).
__host__ __device__ constexpr uint32_t tmem_cols(int groups) { return groups == 1 ? 128 : groups == 2 ? 256 : 512; }

// Block set-up: tables, TMEM, barriers.  Every thread calls it; blockDim = groups * GROUP.
__device__ __forceinline__ Group setup(uint8_t *sm, const P2Params<BabyBear, 16> &p, Mode mode, int last_rem,
                                       uint32_t *err) {
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm), ctrl = base + smem_tables(mode);
  const uint32_t tables = ctrl + 8;  // mbarrier of the image copies
  const int groups = blockDim.x / GROUP;
  if (threadIdx.x == 0) {
    init_barrier(tables);
    for (int i = 0; i < groups; i++) init_barrier(ctrl + 16 + 8 * i);
    init_fence();
    copy_image(base, mode, last_rem, tables);
  }
  for (int t = threadIdx.x; t < 8 * SLAB64 / 16; t += blockDim.x)
    reinterpret_cast<uint4 *>(sm + S_C)[t] = make_uint4(0, 0, 0, 0);
  if (threadIdx.x < 32) tmem_alloc(ctrl, tmem_cols(groups));
  fence_before();
  __syncthreads();
  fence_after();
  tables_or_exit(tables, sm + smem_tables(mode), tmem_cols(groups), err);
  put_constants(sm, p);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  fence_before();
  __syncthreads();
  fence_after();
  const Group g = make_group(sm, smem_tables(mode), ctrl + 16, COLS, err);
  st1(g.tw + COL_W + W_ONE, 1);
  return g;
}
__device__ __forceinline__ void teardown(const Group &g, uint8_t *sm, Mode mode) {
  drain(g);
  st_wait();
  fence_before();
  __syncthreads();
  if (threadIdx.x < 32) {
    fence_after();
    tmem_free(*reinterpret_cast<volatile uint32_t *>(sm + smem_tables(mode)), tmem_cols(blockDim.x / GROUP));
  }
}
#endif  // __CUDACC__

}  // namespace p2t
}  // namespace zkb
