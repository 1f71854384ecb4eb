// p2_tensor_gl.cuh — Goldilocks Poseidon2 (widths 16 and 12) with its linear layers on the tensor cores.
//
// The form of p2_tensor.cuh for 64-bit words: a thread owns one permutation, 128 threads share one
// 8-bit integer product per layer, a word's eight bytes are eight operands, and an output has eight
// accumulators of weights 2^0 .. 2^56.  Goldilocks needs no Montgomery domain, so the input and
// output layers are the external matrix itself.  The 22 partial rounds run in blocks of four: a
// product per block gives the four S-box inputs as functionals of the state that entered the partial
// rounds and of the earlier S-box outputs, six scalar products the multiples inside the block, and one
// last product the state.  Round constants ride on a word whose one set byte names the layer.
#pragma once
#include "field.cuh"
#include "limbs.cuh"
#include "p2_consts.h"
#include "poseidon2.cuh"
#include "tcgen05.cuh"

namespace zkb {
namespace p2g {
using namespace tc;

constexpr int NF = 8, NP = 22, BLOCKS = 6;  // partial rounds in blocks of 4, 4, 4, 4, 4, 2
constexpr int GROUP = 128;
constexpr uint64_t P = Goldilocks::P;

constexpr uint64_t mulp(uint64_t a, uint64_t b) { return (uint64_t)((unsigned __int128)a * b % P); }
constexpr uint64_t addp(uint64_t a, uint64_t b) { return (uint64_t)(((unsigned __int128)a + b) % P); }

template <int W>
struct Shape {
  static constexpr int N = 8 * W;            // accumulator columns of a layer
  static constexpr int ZS = W / 4;           // K steps (32 bytes, 8 TMEM columns) of the state
  static constexpr int WS = 6;               // and of the partial rounds' outputs with the constants' word
  static constexpr int COL_D = 0, COL_Z = N, COL_W = N + 8 * ZS, COLS = N + 8 * ZS + 8 * WS;
  static constexpr int COL_ONE = COL_W + 2 * NP;  // the constants' word
  static constexpr int MAX_GROUPS = 512 / COLS;
  static constexpr int SLAB = N * 32;        // bytes of a K step of a full layer
  static constexpr int YSLAB = 32 * 32;      // of four outputs
  // tables (shared memory; the image has the same layout up to ABS's end)
  static constexpr int EXT = 0;
  static constexpr int Y = EXT + ZS * SLAB;  // block i: ZS + i steps
  static constexpr int y_off(int i) { return Y + (i * ZS + i * (i - 1) / 2) * YSLAB; }
  static constexpr int O = y_off(BLOCKS);    // Z steps, W steps (the last with the first terminal constants)
  static constexpr int ABS = O + (ZS + WS) * SLAB;  // absorb: Z steps, two of the input
  static constexpr int IMAGE = ABS + (ZS + 2) * SLAB;
  static constexpr int C = IMAGE;            // constants of the other full rounds: one step
  static constexpr int YC = C + SLAB;        // of the blocks: one step of four outputs
  static constexpr int CTRL = YC + YSLAB;
  static constexpr int SMEM = CTRL + 16 + 8 * MAX_GROUPS;
};

__host__ __device__ constexpr int acc_col(int l) { return limbs::goldilocks_col(l); }
__host__ __device__ constexpr int slot(int N, int n, int k) {
  return ((k >> 4) * (N >> 3) + (n >> 3)) * 128 + (n & 7) * 16 + (k & 15);
}

constexpr int m_entry(int i, int j) {
  const int m4[4][4] = {{2, 3, 1, 1}, {1, 2, 3, 1}, {1, 1, 2, 3}, {3, 1, 1, 2}};
  return m4[i % 4][j % 4] * (i / 4 == j / 4 ? 2 : 1);
}

template <int W>
struct alignas(16) Image {
  using S = Shape<W>;
  uint8_t b[S::IMAGE];
  uint64_t c[3];  // y_k += c[k - 1 - j] w_j inside a block
  // coefficient of (output i, input word at byte 8 j) of a matrix of N rows
  constexpr void gen(int base, int N, int i, int j, uint64_t v) {
    for (int lp = 0; lp < 8; lp++) {
      for (int l = 0; l < 8; l++) b[base + slot(N, 8 * i + acc_col(l), 8 * j + lp)] = (uint8_t)(v >> (8 * l));
      v = mulp(v, 256);
    }
  }
  constexpr void small(int base, int N, int i, int j, int v) {
    for (int l = 0; l < 8; l++) b[base + slot(N, 8 * i + acc_col(l), 8 * j + l)] = (uint8_t)v;
  }
};

template <int W>
constexpr Image<W> make_image() {
  using S = Shape<W>;
  Image<W> m{};
  const GoldilocksDiag d = goldilocks_diag(W);
  for (int i = 0; i < W; i++)
    for (int j = 0; j < W; j++) {
      m.small(S::EXT, S::N, i, j, m_entry(i, j));
      // absorb a full chunk: words 8.. keep the last permutation's state M z, then M again
      int s = 0;
      for (int l = 8; l < W; l++) s += m_entry(i, l) * m_entry(l, j);
      m.small(S::ABS, S::N, i, j, s);
      if (j < 8) m.small(S::ABS + S::ZS * S::SLAB, S::N, i, j, m_entry(i, j));
    }
  // A = all-ones + diag(d); a = A e0; Abar = A with column 0 cleared (the S-box replaces word 0).
  // y_k = f_k z + sum_j c_{k-1-j} w_j with f_k = e0^T Abar^k M, c_k = e0^T Abar^k a.
  uint64_t c[NP] = {}, f[W] = {};
  f[0] = 1;
  for (int t = 0; t < NP; t++) {
    for (int j = 0; j < W; j++) {
      uint64_t s = 0;
      for (int i = 0; i < W; i++) s = addp(s, mulp(f[i], m_entry(i, j)));
      m.gen(S::y_off(t / 4), 32, t % 4, j, s);
    }
    c[t] = addp(mulp(f[0], d.d[0]), 0);
    for (int i = 0; i < W; i++) c[t] = addp(c[t], f[i]);
    uint64_t sum = 0;
    for (int i = 0; i < W; i++) sum = addp(sum, f[i]);
    uint64_t g[W] = {};
    for (int j = 1; j < W; j++) g[j] = addp(sum, mulp(d.d[j], f[j]));
    for (int j = 0; j < W; j++) f[j] = g[j];
  }
  for (int t = 4; t < NP; t++)
    for (int j = 0; j < t / 4 * 4; j++) m.gen(S::y_off(t / 4) + S::ZS * S::YSLAB, 32, t % 4, j, c[t - 1 - j]);
  for (int i = 0; i < 3; i++) m.c[i] = c[i];
  // the state after the partial rounds, of z and of the w_j
  for (int j = 0; j < W + NP; j++) {
    uint64_t v[W] = {};
    for (int i = 0; i < W; i++) v[i] = j < W ? m_entry(i, j) : i == 0 ? addp(d.d[0], 1) : 1;
    const int steps = j < W ? NP : NP - 1 - (j - W);
    for (int t = 0; t < steps; t++) {
      uint64_t sum = 0;
      for (int i = 1; i < W; i++) sum = addp(sum, v[i]);
      for (int i = 1; i < W; i++) v[i] = addp(sum, mulp(d.d[i], v[i]));
      v[0] = sum;
    }
    for (int i = 0; i < W; i++)
      if (j < W)
        m.gen(S::O, S::N, i, j, v[i]);
      else
        m.gen(S::O + S::ZS * S::SLAB, S::N, i, j - W, v[i]);
  }
  return m;
}
constexpr bool absorb_fits(int w) {
  for (int i = 0; i < w; i++)
    for (int j = 0; j < w; j++) {
      int s = 0;
      for (int l = 8; l < w; l++) s += m_entry(i, l) * m_entry(l, j);
      if (s > 255) return false;
    }
  return true;
}
static_assert(absorb_fits(12) && absorb_fits(16), "the fused absorb layer needs entries below 256");

// The largest sum over a layer's operand bytes of one accumulator column (constants included).
template <int W>
constexpr uint32_t max_column() {
  using S = Shape<W>;
  const Image<W> m = make_image<W>();
  uint32_t best = 0;
  for (int part = 0; part < 2 + BLOCKS; part++) {
    const int base = part == 0 ? S::O : part == 1 ? S::ABS : S::y_off(part - 2);
    const int N = part < 2 ? S::N : 32, steps = part == 0 ? S::ZS + S::WS : part == 1 ? S::ZS + 2 : S::ZS + part - 2;
    for (int n = 0; n < N; n++) {
      uint32_t sum = 1;  // the constant's byte, against a one
      for (int k = 0; k < 32 * steps; k++) sum += m.b[base + slot(N, n, k)];
      best = sum > best ? sum : best;
    }
  }
  return best;
}
static_assert(max_column<12>() <= limbs::MAX_COLUMN && max_column<16>() <= limbs::MAX_COLUMN,
              "accumulators exceed the recombination's range");

template <int W>
bool usable(const P2Params<Goldilocks, W> &p) {
  return p.diag_kind == 1 && p.rounds_f == NF && p.rounds_p == NP;
}

#ifdef __CUDACC__
template <int W>
__device__ const Image<W> kImage = make_image<W>();

// The constants' word as layer r of the full rounds (0..3 the initial ones, 4..6 terminal 1..3, 7 terminal
// 0) or block r of the partial rounds wants it: byte r set.
template <int W>
__device__ __forceinline__ void select_constants(const Group &g, int r) {
  const uint32_t v = 1u << (8 * (r & 3));
  st2(g.tw + Shape<W>::COL_ONE, r < 4 ? v : 0, r < 4 ? 0 : v);
}
template <int W>
__device__ __forceinline__ void put_constants(uint8_t *sm, const P2Params<Goldilocks, W> &p) {
  using S = Shape<W>;
  constexpr int k0 = 8 * NP - 32 * (S::WS - 1);  // the constants' word in the last W step
  for (int t = threadIdx.x; t < NF * W + NP; t += blockDim.x) {
    uint64_t v;
    int base, N, i, r;
    if (t < NF * W) {
      const int round = t / W;
      i = t % W;
      v = p.rc[round < 4 ? t : NP + t];
      r = round < 4 ? round : round == 4 ? 7 : round - 1;
      base = r == 7 ? S::O + (S::ZS + S::WS - 1) * S::SLAB : S::C;
      N = S::N;
    } else {
      const int k = t - NF * W;
      v = p.rc[4 * W + k];
      r = k / 4;
      i = k % 4;
      base = S::YC;
      N = 32;
    }
#pragma unroll
    for (int l = 0; l < 8; l++) sm[base + slot(N, 8 * i + acc_col(l), k0 + r)] = (uint8_t)(v >> (8 * l));
  }
}

// --------------------------------------------------------------------- arithmetic
// An output of the external matrix: accumulators below 2^14 (35 * 255 + 255), in pairs a0 + a2 2^16,
// a1 + a3 2^16, a4 + a6 2^16, a5 + a7 2^16.
__device__ __forceinline__ uint64_t recombine_small(uint32_t p02, uint32_t p13, uint32_t p46, uint32_t p57) {
  const uint64_t e = p02 + ((uint64_t)p13 << 8), f = p46 + ((uint64_t)p57 << 8);
  return limbs::goldilocks_join(e, f);
}
// An output of any layer.
__device__ __forceinline__ uint64_t recombine(const uint32_t *a) { return limbs::goldilocks(a); }

__device__ __forceinline__ void store_words(uint32_t col, const uint64_t (&z)[4]) {
  const uint32_t v[8] = {(uint32_t)z[0], (uint32_t)(z[0] >> 32), (uint32_t)z[1], (uint32_t)(z[1] >> 32),
                         (uint32_t)z[2], (uint32_t)(z[2] >> 32), (uint32_t)z[3], (uint32_t)(z[3] >> 32)};
  st8(col, v);
}
// Four outputs from accumulator column `col` on.
template <bool SMALL>
__device__ __forceinline__ void load_outputs(uint64_t (&o)[4], uint32_t col) {
  uint32_t a[16];
  if constexpr (SMALL) {
    ld16_pack(a, col);
    ld_wait(a);
#pragma unroll
    for (int e = 0; e < 4; e++) o[e] = recombine_small(a[4 * e], a[4 * e + 1], a[4 * e + 2], a[4 * e + 3]);
  } else {
#pragma unroll
    for (int h = 0; h < 2; h++) {
      ld16(a, col + 16 * h);
      ld_wait(a);
      o[2 * h] = recombine(a);
      o[2 * h + 1] = recombine(a + 8);
    }
  }
}

// One layer's outputs to S-box outputs, stored as the next operand, four words at a time.
template <int W, bool SMALL>
__device__ __forceinline__ void full_sbox(const Group &g) {
  using S = Shape<W>;
#pragma unroll 1
  for (int c = 0; c < W / 4; c++) {
    uint64_t z[4];
    load_outputs<SMALL>(z, g.tw + S::COL_D + 32 * c);
#pragma unroll
    for (int e = 0; e < 4; e++) z[e] = Goldilocks::pow7_any(z[e]);
    store_words(g.tw + S::COL_Z + 8 * c, z);
  }
}

// Steps of a full layer: the matrix at `off` against Z, and the constants (named by the word) unless
// none.
template <int W>
__device__ __forceinline__ void layer(const Group &g, int off, bool constants, bool acc = false) {
  using S = Shape<W>;
#pragma unroll
  for (int s = 0; s < S::ZS; s++) mma_slab(g, S::COL_D, S::COL_Z + 8 * s, off + s * S::SLAB, S::N, acc || s > 0);
  if (constants) mma_slab(g, S::COL_D, S::COL_W + 8 * (S::WS - 1), S::C, S::N, true);
}

// The rounds of one permutation after its first layer's products (whose accumulators may need 32
// bits: the fused absorb); leaves the last S-box outputs in the Z columns.
template <int W>
__device__ __forceinline__ void rounds(Group &g) {
  using S = Shape<W>;
#pragma unroll 1
  for (int r = 0; r < 4; r++) {
    if (r == 0)
      full_sbox<W, false>(g);
    else
      full_sbox<W, true>(g);
    if (r == 3) break;
    select_constants<W>(g, r + 1);
    arrive(g);
    if (g.lead) layer<W>(g, S::EXT, true);
    finish(g);
  }
#pragma unroll 1
  for (int i = 0; i < BLOCKS; i++) {
    select_constants<W>(g, i);
    arrive(g);
    if (g.lead) {
      int off = S::Y + (i * S::ZS + i * (i - 1) / 2) * S::YSLAB;
#pragma unroll 1
      for (int s = 0; s < S::ZS + i; s++, off += S::YSLAB) mma_slab(g, S::COL_D, S::COL_Z + 8 * s, off, 32, s > 0);
      mma_slab(g, S::COL_D, S::COL_W + 8 * (S::WS - 1), S::YC, 32, true);
    }
    finish(g);
    uint64_t w[4];
    load_outputs<false>(w, g.tw + S::COL_D);
    const uint64_t c0 = kImage<W>.c[0], c1 = kImage<W>.c[1], c2 = kImage<W>.c[2];
    using G = Goldilocks;
    w[0] = G::pow7_any(w[0]);
    w[1] = G::pow7_any(G::mul_any<true>(c0, w[0], w[1]));
    if (i + 1 < BLOCKS) {  // the last block has two rounds
      w[2] = G::pow7_any(G::mul_any<true>(c0, w[1], G::mul_any<true>(c1, w[0], w[2])));
      w[3] = G::pow7_any(G::mul_any<true>(c0, w[2], G::mul_any<true>(c1, w[1], G::mul_any<true>(c2, w[0], w[3]))));
      store_words(g.tw + S::COL_W + 8 * i, w);
    } else {
      const uint32_t v[4] = {(uint32_t)w[0], (uint32_t)(w[0] >> 32), (uint32_t)w[1], (uint32_t)(w[1] >> 32)};
      st4(g.tw + S::COL_W + 8 * i, v);
    }
  }
  select_constants<W>(g, 7);
  arrive(g);
  if (g.lead) {
#pragma unroll 1
    for (int s = 0; s < S::ZS + S::WS; s++)
      mma_slab(g, S::COL_D, S::COL_Z + 8 * s, S::O + s * S::SLAB, S::N, s > 0);
  }
  finish(g);
#pragma unroll 1
  for (int r = 0; r < 4; r++) {
    if (r == 0)
      full_sbox<W, false>(g);
    else
      full_sbox<W, true>(g);
    if (r == 3) break;
    select_constants<W>(g, r + 4);
    arrive(g);
    if (g.lead) layer<W>(g, S::EXT, true);
    finish(g);
  }
}

// First layer of an absorb step after a permutation; x: the chunk's eight words.
template <int W>
__device__ __forceinline__ void absorb(Group &g, const uint64_t (&x)[8], bool fresh) {
  using S = Shape<W>;
  const uint64_t lo[4] = {x[0], x[1], x[2], x[3]}, hi[4] = {x[4], x[5], x[6], x[7]};
  store_words(g.tw + S::COL_W, lo);
  store_words(g.tw + S::COL_W + 8, hi);
  select_constants<W>(g, 0);
  arrive(g);
  if (g.lead) {
    mma_slab(g, S::COL_D, S::COL_W, S::ABS + S::ZS * S::SLAB, S::N, false);
    mma_slab(g, S::COL_D, S::COL_W + 8, S::ABS + (S::ZS + 1) * S::SLAB, S::N, true);
    if (fresh)
      mma_slab(g, S::COL_D, S::COL_W + 8 * (S::WS - 1), S::C, S::N, true);
    else
      layer<W>(g, S::ABS, true, true);
  }
  finish(g);
}
// First layer over the state words in the Z columns.
template <int W>
__device__ __forceinline__ void enter(Group &g) {
  select_constants<W>(g, 0);
  arrive(g);
  if (g.lead) layer<W>(g, Shape<W>::EXT, true);
  finish(g);
}
// The last layer; then output(g, c) gives state words 4c.. (some representative).
template <int W>
__device__ __forceinline__ void leave(Group &g) {
  arrive(g);
  if (g.lead) layer<W>(g, Shape<W>::EXT, false);
  finish(g);
}
template <int W>
__device__ __forceinline__ void output(const Group &g, int c, uint64_t (&o)[4]) {
  load_outputs<true>(o, g.tw + Shape<W>::COL_D + 32 * c);
#pragma unroll
  for (int e = 0; e < 4; e++) o[e] = Goldilocks::canon(o[e]);
}

template <int W>
__host__ __device__ constexpr uint32_t tmem_cols(int groups) {
  return groups * Shape<W>::COLS <= 256 ? 256 : 512;
}

// Block set-up: every thread calls it; blockDim = groups * GROUP.
template <int W>
__device__ __forceinline__ Group setup(uint8_t *sm, const P2Params<Goldilocks, W> &p, bool sponge, uint32_t *err) {
  using S = Shape<W>;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm), ctrl = base + S::CTRL, tables = ctrl + 8;
  const int groups = blockDim.x / GROUP;
  if (threadIdx.x == 0) {
    init_barrier(tables);
    for (int i = 0; i < groups; i++) init_barrier(ctrl + 16 + 8 * i);
    init_fence();
    const int bytes = sponge ? S::IMAGE : S::ABS;
    expect_bytes(tables, bytes);
    bulk_copy(base, kImage<W>.b, bytes, tables);
  }
  for (int t = threadIdx.x; t < (S::CTRL - S::C) / 16; t += blockDim.x)
    reinterpret_cast<uint4 *>(sm + S::C)[t] = make_uint4(0, 0, 0, 0);
  if (threadIdx.x < 32) tmem_alloc(ctrl, tmem_cols<W>(groups));
  fence_before();
  __syncthreads();
  fence_after();
  tables_or_exit(tables, sm + S::CTRL, tmem_cols<W>(groups), err);
  put_constants<W>(sm, p);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  fence_before();
  __syncthreads();
  fence_after();
  return make_group(sm, S::CTRL, ctrl + 16, S::COLS, err);
}
template <int W>
__device__ __forceinline__ void teardown(const Group &g, uint8_t *sm) {
  drain(g);
  st_wait();
  fence_before();
  __syncthreads();
  if (threadIdx.x < 32) {
    fence_after();
    tmem_free(*reinterpret_cast<volatile uint32_t *>(sm + Shape<W>::CTRL), tmem_cols<W>(blockDim.x / GROUP));
  }
}
#endif  // __CUDACC__

}  // namespace p2g
}  // namespace zkb
