// ntt_tc.cu — Goldilocks NTT passes whose small DFTs run on the tensor cores.
//
// A pass of K = LA + LB index bits is the two-phase tile of ntt_tile.cuh (2^LA-point DFTs, a twist, 2^LB-point
// DFTs, the pass twist).  A DFT of R <= 16 points is an R x R matrix of constants, so it runs as an exact
// 8-bit integer product (tcgen05.cuh): a thread's R inputs are a row of operand A (their bytes, as they
// are), the matrix is operand B, and the accumulators recombine to the outputs in about twenty
// instructions each, against the LR levels of butterflies, each an addition and half a product mod p.
// What bounds them: those round trips, which the other groups of the block cover in part; of 2^18 x 64 the issue
// slots are 51 to 58 % busy, the multiplier and the ALU 45 to 55 %, the tensor pipe 7 to 8 %.
//
// BabyBear passes stay in ntt_tile.cuh: their butterflies are a tenth as long, and the products'
// round trips (about 1,000 cycles for 16 outputs a thread) cost more than they save: 10-bit passes of
// 2^20 x 64 606 us against 479, 8- and 7-bit passes of 2^22 x 256 22.4 ms against 12.9.
//
// A block is persistent, one per SM, of up to five groups of 128 threads (96 TMEM columns each).  A group takes
// tiles of 2^K rows x C columns: one tensor copy (TMA) brings a tile into shared memory while the pass twists
// are staged, both phases exchange in place, and the next tile's copy starts as soon as phase B has read
// its operands, so that it runs under phase B's arithmetic and the other groups' work.
#include <algorithm>

#include "common.cuh"
#include "engine.cuh"
#include "limbs.cuh"
#include "ntt_tc.cuh"
#include "tcgen05.cuh"

namespace zkb {

namespace ntt_tc {
using namespace tc;

constexpr int ROWS = 128, MAX_GROUPS = 5, COLS = 96, COL_A = 64;  // TMEM: D 64 columns, A up to 32

// ------------------------------------------------------------------ DFT matrices
using F = Goldilocks;
using T = uint64_t;
constexpr uint64_t ROOT = 0x185629dcda58878cull;  // 7^((p-1)/2^32)

constexpr uint64_t mulp(uint64_t a, uint64_t b) { return (uint64_t)((unsigned __int128)a * b % F::P); }
constexpr uint64_t powp(uint64_t a, uint64_t e) {
  uint64_t r = 1;
  for (; e; e >>= 1, a = mulp(a, a))
    if (e & 1) r = mulp(r, a);
  return r;
}

// The DFT of R points as products of 64 accumulator columns: [chunk of 64][32-byte K step][k / 16][n / 8][n %
// 8][k % 16].
template <int LR>
struct Dft {
  static constexpr int R = 1 << LR, L = 8;  // operand bytes of an input, accumulators of an output
  static constexpr int NCOL = R * L < 64 ? R * L : 64;  // columns of a chunk
  static constexpr int CHUNKS = R * L / NCOL, OUTS = NCOL / L, STEPS = R * L / 32;
  static constexpr int SLAB = NCOL * 32, BYTES = CHUNKS * STEPS * SLAB;
};
template <int LR>
struct alignas(16) Matrix {
  using D = Dft<LR>;
  uint8_t b[2][D::BYTES];  // forward, inverse
};
template <int LR>
constexpr Matrix<LR> make_matrix() {
  using D = Dft<LR>;
  Matrix<LR> m{};
  for (int inv = 0; inv < 2; inv++) {
    uint64_t w = powp(ROOT, 1ull << (F::TWO_ADICITY - LR));
    if (inv) w = powp(w, F::P - 2);
    uint64_t pw[D::R] = {1};
    for (int i = 1; i < D::R; i++) pw[i] = mulp(pw[i - 1], w);
    for (int f = 0; f < D::R; f++)
      for (int j = 0; j < D::R; j++) {
        uint64_t v = pw[j * f % D::R];
        for (int lp = 0; lp < D::L; lp++) {
          for (int l = 0; l < D::L; l++) {
            const int n = (f % D::OUTS) * D::L + limbs::goldilocks_col(l), k = j * D::L + lp;
            const int at = (f / D::OUTS) * D::STEPS * D::SLAB + ((k >> 4) * (D::NCOL >> 3) + (n >> 3)) * 128 + (n & 7) * 16 + (k & 15);
            m.b[inv][at] = (uint8_t)(v >> (8 * l));
          }
          v = mulp(v, 256);
        }
      }
  }
  return m;
}
// 128 operand bytes: every column sum is in the recombination's range.
static_assert(128 * 255 <= limbs::MAX_COLUMN, "accumulators exceed the recombination's range");

template <int LR>
__device__ const Matrix<LR> kMatrix = make_matrix<LR>();

// ------------------------------------------------------------------------ layout
template <int LA, int LB, int C>
struct Tile {
  static constexpr int RA = 1 << LA, RB = 1 << LB, K = LA + LB, ROWS_T = 1 << K;
  static constexpr int NA = RB * C / ROWS, NB = RA * C / ROWS;  // batches of 128 DFTs
  static_assert(NA * ROWS == RB * C && NB * ROWS == RA * C, "whole batches");
  static constexpr int BYTES = ROWS_T * C * (int)sizeof(T);
  static constexpr int MA = Dft<LA>::BYTES, MB = LA == LB ? 0 : Dft<LB>::BYTES;
  static constexpr int TW = ROWS_T * (int)sizeof(T);
  // shared memory: DFT matrices, phase-A twists, then per group its tile and pass twists, then control
  static constexpr int O_MB = MA, O_TWA = MA + MB, O_GROUP = (O_TWA + TW + 127) / 128 * 128;
  static constexpr int PER_GROUP = (BYTES + TW + 127) / 128 * 128;
  static constexpr int FIT = (225 * 1024 - O_GROUP) / PER_GROUP;
  static constexpr int GROUPS = FIT < MAX_GROUPS ? FIT : MAX_GROUPS;
  static constexpr int O_CTRL = O_GROUP + GROUPS * PER_GROUP;
  static constexpr int SMEM = O_CTRL + 16 + 16 * MAX_GROUPS;
};

// One thread: a tile by one tensor copy.
__device__ __forceinline__ void tile_copy(const T *tile, const CUtensorMap *map, int x, int low, int high, uint32_t mbar,
                                          int bytes) {
  expect_bytes(mbar, bytes);
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], "
      "[%7];" ::"r"((uint32_t)__cvta_generic_to_shared(tile)),
      "l"(map), "r"(x), "r"(low), "r"(0), "r"(0), "r"(high), "r"(mbar)
      : "memory");
}
// The group's tile has come.  `in_flight`: this thread has started its copy; when the wait gives up (or one
// before it has), that thread waits for the copy once more, so that none is under way when the block ends.
__device__ __forceinline__ void group_wait(Group &g, uint32_t mbar, uint32_t &phase, bool &in_flight) {
  if (wait_parity(mbar, phase, g.polls)) {
    phase ^= 1;
  } else {
    g.polls = 0;
    if (in_flight) wait_parity(mbar, phase, WAIT_POLLS);
  }
  in_flight = false;
}
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void group_sync(const Group &g) { asm volatile("bar.sync %0, 128;" ::"r"(g.bar) : "memory"); }

// One DFT per thread: get(j) its inputs, put(f, x) its outputs (some 64-bit representative); after_read() runs once every thread's inputs have been read.
template <int LR, class Get, class Put, class After>
__device__ __forceinline__ void dft(Group &g, int matrix, Get get, Put put, After after_read) {
  using D = Dft<LR>;
#pragma unroll
  for (int s = 0; s < D::R / 4; s++) {
    uint32_t v[8];
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const T x = get(s * 4 + e);
      v[2 * e] = (uint32_t)x;
      v[2 * e + 1] = (uint32_t)(x >> 32);
    }
    st8(g.tw + COL_A + 8 * s, v);
  }
#pragma unroll 1
  for (int q = 0; q < D::CHUNKS; q++) {
    arrive(g);
    if (q == 0) after_read();
    if (g.lead) {
#pragma unroll
      for (int s = 0; s < D::STEPS; s++)
        mma_slab(g, 0, COL_A + 8 * s, matrix + (q * D::STEPS + s) * D::SLAB, D::NCOL, s > 0);
    }
    finish(g);
#pragma unroll
    for (int h = 0; h < D::NCOL / 16; h++) {
      uint32_t a[16];
      ld16(a, g.tw + 16 * h);
      ld_wait(a);
#pragma unroll
      for (int e = 0; e < 2; e++) put(q * D::OUTS + 2 * h + e, limbs::goldilocks(a + 8 * e));
    }
  }
}

template <int LA, int LB, int C>
__global__ void __launch_bounds__(ROWS * Tile<LA, LB, C>::GROUPS, 1)
    pass_kernel(T *out, const PassGeom g, uint64_t tiles, const T *__restrict__ tw, int inverse, T post_scale,
                const __grid_constant__ CUtensorMap map, uint32_t *waits) {
  using S = Tile<LA, LB, C>;
  constexpr int K = S::K, RA = S::RA, RB = S::RB;
  extern __shared__ __align__(128) uint8_t sm[];
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm), ctrl = base + S::O_CTRL;
  const uint32_t loads = ctrl + 16 + 8 * MAX_GROUPS;  // mbarriers of the groups' tile copies
  const int hi = g.lo + K;

  if (threadIdx.x == 0) {
    init_barrier(ctrl + 8);
    for (int i = 0; i < S::GROUPS; i++) {
      init_barrier(ctrl + 16 + 8 * i);
      init_barrier(loads + 8 * i);
    }
    init_fence();
    expect_bytes(ctrl + 8, S::MA + S::MB);
    bulk_copy(base, kMatrix<LA>.b[inverse], S::MA, ctrl + 8);
    if constexpr (S::MB > 0) bulk_copy(base + S::O_MB, kMatrix<LB>.b[inverse], S::MB, ctrl + 8);
  }
  T *tw_a = reinterpret_cast<T *>(sm + S::O_TWA);  // [f1][i] = w_{2^K}^(i f1)
  for (int e = threadIdx.x; e < S::ROWS_T; e += blockDim.x) tw_a[e] = tw[(uint64_t)((e / RB) * (e % RB)) << (g.L - K)];
  if (threadIdx.x < 32) tmem_alloc(ctrl, 512);
  fence_before();
  __syncthreads();
  fence_after();
  tables_or_exit(ctrl + 8, sm + S::O_CTRL, 512, waits);
  Group gr = make_group(sm, S::O_CTRL, ctrl + 16, COLS, waits);

  const int gi = threadIdx.x / ROWS, tid = threadIdx.x % ROWS;
  uint8_t *mine = sm + S::O_GROUP + gi * S::PER_GROUP;
  T *tile = reinterpret_cast<T *>(mine);
  T *tw_b = reinterpret_cast<T *>(mine + S::BYTES);
  const uint32_t load = loads + 8 * gi;
  const uint64_t stride = (uint64_t)gridDim.x * S::GROUPS;
  bool in_flight = false;
  auto fetch = [&](uint64_t t) {  // one thread: the copy of tile t
    in_flight = true;
    const uint32_t chunk = (uint32_t)(t % g.chunks_per_row);
    const uint64_t rest = t / g.chunks_per_row;
    const uint32_t grp = (uint32_t)(rest % g.groups), blk = (uint32_t)(rest / g.groups);
    tile_copy(tile, &map, (int)(chunk * C), (int)(grp & ((1u << g.lo) - 1u)),
              (int)(blk * (g.groups >> g.lo) + (grp >> g.lo)), load, S::BYTES);
  };
  const uint64_t first = (uint64_t)gi * gridDim.x + blockIdx.x;
  if (tid == 0 && first < tiles) fetch(first);
  uint32_t phase = 0, staged = ~0u;
  for (uint64_t t = first; t < tiles; t += stride) {
    const uint32_t chunk = (uint32_t)(t % g.chunks_per_row);
    const uint64_t rest = t / g.chunks_per_row;
    const uint32_t grp = (uint32_t)(rest % g.groups), blk = (uint32_t)(rest / g.groups);
    const uint32_t i_low = grp & ((1u << g.lo) - 1u);
    const uint32_t base_row = ((grp >> g.lo) << hi) | i_low;
    if (g.twist && staged != i_low) {
      group_sync(gr);  // the last tile's uses of the table are over
      for (int e = tid; e < S::ROWS_T; e += ROWS) tw_b[e] = tw[((uint64_t)i_low * e) << (g.L - hi)];
      staged = i_low;  // visible after the barriers of phase A
    }
    group_wait(gr, load, phase, in_flight);
    // ---- phase A: over j of rows j * RB + i; outputs in place, i's low bits xored with f1's so that neither
    // phase's warps meet a bank twice (the xor stays inside the batch)
#pragma unroll 1
    for (int b = 0; b < S::NA; b++) {
      const int i = (b * ROWS + tid) / C, c = tid % C;
      dft<LA>(
          gr, 0, [&](int j) { return tile[(j * RB + i) * C + c]; },
          [&](int f, T x) { tile[(f * RB + (i ^ (f & 3))) * C + c] = F::mul_any(x, tw_a[f * RB + i]); },
          [] {});
    }
    proxy_fence();  // these writes come before the next copy's
    group_sync(gr);
    // ---- phase B: over i, the pass twist, out
#pragma unroll 1
    for (int b = 0; b < S::NB; b++) {
      const int f1 = (b * ROWS + tid) / C, c = tid % C;
      const bool ok = chunk * C + c < g.cols;
      T *p = out + (size_t)blk * g.block_stride + (size_t)chunk * C + c + (size_t)base_row * g.width +
             (((size_t)(__brev(f1) >> (32 - LA)) << LB) * g.width << g.lo);
      const size_t rs = (size_t)g.width << g.lo;
      dft<LB>(
          gr, LA == LB ? 0 : S::O_MB, [&](int i) { return tile[(f1 * RB + (i ^ (f1 & 3))) * C + c]; },
          [&](int f, T x) {
            if (g.twist)
              x = F::mul_any(x, tw_b[f1 + RA * f]);
            else if (post_scale)
              x = F::mul_any(x, post_scale);
            if (ok) p[(size_t)(__brev(f) >> (32 - LB)) * rs] = F::canon(x);
          },
          [&] {
            // every thread of the group has read its last inputs: the tile's memory is free
            if (b == S::NB - 1 && tid == 0 && t + stride < tiles && gr.polls) {
              proxy_fence();
              fetch(t + stride);
            }
          });
    }
  }
  drain(gr);
  st_wait();
  fence_before();
  __syncthreads();
  if (threadIdx.x < 32) {
    fence_after();
    tmem_free(*reinterpret_cast<volatile uint32_t *>(sm + S::O_CTRL), 512);
  }
}

// The fused LDE middle (lde_fused_tile of ntt_tile.cuh): the last inverse pass, every coset's twist and first
// forward pass.  A group keeps the block's coefficients in a second buffer of its shared memory; the
// coset factors are applied as phase A reads them.
template <int LA, int LB, int C>
struct FusedTile {
  using S = Tile<LA, LB, C>;
  static constexpr int M = S::MA + S::MB;  // matrices of one direction
  static constexpr int O_TW = 2 * M, O_GROUP = (O_TW + 2 * S::TW + 127) / 128 * 128;
  static constexpr int PER_GROUP = (2 * S::BYTES + 2 * S::TW + 127) / 128 * 128;
  static constexpr int FIT = (225 * 1024 - O_GROUP) / PER_GROUP;
  static constexpr int GROUPS = FIT < MAX_GROUPS ? FIT : MAX_GROUPS;
  static constexpr int O_CTRL = O_GROUP + GROUPS * PER_GROUP;
  static constexpr int SMEM = O_CTRL + 16 + 16 * MAX_GROUPS;
};

template <int LA, int LB, int C>
__global__ void __launch_bounds__(ROWS * FusedTile<LA, LB, C>::GROUPS, 1)
    fused_kernel(T *out, const FusedGeom g, uint64_t tiles, const T *__restrict__ itw, const T *__restrict__ ftw,
                 const T *__restrict__ ctab_t, const T *__restrict__ ftw_t, const __grid_constant__ CUtensorMap map, uint32_t *waits) {
  using S = Tile<LA, LB, C>;
  using U = FusedTile<LA, LB, C>;
  constexpr int K = S::K, RA = S::RA, RB = S::RB;
  extern __shared__ __align__(128) uint8_t sm[];
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm), ctrl = base + U::O_CTRL;
  const uint32_t loads = ctrl + 16 + 8 * MAX_GROUPS;
  const int lm = g.L - K;
  if (threadIdx.x == 0) {
    init_barrier(ctrl + 8);
    for (int i = 0; i < U::GROUPS; i++) {
      init_barrier(ctrl + 16 + 8 * i);
      init_barrier(loads + 8 * i);
    }
    init_fence();
    expect_bytes(ctrl + 8, 2 * U::M);
    for (int d = 0; d < 2; d++) {  // forward, inverse
      bulk_copy(base + d * U::M, kMatrix<LA>.b[d], S::MA, ctrl + 8);
      if constexpr (S::MB > 0) bulk_copy(base + d * U::M + S::O_MB, kMatrix<LB>.b[d], S::MB, ctrl + 8);
    }
  }
  T *tw_f = reinterpret_cast<T *>(sm + U::O_TW), *tw_i = tw_f + S::ROWS_T;  // [f1][i] = w_{2^K}^(+-i f1)
  for (int e = threadIdx.x; e < S::ROWS_T; e += blockDim.x) {
    const uint64_t at = (uint64_t)((e / RB) * (e % RB)) << lm;
    tw_f[e] = ftw[at];
    tw_i[e] = itw[at];
  }
  if (threadIdx.x < 32) tmem_alloc(ctrl, 512);
  fence_before();
  __syncthreads();
  fence_after();
  tables_or_exit(ctrl + 8, sm + U::O_CTRL, 512, waits);
  Group gr = make_group(sm, U::O_CTRL, ctrl + 16, COLS, waits);

  const int gi = threadIdx.x / ROWS, tid = threadIdx.x % ROWS;
  uint8_t *mine = sm + U::O_GROUP + gi * U::PER_GROUP;
  T *tile = reinterpret_cast<T *>(mine), *coef = reinterpret_cast<T *>(mine + S::BYTES);
  T *cf = reinterpret_cast<T *>(mine + 2 * S::BYTES), *tw_b = cf + S::ROWS_T;
  const uint32_t load = loads + 8 * gi;
  const uint64_t stride = (uint64_t)gridDim.x * U::GROUPS, first = (uint64_t)gi * gridDim.x + blockIdx.x;
  bool in_flight = false;
  auto fetch = [&](uint64_t t) {
    in_flight = true;
    tile_copy(tile, &map, (int)(t % g.chunks_per_row) * C, 0, (int)(t / g.chunks_per_row), load, S::BYTES);
  };
  if (tid == 0 && first < tiles) fetch(first);
  uint32_t phase = 0;
  for (uint64_t t = first; t < tiles; t += stride) {
    const uint32_t chunk = (uint32_t)(t % g.chunks_per_row), B = (uint32_t)(t / g.chunks_per_row);
    const uint32_t m_lo = lm ? (__brev(B) >> (32 - lm)) : 0u;
    auto factors = [&](int jc) {  // coset jc's
      for (int e = tid; e < S::ROWS_T; e += ROWS) cf[e] = ctab_t[(uint64_t)jc * g.n + ((size_t)m_lo << K) + e];
    };
    group_sync(gr);  // the last tile's uses of the tables are over
    for (int e = tid; e < S::ROWS_T; e += ROWS) tw_b[e] = ftw_t[((size_t)m_lo << K) + e];
    factors(0);
    group_wait(gr, load, phase, in_flight);
    // ---- inverse pass: phase A in place, phase B into the coefficients, index e = f1 + RA f2
#pragma unroll 1
    for (int b = 0; b < S::NA; b++) {
      const int i = (b * ROWS + tid) / C, c = tid % C;
      dft<LA>(
          gr, U::M, [&](int j) { return tile[(j * RB + i) * C + c]; },
          [&](int f, T x) { tile[(f * RB + (i ^ (f & 3))) * C + c] = F::mul_any(x, tw_i[f * RB + i]); }, [] {});
    }
    group_sync(gr);
#pragma unroll 1
    for (int b = 0; b < S::NB; b++) {
      const int f1 = (b * ROWS + tid) / C, c = tid % C;
      dft<LB>(
          gr, U::M + (LA == LB ? 0 : S::O_MB), [&](int i) { return tile[(f1 * RB + (i ^ (f1 & 3))) * C + c]; },
          [&](int f, T x) { coef[(f1 + RA * f) * C + c] = x; }, [] {});
    }
    // ---- per coset
#pragma unroll 1
    for (int jc = 0; jc < (1 << g.log_b); jc++) {
      group_sync(gr);  // the coefficients are there (or the last coset is done with the tile)
#pragma unroll 1
      for (int b = 0; b < S::NA; b++) {
        const int i = (b * ROWS + tid) / C, c = tid % C;
        dft<LA>(
            gr, 0, [&](int j) { return F::mul_any(coef[(j * RB + i) * C + c], cf[j * RB + i]); },
            [&](int f, T x) { tile[(f * RB + (i ^ (f & 3))) * C + c] = F::mul_any(x, tw_f[f * RB + i]); }, [] {});
      }
      const bool last = jc + 1 == (1 << g.log_b);
      if (last) proxy_fence();  // these writes come before the next copy's
      group_sync(gr);
      if (!last) factors(jc + 1);
      const uint32_t r = g.log_b ? (__brev((uint32_t)jc) >> (32 - g.log_b)) : 0u;
#pragma unroll 1
      for (int b = 0; b < S::NB; b++) {
        const int f1 = (b * ROWS + tid) / C, c = tid % C;
        const bool ok = chunk * C + c < g.cols;
        const size_t rs = (size_t)g.width << lm;
        T *p = out + (uint64_t)r * g.n * g.width + (size_t)chunk * C + c + (size_t)m_lo * g.width +
               ((size_t)(__brev(f1) >> (32 - LA)) << LB) * rs;
        dft<LB>(
            gr, LA == LB ? 0 : S::O_MB, [&](int i) { return tile[(f1 * RB + (i ^ (f1 & 3))) * C + c]; },
            [&](int f, T x) {
              if (lm > 0) x = F::mul_any(x, tw_b[f1 + RA * f]);
              if (ok) p[(size_t)(__brev(f) >> (32 - LB)) * rs] = F::canon(x);
            },
            [&] {
              if (last && b == S::NB - 1 && tid == 0 && t + stride < tiles && gr.polls) {
                proxy_fence();
                fetch(t + stride);
              }
            });
      }
    }
  }
  drain(gr);
  st_wait();
  fence_before();
  __syncthreads();
  if (threadIdx.x < 32) {
    fence_after();
    tmem_free(*reinterpret_cast<volatile uint32_t *>(sm + U::O_CTRL), 512);
  }
}

template <int LA, int LB, int C>
static int launch(T *out, const PassGeom &g, uint64_t tiles, const T *tw, bool inverse, T scale, const CUtensorMap &map,
                  cudaStream_t s) {
  using S = Tile<LA, LB, C>;
  DeviceContext *ctx;
  ZKB_TRY(current_context(&ctx));
  ZKB_CHECK_CUDA(cudaFuncSetAttribute(pass_kernel<LA, LB, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM));
  const unsigned grid = (unsigned)std::min<uint64_t>(ctx->sm_count, tiles);
  ZKB_LAUNCH("ntt_pass_tc", s, pass_kernel<LA, LB, C><<<grid, ROWS * S::GROUPS, S::SMEM, s>>>(out, g, tiles, tw, inverse ? 1 : 0, scale, map, ctx->wait_word));
  return ZKB_OK;
}

uint32_t chunk(int K) { return K == 6 || K == 7 ? 16 : K == 8 ? 8 : 0; }

int pass(int K, T *out, const PassGeom &g, uint64_t tiles, const T *tw, bool inverse, T scale, const CUtensorMap &map,
         cudaStream_t s) {
  switch (K) {
    case 6: return launch<3, 3, 16>(out, g, tiles, tw, inverse, scale, map, s);
    case 7: return launch<4, 3, 16>(out, g, tiles, tw, inverse, scale, map, s);
    case 8: return launch<4, 4, 8>(out, g, tiles, tw, inverse, scale, map, s);
    default: set_error("internal: NTT pass of %d bits", K); return ZKB_ERR_INTERNAL;
  }
}

template <int LA, int LB, int C>
static int launch_fused(T *out, const FusedGeom &g, uint64_t tiles, const T *itw, const T *ftw, const T *ctab_t,
                        const T *ftw_t, const CUtensorMap &map, cudaStream_t s) {
  using U = FusedTile<LA, LB, C>;
  DeviceContext *ctx;
  ZKB_TRY(current_context(&ctx));
  ZKB_CHECK_CUDA(cudaFuncSetAttribute(fused_kernel<LA, LB, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, U::SMEM));
  const unsigned grid = (unsigned)std::min<uint64_t>(ctx->sm_count, tiles);
  ZKB_LAUNCH("lde_fused_tc", s, fused_kernel<LA, LB, C><<<grid, ROWS * U::GROUPS, U::SMEM, s>>>(out, g, tiles, itw, ftw, ctab_t, ftw_t, map, ctx->wait_word));
  return ZKB_OK;
}

int fused(int K, T *out, const FusedGeom &g, uint64_t tiles, const T *itw, const T *ftw, const T *ctab_t, const T *ftw_t,
          const CUtensorMap &map, cudaStream_t s) {
  switch (K) {
    case 6: return launch_fused<3, 3, 16>(out, g, tiles, itw, ftw, ctab_t, ftw_t, map, s);
    case 7: return launch_fused<4, 3, 16>(out, g, tiles, itw, ftw, ctab_t, ftw_t, map, s);
    case 8: return launch_fused<4, 4, 8>(out, g, tiles, itw, ftw, ctab_t, ftw_t, map, s);
    default: set_error("internal: fused LDE pass of %d bits", K); return ZKB_ERR_INTERNAL;
  }
}

}  // namespace ntt_tc
}  // namespace zkb
