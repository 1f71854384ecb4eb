// p2_tensor.cu — the hashing kernels on the tensor-core form of the BabyBear permutation
// (p2_tensor.cuh): leaf sponges, compressions, the FRI fold with its leaf hash, the batch
// permutation.
//
// All of them are a loop over tiles of 128 rows, one row per thread, a group of four warps per
// tile and up to five groups per block (the TMEM of an SM holds five).  The tile's rows run the same
// number of permutations, so a tile never spans two matrices of different width.
//
// What bounds them: the integer multiplier.  The 564 products of a permutation's S-boxes occupy
// it for 5640 cycles per warp (a wide product 4, a low one 2, a high one 4), everything else for
// 1270.  On a B200 at 1965 MHz a leaf hash of 2^23 x 256 with the alpha-reduction runs 4.30e9
// permutations/s (62.5 ms; 78.2 with the layers as modular additions, p2_permute); of 2^20 x 64 the multiplier
// is 79 % busy, the ALU 31 %, the tensor pipe 11 %.
#include <algorithm>

#include "common.cuh"
#include "engine.cuh"
#include "multitree.cuh"
#include "p2_launch.cuh"
#include "p2_tensor.cuh"

namespace zkb {

namespace p2t {

constexpr int THREADS = GROUP * MAX_GROUPS;
// Shared memory of the many-tree kernels: the tables, then the jobs' starts.
__host__ __device__ constexpr int mt_smem(Mode m, int jobs) {
  return (smem_bytes(m) + 15) / 16 * 16 + jobs * (int)sizeof(uint64_t);
}

// Eight words of a row from column c on (zero past the end).
__device__ __forceinline__ void load8(uint32_t (&x)[8], const uint32_t *rp, uint64_t c, uint64_t width, bool vec) {
  if (vec) {
    const uint4 a = *reinterpret_cast<const uint4 *>(rp + c);
    x[0] = a.x, x[1] = a.y, x[2] = a.z, x[3] = a.w;
    if (c + 4 < width) {
      const uint4 b = *reinterpret_cast<const uint4 *>(rp + c + 4);
      x[4] = b.x, x[5] = b.y, x[6] = b.z, x[7] = b.w;
    } else {
      x[4] = x[5] = x[6] = x[7] = 0;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; i++) x[i] = c + i < width ? rp[c + i] : 0;
  }
}

__device__ __forceinline__ void store8(uint32_t *out, const uint32_t (&o)[8]) {
  uint4 *d = reinterpret_cast<uint4 *>(out);
  d[0] = make_uint4(o[0], o[1], o[2], o[3]);
  d[1] = make_uint4(o[4], o[5], o[6], o[7]);
}

// acc += alpha-reduction of the chunk's columns (apow: one uint4 per column), times 2^32: four products to
// a reduction (4 p^2 < 2^64; hi(t) - hi(m p) lies in (-p, 1.9 p)), the reduced sums in 64 bits.
__device__ __forceinline__ void combine8(int64_t (&acc)[4], const uint32_t (&x)[8], const uint4 *__restrict__ apow,
                                         uint64_t c, uint64_t width) {
  using B = BabyBear;
#pragma unroll
  for (int i = 0; i < 8; i += 4) {
    if (c + i >= width) break;
    uint64_t t[4] = {0, 0, 0, 0};
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint4 w = c + i + k < width ? apow[c + i + k] : make_uint4(0, 0, 0, 0);
      t[0] += (uint64_t)x[i + k] * w.x;
      t[1] += (uint64_t)x[i + k] * w.y;
      t[2] += (uint64_t)x[i + k] * w.z;
      t[3] += (uint64_t)x[i + k] * w.w;
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint32_t m = (uint32_t)t[k] * B::PINV;
      acc[k] += (int64_t)(t[k] >> 32) - (int64_t)__umulhi(m, B::P);
    }
  }
}
// The four sums; the multiple of p keeps a negative one positive (up to 2^32 columns' groups).
__device__ __forceinline__ uint4 combined(const int64_t (&acc)[4]) {
  constexpr int64_t BIAS = (int64_t)BabyBear::P << 31;
  uint32_t r[4];
#pragma unroll
  for (int k = 0; k < 4; k++) r[k] = BabyBear::mont_reduce((uint64_t)(acc[k] + BIAS));
  return make_uint4(r[0], r[1], r[2], r[3]);
}

// Brings a line of a later tile into L2 while this one computes.
__device__ __forceinline__ void prefetch(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// The tiles of 128 rows of a group: spread over the blocks first, so that the SMs' numbers of
// tiles differ by one at most.
#define P2T_TILES(t, tiles)                                                                       \
  for (uint64_t t = (uint64_t)(threadIdx.x / GROUP) * gridDim.x + blockIdx.x; t < (tiles);        \
       t += (uint64_t)gridDim.x * (blockDim.x / GROUP))

// Leaf sponge over the concatenated rows of the matrices in ml; with COMBINE (one matrix) the
// rows' alpha-reductions too.  The next chunk's words are loaded while the permutation runs.
template <bool COMBINE>
__global__ void __launch_bounds__(THREADS)
    leaf_kernel(const MatList ml, uint64_t height, uint32_t *__restrict__ digests,
                const __grid_constant__ P2Params<BabyBear, 16> p, uint32_t *waits, const uint4 *__restrict__ apow,
                uint4 *__restrict__ comb, bool vec) {
  extern __shared__ __align__(128) uint8_t sm[];
  const uint64_t width = ml.col_start[ml.n];
  const int rem = (int)((width - 1) % 8) + 1;
  Group g = setup(sm, p, SPONGE, rem, waits);
  const uint64_t tiles = (height + GROUP - 1) / GROUP;
  P2T_TILES(t, tiles) {
    uint64_t row = t * GROUP + threadIdx.x % GROUP;
    const bool live = row < height;
    if (!live) row = height - 1;
    const uint32_t *rp = (const uint32_t *)ml.ptr[0] + row * ml.width[0];
    auto load = [&](uint32_t(&x)[8], uint64_t c) {
      if (COMBINE || ml.n == 1) {
        load8(x, rp, c, width, vec);
      } else {
#pragma unroll
        for (int i = 0; i < 8; i++) x[i] = c + i < width ? fetch_col<BabyBear>(ml, row, c + i) : 0;
      }
    };
    int64_t acc[4] = {0, 0, 0, 0};
    uint32_t x[8];
    load(x, 0);
#pragma unroll 1
    for (uint64_t c = 0; c < width; c += 8) {
      absorb(g, x, c == 0, c + 8 > width ? S_LAST : S_IN);
      if constexpr (COMBINE) combine8(acc, x, apow, c, width);
      if (c + 8 < width) load(x, c + 8);
      rounds(g);
    }
    uint32_t o[8];
    leave<8>(g, o);
    if (live) {
      store8(digests + row * 8, o);
      if constexpr (COMBINE)
        comb[row] = combined(acc);
    }
  }
  teardown(g, sm, SPONGE);
}

// The same over columns [c0, c0 + ncols) of wider rows: the last S-box outputs carried in `carry`
// (16 words per row) between slabs, digests on the last slab; the reduction written on the
// first slab, added on the others.
template <bool COMBINE>
__global__ void __launch_bounds__(THREADS)
    slab_kernel(const uint32_t *__restrict__ mat, uint64_t stride, uint64_t c0, uint64_t ncols, uint64_t height,
                uint32_t *__restrict__ carry, int first, int last, uint32_t *__restrict__ digests,
                const __grid_constant__ P2Params<BabyBear, 16> p, uint32_t *waits, const uint4 *__restrict__ apow,
                uint4 *__restrict__ comb, bool vec) {
  extern __shared__ __align__(128) uint8_t sm[];
  const int rem = (int)((ncols - 1) % 8) + 1;
  Group g = setup(sm, p, SPONGE, rem, waits);
  const uint64_t tiles = (height + GROUP - 1) / GROUP;
  P2T_TILES(t, tiles) {
    uint64_t row = t * GROUP + threadIdx.x % GROUP;
    const bool live = row < height;
    if (!live) row = height - 1;
    const uint32_t *rp = mat + row * stride + c0;
    uint4 *cp = reinterpret_cast<uint4 *>(carry + row * 16);
    if (!first) {
      uint32_t z[16];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const uint4 v = cp[q];
        z[4 * q] = v.x, z[4 * q + 1] = v.y, z[4 * q + 2] = v.z, z[4 * q + 3] = v.w;
      }
      st8(g.tw + COL_Z, z);
      st8(g.tw + COL_Z + 8, z + 8);
    }
    int64_t acc[4] = {0, 0, 0, 0};
    uint32_t x[8];
    load8(x, rp, 0, ncols, vec);
#pragma unroll 1
    for (uint64_t c = 0; c < ncols; c += 8) {
      absorb(g, x, first && c == 0, c + 8 > ncols ? S_LAST : S_IN);
      if constexpr (COMBINE) combine8(acc, x, apow + c0, c, ncols);
      if (c + 8 < ncols) load8(x, rp, c + 8, ncols, vec);
      rounds(g);
    }
    if (last) {
      uint32_t o[8];
      leave<8>(g, o);
      if (live) store8(digests + row * 8, o);
    } else {
      uint32_t z[16];
      load_z(g, z);
      if (live) {
#pragma unroll
        for (int q = 0; q < 4; q++) cp[q] = make_uint4(z[4 * q], z[4 * q + 1], z[4 * q + 2], z[4 * q + 3]);
      }
    }
    if constexpr (COMBINE) {
      if (live) {
        using B = BabyBear;
        uint4 r = combined(acc);
        if (!first) {
          const uint4 o = comb[row];
          r = make_uint4(B::add(o.x, r.x), B::add(o.y, r.y), B::add(o.z, r.z), B::add(o.w, r.w));
        }
        comb[row] = r;
      }
    }
  }
  teardown(g, sm, SPONGE);
}

__device__ __forceinline__ void load16(uint32_t (&x)[16], const uint32_t *from) {
  const uint4 *f = reinterpret_cast<const uint4 *>(from);
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const uint4 v = f[q];
    x[4 * q] = v.x, x[4 * q + 1] = v.y, x[4 * q + 2] = v.z, x[4 * q + 3] = v.w;
  }
}

// next[i] = compress(prev[2i], prev[2i+1]); with inj, compress(that, i < inj_h ? inj[i] : 0).
__global__ void __launch_bounds__(THREADS)
    compress_kernel(const uint32_t *__restrict__ prev, uint32_t *__restrict__ next, uint64_t n_out,
                    const uint32_t *__restrict__ inj, uint64_t inj_h, const __grid_constant__ P2Params<BabyBear, 16> p, uint32_t *waits) {
  extern __shared__ __align__(128) uint8_t sm[];
  Group g = setup(sm, p, STATE16, 8, waits);
  const uint64_t tiles = (n_out + GROUP - 1) / GROUP;
  P2T_TILES(t, tiles) {
    uint64_t i = t * GROUP + threadIdx.x % GROUP;
    const bool live = i < n_out;
    if (!live) i = n_out - 1;
    uint32_t x[16], o[8];
    load16(x, prev + i * 16);
#pragma unroll 1
    for (int r = 0;; r++) {
      enter16(g, x);
      rounds(g);
      leave<8>(g, o);
      if (!inj || r == 1) break;
#pragma unroll
      for (int k = 0; k < 8; k++) {
        x[k] = o[k];
        x[8 + k] = i < inj_h ? inj[i * 8 + k] : 0;
      }
    }
    if (live) store8(next + i * 8, o);
  }
  teardown(g, sm, STATE16);
}

// Leaf sponges of many matrices: tile t belongs to the last job whose first tile is <= t.
__global__ void __launch_bounds__(THREADS)
    mt_leaf_kernel(const mt::LeafJob *__restrict__ jobs, int n_jobs, uint64_t tiles,
                   const __grid_constant__ P2Params<BabyBear, 16> p, uint32_t *waits) {
  extern __shared__ __align__(128) uint8_t sm[];
  uint64_t *starts = reinterpret_cast<uint64_t *>(sm + mt_smem(SPONGE_ANY, 0));
  for (int i = threadIdx.x; i < n_jobs; i += blockDim.x) starts[i] = jobs[i].tile_start;
  Group g = setup(sm, p, SPONGE_ANY, 8, waits);
  P2T_TILES(t, tiles) {
    const int j = mt::find_job(starts, n_jobs, t);
    const uint64_t rows = jobs[j].rows, width = jobs[j].width;
    const int rem = (int)(width % 8);
    uint64_t row = (t - starts[j]) * GROUP + threadIdx.x % GROUP;
    const bool live = row < rows;
    if (!live) row = rows - 1;
    const uint32_t *rp = (const uint32_t *)jobs[j].data + row * width;
    const bool vec = width % 4 == 0 && ((uintptr_t)jobs[j].data & 15) == 0;
    uint32_t x[8];
    load8(x, rp, 0, width, vec);
#pragma unroll 1
    for (uint64_t c = 0; c < width; c += 8) {
      absorb(g, x, c == 0, c + 8 > width ? S_LAST + (rem - 1) * ABS_BYTES : S_IN);
      if (c + 8 < width) load8(x, rp, c + 8, width, vec);
      rounds(g);
    }
    uint32_t o[8];
    leave<8>(g, o);
    if (live) store8((uint32_t *)jobs[j].digests + row * 8, o);
  }
  teardown(g, sm, SPONGE_ANY);
}

// One level of many trees: each thread finds its own job.
__global__ void __launch_bounds__(THREADS)
    mt_compress_kernel(const mt::CompJob *__restrict__ jobs, int n_jobs, uint64_t total,
                       const __grid_constant__ P2Params<BabyBear, 16> p, uint32_t *waits) {
  extern __shared__ __align__(128) uint8_t sm[];
  uint64_t *starts = reinterpret_cast<uint64_t *>(sm + mt_smem(STATE16, 0));
  for (int i = threadIdx.x; i < n_jobs; i += blockDim.x) starts[i] = jobs[i].start;
  Group g = setup(sm, p, STATE16, 8, waits);
  const uint64_t tiles = (total + GROUP - 1) / GROUP;
  P2T_TILES(t, tiles) {
    uint64_t q = t * GROUP + threadIdx.x % GROUP;
    const bool live = q < total;
    if (!live) q = total - 1;
    const int j = mt::find_job(starts, n_jobs, q);
    const uint64_t i = q - starts[j];
    uint32_t x[16], o[8];
    load16(x, (const uint32_t *)jobs[j].prev + i * 16);
    enter16(g, x);
    rounds(g);
    leave<8>(g, o);
    if (live) store8((uint32_t *)jobs[j].next + i * 8, o);
  }
  teardown(g, sm, STATE16);
}

// fri.cu's fold with the leaf hash of the layer it makes.
template <bool FOLD>
__global__ void __launch_bounds__(THREADS)
    fri_kernel(const uint32_t *__restrict__ e, uint32_t *__restrict__ out, uint64_t n_leaves, int log_out,
               const Ext4Params prm, const uint32_t *__restrict__ itw, uint32_t *__restrict__ digests,
               const __grid_constant__ P2Params<BabyBear, 16> p, uint32_t *waits) {
  extern __shared__ __align__(128) uint8_t sm[];
  Group g = setup(sm, p, SPONGE, 8, waits);
  const uint64_t tiles = (n_leaves + GROUP - 1) / GROUP;
  P2T_TILES(t, tiles) {
    uint64_t j = t * GROUP + threadIdx.x % GROUP;
    const bool live = j < n_leaves;
    if (!live) j = n_leaves - 1;
    const uint4 *in = reinterpret_cast<const uint4 *>(e);
    const uint64_t later = j + (uint64_t)gridDim.x * (blockDim.x / GROUP) * GROUP;
    if (later < n_leaves) prefetch(in + (FOLD ? 4 : 2) * later);
    uint4 a, b;
    if constexpr (FOLD) {
      a = fold_ext4_one(in[4 * j], in[4 * j + 1], 2 * j, log_out, prm, itw);
      b = fold_ext4_one(in[4 * j + 2], in[4 * j + 3], 2 * j + 1, log_out, prm, itw);
      if (live) {
        reinterpret_cast<uint4 *>(out)[2 * j] = a;
        reinterpret_cast<uint4 *>(out)[2 * j + 1] = b;
      }
    } else {
      a = in[2 * j];
      b = in[2 * j + 1];
    }
    const uint32_t x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint32_t o[8];
    absorb(g, x, true, S_IN);
    rounds(g);
    leave<8>(g, o);
    if (live) store8(digests + j * 8, o);
  }
  teardown(g, sm, SPONGE);
}

__global__ void __launch_bounds__(THREADS)
    permute_kernel(uint32_t *__restrict__ states, uint64_t n, bool vec, const __grid_constant__ P2Params<BabyBear, 16> p, uint32_t *waits) {
  extern __shared__ __align__(128) uint8_t sm[];
  Group g = setup(sm, p, PERM16, 8, waits);
  const uint64_t tiles = (n + GROUP - 1) / GROUP;
  P2T_TILES(t, tiles) {
    uint64_t i = t * GROUP + threadIdx.x % GROUP;
    const bool live = i < n;
    if (!live) i = n - 1;
    uint32_t x[16];
    if (vec) {
      load16(x, states + i * 16);
    } else {
#pragma unroll
      for (int k = 0; k < 16; k++) x[k] = states[i * 16 + k];
    }
    enter16(g, x);
    rounds(g);
    leave<16>(g, x);
    if (live) {
#pragma unroll
      for (int k = 0; k < 16; k++) states[i * 16 + k] = x[k];
    }
  }
  teardown(g, sm, PERM16);
}

// Launch shape.  A block runs up to five tiles side by side; an SM's time for k of them is
// TILE_KCLK[k] thousand cycles per permutation (measured: a lone tile waits for its products and its
// own S-box chains, five fill the multiplier).  A block's unit of work is at least 32
// permutations a thread (0.7 ms with five groups), so that its tables (about 2 us) cost
// nothing and it still ends soon enough for other streams' kernels to get SMs in between.
// Below eight such units an SM, the last ones would leave SMs idle: the grid is one block an
// SM then, the tiles spread evenly, with the number of groups that takes the SM's share in
// the least time.
constexpr double TILE_KCLK[MAX_GROUPS + 1] = {0, 17.3, 22.8, 27.4, 33.7, 40.8};
struct Shape {
  unsigned grid, threads;
};
static Shape shape(uint64_t tiles, uint64_t perms, int sms) {
  const uint64_t per_sm = (tiles + sms - 1) / sms;
  const uint64_t unit = MAX_GROUPS * std::max<uint64_t>(1, 32 / std::max<uint64_t>(1, perms));  // tiles
  if (per_sm >= 8 * unit) return {(unsigned)((tiles + unit - 1) / unit), (unsigned)(MAX_GROUPS * GROUP)};
  int best = 1;
  double best_t = 1e30;
  for (int g = 1; g <= MAX_GROUPS; g++) {
    const double t = (double)(per_sm / g) * TILE_KCLK[g] + TILE_KCLK[per_sm % g];
    if (t < best_t) best_t = t, best = g;
  }
  return {(unsigned)std::min<uint64_t>(sms, tiles), (unsigned)(best * GROUP)};
}

// Smallest number of rows (or compressions) in one launch: more than one tile an SM.  Up to there
// the quad form is the faster one (16,384 rows x 32 columns: 46 us against 55; 18,944 x 64: 86
// against 91), from there this one (32,768 x 8: 21.5 us against 24.7, x 64: 109 against 135).
constexpr uint64_t MIN_ROWS = 148ull * GROUP + 1;

bool takes(const P2Params<BabyBear, 16> &p, uint64_t rows) { return rows >= MIN_ROWS && usable(p); }

int hash_rows(const MatList &ml, uint64_t height, uint32_t *digests, const P2Params<BabyBear, 16> &p,
              const uint4 *apow, uint4 *comb, const char *name, cudaStream_t s) {
  DeviceContext *ctx;
  ZKB_TRY(current_context(&ctx));
  const uint64_t width = ml.col_start[ml.n];
  const Shape sh = shape((height + GROUP - 1) / GROUP, (width + 7) / 8, ctx->sm_count);
  const size_t smem = smem_bytes(SPONGE);
  const bool vec = ml.n == 1 && width % 4 == 0 && ((uintptr_t)ml.ptr[0] & 15) == 0;
  if (comb) {
    ZKB_TRY(smem_limit<smem_bytes(SPONGE)>(leaf_kernel<true>));
    ZKB_LAUNCH(name, s, leaf_kernel<true><<<sh.grid, sh.threads, smem, s>>>(ml, height, digests, p, ctx->wait_word, apow, comb, vec));
  } else {
    ZKB_TRY(smem_limit<smem_bytes(SPONGE)>(leaf_kernel<false>));
    ZKB_LAUNCH(name, s, leaf_kernel<false><<<sh.grid, sh.threads, smem, s>>>(ml, height, digests, p, ctx->wait_word, apow, comb, vec));
  }
  return ZKB_OK;
}

int hash_slab(const uint32_t *mat, uint64_t stride, uint64_t c0, uint64_t ncols, uint64_t height, uint32_t *carry,
              bool first, bool last, uint32_t *digests, const P2Params<BabyBear, 16> &p, const uint4 *apow, uint4 *comb,
              const char *name, cudaStream_t s) {
  DeviceContext *ctx;
  ZKB_TRY(current_context(&ctx));
  const Shape sh = shape((height + GROUP - 1) / GROUP, (ncols + 7) / 8, ctx->sm_count);
  const size_t smem = smem_bytes(SPONGE);
  const bool vec = stride % 4 == 0 && c0 % 4 == 0 && ncols % 4 == 0 && ((uintptr_t)mat & 15) == 0;
  if (apow) {
    ZKB_TRY(smem_limit<smem_bytes(SPONGE)>(slab_kernel<true>));
    ZKB_LAUNCH(name, s, slab_kernel<true><<<sh.grid, sh.threads, smem, s>>>(mat, stride, c0, ncols, height, carry, first, last, digests, p, ctx->wait_word, apow, comb, vec));
  } else {
    ZKB_TRY(smem_limit<smem_bytes(SPONGE)>(slab_kernel<false>));
    ZKB_LAUNCH(name, s, slab_kernel<false><<<sh.grid, sh.threads, smem, s>>>(mat, stride, c0, ncols, height, carry, first, last, digests, p, ctx->wait_word, apow, comb, vec));
  }
  return ZKB_OK;
}

int compress(const uint32_t *prev, uint32_t *next, uint64_t n_out, const uint32_t *inj, uint64_t inj_h,
             const P2Params<BabyBear, 16> &p, const char *name, cudaStream_t s) {
  DeviceContext *ctx;
  ZKB_TRY(current_context(&ctx));
  const Shape sh = shape((n_out + GROUP - 1) / GROUP, 1, ctx->sm_count);
  const size_t smem = smem_bytes(STATE16);
  ZKB_TRY(smem_limit<smem_bytes(STATE16)>(compress_kernel));
  ZKB_LAUNCH(name, s, compress_kernel<<<sh.grid, sh.threads, smem, s>>>(prev, next, n_out, inj, inj_h, p, ctx->wait_word));
  return ZKB_OK;
}

int mt_leaf(const mt::LeafJob *d_jobs, int n, uint64_t tiles, uint64_t perms, const P2Params<BabyBear, 16> &p,
            const char *name, cudaStream_t s) {
  DeviceContext *ctx;
  ZKB_TRY(current_context(&ctx));
  const Shape sh = shape(tiles, perms, ctx->sm_count);
  ZKB_REQUIRE(n <= mt::MAX_JOBS, "internal: %d trees in one launch", n);
  const size_t smem = mt_smem(SPONGE_ANY, n);
  ZKB_TRY(smem_limit<mt_smem(SPONGE_ANY, mt::MAX_JOBS)>(mt_leaf_kernel));
  ZKB_LAUNCH(name, s, mt_leaf_kernel<<<sh.grid, sh.threads, smem, s>>>(d_jobs, n, tiles, p, ctx->wait_word));
  return ZKB_OK;
}

int mt_compress(const mt::CompJob *d_jobs, int n, uint64_t total, const P2Params<BabyBear, 16> &p, const char *name,
                cudaStream_t s) {
  DeviceContext *ctx;
  ZKB_TRY(current_context(&ctx));
  const Shape sh = shape((total + GROUP - 1) / GROUP, 1, ctx->sm_count);
  ZKB_REQUIRE(n <= mt::MAX_JOBS, "internal: %d trees in one launch", n);
  const size_t smem = mt_smem(STATE16, n);
  ZKB_TRY(smem_limit<mt_smem(STATE16, mt::MAX_JOBS)>(mt_compress_kernel));
  ZKB_LAUNCH(name, s, mt_compress_kernel<<<sh.grid, sh.threads, smem, s>>>(d_jobs, n, total, p, ctx->wait_word));
  return ZKB_OK;
}

int fri_fold_hash(const uint32_t *e, uint32_t *out, uint64_t n_leaves, int log_out, const Ext4Params *prm,
                  const uint32_t *itw, uint32_t *digests, const P2Params<BabyBear, 16> &p, const char *name,
                  cudaStream_t s) {
  DeviceContext *ctx;
  ZKB_TRY(current_context(&ctx));
  const Shape sh = shape((n_leaves + GROUP - 1) / GROUP, 1, ctx->sm_count);
  const size_t smem = smem_bytes(SPONGE);
  if (prm) {
    ZKB_TRY(smem_limit<smem_bytes(SPONGE)>(fri_kernel<true>));
    ZKB_LAUNCH(name, s, fri_kernel<true><<<sh.grid, sh.threads, smem, s>>>(e, out, n_leaves, log_out, *prm, itw, digests, p, ctx->wait_word));
  } else {
    ZKB_TRY(smem_limit<smem_bytes(SPONGE)>(fri_kernel<false>));
    ZKB_LAUNCH(name, s, fri_kernel<false><<<sh.grid, sh.threads, smem, s>>>(e, out, n_leaves, log_out, Ext4Params{}, itw, digests, p, ctx->wait_word));
  }
  return ZKB_OK;
}

int permute(uint32_t *states, uint64_t n, const P2Params<BabyBear, 16> &p, cudaStream_t s) {
  DeviceContext *ctx;
  ZKB_TRY(current_context(&ctx));
  const Shape sh = shape((n + GROUP - 1) / GROUP, 1, ctx->sm_count);
  const size_t smem = smem_bytes(PERM16);
  ZKB_TRY(smem_limit<smem_bytes(PERM16)>(permute_kernel));
  const bool vec = ((uintptr_t)states & 15) == 0;
  ZKB_LAUNCH("p2_permute", s, permute_kernel<<<sh.grid, sh.threads, smem, s>>>(states, n, vec, p, ctx->wait_word));
  return ZKB_OK;
}

}  // namespace p2t
}  // namespace zkb
