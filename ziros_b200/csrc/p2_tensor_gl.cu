// p2_tensor_gl.cu — the Goldilocks hashing kernels on the tensor-core form of the permutation
// (p2_tensor_gl.cuh): leaf sponges, compressions, the batch permutation.  Loops and tiles as in p2_tensor.cu;
// the TMEM of an SM holds three tiles of width 12 (168 columns each) and two of width 16 (208).
//
// What bounds them: the latency of the chains of 64-bit products (472 in a permutation's S-boxes at width 12, 600
// at 16), which three or two warps a scheduler cover in part: 2^18 x 64 rows keep the multiplier 62 and 53 %
// busy, the ALU 60 and 51 %, the issue slots 54 and 46 %.  On a B200 at 1965 MHz a 2^20 x 64 leaf hash takes
// 6.11 and 8.52 ms; with the layers as modular additions and the partial rounds' diagonal as products, one state
// per thread, it took 11.63 and 15.18 ms.
#include <algorithm>

#include "common.cuh"
#include "engine.cuh"
#include "multitree.cuh"
#include "p2_launch.cuh"
#include "p2_tensor_gl.cuh"

namespace zkb {

namespace p2g {

template <int W>
constexpr int out_words() {
  return W == 16 ? 8 : 4;
}

// Shared memory of the many-tree kernels: the tables, then the jobs' starts.
template <int W>
__host__ __device__ constexpr int mt_smem(int jobs) {
  return (Shape<W>::SMEM + 15) / 16 * 16 + jobs * (int)sizeof(uint64_t);
}

// Eight words of a row from column c on (zero past the end).
__device__ __forceinline__ void load8(uint64_t (&x)[8], const uint64_t *rp, uint64_t c, uint64_t width, bool vec) {
  if (vec && c + 8 <= width) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const ulonglong2 v = reinterpret_cast<const ulonglong2 *>(rp + c)[i];
      x[2 * i] = v.x, x[2 * i + 1] = v.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; i++) x[i] = c + i < width ? rp[c + i] : 0;
  }
}
__device__ __forceinline__ void load4(uint64_t (&x)[4], const uint64_t *from) {
  const ulonglong2 a = reinterpret_cast<const ulonglong2 *>(from)[0], b = reinterpret_cast<const ulonglong2 *>(from)[1];
  x[0] = a.x, x[1] = a.y, x[2] = b.x, x[3] = b.y;
}
__device__ __forceinline__ void store4(uint64_t *to, const uint64_t (&x)[4]) {
  reinterpret_cast<ulonglong2 *>(to)[0] = make_ulonglong2(x[0], x[1]);
  reinterpret_cast<ulonglong2 *>(to)[1] = make_ulonglong2(x[2], x[3]);
}

// The digest of the permutation that has just run.
template <int W>
__device__ __forceinline__ void digest(Group &g, uint64_t *to, bool live) {
  leave<W>(g);
#pragma unroll
  for (int c = 0; c < out_words<W>() / 4; c++) {
    uint64_t o[4];
    output<W>(g, c, o);
    if (live) store4(to + 4 * c, o);
  }
}

// A row's sponge; load(x, c) gives the eight words from column c on.
template <int W, class Load>
__device__ __forceinline__ void sponge(Group &g, uint64_t width, Load load) {
  uint64_t x[8];
  load(x, 0);
#pragma unroll 1
  for (uint64_t c = 0; c < width; c += 8) {
    if (c + 8 <= width) {
      absorb<W>(g, x, c == 0);
      if (c + 8 < width) load(x, c + 8);
    } else {
      // a partial chunk overwrites its own words of the state only
      const int rem = (int)(width - c);
      if (c) leave<W>(g);
#pragma unroll
      for (int q = 0; q < W / 4; q++) {
        uint64_t s[4] = {0, 0, 0, 0};
        if (c) output<W>(g, q, s);
#pragma unroll
        for (int i = 0; i < 4; i++)
          if (4 * q + i < 8 && 4 * q + i < rem) s[i] = x[(4 * q + i) & 7];
        store_words(g.tw + Shape<W>::COL_Z + 8 * q, s);
      }
      enter<W>(g);
    }
    rounds<W>(g);
  }
}

#define P2G_TILES(t, tiles)                                                                       \
  for (uint64_t t = (uint64_t)(threadIdx.x / GROUP) * gridDim.x + blockIdx.x; t < (tiles);        \
       t += (uint64_t)gridDim.x * (blockDim.x / GROUP))

template <int W>
__global__ void __launch_bounds__(GROUP * Shape<W>::MAX_GROUPS, 1)
    leaf_kernel(const MatList ml, uint64_t height, uint64_t *__restrict__ digests,
                const __grid_constant__ P2Params<Goldilocks, W> p, uint32_t *waits, bool vec) {
  extern __shared__ __align__(128) uint8_t sm[];
  Group g = setup<W>(sm, p, true, waits);
  const uint64_t width = ml.col_start[ml.n], tiles = (height + GROUP - 1) / GROUP;
  P2G_TILES(t, tiles) {
    uint64_t row = t * GROUP + threadIdx.x % GROUP;
    const bool live = row < height;
    if (!live) row = height - 1;
    const uint64_t *rp = (const uint64_t *)ml.ptr[0] + row * ml.width[0];
    sponge<W>(g, width, [&](uint64_t(&x)[8], uint64_t c) {
      if (ml.n == 1) {
        load8(x, rp, c, width, vec);
      } else {
#pragma unroll
        for (int i = 0; i < 8; i++) x[i] = c + i < width ? fetch_col<Goldilocks>(ml, row, c + i) : 0;
      }
    });
    digest<W>(g, digests + row * out_words<W>(), live);
  }
  teardown<W>(g, sm);
}

template <int W>
__global__ void __launch_bounds__(GROUP * Shape<W>::MAX_GROUPS, 1)
    mt_leaf_kernel(const mt::LeafJob *__restrict__ jobs, int n_jobs, uint64_t tiles,
                   const __grid_constant__ P2Params<Goldilocks, W> p, uint32_t *waits) {
  extern __shared__ __align__(128) uint8_t sm[];
  uint64_t *starts = reinterpret_cast<uint64_t *>(sm + mt_smem<W>(0));
  for (int i = threadIdx.x; i < n_jobs; i += blockDim.x) starts[i] = jobs[i].tile_start;
  Group g = setup<W>(sm, p, true, waits);
  P2G_TILES(t, tiles) {
    const int j = mt::find_job(starts, n_jobs, t);
    const uint64_t rows = jobs[j].rows, width = jobs[j].width;
    uint64_t row = (t - starts[j]) * GROUP + threadIdx.x % GROUP;
    const bool live = row < rows;
    if (!live) row = rows - 1;
    const uint64_t *rp = (const uint64_t *)jobs[j].data + row * width;
    const bool vec = width % 2 == 0 && ((uintptr_t)jobs[j].data & 15) == 0;
    sponge<W>(g, width, [&](uint64_t(&x)[8], uint64_t c) { load8(x, rp, c, width, vec); });
    digest<W>(g, (uint64_t *)jobs[j].digests + row * out_words<W>(), live);
  }
  teardown<W>(g, sm);
}

// Two digests into the state.
template <int W>
__device__ __forceinline__ void enter_pair(Group &g, const uint64_t *pair) {
#pragma unroll
  for (int q = 0; q < W / 4; q++) {
    uint64_t s[4] = {0, 0, 0, 0};
    if (4 * q < 2 * out_words<W>()) load4(s, pair + 4 * q);
    store_words(g.tw + Shape<W>::COL_Z + 8 * q, s);
  }
  enter<W>(g);
}

template <int W>
__global__ void __launch_bounds__(GROUP * Shape<W>::MAX_GROUPS, 1)
    compress_kernel(const uint64_t *__restrict__ prev, uint64_t *__restrict__ next, uint64_t n_out,
                    const uint64_t *__restrict__ inj, uint64_t inj_h, const __grid_constant__ P2Params<Goldilocks, W> p, uint32_t *waits) {
  extern __shared__ __align__(128) uint8_t sm[];
  constexpr int OUT = out_words<W>();
  Group g = setup<W>(sm, p, false, waits);
  const uint64_t tiles = (n_out + GROUP - 1) / GROUP;
  P2G_TILES(t, tiles) {
    uint64_t i = t * GROUP + threadIdx.x % GROUP;
    const bool live = i < n_out;
    if (!live) i = n_out - 1;
    enter_pair<W>(g, prev + i * 2 * OUT);
#pragma unroll 1
    for (int r = inj ? 0 : 1; r < 2; r++) {
      rounds<W>(g);
      if (r == 1) break;
      // compress(that, injected digest)
      leave<W>(g);
#pragma unroll
      for (int q = 0; q < W / 4; q++) {
        uint64_t s[4] = {0, 0, 0, 0};
        if (4 * q < OUT)
          output<W>(g, q, s);
        else if (4 * q < 2 * OUT && i < inj_h)
          load4(s, inj + i * OUT + 4 * q - OUT);
        store_words(g.tw + Shape<W>::COL_Z + 8 * q, s);
      }
      enter<W>(g);
    }
    digest<W>(g, next + i * OUT, live);
  }
  teardown<W>(g, sm);
}

template <int W>
__global__ void __launch_bounds__(GROUP * Shape<W>::MAX_GROUPS, 1)
    mt_compress_kernel(const mt::CompJob *__restrict__ jobs, int n_jobs, uint64_t total,
                       const __grid_constant__ P2Params<Goldilocks, W> p, uint32_t *waits) {
  extern __shared__ __align__(128) uint8_t sm[];
  constexpr int OUT = out_words<W>();
  uint64_t *starts = reinterpret_cast<uint64_t *>(sm + mt_smem<W>(0));
  for (int i = threadIdx.x; i < n_jobs; i += blockDim.x) starts[i] = jobs[i].start;
  Group g = setup<W>(sm, p, false, waits);
  const uint64_t tiles = (total + GROUP - 1) / GROUP;
  P2G_TILES(t, tiles) {
    uint64_t q = t * GROUP + threadIdx.x % GROUP;
    const bool live = q < total;
    if (!live) q = total - 1;
    const int j = mt::find_job(starts, n_jobs, q);
    const uint64_t i = q - starts[j];
    enter_pair<W>(g, (const uint64_t *)jobs[j].prev + i * 2 * OUT);
    rounds<W>(g);
    digest<W>(g, (uint64_t *)jobs[j].next + i * OUT, live);
  }
  teardown<W>(g, sm);
}

template <int W>
__global__ void __launch_bounds__(GROUP * Shape<W>::MAX_GROUPS, 1)
    permute_kernel(uint64_t *__restrict__ states, uint64_t n, const __grid_constant__ P2Params<Goldilocks, W> p, uint32_t *waits) {
  extern __shared__ __align__(128) uint8_t sm[];
  Group g = setup<W>(sm, p, false, waits);
  const uint64_t tiles = (n + GROUP - 1) / GROUP;
  P2G_TILES(t, tiles) {
    uint64_t i = t * GROUP + threadIdx.x % GROUP;
    const bool live = i < n;
    if (!live) i = n - 1;
    uint64_t *st = states + i * W;
#pragma unroll
    for (int q = 0; q < W / 4; q++) {
      const uint64_t s[4] = {st[4 * q], st[4 * q + 1], st[4 * q + 2], st[4 * q + 3]};
      store_words(g.tw + Shape<W>::COL_Z + 8 * q, s);
    }
    enter<W>(g);
    rounds<W>(g);
    leave<W>(g);
#pragma unroll
    for (int q = 0; q < W / 4; q++) {
      uint64_t o[4];
      output<W>(g, q, o);
      if (live) {
#pragma unroll
        for (int k = 0; k < 4; k++) st[4 * q + k] = o[k];
      }
    }
  }
  teardown<W>(g, sm);
}

// Launch shape, as in p2_tensor.cu: thousands of cycles per permutation for k tiles side by side on
// an SM; a unit of work is at least 16 permutations a thread.
template <int W>
constexpr double tile_kclk(int k) {
  return W == 12 ? (k == 0 ? 0 : k == 1 ? 43.3 : k == 2 ? 61.7 : 81.5) : (k == 0 ? 0 : k == 1 ? 52.0 : 77.6);
}
struct Launch {
  unsigned grid, threads;
};
template <int W>
static Launch shape(uint64_t tiles, uint64_t perms, int sms) {
  constexpr int G = Shape<W>::MAX_GROUPS;
  const uint64_t per_sm = (tiles + sms - 1) / sms;
  const uint64_t unit = G * std::max<uint64_t>(1, 16 / std::max<uint64_t>(1, perms));
  if (per_sm >= 8 * unit) return {(unsigned)((tiles + unit - 1) / unit), (unsigned)(G * GROUP)};
  int best = 1;
  double best_t = 1e30;
  for (int g = 1; g <= G; g++) {
    const double t = (double)(per_sm / g) * tile_kclk<W>(g) + tile_kclk<W>((int)(per_sm % g));
    if (t < best_t) best_t = t, best = g;
  }
  return {(unsigned)std::min<uint64_t>(sms, tiles), (unsigned)(best * GROUP)};
}

// Smallest number of rows (or compressions) in one launch; against quads of threads (p2_quad.cuh),
// width 12 and 16: 4,096 rows x 32 columns 94 us and 113 against 84 and 81, 8,192 100 and 114 against
// 126 and 120, 16,384 98 and 116 against 224 and 216.
constexpr uint64_t MIN_ROWS = 8192;

template <int W>
bool takes(const P2Params<Goldilocks, W> &p, uint64_t rows) {
  return rows >= MIN_ROWS && usable(p);
}

template <int W>
int hash_rows(const MatList &ml, uint64_t height, uint64_t *digests, const P2Params<Goldilocks, W> &p, const char *name,
              cudaStream_t s) {
  DeviceContext *ctx;
  ZKB_TRY(current_context(&ctx));
  const Launch sh = shape<W>((height + GROUP - 1) / GROUP, (ml.col_start[ml.n] + 7) / 8, ctx->sm_count);
  const size_t smem = Shape<W>::SMEM;
  const bool vec = ml.n == 1 && ml.width[0] % 2 == 0 && ((uintptr_t)ml.ptr[0] & 15) == 0;
  ZKB_TRY(smem_limit<Shape<W>::SMEM>(leaf_kernel<W>));
  ZKB_LAUNCH(name, s, leaf_kernel<W><<<sh.grid, sh.threads, smem, s>>>(ml, height, digests, p, ctx->wait_word, vec));
  return ZKB_OK;
}

template <int W>
int compress(const uint64_t *prev, uint64_t *next, uint64_t n_out, const uint64_t *inj, uint64_t inj_h,
             const P2Params<Goldilocks, W> &p, const char *name, cudaStream_t s) {
  DeviceContext *ctx;
  ZKB_TRY(current_context(&ctx));
  const Launch sh = shape<W>((n_out + GROUP - 1) / GROUP, 1, ctx->sm_count);
  const size_t smem = Shape<W>::SMEM;
  ZKB_TRY(smem_limit<Shape<W>::SMEM>(compress_kernel<W>));
  ZKB_LAUNCH(name, s, compress_kernel<W><<<sh.grid, sh.threads, smem, s>>>(prev, next, n_out, inj, inj_h, p, ctx->wait_word));
  return ZKB_OK;
}

template <int W>
int mt_leaf(const mt::LeafJob *d_jobs, int n, uint64_t tiles, uint64_t perms, const P2Params<Goldilocks, W> &p,
            const char *name, cudaStream_t s) {
  DeviceContext *ctx;
  ZKB_TRY(current_context(&ctx));
  const Launch sh = shape<W>(tiles, perms, ctx->sm_count);
  ZKB_REQUIRE(n <= mt::MAX_JOBS, "internal: %d trees in one launch", n);
  const size_t smem = mt_smem<W>(n);
  ZKB_TRY(smem_limit<mt_smem<W>(mt::MAX_JOBS)>(mt_leaf_kernel<W>));
  ZKB_LAUNCH(name, s, mt_leaf_kernel<W><<<sh.grid, sh.threads, smem, s>>>(d_jobs, n, tiles, p, ctx->wait_word));
  return ZKB_OK;
}

template <int W>
int mt_compress(const mt::CompJob *d_jobs, int n, uint64_t total, const P2Params<Goldilocks, W> &p, const char *name,
                cudaStream_t s) {
  DeviceContext *ctx;
  ZKB_TRY(current_context(&ctx));
  const Launch sh = shape<W>((total + GROUP - 1) / GROUP, 1, ctx->sm_count);
  ZKB_REQUIRE(n <= mt::MAX_JOBS, "internal: %d trees in one launch", n);
  const size_t smem = mt_smem<W>(n);
  ZKB_TRY(smem_limit<mt_smem<W>(mt::MAX_JOBS)>(mt_compress_kernel<W>));
  ZKB_LAUNCH(name, s, mt_compress_kernel<W><<<sh.grid, sh.threads, smem, s>>>(d_jobs, n, total, p, ctx->wait_word));
  return ZKB_OK;
}

template <int W>
int permute(uint64_t *states, uint64_t n, const P2Params<Goldilocks, W> &p, cudaStream_t s) {
  DeviceContext *ctx;
  ZKB_TRY(current_context(&ctx));
  const Launch sh = shape<W>((n + GROUP - 1) / GROUP, 1, ctx->sm_count);
  const size_t smem = Shape<W>::SMEM;
  ZKB_TRY(smem_limit<Shape<W>::SMEM>(permute_kernel<W>));
  ZKB_LAUNCH("p2_permute", s, permute_kernel<W><<<sh.grid, sh.threads, smem, s>>>(states, n, p, ctx->wait_word));
  return ZKB_OK;
}

#define P2G_INSTANCE(W)                                                                                              \
  template bool takes<W>(const P2Params<Goldilocks, W> &, uint64_t);                                                 \
  template int hash_rows<W>(const MatList &, uint64_t, uint64_t *, const P2Params<Goldilocks, W> &, const char *,    \
                            cudaStream_t);                                                                           \
  template int compress<W>(const uint64_t *, uint64_t *, uint64_t, const uint64_t *, uint64_t,                       \
                           const P2Params<Goldilocks, W> &, const char *, cudaStream_t);                             \
  template int mt_leaf<W>(const mt::LeafJob *, int, uint64_t, uint64_t, const P2Params<Goldilocks, W> &, const char *, \
                          cudaStream_t);                                                                             \
  template int mt_compress<W>(const mt::CompJob *, int, uint64_t, const P2Params<Goldilocks, W> &, const char *,     \
                              cudaStream_t);                                                                         \
  template int permute<W>(uint64_t *, uint64_t, const P2Params<Goldilocks, W> &, cudaStream_t);
P2G_INSTANCE(12)
P2G_INSTANCE(16)

}  // namespace p2g
}  // namespace zkb
