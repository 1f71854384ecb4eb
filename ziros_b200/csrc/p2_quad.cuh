// p2_quad.cuh — Poseidon2 with one state spread over four threads.
//
// A launch that cannot fill the GPU lasts as long as one permutation, and one thread needs
// thousands of dependent instructions for it (about 12 us on a B200 for BabyBear).  Here lane q of
// a quad holds words 4q..4q+3: the sixteen S-boxes of a full round are four deep instead of
// sixteen, M4 stays inside a lane, the column sums are two shuffles, and in a partial round the sum
// over the state (without the S-box word) and the diagonal products run while the S-box
// does.  Eight permutations a warp take about 2300 instructions, a quarter more than the same eight
// in single lanes, so the form is also the one for middle sizes (2^20 states take 1.5 times as long as one a
// thread).
//
// Tree levels below that size are one launch for up to eight levels: a block takes a run of S nodes
// and computes the whole subtree above them, level by level in shared memory.
#pragma once
#include "common.cuh"
#include "field.cuh"
#include "fri_fold.cuh"
#include "matlist.cuh"
#include "poseidon2.cuh"

namespace zkb {
namespace quad {

template <int W>
__host__ __device__ constexpr int out_words() {
  return W == 16 ? 8 : 4;
}

// Arithmetic of a lane's words: canonical internal-domain values.
template <class F>
struct Ops;
template <>
struct Ops<BabyBear> {
  using T = uint32_t;
  using B = BabyBear;
  static __host__ __device__ T rc(T c) { return c - B::P; }  // kept less p: x + rc fits a signed word
  static __device__ __forceinline__ T sbox(T x, T rcp) {
    const int y = (int)(x + rcp), y2 = B::smul(y, y), y3 = B::smul(y2, y), y4 = B::smul(y2, y2);
    return B::lift(B::smul(y3, y4));
  }
  static __device__ __forceinline__ T mul(T a, T b) { return B::lift(B::smul((int)a, (int)b)); }
  // rest + (1 + d_0) w: d_0 = -2 (P2Params::diag_kind 1, the only diagonal of this width)
  static __device__ __forceinline__ T next_y(T rest, T w, T, T) { return B::sub(rest, w); }
};
template <>
struct Ops<Goldilocks> {
  using T = unsigned long long;
  static __host__ __device__ T rc(T c) { return c; }
  static __device__ __forceinline__ T sbox(T x, T c) { return Goldilocks::canon(Goldilocks::pow7_any(Goldilocks::add(x, c))); }
  static __device__ __forceinline__ T mul(T a, T b) { return Goldilocks::mul(a, b); }
  static __device__ __forceinline__ T next_y(T, T w, T sum, T d0) { return Goldilocks::add(Goldilocks::mul(w, d0), sum); }
};

// Constants in shared memory, four words a lane (width 12: the fourth lane's are zero).
template <class F>
struct Consts {
  typename F::T full[P2_MAX_RC + 16 - P2_MAX_RC % 16];  // [round][16]
  typename F::T part[P2_MAX_RC];
  typename F::T diag[16];
  int half, partial;
};

template <class F, int W>
__device__ __forceinline__ void load_consts(Consts<F> &k, const P2Params<F, W> &p) {
  const int half = p.rounds_f / 2;
  for (int t = threadIdx.x; t < p.rounds_f * 16; t += blockDim.x) {
    const int r = t / 16, i = t % 16;
    k.full[t] = Ops<F>::rc(i < W ? p.rc[r * W + (r < half ? 0 : p.rounds_p) + i] : 0);
  }
  for (int t = threadIdx.x; t < p.rounds_p; t += blockDim.x) k.part[t] = Ops<F>::rc(p.rc[half * W + t]);
  for (int t = threadIdx.x; t < 16; t += blockDim.x) k.diag[t] = t < W ? p.diag[t] : 0;
  if (threadIdx.x == 0) {
    k.half = half;
    k.partial = p.rounds_p;
  }
  __syncthreads();
}

// Every lane of the warp calls this (full-mask shuffles: with a run-time mask each one would be preceded by a warp
// synchronisation).  Written for a short chain: M4's row i is (sum of the four) + s_i + 2 s_{i+1}.
template <class F, int W>
__device__ __forceinline__ void ext_mds(typename F::T (&s)[4], int q) {
  using D = Dom<F>;
  using T = typename F::T;
  const T t = D::add(D::add(s[0], s[1]), D::add(s[2], s[3]));
  T y[4];
#pragma unroll
  for (int i = 0; i < 4; i++) y[i] = D::add(t, D::add(s[i], D::add(s[(i + 1) & 3], s[(i + 1) & 3])));
#pragma unroll
  for (int k = 0; k < 4; k++) {
    T c = D::add(y[k], (T)__shfl_xor_sync(0xFFFFFFFFu, (typename Ops<F>::T)y[k], 1));
    c = D::add(c, (T)__shfl_xor_sync(0xFFFFFFFFu, (typename Ops<F>::T)c, 2));
    s[k] = W == 12 && q == 3 ? 0 : D::add(y[k], c);
  }
}

template <class F, int W>
__device__ __forceinline__ void full_round(typename F::T (&s)[4], const typename F::T (&rc)[4], int q) {
#pragma unroll
  for (int i = 0; i < 4; i++) {
    s[i] = Ops<F>::sbox(s[i], rc[i]);
    if (W == 12 && q == 3) s[i] = 0;
  }
  ext_mds<F, W>(s, q);
}

// The four lanes of a quad hold one state; q: this lane's place among them.  Constants are read a
// round ahead.
template <class F, int W>
__device__ __forceinline__ void permute(typename F::T (&s)[4], const Consts<F> &k, int q) {
  using D = Dom<F>;
  using T = typename F::T;
  using U = typename Ops<F>::T;
  const int half = k.half, partial = k.partial;
  T rc[4], d[4];
#pragma unroll
  for (int i = 0; i < 4; i++) rc[i] = k.full[4 * q + i];
#pragma unroll
  for (int i = 0; i < 4; i++) d[i] = k.diag[4 * q + i];
  ext_mds<F, W>(s, q);
#pragma unroll 1
  for (int h = 0; h < 2; h++) {
#pragma unroll 1
    for (int r = 0; r < half; r++) {
      T nx[4];
      const int at = min(h * half + r + 1, 2 * half - 1) * 16 + 4 * q;
#pragma unroll
      for (int i = 0; i < 4; i++) nx[i] = k.full[at + i];
      full_round<F, W>(s, rc, q);
#pragma unroll
      for (int i = 0; i < 4; i++) rc[i] = nx[i];
    }
    if (h) break;
    // s_0' = rest + (1 + d_0) w, s_i' = d_i s_i + rest + w, with w the S-box output and rest the sum of
    // the other words: the sum and the products do not wait for the S-box, nor it for them.
    T c = k.part[0], y = s[0];  // the first lane's y is the state's word 0
#pragma unroll 1
    for (int pr = 0; pr < partial; pr++) {
      const T cn = k.part[min(pr + 1, partial - 1)];
      T rest = D::add(D::add(q ? s[0] : 0, s[1]), D::add(s[2], s[3]));
      T m[4];
#pragma unroll
      for (int i = 0; i < 4; i++) m[i] = Ops<F>::mul(s[i], d[i]);
      rest = D::add(rest, (T)__shfl_xor_sync(0xFFFFFFFFu, (U)rest, 1));
      const T w0 = Ops<F>::sbox(y, c);
      rest = D::add(rest, (T)__shfl_xor_sync(0xFFFFFFFFu, (U)rest, 2));
      const T w = (T)__shfl_sync(0xFFFFFFFFu, (U)w0, 0, 4), sum = D::add(rest, w);
      y = Ops<F>::next_y(rest, w0, sum, d[0]);
#pragma unroll
      for (int i = 0; i < 4; i++) s[i] = D::add(m[i], sum);
      if (W == 12 && q == 3) s[0] = s[1] = s[2] = s[3] = 0;
      c = cn;
    }
    if (q == 0) s[0] = y;
  }
}

// The same with one word to a lane, sixteen lanes a state (width 12: the last four idle), for the upper tree
// levels, where threads are left over: one S-box deep instead of four, at two
// and a half times the instructions per state.  d: this lane's diagonal word.
template <class F, int W>
__device__ __forceinline__ typename F::T ext_mds_lane(typename F::T s, int lane) {
  using D = Dom<F>;
  using T = typename F::T;
  using U = typename Ops<F>::T;
  const T next = (T)__shfl_sync(0xFFFFFFFFu, (U)s, (lane & ~3) | ((lane + 1) & 3), 16);
  T t = D::add(s, (T)__shfl_xor_sync(0xFFFFFFFFu, (U)s, 1));
  t = D::add(t, (T)__shfl_xor_sync(0xFFFFFFFFu, (U)t, 2));
  const T y = D::add(t, D::add(s, D::add(next, next)));
  T c = D::add(y, (T)__shfl_xor_sync(0xFFFFFFFFu, (U)y, 4));
  c = D::add(c, (T)__shfl_xor_sync(0xFFFFFFFFu, (U)c, 8));
  return W == 12 && lane >= 12 ? 0 : D::add(y, c);
}
template <class F, int W>
__device__ __forceinline__ typename F::T permute_lane(typename F::T s, const Consts<F> &k, int lane) {
  using D = Dom<F>;
  using T = typename F::T;
  using U = typename Ops<F>::T;
  const int half = k.half, partial = k.partial;
  const T d = k.diag[lane];
  T rc = k.full[lane];
  s = ext_mds_lane<F, W>(s, lane);
#pragma unroll 1
  for (int h = 0; h < 2; h++) {
#pragma unroll 1
    for (int r = 0; r < half; r++) {
      const T nx = k.full[min(h * half + r + 1, 2 * half - 1) * 16 + lane];
      s = Ops<F>::sbox(s, rc);
      if (W == 12 && lane >= 12) s = 0;
      s = ext_mds_lane<F, W>(s, lane);
      rc = nx;
    }
    if (h) break;
    T c = k.part[0], y = s;
#pragma unroll 1
    for (int pr = 0; pr < partial; pr++) {
      const T cn = k.part[min(pr + 1, partial - 1)];
      T rest = lane ? s : 0;
      const T m = Ops<F>::mul(s, d);
      rest = D::add(rest, (T)__shfl_xor_sync(0xFFFFFFFFu, (U)rest, 1));
      const T w0 = Ops<F>::sbox(y, c);
      rest = D::add(rest, (T)__shfl_xor_sync(0xFFFFFFFFu, (U)rest, 2));
      rest = D::add(rest, (T)__shfl_xor_sync(0xFFFFFFFFu, (U)rest, 4));
      rest = D::add(rest, (T)__shfl_xor_sync(0xFFFFFFFFu, (U)rest, 8));
      const T w = (T)__shfl_sync(0xFFFFFFFFu, (U)w0, 0, 16), sum = D::add(rest, w);
      y = Ops<F>::next_y(rest, w0, sum, d);
      s = D::add(m, sum);
      if (W == 12 && lane >= 12) s = 0;
      c = cn;
    }
    if (lane == 0) s = y;
  }
  return s;
}

template <class T>
__device__ __forceinline__ void load_words(T (&x)[4], const T *from) {
  if constexpr (sizeof(T) == 4) {
    const uint4 v = *reinterpret_cast<const uint4 *>(from);
    x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
  } else {
    const ulonglong2 a = reinterpret_cast<const ulonglong2 *>(from)[0], b = reinterpret_cast<const ulonglong2 *>(from)[1];
    x[0] = a.x, x[1] = a.y, x[2] = b.x, x[3] = b.y;
  }
}
template <class F>
__device__ __forceinline__ void store_words(typename F::T *to, const typename F::T (&s)[4]) {
  using D = Dom<F>;
  if constexpr (sizeof(typename F::T) == 4) {
    *reinterpret_cast<uint4 *>(to) = make_uint4(D::leave(s[0]), D::leave(s[1]), D::leave(s[2]), D::leave(s[3]));
  } else {
    reinterpret_cast<ulonglong2 *>(to)[0] = make_ulonglong2(D::leave(s[0]), D::leave(s[1]));
    reinterpret_cast<ulonglong2 *>(to)[1] = make_ulonglong2(D::leave(s[2]), D::leave(s[3]));
  }
}
template <class F>
__device__ __forceinline__ void enter(typename F::T (&s)[4]) {
#pragma unroll
  for (int i = 0; i < 4; i++) s[i] = Dom<F>::enter(s[i]);
}

// This thread's quad among the grid's.  Loops over items run warp by warp (a quad past the end
// repeats the last item), so that the shuffles of a permutation always have the whole warp.
struct Lane {
  int q;
  uint64_t warp0, quad, stride;  // first item of the warp, this quad's place in it, quads of the grid
};
__device__ __forceinline__ Lane lane() {
  const int l = threadIdx.x & 31;
  return {l & 3, (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 8, (uint64_t)(l >> 2),
          (uint64_t)gridDim.x * blockDim.x >> 2};
}
#define QUAD_ITEMS(l, item, live, n)                                                    \
  for (uint64_t w_ = (l).warp0, item, live; w_ < (n); w_ += (l).stride)                 \
    if (item = w_ + (l).quad, live = item < (n), item = live ? item : (n) - 1; true)

// Absorbs columns [0, width) of a row read by get(column); the rate is the first two lanes' words.
// The quads of a warp may have rows of different widths: one that is done keeps its state.
template <class F, int W, bool SAME, class Get, class Each>
__device__ __forceinline__ void absorb(typename F::T (&s)[4], uint64_t width, const Consts<F> &k, int q, Get get, Each each) {
  using T = typename F::T;
  T x[4];
  auto load = [&](uint64_t c) {
#pragma unroll
    for (int i = 0; i < 4; i++) x[i] = q < 2 && c + 4 * q + i < width ? get(c + 4 * q + i) : 0;
  };
  load(0);
  for (uint64_t c = 0; SAME ? c < width : __any_sync(0xFFFFFFFFu, c < width); c += 8) {
    T kept[4];
    if (!SAME) {
#pragma unroll
      for (int i = 0; i < 4; i++) kept[i] = s[i];
    }
    if (q < 2) {
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (c + 4 * q + i < width) s[i] = Dom<F>::enter(x[i]);
      each(x, c + 4 * q);
    }
    load(c + 8);  // on its way while the permutation runs
    permute<F, W>(s, k, q);
    if (!SAME && c >= width) {
#pragma unroll
      for (int i = 0; i < 4; i++) s[i] = kept[i];
    }
  }
}

template <class F, int W>
__global__ void __launch_bounds__(128)
    rows_kernel(const MatList ml, uint64_t height, typename F::T *__restrict__ digests,
                const __grid_constant__ P2Params<F, W> p) {
  using T = typename F::T;
  __shared__ Consts<F> k;
  load_consts<F, W>(k, p);
  const Lane l = lane();
  const uint64_t width = ml.col_start[ml.n];
  QUAD_ITEMS(l, row, live, height) {
    T s[4] = {0, 0, 0, 0};
    const T *rp = (const T *)ml.ptr[0] + row * ml.width[0];
    if (ml.n == 1)
      absorb<F, W, true>(s, width, k, l.q, [&](uint64_t c) { return rp[c]; }, [](const T(&)[4], uint64_t) {});
    else
      absorb<F, W, true>(s, width, k, l.q, [&](uint64_t c) { return fetch_col<F>(ml, row, c); },
                   [](const T(&)[4], uint64_t) {});
    if (live && 4 * l.q < out_words<W>()) store_words<F>(digests + row * out_words<W>() + 4 * l.q, s);
  }
}

// Leaves of many matrices (one job each).
template <class F, int W, class Job>
__global__ void __launch_bounds__(256)
    mt_rows_kernel(const Job *__restrict__ jobs, int n_jobs, uint64_t total_rows, const __grid_constant__ P2Params<F, W> p) {
  using T = typename F::T;
  extern __shared__ uint64_t starts[];  // n_jobs entries
  __shared__ Consts<F> k;
  for (int i = threadIdx.x; i < n_jobs; i += blockDim.x) starts[i] = jobs[i].row_start;
  load_consts<F, W>(k, p);
  const Lane l = lane();
  QUAD_ITEMS(l, g, live, total_rows) {
    int lo = 0, hi = n_jobs - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (starts[mid] <= g)
        lo = mid;
      else
        hi = mid - 1;
    }
    const uint64_t row = g - starts[lo], width = jobs[lo].width;
    const T *rp = (const T *)jobs[lo].data + row * width;
    T s[4] = {0, 0, 0, 0};
    absorb<F, W, false>(s, width, k, l.q, [&](uint64_t c) { return rp[c]; }, [](const T(&)[4], uint64_t) {});
    if (live && 4 * l.q < out_words<W>()) store_words<F>((T *)jobs[lo].digests + row * out_words<W>() + 4 * l.q, s);
  }
}

// next[i] = compress(compress(prev[2i], prev[2i+1]), i < inj_h ? inj[i] : 0): an injected level.
template <class F, int W>
__global__ void __launch_bounds__(128)
    inject_kernel(const typename F::T *__restrict__ prev, typename F::T *__restrict__ next, uint64_t n_out,
                  const typename F::T *__restrict__ inj, uint64_t inj_h, const __grid_constant__ P2Params<F, W> p) {
  using T = typename F::T;
  constexpr int OUT = out_words<W>();
  __shared__ Consts<F> k;
  load_consts<F, W>(k, p);
  const Lane l = lane();
  QUAD_ITEMS(l, i, live, n_out) {
    T s[4] = {0, 0, 0, 0};
    if (4 * l.q < 2 * OUT) load_words<T>(s, prev + i * 2 * OUT + 4 * l.q);
    enter<F>(s);
    permute<F, W>(s, k, l.q);
    if (4 * l.q >= OUT) {
      s[0] = s[1] = s[2] = s[3] = 0;
      if (4 * l.q < 2 * OUT && i < inj_h) {
        load_words<T>(s, inj + i * OUT + (4 * l.q - OUT));
        enter<F>(s);
      }
    }
    permute<F, W>(s, k, l.q);
    if (live && 4 * l.q < OUT) store_words<F>(next + i * OUT + 4 * l.q, s);
  }
}

// The subtree of `levels` levels over nodes [block * 2^levels, ...) of a layer: layer(j) is layer j's
// first digest and nodes(j) its number of computed nodes (those past it are zero), j = 0 the layer
// read.  buf: 2^levels digests of shared memory.
template <class F, int W, class Layer, class Nodes>
__device__ __forceinline__ void subtree(uint64_t block, int levels, Layer layer, Nodes nodes, typename F::T *buf,
                                        const Consts<F> &k) {
  using T = typename F::T;
  constexpr int OUT = out_words<W>();
  const int q = threadIdx.x & 3;
  T *from = buf, *to = buf;  // level j's digests: 2^(levels - 1 - j) of them, one after another
  for (int j = 0; j < levels; j++) {
    const uint64_t cnt = 1ull << (levels - 1 - j), base = block * cnt, below = nodes(j), n = nodes(j + 1);
    if (cnt * 16 <= blockDim.x) {  // few enough for a lane to a word
      const int lane = threadIdx.x & 15;
      const uint64_t o = threadIdx.x / 16;
      const bool live = o < cnt && base + o < n;
      if (threadIdx.x / 32 * 2 < cnt) {  // whole warps
        T s = 0;
        const int child = lane / OUT;
        if (live && child < 2) {
          if (j == 0)
            s = layer(0)[(base + o) * 2 * OUT + lane];
          else if (2 * (base + o) + child < below)
            s = from[o * 2 * OUT + lane];
        }
        s = Dom<F>::leave(permute_lane<F, W>(Dom<F>::enter(s), k, lane));
        if (live && lane < OUT) {
          layer(j + 1)[(base + o) * OUT + lane] = s;
          if (j + 1 < levels) to[o * OUT + lane] = s;
        }
      }
      __syncthreads();
      from = to;
      to += cnt * OUT;
      continue;
    }
    for (uint64_t w = threadIdx.x / 32 * 8; w < cnt && base + w < n; w += blockDim.x >> 2) {
      const uint64_t o = w + threadIdx.x % 32 / 4;
      const bool live = o < cnt && base + o < n;
      T s[4] = {0, 0, 0, 0};
      const int child = 4 * q / OUT;  // 0, 1: left, right; 2 and more: none (width 12)
      if (live && child < 2) {
        if (j == 0)
          load_words<T>(s, layer(0) + (base + o) * 2 * OUT + 4 * q);
        else if (2 * (base + o) + child < below)
          load_words<T>(s, from + o * 2 * OUT + 4 * q);
      }
      enter<F>(s);
      permute<F, W>(s, k, q);
      if (live && 4 * q < OUT) {
        store_words<F>(layer(j + 1) + (base + o) * OUT + 4 * q, s);
        if (j + 1 < levels) store_words<F>(to + o * OUT + 4 * q, s);
      }
    }
    __syncthreads();
    from = to;
    to += cnt * OUT;
  }
}

constexpr int MAX_RUN = 8;  // levels of one launch

// Where a tree's layers lie: layer j of the run starts `off[j]` digests into `layers` and has n[j]
// computed nodes.
struct Run {
  void *layers;
  uint64_t off[MAX_RUN + 1];
  uint64_t n[MAX_RUN + 1];
};

template <class F, int W>
__global__ void __launch_bounds__(512)
    levels_kernel(const Run run, int levels, const __grid_constant__ P2Params<F, W> p) {
  using T = typename F::T;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ Consts<F> k;
  load_consts<F, W>(k, p);
  subtree<F, W>(
      blockIdx.x, levels, [&](int j) { return (T *)run.layers + run.off[j] * out_words<W>(); },
      [&](int j) { return run.n[j]; }, (T *)smem, k);
}

// The same for the trees of many jobs (power-of-two rows, layers back to back): the run starts at
// layer `l0` of each; a job that has fewer layers takes part as far as it goes.
template <class F, int W, class Job>
__global__ void __launch_bounds__(512)
    mt_levels_kernel(const Job *__restrict__ jobs, int n_jobs, int l0, int levels, const __grid_constant__ P2Params<F, W> p) {
  using T = typename F::T;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ Consts<F> k;
  __shared__ int s_job;
  __shared__ uint64_t s_block;
  load_consts<F, W>(k, p);
  if (threadIdx.x < 32) {  // the job of this block: a warp adds up the jobs' blocks, 32 at a time
    uint64_t before = 0;
    for (int i0 = 0; i0 < n_jobs; i0 += 32) {
      const int i = i0 + threadIdx.x;
      const uint64_t rows = i < n_jobs ? jobs[i].rows >> l0 : 0;
      const uint64_t mine = rows < 2 ? 0 : (rows + (1ull << levels) - 1) >> levels;
      uint64_t upto = mine;
#pragma unroll
      for (int d = 1; d < 32; d *= 2) {
        const uint64_t v = __shfl_up_sync(0xFFFFFFFFu, (unsigned long long)upto, d);
        if ((int)threadIdx.x >= d) upto += v;
      }
      const uint64_t lo = before + upto - mine;
      if (mine && blockIdx.x >= lo && blockIdx.x < lo + mine) {
        s_job = i;
        s_block = blockIdx.x - lo;
      }
      before += __shfl_sync(0xFFFFFFFFu, (unsigned long long)upto, 31);
      if (blockIdx.x < before) break;
    }
  }
  __syncthreads();
  const uint64_t rows = jobs[s_job].rows;
  T *layers = (T *)jobs[s_job].digests;
  subtree<F, W>(
      s_block, levels,
      [&](int j) { return layers + (2 * rows - ((2 * rows) >> (l0 + j))) * out_words<W>(); },
      [&](int j) { return l0 + j < 63 ? rows >> (l0 + j) : 0; }, (T *)smem, k);
}

template <class F, int W>
__global__ void __launch_bounds__(128)
    states_kernel(typename F::T *__restrict__ states, uint64_t n, const __grid_constant__ P2Params<F, W> p) {
  using T = typename F::T;
  __shared__ Consts<F> k;
  load_consts<F, W>(k, p);
  const Lane l = lane();
  QUAD_ITEMS(l, i, live, n) {
    T s[4] = {0, 0, 0, 0};
    if (4 * l.q < W) {
#pragma unroll
      for (int j = 0; j < 4; j++) s[j] = Dom<F>::enter(states[i * W + 4 * l.q + j]);
    }
    permute<F, W>(s, k, l.q);
    if (live && 4 * l.q < W) {
#pragma unroll
      for (int j = 0; j < 4; j++) states[i * W + 4 * l.q + j] = Dom<F>::leave(s[j]);
    }
  }
}

inline unsigned grid_of(uint64_t items, unsigned threads) { return grid_for(items * 4, threads, 1u << 30); }

// Levels per launch for a run of `total` levels: as few launches as MAX_RUN levels each allow, of
// equal length.
inline int run_levels(int total) {
  const int stages = (total + MAX_RUN - 1) / MAX_RUN;
  return (total + stages - 1) / stages;
}
// Four threads for each of the first level's nodes (up to 512), which is sixteen for each of the third's.
inline unsigned run_threads(int levels) {
  const int t = 4 << (levels - 1);
  return (unsigned)(t < 32 ? 32 : t > 512 ? 512 : t);
}
template <class F, int W>
size_t run_smem(int levels) {
  return ((size_t)1 << levels) * out_words<W>() * sizeof(typename F::T);
}

}  // namespace quad
}  // namespace zkb
