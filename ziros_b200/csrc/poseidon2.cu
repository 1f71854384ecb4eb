// poseidon2.cu — batch Poseidon2 permutation (Poseidon2Accelerator::batch_permute_*).
#include "common.cuh"
#include "engine.cuh"
#include "p2_launch.cuh"
#include "p2_quad.cuh"
#include "poseidon2.cuh"

namespace zkb {

template <class F, int W>
bool build_p2_params(const uint64_t *rc, size_t n_rc, int rounds_f, int rounds_p,
                     const uint64_t *diag, int out, P2Params<F, W> *p) {
  if (rounds_f <= 0 || rounds_f % 2 || rounds_p < 0) return false;
  if ((size_t)rounds_f * W + rounds_p != n_rc || n_rc > (size_t)P2_MAX_RC) return false;
  for (size_t i = 0; i < n_rc; i++) {
    if (rc[i] >= (uint64_t)F::P) return false;
    p->rc[i] = Dom<F>::encode(rc[i]);
  }
  for (int i = 0; i < W; i++) {
    if (diag[i] >= (uint64_t)F::P) return false;
    p->diag[i] = Dom<F>::encode(diag[i]);
  }
  p->rounds_f = rounds_f;
  p->rounds_p = rounds_p;
  p->out = out;
  p->rate = 8;
  p->diag_kind = 0;
  {
    const std::vector<uint64_t> &v = p2_diagonal(sizeof(typename F::T) == 4 ? FIELD_BABYBEAR : FIELD_GOLDILOCKS, W);
    bool same = true;
    for (int i = 0; i < W; i++) same = same && diag[i] == v[i];
    p->diag_kind = same ? 1 : 0;
  }
  return true;
}

template <class F, int W>
bool build_p2_params(const HasherSpec &h, P2Params<F, W> *p) {
  if (h.width != W) return false;
  return build_p2_params<F, W>(h.rc.data(), h.rc.size(), h.rounds_f, h.rounds_p, h.diag.data(),
                               h.out, p);
}

// One state a thread: the form of middle sizes (tensor_batch below), and of large ones for instances that the
// tensor-core kernels are not built for (other numbers of rounds).
template <class F, int W>
__global__ void __launch_bounds__(128)
    states_kernel(typename F::T *__restrict__ states, size_t n, const __grid_constant__ P2Params<F, W> p) {
  using T = typename F::T;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    T s[W];
    T *g = states + i * W;
#pragma unroll
    for (int k = 0; k < W; k++) s[k] = Dom<F>::enter(g[k]);
    p2_permute<F, W>(s, p);
#pragma unroll
    for (int k = 0; k < W; k++) g[k] = Dom<F>::leave(s[k]);
  }
}

// States from which it beats quads of threads (p2_quad.cuh).  BabyBear
// 8 + 22 rounds: 19,000 states 22.5 us against 23.5, 40,000 29.7 against 33.8, 2^20 382 against 611; 8 + 14: equal up to
// 28,000, 2^20 331 against 488.  Goldilocks 8 + 21: 60,000 169 against 155, 70,000 169 against 175, 2^20 1957 against
// 2403.
template <class F>
static constexpr size_t one_per_thread() {
  return sizeof(typename F::T) == 4 ? 148 * 128 + 1 : 1 << 16;
}

// The tensor-core form of a batch: one permutation a state, so its tables and a last round of fewer than five
// tiles an SM are not paid for as a leaf hash's are.  BabyBear by 128-state tiles an SM (148 SMs), against one
// state a thread: two tiles 23.0 us against 21.0, three to five 25.0, 27.1 and 32.5 against 27.2, 27.2 and 33.0, six
// to thirteen slower or equal (100,000 states 45.3 against 43.4, 200,000 70.7 against 68.2), from fourteen on
// faster (400,000 122 against 128, 2^20 273 against 322).  Goldilocks is faster at every size.
template <class F>
static bool tensor_batch(size_t n, int sms) {
  if (sizeof(typename F::T) == 8) return true;
  const uint64_t tiles = ((n + 127) / 128 + sms - 1) / sms;
  return (tiles >= 3 && tiles <= 5) || tiles >= 14;
}

template <class F, int W>
int p2_permute_batch(typename F::T *d_states, size_t n_states, const P2Params<F, W> &p,
                     cudaStream_t s) {
  if (n_states == 0) return ZKB_OK;
  const unsigned threads = 128;
  const bool tensor = tensor_takes<F, W>(p, n_states);
  if (tensor || n_states >= one_per_thread<F>()) {
    DeviceContext *ctx;
    ZKB_TRY(current_context(&ctx));
    if (tensor && tensor_batch<F>(n_states, ctx->sm_count)) {
      if constexpr (std::is_same<F, BabyBear>::value)
        return p2t::permute(d_states, n_states, p, s);
      else
        return p2g::permute<W>(d_states, n_states, p, s);
    }
    const unsigned grid = grid_for(n_states, threads, (unsigned)ctx->sm_count * 16u);
    ZKB_LAUNCH("p2_permute", s, states_kernel<F, W><<<grid, threads, 0, s>>>(d_states, n_states, p));
    return ZKB_OK;
  }
  ZKB_LAUNCH("p2_permute", s, quad::states_kernel<F, W><<<quad::grid_of(n_states, threads), threads, 0, s>>>(d_states, n_states, p));
  return ZKB_OK;
}

template bool build_p2_params<BabyBear, 16>(const uint64_t *, size_t, int, int, const uint64_t *,
                                            int, P2Params<BabyBear, 16> *);
template bool build_p2_params<Goldilocks, 16>(const uint64_t *, size_t, int, int,
                                              const uint64_t *, int, P2Params<Goldilocks, 16> *);
template bool build_p2_params<Goldilocks, 12>(const uint64_t *, size_t, int, int,
                                              const uint64_t *, int, P2Params<Goldilocks, 12> *);
template bool build_p2_params<BabyBear, 16>(const HasherSpec &, P2Params<BabyBear, 16> *);
template bool build_p2_params<Goldilocks, 16>(const HasherSpec &, P2Params<Goldilocks, 16> *);
template bool build_p2_params<Goldilocks, 12>(const HasherSpec &, P2Params<Goldilocks, 12> *);
template int p2_permute_batch<BabyBear, 16>(uint32_t *, size_t, const P2Params<BabyBear, 16> &,
                                            cudaStream_t);
template int p2_permute_batch<Goldilocks, 16>(uint64_t *, size_t,
                                              const P2Params<Goldilocks, 16> &, cudaStream_t);
template int p2_permute_batch<Goldilocks, 12>(uint64_t *, size_t,
                                              const P2Params<Goldilocks, 12> &, cudaStream_t);

}  // namespace zkb
