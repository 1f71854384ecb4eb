// p2_launch.cuh — launches of the tensor-core hashing kernels (p2_tensor.cu).
#pragma once
#include <type_traits>

#include "common.cuh"
#include "fri_fold.cuh"
#include "matlist.cuh"
#include "poseidon2.cuh"

namespace zkb {
namespace mt {
struct LeafJob;
struct CompJob;
constexpr int MAX_JOBS = 1024;  // trees of one launch
}  // namespace mt

// The dynamic shared memory a kernel may be launched with.  The limit belongs to the function and the
// context, not to the calling thread, and a smaller value lowers it for everyone: BYTES is one
// constant per kernel, never the size of the launch at hand.
template <int BYTES, class K>
int smem_limit(K kernel) {
  static_assert(BYTES <= 227 * 1024, "more shared memory than a block can have");
  ZKB_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, BYTES));
  return ZKB_OK;
}

namespace p2t {

// True when a launch over this many rows (or compressions) takes the tensor-core kernels.
bool takes(const P2Params<BabyBear, 16> &p, uint64_t rows);
// Leaf digests of `height` rows (total width at least 1); with comb (one matrix) the rows'
// alpha-reductions too.
int hash_rows(const MatList &ml, uint64_t height, uint32_t *digests, const P2Params<BabyBear, 16> &p,
              const uint4 *apow, uint4 *comb, const char *name, cudaStream_t s);
// A slab of columns; every slab of a matrix goes through the same form (the carried words differ).
int hash_slab(const uint32_t *mat, uint64_t stride, uint64_t c0, uint64_t ncols, uint64_t height, uint32_t *carry,
              bool first, bool last, uint32_t *digests, const P2Params<BabyBear, 16> &p, const uint4 *apow, uint4 *comb,
              const char *name, cudaStream_t s);
int compress(const uint32_t *prev, uint32_t *next, uint64_t n_out, const uint32_t *inj, uint64_t inj_h,
             const P2Params<BabyBear, 16> &p, const char *name, cudaStream_t s);
// Leaves of many matrices: `tiles` 128-row tiles (LeafJob::tile_start), `perms` the largest
// row's permutations.
int mt_leaf(const mt::LeafJob *d_jobs, int n, uint64_t tiles, uint64_t perms, const P2Params<BabyBear, 16> &p,
            const char *name, cudaStream_t s);
int mt_compress(const mt::CompJob *d_jobs, int n, uint64_t total, const P2Params<BabyBear, 16> &p, const char *name,
                cudaStream_t s);
int fri_fold_hash(const uint32_t *e, uint32_t *out, uint64_t n_leaves, int log_out, const Ext4Params *prm,
                  const uint32_t *itw, uint32_t *digests, const P2Params<BabyBear, 16> &p, const char *name,
                  cudaStream_t s);
int permute(uint32_t *states, uint64_t n, const P2Params<BabyBear, 16> &p, cudaStream_t s);

}  // namespace p2t

// The same for Goldilocks, widths 12 and 16 (p2_tensor_gl.cu).
namespace p2g {

template <int W>
bool takes(const P2Params<Goldilocks, W> &p, uint64_t rows);
template <int W>
int hash_rows(const MatList &ml, uint64_t height, uint64_t *digests, const P2Params<Goldilocks, W> &p, const char *name,
              cudaStream_t s);
template <int W>
int compress(const uint64_t *prev, uint64_t *next, uint64_t n_out, const uint64_t *inj, uint64_t inj_h,
             const P2Params<Goldilocks, W> &p, const char *name, cudaStream_t s);
template <int W>
int mt_leaf(const mt::LeafJob *d_jobs, int n, uint64_t tiles, uint64_t perms, const P2Params<Goldilocks, W> &p,
            const char *name, cudaStream_t s);
template <int W>
int mt_compress(const mt::CompJob *d_jobs, int n, uint64_t total, const P2Params<Goldilocks, W> &p, const char *name,
                cudaStream_t s);
template <int W>
int permute(uint64_t *states, uint64_t n, const P2Params<Goldilocks, W> &p, cudaStream_t s);

}  // namespace p2g

// ---- the form of a launch, chosen by its size (rows, compressions or states) ----
// The tensor-core form above its smallest size.
template <class F, int W>
bool tensor_takes(const P2Params<F, W> &p, uint64_t rows) {
  if constexpr (std::is_same<F, BabyBear>::value)
    return p2t::takes(p, rows);
  else
    return p2g::takes<W>(p, rows);
}

}  // namespace zkb
