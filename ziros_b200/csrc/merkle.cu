// merkle.cu — Poseidon2 MMCS: leaf sponge hashing, 2-to-1 compression, tree layers.
//
// Semantics follow p3 MerkleTree::new as vendored in
// vendor/p3-merkle-tree-gpu/src/merkle_tree.rs:84-151 (first_digest_layer :202-266,
// compress_and_inject :272-350, compress :359-403) with
//   leaf  = PaddingFreeSponge<Perm, W, 8, OUT> over the concatenated rows of the
//           tallest matrices (overwrite-mode absorption, partial last chunk keeps
//           the old lanes, zkf-backends/src/wrapping/poseidon2_goldilocks.rs:392-415);
//   node  = TruncatedPermutation<Perm, 2, OUT, W> (poseidon2_goldilocks.rs:373-390);
//   layer lengths padded to even with zero digests except at the root; shorter
//   matrices injected as compress(compress(l, r), hash(rows)).
// Unlike the reference's Metal path (zkf-metal/src/merkle.rs:82-90), which falls back
// to the CPU for rows wider than 8 elements, every width is hashed on the device.
#include <algorithm>
#include <type_traits>
#include <numeric>

#include "common.cuh"
#include "engine.cuh"
#include "matlist.cuh"
#include "p2_launch.cuh"
#include "p2_quad.cuh"
#include "poseidon2.cuh"

namespace zkb {

template <int W>
__host__ __device__ constexpr int p2_out() {
  return W == 16 ? 8 : 4;
}

// The leaf sponge of one BabyBear matrix with the alpha-reduction of each row fused in, or of a slab
// [c0, c0 + ncols) of its columns (row stride `stride`) when it arrives a slab at a time.
// While the row streams through the sponge, comb[row] accumulates sum_j alpha^j * row[j]
// (apow, when given: alpha^j * 2^64 encoded; two columns per reduction, v0*w0 + v1*w1 < 2p^2 <
// p*2^32).  The sponge state comes from `carry` (16 words per row, internal domain; none on the
// first slab) and goes back there, or on the last slab the digest goes to `digests`.  c0 is a
// multiple of 8 (slabs hold whole absorbed chunks; only the last may end in a partial one),
// so the chunks and permutations are exactly the full row's; the slabs' reductions add up to
// the row's.
__global__ void __launch_bounds__(128)
    quad_slab_kernel(const uint32_t *__restrict__ mat, uint64_t stride, uint64_t c0, uint64_t ncols, uint64_t height,
                     uint32_t *__restrict__ carry, int first, int last, uint32_t *__restrict__ digests,
                     const __grid_constant__ P2Params<BabyBear, 16> p, const uint4 *__restrict__ apow,
                     uint4 *__restrict__ comb) {
  using B = BabyBear;
  __shared__ quad::Consts<B> k;
  quad::load_consts<B, 16>(k, p);
  const quad::Lane l = quad::lane();
  QUAD_ITEMS(l, row, live, height) {
    uint32_t s[4] = {0, 0, 0, 0};
    if (!first) quad::load_words<uint32_t>(s, carry + row * 16 + 4 * l.q);
    uint64_t a0 = 0, a1 = 0, a2 = 0, a3 = 0;
    const uint32_t *rp = mat + row * stride + c0;
    const uint4 *ap = apow ? apow + c0 : nullptr;
    quad::absorb<B, 16, true>(
        s, ncols, k, l.q, [&](uint64_t c) { return rp[c]; },
        [&](const uint32_t(&x)[4], uint64_t c) {
          if (!ap) return;
#pragma unroll
          for (int i = 0; i < 4; i += 2) {
            if (c + i >= ncols) break;
            const uint4 w0 = ap[c + i];
            const uint4 w1 = c + i + 1 < ncols ? ap[c + i + 1] : make_uint4(0, 0, 0, 0);
            a0 += B::mont_lazy_sum(x[i], w0.x, x[i + 1], w1.x);
            a1 += B::mont_lazy_sum(x[i], w0.y, x[i + 1], w1.y);
            a2 += B::mont_lazy_sum(x[i], w0.z, x[i + 1], w1.z);
            a3 += B::mont_lazy_sum(x[i], w0.w, x[i + 1], w1.w);
          }
        });
    if (!last) {
      if (live) *reinterpret_cast<uint4 *>(carry + row * 16 + 4 * l.q) = make_uint4(s[0], s[1], s[2], s[3]);
    } else if (live && l.q < 2) {
      quad::store_words<B>(digests + row * 8 + 4 * l.q, s);
    }
    if (ap) {  // the first two lanes have the sums of their columns
      uint32_t r[4] = {B::mont_reduce(a0), B::mont_reduce(a1), B::mont_reduce(a2), B::mont_reduce(a3)};
#pragma unroll
      for (int i = 0; i < 4; i++) r[i] = B::add(r[i], __shfl_xor_sync(0xFFFFFFFFu, r[i], 1));
      if (live && l.q == 0) {
        if (!first) {
          const uint4 o = comb[row];
          r[0] = B::add(o.x, r[0]), r[1] = B::add(o.y, r[1]), r[2] = B::add(o.z, r[2]), r[3] = B::add(o.w, r[3]);
        }
        comb[row] = make_uint4(r[0], r[1], r[2], r[3]);
      }
    }
  }
}

DeviceTree::~DeviceTree() {
  int prev = 0;
  cudaGetDevice(&prev);
  cudaSetDevice(device);
  if (d_layers && !borrowed) dev_free(d_layers, stream);
  for (void *p : owned) dev_free(p, stream);
  cudaSetDevice(prev);
}

static uint64_t next_pow2_u64(uint64_t x) { return ceil_pow2(x); }

static int log2_ceil(uint64_t x) {
  int l = 0;
  while ((1ull << l) < x) l++;
  return l;
}

template <class F, int W>
static int build_tree_impl(const HasherSpec &h, const std::vector<TreeMatrix> &mats,
                           DeviceTree *t, cudaStream_t s, bool fri_layer, const LeafCombine *comb,
                           const LeafFill *fill) {
  const char *leaf_name = fri_layer ? "fri_leaf_hash" : "merkle_leaf_hash";
  const char *comp_name = fri_layer ? "fri_compress" : "merkle_compress";
  using T = typename F::T;
  constexpr int OUT = p2_out<W>();
  P2Params<F, W> p;
  if (!build_p2_params<F, W>(h, &p)) {
    set_error("invalid Poseidon2 parameters");
    return ZKB_ERR_INVALID;
  }
  DeviceContext *ctx;
  ZKB_TRY(current_context(&ctx));

  const size_t nm = mats.size();
  std::vector<size_t> ord(nm);
  std::iota(ord.begin(), ord.end(), 0);
  std::stable_sort(ord.begin(), ord.end(),
                   [&](size_t a, size_t b) { return mats[a].height > mats[b].height; });
  const uint64_t max_h = mats[ord[0]].height;
  ZKB_REQUIRE(max_h > 0, "matrix height 0 not supported");
  const int log_max = log2_ceil(max_h);
  for (size_t i = 0; i < nm; i++) {
    const uint64_t hgt = mats[i].height;
    ZKB_REQUIRE(hgt > 0, "matrix height 0 not supported");
    const int bits_reduced = log_max - log2_ceil(hgt);
    const uint64_t expected = ((max_h - 1) >> bits_reduced) + 1;
    ZKB_REQUIRE(hgt == expected, "matrix height %llu incompatible with tallest height %llu",
                (unsigned long long)hgt, (unsigned long long)max_h);
  }
  for (size_t i = 0; i + 1 < nm; i++) {
    uint64_t a = mats[ord[i]].height, b = mats[ord[i + 1]].height;
    ZKB_REQUIRE(a == b || next_pow2_u64(a) != next_pow2_u64(b),
                "matrix heights that round up to the same power of two must be equal");
  }

  // layer lengths
  t->layer_len.clear();
  t->layer_off.clear();
  uint64_t len = max_h == 1 ? 1 : max_h + (max_h & 1), total = 0;
  for (;;) {
    t->layer_off.push_back(total);
    t->layer_len.push_back(len);
    total += len;
    if (len == 1) break;
    len = len == 2 ? 1 : ((len / 2 + 1) & ~1ull);
  }
  t->spec = h;
  t->stream = s;
  t->device = ctx->device;
  t->mats = mats;
  ZKB_TRY(dev_alloc(&t->d_layers, total * OUT * sizeof(T), s));
  T *layers = (T *)t->d_layers;
  ZKB_CHECK_CUDA(cudaMemsetAsync(layers, 0, total * OUT * sizeof(T), s));

  auto make_list = [&](size_t first, size_t count, MatList *ml) -> int {
    ZKB_REQUIRE(count <= (size_t)MAX_GROUP_MATS, "more than %d matrices share one height",
                MAX_GROUP_MATS);
    ml->n = (int)count;
    ml->col_start[0] = 0;
    for (size_t i = 0; i < count; i++) {
      const TreeMatrix &m = mats[ord[first + i]];
      ml->ptr[i] = m.data;
      ml->width[i] = m.width;
      ml->col_start[i + 1] = ml->col_start[i] + m.width;
    }
    return ZKB_OK;
  };

  size_t ng = 0;
  while (ng < nm && mats[ord[ng]].height == max_h) ng++;
  MatList ml;
  ZKB_TRY(make_list(0, ng, &ml));
  const unsigned thr = 128;
  // Both forms' blocks retire every few milliseconds at most (a quad's after a row or two, the tensor-core
  // form's after a unit of work, p2_tensor.cu: shape), so kernels of other streams (other jobs of the
  // engine, which gives small jobs higher stream priority) get SMs in between.
  // Leaf digests of the matrices in `l` (rows of one height).
  constexpr bool bb = std::is_same<F, BabyBear>::value;
  auto hash = [&](const MatList &l, uint64_t height, T *out, const LeafCombine *c, const char *name) -> int {
    if (l.col_start[l.n] > 0 && tensor_takes<F, W>(p, height)) {
      if constexpr (bb)
        return p2t::hash_rows(l, height, out, p, c ? c->apow : nullptr, c ? c->out : nullptr, name, s);
      else
        return p2g::hash_rows<W>(l, height, out, p, name, s);
    }
    if constexpr (bb) {
      if (c) {
        ZKB_LAUNCH(name, s, quad_slab_kernel<<<quad::grid_of(height, thr), thr, 0, s>>>((const uint32_t *)l.ptr[0], l.width[0], 0, l.width[0], height, nullptr, 1, 1, out, p, c->apow, c->out));
        return ZKB_OK;
      }
    }
    ZKB_LAUNCH(name, s, quad::rows_kernel<F, W><<<quad::grid_of(height, thr), thr, 0, s>>>(l, height, out, p));
    return ZKB_OK;
  };
  if (fill) {
    // the caller writes layer 0 (e.g. slab by slab as the matrix arrives)
    ZKB_REQUIRE(nm == 1 && comb == nullptr, "internal: leaves written by the caller take one matrix");
    ZKB_TRY((*fill)(layers));
  } else {
    if (comb) {
      ZKB_REQUIRE(h.field == FIELD_BABYBEAR, "the fused alpha-reduction is BabyBear width 16 only");
      ZKB_REQUIRE(nm == 1, "the fused alpha-reduction takes one matrix");
    }
    ZKB_TRY(hash(ml, max_h, layers, comb, leaf_name));
  }
  ScratchBuf inj_buf;  // digests of rows injected at one layer (sized for the largest)

  size_t next_m = ng;
  // the matrices injected when layer li is compressed
  auto injected = [&](size_t li) {
    const uint64_t next_layer_len = next_pow2_u64(t->layer_len[li] / 2);
    size_t ni = 0;
    while (next_m + ni < nm && next_pow2_u64(mats[ord[next_m + ni]].height) == next_layer_len) ni++;
    return ni;
  };
  const size_t top = t->layer_len.size() - 1;
  for (size_t li = 0; li < top; li++) {
    const uint64_t half = t->layer_len[li] / 2;
    const size_t ni = injected(li);
    const T *prev = layers + t->layer_off[li] * OUT;
    T *next = layers + t->layer_off[li + 1] * OUT;
    const T *inj = nullptr;
    uint64_t inj_h = 0;
    if (ni) {
      MatList iml;
      ZKB_TRY(make_list(next_m, ni, &iml));
      inj_h = mats[ord[next_m]].height;
      if (!inj_buf.p) ZKB_TRY(inj_buf.alloc(inj_h * OUT * sizeof(T), s));
      ZKB_TRY(hash(iml, inj_h, inj_buf.as<T>(), nullptr, "merkle_inject_hash"));
      inj = inj_buf.as<T>();
    }
    next_m += ni;
    if (tensor_takes<F, W>(p, half)) {
      if constexpr (bb)
        ZKB_TRY(p2t::compress(prev, next, half, inj, inj_h, p, comp_name, s));
      else
        ZKB_TRY(p2g::compress<W>(prev, next, half, inj, inj_h, p, comp_name, s));
      continue;
    }
    if (inj) {
      ZKB_LAUNCH(comp_name, s, quad::inject_kernel<F, W><<<quad::grid_of(half, thr), thr, 0, s>>>(prev, next, half, inj, inj_h, p));
      continue;
    }
    // every level up to the next injection, a few launches of whole subtrees
    size_t end = li + 1;
    while (end < top && injected(end) == 0) end++;
    const int levels = quad::run_levels((int)(end - li));
    for (size_t at = li; at < end; at += levels) {
      const int n = (int)std::min<size_t>(levels, end - at);
      quad::Run run{};
      run.layers = layers;
      for (int j = 0; j <= n; j++) {
        run.off[j] = t->layer_off[at + j];
        run.n[j] = j || at > 0 ? t->layer_len[at + j - 1] / 2 : max_h;
      }
      const uint64_t nodes = t->layer_len[at];
      ZKB_LAUNCH(comp_name, s, quad::levels_kernel<F, W><<<(unsigned)((nodes + (1ull << n) - 1) >> n), quad::run_threads(n), quad::run_smem<F, W>(n), s>>>(run, n, p));
    }
    li = end - 1;
  }
  return ZKB_OK;
}

int mmcs_build_dev(const HasherSpec &h, const std::vector<TreeMatrix> &mats, DeviceTree *tree,
                   cudaStream_t s, bool fri_layer, const LeafCombine *comb, const LeafFill *fill) {
  ZKB_REQUIRE(!mats.empty(), "No matrices given");
  if (h.field == FIELD_BABYBEAR && h.width == 16) return build_tree_impl<BabyBear, 16>(h, mats, tree, s, fri_layer, comb, fill);
  if (h.field == FIELD_GOLDILOCKS && h.width == 16) return build_tree_impl<Goldilocks, 16>(h, mats, tree, s, fri_layer, comb, fill);
  if (h.field == FIELD_GOLDILOCKS && h.width == 12) return build_tree_impl<Goldilocks, 12>(h, mats, tree, s, fri_layer, comb, fill);
  set_error("unsupported hasher: field %d width %d", h.field, h.width);
  return ZKB_ERR_UNSUPPORTED;
}

int hash_rows_slab_dev(const HasherSpec &h, const uint32_t *mat, uint64_t stride, uint64_t c0, uint64_t ncols,
                       uint64_t height, uint32_t *carry, bool first, bool last, uint32_t *digests,
                       const LeafCombine *comb, cudaStream_t s) {
  ZKB_REQUIRE(h.field == FIELD_BABYBEAR && h.width == 16, "internal: slab leaf hashing is BabyBear width 16");
  ZKB_REQUIRE(ncols > 0 && c0 % 8 == 0 && (last || ncols % 8 == 0), "internal: slabs hold whole absorbed chunks");
  P2Params<BabyBear, 16> p;
  if (!build_p2_params<BabyBear, 16>(h, &p)) {
    set_error("invalid Poseidon2 parameters");
    return ZKB_ERR_INVALID;
  }
  const uint4 *apow = comb ? comb->apow : nullptr;
  uint4 *out = comb ? comb->out : nullptr;
  if (p2t::takes(p, height))  // by the height alone: every slab of a matrix takes the same form
    return p2t::hash_slab(mat, stride, c0, ncols, height, carry, first, last, digests, p, apow, out, "merkle_leaf_hash", s);
  const unsigned thr = 128;
  ZKB_LAUNCH("merkle_leaf_hash", s, quad_slab_kernel<<<quad::grid_of(height, thr), thr, 0, s>>>(mat, stride, c0, ncols, height, carry, first ? 1 : 0, last ? 1 : 0, digests, p, apow, out));
  return ZKB_OK;
}

int mmcs_root_to_host(const DeviceTree *tree, void *root_out, cudaStream_t s) {
  const size_t es = field_elem_bytes(tree->spec.field);
  const uint64_t off = tree->layer_off.back() * tree->spec.out;
  ZKB_CHECK_CUDA(cudaMemcpyAsync(root_out, (const char *)tree->d_layers + off * es,
                                 tree->spec.out * es, cudaMemcpyDeviceToHost, s));
  ZKB_TRY(wait_stream(s));
  return ZKB_OK;
}

}  // namespace zkb
