// tcgen05.cuh — the tensor-core instructions the hashing kernels use: 8-bit integer products of 128 rows
// (operand A and the s32 accumulators in TMEM, operand B in shared memory), TMEM loads and
// stores, bounded mbarrier waits.
#pragma once
#include <cstdint>

#include "common.cuh"

namespace zkb {
namespace tc {

#ifdef __CUDACC__
// s32 accumulators, u8 x u8, both operands K-major, M = 128.
__device__ __forceinline__ constexpr uint32_t idesc(int N) {
  return (2u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
// Shared-memory operand without swizzle: 8 x 16-byte core matrices, 128 bytes apart along N and
// (N / 8) * 128 bytes apart along K.
__device__ __forceinline__ uint64_t bdesc(uint32_t addr, int N) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((N / 8) * 128 / 16) << 16) | ((uint64_t)(128 / 16) << 32) |
         (1ull << 46);
}
// Issued by a whole warp with warp-uniform operands; `one` is set in a single lane.
__device__ __forceinline__ void mma(uint32_t d, uint32_t a, uint64_t b, uint32_t id, bool acc, uint32_t one) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\tsetp.ne.u32 p, %4, 0;\n\tsetp.ne.u32 e, %5, 0;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
      "r"(a), "l"(b), "r"(id), "r"((uint32_t)acc), "r"(one)
      : "memory");
}
__device__ __forceinline__ void st8(uint32_t a, const uint32_t *v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(a), "r"(v[0]), "r"(v[1]),
               "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
__device__ __forceinline__ void st4(uint32_t a, const uint32_t *v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(v[0]), "r"(v[1]), "r"(v[2]),
               "r"(v[3])
               : "memory");
}
__device__ __forceinline__ void st2(uint32_t a, uint32_t v, uint32_t w) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1,%2};" ::"r"(a), "r"(v), "r"(w) : "memory");
}
__device__ __forceinline__ void st1(uint32_t a, uint32_t v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void ld16(uint32_t (&v)[16], uint32_t a) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(a)
      : "memory");
}
// The low 16 bits of 32 columns, two adjacent columns to a register.
__device__ __forceinline__ void ld16_pack(uint32_t (&v)[16], uint32_t a) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.pack::16b.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(a)
      : "memory");
}
// Waits for the loads; the registers pass through so that no use moves above the wait.
__device__ __forceinline__ void ld_wait(uint32_t (&v)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                 "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15])::"memory");
}

// Waits for a phase of the mbarrier; false when `polls` polls have run out.
__device__ __forceinline__ bool wait_parity(uint32_t mbar, uint32_t parity, uint32_t polls) {
  uint32_t done = 0;
  for (uint32_t n = 0; n < polls && !done; n++) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(mbar), "r"(parity)
        : "memory");
  }
  return done != 0;
}

// A part of a table, copied by one untiled bulk copy of this GPU's own memory.
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void *src, int bytes, uint32_t mbar) {
  asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(__cvta_generic_to_global(src)), "r"((uint32_t)bytes), "r"(mbar)
               : "memory");
}
__device__ __forceinline__ void expect_bytes(uint32_t mbar, int bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"((uint32_t)bytes) : "memory");
}
__device__ __forceinline__ void init_barrier(uint32_t mbar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// One warp: `cols` (a power of two) columns, the address written to shared memory at `slot`.
__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t addr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Four warps (128 rows) that share a product per layer.
struct Group {
  uint32_t sm;      // shared address of the tables
  uint32_t tm;      // TMEM address of the group's columns
  uint32_t tw;      // the same with this warp's lane base (ld / st)
  uint32_t mbar;    // shared address of the group's mbarrier
  uint32_t phase;
  int bar;          // named barrier of the group
  bool lead;        // this is the warp that issues the products (warp-uniform)
  uint32_t one;     // set in one lane of it
  uint32_t polls;   // limit of a wait (0 once one has run out)
  uint32_t *err;    // DeviceContext::wait_word
};

// D columns += (or =) A columns x the K step of 32 bytes at shared offset `off` (N rows of a matrix
// laid out for L rows).
__device__ __forceinline__ void mma_slab(const Group &g, int d_col, int a_col, int off, int N, bool acc, int L = 0) {
  mma(g.tm + d_col, g.tm + a_col, bdesc(g.sm + off, L ? L : N), idesc(N), acc, g.one);
}
// Before the products: this thread's operand stores are complete and its accumulator loads done.
__device__ __forceinline__ void arrive(const Group &g) {
  st_wait();
  fence_before();
  asm volatile("bar.sync %0, 128;" ::"r"(g.bar) : "memory");
  if (g.lead) fence_after();
}
// The products issued so far by the lane that has `one` set arrive on mbar when they are done.
__device__ __forceinline__ void commit(uint32_t mbar, uint32_t one) {
  asm volatile(
      "{\n\t.reg .pred e;\n\tsetp.ne.u32 e, %1, 0;\n\t"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(mbar),
      "r"(one)
      : "memory");
}
// After the lead warp has issued the products: everyone waits for them (bounded: a thread whose wait runs
// out goes on without waiting, so every block ends, and reports it there, see drain: the report at every wait
// made the hashing kernels 1 to 4 % longer, as a call 3 % that of column slabs).
__device__ __forceinline__ void finish(Group &g) {
  if (g.lead) commit(g.mbar, g.one);
  if (!wait_parity(g.mbar, g.phase, g.polls)) g.polls = 0;
  g.phase ^= 1;
  fence_after();
}
// Before the block gives its TMEM and shared memory back: a thread whose wait gave up reports it, and as products
// may still be under way then, the lane that issued them waits for all of them on an mbarrier of its own
// (bounded), in the first words of the tables, which nothing correct needs any more.
__device__ __forceinline__ void drain(const Group &g, uint32_t polls = WAIT_POLLS) {
  if (g.polls) return;
  report_wait(g.err);
  if (!g.one) return;
  const uint32_t mbar = g.sm + 8 * (g.bar - 1);
  init_barrier(mbar);
  init_fence();
  commit(mbar, 1);
  wait_parity(mbar, 0, polls);
}
// The tables' copies (on the mbarrier `tables`) have landed; or they have not within the limit, and the
// block reports that, waits once more, frees its TMEM (address at `slot`) and ends.  Every thread calls it.
__device__ __forceinline__ void tables_or_exit(uint32_t tables, const uint8_t *slot, uint32_t cols, uint32_t *err,
                                               uint32_t polls = WAIT_POLLS) {
  if (__syncthreads_and(wait_parity(tables, 0, polls))) return;
  if (threadIdx.x == 0) report_wait(err);
  wait_parity(tables, 0, polls);
  __syncthreads();
  if (threadIdx.x < 32) tmem_free(*reinterpret_cast<const volatile uint32_t *>(slot), cols);
  asm volatile("exit;");
}
// This thread's group: `cols` TMEM columns each from the address at sm + slot on, mbarriers at
// `mbars`, tables at `sm`.
__device__ __forceinline__ Group make_group(const uint8_t *sm, int slot, uint32_t mbars, int cols, uint32_t *err) {
  // warp-uniform by construction; the shuffles let the compiler keep them in uniform registers
  const int warp = __shfl_sync(0xFFFFFFFFu, (int)threadIdx.x / 32, 0), gi = warp / 4;
  Group g;
  g.sm = (uint32_t)__cvta_generic_to_shared(sm);
  g.tm = __shfl_sync(0xFFFFFFFFu, *reinterpret_cast<const volatile uint32_t *>(sm + slot), 0) + gi * cols;
  g.tw = g.tm + ((warp % 4) << 21);
  g.mbar = mbars + 8 * gi;
  g.phase = 0;
  g.bar = 1 + gi;
  g.lead = warp % 4 == 0;
  g.one = threadIdx.x % 128 == 0;
  g.polls = WAIT_POLLS;
  g.err = err;
  return g;
}
#endif  // __CUDACC__

}  // namespace tc
}  // namespace zkb
