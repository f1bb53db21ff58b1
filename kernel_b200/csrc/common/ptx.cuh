// Thin inline-PTX layer for sm_100a: mbarrier, TMA (non-multicast only),
// tcgen05 (TMEM alloc / MMA / commit / ld), system-scope flag traffic for
// peer GPUs, and time-bounded waits.
//
// Every wait in this file gives up after a deadline and reports failure to its
// caller; nothing here spins forever and nothing traps.
#pragma once
#include <cstdint>
#include <cuda_bf16.h>

namespace kb {

// ---------------------------------------------------------------- misc ----
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ uint32_t lane_id() {
  uint32_t l;
  asm volatile("mov.u32 %0, %%laneid;" : "=r"(l));
  return l;
}

// ------------------------------------------------------------ mbarrier ----
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// try_wait with a suspend-time hint: the thread may stay suspended for up to
// `hint_ns` before the instruction returns false; the phase's completion wakes it.
__device__ __forceinline__ bool mbar_try_wait_hint(uint64_t* bar, uint32_t parity, uint32_t hint_ns) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(hint_ns)
      : "memory");
  return ok != 0;
}
// Waits until the barrier's phase with the given parity has completed, or until
// `limit_ns` has elapsed.  Returns false on expiry (caller must unwind).
// `hint_ns` > 0: a role that can afford it (an epilogue warp waiting for a whole
// tile, a producer waiting for a stage) lets the hardware suspend it between polls
// instead of issuing a poll every few cycles; the issue slots and the energy of a
// persistent kernel's idle roles are not free under a power cap.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, uint64_t limit_ns, uint32_t hint_ns = 0) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  uint32_t spins = 0;
  while (!(hint_ns ? mbar_try_wait_hint(bar, parity, hint_ns) : mbar_try_wait(bar, parity))) {
    if ((++spins & (hint_ns ? 0xfu : 0x3ffu)) == 0 && globaltimer_ns() - t0 > limit_ns) return false;
  }
  return true;
}

// Cluster-scope acquire form of the bounded wait: for a barrier whose arrival
// orders ordinary stores that a thread of ANOTHER CTA of the cluster made to this
// CTA's shared memory (st.shared::cluster + mbarrier.arrive.release.cluster).
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_bounded_cluster(uint64_t* bar, uint32_t parity, uint64_t limit_ns) {
  if (mbar_try_wait_cluster(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  uint32_t spins = 0;
  while (!mbar_try_wait_cluster(bar, parity)) {
    if ((++spins & 0x3ffu) == 0 && globaltimer_ns() - t0 > limit_ns) return false;
  }
  return true;
}
// 32-bit store into the shared memory of another CTA of the cluster (address from map_to_cta).
__device__ __forceinline__ void st_shared_cluster_u32(uint32_t cluster_addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}

// 16-byte accesses to this CTA's shared memory by address (a pointer that went through
// integer arithmetic has lost its address space and would be accessed generically).
__device__ __forceinline__ float4 ld_shared_v4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void st_shared_cluster_v4(uint32_t cluster_addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// ----------------------------------------------------------------- TMA ----
// 2-D tiled load global -> shared of one box, completion on an mbarrier.
// Plain (single-CTA) form only.  x is the innermost coordinate and must keep
// x * elem_size a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const void* tmap, uint64_t* bar, int32_t x, int32_t y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(tmap), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
// 3-D form (innermost coordinate x, then y, z), called by a converged warp: one elected
// lane issues.  kPair: the completion is counted on the mbarrier at cluster address
// `bar` (the leader of a CTA pair); otherwise `bar` is the shared-memory address of one
// of this CTA's own barriers.
template <bool kPair>
__device__ __forceinline__ void tma_load_3d_warp(uint32_t smem_dst, const void* tmap, uint32_t bar, int32_t x, int32_t y, int32_t z) {
  if constexpr (kPair) {
    asm volatile(
        "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
        "@q cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n\t}"
        ::"r"(smem_dst), "l"(tmap), "r"(bar), "r"(x), "r"(y), "r"(z)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
        "@q cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n\t}"
        ::"r"(smem_dst), "l"(tmap), "r"(bar), "r"(x), "r"(y), "r"(z)
        : "memory");
  }
}
template <bool kPair>
__device__ __forceinline__ void tma_load_4d_warp(uint32_t smem_dst, const void* tmap, uint32_t bar, int32_t x, int32_t y, int32_t z, int32_t w) {
  if constexpr (kPair) {
    asm volatile(
        "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
        "@q cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];\n\t}"
        ::"r"(smem_dst), "l"(tmap), "r"(bar), "r"(x), "r"(y), "r"(z), "r"(w)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
        "@q cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];\n\t}"
        ::"r"(smem_dst), "l"(tmap), "r"(bar), "r"(x), "r"(y), "r"(z), "r"(w)
        : "memory");
  }
}
// Two boxes of a 3-D map, at rows y0 and y1, for one election.
template <bool kPair>
__device__ __forceinline__ void tma_load_3d_two_warp(uint32_t dst0, uint32_t dst1, const void* tmap, uint32_t bar, int32_t x, int32_t y0, int32_t y1, int32_t z) {
#define KB_LOAD_TWO(GROUP)                                                                                                           \
  asm volatile(                                                                                                                      \
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"                                                                       \
      "@q cp.async.bulk.tensor.3d" GROUP ".shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%2, {%4, %5, %7}], [%3];\n\t"    \
      "@q cp.async.bulk.tensor.3d" GROUP ".shared::cluster.global.mbarrier::complete_tx::bytes [%1], [%2, {%4, %6, %7}], [%3];\n\t}"   \
      ::"r"(dst0), "r"(dst1), "l"(tmap), "r"(bar), "r"(x), "r"(y0), "r"(y1), "r"(z)                                                  \
      : "memory")
  if constexpr (kPair) KB_LOAD_TWO(".cta_group::2");
  else KB_LOAD_TWO("");
#undef KB_LOAD_TWO
}
// The expected bytes (0: this CTA expects none) and one box of a 4-D map, issued by one elected lane.
template <bool kPair>
__device__ __forceinline__ void tma_load_4d_expect_warp(uint32_t own_bar, uint32_t tx_bytes, uint32_t bar, uint32_t dst, const void* map, int32_t x,
                                                        int32_t y, int32_t z, int32_t w) {
#define KB_LOAD_EXPECT(GROUP)                                                                                                          \
  asm volatile(                                                                                                                        \
      "{\n\t.reg .pred q, e;\n\telect.sync _|q, 0xffffffff;\n\t"                                                                       \
      "setp.ne.and.u32 e, %1, 0, q;\n\t"                                                                                               \
      "@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t"                                                                  \
      "@q cp.async.bulk.tensor.4d" GROUP ".shared::cluster.global.mbarrier::complete_tx::bytes [%3], [%4, {%5, %6, %7, %8}], [%2];\n\t}" \
      ::"r"(own_bar), "r"(tx_bytes), "r"(bar), "r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(w)                                      \
      : "memory")
  if constexpr (kPair) KB_LOAD_EXPECT(".cta_group::2");
  else KB_LOAD_EXPECT("");
#undef KB_LOAD_EXPECT
}
__device__ __forceinline__ void mbar_expect_tx_warp(uint32_t bar, uint32_t bytes) {
  asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
               "@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}" ::"r"(bar), "r"(bytes) : "memory");
}
// The expected bytes (0: this CTA expects none) and one box, issued by one elected lane.
template <bool kPair>
__device__ __forceinline__ void tma_load_expect_warp(uint32_t own_bar, uint32_t tx_bytes, uint32_t bar, uint32_t dst, const void* map, int32_t x,
                                                     int32_t y, int32_t z) {
#define KB_LOAD_EXPECT(GROUP)                                                                                                      \
  asm volatile(                                                                                                                    \
      "{\n\t.reg .pred q, e;\n\telect.sync _|q, 0xffffffff;\n\t"                                                                   \
      "setp.ne.and.u32 e, %1, 0, q;\n\t"                                                                                           \
      "@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t"                                                              \
      "@q cp.async.bulk.tensor.3d" GROUP ".shared::cluster.global.mbarrier::complete_tx::bytes [%3], [%4, {%5, %6, %7}], [%2];\n\t}" \
      ::"r"(own_bar), "r"(tx_bytes), "r"(bar), "r"(dst), "l"(map), "r"(x), "r"(y), "r"(z)                                          \
      : "memory")
  if constexpr (kPair) KB_LOAD_EXPECT(".cta_group::2");
  else KB_LOAD_EXPECT("");
#undef KB_LOAD_EXPECT
}
// One stage of a GEMM: the expected bytes (0: this CTA expects none) and the boxes of both
// operands, issued by one elected lane.  One election instead of three: the issuing
// warp is what bounds narrow tiles.
template <bool kPair>
__device__ __forceinline__ void tma_load_ab_warp(uint32_t own_bar, uint32_t tx_bytes, uint32_t bar, uint32_t a_dst, const void* a_map, int32_t ax,
                                                 int32_t ay, int32_t az, uint32_t b_dst, const void* b_map, int32_t bx, int32_t by, int32_t bz) {
#define KB_LOAD_AB(GROUP)                                                                                                          \
  asm volatile(                                                                                                                    \
      "{\n\t.reg .pred q, e;\n\telect.sync _|q, 0xffffffff;\n\t"                                                                   \
      "setp.ne.and.u32 e, %1, 0, q;\n\t"                                                                                           \
      "@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t"                                                              \
      "@q cp.async.bulk.tensor.3d" GROUP ".shared::cluster.global.mbarrier::complete_tx::bytes [%3], [%4, {%5, %6, %7}], [%2];\n\t"    \
      "@q cp.async.bulk.tensor.3d" GROUP ".shared::cluster.global.mbarrier::complete_tx::bytes [%8], [%9, {%10, %11, %12}], [%2];\n\t}" \
      ::"r"(own_bar), "r"(tx_bytes), "r"(bar), "r"(a_dst), "l"(a_map), "r"(ax), "r"(ay), "r"(az), "r"(b_dst), "l"(b_map), "r"(bx), \
      "r"(by), "r"(bz)                                                                                                             \
      : "memory")
  if constexpr (kPair) KB_LOAD_AB(".cta_group::2");
  else KB_LOAD_AB("");
#undef KB_LOAD_AB
}
__device__ __forceinline__ void tma_prefetch_desc(const void* tmap) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(tmap) : "memory");
}
// Generic-proxy writes (plain stores, also those that arrived from a peer GPU)
// must be fenced before the async proxy (TMA) reads the same bytes.
__device__ __forceinline__ void fence_proxy_async_global() {
  asm volatile("fence.proxy.async.global;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// 2-D tiled store shared -> global of one box (bulk async group of the issuing
// thread).  Rows and columns of the box that fall outside the tensor are not
// written.  x * elem_size must be a multiple of 16 bytes.
__device__ __forceinline__ void tma_store_2d(const void* tmap, const void* smem_src, int32_t x, int32_t y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(tmap),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tma_store_3d(const void* tmap, const void* smem_src, int32_t x, int32_t y, int32_t z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(tmap),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z)
               : "memory");
}
// Untiled bulk copies (the same engine as TMA, no tensor map): both addresses
// 16-byte aligned, size a multiple of 16 bytes.  The load completes on an
// mbarrier of this CTA; the store belongs to the issuing thread's bulk group.
// Never multicast: one CTA, one destination.
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* gmem_src, int bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(smem_dst)),
               "l"(gmem_src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void bulk_store(void* gmem_dst, const void* smem_src, int bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(gmem_dst), "r"(smem_u32(smem_src)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_commit_group() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// Waits until at most N of this thread's bulk groups still read their source.
template <int N>
__device__ __forceinline__ void bulk_wait_group_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
// Waits until at most N of this thread's bulk groups are incomplete.
template <int N>
__device__ __forceinline__ void bulk_wait_group() {
  asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}

// ------------------------------------------------------------- tcgen05 ----
// TMEM allocation: whole warp, `ncols` a power of two in [32, 512].
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before_sync() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after_sync() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// D[tmem] (+)= A[smem] * B[smem], bf16/f16 inputs, fp32 accumulate, one CTA.
__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive (count 1) on a CTA-local mbarrier once all MMAs issued so far by this
// thread have finished.  Single-CTA form; implies fence::before_thread_sync.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
// 32 lanes x 32 consecutive fp32 columns: thread i of the warp receives lane
// (32 * (warp_id % 4) + i), registers run along columns.
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_32x8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// ------------------------------------------------ CTA pairs (cta_group::2) ----
// Two CTAs of a cluster share one 256-row MMA: each holds its 128 rows of A, its
// half of B and its 128 accumulator rows; the even CTA (the leader) issues.
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// Address of the same shared-memory location in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Without memory ordering: for arrivals that only say that tensor memory has been read (the values are in registers by then).  A
// release at cluster scope waits until the thread's earlier stores have been performed, 2000 cycles behind an epilogue's.
__device__ __forceinline__ void mbar_arrive_cluster_relaxed(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Each CTA of the pair loads its own box into its own shared memory; the bytes
// are counted on the LEADER's mbarrier (`leader_bar` is a cluster address).
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const void* tmap, uint32_t leader_bar, int32_t x,
                                                 int32_t y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(tmap), "r"(leader_bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                              uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on ONE mbarrier (given by its cluster address, in either CTA of the
// pair) once all MMAs issued so far have finished in both CTAs.
__device__ __forceinline__ void umma_commit_pair(uint32_t cluster_bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(cluster_bar)
               : "memory");
}

// Warp-converged forms: every lane of the warp calls them with the same arguments and
// one elected lane issues.  With the loop around them free of divergence the compiler
// keeps addresses and descriptors in uniform registers, where tcgen05 wants its
// operands; issued from inside an `if (lane == 0)` the same instructions cost a move
// per operand register, which made the issuing thread the bottleneck of the mainloop
// (640 instead of 512 cycles per 64-wide k block of a 256 x 256 pair tile).
//
// Four consecutive K steps (64 elements) of D (+)= A * B; the descriptors advance by
// `a_step` / `b_step` 16-byte units per step.
template <bool kPair>
__device__ __forceinline__ void umma_f16_x4(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                            uint32_t a_step, uint32_t b_step, uint32_t idesc, uint32_t accumulate) {
#define KB_UMMA_X4(GROUP)                                                                                          \
  asm volatile(                                                                                                    \
      "{\n\t.reg .pred q, p;\n\t.reg .b32 al, bl;\n\t.reg .b64 da, db;\n\t"                                             \
      "elect.sync _|q, 0xffffffff;\n\t"                                                                            \
      "setp.ne.b32 p, %8, 0;\n\t"                                                                                  \
      "mov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %4};\n\t"                                                        \
      "@q tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], da, db, %7, p;\n\t"                                     \
      "add.u32 al, %1, %5;\n\tadd.u32 bl, %3, %6;\n\tmov.b64 da, {al, %2};\n\tmov.b64 db, {bl, %4};\n\t"        \
      "@q tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], da, db, %7, 1;\n\t"                                     \
      "add.u32 al, al, %5;\n\tadd.u32 bl, bl, %6;\n\tmov.b64 da, {al, %2};\n\tmov.b64 db, {bl, %4};\n\t"        \
      "@q tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], da, db, %7, 1;\n\t"                                     \
      "add.u32 al, al, %5;\n\tadd.u32 bl, bl, %6;\n\tmov.b64 da, {al, %2};\n\tmov.b64 db, {bl, %4};\n\t"        \
      "@q tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], da, db, %7, 1;\n\t}"                                    \
      ::"r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(a_step), "r"(b_step), "r"(idesc), "r"(accumulate) \
      : "memory")
  if constexpr (kPair) KB_UMMA_X4("2");
  else KB_UMMA_X4("1");
#undef KB_UMMA_X4
}
// Commit of the elected lane; `bar`: shared-memory address (cluster address for a pair).
template <bool kPair>
__device__ __forceinline__ void umma_commit_warp(uint32_t bar) {
  if constexpr (kPair) {
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
                 "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar) : "memory");
  } else {
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
                 "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar) : "memory");
  }
}

// Shared-memory operand descriptor for a K-major bf16 tile stored as rows of
// 128 bytes (64 elements) with the 128-byte swizzle TMA produces; 8-row groups
// are 1024 bytes apart.  `addr` is the 1024-byte aligned tile base plus
// 32 bytes per 16-element K step.
__device__ __forceinline__ uint64_t umma_desc_k_sw128(uint32_t addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((addr & 0x3ffffu) >> 4);   // start address, 16-byte units
  d |= static_cast<uint64_t>(1) << 16;                  // leading byte offset (unused with swizzle)
  d |= static_cast<uint64_t>(1024 >> 4) << 32;          // stride byte offset between 8-row groups
  d |= static_cast<uint64_t>(1) << 46;                  // descriptor version for sm_100
  d |= static_cast<uint64_t>(2) << 61;                  // 128-byte swizzle
  return d;
}
// Instruction descriptor: bf16 x bf16 -> fp32, both operands K-major, M x N tile.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(uint32_t m, uint32_t n) {
  return (1u << 4)            // D format fp32
         | (1u << 7)          // A format bf16
         | (1u << 10)         // B format bf16
         | ((n >> 3) << 17)   // N / 8
         | ((m >> 4) << 24);  // M / 16
}

// ------------------------------------------------- system-scope traffic ----
__device__ __forceinline__ void st_release_sys_u32(uint32_t* p, uint32_t v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_acquire_sys_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_relaxed_sys_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void fence_sys() { asm volatile("fence.acq_rel.sys;" ::: "memory"); }
// Plain system-scope store for a flag whose ordering is provided by a
// fence_sys() the same thread executed just before (fence + relaxed store is a
// release pattern; st.release would pay for a second fence).
__device__ __forceinline__ void st_relaxed_sys_u32(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// 16-byte loads that never use the non-coherent path (data may have been
// written by a peer GPU during this kernel).
__device__ __forceinline__ uint4 ld_sys_v4(const void* p) {
  uint4 v;
  asm volatile("ld.relaxed.sys.global.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p)
               : "memory");
  return v;
}
__device__ __forceinline__ void st_sys_v4(void* p, const uint4& v) {
  asm volatile("st.relaxed.sys.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z),
               "r"(v.w)
               : "memory");
}
// ------------------------------------------------- NVLS (multimem) traffic ----
// `mc` is an address inside the multicast mapping of the symmetric heap: a store
// lands at the same offset of every rank's segment, a ld_reduce returns the sum
// of the values at that offset of every rank's segment, added in the switch.
__device__ __forceinline__ void multimem_st_v4(void* mc, const uint4& v) {
  asm volatile("multimem.st.relaxed.sys.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(mc), "r"(v.x), "r"(v.y), "r"(v.z),
               "r"(v.w)
               : "memory");
}
// Eight bf16 values per call, accumulated in fp32 inside the switch, returned as bf16 pairs.
__device__ __forceinline__ uint4 multimem_ld_reduce_bf16x8(const void* mc) {
  uint4 v;
  asm volatile("multimem.ld_reduce.relaxed.sys.global.add.acc::f32.v4.bf16x2 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(mc)
               : "memory");
  return v;
}

// 32 bytes per thread (a whole L2 sector); the address is a multiple of 32.
__device__ __forceinline__ void st_global_v8(void* p, const uint4& a, const uint4& b) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w),
               "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
               : "memory");
}

// 32 bytes per thread; the address is a multiple of 32.
__device__ __forceinline__ void ld_stream_v8(const void* p, uint4& a, uint4& b) {
  asm volatile("ld.global.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
               : "l"(p));
}

// Streaming read of data that is read-only for the whole kernel.
__device__ __forceinline__ uint4 ld_nc_v4(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

// The same without the non-coherent path, for kernels that begin before the previous kernel of the
// stream has ended: what that one wrote is not read-only for the whole of this one, which
// is what ld.global.nc (__ldg) asks for.  Volatile: stays behind wait_for_previous_launch().
__device__ __forceinline__ uint4 ld_stream_v4(const void* p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 ld_stream_v2(const void* p) {
  uint2 v;
  asm volatile("ld.global.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ uint4 ld_global_v4(const void* p) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// Start of a kernel launched with the overlap_launch attribute: waits until the previous
// kernel of the stream has ended and its writes are visible, then lets the next one be set up.
// Nothing that the previous kernel may write, and no output, is touched before it.  What was written before
// that kernel began may be read earlier if that kernel passes its own wait before it lets this one start, as all kernels that call
// this do (`early` in gemm_swap.cuh).  Without the attribute the wait returns at once.
__device__ __forceinline__ void wait_for_previous_launch() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Brings `bytes` (a multiple of 16, 16-byte aligned) into the L2.
__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
// Loads 16 bytes and drops them: the line is in L1 afterwards.
__device__ __forceinline__ void touch_global(const void* p) {
  asm volatile("{\n\t.reg .b32 a, b, c, d;\n\tld.global.v4.u32 {a, b, c, d}, [%0];\n\t}" ::"l"(p));
}

// Device-scope counterparts for words that only threads of this GPU touch.
__device__ __forceinline__ void st_release_gpu_u32(uint32_t* p, uint32_t v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_relaxed_gpu_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// Spin on a 32-bit flag until it reaches `want` (flags only grow).  Returns
// false if `limit_ns` passes first.
//
// Polls with relaxed loads and pays for one acquire fence once the flag is
// there.  The pause between polls doubles up to `max_pause_ns`: where many
// CTAs poll words of the same cache line an unthrottled spin takes L2 bandwidth
// away from the very stores it is waiting for.  A single poller of a line passes
// 0 and spins without pausing (a pause costs about a microsecond of reaction
// time).  `sys` false: the word is written by this GPU only, device scope is
// enough for the polls and the fence.  `acquire_loads`: poll with ld.acquire.sys
// and skip the fence; for a lone poller that is cheaper than relaxed polls plus
// fence.acq_rel.sys, which also waits for the acknowledgements of every store this
// GPU has in flight to its peers (several microseconds on an NVSwitch system).
__device__ __forceinline__ bool wait_flag_ge(const uint32_t* flag, uint32_t want, uint64_t limit_ns,
                                             uint32_t max_pause_ns = 512, bool sys = true, bool acquire_loads = false) {
  auto poll = [&]() -> bool {
    const uint32_t v = !sys ? ld_relaxed_gpu_u32(flag) : (acquire_loads ? ld_acquire_sys_u32(flag) : ld_relaxed_sys_u32(flag));
    return static_cast<int32_t>(v - want) >= 0;
  };
  auto acquire = [&]() {
    if (!sys) fence_gpu();
    else if (!acquire_loads) fence_sys();
  };
  if (poll()) {
    acquire();
    return true;
  }
  const uint64_t t0 = globaltimer_ns();
  uint32_t spins = 0;
  uint32_t pause = 32;
  for (;;) {
    if (max_pause_ns != 0) {
      __nanosleep(pause);
      if (pause < max_pause_ns) pause *= 2;
    }
    if (poll()) {
      acquire();
      return true;
    }
    if ((++spins & 0x3fu) == 0 && globaltimer_ns() - t0 > limit_ns) return false;
  }
}

// ---------------------------------------------------------- conversions ----
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack_bf16x2(uint32_t u) {
  __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&u);
  return __bfloat1622float2(v);
}

}  // namespace kb
