// Thin inline-PTX wrappers for the sm_100a features the weight-only GEMM uses:
// mbarrier, TMA (cp.async.bulk.tensor, never multicast), tcgen05 (TMEM alloc,
// st/ld, MMA, commit, fences).  Every wait is bounded: a wait that runs out
// returns false so the caller can record an error code and leave the kernel
// with its TMEM freed, instead of hanging the GPU.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "tile_counter.h"

namespace dx {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(pred));
  return pred != 0;
}

// ---------------------------------------------------------------- mbarrier --
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Same test, but the hardware may park the thread for up to `hint_ns` until the
// phase completes, instead of returning at once: a waiting warp then costs no
// issue slots and is woken by the barrier itself.  (Loops of the plain form and of
// mbarrier.test_wait were measured as well: the same or slightly slower.)
__device__ __forceinline__ bool mbar_try_wait_parked(uint32_t bar, uint32_t parity,
                                                     uint32_t hint_ns) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(hint_ns)
      : "memory");
  return ok != 0;
}

// Upper bound of one wait: kWaitTries parked attempts of kWaitHintNs each (about
// one second in all, whatever the clock).
constexpr uint32_t kWaitHintNs = 1000000u;
constexpr uint32_t kWaitTries = 1000u;

// Bounded wait on an mbarrier phase.  `abort_flag` is a CTA-shared word: once
// any role gives up it is set, and every other wait in the CTA returns false
// at its next poll so the whole CTA drains to its tear-down.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_try_wait(bar, parity)) return true;
  for (uint32_t tries = 0; tries < kWaitTries; ++tries) {
    if (mbar_try_wait_parked(bar, parity, kWaitHintNs)) return true;
    if (*abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}
// The same for all lanes of a warp, which get one answer: what follows a wait are warp-wide instructions
// (tcgen05.ld / st, __syncwarp), and lanes that saw the abort flag while others saw the phase complete would
// leave the rest of their warp waiting for them without a limit.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}

// --------------------------------------------------------------------- TMA --
__device__ __forceinline__ void tma_prefetch_desc(const void* tmap) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(tmap)) : "memory");
}
// 2-D tiled load, global -> this CTA's shared memory, completion on `bar`.
// x is the innermost coordinate; x * element size must be a multiple of 16 B.
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const void* tmap, uint32_t bar, int x,
                                            int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
// The same with an L2 eviction priority: one of the words that createpolicy.fractional yields on this architecture, which
// tests/test_gpu_l2_policy.py compares with what it gives on the device.  They are kept here and travel as a kernel
// parameter because the load wants its policy in a uniform register, where a parameter already is; made
// by createpolicy in the kernel, 8 tokens 3072 x 9216 take 7.37 us instead of 7.24.
constexpr uint64_t kL2EvictFirst = 0x12F0000000000000ull;      // L2::evict_first, all lines
constexpr uint64_t kL2EvictFirstHalf = 0x1270000000000000ull;  // L2::evict_first, half of them
constexpr uint64_t kL2EvictNormal = 0x16F0000000000000ull;     // L2::evict_normal
__device__ __forceinline__ void tma_load_2d_policy(uint32_t dst, const void* tmap, uint32_t bar, int x, int y,
                                                   uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4}], [%2], %5;"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar), "r"(x), "r"(y), "l"(policy)
      : "memory");
}
// 3-D tiled load (x innermost).
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const void* tmap, uint32_t bar, int x,
                                            int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}
// -------------------------------------------------- flags in global memory --
__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
// Bounded wait (one calling thread) until all sums of a tile are parked.  Gives up after about a second
// or as soon as another role of the CTA has given up, setting the CTA's abort flag.
constexpr uint32_t kFlagTries = 4000000u;
__device__ __forceinline__ bool wait_tile_parked(const int* counter, int sharers, volatile int* abort_flag) {
  for (uint32_t tries = 0; tries < kFlagTries; ++tries) {
    if (tile_all_parked(static_cast<unsigned>(ld_acquire_gpu(counter)), sharers)) return true;
    if (*abort_flag) return false;
    __nanosleep(tries < 64 ? 32 : 256);
  }
  *abort_flag = 1;
  return false;
}
// One thread, after its CTA's sums are out (or once it has given up).
__device__ __forceinline__ void tile_leave(int* counter, int sharers, bool parked) {
  const unsigned before = atomicAdd(reinterpret_cast<unsigned*>(counter), tile_leave_add(parked));
  if (tile_all_left(before, sharers)) *counter = 0;
}

// ------------------------------------------- programmatic dependent launch --
// A kernel launched with programmatic stream serialisation may start while the kernel
// before it in the stream is still running.  `pdl_wait` blocks until that kernel has
// finished and its writes are visible; `pdl_launch_dependents` lets the NEXT kernel in
// the stream start early.  Both are no-ops for ordinary launches.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ------------------------------------------------- thread-block clusters --
// Address of the same shared-memory location in CTA `rank` of this cluster.
__device__ __forceinline__ uint32_t dsmem_addr(uint32_t local_addr, uint32_t rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local_addr), "r"(rank));
  return remote;
}
__device__ __forceinline__ void st_dsmem_b32x4(uint32_t cluster_addr, uint32_t a, uint32_t b,
                                               uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_addr), "r"(a),
               "r"(b), "r"(c), "r"(d)
               : "memory");
}
__device__ __forceinline__ float4 ld_smem_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}
// Rank of this CTA in its cluster and index of the cluster in the grid (x), read from the
// special registers: no division by the cluster size.
__device__ __forceinline__ uint32_t cluster_cta_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_id_x() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
  return r;
}
// Hardware barrier over every thread of the cluster; release/acquire at cluster scope,
// so shared-memory writes made before it are visible to peer CTAs after it.
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Its two halves: arrive without ordering memory (only "this CTA has started"), and wait.
__device__ __forceinline__ void cluster_arrive_relaxed() {
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// ----------------------------------------------------------------- tcgen05 --
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// Arrive once on `bar` when every tcgen05.mma issued so far by this thread is done.
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   bar)
               : "memory");
}

// ---- CTA pairs (cta_group::2): two CTAs of a cluster work on one M = 256 tile.  TMEM is allocated by one
// warp of each; the leader (rank 0) issues the MMAs for both, which read A and write D in each CTA's own
// TMEM (rows 0-127 / 128-255) and take half of B's rows from each CTA's shared memory.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// Arrive once on `bar` of BOTH CTAs when every pair MMA issued so far by this thread is done.
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
      "h"(static_cast<uint16_t>(3))
      : "memory");
}
__device__ __forceinline__ void mma_ts_pair(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 b;\n\t"
      "setp.ne.b32 p, %5, 0;\n\tmov.b64 b, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], b, %4, p;\n\t}\n"
      ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Across the pair, at cluster scope.  An arrival announces what its warp has read from or written to TMEM, which
// tcgen05.wait and tcgen05.fence::before_thread_sync / after_thread_sync order around it, so it is relaxed: it
// makes no shared or global memory visible.  (Activations do not pass through a thread: their copies complete
// on the leader's barrier themselves, see tma_load_3d_pair.)  So are waits for a commit of the leader's; the
// leader's own waits, which also stand for those copies, acquire.  (Arrivals that release as well: 913 x 13824 x
// 5120 147 us instead of 98.)
__device__ __forceinline__ void mbar_arrive_pair(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
template <bool ACQUIRE>
__device__ __forceinline__ bool mbar_try_wait_pair(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  if (ACQUIRE)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(kWaitHintNs)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.relaxed.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(kWaitHintNs)
        : "memory");
  return ok != 0;
}
template <bool ACQUIRE>
__device__ __forceinline__ bool mbar_wait_pair(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  for (uint32_t tries = 0; tries < kWaitTries; ++tries) {
    if (mbar_try_wait_pair<ACQUIRE>(bar, parity)) return true;
    if (*abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}
// Loads into this CTA's shared memory that complete on a barrier of either CTA of the pair.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const void* tmap, uint32_t cluster_bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2"
      " [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(cluster_bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const void* tmap, uint32_t cluster_bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2"
      " [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(cluster_bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}

// D[tmem] (+)= A[tmem] * B[smem desc]; bf16 inputs, fp32 sums.  A is K-major: lane = row, two bf16 per column.
// B's descriptor comes in halves: steps along K and from stage to stage only change the lower one, without carries.
__device__ __forceinline__ void mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 b;\n\t"
      "setp.ne.b32 p, %5, 0;\n\tmov.b64 b, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p;\n\t}\n"
      ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Instruction descriptor of kind::f16 with bf16 A/B (both K-major) and fp32 D.
__host__ __device__ constexpr uint32_t idesc_bf16_f32(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) |
         (static_cast<uint32_t>(m >> 4) << 24);
}
// Shared-memory matrix descriptor: K-major tile whose rows are 128 B (64 bf16),
// 128-byte swizzle, 8-row groups 1024 B apart.  `addr` is the CTA-shared byte
// address of the (1024 B aligned) tile, plus 32 B per 16-element step along K.
__device__ __forceinline__ uint64_t smem_desc_kmajor_sw128(uint32_t addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((addr & 0x3FFFF) >> 4);  // start address
  d |= static_cast<uint64_t>(1) << 16;                // leading byte offset (unused when swizzled)
  d |= static_cast<uint64_t>(1024 >> 4) << 32;        // stride byte offset
  d |= static_cast<uint64_t>(1) << 46;                // descriptor version (sm_100)
  d |= static_cast<uint64_t>(2) << 61;                // SWIZZLE_128B
  return d;
}

// TMEM address: lane in bits 31..16, column in bits 15..0.
__device__ __forceinline__ uint32_t tmem_addr(uint32_t base, uint32_t lane, uint32_t col) {
  return base + (lane << 16) + col;
}

// 16 lanes x 128 bit, repeated 4 times along the columns (16 columns in all).
// Thread t of the warp holds, for repeat j in 0..3 and h in 0..1, register
// r[2*j + h] = (lane base + 8*h + t/4, column 4*j + t%4): the layout of an
// mma.sync m16n8k16 A fragment, so a pair of consecutive-k bf16 values for one
// row travels in one register.
__device__ __forceinline__ void tmem_st_16x128b_x4(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
      "r"(r[7])
      : "memory");
}

// Load counterpart of tmem_st_16x128b_x4: same (thread, register) -> (lane, column) map.
__device__ __forceinline__ void tmem_ld_16x128b_x4(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x128b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7])
      : "r"(taddr)
      : "memory");
}

}  // namespace dx
