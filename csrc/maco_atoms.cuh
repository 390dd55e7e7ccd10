// Synchronisation and data-movement primitives for sm_100a, as inline PTX.
//
// Covers what the reference's maco/csrc/maco_atoms.cuh:34-197 offers (acquire/release
// loads, stores and atomics at .gpu and .sys scope, nanosleep, warp-leader election) and adds
// what a Blackwell kernel needs on top: mbarriers, async-proxy fences, TMA tile loads,
// tcgen05 (MMA issue, commit, TMEM alloc/ld), multimem loads/stores through an NVSwitch
// multicast address, and *bounded* waits. Every wait in this file gives up after a time
// budget and reports failure to its caller instead of spinning forever.
#pragma once
#include <cstdint>
#include <cuda_bf16.h>

namespace maco {

#define MACO_DEVICE __device__ __forceinline__

// ---------------------------------------------------------------------------------------------
// Scoped loads / stores / atomics on global memory
// ---------------------------------------------------------------------------------------------
MACO_DEVICE uint64_t ld_acquire_gpu_u64(const uint64_t* p) {
  uint64_t v; asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory"); return v;
}
MACO_DEVICE void st_release_gpu_u64(uint64_t* p, uint64_t v) {
  asm volatile("st.release.gpu.global.u64 [%0], %1;" :: "l"(p), "l"(v) : "memory");
}
MACO_DEVICE uint64_t ld_relaxed_gpu_u64(const uint64_t* p) {
  uint64_t v; asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory"); return v;
}
MACO_DEVICE void st_relaxed_gpu_u64(uint64_t* p, uint64_t v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" :: "l"(p), "l"(v) : "memory");
}
MACO_DEVICE uint64_t atom_add_release_gpu_u64(uint64_t* p, uint64_t v) {
  uint64_t old; asm volatile("atom.add.release.gpu.global.u64 %0, [%1], %2;" : "=l"(old) : "l"(p), "l"(v) : "memory"); return old;
}
MACO_DEVICE uint64_t atom_add_relaxed_gpu_u64(uint64_t* p, uint64_t v) {
  uint64_t old; asm volatile("atom.add.relaxed.gpu.global.u64 %0, [%1], %2;" : "=l"(old) : "l"(p), "l"(v) : "memory"); return old;
}
MACO_DEVICE uint64_t atom_cas_release_gpu_u64(uint64_t* p, uint64_t cmp, uint64_t val) {
  uint64_t old; asm volatile("atom.cas.release.gpu.global.b64 %0, [%1], %2, %3;" : "=l"(old) : "l"(p), "l"(cmp), "l"(val) : "memory"); return old;
}
MACO_DEVICE uint32_t ld_acquire_gpu_u32(const uint32_t* p) {
  uint32_t v; asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory"); return v;
}
MACO_DEVICE uint32_t ld_relaxed_gpu_u32(const uint32_t* p) {
  uint32_t v; asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory"); return v;
}
MACO_DEVICE void st_release_gpu_u32(uint32_t* p, uint32_t v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" :: "l"(p), "r"(v) : "memory");
}
MACO_DEVICE void st_relaxed_gpu_u32(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" :: "l"(p), "r"(v) : "memory");
}
MACO_DEVICE uint32_t atom_add_release_gpu_u32(uint32_t* p, uint32_t v) {
  uint32_t old; asm volatile("atom.add.release.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory"); return old;
}
MACO_DEVICE uint32_t atom_add_acq_rel_gpu_u32(uint32_t* p, uint32_t v) {
  uint32_t old; asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory"); return old;
}
MACO_DEVICE uint32_t atom_add_relaxed_gpu_u32(uint32_t* p, uint32_t v) {
  uint32_t old; asm volatile("atom.add.relaxed.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory"); return old;
}
MACO_DEVICE void red_add_release_gpu_u32(uint32_t* p, uint32_t v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" :: "l"(p), "r"(v) : "memory");
}
MACO_DEVICE void red_add_relaxed_gpu_u32(uint32_t* p, uint32_t v) {
  asm volatile("red.relaxed.gpu.global.add.u32 [%0], %1;" :: "l"(p), "r"(v) : "memory");
}

// .sys scope: flags that another GPU (over NVLink) or the host reads or writes.
MACO_DEVICE uint64_t ld_acquire_sys_u64(const uint64_t* p) {
  uint64_t v; asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory"); return v;
}
MACO_DEVICE void st_release_sys_u64(uint64_t* p, uint64_t v) {
  asm volatile("st.release.sys.global.u64 [%0], %1;" :: "l"(p), "l"(v) : "memory");
}
MACO_DEVICE uint64_t atom_add_release_sys_u64(uint64_t* p, uint64_t v) {
  uint64_t old; asm volatile("atom.add.release.sys.global.u64 %0, [%1], %2;" : "=l"(old) : "l"(p), "l"(v) : "memory"); return old;
}
MACO_DEVICE uint32_t ld_acquire_sys_u32(const uint32_t* p) {
  uint32_t v; asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory"); return v;
}
MACO_DEVICE uint32_t ld_relaxed_sys_u32(const uint32_t* p) {
  uint32_t v; asm volatile("ld.relaxed.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory"); return v;
}
MACO_DEVICE void st_release_sys_u32(uint32_t* p, uint32_t v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" :: "l"(p), "r"(v) : "memory");
}
MACO_DEVICE void st_relaxed_sys_u32(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.sys.global.u32 [%0], %1;" :: "l"(p), "r"(v) : "memory");
}
MACO_DEVICE void red_add_release_sys_u32(uint32_t* p, uint32_t v) {
  asm volatile("red.release.sys.global.add.u32 [%0], %1;" :: "l"(p), "r"(v) : "memory");
}
MACO_DEVICE void red_add_relaxed_sys_u32(uint32_t* p, uint32_t v) {
  asm volatile("red.relaxed.sys.global.add.u32 [%0], %1;" :: "l"(p), "r"(v) : "memory");
}
MACO_DEVICE uint32_t atom_add_release_sys_u32(uint32_t* p, uint32_t v) {
  uint32_t old; asm volatile("atom.add.release.sys.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory"); return old;
}
MACO_DEVICE void fence_acq_rel_sys() { asm volatile("fence.acq_rel.sys;" ::: "memory"); }
MACO_DEVICE void fence_acq_rel_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// 16-byte vector accesses used by the copy / reduce kernels (peer memory included).
MACO_DEVICE uint4 ld_global_v4(const void* p) {
  uint4 v; asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory"); return v;
}
MACO_DEVICE uint4 ld_global_nc_v4(const void* p) {
  uint4 v; asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p)); return v;
}
MACO_DEVICE void st_global_v4(void* p, uint4 v) {
  asm volatile("st.global.v4.u32 [%0], {%1,%2,%3,%4};" :: "l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// ---------------------------------------------------------------------------------------------
// Time, sleep, election
// ---------------------------------------------------------------------------------------------
MACO_DEVICE uint64_t globaltimer_ns() {
  uint64_t t; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t)); return t;
}
MACO_DEVICE void maco_nanosleep(uint32_t ns = 20) { __nanosleep(ns); }
MACO_DEVICE uint32_t smid() { uint32_t r; asm volatile("mov.u32 %0, %%smid;" : "=r"(r)); return r; }
MACO_DEVICE uint32_t lane_id() { return threadIdx.x & 31; }
MACO_DEVICE bool elect_one() {
  uint32_t pred;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.b32 %0, 1, 0, p;\n}" : "=r"(pred));
  return pred != 0;
}
// Lane 0's value in every lane: values read from memory become ones the compiler knows to be uniform.
template <typename T> MACO_DEVICE T warp_uniform(T v) { return __shfl_sync(0xffffffffu, v, 0); }
MACO_DEVICE uint32_t elect_warp_leader() { return __ffs(__activemask()) - 1; }
MACO_DEVICE bool is_warp_leader() { return lane_id() == elect_warp_leader(); }

// Bounded wait on a global flag: returns true once *flag >= expect, false when budget_ns ran out
// or the kernel-wide abort word became non-zero. Never spins forever.
template <bool kSys>
MACO_DEVICE bool wait_flag_ge_u32(const uint32_t* flag, uint32_t expect, uint64_t budget_ns,
                                  const uint32_t* abort_word = nullptr) {
  uint32_t v = kSys ? ld_acquire_sys_u32(flag) : ld_acquire_gpu_u32(flag);
  if ((int32_t)(v - expect) >= 0) return true;
  const uint64_t t0 = globaltimer_ns();
  uint32_t spins = 0;
  while (true) {
    v = kSys ? ld_acquire_sys_u32(flag) : ld_acquire_gpu_u32(flag);
    if ((int32_t)(v - expect) >= 0) return true;
    if ((++spins & 63u) == 0) {
      if (abort_word != nullptr && ld_relaxed_gpu_u32(abort_word) != 0) return false;
      if (globaltimer_ns() - t0 > budget_ns) return false;
    }
    __nanosleep(20);
  }
}

// ---------------------------------------------------------------------------------------------
// Shared-memory addresses, mbarriers, proxy fences
// ---------------------------------------------------------------------------------------------
MACO_DEVICE uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

MACO_DEVICE void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(bar)), "r"(count) : "memory");
}
MACO_DEVICE void mbar_inval(uint64_t* bar) {
  asm volatile("mbarrier.inval.shared::cta.b64 [%0];" :: "r"(smem_u32(bar)) : "memory");
}
MACO_DEVICE void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
MACO_DEVICE void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
MACO_DEVICE void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }
MACO_DEVICE void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(smem_u32(bar)) : "memory");
}
MACO_DEVICE void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(smem_u32(bar)), "r"(bytes) : "memory");
}
MACO_DEVICE bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.b32 %0, 1, 0, p;\n}"
               : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}
// Bounded mbarrier wait. `abort_smem` is a CTA-local word any role sets when it gives up, so
// the other roles of the CTA leave their waits too.
MACO_DEVICE bool mbar_wait(uint64_t* bar, uint32_t parity, uint64_t budget_ns, volatile uint32_t* abort_smem) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  uint32_t spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++spins & 255u) == 0) {
      if (*abort_smem != 0) return false;
      if (globaltimer_ns() - t0 > budget_ns) { *abort_smem = 1; return false; }
    }
  }
  return true;
}

// The same for a whole, converged warp, with one verdict for all lanes: a lane that gave up while another saw the phase complete would
// leave that one alone at the next elect.sync.
MACO_DEVICE bool mbar_wait_warp(uint64_t* bar, uint32_t parity, uint64_t budget_ns, volatile uint32_t* abort_smem) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  const uint64_t t0 = globaltimer_ns();
  uint32_t spins = 0;
  while (!__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) {
    if ((++spins & 255u) == 0) {
      const bool late = globaltimer_ns() - t0 > budget_ns;
      if (late) *abort_smem = 1;
      if (__any_sync(0xffffffffu, late || *abort_smem != 0)) return false;
    }
  }
  return true;
}

MACO_DEVICE void cp_async16(uint32_t sdst, const void* gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(sdst), "l"(gsrc) : "memory");
}
MACO_DEVICE void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> MACO_DEVICE void cp_async_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }

// ---------------------------------------------------------------------------------------------
// TMA (tile mode, no cluster qualifier: every CTA fetches its own tiles)
// ---------------------------------------------------------------------------------------------
MACO_DEVICE void tma_load_2d(void* smem_dst, const void* tmap, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      :: "r"(smem_u32(smem_dst)), "l"(tmap), "r"(smem_u32(bar)), "r"(x), "r"(y) : "memory");
}
MACO_DEVICE void tma_load_3d(void* smem_dst, const void* tmap, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      :: "r"(smem_u32(smem_dst)), "l"(tmap), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z) : "memory");
}
MACO_DEVICE void tma_prefetch_desc(const void* tmap) {
  asm volatile("prefetch.tensormap [%0];" :: "l"(tmap) : "memory");
}
MACO_DEVICE void tma_store_2d(const void* tmap, const void* smem_src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               :: "l"(tmap), "r"(smem_u32(smem_src)), "r"(x), "r"(y) : "memory");
}
// Untiled bulk copies (both addresses 16-byte aligned, size a multiple of 16 bytes).
MACO_DEVICE void bulk_load(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               :: "r"(smem_u32(smem_dst)), "l"(gsrc), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
MACO_DEVICE void bulk_store(void* gdst, const void* smem_src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
               :: "l"(gdst), "r"(smem_u32(smem_src)), "r"(bytes) : "memory");
}
MACO_DEVICE void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N> MACO_DEVICE void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" :: "n"(N) : "memory"); }
template <int N> MACO_DEVICE void tma_store_wait() { asm volatile("cp.async.bulk.wait_group %0;" :: "n"(N) : "memory"); }

// ---------------------------------------------------------------------------------------------
// tcgen05: tensor memory and the 5th-generation MMA
// ---------------------------------------------------------------------------------------------
MACO_DEVICE void tmem_alloc(uint32_t* smem_slot, uint32_t ncols) {   // whole warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(smem_slot)), "r"(ncols) : "memory");
}
MACO_DEVICE void tmem_relinquish() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory"); }
MACO_DEVICE void tmem_dealloc(uint32_t taddr, uint32_t ncols) {      // whole warp
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(taddr), "r"(ncols) : "memory");
}
MACO_DEVICE void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
MACO_DEVICE void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Arrive on an mbarrier once every MMA issued so far by this thread has finished.
MACO_DEVICE void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(smem_u32(bar)) : "memory");
}
// D[tmem] (+)= A[smem desc] * B[smem desc]; one thread issues for the CTA.
MACO_DEVICE void tc_mma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
      :: "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
MACO_DEVICE void tc_mma_tf32(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}"
      :: "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// 32 lanes x 32 consecutive fp32 columns: thread t of the warp receives lane (base_lane + t).
MACO_DEVICE void tmem_ld_32x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}
MACO_DEVICE void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}
MACO_DEVICE void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// ---- two-CTA forms (cta_group::2): a pair of CTAs in one cluster works on one 256-row tile -----------------
// The MMA is issued by the pair's leader (cluster rank 0) and reads operand tiles at the same shared-memory
// offset in both CTAs; each CTA's TMEM receives its 128 rows of the accumulator. Every tcgen05 instruction of
// a kernel uses the same cta_group, so a kernel is built either from the forms above or from these.
MACO_DEVICE uint32_t cluster_ctarank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
MACO_DEVICE void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
MACO_DEVICE void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// shared::cluster address of `smem_addr` (a shared::cta address of this CTA) in the CTA of cluster rank `rank`
MACO_DEVICE uint32_t mapa_u32(uint32_t smem_addr, uint32_t rank) {
  uint32_t r; asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank)); return r;
}
MACO_DEVICE void mbar_arrive_cluster(uint32_t cluster_addr) {      // arrive on a barrier of any CTA of the cluster
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" :: "r"(cluster_addr) : "memory");
}
MACO_DEVICE void tmem_alloc2(uint32_t* smem_slot, uint32_t ncols) {   // one whole warp in EACH CTA of the pair
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(smem_slot)), "r"(ncols) : "memory");
}
MACO_DEVICE void tmem_relinquish2() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory"); }
MACO_DEVICE void tmem_dealloc2(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" :: "r"(taddr), "r"(ncols) : "memory");
}
// Arrive on the barrier at shared::cluster address `cluster_addr` once every MMA issued so far has finished.
MACO_DEVICE void tc_commit2(uint32_t cluster_addr) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(cluster_addr) : "memory");
}
// The same arrival on the barrier at this offset in BOTH CTAs of the pair (mask 0b11), one instruction.
MACO_DEVICE void tc_commit2_both(uint32_t bar_addr) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               :: "r"(bar_addr), "h"((uint16_t)3) : "memory");
}
MACO_DEVICE void tc_mma2_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}"
      :: "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// TMA tile load into THIS CTA's shared memory whose byte count is credited to a barrier that may live in the
// pair's other CTA (`bar_cluster_addr` is a shared::cluster address). No other CTA receives the data.
MACO_DEVICE void tma_load_2d_pair(void* smem_dst, const void* tmap, uint32_t bar_cluster_addr, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      :: "r"(smem_u32(smem_dst)), "l"(tmap), "r"(bar_cluster_addr), "r"(x), "r"(y) : "memory");
}

// Lean issue forms for the main loops: the descriptor's high word (offsets, version, swizzle) is constant per
// operand, only the low word (start address >> 4) moves, so the issuing thread spends one add per MMA.
MACO_DEVICE void tc_mma_f16_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                               uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 da, db;\n setp.ne.b32 p, %6, 0;\n mov.b64 da, {%1, %2};\n mov.b64 db, {%3, %4};\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n}"
      :: "r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate) : "memory");
}
MACO_DEVICE void tc_mma_tf32_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 da, db;\n setp.ne.b32 p, %6, 0;\n mov.b64 da, {%1, %2};\n mov.b64 db, {%3, %4};\n"
      " tcgen05.mma.cta_group::1.kind::tf32 [%0], da, db, %5, p;\n}"
      :: "r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate) : "memory");
}
MACO_DEVICE void tc_mma2_f16_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 da, db;\n setp.ne.b32 p, %6, 0;\n mov.b64 da, {%1, %2};\n mov.b64 db, {%3, %4};\n"
      " tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %5, p;\n}"
      :: "r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate) : "memory");
}

// Shared-memory matrix descriptor for tcgen05.mma. Addresses and offsets are in 16-byte units.
//   layout_type: 0 none, 2 = 128-byte swizzle, 4 = 64-byte, 6 = 32-byte.
MACO_DEVICE uint64_t make_smem_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes, uint32_t layout_type) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;                       // descriptor version for sm_100
  d |= (uint64_t)(layout_type & 7u) << 61;
  return d;
}
// Instruction descriptor for kind::f16 / kind::tf32 with an fp32 accumulator.
//   ab_format: 0 fp16, 1 bf16, 2 tf32.  *_mn_major: 0 = K-major operand, 1 = MN-major.
__host__ __device__ constexpr uint32_t make_idesc(uint32_t ab_format, uint32_t m, uint32_t n,
                                                  uint32_t a_mn_major, uint32_t b_mn_major) {
  return (1u << 4) | (ab_format << 7) | (ab_format << 10) | (a_mn_major << 15) | (b_mn_major << 16) |
         ((n >> 3) << 17) | ((m >> 4) << 24);
}

// ---------------------------------------------------------------------------------------------
// multimem: loads that reduce across, and stores that broadcast to, every GPU bound to an
// NVSwitch multicast address.
// ---------------------------------------------------------------------------------------------
MACO_DEVICE uint4 multimem_ld_reduce_bf16x8(const void* mc_ptr) {
  uint4 v;
  asm volatile("multimem.ld_reduce.relaxed.sys.global.add.acc::f32.v4.bf16x2 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(mc_ptr) : "memory");
  return v;
}
MACO_DEVICE uint4 multimem_ld_reduce_f16x8(const void* mc_ptr) {
  uint4 v;
  asm volatile("multimem.ld_reduce.relaxed.sys.global.add.acc::f32.v4.f16x2 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(mc_ptr) : "memory");
  return v;
}
MACO_DEVICE float4 multimem_ld_reduce_f32x4(const void* mc_ptr) {
  float4 v;
  asm volatile("multimem.ld_reduce.relaxed.sys.global.add.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(mc_ptr) : "memory");
  return v;
}
MACO_DEVICE void multimem_st_v4(void* mc_ptr, uint4 v) {
  asm volatile("multimem.st.relaxed.sys.global.v4.f32 [%0], {%1,%2,%3,%4};"
               :: "l"(mc_ptr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
MACO_DEVICE void multimem_st_v4_weak(void* mc_ptr, uint4 v) {
  asm volatile("multimem.st.weak.global.v4.f32 [%0], {%1,%2,%3,%4};"
               :: "l"(mc_ptr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
MACO_DEVICE void multimem_red_add_u32(uint32_t* mc_ptr, uint32_t v) {
  asm volatile("multimem.red.release.sys.global.add.u32 [%0], %1;" :: "l"(mc_ptr), "r"(v) : "memory");
}

// ---------------------------------------------------------------------------------------------
// Small numeric helpers
// ---------------------------------------------------------------------------------------------
MACO_DEVICE uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
MACO_DEVICE float2 unpack_bf16x2(uint32_t u) {
  __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&u);
  return __bfloat1622float2(v);
}
MACO_DEVICE float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
MACO_DEVICE float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// tanh-GELU, 0.5 x (1 + tanh u) = x / (1 + exp(-2u)), in two forms. For results that are rounded to 16 bits: one fast
// exponential and one fast division (a few 2^-23 off, far below the rounding), where tanhf is a branchy 30-instruction sequence.
MACO_DEVICE float gelu_tanh(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  return __fdividef(x, 1.f + __expf(-2.f * k0 * (x + k1 * x * x * x)));
}
// d/dx: s + 2 x s (1 - s) k0 (1 + 3 k1 x^2) with s = 1 / (1 + e), 1 - s = e s, e = exp(-2u) kept finite. Beyond |x| = 10
// (e = 10^-38 or 10^38) the derivative is 1 or 0 to the last bit, while the formula's x^3 would grow against the clamped
// e (-3.9e9 at x = -1e15) and then overflow; x - x keeps an infinity visible as NaN.
MACO_DEVICE float gelu_tail(float x, float d) { return fabsf(x) > 10.f ? (x > 0.f ? 1.f : 0.f) + (x - x) : d; }
MACO_DEVICE float gelu_tanh_grad(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  const float e = __expf(fminf(-2.f * k0 * (x + k1 * x * x * x), 80.f));
  const float s = __fdividef(1.f, 1.f + e);
  return gelu_tail(x, s + 2.f * x * s * (e * s) * k0 * (1.f + 3.f * k1 * x * x));
}
// For results that stay fp32: tanhf where 1 + tanh(u) keeps its bits, the logistic form with a full-precision exponential
// and division where it would cancel. 2-norm of the error relative to 64 bits, against tanhf everywhere: equal for
// x > -0.3, 1.4e-7 against 4e-7 for x in (-2, -1.5), 3e-7 against 5e-5 in (-5, -3). The derivative also leaves tanhf above 1.75,
// where 1 - tanh^2 cancels (5e-8 against 2.7e-7 in (3, 5)).
MACO_DEVICE float gelu_tanh_f32(float x) {
  const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
  return x > -0.3f ? 0.5f * x * (1.f + tanhf(u)) : x / (1.f + expf(-2.f * u));
}
MACO_DEVICE float gelu_tanh_grad_f32(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  const float u = k0 * (x + k1 * x * x * x), du = k0 * (1.f + 3.f * k1 * x * x);
  if (x > -0.3f && x < 1.75f) {
    const float t = tanhf(u);
    return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * du;
  }
  const float e = expf(fminf(-2.f * u, 80.f)), s = 1.f / (1.f + e);
  return gelu_tail(x, s + 2.f * x * s * (e * s) * du);
}
// (out of line for the unrolled GEMM epilogues, whose fp32 results are the rare case)
static __device__ __noinline__ float gelu_tanh_f32_call(float x) { return gelu_tanh_f32(x); }
static __device__ __noinline__ float gelu_tanh_grad_f32_call(float x) { return gelu_tanh_grad_f32(x); }
MACO_DEVICE float silu(float x) { return x / (1.f + __expf(-x)); }
// The same quotient for unrolled epilogues, whose code would mostly be inlined divisions (an SM that runs them for the first time in a
// launch fetches that code from L2): the product with the approximate reciprocal, corrected once by its residual (Markstein, 1990).
// Both operands are quartered, so that the reciprocal stays normal up to the largest finite 1 + exp(-x). Against silu() over every float: the
// same fp16 values; the same bf16 values but for 512 floats below 2^-124 in magnitude, where x / 4 is subnormal and the result off by up to
// one subnormal unit; above that the same fp32 bits but for two floats. (Forms exact there too cost linears with SiLU 4 to 12 %.) The
// product alone has an rms error of 1.40e-7 instead of 1.37e-7 and was 0 below -87.3. One B200, us, product alone /
// corrected / division or a longer guard: SwiGLU block of 1003 rows 105.9 / 106.9 / 115, expert layer of 256 tokens 103 / 106 / 111.
MACO_DEVICE float silu_16(float x) {
  const float y4 = fmaf(__expf(-x), 0.25f, 0.25f), x4 = 0.25f * x;
  float r;                                             // 4 / (1 + exp(-x))
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y4));
  const float q = x4 * r, e = fmaf(-q, y4, x4);
  return fabsf(e) > 0.f ? fmaf(e, r, q) : q;           // (no residual: the quotient is exact, or x or exp(-x) is infinite)
}

}  // namespace maco
