// Thin inline-PTX layer for sm_100a: mbarrier, TMA (cp.async.bulk[.tensor]),
// tcgen05 (TMEM alloc / mma / commit / ld) and system-scope flag traffic.
//
// Every wait in here is bounded by wall time (%globaltimer).  A wait that runs
// out returns false; the caller records a status code and tears down.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include "status.h"

namespace rf {

// ---------------------------------------------------------------- misc ----
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ uint64_t global_timer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }
// True in one lane of a fully converged warp.  A role whose whole warp runs the loop around it keeps its operands in uniform registers,
// where the tcgen05 and bulk-copy instructions want them.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n selp.b32 %0, 1, 0, q;\n}" : "=r"(p));
  return p != 0;
}

// Wait limits.  Local waits (smem barriers) cover at most one tile of work;
// peer waits cover a whole kernel on another GPU.
constexpr uint64_t kLocalWaitNs = 2000ull * 1000ull * 1000ull;  // 2 s
constexpr uint64_t kPeerWaitNs = 1000ull * 1000ull * 1000ull;   // 1 s

__device__ __forceinline__ void report_status(int32_t* status, int32_t code, int32_t tag,
                                              int32_t detail) {
  if (status == nullptr) return;
  if (atomicCAS(status, 0, code) == 0) {
    status[1] = static_cast<int32_t>(blockIdx.x);
    status[2] = tag;
    status[3] = detail;
  }
}

// ------------------------------------------- programmatic dependent launch ----
// Every kernel in this library starts with pdl_prologue(): it lets the next
// kernel in the stream begin launching at once and then blocks until the
// previous kernel has completed and flushed.  Work that does not depend on the
// previous kernel (barrier set-up, TMEM allocation, weight prefetch) may be
// placed between launch_dependents and wait.
__device__ __forceinline__ void pdl_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_prologue() {
  pdl_launch_dependents();
  pdl_wait();
}

// ------------------------------------------------------------ mbarrier ----
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.shared::cta.b64 st, [%0];\n}" ::"r"(
                   smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile(
      "{\n .reg .b64 st;\n mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}" ::"r"(
          smem_u32(bar)),
      "r"(bytes)
      : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n"
      " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.b32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait on one phase of an mbarrier.  Returns false on timeout.
// backoff_ns > 0: sleep between polls, for single-lane roles (TMA producer, MMA issuer) whose spinning would
// otherwise take issue slots from the compute warps that share their scheduler.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity,
                                          uint64_t limit_ns = kLocalWaitNs, uint32_t backoff_ns = 0) {
  if (mbar_try_wait(bar, parity)) return true;
  if (limit_ns == 0) return false;
  const uint64_t t0 = global_timer_ns();
  while (true) {
#pragma unroll 1
    for (int i = 0; i < 64; ++i) {
      if (mbar_try_wait(bar, parity)) return true;
      if (backoff_ns) __nanosleep(backoff_ns);
    }
    if (global_timer_ns() - t0 > limit_ns) return false;
  }
}

// What happens once in a launch's life or never stands out of line: inside the kernels it cost a GEMM of 93 rows half a microsecond of instruction
// fetches (prompt of 93 tokens, 16 layers, us: 1236, so 1192).
static __device__ __noinline__ void role_gives_up(int32_t* gave_up, int32_t* status, int32_t code, int32_t tag, int32_t detail, uint32_t peer) {
  volatile int32_t* flag = gave_up;
  if (!*flag) report_status(status, code, tag, detail);
  *flag = 1;
  if (peer) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(peer), "r"(1u) : "memory");
  asm volatile("fence.acq_rel.cluster;" ::: "memory");
}
// A wait of a role that its whole warp runs; the answer is the lane's own.  When it runs out, `code` is reported (by the first role of the CTA to give
// up), `gave_up` is set, ahead of anything that the role does next, and its later waits have no patience.  Behind that
//   * a role that writes what others may still use (copies into a ring, a new accumulator, stores, arrivals) starts nothing more;
//   * the MMA role alone goes on through the k blocks of an accumulator whose operands did not come: it writes nothing but that accumulator, and
//     whoever is told that it is complete looks at `gave_up` before taking it.  A test or a vote between barrier and MMA would cost every launch
//     (prefill attention, a chain of such waits, 2 to 10 per cent).  It gives no ring stage back any more, whose copies may still be under way: a
//     barrier armed again with bytes of its phase outstanding has no meaning;
//   * the teardown waits for what was started (settle_copies, settle_mmas).
// `peer`: the flag of the pair's other CTA (a shared::cluster address), 0 for none.
__device__ __forceinline__ bool role_wait(uint64_t* bar, uint32_t parity, uint64_t* limit_ns, int32_t* gave_up, int32_t* status, int32_t code,
                                          int32_t tag, int32_t detail, uint32_t backoff_ns = 0, uint32_t peer = 0) {
  if (mbar_wait(bar, parity, *limit_ns, backoff_ns)) return true;
  role_gives_up(gave_up, status, code, tag, detail, peer);
  *limit_ns = 0;
  return false;
}
// Whether a wait came true in every lane: the warp leaves a loop together.
__device__ __forceinline__ bool agreed(bool ok) { return __all_sync(0xffffffffu, ok); }
// Teardown after a role gave up, when every role has stopped: what was started has to end before the CTA's memory goes.  Copies: the last `stages`
// of `issued` fills of a ring, each of which completes a phase of its stage's barrier.
constexpr uint64_t kSettleNs = 20ull * 1000 * 1000;
static __device__ __noinline__ void settle_copies(uint64_t* full, int stages, int issued) {
  for (int i = issued > stages ? issued - stages : 0; i < issued; ++i) mbar_wait(&full[i % stages], (uint32_t)(i / stages) & 1u, kSettleNs);
}

// ----------------------------------------------------------------- TMA ----
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
// 2-D tiled load global -> this CTA's shared memory, completion on an mbarrier.
// c0 is the innermost (contiguous) coordinate: c0 * elem_size must be a
// multiple of 16 bytes.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* m, uint64_t* bar,
                                            int32_t c0, int32_t c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_2d_hint(void* smem_dst, const CUtensorMap* m,
                                                 uint64_t* bar, int32_t c0, int32_t c1,
                                                 uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4}], [%2], %5;" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "l"(policy)
      : "memory");
}
__device__ __forceinline__ uint64_t l2_policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t l2_policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
// Untiled bulk copy global -> shared.  Both addresses 16-byte aligned, bytes a
// multiple of 16.
__device__ __forceinline__ void bulk_load_1d(void* smem_dst, const void* gsrc, uint32_t bytes,
                                             uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(gsrc)), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
// The same with an L2 cache policy (createpolicy): evict_first for data that is read once.
__device__ __forceinline__ void bulk_load_1d_hint(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar,
                                                  uint64_t policy) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::
          "r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(gsrc)), "r"(bytes), "r"(smem_u32(bar)), "l"(policy)
      : "memory");
}
// Tiled bulk store shared -> global of one box of a 2-D tensor map (x = innermost coordinate, a multiple of
// 16 bytes; parts of the box outside the tensor are not written).  The issuing thread owns the bulk group.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* m, const void* smem_src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(m)),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y)
               : "memory");
}
// Untiled bulk copy shared -> global (both 16-byte aligned, bytes a multiple of 16); the issuing thread owns the bulk group.
__device__ __forceinline__ void bulk_store_1d(void* gdst, const void* smem_src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(reinterpret_cast<uint64_t>(gdst)),
               "r"(smem_u32(smem_src)), "r"(bytes)
               : "memory");
}
// all but the newest bulk group of this thread have finished reading shared memory
__device__ __forceinline__ void bulk_wait_read_1() { asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); }
__device__ __forceinline__ void bulk_commit_group() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// all bulk groups of this thread have finished READING shared memory (the source may be overwritten)
__device__ __forceinline__ void bulk_wait_read_all() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// all bulk groups of this thread are complete (their global writes are done)
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// Fire-and-forget prefetch of a contiguous global range into L2 (16-byte aligned, bytes a multiple of 16).
// Lets a kernel keep far more bytes in flight towards DRAM than its shared-memory ring can hold: the later
// bulk copy of the same range then completes with L2 latency.
__device__ __forceinline__ void bulk_prefetch_l2(const void* gsrc, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(reinterpret_cast<uint64_t>(gsrc)), "r"(bytes)
               : "memory");
}
// The same for one box of a 2-D tensor map.
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap* tm, int x, int y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(reinterpret_cast<uint64_t>(tm)),
               "r"(x), "r"(y)
               : "memory");
}

// ------------------------------------------------------------- tcgen05 ----
// TMEM allocation: whole warp executes; ncols a power of two in [32, 512].
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_holder, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_holder)),
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
__device__ __forceinline__ void tc_fence_before_sync() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after_sync() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// D[tmem] (+)= A[smem desc] * B[smem desc]; one thread issues.
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b,
                                         uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// The same with A in tensor memory: lane r holds row r, a 32-bit column two neighbouring values of K.
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// mbarrier arrives once every MMA issued so far by this thread has finished.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}
// Teardown after a role gave up, by the warp whose elected lane issued (elect_one names the same one again): its MMAs end before tensor memory is
// handed back.
static __device__ __noinline__ void settle_mmas(uint64_t* bar) {
  if (elect_one()) umma_commit(bar);
  __syncwarp();
  mbar_wait(bar, 0, kSettleNs);
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// Each lane reads 16 consecutive 32-bit columns of its own TMEM lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32"
      " {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

// Each lane reads 32 consecutive 32-bit columns of its own TMEM lane.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32"
      " {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15,"
      " %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
// Each lane writes 32 consecutive 32-bit columns of its own TMEM lane.
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0],"
      " {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16,"
      " %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// 64-bit shared-memory matrix descriptor for a K-major operand tile whose rows
// are 128 bytes (64 x 16-bit) laid out with the 128-byte swizzle that a TMA
// box of inner extent 128 bytes produces: 8-row groups of 1024 bytes.
//   bits [0,14)  start address >> 4      bits [16,30) leading byte offset >> 4
//   bits [32,46) stride byte offset >> 4 bits [46,48) descriptor version (1)
//   bits [61,64) layout type (2 = 128-byte swizzle)
__device__ __forceinline__ uint64_t umma_desc_k128(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>(1) << 16;             // LBO: unused with swizzle, canonical 1
  d |= static_cast<uint64_t>(1024 >> 4) << 32;     // SBO: next 8-row group
  d |= static_cast<uint64_t>(1) << 46;             // version
  d |= static_cast<uint64_t>(2) << 61;             // SWIZZLE_128B
  return d;
}
// Descriptor of an MN-major operand (its M or N index is the contiguous one) in the 128-byte swizzle:
// the tile is a stack of [k rows x 64 elements] slabs, row pitch 128 bytes, 8-row groups 1024 bytes apart
// (stride byte offset); the next 64 elements along M/N start `mn_chunk_bytes` later (leading byte offset).
// This is the image a TMA box of 64 elements x rows leaves for a row-major [k, mn] matrix, e.g. V[token, d]
// used as the B operand of P.V.
__device__ __forceinline__ uint64_t umma_desc_mn128(uint32_t smem_addr, uint32_t mn_chunk_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>((mn_chunk_bytes >> 4) & 0x3FFF) << 16;   // LBO: next 64-element chunk along M/N
  d |= static_cast<uint64_t>(1024 >> 4) << 32;                        // SBO: next 8 k-rows
  d |= static_cast<uint64_t>(1) << 46;                                // version
  d |= static_cast<uint64_t>(2) << 61;                                // SWIZZLE_128B
  return d;
}
// 32-bit instruction descriptor, kind::f16, fp32 accumulate, both operands
// K-major.  ab_fmt: 0 = fp16, 1 = bf16.
__host__ __device__ __forceinline__ uint32_t umma_idesc_f16(int m, int n, int ab_fmt, int b_mn_major = 0) {
  uint32_t d = 0;
  d |= static_cast<uint32_t>(b_mn_major & 1) << 16;  // B operand major-ness: 0 = K, 1 = M/N
  d |= 1u << 4;                                   // D format: fp32
  d |= static_cast<uint32_t>(ab_fmt) << 7;        // A format
  d |= static_cast<uint32_t>(ab_fmt) << 10;       // B format
  d |= static_cast<uint32_t>(n >> 3) << 17;       // N / 8
  d |= static_cast<uint32_t>(m >> 4) << 24;       // M / 16
  return d;
}


// ------------------------------------------------- clusters and DSMEM ----
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// All threads of every CTA in the cluster must execute both halves.
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The same rendezvous without memory ordering: for "every CTA has finished reading its peers' shared memory" before any of
// them exits, where the reads' values were already consumed and nothing written needs to become visible.
__device__ __forceinline__ void cluster_sync_relaxed() {
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
}
// Address of the same shared-memory location in CTA `rank` of this cluster.
__device__ __forceinline__ uint32_t dsmem_addr(uint32_t local_smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_dsmem_u32(uint32_t addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ float2 ld_dsmem_f32x2(uint32_t addr) {   // addr: 8-byte aligned
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float ld_dsmem_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

// ---------------------------------------- CTA pairs (cta_group::2) ----
// Two CTAs of a cluster whose ranks differ in the last bit work on one MMA: each holds half of the rows of A and of D and half of
// the rows of B.  The even rank issues; barriers may lie in its shared memory for both.
__device__ __forceinline__ void pair_tmem_alloc(uint32_t* smem_holder, uint32_t ncols) {      // one warp of each CTA
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_holder)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void pair_tmem_relinquish() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void pair_tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void pair_umma_f16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// The barrier at this offset in BOTH CTAs' shared memory (or those of `ctas`) arrives once every MMA issued so far by this thread has finished.
__device__ __forceinline__ void pair_umma_commit(uint64_t* bar, uint16_t ctas = 3) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "h"(ctas)
               : "memory");
}
// Tiled load into this CTA's shared memory that completes on a barrier of either CTA of the pair (`bar`: a shared::cluster address).
__device__ __forceinline__ void pair_tma_load_2d(void* smem_dst, const CUtensorMap* m, uint32_t bar, int32_t c0, int32_t c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
// Arrival on a barrier of any CTA of the cluster (`bar`: a shared::cluster address).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}

// ----------------------------------------------- system-scope flag I/O ----
__device__ __forceinline__ void st_release_sys(uint32_t* p, uint32_t v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_acquire_sys(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_acquire_gpu(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_sys_add(uint32_t* p, uint32_t v) {
  asm volatile("red.release.sys.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Bounded spin until *p >= target (flags only grow).  Returns false on timeout.
__device__ __forceinline__ bool wait_flag_ge_sys(const uint32_t* p, uint32_t target,
                                                 uint64_t limit_ns = kPeerWaitNs) {
  if (static_cast<int32_t>(ld_acquire_sys(p) - target) >= 0) return true;
  const uint64_t t0 = global_timer_ns();
  while (true) {
#pragma unroll 1
    for (int i = 0; i < 32; ++i)
      if (static_cast<int32_t>(ld_acquire_sys(p) - target) >= 0) return true;
    if (global_timer_ns() - t0 > limit_ns) return false;
  }
}

}  // namespace rf
