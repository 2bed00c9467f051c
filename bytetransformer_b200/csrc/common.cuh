// Device-side building blocks shared by the sm_100a kernels: mbarrier, TMA,
// tcgen05 (UMMA + tensor memory) wrappers, shared-memory matrix descriptors and
// bounded waits.  Everything here is inline PTX; there is no CUTLASS dependency.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace bt {

// ---------------------------------------------------------------------------
// Device status word codes (written by kernels, read by bt_device_status()).
// A non-zero code means a bounded wait gave up or a bounds check tripped; the
// kernel that saw it returned early and its output is not valid.
// ---------------------------------------------------------------------------
enum StatusCode : int {
  kStatusOk = 0,
  kStatusGemmProducerTimeout = 0x101,
  kStatusGemmMmaTimeout = 0x102,
  kStatusGemmEpilogueTimeout = 0x103,
  kStatusMhaLoadTimeout = 0x201,
  kStatusMhaMmaTimeout = 0x202,
  kStatusMhaSoftmaxTimeout = 0x203,
  kStatusBadOffsets = 0x301,
  kStatusSelfTestTimeout = 0x7F1,  // bt_selftest_bounded_wait(): the wait that nothing satisfies ran out, as intended
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}\n"
      : "=r"(pred));
  return pred != 0;
}

// ------------------------------------------------- programmatic dependent launch
// pdl_launch_dependents(): the next kernel of the stream may be launched as soon as all CTAs of this one have said so
// (or have ended).  pdl_wait(): returns once the preceding kernel has completed and its writes are visible; every CTA
// of every kernel calls it before it ends, so a kernel that has completed tells that all before it have.  Without the
// launch attribute both are no-ops.  What holds between the kernels of a call:
//  * The first one is launched the ordinary way (pdl_next_launch_plain), so all that the caller's stream did before the
//    call is complete and visible to every kernel of the call, before its pdl_wait() too.  Weights, bias, gamma, beta and
//    a packed call's offsets may therefore be read ahead of the wait.
//  * Kernels say pdl_launch_dependents() first thing - except those that run second in a call (pack_rows,
//    embedding_layernorm, mask_bits), which say it after their own pdl_wait().  So from the third kernel on, what the
//    FIRST kernel of the call wrote is complete and visible ahead of the wait as well: the attention kernels read the
//    offsets there (MhaLaunch::early_offsets), the GEMM + LayerNorm kernels the row count.
//  * Anything else that an earlier kernel may have written or may still read is touched after pdl_wait() only.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Hint: bring the 128-byte line at `p` into L1 (constants such as bias, gamma and beta, asked for
// while the kernel still waits for its predecessor).
__device__ __forceinline__ void prefetch_l1(const void* p) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

// ------------------------------------------------------------------ mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
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
      "{\n\t"
      ".reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Non-blocking test of a phase (try_wait may suspend the thread for a while before it answers).
__device__ __forceinline__ bool mbar_test_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Wait for a phase with an upper bound.  Returns false when the bound ran out
// or another role of this CTA already gave up (`*abort_flag` non-zero).  The answer
// is the calling lane's own: what a warp waits for goes through the forms below.
// The bound is ~2^31 SM cycles (about a second) unless the caller gives another,
// checked every 256 polls; once the flag is up, a wait ends after nine (not after
// its first: a look at the flag between two polls that a K loop's wait does need was
// seen in the GEMMs' time).
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity,
                                                  volatile int* abort_flag, int* status, int code,
                                                  long long max_cycles = (1ll << 31)) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  uint32_t polls = 0;
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    ++polls;
    if ((polls & 255u) == 8u && *abort_flag != 0) return false;
    if ((polls & 255u) == 0u) {
      if (clock64() - t0 > max_cycles) {
        *abort_flag = 1;
        if (status != nullptr) atomicCAS(status, 0, code);
        return false;
      }
    }
  }
}

// The same for a warp whose 32 lanes all wait: one answer for the warp.  No kernel branches on a lane's own answer:
// lanes that parted ways where a wait gave up would hang in the next warp-wide instruction (elect.sync, tcgen05.ld,
// __syncwarp), bound or no bound.  A role votes (this form), goes on to the end of its K loop and votes there
// (mbar_wait_latched), or goes on regardless (mbar_wait_anyway).
// Every branch here is on a vote.  With a branch on the lanes' own answers - a vote behind the loop is too late - the
// compiler has to take all code behind the wait for code that a part of the warp may run, and forms the operands of the
// tcgen05 and TMA instructions there lane by lane: a K block of four 128 x 64 x 16 MMAs took 314 clocks behind such a
// wait and takes 240 behind this one (198 without a wait).
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status,
                                               int code, long long max_cycles = (1ll << 31)) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  const long long t0 = clock64();
  uint32_t polls = 0;
  while (true) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    ++polls;
    if ((polls & 255u) == 8u && __any_sync(0xffffffffu, *abort_flag != 0)) return false;
    if ((polls & 255u) == 0u && __any_sync(0xffffffffu, clock64() - t0 > max_cycles)) {
      *abort_flag = 1;
      if (status != nullptr) atomicCAS(status, 0, code);
      return false;
    }
  }
}

// The wait of a role that can go on whatever the answer: where it gives up the status word is set, the CTA's flag is up,
// later waits end after nine polls, and what the role makes of the bytes that did not arrive is as invalid as the launch's
// output is then.  For waits in the middle of a tile.  The GEMMs' epilogues use the form whose branches are votes (see
// above; us per forward, lane form / this one: 16 x 512 1111 / 1097, 16 x 128 595 / 591); the softmax warps of the
// attention kernels, whose registers are all taken, the lane form (one sequence of 614 tokens 528.3 against 529.8).
__device__ __forceinline__ void mbar_wait_anyway(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status,
                                                 int code) {
  (void)mbar_wait_warp(bar, parity, abort_flag, status, code);
}
__device__ __forceinline__ void mbar_wait_anyway_lane(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status,
                                                      int code) {
  (void)mbar_wait_bounded(bar, parity, abort_flag, status, code);
}

// The wait of a K loop, which goes on to its end when a wait gave up: `ok` is the answer so far; the loop ends in a vote
// over it.  `landed` is what a test of this barrier and phase, made ahead of the MMAs of the block before, said to the lane:
// the test's latency then passes under the issue of those MMAs (240 -> 218 clocks per K block, see mbar_wait_warp).
// The blocks that are left after a wait gave up are polled nine times each, because the flag is up: the time to give
// up stays one bound however many they are.
__device__ __forceinline__ bool mbar_wait_latched(bool ok, bool landed, uint64_t* bar, uint32_t parity,
                                                  volatile int* abort_flag, int* status, int code,
                                                  long long max_cycles = (1ll << 31)) {
  if (__all_sync(0xffffffffu, landed)) return ok;
  return mbar_wait_warp(bar, parity, abort_flag, status, code, max_cycles) && ok;
}

// Whether no role of the CTA will touch tensor memory any more: the MMA warp's question after its last tile.  It waits for
// the epilogue to hand back the accumulators of the `tiles` tiles that were begun (`acc_empty`: two buffers by turns).
// The answer is the CTA's flag: a wait that gives up raises it (or found it up), the MMA warp's own among them, and the
// epilogue, which goes on after such a wait (mbar_wait_anyway) with loads of tensor memory and with arrivals that say
// nothing, raises it ahead of them.  One answer for the warp.
__device__ __forceinline__ bool accumulators_back(uint64_t* acc_empty, int tiles, volatile int* abort_flag, int* status, int code,
                                                  long long max_cycles = (1ll << 31)) {
  for (int it = tiles < 2 ? 0 : tiles - 2; it < tiles; ++it)
    (void)mbar_wait_warp(&acc_empty[it & 1], (it >> 1) & 1, abort_flag, status, code, max_cycles);
  return __all_sync(0xffffffffu, *abort_flag == 0) != 0;
}

// ------------------------------------------------------------ warp-uniform roles
// tcgen05 and TMA instructions take their descriptors, addresses and coordinates from uniform registers.  In a
// branch that one lane takes (`if (lane == 0)`) every operand of every instruction is moved there first, and that
// cost more than the instruction.  So the single-thread roles are
// walked by their whole warp - role, loop bounds and shared values go through uniform_int(), waits branch on votes - and
// only the instructions themselves are predicated on an elected lane, all MMAs of a K block and their commit on one
// election (umma_k_block).  Clocks per K block of four 128 x 64 x 16 MMAs in the main loop: 525 with one lane, 330 with
// the whole warp and waits that branched on the lanes' own answers, 225 now.
// Because elect.sync needs the whole warp, a warp's lanes must not part ways after a wait that gave up: see
// the forms of a warp's wait above.
// (A reduction, not a shuffle: its result is born in a uniform register, so a branch on it is one the whole warp takes.
// us per forward, shuffle / reduction: 16 x 512 causal 1822 / 1787, 16 x 512 1110 / 1097, one of 38 tokens 364.7 / 365.6.)
// All lanes hold the same value.
__device__ __forceinline__ uint32_t uniform_u32(uint32_t v) { return __reduce_or_sync(0xffffffffu, v); }
__device__ __forceinline__ int uniform_int(int v) { return static_cast<int>(uniform_u32(static_cast<uint32_t>(v))); }

// ----------------------------------------------------------------------- TMA
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* tmap) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(tmap)) : "memory");
}
// 2-D tiled load global -> shared, completion counted in bytes on `bar`.
// `x` is the innermost (contiguous) coordinate and must keep x*elem_size a
// multiple of 16 bytes.  No cluster multicast is used anywhere in this library.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* tmap, uint64_t* bar,
                                            int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
// 2-D tiled store shared -> global (bulk async group completion).
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* tmap, const void* smem_src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(tmap)),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// all but the newest 0 bulk groups of this thread have finished READING shared memory
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// Makes generic-proxy shared-memory writes visible to the async proxy (UMMA/TMA).
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ------------------------------------------------------ cluster launch control
// A running block takes over a block of its own grid that has not started yet: the hardware cancels that launch and
// hands its index out.  The answer (16 bytes at `resp`, 16-byte aligned) is counted in bytes on `bar`.  One thread of
// the block asks; after an answer without a block it must not ask again.
__device__ __forceinline__ void launch_control_ask(void* resp, uint64_t* bar) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the last answer has been read
  mbar_arrive_expect_tx(bar, 16);
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(
                   smem_u32(resp)),
               "r"(smem_u32(bar))
               : "memory");
}
// The index (x) of the block taken over, or -1 if none was left.
__device__ __forceinline__ int launch_control_answer(const void* resp) {
  int x;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      ".reg .b128 r;\n\t"
      "ld.shared.b128 r, [%1];\n\t"
      "mov.b32 %0, -1;\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %0, r;\n\t"
      "}\n"
      : "=r"(x)
      : "r"(smem_u32(resp))
      : "memory");
  return x;
}

// ------------------------------------------------------------------- tcgen05
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
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// One K block of a GEMM main loop, D[tmem] (+)= A[smem] * B[smem], fp16 inputs, fp32 accumulation: four MMAs of 16 K elements each (operands `astep` / `bstep` descriptor units
// apart) and the commit that frees the block's stage.  Called by a whole warp; one elect for the five instructions,
// which are predicated on it.  `accumulate` = 0 overwrites the accumulator with the first product.  PAIR: cta_group::2,
// the commit arrives on the barrier at the same offset in both CTAs.
template <bool PAIR>
__device__ __forceinline__ void umma_k_block(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t astep, uint32_t bstep,
                                             uint32_t idesc, uint32_t accumulate, uint64_t* bar) {
#define BT_UMMA_K_BLOCK(GROUP, COMMIT)                                                                       \
  asm volatile(                                                                                              \
      "{\n\t"                                                                                                \
      ".reg .pred p, q, t;\n\t"                                                                              \
      ".reg .b64 a1, a2, a3, b1, b2, b3, sa, sb;\n\t"                                                        \
      ".reg .b16 m;\n\t"                                                                                     \
      "cvt.u64.u32 sa, %3;\n\t"                                                                              \
      "cvt.u64.u32 sb, %4;\n\t"                                                                              \
      "add.u64 a1, %1, sa;\n\t"                                                                              \
      "add.u64 a2, a1, sa;\n\t"                                                                              \
      "add.u64 a3, a2, sa;\n\t"                                                                              \
      "add.u64 b1, %2, sb;\n\t"                                                                              \
      "add.u64 b2, b1, sb;\n\t"                                                                              \
      "add.u64 b3, b2, sb;\n\t"                                                                              \
      "mov.b16 m, 3;\n\t"                                                                                    \
      "elect.sync _|q, 0xffffffff;\n\t"                                                                      \
      "setp.ne.b32 p, %6, 0;\n\t"                                                                            \
      "setp.eq.u32 t, 0, 0;\n\t"                                                                             \
      "@q tcgen05.mma." GROUP ".kind::f16 [%0], %1, %2, %5, p;\n\t"                                          \
      "@q tcgen05.mma." GROUP ".kind::f16 [%0], a1, b1, %5, t;\n\t"                                          \
      "@q tcgen05.mma." GROUP ".kind::f16 [%0], a2, b2, %5, t;\n\t"                                          \
      "@q tcgen05.mma." GROUP ".kind::f16 [%0], a3, b3, %5, t;\n\t"                                          \
      "@q tcgen05.commit." GROUP ".mbarrier::arrive::one.shared::cluster" COMMIT ";\n\t"                     \
      "}\n" ::"r"(d_tmem),                                                                                   \
      "l"(adesc), "l"(bdesc), "r"(astep), "r"(bstep), "r"(idesc), "r"(accumulate), "r"(smem_u32(bar))        \
      : "memory")
  if (PAIR)
    BT_UMMA_K_BLOCK("cta_group::2", ".multicast::cluster.b64 [%7], m");
  else
    BT_UMMA_K_BLOCK("cta_group::1", ".b64 [%7]");
#undef BT_UMMA_K_BLOCK
}
// Arrive on `bar` once every tcgen05 operation issued so far by this thread is done.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// 32 lanes x 32 consecutive fp32 columns: thread i of the warp receives lane
// (base_lane + i), columns [col, col+32).  A warp may only touch the lane
// quarter (warp_id % 4) * 32.
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}

// tcgen05.ld 32x32b.x32 into elements [B, B + 32) of a longer register array (no address of the array
// is formed, so it stays in registers).
template <int B, int N>
__device__ __forceinline__ void tmem_ld_32x32_at(uint32_t taddr, uint32_t (&r)[N]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[B + 0]), "=r"(r[B + 1]), "=r"(r[B + 2]), "=r"(r[B + 3]), "=r"(r[B + 4]), "=r"(r[B + 5]), "=r"(r[B + 6]),
        "=r"(r[B + 7]), "=r"(r[B + 8]), "=r"(r[B + 9]), "=r"(r[B + 10]), "=r"(r[B + 11]), "=r"(r[B + 12]), "=r"(r[B + 13]),
        "=r"(r[B + 14]), "=r"(r[B + 15]), "=r"(r[B + 16]), "=r"(r[B + 17]), "=r"(r[B + 18]), "=r"(r[B + 19]), "=r"(r[B + 20]),
        "=r"(r[B + 21]), "=r"(r[B + 22]), "=r"(r[B + 23]), "=r"(r[B + 24]), "=r"(r[B + 25]), "=r"(r[B + 26]), "=r"(r[B + 27]),
        "=r"(r[B + 28]), "=r"(r[B + 29]), "=r"(r[B + 30]), "=r"(r[B + 31])
      : "r"(taddr)
      : "memory");
}
// Register -> tensor memory, same lane / column mapping as the loads above.
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ------------------------------------------------- UMMA descriptors (sm_100)
// Shared-memory matrix descriptor, 64 bit:
//   [ 0,14) start address >> 4      [16,30) leading byte offset >> 4
//   [32,46) stride byte offset >> 4 [46,48) version = 1
//   [49,52) base offset = 0         [61,64) layout: 0 none, 2 = 128-byte swizzle
// K-major, 128B swizzle  (rows of 64 fp16 = 128 B, 8-row groups of 1024 B):
//   SBO = distance between 8-row groups; LBO unused.
// MN-major, 128B swizzle (64 contiguous MN elements per k row, 8 k rows = 1024 B):
//   LBO = distance between 64-element chunks along MN; SBO = distance between
//   8-k groups.
__host__ __device__ constexpr uint64_t make_smem_desc_hi(uint32_t lbo_bytes, uint32_t sbo_bytes) {
  return (static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16) |
         (static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ uint64_t smem_desc(uint64_t hi_template, uint32_t smem_addr) {
  return hi_template | static_cast<uint64_t>((smem_addr >> 4) & 0x3FFFu);
}
// Instruction descriptor for kind::f16, fp16 A/B, fp32 D.
//   [4,6) D format 1 = f32; [7,10) A fmt 0 = f16; [10,13) B fmt 0 = f16;
//   bit 15 A major (0 K / 1 MN); bit 16 B major; [17,23) N>>3; [24,29) M>>4.
__host__ __device__ constexpr uint32_t make_idesc_f16(int M, int N, int a_mn_major, int b_mn_major) {
  return (1u << 4) | (static_cast<uint32_t>(a_mn_major) << 15) | (static_cast<uint32_t>(b_mn_major) << 16) |
         (static_cast<uint32_t>(N >> 3) << 17) | (static_cast<uint32_t>(M >> 4) << 24);
}

// -------------------------------------------------------------------- maths
__device__ __forceinline__ float gelu_erf(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
// Exact-form GELU, x * Phi(x), with one special-function op:
//   gelu(x) = max(x, 0) - 0.5 * |x| * erfc(|x| / sqrt(2)),   erfc(z) = 2^p(z),
// p = degree-5 polynomial fit of log2(erfc(z)) on [0, 4.3] (z is clamped there; beyond,
// erfc < 2e-9).  Maximum absolute error of the result against 0.5*x*(1+erf(x/sqrt 2)) in
// fp32 arithmetic: 6.4e-7 over x in [-8, 8] — far below fp16 resolution of the output.
__device__ __forceinline__ float gelu_erf_fast(float x) {
  const float ax = fabsf(x);
  const float z = fminf(ax * 0.70710678118654752f, 4.3f);
  float p = fmaf(-0.002677350537851453f, z, 0.02833780087530613f);
  p = fmaf(p, z, -0.1465892493724823f);
  p = fmaf(p, z, -0.9199854135513306f);
  p = fmaf(p, z, -1.6274596452713013f);
  p = fmaf(p, z, -3.764020948437974e-05f);
  float e;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(p));
  return fmaf(-0.5f * ax, e, fmaxf(x, 0.f));
}
// Two values at once with the packed fp32 instructions of sm_100 (fma.rn.f32x2: one issue slot for two
// lanes of a 64-bit register pair).
__device__ __forceinline__ unsigned long long pack_f32x2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long fma_f32x2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long add_f32x2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// gelu_erf_fast for two values, with the constants folded together: n = -|x|, clamped, takes the place of z, and the
// factor 1/2 is in the exponent,
//   gelu(x) = max(x, 0) + n * 2^q(n),   q(n) = p(-n / sqrt(2)) - 1.
// Maximum absolute error 6.4e-7 as above.  A NaN stays one (by way of the maximum; n drops it), and an infinity
// gives what its limit is.  Clocks for the GELU epilogue of a 128 x 256 tile by itself, eight warps: 4322 with the two
// halvings and the scaling as instructions of their own, 3787 so.
__device__ __forceinline__ void gelu_erf_fast_pair(float& x0, float& x1) {
  const unsigned long long n = pack_f32x2(fmaxf(-fabsf(x0), -6.0811183f), fmaxf(-fabsf(x1), -6.0811183f));
  unsigned long long q = fma_f32x2(pack_f32x2(0.00047329318476840854f, 0.00047329318476840854f), n, pack_f32x2(0.007084450218826532f, 0.007084450218826532f));
  q = fma_f32x2(q, n, pack_f32x2(0.05182712525129318f, 0.05182712525129318f));
  q = fma_f32x2(q, n, pack_f32x2(-0.4599927067756653f, -0.4599927067756653f));
  q = fma_f32x2(q, n, pack_f32x2(1.1507877111434937f, 1.1507877111434937f));
  q = fma_f32x2(q, n, pack_f32x2(-1.000037670135498f, -1.000037670135498f));
  float q0, q1, e0, e1, m0, m1;
  unpack_f32x2(q, q0, q1);
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(q0));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(q1));
  asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(m0) : "f"(x0));
  asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(m1) : "f"(x1));
  unpack_f32x2(fma_f32x2(n, pack_f32x2(e0, e1), pack_f32x2(m0, m1)), x0, x1);
}
// a += low half of h, b += high half: mixed-precision additions (one instruction each, no conversion first).
__device__ __forceinline__ void add_half2(float& a, float& b, uint32_t h) {
  asm("{\n\t"
      ".reg .f16 lo, hi;\n\t"
      "mov.b32 {lo, hi}, %2;\n\t"
      "add.f32.f16 %0, lo, %0;\n\t"
      "add.f32.f16 %1, hi, %1;\n\t"
      "}"
      : "+f"(a), "+f"(b)
      : "r"(h));
}
__device__ __forceinline__ float gelu_tanh(float x) {
  // 0.5 x (1 + tanh( sqrt(2/pi) (x + 0.044715 x^3) ))
  const float u = 0.7978845608028654f * x * (1.0f + 0.044715f * x * x);
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(u));
  return 0.5f * x * (1.0f + t);
}
__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

}  // namespace bt
