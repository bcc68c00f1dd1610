// Newton-Schulz GEMMs for sm_100a: D[M][N] = A * B^T on the 5th-generation tensor cores.
//
//   tcgen05.mma (kind::f16, BF16 or F16 operands, FP32 accumulators in TMEM), operands staged
//   in shared memory by TMA (cp.async.bulk.tensor, 128-byte swizzle), mbarrier pipeline,
//   warp-specialised persistent CTAs walking a tile list that spans every matrix of the plan.
//
// One kernel, three uses per iteration (crates/cuda-kernels/src/gpt/optimizer/muon/polar/
// fused.rs:64-92 in the reference):
//   Gram   G = X X^T                     (reference: tiles/symmetric.rs:28-40)
//   Poly   Q = c G G + b G + a I         (reference: tiles/symmetric.rs:42-65, store/plain.rs:175-178)
//   Apply  X' = Q X                      (reference: tiles.rs:14-38)
// Operands are read in their storage orientation: an operand whose reduction dimension is
// the slow one is described to the tensor core as MN-major, so no transpose is ever
// materialised.  Results go from registers straight to memory, a whole 32-byte sector per lane; the FP32 Gram
// values that the polynomial epilogue needs are kept in a private scratch in the order of the
// registers, so both sides access it fully coalesced.
//
// Tiles (the choice is in api.cu):
//   PAIR  : a cluster of two CTAs computes 256 x 256 or 128 x 128 with cta_group::2 MMAs.  Each CTA stages half of the rows
//           of A and half of those of B, so a k-block of 256 x 256 costs 32 KB of loads per SM instead of 48 KB, and one of
//           128 x 128 16 KB instead of the 32 KB that one CTA needs for it.  No multicast load is used.
//   single: one CTA computes 128 x BN (BN = 128 or 256).
// In every configuration a tile's sum runs over all of K in one order, so a matrix's result does not depend on which
// other matrices share its plan: a sharded run and a single GPU compute the same bits.  (Splitting K of the long Gram
// tiles of a small plan over several CTAs took one 3072 x 768 from 166 to 150 us and broke that.)
//
// What bounds it.
//   Many tiles.  A k-block (64 of K) of a 256 x 256 pair tile is 512 clocks of MMA, in which an SM takes in 32 KB, the 64
//   bytes per clock that it can (every shape comes to that rate, with 12 CTAs running or with 148), and its shared memory
//   serves 32 KB read and 32 KB written, 128 bytes per clock.  k-blocks take 510 to 630 clocks.  Beyond that the 1000 W cap
//   decides: with real data the clock falls to 1.4 - 1.7 GHz (GPT-2 small) and 1.1 - 1.4 (XL), where the same launches on
//   operands of zeros keep 1.8.  What the epilogue does to shared memory therefore counts twice, in port time and in energy:
//   through a slab for whole-line stores every result byte passed the port three times; directly from registers it passes
//   once (Newton-Schulz loop, before and after: 48 matrices of GPT-2 small 1284 -> 1213 us, six layers of XL 4625 -> 4450).
//   Whole lines without the slab, by exchanging pieces between the four lanes of a row, were slower for pairs (Apply of six
//   XL layers 334 -> 364 us).
//   Few tiles.  A launch is a chain: 2.0 us from the end of the launch in front to griddepcontrol.wait, 1.2 us to the first
//   MMA, the k-blocks at what an SM takes in (512 clocks where a CTA stages 32 KB of a k-block, 256 where it stages 16),
//   and the epilogue, 1400 clocks for 32 columns a warp.  That was 2500 while the arrival that hands an accumulator back had
//   release semantics at cluster scope, which waits for the thread's stores.
//   A thread spends 115 (one 3072 x 768) to 195 clocks (GPT-2 small, XL) on issuing a copy, beside the barrier rounds.  One for
//   both operands was the slowest role of the pipeline, so each operand has a producer of its own and takes one copy per k-block;
//   an MN-major operand of 128 rows is one copy of a three-dimensional map instead of two (six layers of XL 4280 -> 4160 us).
//   The MMA loop is warp-uniform, and a scheduler warp keeps a ring of decoded tiles in shared memory: the tile list and the
//   problem table are two dependent reads of L2.
//
// Three ways to launch the loop (the template parameter CHAINED separates the first from the other two), and a fourth for
// matrices that fit one SM (k_ns_small below):
//   per phase : one launch per GEMM flavour and iteration, tiles dealt round-robin, launches chained with
//               programmatic dependent launch.  The default.
//   chained   : one persistent grid over a work list of every tile of every iteration; CTAs draw tiles with an
//               atomic ticket and a per-matrix progress count orders a tile after the tiles it reads from.
//   fused     : a ticketed launch whose entries are a Gram tile AND the polynomial tile of the same position:
//               the FP32 Gram accumulator stays in tensor memory between the two.
//
// Every mbarrier wait, ring read and dependency wait is bounded: on expiry the CTA raises a status word, drains
// and frees its TMEM before returning.
#include <algorithm>

#include <cuda.h>

#include "common.cuh"
#include "internal.h"

namespace b2 {

namespace {

constexpr int kBoxBytes = 64 * 128;          // 64 rows x 128 bytes
constexpr int kSmemLimit = 227 * 1024;
constexpr uint32_t kSpinLimit = 1u << 24;    // hard cap on polls, whatever the timer says
constexpr uint64_t kWaitLimitNs = 2000000000ull;

// TM x BN is the tile of a CTA, or of a pair of CTAs; a pair's CTAs hold half of its rows of A and half of its rows of B each.
template <int TM, int BN, bool PAIR, bool CHAINED>
struct Cfg {
    static constexpr int kTileM = TM;
    static constexpr int kRows = PAIR ? TM / 2 : TM;        // output rows of this CTA, and rows of A it stages per k-block
    static constexpr int kBRows = PAIR ? BN / 2 : BN;       // rows of B this CTA stages per k-block
    static constexpr int kABytes = kRows * 128, kBBytes = kBRows * 128;
    static constexpr int kKbBytes = kABytes + kBBytes;
    // k-blocks per pipeline stage: with 16 KB each, one per stage would leave the roles 256 clocks for a barrier round
    static constexpr int kStageKb = kKbBytes <= 16 * 1024 ? 2 : 1;
    static constexpr int kStageBytes = kStageKb * kKbBytes;
    // An accumulator of 64 rows per CTA lies in all 128 lanes: columns 0 .. BN/2-1 in lanes 0 .. 63, the others above.
    static constexpr int kAccCols = kRows == 64 ? BN / 2 : BN;
    // warp 0: TMA producer of A, warp 1: MMA issuer, then four epilogue warps (one per TMEM lane quarter) for every
    // kEpiCols tensor-memory columns, the TMA producer of B and the tile scheduler.  Narrow tiles: 32 columns a warp shorten
    // the epilogue, but in the ticketed form every warp publishes its part of a tile with a fence and an atomic, and twice as
    // many of these cost more than that (128 x 128, one CTA, 32 -> 64 columns in the chained loop: one layer of width 768
    // 247 -> 215 us, the eighth of GPT-2 small 302 -> 265; launch per phase 203 with 32).
    static constexpr int kEpiCols = BN == 256 || CHAINED ? 64 : 32;
    static constexpr int kEpiWarps = 4 * (kAccCols / kEpiCols);
    static constexpr int kProducerA = 0, kMmaWarp = 1, kEpiWarp0 = 2, kProducerB = 2 + kEpiWarps, kSchedulerWarp = 3 + kEpiWarps;
    static constexpr int kThreads = 32 * (4 + kEpiWarps);
    static constexpr int kTmemCols = 2 * kAccCols;
    static constexpr int kBarrierBytes = 768;   // mbarriers, flags, the tile ring and the hand-over ring of the chained launch
    static_assert(kRows == 128 || (kRows == 64 && kBRows == 64), "boxes of the operand maps");
    static constexpr int kMaxStages = (kSmemLimit - kBarrierBytes - 1024) / kStageBytes;
    static constexpr int kStages = kMaxStages < 8 ? kMaxStages : 8;
    static constexpr int kSmemBytes = kStages * kStageBytes + kBarrierBytes + 1024;
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
// shared::cluster address of the same offset in CTA `rank` of this cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ uint32_t cluster_cta_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Arrive on a barrier given by its shared::cluster address (own or peer CTA).  For tensor memory that has been read, whose order
// tcgen05.fence::before_thread_sync keeps: relaxed, because release semantics at cluster scope would make the thread wait for
// its stores.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok;
}
// Non-blocking probe of a barrier phase.  (mbarrier.try_wait may suspend the thread for a system-dependent time,
// measured here at about 5 us, before it reports that the phase is not complete; that is right for a wait, not
// for a probe.)
__device__ __forceinline__ uint32_t mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok;
}
__device__ __forceinline__ uint64_t global_timer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Bounded wait (about two seconds of wall clock).  Returns false when the limit ran out or
// another role of this CTA already gave up.
__device__ __noinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity, volatile uint32_t *abort_flag) {
#pragma unroll 1
    for (int it = 0; it < 128; ++it)
        if (mbar_try_wait(bar, parity)) return true;
    const uint64_t start = global_timer_ns();
#pragma unroll 1
    for (uint32_t it = 0; it < kSpinLimit; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if (global_timer_ns() - start > kWaitLimitNs) break;
        __nanosleep(it >= 1024 ? 256 : 32);
    }
    *abort_flag = 1;
    return false;
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile uint32_t *abort_flag) {
    return mbar_try_wait(bar, parity) || mbar_wait_slow(bar, parity, abort_flag);
}

__device__ __forceinline__ uint32_t ld_acquire_gpu(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t ld_relaxed_gpu(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// orders this thread's generic-proxy accesses against its async-proxy ones (TMA loads and stores)
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }

// Chained launch: words shared by every CTA.  All zero between launches; the last CTA to leave clears them.
struct ChainSync {
    uint32_t abort;      // a bounded wait ran out somewhere: everybody leaves
    uint32_t exited;
    uint32_t ticket;     // next unclaimed entry of the work list
    uint32_t reserved;
    uint32_t progress[1];  // per slot: epilogue warps that have finished a tile of the slot, over all phases
};
// Bounded wait until `*counter >= need`.  Returns false when the limit ran out or the launch is aborting.
//
// How a tile's outputs reach the CTA that reads them.  Every lane of the writer's epilogue warp orders its
// stores before what follows (__threadfence), the warp converges, and one lane raises the matrix's progress
// count with an atomic.
// The reader polls the count with relaxed loads that bypass L1; once it is high enough it reads it once more
// with acquire semantics and issues fence.proxy.async before its first TMA copy, which is what the PTX memory
// model asks for between a generic-proxy flag and async-proxy accesses.  Both fences were measured against a
// build without them: no difference beyond run-to-run noise.
__device__ __forceinline__ bool chain_wait(const uint32_t *counter, uint32_t need, uint32_t *launch_abort,
                                           volatile uint32_t *abort_flag) {
    if (ld_relaxed_gpu(counter) >= need) return true;
    const uint64_t start = global_timer_ns();
#pragma unroll 1
    for (uint32_t it = 0; it < kSpinLimit; ++it) {
        if (ld_relaxed_gpu(counter) >= need) return true;
        if (*abort_flag || ld_relaxed_gpu(launch_abort) != 0u) break;
        if (global_timer_ns() - start > kWaitLimitNs) break;
        __nanosleep(it >= 64 ? 128 : 20);
    }
    *abort_flag = 1;
    atomicExch(launch_abort, 1u);
    return false;
}

// Chained launch: which tile a CTA pair works on next is decided at run time (an atomic ticket over the work list,
// claimed by the leader's scheduler), so the peer CTA learns it through a small ring in its shared memory: entry k
// holds (k + 1) << 32 | tile for the k-th tile of the pair.  The leader's scheduler is never more than the tile ring
// and the pipeline ahead of the peer's, far less than this ring's length.
constexpr uint32_t kHandRing = 16;
constexpr uint32_t kNoTile = 0xffffffffu;
__device__ __forceinline__ void hand_put(uint32_t hand_cluster_addr, uint32_t seq, uint32_t tile) {
    const uint64_t v = ((uint64_t)(seq + 1u) << 32) | tile;
    asm volatile("st.volatile.shared::cluster.u64 [%0], %1;" ::"r"(hand_cluster_addr + 8u * (seq % kHandRing)), "l"(v)
                 : "memory");
}
// Bounded: gives kNoTile when the CTA is aborting or nothing arrives within the wait limit.
__device__ __forceinline__ uint32_t hand_get(volatile uint64_t *ring, uint32_t seq, volatile uint32_t *abort_flag) {
    const uint64_t want = (uint64_t)(seq + 1u);
    uint64_t v = ring[seq % kHandRing];
    if ((v >> 32) == want) return (uint32_t)v;
    const uint64_t start = global_timer_ns();
#pragma unroll 1
    for (uint32_t it = 0; it < kSpinLimit; ++it) {
        v = ring[seq % kHandRing];
        if ((v >> 32) == want) return (uint32_t)v;
        if (*abort_flag) return kNoTile;
        if (global_timer_ns() - start > kWaitLimitNs) break;
        __nanosleep(20);
    }
    *abort_flag = 1;
    return kNoTile;
}

template <bool PAIR>
__device__ __forceinline__ void tma_load_2d(uint32_t dst, uint64_t map, uint32_t bar, int x, int y) {
    if (PAIR)
        asm volatile(
            "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
            ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y)
            : "memory");
    else
        asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
            ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y)
            : "memory");
}
template <bool PAIR>
__device__ __forceinline__ void tma_load_3d(uint32_t dst, uint64_t map, uint32_t bar, int x, int y, int z) {
    if (PAIR)
        asm volatile(
            "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
            ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z)
            : "memory");
    else
        asm volatile(
            "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
            ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z)
            : "memory");
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Arrive on `bar` once every MMA issued so far has retired.  PAIR: the arrival is delivered
// to the barrier at this offset in both CTAs of the pair.
template <bool PAIR>
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    if (PAIR)
        asm volatile(
            "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
            ::"r"(bar), "h"((uint16_t)3)
            : "memory");
    else
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                     : "memory");
}
template <bool PAIR>
__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                       uint32_t accumulate) {
    if (PAIR)
        asm volatile(
            "{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p; }"
            ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    else
        asm volatile(
            "{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }"
            ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
}
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile("{ .reg .pred p; elect.sync _|p, 0xffffffff; selp.u32 %0, 1, 0, p; }" : "=r"(r));
    return r != 0u;
}
// 32 lanes x 32 consecutive 32-bit columns: thread i of the warp receives row (lane base + i).
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t *r) {
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
// 32 lanes x 16 consecutive 32-bit columns
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t *r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
// 16 lanes x 64 consecutive 32-bit columns, in the layout of an MMA accumulator: thread i receives columns 8 j + 2 (i % 4) and
// the next one of row i / 4 in r[4 j], r[4 j + 1], those of row 8 + i / 4 in r[4 j + 2], r[4 j + 3].
__device__ __forceinline__ void tc_ld_16x64(uint32_t taddr, uint32_t *r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x8.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
// Four words of each of four neighbouring lanes, transposed: word k of lane s becomes word s of lane k.
__device__ __forceinline__ void quad_transpose(uint32_t &w0, uint32_t &w1, uint32_t &w2, uint32_t &w3, uint32_t lane) {
    const bool odd = lane & 1u, high = lane & 2u;
    const uint32_t p = __shfl_xor_sync(0xffffffffu, odd ? w0 : w1, 1), r = __shfl_xor_sync(0xffffffffu, odd ? w2 : w3, 1);
    if (odd) { w0 = p; w2 = r; } else { w1 = p; w3 = r; }
    const uint32_t t = __shfl_xor_sync(0xffffffffu, high ? w0 : w2, 2), u = __shfl_xor_sync(0xffffffffu, high ? w1 : w3, 2);
    if (high) { w0 = t; w1 = u; } else { w2 = t; w3 = u; }
}
// 32 bytes, one sector, to a 32-byte aligned address
__device__ __forceinline__ void st_global_32(void *p, const uint32_t *v) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
                 "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ void tc_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor, 128-byte swizzle, descriptor version 1 (sm_100).
//   K-major operand  (rows = M/N index, 128 bytes of K per row): 8-row groups are 1024 bytes
//   apart (stride byte offset); the leading byte offset is unused.
//   MN-major operand (rows = K index, 128 bytes = 64 M/N elements per row): 8-row groups of K
//   are 1024 bytes apart (stride), 64-element groups of M/N are one 64 x 64 box (8192 bytes)
//   apart (leading).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3ffffu) >> 4);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3fffu) << 16;
    d |= (uint64_t)((sbo_bytes >> 4) & 0x3fffu) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// Instruction descriptor for kind::f16: FP32 accumulate, A/B format F16 (0) or BF16 (1),
// per-operand major bit, N >> 3 at bit 17, M >> 4 at bit 24.
__device__ __forceinline__ uint32_t instr_desc(int m, int n, int f16, uint32_t a_mn, uint32_t b_mn) {
    uint32_t fmt = f16 ? 0u : 1u;
    return (1u << 4) | (fmt << 7) | (fmt << 10) | (a_mn << 15) | (b_mn << 16) |
           ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// What the roles of a CTA need to know about the tile they work on, written by the CTA's scheduler warp into a
// small ring in shared memory.  The tile list and the problem table are two dependent reads of L2 (about 700 clocks
// each); with the ring they are off the path of the roles, which read an entry in a few tens of clocks.
struct alignas(16) TileEntry {
    uint64_t map_a, map_b;   // tensor maps of the operands
    uint64_t out;            // 16-bit result, or the FP32 one (kEpiApplyLast)
    uint64_t frag;
    uint32_t M, N, num_kb, pitch_bytes;
    uint32_t tile;           // tile_m | tile_n << 16
    uint32_t flags;
    uint32_t frag_units, slot;
};
static_assert(sizeof(TileEntry) == 64, "control region layout");
constexpr uint32_t kRing = 4;
// flags of an entry
constexpr uint32_t kTileAMn = 1u, kTileBMn = 2u, kTileMirror = 4u;
constexpr uint32_t kTileShared = 8u;      // B is the A tile: loaded once, read twice
constexpr uint32_t kTileDependent = 16u;  // the operands were written by this launch
constexpr uint32_t kTileEnd = 32u;        // no more tiles
constexpr int kTileEpiShift = 8, kTileScaleShift = 12, kTileIterShift = 16, kTileNShift = 24;

// Fills in everything but `flags` bits that come from the list entry.  The MMA's N is the width of the tile that
// exists, rounded up: a 1600-wide output has a last tile column of 64, which a 256-wide MMA would spend four times as
// long on.  K-major B: steps of 64 (a pair splits N in two halves of at least 32 rows); MN-major B: steps of 128, so
// that each half is made of whole 64-element swizzle atoms.
template <typename C, int BN, bool PAIR>
__device__ __forceinline__ void fill_entry(TileEntry &e, const GemmProblem *p, uint32_t tile_m, uint32_t tile_n, uint32_t epilogue,
                                           uint32_t flags) {
    e.map_a = p->map_a;
    e.map_b = p->map_b;
    e.frag = p->frag32;
    e.M = p->M;
    e.N = p->N;
    e.num_kb = (p->K + kGemmBlockK - 1) / kGemmBlockK;
    e.frag_units = p->frag_units;
    const bool last = epilogue == kEpiApplyLast;
    e.out = last ? p->out32 : p->out16;
    e.pitch_bytes = last ? p->pitch32 * 4u : p->pitch16 * 2u;
    e.tile = tile_m | (tile_n << 16);
    const uint32_t a_mn = p->a_mn_major, b_mn = p->b_mn_major;
    const uint32_t step = b_mn ? 128u : 64u;
    const uint32_t left = e.N - tile_n * BN;
    // (64 rows per CTA: always BN, which fixes where the columns lie in tensor memory)
    const uint32_t n_mma = C::kRows == 64 ? (uint32_t)BN : min((uint32_t)BN, (left + step - 1u) / step * step);
    // a diagonal tile of X X^T or G G: this CTA's rows of B are its rows of A, in the same shared-memory layout
    const bool shared = C::kTileM == BN && tile_m == tile_n && e.map_a == e.map_b && a_mn == b_mn && n_mma == (uint32_t)BN;
    e.flags = flags | (a_mn ? kTileAMn : 0u) | (b_mn ? kTileBMn : 0u) | (shared ? kTileShared : 0u) |
              (epilogue << kTileEpiShift) | ((n_mma / 32u) << kTileNShift);
}

template <int TM, int BN, bool PAIR, bool CHAINED>
__global__ void __launch_bounds__((Cfg<TM, BN, PAIR, CHAINED>::kThreads), 1)
k_ns_gemm(const GemmProblem *__restrict__ problems, const void *__restrict__ tiles,
          uint32_t tile_count, uint32_t epilogue_arg, int f16, GemmCoefficients coef,
          const float *__restrict__ slot_scale, uint32_t scale_pow_arg, uint32_t *status, ChainSync *sync,
          uint32_t slot_count) {
    using C = Cfg<TM, BN, PAIR, CHAINED>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *stage_base = smem;
    uint8_t *control = smem + C::kStages * C::kStageBytes;
    uint64_t *bars = reinterpret_cast<uint64_t *>(control);
    // bars: full[S], empty[S], tmem_full[2], tmem_empty[2], ring_full[kRing], ring_empty[kRing]
    constexpr int kBars = 2 * C::kStages + 4 + 2 * (int)kRing;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + kBars);
    volatile uint32_t *abort_flag = tmem_slot + 1;
    TileEntry *ring = reinterpret_cast<TileEntry *>(control + 256);
    volatile uint64_t *hand = reinterpret_cast<volatile uint64_t *>(control + 256 + kRing * sizeof(TileEntry));
    static_assert(kBars * 8 + 8 <= 256 && 256 + kRing * sizeof(TileEntry) + kHandRing * 8 <= C::kBarrierBytes, "control region layout");

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = PAIR ? cluster_cta_rank() : 0u;       // 0 = leader of the pair
    const uint32_t first_tile = PAIR ? blockIdx.x / 2 : blockIdx.x;
    const uint32_t tile_stride = PAIR ? gridDim.x / 2 : gridDim.x;
    const uint32_t bar0 = smem_u32(bars);
    auto full_bar = [&](uint32_t s) { return bar0 + 8u * s; };
    auto empty_bar = [&](uint32_t s) { return bar0 + 8u * (C::kStages + s); };
    auto tfull_bar = [&](uint32_t a) { return bar0 + 8u * (2 * C::kStages + a); };
    auto tempty_bar = [&](uint32_t a) { return bar0 + 8u * (2 * C::kStages + 2 + a); };
    auto ring_full = [&](uint32_t k) { return bar0 + 8u * (2 * C::kStages + 4 + k % kRing); };
    auto ring_empty = [&](uint32_t k) { return bar0 + 8u * (2 * C::kStages + 4 + kRing + k % kRing); };
    auto ring_parity = [&](uint32_t k) { return (k / kRing) & 1u; };

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::kStages; ++s) {
            mbar_init(full_bar(s), 2);    // one arrival from each of the leader's two TMA producers
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(tfull_bar(a), 1);
            mbar_init(tempty_bar(a), PAIR ? 2 * C::kEpiWarps : C::kEpiWarps);
        }
        for (uint32_t k = 0; k < kRing; ++k) {
            mbar_init(ring_full(k), 1);
            mbar_init(ring_empty(k), C::kEpiWarps + 2 + (rank == 0 ? 1 : 0));
        }
        *abort_flag = 0;
        if (CHAINED)
            for (uint32_t k = 0; k < kHandRing; ++k) hand[k] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (warp == C::kMmaWarp) {
        if (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                         "r"((uint32_t)C::kTmemCols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                         "r"((uint32_t)C::kTmemCols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync_all();  // the peer's barriers are initialised before anything signals them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // Programmatic dependent launch: the next launch of the stream may start its own prologue on SMs this grid has
    // left.  What the previous launch wrote may be read only below the wait (a no-op without the launch attribute);
    // the tile list, the problem table and the tensor maps belong to the plan, so the scheduler warp of a plain launch
    // does not wait and has the first entries in the ring, and their tensor maps fetched, by then.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (CHAINED || warp != C::kSchedulerWarp) asm volatile("griddepcontrol.wait;" ::: "memory");

    if (warp == C::kSchedulerWarp) {
        // ------------------------------------------------------------------ tile scheduler
        if (lane == 0) {
            uint32_t k = 0;   // ring sequence number
            bool ok = true;
            auto claim_slot = [&]() { return mbar_wait(ring_empty(k), ring_parity(k) ^ 1u, abort_flag); };
            auto publish_entry = [&]() {
                mbar_arrive(ring_full(k));
                ++k;
            };
            if (!CHAINED) {
                // tile first_tile + i * tile_stride; the list is read one tile ahead
                const GemmTile *list = reinterpret_cast<const GemmTile *>(tiles);
                uint32_t t = first_tile;
                GemmTile next = {};
                if (t < tile_count) next = list[t];
                while (t < tile_count) {
                    const GemmTile tl = next;
                    t += tile_stride;
                    if (t < tile_count) next = list[t];
                    if (!claim_slot()) { ok = false; break; }
                    TileEntry &e = ring[k % kRing];
                    fill_entry<C, BN, PAIR>(e, problems + tl.problem, tl.tile_m, tl.tile_n, epilogue_arg,
                                         (tl.reserved ? kTileMirror : 0u) | (scale_pow_arg << kTileScaleShift));
                    e.slot = tl.problem;
                    if (k < 2) {
                        asm volatile("prefetch.tensormap [%0];" ::"l"(e.map_a) : "memory");
                        asm volatile("prefetch.tensormap [%0];" ::"l"(e.map_b) : "memory");
                    }
                    publish_entry();
                }
            } else {
                // The leader claims list entries in order with an atomic ticket (a tile only ever waits for tiles with
                // smaller tickets, which running CTAs hold, so the launch makes progress however many CTAs are
                // resident; the CTAs stay within a few tiles of each other in the list, which keeps a matrix's
                // operands in L2 while its tiles are worked on; and a slower SM simply takes fewer tiles) and hands
                // them to the peer CTA.  An entry goes into the ring once the tiles it reads from have been stored and
                // published.  A fused Gram + polynomial entry becomes two; its second part waits for tiles with LARGER
                // tickets, and the next ticket is drawn only after that wait, so a CTA never sits on a ticket it has
                // not started while it waits for one.
                const bool claims = !PAIR || rank == 0;
                const uint32_t peer_hand = PAIR ? map_to_cta(smem_u32(const_cast<uint64_t *>(hand)), 1) : 0u;
                for (uint32_t seq = 0; ok; ++seq) {
                    uint32_t t;
                    if (claims) {
                        t = atomicAdd(&sync->ticket, 1u);
                        if (PAIR) hand_put(peer_hand, seq, t);
                    } else {
                        t = hand_get(hand, seq, abort_flag);
                    }
                    if (t >= tile_count) break;
                    const uint4 c = __ldg(reinterpret_cast<const uint4 *>(tiles) + 2 * (size_t)t);
                    const uint4 d = __ldg(reinterpret_cast<const uint4 *>(tiles) + 2 * (size_t)t + 1);
                    const uint32_t slot = c.z & 0xffffu, epilogue = (c.z >> 16) & 0xffu;
                    const bool two = epilogue == kEpiGramPoly;
                    const uint32_t flags = (((c.z >> 24) & 1u) ? kTileMirror : 0u) | (((c.z >> 25) & 3u) << kTileScaleShift) |
                                           (((c.z >> 27) & 31u) << kTileIterShift);
                    for (uint32_t part = 0; ok && part < (two ? 2u : 1u); ++part) {
                        const uint32_t need = part ? d.y : c.w;
                        if (need != 0u) {
                            if (!chain_wait(&sync->progress[slot], need, &sync->abort, abort_flag)) { ok = false; break; }
                            (void)ld_acquire_gpu(&sync->progress[slot]);
                        }
                        if (!claim_slot()) { ok = false; break; }
                        TileEntry &e = ring[k % kRing];
                        fill_entry<C, BN, PAIR>(e, problems + (part ? d.x : c.x), c.y & 0xffffu, c.y >> 16,
                                             two ? (part ? kEpiPolyFused : kEpiGramHold) : epilogue,
                                             flags | (need != 0u ? kTileDependent : 0u));
                        e.slot = slot;
                        publish_entry();
                    }
                }
            }
            if (ok && claim_slot()) {
                ring[k % kRing].flags = kTileEnd;
                publish_entry();
            }
        }
    } else if (warp == C::kProducerA || warp == C::kProducerB) {
        // ------------------------------------------------------------------ TMA producers, one per operand
        if (lane == 0) {
            const bool for_b = warp == C::kProducerB;
            const uint32_t leader_full = PAIR ? map_to_cta(full_bar(0), 0) : full_bar(0);
            uint32_t stage = 0, phase = 0, turn = 0;   // turn: parity of the k-blocks so far, over all tiles
            bool ok = true;
            for (uint32_t k = 0; ok; ++k) {
                if (!mbar_wait(ring_full(k), ring_parity(k), abort_flag)) break;
                const TileEntry &e = ring[k % kRing];
                const uint32_t flags = e.flags, tile = e.tile;
                const int num_kb = (int)e.num_kb;
                const uint64_t map_a = e.map_a, map_b = e.map_b;
                mbar_arrive(ring_empty(k));
                if (flags & kTileEnd) break;
                // the operands were stored by other CTAs of this launch: the scheduler has seen their counts
                if (CHAINED && (flags & kTileDependent)) fence_proxy_async_all();
                // A tile whose B is its A: the two producers take every other k-block.  (Both have to take part: a
                // producer that the pipeline could do without might fall two phases of a stage's barrier behind, or run
                // two ahead, and a parity wait cannot tell two phases apart.)
                const bool shared = (flags & kTileShared) != 0u;
                const bool as_b = for_b && !shared;
                const uint64_t map = as_b ? map_b : map_a;
                const bool mn = (flags & (as_b ? kTileBMn : kTileAMn)) != 0u;
                const int n_half = (int)(flags >> kTileNShift) * 16;   // half of the MMA's N
                const int row0 = as_b ? (int)(tile >> 16) * BN + (PAIR ? (int)rank * n_half : 0)
                                      : (int)(tile & 0xffffu) * C::kTileM + (int)rank * C::kRows;
                const uint32_t dst0 = smem_u32(stage_base) + (as_b ? (uint32_t)C::kABytes : 0u);
                const int operand_rows = as_b ? C::kBRows : C::kRows;
                for (int kb = 0; kb < num_kb; kb += C::kStageKb) {
                    turn ^= 1u;
                    if (!shared || turn == (for_b ? 1u : 0u)) {
                        const int subs = min(C::kStageKb, num_kb - kb);
                        if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag)) { ok = false; break; }
                        if (!PAIR || rank == 0) {
                            // PAIR: both CTAs' copies complete on the leader's barrier, which expects the bytes of both
                            mbar_expect_tx(full_bar(stage), (uint32_t)(operand_rows * 128 * subs) * (PAIR ? 2u : 1u));
                            if (shared) mbar_arrive(full_bar(stage));   // in the other producer's place
                        }
                        const uint32_t fb = leader_full + 8u * stage;
#pragma unroll
                        for (int sub = 0; sub < C::kStageKb; ++sub) {
                            if (sub >= subs) break;
                            const uint32_t dst = dst0 + stage * (uint32_t)C::kStageBytes + sub * C::kKbBytes;
                            const int k0 = (kb + sub) * kGemmBlockK;
                            if (C::kRows == 64) {   // (B has 64 rows too) one box of 64 x 64: x = M or N index, y = K index, or K, rows
                                tma_load_2d<PAIR>(dst, map, fb, mn ? row0 : k0, mn ? k0 : row0);
                            } else {
#pragma unroll
                                for (int j = 0; j < (C::kBRows > 128 ? 2 : 1); ++j) {
                                    if (128 * j >= operand_rows) break;
                                    // 128 rows: two boxes of 64 x 64, z = M or N index / 64, or one of 64 (K) x 128
                                    if (mn) tma_load_3d<PAIR>(dst + j * 16384, map, fb, 0, k0, row0 / 64 + 2 * j);
                                    else tma_load_2d<PAIR>(dst + j * 16384, map, fb, k0, row0 + 128 * j);
                                }
                            }
                        }
                    }
                    if (++stage == C::kStages) { stage = 0; phase ^= 1u; }
                }
            }
        }
    } else if (warp == C::kMmaWarp) {
        // ------------------------------------------------------------------ MMA issuer
        // The whole warp walks the loop and one elected lane issues: with warp-uniform control flow and operands the
        // issue of a k-block is about 100 clocks shorter than from a single diverged lane.
        if (rank == 0) {
            const uint64_t desc0 = smem_desc(__shfl_sync(0xffffffffu, smem_u32(stage_base), 0), 0, 1024);
            const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
            uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0;
            bool ok = true;
            for (uint32_t k = 0; ok; ++k) {
                if (!__all_sync(0xffffffffu, mbar_wait(ring_full(k), ring_parity(k), abort_flag))) break;
                const uint32_t flags = __shfl_sync(0xffffffffu, ring[k % kRing].flags, 0);
                const uint32_t num_kb = __shfl_sync(0xffffffffu, ring[k % kRing].num_kb, 0);
                __syncwarp();
                if (lane == 0) mbar_arrive(ring_empty(k));
                if (flags & kTileEnd) break;
                const uint32_t a_mn = flags & kTileAMn ? 1u : 0u, b_mn = flags & kTileBMn ? 1u : 0u;
                const uint32_t idesc = instr_desc(C::kTileM, (int)(flags >> kTileNShift) * 32, f16, a_mn, b_mn);
                // leading byte offset (unused by a K-major operand) and the step of 16 in K, in units of 16 bytes
                const uint64_t a0 = desc0 + ((uint64_t)(a_mn ? kBoxBytes >> 4 : 1) << 16);
                const uint64_t b0 = desc0 + ((uint64_t)(b_mn ? kBoxBytes >> 4 : 1) << 16) + (flags & kTileShared ? 0u : (uint32_t)(C::kABytes >> 4));
                const uint32_t a_step = a_mn ? 128u : 2u, b_step = b_mn ? 128u : 2u;
                if (!__all_sync(0xffffffffu, mbar_wait(tempty_bar(acc), acc_phase ^ 1u, abort_flag))) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem + acc * C::kAccCols;
                for (uint32_t kb = 0; kb < num_kb; kb += C::kStageKb) {
                    if (!__all_sync(0xffffffffu, mbar_wait(full_bar(stage), phase, abort_flag))) { ok = false; break; }
                    tc_fence_after();
                    const uint64_t ad = a0 + stage * (uint32_t)(C::kStageBytes >> 4), bd = b0 + stage * (uint32_t)(C::kStageBytes >> 4);
                    if (elect_one()) {
#pragma unroll
                        for (uint32_t sub = 0; sub < (uint32_t)C::kStageKb; ++sub) {
                            if (C::kStageKb > 1 && kb + sub >= num_kb) break;
#pragma unroll
                            for (uint32_t j = 0; j < kGemmBlockK / 16; ++j)
                                tc_mma<PAIR>(d_tmem, ad + sub * (uint32_t)(C::kKbBytes >> 4) + j * a_step,
                                             bd + sub * (uint32_t)(C::kKbBytes >> 4) + j * b_step, idesc,
                                             sub != 0 || j != 0 ? 1u : (uint32_t)(kb != 0));
                        }
                        tc_commit<PAIR>(empty_bar(stage));
                        if (kb + C::kStageKb >= num_kb) tc_commit<PAIR>(tfull_bar(acc));
                    }
                    __syncwarp();
                    if (++stage == C::kStages) { stage = 0; phase ^= 1u; }
                }
                acc ^= 1u;
                if (acc == 0) acc_phase ^= 1u;
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue warps
        // Warp w may read TMEM lanes 32 (w % 4) .. +31; the warps of a lane quarter each take kEpiCols columns, so an
        // accumulator buffer is free again after that many have been read.  Results go from registers to memory in 32-byte
        // pieces, one whole sector per lane: through a slab in shared memory, for stores of whole 128-byte lines, every byte
        // would pass the shared-memory port twice more, and that port is what the MMAs and their operands fill.
        const int q = warp & 3;
        const int chunk = (warp - C::kEpiWarp0) >> 2;
        const int taddr_col = chunk * C::kEpiCols;
        // rows and columns of the tile: 64 rows per CTA lie in two halves of the lanes
        const int c0 = taddr_col + (C::kRows == 64 ? (q >> 1) * (BN / 2) : 0);
        const int row_in_cta = 32 * (C::kRows == 64 ? q & 1 : q) + lane;
        const uint32_t tempty_leader0 = PAIR ? map_to_cta(tempty_bar(0), 0) : tempty_bar(0);
        uint32_t acc = 0, acc_phase = 0;
        // Chained launch: a finished tile is published to the other CTAs by raising its matrix's progress count
        // once this warp's stores are ordered before it (every lane fences its own).  The fence is put off until
        // the next tile's accumulator has been read (the stores then had that long to land) unless the next
        // accumulator is not ready yet, in which case it is done first: a warp never blocks on other CTAs with a
        // count unpublished.
        constexpr uint32_t kNoSlot = 0xffffffffu;
        uint32_t unpublished = kNoSlot;
        auto publish = [&]() {
            __threadfence();
            __syncwarp();
            if (lane == 0) atomicAdd(&sync->progress[unpublished], 1u);
            unpublished = kNoSlot;
        };
        for (uint32_t k = 0;; ++k) {
            if (CHAINED && unpublished != kNoSlot && !__all_sync(0xffffffffu, mbar_test(ring_full(k), ring_parity(k)))) publish();
            if (!__all_sync(0xffffffffu, mbar_wait(ring_full(k), ring_parity(k), abort_flag))) break;
            const TileEntry &entry = ring[k % kRing];
            const uint32_t flags = entry.flags, M = entry.M, N = entry.N, slot = entry.slot;
            uint8_t *out = reinterpret_cast<uint8_t *>(entry.out);
            const size_t pitch = entry.pitch_bytes;
            const uint64_t entry_frag = entry.frag;
            const int tile_m = (int)(entry.tile & 0xffffu), tile_n = (int)(entry.tile >> 16);
            const uint32_t frag_units = entry.frag_units;
            __syncwarp();
            if (lane == 0) mbar_arrive(ring_empty(k));
            if (flags & kTileEnd) break;
            const uint32_t epilogue = CHAINED ? (flags >> kTileEpiShift) & 15u : epilogue_arg;
            const uint32_t scale_pow = (flags >> kTileScaleShift) & 3u;
            // the iteration's coefficient triple, picked without indexing the argument block by a register
            float ca = coef.v[0], cb = coef.v[1], cc = coef.v[2];
            if (CHAINED) {
                const uint32_t iter = (flags >> kTileIterShift) & 31u;
#pragma unroll
                for (uint32_t i = 1; i < kMaxChainIterations; ++i)
                    if (iter == i) { ca = coef.v[3 * i]; cb = coef.v[3 * i + 1]; cc = coef.v[3 * i + 2]; }
            }
            const bool hold = CHAINED && epilogue == kEpiGramHold;    // the accumulator stays for the next part
            const bool fused = CHAINED && epilogue == kEpiPolyFused;  // combines with the held accumulator
            // symmetric outputs (Gram, Poly): tiles below the diagonal are not computed; the tile
            // above writes them as its transpose (reference: tiles/symmetric.rs:76-92)
            const bool mirror = (flags & kTileMirror) != 0u;
            const int grow = tile_m * C::kTileM + (int)rank * C::kRows + row_in_cta;   // this lane's row
            const int warp_row0 = grow - lane, col0 = tile_n * BN + c0;
            const bool in_range = col0 < (int)N && warp_row0 < (int)M;   // warp-uniform
            // FP32 Gram values: [128 rows][32-column unit][float4 index][row]
            float4 *frag = reinterpret_cast<float4 *>(entry_frag) +
                           ((size_t)(grow / kGemmBlockM) * frag_units + (size_t)(col0 / 32)) * (8 * kGemmBlockM) + grow % kGemmBlockM;

            // The polynomial epilogue needs the FP32 Gram tile: fetch the first 32 columns before the accumulator is
            // ready so the latency hides behind the MMAs.  (Chained: an entry is in the ring only once the matrix's
            // Gram phase is complete.)
            float4 g[8];
            if (epilogue == kEpiPoly && in_range) {
#pragma unroll
                for (int j = 0; j < 8; ++j) g[j] = __ldcg(frag + j * kGemmBlockM);
            }
            if (CHAINED && unpublished != kNoSlot && !__all_sync(0xffffffffu, mbar_test(tfull_bar(acc), acc_phase))) publish();
            if (!__all_sync(0xffffffffu, mbar_wait(tfull_bar(acc), acc_phase, abort_flag))) break;
            tc_fence_after();
            const uint32_t taddr = tmem_base + ((uint32_t)(32 * q) << 16) + acc * C::kAccCols + taddr_col;
            // fused: the Gram accumulator of this tile sits in the other buffer
            const uint32_t held_taddr = tmem_base + ((uint32_t)(32 * q) << 16) + (acc ^ 1u) * C::kAccCols + taddr_col;
            const uint32_t tempty = tempty_leader0 + 8u * acc;
            const uint32_t held_tempty = tempty_leader0 + 8u * (acc ^ 1u);
            // One-pass prepare: the operand of the first iteration is the un-normalised update, and
            // s = 1 / (1.01 |u| + 1e-7) of the tile's matrix enters here: G = (s s) X X^T, X1 = s (Q X).
            // (A fused polynomial part scales the held Gram accumulator, not its own.)
            float out_scale = 1.0f;
            if (slot_scale != nullptr && scale_pow != 0u && epilogue != kEpiPoly) {
                const float sv = __ldcg(slot_scale + slot);
                out_scale = scale_pow == 2u ? sv * sv : sv;
            }
            const bool scaled = out_scale != 1.0f;   // warp-uniform

#pragma unroll
            for (int sub = 0; sub < C::kEpiCols / 32; ++sub) {
                constexpr int kLastSub = C::kEpiCols / 32 - 1;
                const int col = col0 + 32 * sub;
                uint32_t packed[16];
                if (CHAINED && fused) {
                    // two halves of 16 columns: this tile's accumulator and the held Gram accumulator, which enters as the
                    // unfused form would have read it back from memory
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        uint32_t v[16], h[16];
                        tc_ld16(taddr + 32 * sub + 16 * half, v);
                        tc_ld16(held_taddr + 32 * sub + 16 * half, h);
                        tc_ld_wait();
                        if (sub == kLastSub && half == 1) {
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) { mbar_arrive_cluster(tempty); mbar_arrive_cluster(held_tempty); }
                        }
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const float ident = (col + 16 * half + j == grow) ? ca : 0.0f;
                            const float base = scaled ? __uint_as_float(h[j]) * out_scale : __uint_as_float(h[j]);
                            // store/plain.rs:175-178: fma(c, acc, fma(b, base, identity))
                            v[j] = __float_as_uint(fmaf(cc, __uint_as_float(v[j]), fmaf(cb, base, ident)));
                        }
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            packed[8 * half + j] = pack_operands(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]), f16);
                    }
                } else {
                    uint32_t v[32];
                    tc_ld32(taddr + 32 * sub, v);
                    tc_ld_wait();
                    if (sub == kLastSub && !hold) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive_cluster(tempty);
                    }
                    if (scaled) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * out_scale);
                    }
                    if (epilogue == kEpiApplyLast) {   // FP32 result in the storage layout
                        if (CHAINED && unpublished != kNoSlot) publish();
                        if (in_range && grow < (int)M) {
                            uint8_t *dst = out + (size_t)grow * pitch + (size_t)col * 4;
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                if (col * 4 + 32 * j < (int)pitch) st_global_32(dst + 32 * j, v + 8 * j);
                        }
                        continue;
                    }
                    if (in_range && col < (int)N && (epilogue == kEpiGram || epilogue == kEpiPoly)) {
                        float4 *unit = frag + (size_t)sub * (8 * kGemmBlockM);
                        if (epilogue == kEpiGram) {
#pragma unroll
                            for (int j = 0; j < 8; ++j)
                                __stcg(unit + j * kGemmBlockM,
                                       make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]),
                                                   __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3])));
                        } else {
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                const float gg[4] = {g[j].x, g[j].y, g[j].z, g[j].w};
#pragma unroll
                                for (int e = 0; e < 4; ++e) {
                                    const float ident = (col + 4 * j + e == grow) ? ca : 0.0f;
                                    // store/plain.rs:175-178: fma(c, acc, fma(b, base, identity))
                                    v[4 * j + e] = __float_as_uint(fmaf(cc, __uint_as_float(v[4 * j + e]), fmaf(cb, gg[e], ident)));
                                }
                            }
                            if (sub < kLastSub && col + 32 < (int)N) {   // the next 32 columns, while these are packed and stored
#pragma unroll
                                for (int j = 0; j < 8; ++j) g[j] = __ldcg(unit + (8 + j) * kGemmBlockM);
                            }
                        }
                    }
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        packed[j] = pack_operands(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]), f16);
                }
                if (CHAINED && unpublished != kNoSlot) publish();
                if (in_range && col < (int)N) {
                    if (grow < (int)M) {
                        uint8_t *dst = out + (size_t)grow * pitch + (size_t)col * 2;
                        if ((pitch & 31u) == 0u) {
#pragma unroll
                            for (int j = 0; j < 2; ++j)
                                if (col * 2 + 32 * j < (int)pitch) st_global_32(dst + 32 * j, packed + 8 * j);
                        } else {
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                if (col * 2 + 16 * j < (int)pitch)
                                    *reinterpret_cast<uint4 *>(dst + 16 * j) =
                                        make_uint4(packed[4 * j], packed[4 * j + 1], packed[4 * j + 2], packed[4 * j + 3]);
                        }
                    }
                    if (mirror) {
                        // the transposed block: lanes pair up, the even one stores two rows of one column, the odd one two of
                        // the next, so a store writes 64 bytes of two rows of the result
                        uint8_t *dst = out + (size_t)(col + (lane & 1)) * pitch + (size_t)(warp_row0 + (lane & ~1)) * 2;
                        const bool inside = (warp_row0 + (lane & ~1)) * 2 < (int)pitch;
#pragma unroll
                        for (int c = 0; c < 32; c += 2) {
                            const uint32_t mine = packed[c >> 1];
                            const uint32_t other = __shfl_xor_sync(0xffffffffu, mine, 1);
                            const uint32_t two = (lane & 1) ? __byte_perm(other, mine, 0x7632) : __byte_perm(mine, other, 0x5410);
                            if (inside && col + c + (lane & 1) < (int)M) *reinterpret_cast<uint32_t *>(dst + (size_t)c * pitch) = two;
                        }
                    }
                }
            }
            if (CHAINED) {
                if (unpublished != kNoSlot) publish();   // (a tile whose stores were all skipped)
                unpublished = slot;
                // the other CTAs wait for a held Gram tile before they can go on: publish it at once
                if (hold) publish();
            }
            acc ^= 1u;
            if (acc == 0) acc_phase ^= 1u;
        }
        if (CHAINED && unpublished != kNoSlot) publish();
    }

    __syncthreads();
    if (*abort_flag) {
        // A wait ran out: give copies and MMAs still in flight time to land before the shared
        // memory and TMEM are released, then report.
        for (int i = 0; i < 4096; ++i) __nanosleep(512);
        if (threadIdx.x == 0) atomicExch(status, 1u);
        __syncthreads();
    }
    if (PAIR) cluster_sync_all();  // neither CTA leaves while its peer may still touch it
    if (CHAINED && threadIdx.x == 0) {
        // leave the shared words as the next launch expects them
        if (*abort_flag) atomicExch(&sync->abort, 1u);
        __threadfence();
        if (atomicAdd(&sync->exited, 1u) == gridDim.x - 1) {
            for (uint32_t k = 0; k < slot_count; ++k) sync->progress[k] = 0;
            sync->abort = 0;
            sync->ticket = 0;
            sync->exited = 0;
        }
    }
    if (warp == C::kMmaWarp) {
        if (PAIR)
            asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                         "r"((uint32_t)C::kTmemCols) : "memory");
        else
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                         "r"((uint32_t)C::kTmemCols) : "memory");
    }
}

// ---- the whole Newton-Schulz loop of a small matrix in one CTA ---------------------------------------------------
// A matrix whose smaller dimension is at most 128 and whose larger one at most 512 fits one SM: the operand (up to
// 128 KB), G and Q (32 KB each) stay in shared memory over all iterations, and the FP32 accumulators of a phase in
// tensor memory (the result of the Apply phase fills its 512 columns).  With one launch per phase such a matrix spends
// its time on launches and on the way through L2 between them (4.4 to 5.6 us per phase whose MMAs take well below one);
// here a phase costs its MMAs, one commit, the accumulator's way through registers and two barriers.
// The operand keeps its storage orientation: panels of 64 columns x 128-row blocks as TMA delivers them (128-byte
// swizzle), read K-major along a row and MN-major across rows, so one copy serves both GEMMs it takes part in:
//   wide (rows <= cols)  Gram K-major,  X' = Q X with X as an MN-major B;   tall  Gram MN-major,  X' = X Q with X as a
//   K-major A.
// What TMA fills in beyond the matrix is zero and stays zero, so that MMAs, whose K goes in steps of 16, need no bound.  It
// stays zero by itself while everything is finite.  RAGGED, for plans with a row count that is no multiple of 16 (columns
// always are): what an MMA may read again is cleared, because 0 times an infinity is not 0; a template parameter because the
// code for it costs the others 3 %.  Rounding points, operand values and the order of every sum are those of k_ns_gemm.
// What bounds it: the chain of a phase.  For 64 x 64 that is 330 clocks of MMAs and their barrier, 210 to 360 of reading,
// converting and storing 32 columns a warp, 220 of proxy fence and block barrier, and 100 to 500 between them; up to
// 128 x 512 the MMAs (64 clocks each) and the conversion of 128 x 128 blocks (600 clocks).  So nothing is done for padding
// (units of 32 x 32 that lie beyond G and Q are neither computed nor stored), a warp of its own issues, the inner product of
// the polynomial is formed while its MMAs run, the blocks of Apply have a barrier each, and what memory keeps of G, Q and the
// operands leaves as bulk copies.  Newton-Schulz loop, before and after: 64 x 64 34800 -> 21600 clocks, 128 x 128 49900 ->
// 31600, 128 x 512 103600 -> 61000; whole steps: 64-wide fixture 32.8 -> 24.5 us, one layer of width 128 70.7 -> 46.1, twelve
// 86.8 -> 63.5.  (In twelve layers the larger dimension is 512 and a matrix has one SM to itself.)
constexpr int kSmallWarps = 8;                       // of the epilogue; one more issues MMAs and copies
constexpr int kSmallThreads = 32 * (kSmallWarps + 1);
constexpr uint32_t kSmallPanel = 128 * 128;   // bytes: 128 rows x 64 16-bit values
constexpr uint32_t kSmallTmemCols = 512;
constexpr uint32_t kSmallBlocks = 4;          // of 128 columns of tensor memory: a result of up to 128 x 512

struct SmallLoop {
    uint32_t iterations;
    int last16;           // the last result leaves in the operand type (into the operand buffer that is its turn)
    GemmCoefficients coef;
};

// Which of the loop's results the operand buffers in memory keep.  The buffers take turns, so after a launch per phase they
// hold the last two 16-bit results.  Earlier ones are not stored: the bulk copies of two results to one buffer would be in
// no order (what the issuer waits for before it reuses the panels is only that they have been read).
__host__ __device__ constexpr bool small_keeps(uint32_t it, uint32_t iterations, bool last16) { return it + (last16 ? 2u : 3u) >= iterations; }

__device__ __forceinline__ uint32_t small_swizzled(uint32_t row, uint32_t chunk) { return row * 128u + ((chunk ^ (row & 7u)) << 4); }

template <bool RAGGED, int F16>
__global__ void __launch_bounds__(kSmallThreads, 1)
k_ns_small(const GemmProblem *__restrict__ gram, const GemmProblem *__restrict__ poly, const GemmProblem *__restrict__ apply0,
           const GemmProblem *__restrict__ apply1, const GemmProblem *__restrict__ last, SmallLoop loop,
           const float *__restrict__ slot_scale, uint32_t *status) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *g_panels = smem, *q_panels = smem + 2 * kSmallPanel, *x_panels = smem + 4 * kSmallPanel;
    __shared__ uint64_t bars[2 + kSmallBlocks];   // operand loaded; MMAs of Gram or Poly retired; those of a block of Apply
    __shared__ uint32_t tmem_slot, abort_word;
    __shared__ float coef[3 * kMaxChainIterations];
    volatile uint32_t *abort_flag = &abort_word;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t slot = blockIdx.x;
    const uint32_t load_bar = smem_u32(bars), mma_bar = load_bar + 8, block_bar = load_bar + 16;
    const GemmProblem *ap = apply0 + slot;
    const uint32_t rows = ap->M, cols = ap->N;   // of the storage layout
    const bool empty = rows == 0u;
    const bool tall = gram[slot].a_mn_major != 0u;
    const bool issuer = warp == kSmallWarps;
    const uint32_t n = tall ? cols : rows;
    // maps of 64 x 128 boxes, and results in memory: they belong to the plan.  (The second operand buffer's problems follow the
    // first one's, a matrix per CTA.)
    const uint64_t x0_map = tall ? ap->map_a : gram[slot].map_a, x1_map = tall ? apply1[slot].map_a : gram[gridDim.x + slot].map_a;
    const uint64_t g_map = poly[slot].map_a, q_map = tall ? ap->map_b : ap->map_a;
    uint8_t *out32 = reinterpret_cast<uint8_t *>(last[slot].out32);
    const uint32_t panels = tall ? 2u : (cols + 63u) / 64u, blocks = tall ? (rows + 127u) / 128u : 1u;

    if (threadIdx.x == 0) {
        mbar_init(load_bar, 1);
        mbar_init(mma_bar, 1);
        for (uint32_t j = 0; j < kSmallBlocks; ++j) mbar_init(block_bar + 8u * j, 1);
        abort_word = 0;
        fence_async_smem();
#pragma unroll
        for (uint32_t i = 0; i < 3 * kMaxChainIterations; ++i) coef[i] = loop.coef.v[i];
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(kSmallTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");

    if (!empty) {
        if (threadIdx.x == 32 * kSmallWarps) {
            mbar_expect_tx(load_bar, panels * blocks * kSmallPanel);
            for (uint32_t p = 0; p < panels; ++p)
                for (uint32_t j = 0; j < blocks; ++j)
                    tma_load_2d<false>(smem_u32(x_panels) + (p * blocks + j) * kSmallPanel, x0_map, load_bar, (int)(64 * p), (int)(128 * j));
        }
        const float slot_s = slot_scale != nullptr ? __ldcg(slot_scale + slot) : 1.0f;
        const uint32_t q = warp & 3, half = (warp >> 2) & 1;
        const uint32_t row = 32 * q + lane;                          // TMEM lane
        const uint32_t lane_base = tmem + ((32u * q) << 16);
        const uint32_t k16_n = (n + 15u) / 16u;                       // steps of 16 over the smaller dimension
        // What there is of G and Q in units of 32 x 32: a warp whose 32 rows lie beyond it only waits, and the two warps of a
        // lane quarter take its units in turn.
        const uint32_t units_n = (n + 31u) / 32u;
        const bool active = !issuer && q < units_n;
        const uint64_t g_desc = smem_desc(smem_u32(g_panels), 16, 1024), q_desc = smem_desc(smem_u32(q_panels), 16, 1024);
        const uint64_t x_k_desc = smem_desc(smem_u32(x_panels), 16, 1024);                                           // read along a row
        const uint64_t x_mn_desc = smem_desc(smem_u32(x_panels), (tall ? blocks : 1u) * kSmallPanel, 1024);          // read across rows
        constexpr uint32_t kPanel16 = kSmallPanel >> 4;                // a panel in the descriptors' units of 16 bytes
        auto k_step = [](uint32_t k) { return (k >> 2) * kPanel16 + (k & 3u) * 2u; };   // 16 columns along 64-column panels
        // What a plan keeps in memory of G, Q and the operands leaves as bulk copies of the panels, beside the MMAs.  (Stored by the
        // epilogue, a row per lane, they were a quarter of the time of a 128 x 512 matrix.)
        auto store_panels = [&](uint64_t map, uint32_t smem_addr, uint32_t count, uint32_t rows128) {
            for (uint32_t p = 0; p < count; ++p)
                for (uint32_t j = 0; j < rows128; ++j)
                    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map), "r"((int)(64 * p)),
                                 "r"((int)(128 * j)), "r"(smem_addr + (p * rows128 + j) * kSmallPanel)
                                 : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        };
        (void)mbar_wait(load_bar, 0, abort_flag);   // on expiry the flag ends the loop at its next barrier
        auto wait_mma = [&](uint32_t bar, uint32_t parity) {
            __syncwarp();
            (void)mbar_wait(bar, parity, abort_flag);
            tc_fence_after();
        };
        // what this thread stored to shared memory is visible to the next phase's MMAs, and its TMEM reads are done
        auto hand_over = [&]() {
            fence_async_smem();
            tc_fence_before();
            __syncthreads();
        };
        auto pack8 = [&](const uint32_t *v) {
            uint4 w;
            w.x = pack_operands(__uint_as_float(v[0]), __uint_as_float(v[1]), F16);
            w.y = pack_operands(__uint_as_float(v[2]), __uint_as_float(v[3]), F16);
            w.z = pack_operands(__uint_as_float(v[4]), __uint_as_float(v[5]), F16);
            w.w = pack_operands(__uint_as_float(v[6]), __uint_as_float(v[7]), F16);
            return w;
        };
        auto clear_columns = [&](uint32_t col, uint32_t *v) {   // those from n on, of 32 from `col`
            if (RAGGED && (n & 15u) != 0u && col + 32u > n) {
#pragma unroll
                for (int j = 0; j < 32; ++j)
                    if (col + j >= n) v[j] = 0u;
            }
        };
        // byte offsets of this thread's row in a panel, for the four 16-byte pieces of a unit's 64 bytes
        uint32_t piece[2][4];
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int j = 0; j < 4; ++j) piece[u][j] = small_swizzled(row, (uint32_t)(4 * u + j));
        auto store_unit = [&](uint8_t *panel, uint32_t unit, const uint4 *w) {   // into the panel that holds 32-column unit `unit`
#pragma unroll
            for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4 *>(panel + ((unit & 1u) ? piece[1][j] : piece[0][j])) = w[j];
        };
        __syncthreads();
        for (uint32_t it = 0; it < loop.iterations; ++it) {
            const float ca = coef[3 * it], cb = coef[3 * it + 1], cc = coef[3 * it + 2];
            const bool final = it + 1 == loop.iterations;
            const bool scaled = it == 0 && slot_s != 1.0f;
            const float s1 = slot_s, s2 = s1 * s1;
            auto store_nn = [&](uint8_t *panels0, uint32_t unit, const uint32_t *v) {
                uint4 w[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) w[j] = pack8(v + 8 * j);
                store_unit(panels0 + (unit >> 1) * kSmallPanel, unit, w);
            };
            // ---- Gram: columns 0 .. 127 of tensor memory
            if (issuer && elect_one()) {
                tc_fence_after();
                // (read across rows, N is made of whole 64-column swizzle atoms)
                const uint32_t idesc = instr_desc(128, (int)(tall ? (n + 63u) / 64u * 64u : 32 * units_n), F16, tall ? 1u : 0u, tall ? 1u : 0u);
                if (tall) {
                    const uint32_t steps = (rows + 15u) / 16u;
                    for (uint32_t k = 0; k < steps; ++k) tc_mma<false>(tmem, x_mn_desc + 128u * k, x_mn_desc + 128u * k, idesc, k != 0);
                } else {
                    const uint32_t steps = (cols + 15u) / 16u;
                    for (uint32_t k = 0; k < steps; ++k) tc_mma<false>(tmem, x_k_desc + k_step(k), x_k_desc + k_step(k), idesc, k != 0);
                }
                tc_commit<false>(mma_bar);
            }
            uint32_t base[2][32];   // the Gram accumulator, which the polynomial starts from
            if (!issuer) wait_mma(mma_bar, 0);
            if (active) {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const uint32_t unit = half + 2 * u;
                    if (unit >= units_n) break;   // warp-uniform
                    tc_ld32(lane_base + 32 * unit, base[u]);
                    tc_ld_wait();
                    if (scaled) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) base[u][j] = __float_as_uint(__uint_as_float(base[u][j]) * s2);
                    }
                    uint32_t v[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = base[u][j];
                    clear_columns(32 * unit, v);
                    store_nn(g_panels, unit, v);
                }
            }
            hand_over();
            // ---- Poly: columns 128 .. 255
            if (issuer && elect_one()) {
                tc_fence_after();
                const uint32_t idesc = instr_desc(128, (int)(32 * units_n), F16, 0u, 0u);
                for (uint32_t k = 0; k < k16_n; ++k) tc_mma<false>(tmem + 128u, g_desc + k_step(k), g_desc + k_step(k), idesc, k != 0);
                tc_commit<false>(mma_bar);
                if (final) store_panels(g_map, smem_u32(g_panels), (n + 63u) / 64u, 1u);
            }
            if (active) {   // store/plain.rs:175-178: fma(c, acc, fma(b, base, identity)): the inner one while the MMAs run
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const uint32_t unit = half + 2 * u;
                    if (unit >= units_n) break;
                    if (unit == q) {   // on the diagonal; rows and columns beyond the matrix stay zero
                        const float a = row < n ? ca : 0.0f;
#pragma unroll
                        for (int j = 0; j < 32; ++j) base[u][j] = __float_as_uint(fmaf(cb, __uint_as_float(base[u][j]), j == lane ? a : 0.0f));
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; ++j) base[u][j] = __float_as_uint(fmaf(cb, __uint_as_float(base[u][j]), 0.0f));
                    }
                }
            }
            if (!issuer) wait_mma(mma_bar, 1);   // (two completions per iteration)
            if (active) {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const uint32_t unit = half + 2 * u;
                    if (unit >= units_n) break;
                    uint32_t v[32];
                    tc_ld32(lane_base + 128u + 32 * unit, v);
                    tc_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(fmaf(cc, __uint_as_float(v[j]), __uint_as_float(base[u][j])));
                    clear_columns(32 * unit, v);
                    store_nn(q_panels, unit, v);
                }
            }
            hand_over();
            // ---- Apply: a block of 128 columns of tensor memory is 128 x 128 of the result, with a barrier of its own, so that
            // the first ones are converted while the MMAs of the others run.  A block's result goes where only its own MMAs
            // have read: the same panels (wide), the same rows (tall).
            if (issuer && elect_one()) {
                tc_fence_after();
                // the copies of the panels that this phase overwrites have been read
                asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                if (tall) {
                    const uint32_t idesc = instr_desc(128, (int)(32 * units_n), F16, 0u, 0u);
                    for (uint32_t j = 0; j < blocks; ++j) {
                        for (uint32_t k = 0; k < k16_n; ++k)
                            tc_mma<false>(tmem + 128u * j, x_k_desc + ((k >> 2) * blocks + j) * kPanel16 + (k & 3u) * 2u, q_desc + k_step(k),
                                          idesc, k != 0);
                        tc_commit<false>(block_bar + 8u * j);
                    }
                } else {
                    for (uint32_t p = 0; p < panels; p += 2) {
                        const uint32_t idesc = instr_desc(128, p + 1 < panels ? 128 : 64, F16, 0u, 1u);
                        for (uint32_t k = 0; k < k16_n; ++k)
                            tc_mma<false>(tmem + 64u * p, q_desc + k_step(k), x_mn_desc + p * kPanel16 + 128u * k, idesc, k != 0);
                        tc_commit<false>(block_bar + 4u * p);
                    }
                }
                if (final) store_panels(q_map, smem_u32(q_panels), (n + 63u) / 64u, 1u);
            }
            const bool fp32 = final && !loop.last16;
            const uint32_t result_blocks = issuer ? 0u : tall ? blocks : (panels + 1) / 2;
#pragma unroll 1
            for (uint32_t j = 0; j < result_blocks; ++j) {
                wait_mma(block_bar + 8u * j, it & 1u);
                const uint32_t r = tall ? 128 * j + row : row, units = tall ? units_n : min(4u, (cols - 128 * j + 31u) / 32u);
                if (32 * q + (tall ? 128 * j : 0u) >= rows) continue;   // warp-uniform
                if (fp32) {
                    // 16 rows x 64 columns at a time; the four lanes of a row exchange pairs until each holds 32 bytes in a row, so
                    // that a store writes whole 128-byte lines (128 x 128: 2800 clocks, 4600 with a row per lane)
                    const uint32_t r0 = (tall ? 128 * j : 0u) + 32 * q + 16 * half + (lane >> 2);
#pragma unroll 1
                    for (uint32_t c = 0; c < units; c += 2) {
                        uint32_t v[32];
                        tc_ld_16x64(lane_base + ((16u * half) << 16) + 128 * j + 32 * c, v);
                        tc_ld_wait();
                        if (scaled) {
#pragma unroll
                            for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * s1);
                        }
#pragma unroll
                        for (int h = 0; h < 2; ++h) {       // rows r0 and r0 + 8
#pragma unroll
                            for (int g = 0; g < 2; ++g) {   // 32 columns each
                                uint32_t a[4], b[4], w[8];
#pragma unroll
                                for (int k = 0; k < 4; ++k) {
                                    a[k] = v[16 * g + 4 * k + 2 * h];
                                    b[k] = v[16 * g + 4 * k + 2 * h + 1];
                                }
                                quad_transpose(a[0], a[1], a[2], a[3], lane);
                                quad_transpose(b[0], b[1], b[2], b[3], lane);
#pragma unroll
                                for (int k = 0; k < 4; ++k) { w[2 * k] = a[k]; w[2 * k + 1] = b[k]; }
                                const uint32_t r = r0 + 8 * h, col = (tall ? 0u : 128 * j) + 32 * (c + g) + 8 * (lane & 3);
                                if (r < rows && col < cols) st_global_32(out32 + ((size_t)r * cols + col) * 4, w);
                            }
                        }
                    }
                    continue;
                }
#pragma unroll 1
                for (uint32_t unit = half; unit < units; unit += 2) {
                    uint32_t v[32];
                    tc_ld32(lane_base + 128 * j + 32 * unit, v);
                    tc_ld_wait();
                    if (scaled) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * s1);
                    }
                    if (RAGGED && r >= rows) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i] = 0u;
                    }
                    uint4 w[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) w[i] = pack8(v + 8 * i);
                    store_unit(x_panels + (tall ? (unit >> 1) * blocks + j : 2 * j + (unit >> 1)) * kSmallPanel, unit, w);
                }
            }
            hand_over();
            if (*abort_flag) break;   // a wait ran out: written before the barrier, so every thread sees it
            if (issuer && !fp32 && small_keeps(it, loop.iterations, loop.last16 != 0) && elect_one())
                store_panels((it & 1u) ? x0_map : x1_map, smem_u32(x_panels), tall ? (n + 63u) / 64u : panels, blocks);
        }
        if (issuer) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        if (*abort_flag) {
            // copies or MMAs may still be in flight: give them time to land before the memory is released
            for (int i = 0; i < 4096; ++i) __nanosleep(512);
            if (threadIdx.x == 0) atomicExch(status, 1u);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kSmallTmemCols) : "memory");
}

template <int TM, int BN, bool PAIR, bool CHAINED>
cudaError_t launch_impl(const GemmProblem *problems, const void *tiles, uint32_t tile_count, uint32_t epilogue,
                        int f16, const GemmCoefficients &coef, const float *slot_scale, uint32_t scale_pow,
                        uint32_t *status, void *sync, uint32_t slot_count, uint32_t debug_flags, int grid,
                        cudaStream_t s) {
    using C = Cfg<TM, BN, PAIR, CHAINED>;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    unsigned n_attr = 0;
    bool chained = true;
#ifdef B2_MEASURE
    chained = !(debug_flags & 32u);   // plain stream order
#endif
    if (chained) {
        attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n_attr].val.programmaticStreamSerializationAllowed = 1;
        ++n_attr;
    }
    if (PAIR) {
        int clusters = grid / 2;
        if ((uint32_t)clusters > tile_count) clusters = (int)tile_count;
        if (clusters < 1) clusters = 1;
        grid = 2 * clusters;
        attr[n_attr].id = cudaLaunchAttributeClusterDimension;
        attr[n_attr].val.clusterDim.x = 2;
        attr[n_attr].val.clusterDim.y = 1;
        attr[n_attr].val.clusterDim.z = 1;
        ++n_attr;
    } else if ((uint32_t)grid > tile_count) {
        grid = (int)tile_count;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n_attr;
    cfg.gridDim = dim3((unsigned)grid, 1, 1);
    cfg.blockDim = dim3((unsigned)C::kThreads, 1, 1);
    cfg.dynamicSmemBytes = C::kSmemBytes;
    cfg.stream = s;
    return cudaLaunchKernelEx(&cfg, k_ns_gemm<TM, BN, PAIR, CHAINED>, problems, tiles, tile_count, epilogue, f16, coef,
                              slot_scale, scale_pow, status, static_cast<ChainSync *>(sync), slot_count);
}

template <int TM, int BN, bool PAIR>
struct Shape {
    static constexpr bool is(const GemmShape &g) { return g.tm == TM && g.bn == BN && (g.pair != 0) == PAIR; }
};
// Calls f<TM, BN, PAIR>() for the shape, from those that exist with or without the ticketed form.
#define B2_FOR_SHAPE(shape, F, ...)                                                  \
    if (Shape<256, 256, true>::is(shape)) return F<256, 256, true>(__VA_ARGS__);      \
    if (Shape<128, 256, false>::is(shape)) return F<128, 256, false>(__VA_ARGS__);    \
    if (Shape<128, 128, false>::is(shape)) return F<128, 128, false>(__VA_ARGS__);
#define B2_FOR_PLAIN_SHAPE(shape, F, ...)                                            \
    if (Shape<128, 128, true>::is(shape)) return F<128, 128, true>(__VA_ARGS__);

template <int TM, int BN, bool PAIR>
cudaError_t launch_plain(const GemmProblem *problems, const GemmTile *tiles, uint32_t tile_count, uint32_t epilogue, int f16,
                         const GemmCoefficients &coef, const float *slot_scale, uint32_t scale_pow, uint32_t *status,
                         uint32_t debug_flags, int grid, cudaStream_t s) {
    return launch_impl<TM, BN, PAIR, false>(problems, tiles, tile_count, epilogue, f16, coef, slot_scale, scale_pow, status,
                                            nullptr, 0u, debug_flags, grid, s);
}
template <int TM, int BN, bool PAIR>
cudaError_t launch_ticketed(const GemmProblem *problems, const ChainTile *tiles, uint32_t tile_count, int f16,
                            const GemmCoefficients &coef, const float *slot_scale, uint32_t *status, void *sync,
                            uint32_t slot_count, uint32_t debug_flags, int grid, cudaStream_t s, bool fused_list) {
    // the epilogue argument of the plain launch carries the list kind here
    return launch_impl<TM, BN, PAIR, true>(problems, tiles, tile_count, fused_list ? 1u : 0u, f16, coef, slot_scale, 0u, status,
                                           sync, slot_count, debug_flags, grid, s);
}
template <int TM, int BN, bool PAIR>
cudaError_t configure_plain() {
    return cudaFuncSetAttribute(k_ns_gemm<TM, BN, PAIR, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<TM, BN, PAIR, false>::kSmemBytes);
}
template <int TM, int BN, bool PAIR>
cudaError_t configure(bool ticketed) {
    const cudaError_t e = configure_plain<TM, BN, PAIR>();
    if (e != cudaSuccess || !ticketed) return e;
    return cudaFuncSetAttribute(k_ns_gemm<TM, BN, PAIR, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<TM, BN, PAIR, true>::kSmemBytes);
}
template <int TM, int BN, bool PAIR>
int resident_groups(int sm_count) {
    using C = Cfg<TM, BN, PAIR, true>;
    if (PAIR) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        cfg.gridDim = dim3((unsigned)(sm_count & ~1), 1, 1);
        cfg.blockDim = dim3((unsigned)C::kThreads, 1, 1);
        cfg.dynamicSmemBytes = C::kSmemBytes;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, k_ns_gemm<TM, BN, PAIR, true>, &cfg) != cudaSuccess) {
            (void)cudaGetLastError();
            return 0;
        }
        return clusters;
    }
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_ns_gemm<TM, BN, PAIR, true>, C::kThreads, C::kSmemBytes) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    return per_sm > 0 ? sm_count : 0;   // one CTA per SM is all a launch ever uses
}
}  // namespace

cudaError_t gemm_configure(const GemmShape &shape, bool ticketed) {
    B2_FOR_SHAPE(shape, configure, ticketed)
    B2_FOR_PLAIN_SHAPE(shape, configure_plain)
    return cudaErrorInvalidValue;
}
int gemm_resident_groups(const GemmShape &shape, int sm_count) {
    B2_FOR_SHAPE(shape, resident_groups, sm_count)
    return 0;
}
cudaError_t launch_ns_gemm(const GemmShape &shape, const GemmProblem *problems, const GemmTile *tiles,
                           uint32_t tile_count, uint32_t epilogue, int f16, float ca, float cb,
                           float cc, const float *slot_scale, uint32_t scale_pow, uint32_t *status,
                           uint32_t debug_flags, int grid, cudaStream_t s) {
    if (tile_count == 0) return cudaSuccess;
    GemmCoefficients coef = {};
    coef.v[0] = ca; coef.v[1] = cb; coef.v[2] = cc;
    B2_FOR_SHAPE(shape, launch_plain, problems, tiles, tile_count, epilogue, f16, coef, slot_scale, scale_pow, status, debug_flags, grid, s)
    B2_FOR_PLAIN_SHAPE(shape, launch_plain, problems, tiles, tile_count, epilogue, f16, coef, slot_scale, scale_pow, status, debug_flags, grid, s)
    return cudaErrorInvalidValue;
}
bool ns_small_fits(uint32_t rows, uint32_t cols) { return std::min(rows, cols) <= 128u && std::max(rows, cols) <= 512u; }
namespace {
// what the largest matrix that fits needs: G and Q, two panels each, and an operand of eight
constexpr uint32_t kSmallMaxSmem = 1024u + 12u * kSmallPanel;
static_assert(kSmallMaxSmem <= (uint32_t)kSmemLimit, "one SM holds the largest matrix");
}  // namespace
uint32_t ns_small_smem(uint32_t rows, uint32_t cols) {
    const uint32_t x = rows > cols ? 2u * ((rows + 127u) / 128u) : (cols + 63u) / 64u;
    // at least half of an SM's: a second CTA on it would only wait for the first one's tensor memory, all of which it takes
    return std::max(1024u + (4u + x) * kSmallPanel, 116u * 1024u);
}
// The limit belongs to the function, not to a plan: it is always the largest, so that no plan takes it from another.
namespace {
auto small_kernel(bool ragged, int f16) {
    return ragged ? (f16 ? k_ns_small<true, 1> : k_ns_small<true, 0>) : (f16 ? k_ns_small<false, 1> : k_ns_small<false, 0>);
}
}  // namespace
cudaError_t ns_small_configure(bool ragged, int f16) {
    return cudaFuncSetAttribute(small_kernel(ragged, f16), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallMaxSmem);
}
cudaError_t launch_ns_small(const GemmProblem *gram, const GemmProblem *poly, const GemmProblem *apply0, const GemmProblem *apply1,
                            const GemmProblem *last, uint32_t slot_count, uint32_t iterations, int f16, int last16,
                            const GemmCoefficients &coef, const float *slot_scale, uint32_t smem_bytes, bool ragged,
                            uint32_t *status, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(slot_count, 1, 1);
    cfg.blockDim = dim3(kSmallThreads, 1, 1);
    cfg.dynamicSmemBytes = smem_bytes;
    cfg.stream = s;
    SmallLoop loop = {iterations, last16, coef};
    return cudaLaunchKernelEx(&cfg, small_kernel(ragged, f16), gram, poly, apply0, apply1, last, loop, slot_scale, status);
}
size_t chain_sync_bytes(uint32_t slot_count) { return sizeof(ChainSync) + sizeof(uint32_t) * slot_count; }
namespace {
template <int TM, int BN, bool PAIR>
uint32_t epilogue_warps() { return (uint32_t)Cfg<TM, BN, PAIR, true>::kEpiWarps * (PAIR ? 2u : 1u); }
}  // namespace
uint32_t chain_epilogue_warps(const GemmShape &shape) {
    B2_FOR_SHAPE(shape, epilogue_warps)
    return 0;
}
cudaError_t launch_ns_chain(const GemmShape &shape, const GemmProblem *problems, const ChainTile *tiles,
                            uint32_t tile_count, int f16, const GemmCoefficients &coef, const float *slot_scale,
                            uint32_t *status, void *sync, uint32_t slot_count, uint32_t debug_flags, int grid,
                            cudaStream_t s, bool fused_list) {
    if (tile_count == 0) return cudaSuccess;
    B2_FOR_SHAPE(shape, launch_ticketed, problems, tiles, tile_count, f16, coef, slot_scale, status, sync, slot_count, debug_flags, grid, s,
                 fused_list)
    return cudaErrorInvalidValue;
}

}  // namespace b2
