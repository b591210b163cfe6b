// Grouped block-INT8 GEMM for sm_100a: TMA-fed tcgen05 kind::i8 MMAs with int32
// partial sums in tensor memory, promoted to fp32 register sums once per 128-wide K block.
//
// Orientation ("swap-AB").  The 128 rows of a weight tile are the M side of the
// MMA and the tokens of one expert are its N side (N = tokens rounded up to 16,
// at most 160 in the block-scaled modes, 256 per channel).  A chunk of 1..160
// tokens therefore costs one pass over the weight tile with no padding to 128
// rows, which is what a weight-streaming (HBM-bound) MoE needs, and the same
// kernel serves prefill and decode sizes.  In tensor memory a lane is an output
// column n and a column is a token.
//
// Work item = (chunk of expert-sorted rows, 128-row output tile; for gate_up the gate tile and
// the up tile of the same 128 output columns, run as two passes over K).  Items are ordered
// chunk-major so that CTAs running side by side share the chunk's activation rows, and the
// chunks of one expert (adjacent in the table) read the same weight tiles at about the same
// time: weight tiles are loaded with an evict-first L2 policy unless the chunk table says that
// another chunk of the expert follows.  Persistent CTAs take items round-robin.
//
// Warp roles in a CTA of 16 warps (block-scaled modes):
//   warp 0       : weight producer: streams the weight tiles (HBM) into ring w[] by TMA
//   warp 1       : MMA issuer (of a pair of CTAs: rank 0's; the other's passes consumed[] on).  Two lanes follow the two barriers of a step (operands ready, partial buffer free), poll in
//                  the same instruction and agree by a vote; one elected lane issues the four MMAs of the step and one
//                  commit to done[].  Owns the tensor-memory allocation.
//   warp 2       : scale producer: token scales times weight-block scale, tables of four steps at a time
//   warp 3       : activation producer: the chunk's token rows (L2) into ring a[] by TMA.  Token rows are read from an
//                  expert-sorted copy of the activations, so a chunk is a run of consecutive rows.
//   warps 4..11  : promotion, four warps (one per lane quarter of tensor memory) per column group; the chunk's tokens are
//                  dealt to the two groups in pieces of 16.  The warps keep the fp32 running sums of their columns in
//                  registers: per K block they load the int32 partials, convert and do one fused multiply-add per value.
//   warps 12..15 : output: carry the finished tile from shared memory to global memory while the promotion warps are
//                  already on the next item
// Pipelines: the two shared-memory rings, refilled when done[] says the MMAs that read a slot have completed; NBUF
// tensor-memory partial buffers between the issuer and the promotion warps (done[] as "full", consumed[] as "free"); the ring
// of scale tables; and the staging tile between the promotion and the output warps.
//
// Epilogues go through the staging tile in shared memory, so that the global stores are whole rows: gate_up keeps
// bf16(gate) there during the up pass, then SiLU(gate)*up in its place; the output warps take the 128-wide group maximum and
// write the int8 row.  down stages bf16 rows, and the output warps apply the routed weight on the way out.
//
// What it measured (DeepSeek-V3 shape, one layer, sustained at the 1000 W power cap; before = a per-step hand-over of scales
// through the issuer, a thread on one channel and 16 tokens, two issuer warps and the output in the promotion warps):
// 64 tokens 1764 -> 1480 us, 777 tokens 2290 -> 1880 us, 4096 tokens 3850 -> 3340 us on one board (others: 1415 to 1440, 1740 to 1840, 2880
// to 3050 now).  The board is at its power cap in all of these (SM clock 1.35 to 1.5 GHz), so what a change saves in cycles comes back
// as time only in part.  Instructions besides the arithmetic cost at the cap as well: shorter waits and a scale loop of half the length
// made 4096 tokens 4 to 6 % and Zipf routing 7 % faster there (at burst clocks the launches take the same time; down GEMM without an
// instruction to issue 1.13 -> 0.90 warps per issue).
//
// Per-channel mode (one scale per token and one per output channel instead of 128x128 blocks) uses the same feed without the
// promotion: a tensor-memory buffer is the int32 accumulator of a whole item, summed over every K block by the tensor core, and
// 16 or 20 warps run an epilogue (int32 -> fp32, times token scale, times channel scale) while the MMAs of the next items fill
// the other buffers.  The scale producer idles and there are no output warps in that mode.
//
// Pairs.  Wide chunks of calls with enough work run on clusters of two CTAs (see grouped_gemm_on_pairs()): two neighbouring tiles of a chunk are one MMA of
// 256 rows (cta_group::2), for which each CTA loads its own weight tile and half of the chunk's token rows.  The rows of a chunk, which each
// tile reads again from L2, cross to the SMs half as often, take half of the shared memory (the weight ring of 160-row chunks has 7 slots
// instead of 5, per channel that of 256-row ones 9 instead of 5) and are read from there by one MMA instead of two.  Rank 0 issues for both: the loads of both CTAs complete on its ready[],
// its commits arrive at done[] of both, and the other CTA's warp 1 passes on what its own promotion warps hand back.  Everything behind the
// MMAs (promotion, scales, output) stays with each CTA's tile.
//
// Every wait is bounded: after about a second a waiter records a timeout in the
// status word, raises a CTA-wide abort flag, and all roles fall through to the
// common exit where tensor memory is released.
#include "common.h"
#include <cuda.h>
#include <cudaTypedefs.h>
#include <mutex>
#include <map>
#include <tuple>
#include <type_traits>

namespace lo {
namespace {

// How a wait polls, by the chunk cap of the instantiation (see Smem::POLL).  The plain form is the shortest in the loops of all roles,
// which share the instruction caches and the power: with sleeps and hints in their place 4096 tokens took 3147 us instead of 3091, Qwen3 2048 Zipf 935 instead of
// 892, sharded 8192 797 instead of 789.  Where the weights bound the kernel, the board's power does: 32 tokens in a graph 1066 plain, 1055
// with sleeps.  With a cap of 64 rows a hint saves 0.2 to 0.3 %, which three runs of each side in turn tell apart at the DeepSeek-V3 shape (40
// tokens 1218.7 to 1221.6 with a hint, 1223.2 to 1223.9 plain; 64 1436.9 to 1437.5, 1440.1 to 1440.8; 256 1730.6 to 1733.1, 1736.3 to 1738.5);
// the same sign within the spread for 777 tokens and at the Qwen3 shape (64 tokens 359.7 to 360.8, 359.7 to 363.1); sleeps cost 0.3 to 0.6 %.
enum Poll { PLAIN, HINT, SLEEP };
// SLEEP: interval between two polls in nanoseconds, by role
constexpr uint32_t LO_SLEEP_PRODUCER = 128u, LO_SLEEP_SCALE = 128u, LO_SLEEP_MMA = 20u, LO_SLEEP_PROMO = 32u, LO_SLEEP_OUT = 256u;

constexpr int TILE_N = 128;      // weight rows per accumulator (MMA M)
constexpr int TILE_K = 128;      // int8 elements (= bytes) per K block
constexpr int T_MAX = 128;       // default bound of the rows of a chunk
constexpr int T_WIDE = 160;      // widest block-scaled chunk: three partial buffers of 160 columns fill tensor memory
constexpr int FIRST_EPI_WARP = 4;
constexpr int OUT_WARPS = 4;     // block-scaled modes: warps that carry the finished tile to global memory
// Register budgets of the wide block-scaled instantiations, by role (setmaxnreg): 16 warps start with 128 registers each;
// the feeding and the output warps give up some, the promotion warps (80 sums and three sets of 16 partials a thread) take
// them: 80 + 2 x 184 + 64 = 512, the 512 registers that a lane of the four warp groups has.  (168 for the promotion warps
// spilled at 160 rows.)
constexpr int REGS_FEED = 80, REGS_PROMO = 184, REGS_OUT = 64;
static_assert(REGS_FEED + 2 * REGS_PROMO + REGS_OUT <= 4 * 128, "the register split must not exceed what the block is launched with");
constexpr int W_TILE_BYTES = TILE_N * TILE_K;   // 16 KiB
constexpr int OUT_ROW_BYTES = TILE_N * 2 + 16;  // one token's 128 outputs as bf16 in the staging tile; 16 bytes of padding: 8 rows = 32 banks
constexpr uint32_t TMEM_COLS = 512;
constexpr int SC_STEPS = 4, SC_BATCHES = 3;     // scale-product tables: K-block steps per batch, batches in the ring
constexpr int ND = 16;                          // completion ring, see Smem::done
constexpr int SMEM_LIMIT = 227 * 1024;          // dynamic shared memory a CTA can be given on this part

// A_ROWS is the largest chunk (token count) the instantiation accepts: with few tokens per call no
// expert can receive more than that many rows, the activation tiles shrink and more weight tiles fit
// into shared memory (more weight bytes in flight per SM).
template <int MODE, int A_ROWS, bool PAIR = false> struct Cfg {
  // gate_up: an item is two passes over K on the same chunk, first the gate tile, then the up tile
  static constexpr int PHASES = MODE == GEMM_GATE_UP ? 2 : 1;
  // Column groups: the chunk's tokens are dealt, in pieces of 16, to this many sets of four warps (one warp per lane quarter
  // of tensor memory).  Block-scaled: two groups of up to five pieces, so that what a step costs a warp besides its pieces
  // (barriers, addresses: as much as two pieces) is paid by eight warps, not twenty.
  static constexpr int NCG = MODE == GEMM_CHANNEL ? (A_ROWS > 64 ? 5 : 4) : 2;
  static constexpr int EPI_WARPS = 4 * NCG;
  static constexpr int NUM_THREADS = (FIRST_EPI_WARP + EPI_WARPS + (MODE == GEMM_CHANNEL ? 0 : OUT_WARPS)) * 32;
  static constexpr bool SPLIT_REGS = MODE != GEMM_CHANNEL && A_ROWS > 64;
  static_assert(!SPLIT_REGS || NUM_THREADS == 512, "the register split is made for four warp groups");
  // a pair of CTAs shares a chunk's rows: each keeps half of them
  static constexpr int A_TILE_BYTES = (PAIR ? A_ROWS / 2 : A_ROWS) * TILE_K;
  // Two rings.  Activation tiles come from L2 (the chunk's rows are read by every output tile of the expert): a
  // slot is refilled only after the MMAs that read it have completed, so the ring has to cover the load latency
  // plus the MMA queue, four K blocks at least.  Weight tiles come from HBM and get the shared memory that is left.
  static constexpr int NA_FIT = (64 * 1024) / A_TILE_BYTES;
  static constexpr int NA = NA_FIT < 4 ? 4 : (NA_FIT > 8 ? 8 : NA_FIT);
  // staging tile of the epilogue: A_ROWS rows of 128 bf16 (gate_up keeps the gate values there during the up pass)
  static constexpr int STAGING_BYTES = MODE == GEMM_CHANNEL ? 0 : A_ROWS * OUT_ROW_BYTES;
  static constexpr int FIXED_BYTES = 10 * 1024;   // scale tables, barriers, alignment slack (checked below)
  static constexpr int NW_FIT = (SMEM_LIMIT - FIXED_BYTES - STAGING_BYTES - NA * A_TILE_BYTES) / W_TILE_BYTES;
  static constexpr int NW = NW_FIT;
  // tensor memory is cut into partial buffers of A_ROWS columns, one int32 accumulator each (at most 8 are used):
  // the partial of one 128-wide K block in the block-scaled modes (the fp32 running sums live in the registers of
  // the promotion warps), the accumulator of a whole item in the per-channel mode
  static constexpr int NBUF = (int)TMEM_COLS / A_ROWS > 8 ? 8 : (int)TMEM_COLS / A_ROWS;
  // Ring of scale-product tables: SC_BATCHES batches of SC_STEPS K-block steps each
  static constexpr int SC_SLOTS = MODE == GEMM_CHANNEL ? 1 : SC_BATCHES * SC_STEPS;
};

// The figures that the chunk rules of the layers give as their reasons.
template <int MODE, int A_ROWS> constexpr bool ring_depths(int weight_slots, int buffers) {
  return Cfg<MODE, A_ROWS>::NW == weight_slots && Cfg<MODE, A_ROWS>::NBUF == buffers;
}
static_assert(ring_depths<GEMM_SINGLE, 32>(11, 8) && ring_depths<GEMM_SINGLE, 64>(8, 8) && ring_depths<GEMM_SINGLE, 128>(7, 4) &&
              ring_depths<GEMM_SINGLE, T_WIDE>(5, 3), "block-scaled: weight slots and partial buffers as the chunk rule states them");
static_assert(Cfg<GEMM_SINGLE, T_WIDE, true>::NW == 7 && Cfg<GEMM_CHANNEL, 256, true>::NW == 9, "pairs: weight slots as the head of this file states them");
static_assert(ring_depths<GEMM_CHANNEL, 64>(9, 8) && ring_depths<GEMM_CHANNEL, 128>(9, 4) && ring_depths<GEMM_CHANNEL, T_WIDE>(8, 3) &&
              ring_depths<GEMM_CHANNEL, 256>(5, 2), "per channel: weight slots and accumulators as the chunk rule states them");

template <int MODE, int A_ROWS, bool PAIR = false> struct Smem {
  using C = Cfg<MODE, A_ROWS, PAIR>;
  static constexpr int POLL = A_ROWS <= 32 ? SLEEP : (A_ROWS <= 64 && MODE != GEMM_CHANNEL ? HINT : PLAIN);
  // operand tiles first: each is a multiple of 1024 bytes, base is 1024-aligned
  uint8_t w[C::NW][W_TILE_BYTES];
  uint8_t a[C::NA][C::A_TILE_BYTES];
  // epilogue staging, row = token (column of the chunk)
  alignas(16) uint8_t staging[C::STAGING_BYTES > 0 ? C::STAGING_BYTES : 16];
  alignas(16) float sc[C::SC_SLOTS][A_ROWS];   // token scale x weight-block scale, see scale_place()
  // Barriers of K-block step u, each a ring of ND indexed by u % ND whatever the depths of the operand rings: position and
  // phase follow from the step number alone.  ND exceeds every ring depth, so that a waiter cannot be overtaken by a
  // barrier's next phase.
  uint64_t ready[ND];                      // weights and activations of the step are in place
  // The MMAs of the step have completed.  One tcgen05.commit per step serves everybody who waits for that event: the
  // producers (a weight slot is free NW steps later, an activation slot NA steps later) and in the block-scaled modes the
  // promotion warps (the partial of the step is in its buffer).
  uint64_t done[ND];
  uint64_t consumed[ND];                   // block-scaled modes: the partial of the step has been read, its buffer is free
  uint64_t peer_consumed[PAIR ? ND : 1];   // pairs, block-scaled modes, leader: consumed[] of the other CTA
  uint64_t scales[SC_BATCHES];             // block-scaled modes: the batch's scale products are in place
  uint64_t tmem_full[C::NBUF];             // per-channel mode: the accumulator of an item is complete
  uint64_t tmem_empty[C::NBUF];            // per-channel mode: the accumulator has been read
  uint64_t stg_full;                       // the item's tile is in the staging buffer (promotion warps -> output warps)
  uint64_t stg_free;                       // its rows have been read (output warps -> promotion warps)
  uint32_t tmem_base;
  volatile int abort_flag;
};

// ------------------------------ PTX wrappers --------------------------------

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// One poll; the hardware may park the thread for a short while, or for up to the hint's time, before it answers no.
template <int POLL> __device__ __forceinline__ bool mbar_try_wait_addr(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  if (POLL == HINT)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(200000u)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  return ok != 0;
}
// Upper bound of one wait, in SM clock cycles (about 1.5 s at 1.9 GHz; below 2^32, so the low half of the clock measures it).
constexpr uint32_t WAIT_LIMIT_CYCLES = 3000000000u;

// Bounded wait.  Returns false when the CTA is aborting (this waiter timed out or another one did); `code` identifies the waiter
// in the status word.  Short on purpose: it is inlined into the loops of all roles, which share the instruction caches.
template <class S>
__device__ __forceinline__ bool mbar_wait_addr(S &sm, uint32_t bar, uint32_t parity, int32_t *status, int code, uint32_t sleep_ns = LO_SLEEP_PROMO) {
  if (mbar_try_wait_addr<S::POLL>(bar, parity)) return true;
  const uint32_t t0 = (uint32_t)clock();
#pragma unroll 1
  while (!mbar_try_wait_addr<S::POLL>(bar, parity)) {
    if (sm.abort_flag) return false;
    if ((uint32_t)clock() - t0 > WAIT_LIMIT_CYCLES) {
      sm.abort_flag = 1;
      if (status) atomicCAS(status, 0, code);
      return false;
    }
    if (S::POLL == SLEEP) __nanosleep(sleep_ns);
  }
  return true;
}
template <class S>
__device__ __forceinline__ bool mbar_wait(S &sm, uint64_t *bar, uint32_t parity, int32_t *status, int code, uint32_t sleep_ns = LO_SLEEP_PROMO) {
  return mbar_wait_addr(sm, smem_u32(bar), parity, status, code, sleep_ns);
}
// One non-blocking look at a barrier: has the phase of this parity completed?
__device__ __forceinline__ bool mbar_test_addr(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void mbar_arrive_addr(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Barriers of the CTA that issues a pair's MMAs (rank 0 of the cluster), by their address in the cluster.  The arrival says that values have
// left tensor memory, which their tcgen05.wait::ld has seen to; it publishes no data, and asks for no release at cluster scope: with one
// (mbarrier.arrive.release.cluster) every step of a pair waited for it, 4096 tokens 2797 -> 5944 us.
struct ClusterBarrier {
  uint32_t addr;
};
__device__ __forceinline__ ClusterBarrier operator+(ClusterBarrier b, uint32_t bytes) { return ClusterBarrier{b.addr + bytes}; }
__device__ __forceinline__ void mbar_arrive_addr(ClusterBarrier bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar.addr) : "memory");
}
template <bool PAIR> __device__ __forceinline__ auto issuer_barrier(uint32_t addr) {
  if constexpr (PAIR) {
    ClusterBarrier b;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(b.addr) : "r"(addr));
    return b;
  } else {
    return addr;
  }
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ void fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ uint64_t policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t policy_evict_normal() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}

// 2-D tiled TMA load global -> shared (this CTA), completion on an mbarrier of this CTA or of the pair's issuer.
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int32_t x, int32_t y, uint32_t bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%2, %3}], [%4], %5;"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int32_t x, int32_t y, ClusterBarrier bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2.L2::cache_hint"
      " [%0], [%1, {%2, %3}], [%4], %5;"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar.addr), "l"(policy)
      : "memory");
}

// One lane of a converged warp, always the same one.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(pred));
  return pred != 0;
}

// Shared-memory matrix descriptor: K-major operand, rows of 128 bytes, 128-byte
// swizzle, 8-row groups 1024 bytes apart (tile base 1024-aligned).
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3ffffu) >> 4);   // start address, 16-byte units
  d |= (uint64_t)1 << 16;                     // leading byte offset (unused with swizzle), 16-byte units
  d |= (uint64_t)(1024 >> 4) << 32;           // stride byte offset between 8-row groups
  d |= (uint64_t)1 << 46;                     // descriptor version (sm_100)
  d |= (uint64_t)2 << 61;                     // layout: 128-byte swizzle
  return d;
}

// Instruction descriptor: int8 x int8 -> int32, both operands K-major, M = m, N = n.
__device__ __forceinline__ uint32_t make_idesc(uint32_t m, uint32_t n) {
  uint32_t d = 0;
  d |= 2u << 4;            // accumulator format: S32
  d |= 1u << 7;            // A format: signed 8-bit
  d |= 1u << 10;           // B format: signed 8-bit
  d |= (n >> 3) << 17;     // N / 8
  d |= (m >> 4) << 24;     // M / 16
  return d;
}

// The descriptors' upper halves are the same for every operand; the lower ones hold the start address.  PAIR: one MMA on the operands and the
// tensor memory of both CTAs, at the same places in each.
template <bool PAIR>
__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint32_t adesc_lo, uint32_t bdesc_lo, uint32_t desc_hi, uint32_t idesc, uint32_t accumulate) {
  if (PAIR)
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
        "mov.b64 a, {%1, %3};\n\tmov.b64 b, {%2, %3};\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], a, b, %4, p;\n\t}"
        ::"r"(tmem_d), "r"(adesc_lo), "r"(bdesc_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
        "mov.b64 a, {%1, %3};\n\tmov.b64 b, {%2, %3};\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], a, b, %4, p;\n\t}"
        ::"r"(tmem_d), "r"(adesc_lo), "r"(bdesc_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate)
        : "memory");
}
// An arrival at the barrier (of both CTAs of a pair) when the MMAs issued so far have completed.
template <bool PAIR> __device__ __forceinline__ void umma_commit_addr(uint32_t bar) {
  if (PAIR)
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
  else
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// 16 consecutive tensor-memory columns of this thread's lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

// Wait for this thread's outstanding tensor-memory loads; the registers are operands so that nothing that uses
// them can be scheduled ahead of the wait.
__device__ __forceinline__ void tmem_ld_wait16(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :: "memory");
}
// Partial sums, 16 registers a thread at a time ("unit"), four threads to a channel: two pieces (32 columns) of one half of the
// warp's channels (16 lanes, taddr points at the first of them).  Register 8v + r is piece v, and of that piece
//   ROW4  (16x128b loads): channel 8(r & 1) + lane / 4, token 4(r >> 1) + lane % 4
//   !ROW4 (16x256b loads, the layout of an MMA accumulator fragment): channel 8((r >> 1) & 1) + lane / 4,
//         token 8(r >> 2) + 2(lane % 4) + (r & 1)
// In a loop of loads alone the first form moves 128 bytes per clock and scheduler, the second 64.  Calls with a chunk table (layers,
// expert rows, the grouped GEMM on its own) take the first, dense calls the second.  First, second, in us a pass, medians of three
// turns on one board whose turns differ by 0.1 to 2.5 % (the stand-alone GEMM's by up to 8):
//   layer of 1024 tokens 1877, 1891    2048 2301, 2354    4096 3177, 3233    Qwen3 2048 805, 822 (Zipf 913, 916)    64, 777: the same
//   8192 tokens of a shard 785, 799    4096 expert rows 433, 441    16384 1429, 1454    grouped GEMM of 4096 rows 318, 325
//   dense 4096 x 4096 x 7168 173.6, 169.4    1000 x 4096 x 7168 50.5, 48.8    4096 x 7168 x 2048 104.0, 103.2    smaller: the same
// Why the dense ones lose is not known.
template <bool ROW4> __device__ __forceinline__ void tmem_ld_two(uint32_t taddr, uint32_t (&r)[16]) {
  if (ROW4)
    asm volatile("tcgen05.ld.sync.aligned.16x128b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr)
                 : "memory");
  else
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr)
                 : "memory");
}
// ... or one piece (16 columns) of both halves: register 8k + r is half k (channels 16k ..), r as above.
template <bool ROW4> __device__ __forceinline__ void tmem_ld_one(uint32_t taddr, uint32_t (&r)[16]) {
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    uint32_t *h = &r[8 * k];
    if (ROW4)
      asm volatile("tcgen05.ld.sync.aligned.16x128b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                   : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3]), "=r"(h[4]), "=r"(h[5]), "=r"(h[6]), "=r"(h[7]) : "r"(taddr + (uint32_t)k * (16u << 16)) : "memory");
    else
      asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                   : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3]), "=r"(h[4]), "=r"(h[5]), "=r"(h[6]), "=r"(h[7]) : "r"(taddr + (uint32_t)k * (16u << 16)) : "memory");
  }
}
// A thread's four tokens of a piece, j = 0 .. 3, with i = lane % 4; and the place of token t of a piece in its 16-entry row of the scale
// table: the four scales of a thread are one 16-byte load, in the order of j.
template <bool ROW4> __device__ __forceinline__ int token_of(int i, int j) { return ROW4 ? 4 * j + i : (j >> 1) * 8 + 2 * i + (j & 1); }
template <bool ROW4> __device__ __forceinline__ int scale_place(int t) {
  return ROW4 ? (t & ~15) | (t & 3) << 2 | ((t >> 2) & 3) : (t & ~15) | ((t >> 1) & 3) << 2 | ((t >> 3) & 1) << 1 | (t & 1);
}
// Row of an eight-token block that column c of a transposed matrix store is: a thread's pair of values is columns 2i and 2i + 1.
template <bool ROW4> __device__ __forceinline__ int block_row(int c) { return ROW4 ? (c >> 1) + 4 * (c & 1) : c; }

// acc = fma(float(raw), scale product, acc) on eight values, one half of a piece: s[j] = the scale product of token j of this thread.
// The 128-long int8 dot is below 2^21 in magnitude, so the conversion is exact; one rounding per
// K block.  Two tokens of one channel at a time: acc[4c + 2h + e] is channel 8h + lane / 4, token 2c + e of the thread's four.
template <bool ROW4> __device__ __forceinline__ void promote8(float *acc, const uint32_t *raw, const float (&s)[4]) {
#pragma unroll
  for (int j = 0; j < 8; j += 2) {
    const int a = ROW4 ? (j & 4) + ((j >> 1) & 1) : j, b = ROW4 ? a + 2 : j + 1;
    const float f0 = __int2float_rn((int32_t)raw[a]), f1 = __int2float_rn((int32_t)raw[b]);
    asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%0, %1};\n\t"
        "fma.rn.f32x2 c, a, b, c;\n\tmov.b64 {%0, %1}, c;\n\t}"
        : "+f"(acc[j]), "+f"(acc[j + 1]) : "f"(f0), "f"(f1), "f"(s[(j >> 1) & 2]), "f"(s[((j >> 1) & 2) + 1]));
  }
}
__device__ __forceinline__ void lds4(uint32_t addr, float (&s)[4]) {
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(s[0]), "=f"(s[1]), "=f"(s[2]), "=f"(s[3]) : "r"(addr));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t *>(&v);
}
// Four 8 x 8 blocks of bf16 fragments to / from shared memory, transposed: fragment column (token) = row there.
__device__ __forceinline__ void stmatrix4_t(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void ldmatrix4_t(uint32_t addr, uint32_t (&v)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr) : "memory");
}

// Element i of a small register array (no dynamic indexing: a chain of selects).
template <typename T, int N> __device__ __forceinline__ T pick(const T (&v)[N], int i) {
  T r = v[0];
#pragma unroll
  for (int u = 1; u < N; ++u) r = i == u ? v[u] : r;
  return r;
}

// Maximum that is NaN when an operand is (fmaxf gives the other operand).
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
struct KParams {
  const float *a_scale;     // [positions, KB]
  const float *b_scale;
  int64_t n_rows_per_expert;
  int64_t n_store;          // output columns that exist (< n_tiles*128 only for a dense E = 1 call)
  int KB;
  int n_tiles;
  const int32_t *sorted_ids;
  int64_t numel_valid;
  const Chunk *chunks;
  const int32_t *num_chunks;
  int8_t *act_q;
  float *act_s;
  __nv_bfloat16 *C;
  const float *topk_weights;
  int weight_mode;
  float act_eps;
  int32_t *status;
  int out_by_position;      // bf16 output row = sorted position instead of the sorted id
  int vec_store;            // block-scaled bf16 output: every group of 8 columns of every row begins on a 16-byte boundary
  const int64_t *row_dst;   // single mode: address of the output row of every sorted id (null: C + id * n_store)
  // Without a chunk table (chunks == null) the chunks follow from arithmetic: fixed_chunks of them, of at most chunk_rows rows.
  int fixed_chunks;
  int chunk_rows;
  const int32_t *masked_m;  // per-channel mode: rows of each expert, in a layout of max_m rows an expert
  int64_t max_m;
  int64_t dense_rows;       // single mode: rows of the one expert
  // Single mode: K blocks per item when the K extent of a tile is dealt to several items (0: not split); the int32 sum of every
  // K block then goes to partial[kb][row][n] instead of C, without scales.
  int split_steps;
  int n_split;
  int32_t *partial;
};

// Four tensor maps of the sorted activation matrix, box heights 16 / 32 / 64 / 128 rows.  A chunk of
// more than 128 rows is fetched as a 128-row box plus a second box for the rest; the halves of a pair's chunk (a multiple of 16 rows each) as one
// box or two that cover no other rows, where two can.
struct AMaps {
  CUtensorMap m[4];
};

__device__ __forceinline__ int a_map_index(int T) { return T <= 16 ? 0 : (T <= 32 ? 1 : (T <= 64 ? 2 : 3)); }

// Walks this CTA's items (chunk, output tile): blockIdx.x, blockIdx.x + gridDim.x, ... in chunk-major order.  Every role has
// its own; the descriptor of the item after the current one is already on its way while the current one is worked on
// (a round trip to L2 and two divisions between two items were a tenth of a down-GEMM item).
// Where the chunks come from is part of the instantiation (a branch for it in the common kernel cost the block-scaled loops
// registers and 3 to 9 % at 4096 rows).
enum Form { TABLE, DENSE, SPLIT };      // chunk table / one expert, from arithmetic / the same with the K extent of a tile split
template <int MODE, int FORM, bool PAIR> struct ItemCursor {
  const KParams &p;
  int num_chunks, n_tiles, ci, nt, step_c, step_t;
  int k0, kn;            // K blocks of the item taken last
  int4 next;
  __device__ __forceinline__ void fetch() {
    if (ci >= num_chunks) return;
    if (FORM != TABLE || (MODE == GEMM_CHANNEL && p.chunks == nullptr)) {
      if (MODE == GEMM_CHANNEL) {
        const int per = (int)((p.max_m + p.chunk_rows - 1) / p.chunk_rows), e = ci / per, first = (ci - e * per) * p.chunk_rows;
        const int64_t left = min((int64_t)p.masked_m[e], p.max_m) - first;
        const int rows = left <= 0 ? 0 : (int)min(left, (int64_t)p.chunk_rows);
        next = make_int4(rows > 0 ? e : -1, (int)(e * p.max_m) + first, rows, left > p.chunk_rows ? 1 : 0);
      } else {
        const int64_t first = (int64_t)ci * p.chunk_rows;
        next = make_int4(0, (int)first, (int)min((int64_t)p.chunk_rows, p.dense_rows - first), 0);
      }
      return;
    }
    next = *reinterpret_cast<const int4 *>(p.chunks + ci);
  }
  __device__ __forceinline__ ItemCursor(const KParams &params, int n_chunks)
      : p(params), num_chunks(n_chunks), n_tiles(FORM == SPLIT ? params.n_tiles * params.n_split : (PAIR ? params.n_tiles / 2 : params.n_tiles)),
        k0(0), kn(params.KB), next(make_int4(-1, 0, 0, 0)) {
    // a pair walks the items as one: two tiles of a chunk, one for each CTA
    const int self = PAIR ? (int)blockIdx.x / 2 : (int)blockIdx.x, all = PAIR ? (int)gridDim.x / 2 : (int)gridDim.x;
    ci = self / n_tiles; nt = self % n_tiles;
    step_c = all / n_tiles; step_t = all % n_tiles;
    fetch();
  }
  __device__ __forceinline__ bool take(Chunk &ch, int &tile) {
    if (ci >= num_chunks) return false;
    ch.expert = next.x; ch.row0 = next.y; ch.rows = next.z; ch.pad = next.w;
    tile = PAIR ? 2 * nt + (int)(blockIdx.x & 1) : nt;
    if constexpr (FORM == SPLIT) {
      const int part = nt / p.n_tiles;
      tile = nt - part * p.n_tiles;
      k0 = part * p.split_steps;
      kn = min(p.split_steps, p.KB - k0);
    }
    ci += step_c;
    nt += step_t;
    if (nt >= n_tiles) { nt -= n_tiles; ++ci; }
    fetch();
    return true;
  }
};

template <int MODE, int A_ROWS, int FORM, bool PAIR>
__global__ void __launch_bounds__((Cfg<MODE, A_ROWS, PAIR>::NUM_THREADS), 1)
grouped_gemm_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ AMaps a_maps, const KParams p) {
  using SM = Smem<MODE, A_ROWS, PAIR>;
  using CF = Cfg<MODE, A_ROWS, PAIR>;
  constexpr int NW = CF::NW;
  constexpr int NA = CF::NA;
  constexpr int NBUF = CF::NBUF;
  constexpr int PHASES = CF::PHASES;
  constexpr int NCG = CF::NCG;
  constexpr int EPI_WARPS = CF::EPI_WARPS;
  constexpr bool ROW4 = FORM == TABLE;                           // see tmem_ld_two
  constexpr bool RESPLIT = CF::SPLIT_REGS && FORM != SPLIT;      // (a split K extent has no running sums)
  extern __shared__ uint8_t smem_raw[];
  SM &sm = *reinterpret_cast<SM *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

  const int tid = threadIdx.x;
  // broadcast from lane 0 so that the compiler knows the warp index (and everything derived from it:
  // roles, tensor-memory addresses, barrier addresses) is uniform across the warp
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int lane = tid & 31;
  const uint32_t rank = PAIR ? cluster_rank() : 0u;      // 0: the CTA that issues the pair's MMAs

  // ------------------------------ set-up -----------------------------------
  if (tid == 0) {
    for (int s = 0; s < ND; ++s) {
      mbar_init(&sm.ready[s], 2);            // the two producers
      mbar_init(&sm.done[s], 1);             // tcgen05.commit of the MMA thread
      mbar_init(&sm.consumed[s], EPI_WARPS * 32);      // every lane of the promotion warps
      if (PAIR) mbar_init(&sm.peer_consumed[PAIR ? s : 0], 1);
    }
    for (int b = 0; b < SC_BATCHES; ++b) mbar_init(&sm.scales[b], 1);
    for (int b = 0; b < NBUF; ++b) {
      mbar_init(&sm.tmem_full[b], 1);
      mbar_init(&sm.tmem_empty[b], (PAIR ? 2 : 1) * EPI_WARPS);
    }
    mbar_init(&sm.stg_full, EPI_WARPS);
    mbar_init(&sm.stg_free, OUT_WARPS);
    sm.abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    if (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)), "r"(TMEM_COLS)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)), "r"(TMEM_COLS)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  if (tid == 32) {
    // descriptors into the descriptor cache while the set-up runs
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&w_map)) : "memory");
#pragma unroll
    for (int i = 0; i < 4; ++i)
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&a_maps.m[i])) : "memory");
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync();      // the other CTA's barriers are there
  tc_fence_after();
  const uint32_t tmem_base = sm.tmem_base;

  // Everything above touches this CTA's shared and tensor memory only and may run while the kernel before this
  // one in the stream is still at work (dependent launch); its outputs (chunk table, activations, scales) are
  // read from here on.
  dependency_wait();
  dependency_release();

  static_assert(FORM == TABLE || (MODE == GEMM_SINGLE && A_ROWS <= T_MAX), "dense calls come with at most T_MAX rows a chunk");
  const int num_chunks = FORM != TABLE || (MODE == GEMM_CHANNEL && p.chunks == nullptr) ? p.fixed_chunks : *p.num_chunks;
  const int KB = p.KB;
  Chunk ch;      // the item at hand: chunk and output tile
  int nt = 0;

  if (warp < FIRST_EPI_WARP) {
    if constexpr (RESPLIT) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_FEED));
    if (warp == 0) {
      // ============ weight producer: one 128 x 128 tile per K block (gate_up: gate pass, then up pass) ============
      if (lane == 0) {
        const uint64_t pol_stream = policy_evict_first();
        const uint64_t pol_keep = policy_evict_normal();
        const auto ready0 = issuer_barrier<PAIR>(smem_u32(&sm.ready[0]));
        uint32_t it = 0;
        int s = 0;
        bool ok = true;
        for (ItemCursor<MODE, FORM, PAIR> items(p, num_chunks); ok && items.take(ch, nt);) {
          if (ch.expert < 0) continue;
          // weight tiles are streamed (evict-first) unless another chunk of the same expert is about to read
          // them again: those stay in L2 under the normal policy
          const uint64_t pol_w = ch.pad ? pol_keep : pol_stream;
          for (int ph = 0; ph < PHASES && ok; ++ph) {
            const int32_t row_g = (int32_t)(ch.expert * p.n_rows_per_expert + (int64_t)(ph * p.n_tiles + nt) * TILE_N);
            for (int kb = FORM == SPLIT ? items.k0 : 0; kb < (FORM == SPLIT ? items.k0 + items.kn : KB); ++kb, ++it) {
              // slot s was read by step it - NW
              if (it >= (uint32_t)NW && !mbar_wait(sm, &sm.done[(it - NW) % ND], ((it - NW) / ND) & 1u, p.status, 1, LO_SLEEP_PRODUCER)) { ok = false; break; }
              const auto bar = ready0 + 8u * (it % ND);
              if (rank == 0) mbar_arrive_expect_tx(&sm.ready[it % ND], (PAIR ? 2 : 1) * W_TILE_BYTES);
              tma_load_2d(sm.w[s], &w_map, kb * TILE_K, row_g, bar, pol_w);
              s = s + 1 == NW ? 0 : s + 1;
            }
          }
        }
        if constexpr (MODE == GEMM_CHANNEL) {
          // The commits of an item's steps arrive at done[] each for itself, in no promised order with the one that the epilogue waits for.
          // The last ones are waited for here, so that none arrives at the memory of a CTA that has left (the block-scaled modes wait for the
          // commit of every step anyway).
          for (uint32_t u = it < (uint32_t)NW ? 0u : it - NW; ok && u < it; ++u) ok = mbar_wait(sm, &sm.done[u % ND], (u / ND) & 1u, p.status, 12, LO_SLEEP_PRODUCER);
        }
      }
    } else if (warp == 3) {
      // ============ activation producer: the chunk's token rows of every K block.  Token rows are read from an
      // expert-sorted copy of the activations, so a chunk is a run of consecutive rows and one tiled load fetches
      // it (a second one for the rows beyond 128).
      if (lane == 0) {
        const uint64_t pol_a = policy_evict_last();
        const auto ready0 = issuer_barrier<PAIR>(smem_u32(&sm.ready[0]));
        uint32_t it = 0;
        int s = 0;
        bool ok = true;
        for (ItemCursor<MODE, FORM, PAIR> items(p, num_chunks); ok && items.take(ch, nt);) {
          if (ch.expert < 0) continue;
          // one box, or two: the rows beyond 128, and for pairs, whose half of the rows is a multiple of 16, what is beyond a power of two
          const int T = PAIR ? (ch.rows + 31) / 32 * 16 : (ch.rows + 15) & ~15;
          const int mi = PAIR ? 27 - __clz(T) : a_map_index(T > 128 ? 128 : T);
          const int T0 = PAIR || T > 128 ? 16 << mi : T;
          const int mi2 = T > T0 ? a_map_index(T - T0) : -1;
          const uint32_t a_bytes = (16u << mi) * TILE_K + (mi2 >= 0 ? (16u << mi2) * TILE_K : 0u);
          const int row0 = ch.row0 + (PAIR ? (int)rank * T : 0);
          for (int ph = 0; ph < PHASES && ok; ++ph) {
            for (int kb = FORM == SPLIT ? items.k0 : 0; kb < (FORM == SPLIT ? items.k0 + items.kn : KB); ++kb, ++it) {
              // slot s was read by step it - NA
              if (it >= (uint32_t)NA && !mbar_wait(sm, &sm.done[(it - NA) % ND], ((it - NA) / ND) & 1u, p.status, 6, LO_SLEEP_PRODUCER)) { ok = false; break; }
              const auto bar = ready0 + 8u * (it % ND);
              if (rank == 0) mbar_arrive_expect_tx(&sm.ready[it % ND], (PAIR ? 2u : 1u) * a_bytes);
              tma_load_2d(sm.a[s], &a_maps.m[mi], kb * TILE_K, row0, bar, pol_a);
              if constexpr (PAIR || A_ROWS > 128) {
                if (mi2 >= 0) tma_load_2d(sm.a[s] + T0 * TILE_K, &a_maps.m[mi2], kb * TILE_K, row0 + T0, bar, pol_a);
              }
              s = s + 1 == NA ? 0 : s + 1;
            }
          }
        }
      }
    } else if (warp == 2) {
      // ============ scale producer (block-scaled modes) ============
      // Lane g multiplies the token scales of tokens g, g + 32, ... with the weight-block scale.  The promotion warps wait
      // for the tables by themselves, four K-block steps at a time: a hand-over per step through the MMA issuer made this
      // warp's chain (wait, multiply, store, arrive: 900 cycles) the slowest of the kernel.  Scales come from L2 (the chunk's
      // scale rows are read by every output tile of the expert), one batch ahead, across the ends of passes and items.  Rows
      // of scales whose length is a multiple of four are read with 16-byte loads, in a loop of its own: with the choice inside the loop
      // its code was twice as long, at the cost of the promotion warps on the same scheduler too
      // (4096 tokens 3091 -> 3015 us, Qwen3 2048 Zipf 892 -> 867).
      if constexpr (MODE != GEMM_CHANNEL && FORM != SPLIT) {
        constexpr int NU = (A_ROWS + 31) / 32;
        const int64_t nblk = (p.n_rows_per_expert + TILE_N - 1) / TILE_N;
        auto produce = [&](auto by_four) {
        constexpr bool vec = decltype(by_four)::value;
        ItemCursor<MODE, FORM, PAIR> items(p, num_chunks);
        struct Batch { Chunk ch; int nt, ph, kb; bool valid; };     // K blocks kb .. kb + 3 of a pass over an item
        float a_cur[NU][4], b_cur[4], a_nxt[NU][4], b_nxt[4];
        auto next_item = [&](Batch &b) {
          do { b.valid = items.take(b.ch, b.nt); } while (b.valid && b.ch.expert < 0);
        };
        auto advance = [&](Batch &b) {
          b.kb += SC_STEPS;
          if (b.kb >= KB) {
            b.kb = 0;
            if (++b.ph == PHASES) { b.ph = 0; next_item(b); }
          }
        };
        // a token beyond the chunk reads row 0; its products are zeroed below
        auto fetch = [&](const Batch &bt, float (&a)[NU][4], float (&b)[4]) {
          const float *as_base = p.a_scale + (int64_t)bt.ch.row0 * KB + bt.kb;
#pragma unroll
          for (int u = 0; u < NU; ++u) {
            const int t = lane + u * 32;
            const float *src = as_base + (int64_t)(t < bt.ch.rows ? t : 0) * KB;
            if (vec) {
              const float4 v = __ldg(reinterpret_cast<const float4 *>(src));
              a[u][0] = v.x; a[u][1] = v.y; a[u][2] = v.z; a[u][3] = v.w;
            } else {
#pragma unroll
              for (int i = 0; i < 4; ++i) a[u][i] = bt.kb + i < KB ? __ldg(src + i) : 0.f;
            }
          }
          const float *bs = p.b_scale + ((int64_t)bt.ch.expert * nblk + bt.nt + (int64_t)bt.ph * p.n_tiles) * KB + bt.kb;
          if (vec) {
            const float4 v = __ldg(reinterpret_cast<const float4 *>(bs));
            b[0] = v.x; b[1] = v.y; b[2] = v.z; b[3] = v.w;
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) b[i] = bt.kb + i < KB ? __ldg(bs + i) : 0.f;
          }
        };
        Batch cur{ch, 0, 0, 0, false};
        next_item(cur);
        if (cur.valid) fetch(cur, a_cur, b_cur);
        Batch nxt = cur;
        if (nxt.valid) advance(nxt);
        uint32_t n_batch = 0, slot = 0, it = 0;      // batches written, ring position, K-block steps written
        uint32_t end_of[SC_BATCHES];                 // last step of the batch SC_BATCHES - i before this one
#pragma unroll
        for (int i = 0; i < SC_BATCHES; ++i) end_of[i] = 0u;
        while (cur.valid) {
          if (nxt.valid) fetch(nxt, a_nxt, b_nxt);
          // the slot's previous batch has been read when the partial of its last step has been consumed
          if (n_batch >= (uint32_t)SC_BATCHES &&
              !__all_sync(0xffffffffu, mbar_wait(sm, &sm.consumed[end_of[0] % ND], (end_of[0] / ND) & 1u, p.status, 4, LO_SLEEP_SCALE))) break;
          const int T = (cur.ch.rows + 15) & ~15;
          float *sc = &sm.sc[slot * SC_STEPS][0];
#pragma unroll
          for (int u = 0; u < NU; ++u) {
            const int t = lane + u * 32;
            if (t < T) {
              const float live = t < cur.ch.rows ? 1.f : 0.f;
#pragma unroll
              for (int i = 0; i < SC_STEPS; ++i) sc[i * A_ROWS + scale_place<ROW4>(t)] = live != 0.f ? __fmul_rn(a_cur[u][i], b_cur[i]) : 0.f;
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&sm.scales[slot]);
          slot = slot + 1 == (uint32_t)SC_BATCHES ? 0u : slot + 1;
          ++n_batch;
          const int k_left = KB - cur.kb;
          it += (uint32_t)(k_left < SC_STEPS ? k_left : SC_STEPS);
#pragma unroll
          for (int i = 0; i + 1 < SC_BATCHES; ++i) end_of[i] = end_of[i + 1];
          end_of[SC_BATCHES - 1] = it - 1;
#pragma unroll
          for (int u = 0; u < NU; ++u)
#pragma unroll
            for (int i = 0; i < 4; ++i) a_cur[u][i] = a_nxt[u][i];
#pragma unroll
          for (int i = 0; i < 4; ++i) b_cur[i] = b_nxt[i];
          cur = nxt;
          if (nxt.valid) advance(nxt);
        }
        };
        if ((KB & 3) == 0) produce(std::true_type{});
        else produce(std::false_type{});
      }
    } else if (PAIR && rank != 0) {
      // ============ second CTA of a pair, warp 1: passes the partial buffers that its promotion warps hand back on to the issuer ============
      // (One arrival a step across the cluster instead of one of every lane.  Per-channel accumulators are handed back once an item, by the
      // epilogue warps themselves.)
      if (MODE != GEMM_CHANNEL && lane == 0) {
        const uint32_t consumed0 = smem_u32(&sm.consumed[0]);
        const auto peer0 = issuer_barrier<PAIR>(smem_u32(&sm.peer_consumed[0]));
        uint32_t it = 0;
        bool ok = true;
        for (ItemCursor<MODE, FORM, PAIR> items(p, num_chunks); ok && items.take(ch, nt);) {
          if (ch.expert < 0) continue;
#pragma unroll 1
          for (uint32_t u = 0; u < (uint32_t)(PHASES * KB); ++u, ++it) {
            const uint32_t at = 8u * (it & (uint32_t)(ND - 1));
            if (!mbar_wait_addr(sm, consumed0 + at, (it >> 4) & 1u, p.status, 11, LO_SLEEP_MMA)) { ok = false; break; }
            tc_fence_after();
            tc_fence_before();
            mbar_arrive_addr(peer0 + at);
          }
        }
      }
    } else {
      // ============================ MMA issuer (warp 1) ================================
      // A step of this role is a chain of dependent instructions and barrier round trips, which takes longer than the
      // tensor core needs for the step's MMAs.  So: lanes 0 and 1 each own one of the step's two barriers (operands ready,
      // partial buffer free) and look at it in the same instruction; everything the MMAs take (ring positions,
      // descriptors) is computed from values all lanes share, which keeps it in uniform registers (-11 % on the per-channel layer at 20
      // rows per expert against operands shuffled from the polling lanes).  Per-channel mode accumulates an item's steps into one buffer:
      // lane 1 waits for the accumulator once per item.
      // The look at the next step's barriers comes behind this step's MMAs: the warp stands still until a look has its answer (some 100
      // cycles), and what a partial buffer waits for, from its hand-back to the MMAs and on to the promotion, is part of the loop that bounds
      // wide chunks (in front and behind, us: 4096 tokens 2970, 2936; Qwen3 2048 Zipf 815, 808; dense 4096 x 4096 x 7168 196, 193; per channel 2999
      // 2246, 2228; 128 tokens in a graph 1656, 1652; 48 1289, 1286).  With the narrow caps the weights are what is waited for, and the look
      // stands in front: 32 tokens in a graph 1077, behind 1085; 16 x 4096 x 7168 16.7, 17.1; per channel with 64-row chunks (Qwen3 300, composed)
      // 427, 432.  One thread for barriers and MMAs without votes is no faster than with the look in front, predicated MMAs without a
      // branch are 3 % slower.
      uint32_t it = 0;
      // ring positions of the step's operands and partial buffer
      uint32_t sw = 0, sa = 0, sb = 0;
      const uint32_t desc_w0 = (uint32_t)make_smem_desc(smem_u32(sm.w[0])), desc_a0 = (uint32_t)make_smem_desc(smem_u32(sm.a[0]));
      const uint32_t desc_hi = (uint32_t)(make_smem_desc(0u) >> 32);
      const uint32_t tm0 = __shfl_sync(0xffffffffu, tmem_base, 0);
      const uint32_t done0 = smem_u32(&sm.done[0]);
      // this lane's barrier of step u is number (u + my_off) % ND of its ring; a buffer is waited for with the step that
      // used it before (the steps before the first one read as complete: parity 1 of a fresh barrier)
      constexpr int WAITERS = PAIR && MODE != GEMM_CHANNEL ? 3 : 2;      // pairs: lane 2 has the other CTA's partial buffer
      const uint32_t my_base = smem_u32(lane == 0 ? &sm.ready[0] : (lane == 1 ? &sm.consumed[0] : &sm.peer_consumed[0]));
      const uint32_t my_off = lane == 0 ? 0u : 0u - (uint32_t)NBUF;
      uint32_t acc_par = 1;              // per-channel mode: phase of the accumulator ring
      constexpr bool LOOK_BEHIND = A_ROWS > (MODE == GEMM_CHANNEL ? 64 : 32);
      bool ok = true, seen = lane >= WAITERS;
      for (ItemCursor<MODE, FORM, PAIR> items(p, num_chunks); ok && items.take(ch, nt);) {
        if (ch.expert < 0) continue;
        // (a pair's N is a multiple of 32)
        constexpr uint32_t GRAN = PAIR ? 32u : 16u;
        const uint32_t idesc = make_idesc(PAIR ? 256u : 128u, ((uint32_t)__shfl_sync(0xffffffffu, ch.rows, 0) + GRAN - 1u) & ~(GRAN - 1u));
        const uint32_t steps = (uint32_t)(FORM == SPLIT ? items.kn : PHASES * KB);
#pragma unroll 1
        for (uint32_t u = 0; u < steps; ++u, ++it) {
          if (!__all_sync(0xffffffffu, seen)) {
            if (!seen) {
              uint32_t bar = my_base + 8u * ((it + my_off) & (uint32_t)(ND - 1)), par = ((it + my_off) >> 4) & 1u;
              if (MODE == GEMM_CHANNEL && lane == 1) { bar = smem_u32(&sm.tmem_empty[sb]); par = acc_par; }
              seen = mbar_wait_addr(sm, bar, par, p.status, lane == 2 ? 10 : 3 + lane, LO_SLEEP_MMA);
            }
            if (!__all_sync(0xffffffffu, seen)) { ok = false; break; }
            __syncwarp();      // what one lane has seen holds for the lane that issues (a vote does not order memory)
          }
          tc_fence_after();
          const bool last = u == steps - 1;
          auto look = [&] {
            const uint32_t nx = it + 1u + my_off;
            if (MODE == GEMM_CHANNEL) seen = lane > 1 || (lane == 1 && !last) || (lane == 0 && mbar_test_addr(my_base + 8u * (nx & (uint32_t)(ND - 1)), (nx >> 4) & 1u));
            else seen = lane >= WAITERS || mbar_test_addr(my_base + 8u * (nx & (uint32_t)(ND - 1)), (nx >> 4) & 1u);
          };
          if (!LOOK_BEHIND) look();
          // descriptor start addresses are in 16-byte units
          const uint32_t adesc = desc_w0 + sw * (uint32_t)(W_TILE_BYTES >> 4);
          const uint32_t bdesc = desc_a0 + sa * (uint32_t)(CF::A_TILE_BYTES >> 4);
          const uint32_t d = tm0 + sb * (uint32_t)A_ROWS;
          if (elect_one()) {
#pragma unroll
            for (int k4 = 0; k4 < TILE_K / 32; ++k4)
              umma_i8<PAIR>(d, adesc + (uint32_t)(k4 * 2), bdesc + (uint32_t)(k4 * 2), desc_hi, idesc,
                      (MODE == GEMM_CHANNEL ? (u | (uint32_t)k4) : (uint32_t)k4) != 0u ? 1u : 0u);
            umma_commit_addr<PAIR>(done0 + 8u * (it & (uint32_t)(ND - 1)));
            if (MODE == GEMM_CHANNEL && last) umma_commit_addr<PAIR>(smem_u32(&sm.tmem_full[sb]));
          }
          if (LOOK_BEHIND) look();
          __syncwarp();
          sw = sw + 1 == (uint32_t)NW ? 0u : sw + 1;
          sa = sa + 1 == (uint32_t)NA ? 0u : sa + 1;
          if (MODE != GEMM_CHANNEL || last) {
            if (++sb == (uint32_t)NBUF) { sb = 0; acc_par ^= 1u; }
          }
        }
      }
    }
  } else if (MODE != GEMM_CHANNEL && warp >= FIRST_EPI_WARP + EPI_WARPS) {
    // ====================== output warps (block-scaled modes) ======================
    // They turn the finished tile in the staging buffer (bf16, row = token) into rows of global memory while the
    // promotion warps are already on the next item.
    if constexpr (RESPLIT) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_OUT));
    const int ow = warp - (FIRST_EPI_WARP + EPI_WARPS);
    uint32_t par = 0;
    // (the parts of a split K extent leave the kernel as int32 sums, straight from the promotion warps)
    for (ItemCursor<MODE, FORM, PAIR> items(p, FORM == SPLIT ? 0 : num_chunks); items.take(ch, nt);) {
      if (ch.expert < 0) {
        // block of a non-local expert: its output rows are zero
        if (MODE == GEMM_SINGLE && p.C != nullptr) {
          for (int t = ow; t < ch.rows; t += OUT_WARPS) {
            const int32_t sid = FORM == TABLE && p.sorted_ids ? p.sorted_ids[ch.row0 + t] : ch.row0 + t;
            if (sid >= 0 && sid < p.numel_valid)
              for (int64_t n = (int64_t)nt * TILE_N + lane; n < (int64_t)(nt + 1) * TILE_N && n < p.n_store; n += 32)
                p.C[(int64_t)(p.out_by_position ? ch.row0 + t : sid) * p.n_store + n] = __float2bfloat16_rn(0.f);
          }
        }
        continue;
      }
      if constexpr (MODE == GEMM_GATE_UP) {
        // A row of the tile is one token's 128-channel quantisation group: |act| maximum over the warp (four channels
        // per lane), scale = max / 127, q = trunc(clamp(act / scale)), one 4-byte store per lane.
        if (!__all_sync(0xffffffffu, mbar_wait(sm, &sm.stg_full, par, p.status, 9, LO_SLEEP_OUT))) break;
        const int64_t I = (int64_t)p.n_tiles * TILE_N;
        int8_t *q_out = p.act_q + (int64_t)ch.row0 * I + (int64_t)nt * TILE_N + lane * 4;
        float *s_out = p.act_s + (int64_t)ch.row0 * p.n_tiles + nt;
        constexpr int UN = 4;          // tokens in flight per warp
#pragma unroll 1
        for (int t0 = ow * UN; t0 < ch.rows; t0 += OUT_WARPS * UN) {
          float v[UN][4];
          uint32_t m[UN];
#pragma unroll
          for (int e = 0; e < UN; ++e) {
            // (rows of the tile beyond the chunk are inside the staging buffer: T is a multiple of 16)
            const uint2 raw = *reinterpret_cast<const uint2 *>(&sm.staging[(t0 + e) * OUT_ROW_BYTES + lane * 8]);
            v[e][0] = __uint_as_float(raw.x << 16);
            v[e][1] = __uint_as_float(raw.x & 0xffff0000u);
            v[e][2] = __uint_as_float(raw.y << 16);
            v[e][3] = __uint_as_float(raw.y & 0xffff0000u);
            // (a NaN is kept, and as a bit pattern it is above every number in the warp's maximum below: the group's scale does not
            // depend on which of its channels holds one)
            m[e] = __float_as_uint(max_nan(max_nan(fabsf(v[e][0]), fabsf(v[e][1])), max_nan(fabsf(v[e][2]), fabsf(v[e][3]))));
          }
#pragma unroll
          for (int e = 0; e < UN; ++e) m[e] = __reduce_max_sync(0xffffffffu, m[e]);
          // lane e forms the scale of token e, the others fetch it
          uint32_t m_own = m[0];
#pragma unroll
          for (int e = 1; e < UN; ++e) m_own = lane == e ? m[e] : m_own;
          const float scale_own = __fdiv_rn(fmaxf(__uint_as_float(m_own), p.act_eps), 127.0f);
          if (lane < UN && t0 + lane < ch.rows) s_out[(int64_t)(t0 + lane) * p.n_tiles] = scale_own;
          const float rcp_own = rcp_refined(scale_own);
#pragma unroll
          for (int e = 0; e < UN; ++e) {
            const float scale = __shfl_sync(0xffffffffu, scale_own, e), rcp = __shfl_sync(0xffffffffu, rcp_own, e);
            uint32_t packed = 0u;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float r = fminf(fmaxf(div_by(v[e][i], scale, rcp), -128.0f), 127.0f);
              packed |= ((uint32_t)__float2int_rz(r) & 0xffu) << (8 * i);
            }
            if (t0 + e < ch.rows) *reinterpret_cast<uint32_t *>(q_out + (int64_t)(t0 + e) * I) = packed;
          }
        }
      } else {
        // Two token rows per step and warp, sixteen lanes x 16 bytes each.  The rows' ids, weights and addresses are
        // fetched before the wait: lane l of set i / 16 holds those of row half l & 1 of step i with i % 16 == l / 2.
        constexpr int NSET = (A_ROWS / (2 * OUT_WARPS) + 15) / 16;
        unsigned long long rowp_r[NSET];      // address of the row's first output column, 0 = no row
        float wgt_r[NSET];
#pragma unroll
        for (int u = 0; u < NSET; ++u) {
          rowp_r[u] = 0ull;
          wgt_r[u] = 0.f;
          const int t = (u * 16 + (lane >> 1)) * (2 * OUT_WARPS) + ow * 2 + (lane & 1);
          if (t < ch.rows) {
            // without a sorted-id table the id of a row is its position
            const int32_t sid = FORM == TABLE && p.sorted_ids ? p.sorted_ids[ch.row0 + t] : ch.row0 + t;
            if (sid >= 0 && sid < p.numel_valid) {
              if (p.weight_mode == LO_WEIGHT_BF16_PRODUCT) wgt_r[u] = p.topk_weights[sid];
              rowp_r[u] = FORM == TABLE && p.row_dst != nullptr ? (unsigned long long)p.row_dst[sid]
                                               : (unsigned long long)(p.C + (int64_t)(p.out_by_position ? ch.row0 + t : sid) * p.n_store);
            }
          }
        }
        if (!__all_sync(0xffffffffu, mbar_wait(sm, &sm.stg_full, par, p.status, 9, LO_SLEEP_OUT))) break;
        const int64_t n0 = (int64_t)nt * TILE_N + (lane & 15) * 8;
        const int n_steps = (ch.rows + 2 * OUT_WARPS - 1) / (2 * OUT_WARPS);
#pragma unroll 4
        for (int i = 0; i < n_steps; ++i) {
          const int src_lane = (i & 15) * 2 + (lane >> 4);
          const unsigned long long rowp = __shfl_sync(0xffffffffu, pick(rowp_r, i >> 4), src_lane);
          // bf16-product order: bf16(sum) * bf16(w), rounded once more: one packed multiply per two outputs
          const __nv_bfloat162 w2 = __float2bfloat162_rn(__shfl_sync(0xffffffffu, pick(wgt_r, i >> 4), src_lane));
          const int t = i * (2 * OUT_WARPS) + ow * 2 + (lane >> 4);
          if (rowp != 0ull && n0 < p.n_store) {
            __nv_bfloat16 *dst = reinterpret_cast<__nv_bfloat16 *>(rowp) + n0;
            uint4 v = *reinterpret_cast<const uint4 *>(&sm.staging[t * OUT_ROW_BYTES + (lane & 15) * 16]);
            if (p.weight_mode == LO_WEIGHT_BF16_PRODUCT) {
              __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&v);
#pragma unroll
              for (int e = 0; e < 4; ++e) h[e] = __hmul2(h[e], w2);
            }
            if (p.vec_store) {
              *reinterpret_cast<uint4 *>(dst) = v;
            } else {
              for (int e = 0; e < 8 && n0 + e < p.n_store; ++e) dst[e] = reinterpret_cast<const __nv_bfloat16 *>(&v)[e];
            }
          }
        }
      }
      par ^= 1u;
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.stg_free);
    }
  } else {
    // ====================== promotion (block-scaled modes) / epilogue (per-channel mode) ======================
    if constexpr (RESPLIT) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_PROMO));
    const int pw = warp - FIRST_EPI_WARP;
    const int q = warp & 3;              // lane quarter of tensor memory this warp may access
    const int cg = pw >> 2;              // column group: which share of the chunk's tokens
    const uint32_t lane_off = (uint32_t)(q * 32) << 16;
    const int n_local = q * 32 + lane;
    uint32_t ab = 0, fph = 1;                    // per-channel accumulator count; parity of the staging buffer's "free"
    uint32_t sc_slot = 0, sc_par = 0;            // ring of scale batches
    uint32_t buf = 0, step = 0;                  // block-scaled modes: partial buffer and count of the K-block step
    bool ok = true;
    for (ItemCursor<MODE, FORM, PAIR> items(p, num_chunks); ok && items.take(ch, nt);) {
      if (ch.expert < 0) {
        // block of a non-local expert: its output rows are zero (the block-scaled modes leave that to the output warps)
        if (MODE == GEMM_CHANNEL && p.C != nullptr) {
          for (int t = cg; t < ch.rows; t += NCG) {
            const int32_t sid = FORM == TABLE && p.sorted_ids ? p.sorted_ids[ch.row0 + t] : ch.row0 + t;
            if (sid >= 0 && sid < p.numel_valid && (int64_t)nt * TILE_N + n_local < p.n_store)
              p.C[(int64_t)(p.out_by_position ? ch.row0 + t : sid) * p.n_store + (int64_t)nt * TILE_N + n_local] =
                  __float2bfloat16_rn(0.f);
          }
        }
        continue;
      }
      // The chunk's T columns (a multiple of 16) are dealt to the column groups in pieces of 16, as evenly as
      // that allows.
      const int T = (ch.rows + 15) & ~15;
      const int n_pieces = T >> 4;
      const int my_p = n_pieces / NCG + (cg < n_pieces % NCG ? 1 : 0);
      const int col_begin = (cg * (n_pieces / NCG) + min(cg, n_pieces % NCG)) * 16;

      if constexpr (MODE == GEMM_CHANNEL) {
        // ---------------- per-channel mode: one pass over the finished int32 accumulator ----------------
        // Row id and routed weight of token col_begin + 32 * u + lane, fetched now so that the latency is
        // hidden behind the K loop; broadcast by shuffle in the epilogue: piece pc of the group is in
        // register set pc / 2, lanes 16 * (pc & 1) .. + 15.
        constexpr int NPF = ((A_ROWS / 16 + NCG - 1) / NCG + 1) / 2;   // sets of 32 tokens that cover a group's pieces
        int32_t sid_r[NPF];
        float wgt_r[NPF];
        // token scale of column col_begin + lane (broadcast by shuffle) and the scale of this thread's channel
        float as_r[NPF];
#pragma unroll
        for (int u = 0; u < NPF; ++u) {
          sid_r[u] = -1;
          wgt_r[u] = 0.f;
          as_r[u] = 0.f;
          const int t = col_begin + u * 32 + lane;
          if (u * 32 + lane < my_p * 16 && t < ch.rows) {
            // without a sorted-id table the id of a row is its position
            int32_t sid = FORM == TABLE && p.sorted_ids ? p.sorted_ids[ch.row0 + t] : ch.row0 + t;
            if (sid < 0 || sid >= p.numel_valid) sid = -1;
            if (sid >= 0 && p.weight_mode != LO_WEIGHT_NONE) wgt_r[u] = p.topk_weights[sid];
            if (sid >= 0 && p.out_by_position) sid = ch.row0 + t;
            sid_r[u] = sid;
            as_r[u] = __ldg(p.a_scale + ch.row0 + t);
          }
        }
        const int64_t n_glob = (int64_t)nt * TILE_N + n_local;
        const bool n_ok = n_glob < p.n_store;
        const float bs = n_glob < p.n_rows_per_expert ? __ldg(p.b_scale + (int64_t)ch.expert * p.n_rows_per_expert + n_glob) : 0.f;
        const uint32_t b = ab % NBUF;
        const auto empty = issuer_barrier<PAIR>(smem_u32(&sm.tmem_empty[b]));      // the accumulator goes back to the warp that issues the MMAs
        const uint32_t aph = (ab / NBUF) & 1u;
        ++ab;
        if (!__all_sync(0xffffffffu, mbar_wait(sm, &sm.tmem_full[b], aph, p.status, 5))) { ok = false; break; }
        tc_fence_after();
        const uint32_t part = tmem_base + lane_off + b * (uint32_t)A_ROWS + (uint32_t)col_begin;
#pragma unroll 1
        for (int pc = 0; pc < my_p; ++pc) {
          uint32_t raw[16];
          tmem_ld16(part + pc * 16, raw);
          tmem_ld_wait16(raw);
          if (pc == my_p - 1) {
            // every value this warp needs is in registers: hand the buffer back before the stores
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_addr(empty);
          }
          // piece pc holds tokens 16 * pc .. 16 * pc + 15 of this group: register set pc / 2, lanes 16 * (pc & 1) ..
          const int32_t sid_u = pick(sid_r, pc >> 1);
          const float wgt_u = pick(wgt_r, pc >> 1);
          const float as_u = pick(as_r, pc >> 1);
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int src = (pc & 1) * 16 + j;
            const int32_t sid = __shfl_sync(0xffffffffu, sid_u, src);
            const float wgt = __shfl_sync(0xffffffffu, wgt_u, src);
            const float as = __shfl_sync(0xffffffffu, as_u, src);
            if (sid >= 0 && n_ok) {
              float v = __int2float_rn((int32_t)raw[j]);
              if (p.weight_mode == LO_WEIGHT_FP32) v = __fmul_rn(v, wgt);
              v = __fmul_rn(__fmul_rn(v, as), bs);
              if (p.weight_mode == LO_WEIGHT_BF16_PRODUCT) v = bf16_round(v) * bf16_round(wgt);
              p.C[(int64_t)sid * p.n_store + n_glob] = __float2bfloat16_rn(v);
            }
          }
        }
        if (my_p == 0) {
          __syncwarp();
          if (lane == 0) mbar_arrive_addr(empty);
        }
      } else if constexpr (FORM == SPLIT) {
        // ---------------- a part of the K extent: the int32 sum of every K block as it is ----------------
        // What comes after them (scales, fp32 sum, rounding) is left to the kernel that follows, which takes the K blocks in
        // their order: the result has the bits of the undivided form.  Lane = output channel, so a store of a warp is 128
        // consecutive bytes of one token's row.
        const int64_t n = (int64_t)nt * TILE_N + n_local;
        const int64_t slab = p.dense_rows * p.n_store;
        int32_t *dst = p.partial + items.k0 * slab + (int64_t)(ch.row0 + col_begin) * p.n_store + n;
        const int my_rows = n < p.n_store ? min(ch.rows - col_begin, my_p * 16) : 0;
        for (int kb = 0; kb < items.kn; ++kb, ++step, dst += slab) {
          const uint32_t slot = step % ND;
          if (!__all_sync(0xffffffffu, mbar_wait(sm, &sm.done[slot], (step / ND) & 1u, p.status, 5))) { ok = false; break; }
          tc_fence_after();
          const uint32_t part = tmem_base + lane_off + buf * (uint32_t)A_ROWS + (uint32_t)col_begin;
#pragma unroll 1
          for (int pc = 0; pc < my_p; ++pc) {
            uint32_t raw[16];
            tmem_ld16(part + pc * 16, raw);
            tmem_ld_wait16(raw);
            if (pc == my_p - 1) {
              tc_fence_before();
              mbar_arrive(&sm.consumed[slot]);
            }
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (pc * 16 + j < my_rows) dst[(int64_t)(pc * 16 + j) * p.n_store] = (int32_t)raw[j];
          }
          if (my_p == 0) mbar_arrive(&sm.consumed[slot]);
          buf = buf + 1 == (uint32_t)NBUF ? 0u : buf + 1;
        }
      } else {
        // ---------------- block-scaled modes: promotion once per K block, sums in registers ----------------
        // This warp owns the columns [col_begin, col_begin + 16 * my_p) of its 32 lanes.  Their fp32 running sums
        // stay in registers over the whole K loop, so tensor memory holds nothing but partial buffers and a
        // K block costs one tensor-memory load per piece of 16 columns.
        constexpr int NP = (A_ROWS / 16 + NCG - 1) / NCG;
        float acc[NP][16];
        // Addresses of this item, formed once: the loops below only add constants to them.  Ring positions
        // (scale slot, partial buffer and its phase) are carried as counters instead of being divided out of
        // the step numbers.
        const uint32_t part0 = tmem_base + lane_off + (uint32_t)col_begin;
        const uint32_t sc0 = smem_u32(&sm.sc[0][0]) + (uint32_t)col_begin * 4u + (uint32_t)(lane & 3) * 16u;
        const uint32_t done0 = smem_u32(&sm.done[0]), consumed0 = smem_u32(&sm.consumed[0]), scales0 = smem_u32(&sm.scales[0]);
        // this lane's row of the staging tile for the matrix stores and loads of a piece: lanes 8m .. 8m + 7 address the
        // token rows of block m, blocks 0 / 1 are channels 0..7 / 8..15 of tokens 0..7, blocks 2 / 3 of tokens 8..15
        const uint32_t stg_mine = smem_u32(&sm.staging[0]) + (uint32_t)(col_begin + (lane >> 4) * 8 + block_row<ROW4>(lane & 7)) * OUT_ROW_BYTES +
                                  (uint32_t)(q * 32 + ((lane >> 3) & 1) * 8) * 2u;
        // fp32 routed weight of token t of the chunk (0 where there is no row)
        auto weight_of = [&](int t) {
          const int32_t sid = t < ch.rows ? (FORM == TABLE && p.sorted_ids ? p.sorted_ids[ch.row0 + t] : ch.row0 + t) : -1;
          return sid >= 0 && sid < p.numel_valid ? __ldg(p.topk_weights + sid) : 0.f;
        };
#pragma unroll 1
        for (int ph = 0; ph < PHASES; ++ph) {
#pragma unroll
          for (int pc = 0; pc < NP; ++pc)
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[pc][j] = 0.f;
          // The K loop, instantiated for the number of pieces this warp owns in the chunk (and not unrolled further: the two
          // groups run different instantiations, and with four steps unrolled the pair missed the instruction cache, +35 %).
          // What bounds it is neither a pipe nor the issue slots but the chain of one warp (barrier, tensor-memory load,
          // conversion, multiply-add, hand-back: 890 to 1100 cycles a step in the plain order of these, 710 to 790 so).  Every
          // tensor-memory load is issued one unit ahead of its use, the first one of the next step included, and a buffer goes
          // back to the MMA warp as soon as its last unit is in registers, before that unit is promoted.
          auto k_loop = [&](auto pcs) {
            constexpr int PC = decltype(pcs)::value;
            static_assert(PC <= NP, "more pieces than sums");
            constexpr int U = PC;                     // units of a step: two per pair of pieces, one for an odd last piece
            // Units alternate between two register sets.  The next step's first unit goes into set 0 while the last one is
            // promoted: with an odd number of units the last one takes a third set (a single unit: two steps per turn).
            constexpr int UNROLL = PC == 1 ? 2 : 1;
            constexpr int SETS = PC > 1 && (PC & 1) ? 3 : 2;
            uint32_t raw[SETS][16];
            auto load_unit = [&](int u, uint32_t part, uint32_t (&r)[16]) {
              if ((PC & 1) && u == U - 1) tmem_ld_one<ROW4>(part + 16u * (PC - 1), r);
              else tmem_ld_two<ROW4>(part + 32u * (u >> 1) + ((u & 1) ? 16u << 16 : 0u), r);
            };
            uint32_t dn = step & (uint32_t)(ND - 1), dph = (step >> 4) & 1u;      // the step's place in the rings of ND
            if (!__all_sync(0xffffffffu, mbar_wait_addr(sm, done0 + 8u * dn, dph, p.status, 5))) { ok = false; return; }
            tc_fence_after();
            if (PC > 0) load_unit(0, part0 + buf * (uint32_t)A_ROWS, raw[0]);
            uint32_t sc_at = 0;
#pragma unroll 1
            for (int kb0 = 0; kb0 < KB; kb0 += UNROLL) {
              if ((kb0 & (SC_STEPS - 1)) == 0) {
                // the scale products of the coming four steps
                if (PC > 0 && !__all_sync(0xffffffffu, mbar_wait_addr(sm, scales0 + 8u * sc_slot, sc_par, p.status, 7))) { ok = false; return; }
                sc_at = sc0 + sc_slot * (uint32_t)(SC_STEPS * A_ROWS * 4);
                if (++sc_slot == (uint32_t)SC_BATCHES) { sc_slot = 0; sc_par ^= 1u; }
              }
#pragma unroll
              for (int i = 0; i < UNROLL; ++i) {
                if (i > 0 && kb0 + i >= KB) break;
                const uint32_t part = part0 + buf * (uint32_t)A_ROWS;
                const uint32_t used = consumed0 + 8u * dn;
                buf = buf + 1 == (uint32_t)NBUF ? 0u : buf + 1;
                ++step;
                dn = step & (uint32_t)(ND - 1);
                dph = (step >> 4) & 1u;
                float s0[4], s1[4];      // scale products of the pieces at hand
                bool next_done = false;
#pragma unroll
                for (int u = 0; u < (U > 0 ? U : 1); ++u) {
                  const bool last = u == (U > 0 ? U - 1 : 0);
                  const int set = PC == 1 ? i : (SETS == 3 && last ? 2 : u & 1);
                  const int next_set = PC == 1 ? i ^ 1 : (last ? 0 : (SETS == 3 && u + 1 == U - 1 ? 2 : (u + 1) & 1));
                  const bool single = (PC & 1) && u == U - 1;
                  if (PC > 0 && (single || (u & 1) == 0)) {
                    const int pc = single ? PC - 1 : u;
                    lds4(sc_at + (uint32_t)(pc * 64), s0);
                    if (!single) lds4(sc_at + (uint32_t)((pc + 1) * 64), s1);
                  }
                  if (last) next_done = mbar_test_addr(done0 + 8u * dn, dph);
                  if (PC > 0) tmem_ld_wait16(raw[set]);
                  if (!last) {
                    load_unit(u + 1, part, raw[next_set]);
                  } else {
                    // Every value of the partial is in registers: the buffer goes back, the next step's first unit is asked for.
                    // Every lane arrives for itself: what it has read, of the partial and of the batch's scale products, is ordered before
                    // its own arrive.  (One arrive a warp needs a __syncwarp() in front, which cost the chunks of 160 rows 2 to 4 %:
                    // 4096 tokens 2965 -> 3100 us, sharded 8192 788 -> 820 us; arriving with all lanes 2965 -> 2980 us.)
                    tc_fence_before();
                    mbar_arrive_addr(used);
                    if (kb0 + i + 1 < KB) {
                      // warp-uniform outcome: the accesses to tensor memory are warp-collective
                      if (!__all_sync(0xffffffffu, next_done) &&
                          !__all_sync(0xffffffffu, mbar_wait_addr(sm, done0 + 8u * dn, dph, p.status, 5))) { ok = false; return; }
                      tc_fence_after();
                      if (PC > 0) load_unit(0, part0 + buf * (uint32_t)A_ROWS, raw[next_set]);
                    }
                  }
                  if (PC > 0) {
                    if (single) {
                      promote8<ROW4>(&acc[PC > 0 ? PC - 1 : 0][0], &raw[set][0], s0);
                      promote8<ROW4>(&acc[PC > 0 ? PC - 1 : 0][8], &raw[set][8], s0);
                    } else {
                      promote8<ROW4>(&acc[u & ~1][8 * (u & 1)], &raw[set][0], s0);
                      promote8<ROW4>(&acc[(u | 1) < NP ? (u | 1) : 0][8 * (u & 1)], &raw[set][8], s1);
                    }
                  }
                }
                sc_at += (uint32_t)(A_ROWS * 4);
              }
            }
          };
          // (each count is instantiated once: a lambda called from two places is not inlined, and its sums would go to memory)
          if (my_p == 0) k_loop(std::integral_constant<int, 0>{});
          else if (NP == 1 || my_p == 1) k_loop(std::integral_constant<int, 1>{});
          if constexpr (NP >= 2) {
            if (NP == 2 ? my_p >= 2 : my_p == 2) k_loop(std::integral_constant<int, 2>{});
          }
          if constexpr (NP >= 3) {
            if (NP == 3 ? my_p >= 3 : my_p == 3) k_loop(std::integral_constant<int, 3>{});
          }
          if constexpr (NP >= 4) {
            if (NP == 4 ? my_p >= 4 : my_p == 4) k_loop(std::integral_constant<int, 4>{});
          }
          if constexpr (NP >= 5) {
            if (my_p >= 5) k_loop(std::integral_constant<int, 5>{});
          }
          if (!ok) break;
          // routed weight on the fp32 sums (before their rounding), where the mode asks for it
          if (FORM == TABLE && p.weight_mode == LO_WEIGHT_FP32) {
#pragma unroll
            for (int pc = 0; pc < NP; ++pc) {
              if (pc < my_p) {
                float w[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) w[i] = weight_of(col_begin + pc * 16 + token_of<ROW4>(lane & 3, i));
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[pc][j] *= w[((j >> 1) & 2) + (j & 1)];
              }
            }
          }
          if (MODE == GEMM_SINGLE || ph == 0) {
            // The sums (gate_up: those of the gate pass, read back by the same warp below) go to the staging tile as
            // bf16, once the output warps are done with the previous item's tile.
            if (!__all_sync(0xffffffffu, mbar_wait(sm, &sm.stg_free, fph, p.status, 8))) { ok = false; break; }
            fph ^= 1u;
#pragma unroll
            for (int pc = 0; pc < NP; ++pc) {
              if (pc < my_p) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                  const float *a = &acc[pc][8 * h];
                  stmatrix4_t(stg_mine + (uint32_t)(pc * 16 * OUT_ROW_BYTES + h * 32), pack_bf16(a[0], a[1]), pack_bf16(a[2], a[3]),
                              pack_bf16(a[4], a[5]), pack_bf16(a[6], a[7]));
                }
              }
            }
          } else {
            // act = bf16(bf16(silu(bf16(gate))) * bf16(up)) in place of the gate values.  One rolled loop over the pieces:
            // the body always works on piece 0 of the sums (bf16 by then) and the others move down one place afterwards
            // (registers cannot be indexed by a loop counter, and a body unrolled over the pieces would be fetched cold once
            // per item).
            uint32_t up[NP][8];
#pragma unroll
            for (int pc = 0; pc < NP; ++pc)
#pragma unroll
              for (int j = 0; j < 8; ++j) up[pc][j] = pack_bf16(acc[pc][2 * j], acc[pc][2 * j + 1]);
#pragma unroll 1
            for (int pc = 0; pc < my_p; ++pc) {
              const uint32_t addr = stg_mine + (uint32_t)(pc * 16 * OUT_ROW_BYTES);
              uint32_t g2[2][4];
              ldmatrix4_t(addr, g2[0]);
              ldmatrix4_t(addr + 32u, g2[1]);
#pragma unroll
              for (int h = 0; h < 2; ++h) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  float a[2];
#pragma unroll
                  for (int e = 0; e < 2; ++e) {
                    // SiLU as in silu_of_bf16(), but for denominators beyond 2^126, whose reciprocal is flushed (the quotient would be below 1e-36),
                    // and for an infinite sum, which leaves a NaN in its quantisation group
                    const float gte = __uint_as_float(e ? g2[h][j] & 0xffff0000u : g2[h][j] << 16);
                    a[e] = __fmaf_rn(gte, rcp_approx(silu_denominator(gte)), gte * 0.0f);
                  }
                  // bf16(silu) * bf16(up), rounded once: the packed bf16 product
                  const uint32_t sl = pack_bf16(a[0], a[1]);
                  const __nv_bfloat162 act = __hmul2(*reinterpret_cast<const __nv_bfloat162 *>(&sl), *reinterpret_cast<const __nv_bfloat162 *>(&up[0][4 * h + j]));
                  g2[h][j] = *reinterpret_cast<const uint32_t *>(&act);
                }
                stmatrix4_t(addr + 32u * h, g2[h][0], g2[h][1], g2[h][2], g2[h][3]);
              }
#pragma unroll
              for (int pp = 0; pp + 1 < NP; ++pp)
#pragma unroll
                for (int j = 0; j < 8; ++j) up[pp][j] = up[pp + 1][j];
            }
          }
        }
        if (!ok) break;
        // the finished tile is in the staging buffer: over to the output warps
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.stg_full);
      }
    }
  }

  // ------------------------------ teardown -----------------------------------
  tc_fence_before();
  __syncthreads();
  if (sm.abort_flag) {
    // give copies that may still be in flight time to land before the CTA's shared memory is released
    const long long t0 = clock64();
    while (clock64() - t0 < 400000ll) {
    }
  }
  if (PAIR) cluster_sync();      // neither CTA leaves, or frees its tensor memory, while the other may use it
  if (warp == 1) {
    tc_fence_after();
    if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// ------------------------------ host side ----------------------------------

PFN_cuTensorMapEncodeTiled_v12000 get_encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
  });
  return fn;
}

// Tensor map of a [rows, K] int8 matrix, box `box_rows` x 128 bytes, 128-byte swizzle.
// Encoded maps are cached by (base, rows, K, box_rows).
int make_tile_map(CUtensorMap *map, const int8_t *base, int64_t rows, int64_t K, int box_rows) {
  static std::mutex mu;
  static std::map<std::tuple<const void *, int64_t, int64_t, int>, CUtensorMap> cache;
  std::lock_guard<std::mutex> lock(mu);
  auto key = std::make_tuple((const void *)base, rows, K, box_rows);
  auto itc = cache.find(key);
  if (itc != cache.end()) {
    *map = itc->second;
    return LO_OK;
  }
  auto encode = get_encode_fn();
  if (!encode) return fail(LO_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the CUDA driver");
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)K};
  cuuint32_t box[2] = {TILE_K, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<int8_t *>(base), dims, strides, box, estr,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(LO_ERR_CUDA, "cuTensorMapEncodeTiled failed with code %d", (int)r);
  if (cache.size() > 1024) cache.clear();
  cache[key] = *map;
  return LO_OK;
}

template <int MODE, int A_ROWS, int FORM = TABLE, bool PAIR = false>
int launch_mode(const GemmArgs &a, cudaStream_t stream) {
  using SM = Smem<MODE, A_ROWS, PAIR>;
  using CF = Cfg<MODE, A_ROWS, PAIR>;
  static_assert(sizeof(SM) + 1024 <= SMEM_LIMIT, "shared-memory layout exceeds what a CTA can be given");
  static_assert(ND == 16, "the promotion warps take the completion-ring phase from bit 4 of the step count");
  static_assert(CF::NW >= 4, "too few weight stages");
  static_assert(CF::NW < ND && CF::NA < ND && CF::NBUF < ND, "completion ring too short");
  const size_t smem_bytes = sizeof(SM) + 1024;
  // the attribute belongs to the (kernel, device) pair: set it once per device this thread launches on
  static thread_local uint64_t configured_devices = 0;
  int dev = 0;
  LO_CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !((configured_devices >> dev) & 1u)) {
    LO_CUDA_OK(cudaFuncSetAttribute(grouped_gemm_kernel<MODE, A_ROWS, FORM, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes));
    if (dev >= 0 && dev < 64) configured_devices |= (uint64_t)1 << dev;
  }
  CUtensorMap wmap;
  int rc = make_tile_map(&wmap, a.B, (int64_t)a.E * a.n_rows_per_expert, a.K, TILE_N);
  if (rc != LO_OK) return rc;
  AMaps amaps;
  for (int i = 0; i < 4; ++i) {
    rc = make_tile_map(&amaps.m[i], a.A, a.rows_a, a.K, 16 << i);
    if (rc != LO_OK) return rc;
  }
  KParams p;
  p.a_scale = a.a_scale; p.b_scale = a.b_scale;
  p.n_rows_per_expert = a.n_rows_per_expert; p.n_store = a.n_store > 0 ? a.n_store : a.n_rows_per_expert; p.KB = (int)(a.K / TILE_K); p.n_tiles = a.n_tiles;
  p.sorted_ids = a.sorted_ids; p.numel_valid = a.numel_valid;
  p.chunks = a.chunks; p.num_chunks = a.num_chunks; p.act_q = a.act_q; p.act_s = a.act_s; p.C = a.C; p.row_dst = a.row_dst;
  p.topk_weights = a.topk_weights; p.weight_mode = a.weight_mode; p.act_eps = a.act_eps; p.status = a.status;
  p.out_by_position = a.out_by_position;
  // (C is the caller's: a view may begin anywhere; a table of row addresses holds 16-byte aligned ones)
  p.vec_store = (p.n_store & 7) == 0 && (a.row_dst != nullptr || (reinterpret_cast<uintptr_t>(a.C) & 15) == 0) ? 1 : 0;
  p.fixed_chunks = a.fixed_chunks; p.chunk_rows = a.max_chunk_rows; p.masked_m = a.masked_m; p.max_m = a.max_m; p.dense_rows = a.rows_a;
  p.n_split = a.partial != nullptr ? (int)ceil_div(p.KB, a.split_steps) : 1; p.split_steps = a.split_steps; p.partial = a.partial;
  int grid = sm_count();
  if (grid <= 0) return fail(LO_ERR_CUDA, "no CUDA device");
  // No more CTAs than there can be items: each takes its SM's shared memory and the start of the next kernel waits for all of them.  One CTA a SM and
  // so, in us: layer of 32 tokens of the tiny shape in a graph 18.4, 16.4; DeepSeek-V3 one token 71.2, 70.4; dense 40 x 7168 x 2048 10.7, 8.8, 100 x 2304 x
  // 1280 10.1, 9.2.  A split K extent, which comes out near one item a SM, keeps one CTA a SM (6 x 576 x 7168 11.5, 12.1; why is not known).
  if (FORM != SPLIT) {
    const int64_t items = (a.chunks == nullptr ? (int64_t)a.fixed_chunks : (a.max_chunks > 0 ? a.max_chunks : grid)) * a.n_tiles;
    if (items < grid) grid = (int)items;
  }
  LO_CUDA_OK(launch_dependent_clusters(PAIR ? 2 : 1, grouped_gemm_kernel<MODE, A_ROWS, FORM, PAIR>, dim3(PAIR ? grid & ~1 : grid),
                                       dim3(CF::NUM_THREADS), smem_bytes, stream, wmap, amaps, p));
  if (PAIR) g_pair_launch_count.fetch_add(1, std::memory_order_relaxed);
  return LO_OK;
}

// Whether a call with wide chunks runs on pairs of CTAs: tiles come in twos (a pair with one tile idle would waste half of it), and what a
// pair saves, half of the loads of the chunk's rows, has to make up for its start, which waits for the other CTA (0.5 us), and for the slower of
// two CTAs in every step.  So the rule counts the rows that an SM loads: K-block steps (a call with a chunk table has a chunk an expert or more) times
// rows a chunk.  One CTA / pairs, in us, by steps x rows in thousands:
//   dense linear     7 (600 x 4096 x 7168) 44.4 / 44.9      8 (1200 x 7168 x 2048) 33.3 / 34.4     12 (1000 x 4096 x 7168) 52.1 / 51.8
//                   18 (1500 x 4096 x 7168) 77.8 / 76.5    25 (2000 x 4096 x 7168) 104.3 / 102.7   50 (4096 x 4096 x 7168) 204 / 197
//   layers          11 (Qwen3, 4096 tokens of a shard of eight) 200.7 / 202.2    42 (Qwen3 700, Zipf) 431 / 424    85 (Qwen3 2048, Zipf) 887 / 838
//                  400 (DeepSeek-V3 4096) 3160 / 3112
//   per channel, masked layout (both GEMMs), experts of 7168 x 2048: 32 with 1 row 158.7 / 161.2    6 rows 214.6 / 217.8    16 231.7 / 231.3 (6, 3)
//                   24 243.5 / 239.2 (9, 5)     100 319.7 / 316.1        of 4096 x 1536: 32 with 24 rows 113.8 / 115.5 (4, 2)   16 with 80 76.9 / 75.3 (7, 3)
constexpr int64_t PAIR_MIN_ROWS = 12000, PAIR_MIN_ROWS_CHANNEL = 7000;
}  // namespace

bool grouped_gemm_on_pairs(GemmMode mode, int64_t chunks, int64_t rows, int n_tiles, int64_t K) {
  if (n_tiles % 2 != 0 || sm_count() < 2) return false;
  const int64_t steps = chunks * n_tiles * (mode == GEMM_GATE_UP ? 2 : 1) * (K / TILE_K) / sm_count();
  return steps * rows >= (mode == GEMM_CHANNEL ? PAIR_MIN_ROWS_CHANNEL : PAIR_MIN_ROWS);
}

int launch_grouped_gemm(GemmMode mode, const GemmArgs &a, cudaStream_t stream) {
  LO_REQUIRE(a.K % TILE_K == 0 && a.K >= TILE_K, "grouped gemm: K=%lld must be a positive multiple of 128", (long long)a.K);
  LO_REQUIRE(a.n_rows_per_expert % TILE_N == 0 || (a.E == 1 && mode != GEMM_GATE_UP),
             "grouped gemm: N=%lld must be a multiple of 128", (long long)a.n_rows_per_expert);
  LO_REQUIRE((int64_t)a.E * a.n_rows_per_expert < (1LL << 31), "grouped gemm: E*N exceeds the tensor-map row range");
  LO_REQUIRE(a.rows_a >= 1 && a.rows_a < (1LL << 31), "grouped gemm: activation row count out of range");
  LO_REQUIRE((reinterpret_cast<uintptr_t>(a.B) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.A) & 15) == 0 &&
                 (reinterpret_cast<uintptr_t>(a.a_scale) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.b_scale) & 15) == 0,
             "grouped gemm: operands and scales must be 16-byte aligned");
  LO_REQUIRE(a.weight_mode == LO_WEIGHT_NONE || a.topk_weights != nullptr, "grouped gemm: weight mode %d needs topk_weights", a.weight_mode);
  LO_REQUIRE(a.row_dst == nullptr || (mode == GEMM_SINGLE && a.n_rows_per_expert % 8 == 0 && a.out_by_position == 0),
             "grouped gemm: a table of row addresses serves the single block-scaled mode with N a multiple of 8");
  LO_REQUIRE(mode == GEMM_GATE_UP || a.C != nullptr || a.row_dst != nullptr, "grouped gemm: no output");
  LO_REQUIRE((reinterpret_cast<uintptr_t>(a.C) & 1) == 0, "grouped gemm: the output must be aligned to its bf16 elements");
  LO_REQUIRE(a.chunks != nullptr || (a.fixed_chunks >= 1 && a.max_chunk_rows >= 1 && ((mode == GEMM_SINGLE && a.max_chunk_rows <= T_MAX) || (mode == GEMM_CHANNEL && a.masked_m != nullptr))),
             "grouped gemm: no chunk table");
  LO_REQUIRE(a.partial == nullptr || (mode == GEMM_SINGLE && a.chunks == nullptr && a.max_chunk_rows <= T_MAX && a.split_steps >= 1 &&
                                      a.weight_mode == LO_WEIGHT_NONE),
             "grouped gemm: the K extent is split for dense calls only");
  // no chunk can hold more rows than max_chunk_rows (a bound the caller derives from the token count)
  const int cap = a.max_chunk_rows <= 0 ? T_MAX : a.max_chunk_rows;
  const bool pair = a.partial == nullptr && grouped_gemm_on_pairs(mode, a.chunks != nullptr ? a.E : a.fixed_chunks, a.expected_rows < cap ? a.expected_rows : cap, a.n_tiles, a.K);
  if (mode == GEMM_GATE_UP) {
    LO_REQUIRE(a.n_rows_per_expert == 2 * (int64_t)a.n_tiles * TILE_N, "grouped gemm: gate_up needs N = 2*I");
    LO_REQUIRE(cap <= T_WIDE, "grouped gemm: block-scaled chunks hold at most 160 rows");
    if (cap <= 32) return launch_mode<GEMM_GATE_UP, 32>(a, stream);
    if (cap <= 64) return launch_mode<GEMM_GATE_UP, 64>(a, stream);
    if (cap <= 128) return pair ? launch_mode<GEMM_GATE_UP, 128, TABLE, true>(a, stream) : launch_mode<GEMM_GATE_UP, 128>(a, stream);
    return pair ? launch_mode<GEMM_GATE_UP, T_WIDE, TABLE, true>(a, stream) : launch_mode<GEMM_GATE_UP, T_WIDE>(a, stream);
  }
  LO_REQUIRE((int64_t)a.n_tiles * TILE_N >= a.n_rows_per_expert && (int64_t)(a.n_tiles - 1) * TILE_N < a.n_rows_per_expert,
             "grouped gemm: tile count mismatch");
  if (mode == GEMM_CHANNEL) {
    LO_REQUIRE(cap <= 256, "grouped gemm: per-channel chunks hold at most 256 rows");
    if (cap <= 32) return launch_mode<GEMM_CHANNEL, 32>(a, stream);
    if (cap <= 64) return launch_mode<GEMM_CHANNEL, 64>(a, stream);
    if (cap <= 128) return pair ? launch_mode<GEMM_CHANNEL, 128, TABLE, true>(a, stream) : launch_mode<GEMM_CHANNEL, 128>(a, stream);
    if (cap <= T_WIDE) return pair ? launch_mode<GEMM_CHANNEL, T_WIDE, TABLE, true>(a, stream) : launch_mode<GEMM_CHANNEL, T_WIDE>(a, stream);
    return pair ? launch_mode<GEMM_CHANNEL, 256, TABLE, true>(a, stream) : launch_mode<GEMM_CHANNEL, 256>(a, stream);
  }
  LO_REQUIRE(cap <= T_WIDE, "grouped gemm: block-scaled chunks hold at most 160 rows");
  if (a.partial != nullptr) {
    if (cap <= 32) return launch_mode<GEMM_SINGLE, 32, SPLIT>(a, stream);
    if (cap <= 64) return launch_mode<GEMM_SINGLE, 64, SPLIT>(a, stream);
    return launch_mode<GEMM_SINGLE, 128, SPLIT>(a, stream);
  }
  if (a.chunks == nullptr) {
    if (cap <= 32) return launch_mode<GEMM_SINGLE, 32, DENSE>(a, stream);
    if (cap <= 64) return launch_mode<GEMM_SINGLE, 64, DENSE>(a, stream);
    return pair ? launch_mode<GEMM_SINGLE, 128, DENSE, true>(a, stream) : launch_mode<GEMM_SINGLE, 128, DENSE>(a, stream);
  }
  if (cap <= 32) return launch_mode<GEMM_SINGLE, 32>(a, stream);
  if (cap <= 64) return launch_mode<GEMM_SINGLE, 64>(a, stream);
  if (cap <= 128) return pair ? launch_mode<GEMM_SINGLE, 128, TABLE, true>(a, stream) : launch_mode<GEMM_SINGLE, 128>(a, stream);
  return pair ? launch_mode<GEMM_SINGLE, T_WIDE, TABLE, true>(a, stream) : launch_mode<GEMM_SINGLE, T_WIDE>(a, stream);
}

}  // namespace lo
