// The latent decode attention on the Blackwell tensor cores (tcgen05.mma with accumulators in tensor memory), for
// head_dim 128, int8 or f16 latents and ranks up to 64: split-KV stage 1 and, in the balanced mode, also the merge, the
// U_v projection and the head all-gather.
//
// Scores.  For one head, query q and position s
//   z_s = c * sk_s * sum_r Lk[s,r] * W[s,r],
//   W[s,r] = sum_i cos(s f_i) P[r,i] + sin(s f_i) Q[r,i],
//   P[r,i] = q_i U[i,r] + q_{i+64} U[i+64,r],   Q[r,i] = q_{i+64} U[i,r] - q_i U[i+64,r]
// which is the reference's reconstruct -> RoPE -> q.K' chain
// (efficiency/kernel/flash_int8_latent_per_head_decoding_rope_stage1.py:149-169,
// flash_latent_per_head_decoding_rope_stage1.py:84-165 for f16 latents) with the sums reordered: the rotation is moved
// from K onto the query side.  W is one f16 GEMM
//   [128 positions x 128 (cos|sin)] x [128 x 64*(heads of a pair)]
// per tile of 128 positions and pair of heads: the A operand is a tile of a position table of cos/sin values (f16, shared
// by every head and sequence, read from L2 by TMA), the B operand [P;Q] is built once per work item and stays in shared
// memory, the accumulator is fp32 in tensor memory (three 128-column buffers).  Each epilogue thread owns one token: it
// reads its row of W from tensor memory and dots it in fp32 with the token's K row, which it copied from its slot into
// registers at the top of the tile (so that the slot is refilled long before its next use).
//
// Values.  O[r] = sum_s p_s sv_s Lv[s,r] is a true contraction over the tokens and runs on the tensor cores: the A operand
// is a quarter of the V tile exactly as TMA wrote it (32 tokens, swizzled = the MN-major canonical layout), the B operand
// is the tile's weights, written by their owner threads.
//  - int8 V: kind::i8.  a_s = 2^(y_s - max y), y_s = z_s + log2 sv_s, as three unsigned 8-bit digit planes of
//    round(a_s * (2^24 - 256)); the int32 accumulator (64 ranks x 8 columns per (head, warp)) is read back once per tile and
//    folded into a running fp32 sum under a running reference max(y).  The weights lose nothing that fp32 would keep: 24
//    bits relative to the largest weight of the warp's 32 tokens.
//  - f16 V: kind::f16, the weights as three f16 terms of 11 bits each; the fp32 accumulators add up over tiles until a
//    weight outgrows the warp's reference (HeadSums).
// The softmax denominator is accumulated by the owner threads in fp32.
//
// Work.  A work item is a run of consecutive tiles of one (sequence, group of heads: four for int8 latents, two for f16,
// whose rows take twice the shared memory); it ends in one partial result (normalised latent-space row + log-sum-exp per
// head) for the merge.
//  - Balanced mode: all tiles of the batch, ordered by (sequence, head group, tile), are cut
//    into equal shares, one per persistent CTA (one CTA per SM).  A share covers a few items: the
//    tail of one (sequence, head group), whole ones, the head of another.  No SM idles in a
//    partial last wave whatever the sequence lengths, the [P;Q] build is paid once per item, and
//    tensor memory is allocated once.  Every CTA computes its share itself from the sequence
//    lengths.  The partial of item (sequence b, head group hg) of CTA c goes to slot (b * n_hg + hg + c),
//    which is unique because along the tile order every new item advances the (sequence, head group)
//    index or the CTA index.
//    With arrival counters (one per (sequence, head), zeroed before the launch) the kernel is the
//    whole op: the CTA that completes a head's last partial merges the partials, multiplies by
//    the head's slice of U_v and writes the output row; an item that one CTA covers alone skips
//    the partials altogether.  With a peer set on top, the row goes to every rank's gathered
//    buffer (16-byte peer stores) and the CTA that exits last runs the group's barrier.  Without
//    counters the partials and the prefix sums are left for the merge kernel.
//  - Split mode (int8, whole 16-byte rows): CTA blockIdx.x handles split blockIdx.x % n_splits of a fixed-length
//    split plan, partials in the [B, Hq, n_splits] layout of the reference's stage 1.
// Warps (int8: 20, f16: 11):
//   epilogue     4 per head: warp w owns tensor-memory lanes 32*(w%4)..+31, i.e. tokens 32*(w%4).. of every tile of
//                head w/4
//   score MMAs   one warp
//   copies       one warp: table tiles, K and V rows
//   values       one warp per pair of heads: value MMAs
// Every role walks the CTA's items for itself and none waits for the others at an item's end: the phases of the barriers
// run on, the next item's copies start while the last tiles of this one are worked on, and a head's merge and projection
// run while the next item's first score MMAs do.  With int8 latents the epilogue warps and the control warps are two
// register groups: after the launch the control warpgroup gives registers back and the epilogue warpgroups take them
// (setmaxnreg).
// In the busy SM a control thread needs 20-40 cycles per instruction, so waiting for a slot and issuing one copy costs
// 600-800 cycles whatever the size of the copy: hence few and large copies, one tile of all heads at a time where the
// token slots allow it (copy_role).
// What bounds it (13B shape, 16 x 8192 tokens, rank 64): int8 159 us against 107 us for reading the cache at the measured
// HBM rate; neither issue alone (without the dot of the scores 153 us) nor the copies alone: the round trip of the one K slot
// (16 warps copy their rows out, request, arrival) and a tile's work are about as long.  f16 latents 232 us against 208 us.
// Every wait inside the tile loop is an mbarrier wait with a time limit; on a time-out the
// kernel records a status code and every role falls through to the common exit, which frees
// the tensor memory.
#include <cuda.h>
#include <string.h>

#include <atomic>

#include "common.cuh"

namespace wsvd {
namespace tc {

constexpr int kTile = 128;     // positions per MMA tile (= tensor-memory lanes)
constexpr int kRkMax = 64;
constexpr uint32_t kAHalfBytes = kTile * 128;       // 128 rows x 64 f16
constexpr uint32_t kABufBytes = 2 * kAHalfBytes;    // cos half + sin half
constexpr uint32_t kTmemCols = 512;
constexpr float kNone = -3.0e38f;                   // log2-domain reference of something that is still empty

// Shape of the CTA, for int8 latents (four heads) and f16 latents (two heads, whose rows take twice the room).
// ANY: ranks and row addresses that the tensor copies cannot take (rank 62, say).  Every thread then fetches its own
// token's rows in the 16-byte pieces that hold them, K by asynchronous copies a tile ahead, and shifts them into place in
// registers; the rings for K and V rows are not used.
template <bool F16, bool ANY>
struct Cfg {
  static constexpr bool kF16 = F16;
  static constexpr bool kAny = ANY;
  static constexpr int kG = F16 ? 2 : 4;           // heads per CTA
  static constexpr int kEpiWarps = 4 * kG;
  static constexpr int kMmaWarp = kEpiWarps;       // score MMAs
  static constexpr int kLoadWarp = kEpiWarps + 1;  // copies
  static constexpr int kValWarp = kEpiWarps + 2;   // value MMAs: one warp per pair of heads
  static constexpr int kThreads = (kEpiWarps + 2 + kG / 2) * 32;
  static constexpr int kRowBytes = F16 ? 128 : 64; // a latent row in shared memory (rank < 64: zero-filled)
  static constexpr int kKSlots = F16 ? 2 : 1;      // tiles of K: a tile's rows are copied to registers at the top of the tile
  static constexpr int kVSlots = ANY ? 1 : 2;      // tiles of V: the tile whose value MMAs are pending, and the next tile in flight
  static constexpr int kABufs = ANY ? 1 : 2;       // tiles of the position table
  static constexpr uint32_t kRawPitch = kRowBytes + 16;  // ANY: a row as fetched; 16 bytes more than a row: no bank conflicts
  static constexpr int kWBufs = 3;                 // W accumulators of 128 columns (one pair of heads each)
  // int8: 640 threads leave the compiler 96 registers a thread, and the two groups of warps re-balance them.
  // The pool is the CTA's own: what the control warpgroup hands back, (96 - 64) * 128, is exactly what the
  // epilogue warpgroups take, (104 - 96) * 512.  (A request the pool cannot satisfy would block for ever.)
  // f16: 352 threads have 184 each, nothing to re-balance.
  static constexpr int kLaunchRegs = 96;
  static constexpr int kEpiRegs = 104;
  static constexpr int kCtlRegs = 64;
  static_assert(F16 || (kLaunchRegs - kCtlRegs) * 4 * 32 >= (kEpiRegs - kLaunchRegs) * kEpiWarps * 32, "register pool");
  static_assert(F16 || kThreads == (kEpiWarps + 4) * 32, "the control warps must form one warpgroup (4 warps) for setmaxnreg");

  static constexpr uint32_t kHeadBytes = kTile * kRowBytes;  // one head's part of a ring slot
  static constexpr uint32_t kUnitBytes = kG * kHeadBytes;    // a ring slot: one tile of K or V for the group's KV heads
  static constexpr uint32_t kBHalfBytes = kG * kRkMax * 128; // rows of 64 f16
  static constexpr uint32_t kPlaneBytes = F16 ? 512 : 256;   // per pair of warps: 32 tokens x 8 rows of digits
  static constexpr uint32_t kTmemD = kWBufs * 128;           // first column of the value accumulators
  static constexpr uint32_t kDCols = F16 ? 16 : 8;           // per (head, warp): f16 has two of 8 columns
  static_assert(kTmemD + kG * 4 * kDCols <= kTmemCols, "tensor memory");
  // Weights of the value MMA.  int8 V: integers in three digits of 8 bits, relative to the largest of the warp's 32 tokens
  // (a weight of 1 is 2^24 - 256), summed per tile.  f16 V: three f16 terms, each 2^11 below the one before, relative to the
  // warp's reference 2^my_ref (a weight of 1 is 2^15), summed over tiles in tensor memory.
  static constexpr float kPlaneScale = F16 ? 32768.f : 16776960.f;
  // f16: tiles after which a warp goes over to its other accumulator in any case, so that a sum in tensor memory is never
  // more than 32 additions long
  static constexpr int kRenewTiles = 16;

  // shared-memory map (offsets from a 1024-byte aligned base)
  static constexpr uint32_t kOffB = 0;
  static constexpr uint32_t kOffA = kOffB + 2 * kBHalfBytes;
  static constexpr uint32_t kOffV = kOffA + kABufs * kABufBytes;
  static constexpr uint32_t kOffK = kOffV + kVSlots * kUnitBytes;
  static constexpr uint32_t kOffPlanes = kOffK + (ANY ? 2 * kTile * kG * kRawPitch : kKSlots * kUnitBytes);
  static constexpr uint32_t kOffVRaw = kOffK + kTile * kG * kRawPitch;  // ANY
  static constexpr uint32_t kOffRef = kOffPlanes + 2 * kG * kPlaneBytes;  // [head][tile parity][warp] int8: reference of the tile's planes; f16: reference that a warp left with this tile
  static constexpr uint32_t kOffSum = kOffRef + kG * 2 * 4 * 4;           // [head][warp] (max z, denominator) at the end
  static constexpr uint32_t kOffNeg = kOffSum + kG * 4 * 8;               // int8 ANY: [head] four sums, four references, see odd_scales
  static constexpr uint32_t kOffMode = kOffNeg + (!F16 && ANY ? kG * 4 * 8 : 0);  // [4] how the K and V rows of a tile arrive (ring)
  static constexpr uint32_t kOffItem = kOffMode + 16;                     // [head][item parity] ItemState
  static constexpr uint32_t kOffBar = kOffItem + kG * 2 * 64;
  // barriers: V and K full/empty per ring slot, table full/empty, W full/empty, per head: D full,
  // planes ready; [P;Q] ready.  All are initialised once: their phases run on from one item to the next.
  static constexpr int kBarVFull = 0;
  static constexpr int kBarKFull = kBarVFull + kVSlots;
  static constexpr int kBarVEmpty = kBarKFull + kKSlots;
  static constexpr int kBarKEmpty = kBarVEmpty + kVSlots;
  static constexpr int kBarAFull = kBarKEmpty + kKSlots;
  static constexpr int kBarAEmpty = kBarAFull + kABufs;
  static constexpr int kBarWFull = kBarAEmpty + kABufs;
  static constexpr int kBarWEmpty = kBarWFull + kWBufs;
  static constexpr int kBarDFull = kBarWEmpty + kWBufs;
  static constexpr int kBarPlanes = kBarDFull + kG;
  static constexpr int kBarPq = kBarPlanes + kG;
  static constexpr int kNumBars = kBarPq + 1;
  static constexpr uint32_t kOffTmemSlot = kOffBar + kNumBars * 8;
  static constexpr uint32_t kSmemBytes = kOffTmemSlot + 16;  // the dynamic shared-memory base is 1024-byte aligned
  static_assert(kOffA % 1024 == 0 && kOffV % 1024 == 0 && kOffPlanes % 256 == 0 && kOffBar % 8 == 0, "alignment");
  static_assert(kSmemBytes <= 232448, "shared memory budget");

  // Byte offset, inside one head's part of a ring slot, of 16-byte chunk c of token tok (0..127): rows of 64 bytes
  // with the 64-byte swizzle, or of 128 bytes with the 128-byte swizzle.
  static __device__ __forceinline__ uint32_t row_off(int tok, int c) {
    return F16 ? (uint32_t)(tok * 128 + ((c ^ (tok & 7)) << 4)) : (uint32_t)(tok * 64 + ((c ^ ((tok >> 1) & 3)) << 4));
  }
};
static_assert(Cfg<false, false>::kG == kBalancedGroup && Cfg<true, false>::kG == kBalancedGroupF16, "the merge kernel indexes balanced partials by groups of kG heads");

enum Status : unsigned int { kOk = 0, kTimeoutProducer = 1, kTimeoutMma = 2, kTimeoutEpilogue = 3, kBadSmemAlignment = 4 };

__device__ unsigned int g_status = 0;

// ------------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_n(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// try_wait with a suspend-time hint: the waiting thread is parked by the hardware until
// the phase completes or the hint (ns) expires, instead of spinning on issue slots.
constexpr uint32_t kWaitHintNs = 20000;
constexpr uint32_t kSpinSleepNs = 32;
__device__ __forceinline__ uint32_t mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(kWaitHintNs)
      : "memory");
  return ok;
}
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
// Bounded wait: gives up after about two seconds and reports false.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  if (mbar_try(bar, parity)) return true;
  const uint64_t t0 = global_ns();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 256; ++i) {
      if (mbar_try(bar, parity)) return true;
      __nanosleep(kSpinSleepNs);  // leave the issue slots to the warps this one is waiting for
    }
    if (global_ns() - t0 > 2000000000ull) return false;
  }
}
// The same for a whole warp: every lane waits, and the warp agrees on the outcome so that no
// lane leaves a loop that the others stay in.  (The epilogue's tile loop calls mbar_wait without
// the vote: its lanes run in lockstep, wait on the same barrier and read the same timer, so they
// reach the same verdict, and the three votes per tile were 1 % of the kernel's time.)
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity));
}
// one lane of a converged warp (the same one every time): what it guards stays warp-uniform code
__device__ __forceinline__ bool elect_one() {
  uint32_t on;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(on));
  return on != 0;
}
// The thread index, read anew: what is derived from it here is not kept in registers from an earlier phase.
__device__ __forceinline__ int fresh_tid() {
  int t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_but_one() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_i8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr)
               : "memory");
}
// the loaded registers pass through the wait, so that nothing that uses them can be moved in front of it
template <int N>
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&r)[N]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < N; ++i) asm volatile("" : "+r"(r[i]));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// warp-wide maximum in one instruction (sm_100a)
__device__ __forceinline__ float warp_max_redux(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
// the same, NaN if any lane's value is
__device__ __forceinline__ float warp_max_redux_nan(float v) {
  float r;
  asm volatile("redux.sync.max.NaN.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float fast_log2(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Four int8 packed in `w` (already XORed with 0x80808080) -> two fp32 pairs holding the exact
// signed values: byte -> low mantissa of 2^23, then subtract 2^23 + 128.  Packed fp32 arithmetic
// (sm_100 float2 intrinsics): the compiler keeps the pairs in aligned register pairs.
__device__ __forceinline__ void cvt4(uint32_t w, float2& lo, float2& hi) {
  const uint32_t magic = 0x4B000000u;
  const float2 bias = make_float2(-8388736.f, -8388736.f);
  lo = __fadd2_rn(make_float2(__uint_as_float(__byte_perm(w, magic, 0x7650)), __uint_as_float(__byte_perm(w, magic, 0x7651))), bias);
  hi = __fadd2_rn(make_float2(__uint_as_float(__byte_perm(w, magic, 0x7652)), __uint_as_float(__byte_perm(w, magic, 0x7653))), bias);
}

// UMMA shared-memory descriptors (sm_100 descriptor version 1).
// K-major operand, 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);
  d |= (uint64_t)1 << 16;                       // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;             // stride byte offset between 8-row groups
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;                       // SWIZZLE_128B
  return d;
}
// MN-major operand, 64-byte swizzle: 64 bytes along M per K index, 8 K indices per 512 bytes.
__device__ __forceinline__ uint64_t smem_desc_mn_sw64(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);
  d |= (uint64_t)1 << 16;                       // leading byte offset (one 64-byte atom along M: unused)
  d |= (uint64_t)(512 >> 4) << 32;              // stride byte offset between groups of 8 K indices
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)4 << 61;                       // SWIZZLE_64B
  return d;
}
// MN-major operand, 128-byte swizzle: 128 bytes along M per K index, 8 K indices per 1024 bytes.
__device__ __forceinline__ uint64_t smem_desc_mn_sw128(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);
  d |= (uint64_t)1 << 16;                       // leading byte offset (one 128-byte atom along M: unused)
  d |= (uint64_t)(1024 >> 4) << 32;             // stride byte offset between groups of 8 K indices
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;                       // SWIZZLE_128B
  return d;
}
// K-major operand without swizzle, 8 rows: 16-byte K chunks 128 bytes apart, rows 16 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_k_plain(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);
  d |= (uint64_t)(128 >> 4) << 16;              // leading byte offset: between the K chunks
  d |= (uint64_t)(256 >> 4) << 32;              // stride byte offset between 8-row groups (one group: unused)
  d |= (uint64_t)1 << 46;
  return d;
}
__device__ __forceinline__ uint64_t join64(uint32_t lo, uint32_t hi) { return ((uint64_t)hi << 32) | lo; }
// Instruction descriptors.  f16 x f16 -> f32, both operands K-major.
__device__ __forceinline__ uint32_t instr_desc_f16(int m, int n) {
  return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
// s8 (A, MN-major) x u8 (B, K-major) -> s32.
__device__ __forceinline__ uint32_t instr_desc_i8(int m, int n) {
  return (2u << 4) | (1u << 7) | (0u << 10) | (1u << 15) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

struct TcArgs {
  KArgs k;
  int32_t table_rows;
  int32_t use_tma;         // 0: every latent row is gathered by the thread that owns its token
  int32_t box_heads;       // KV heads one tensor copy of a whole tile fetches: up to kG
  int32_t balanced;        // 0: split mode
  int32_t* prefix_out;     // balanced mode: [batch + 2] tile prefix sums and share count for the merge kernel, or null
  unsigned int* arrivals;  // balanced mode: [batch * n_q_heads] zeroed arrival counters = merge inside this kernel, or null
  int32_t has_peers;       // with arrivals: output rows go to every rank's gathered buffer, group barrier at the end
  PeerArgs peers;
  alignas(64) CUtensorMap tmap_k;      // latents as 3-D tensors [KV head][slot][rank]: box rank x 128 slots x box_heads,
  alignas(64) CUtensorMap tmap_v;      // swizzled over the row of shared memory
  alignas(64) CUtensorMap tmap_runs[4];  // the same with boxes of 64 slots x 1 head (K, V) and of 16 slots x 1 head (K, V),
                                         // for tiles made of several runs of slots (a paged cache)
  alignas(64) CUtensorMap tmap_table;  // [2][rows][64] f16, box 64 x 128 x 2 (cos and sin tile), 128-byte swizzle
};

// ------------------------------------------------------------------ position table
// [2][rows][64] f16: plane 0 cos(pos * f_i), plane 1 sin(pos * f_i).
__global__ void rope_table_kernel(__half* table, int rows, KArgs a) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  const int pos = idx >> 6, i = idx & 63;
  if (pos >= rows) return;
  float sn, cs;
  sincosf((float)pos * a.inv_freq[i], &sn, &cs);
  table[(size_t)pos * 64 + i] = __float2half_rn(cs);
  table[((size_t)rows + pos) * 64 + i] = __float2half_rn(sn);
}

// How the K and V rows of a tile reach shared memory: the copying warp publishes 2 * tile + 1 when the epilogue's threads
// are to fetch them, 2 * tile when it copies them, in word tile % 4, before the tile's K slot is handed over (and as
// early as it knows: the epilogue looks a tile ahead).

// A CTA's place in the list of work.
struct Share {
  int b, hg, t_first, tiles_left;  // first item: sequence, head group, tile; tiles of the whole share
  int before_b;                    // tiles in the sequences before b
  int shares;                      // CTAs that have a share
  int64_t total;                   // entries of the tile list
};

// The walk over a CTA's work items.  Every role makes it for itself, so that a role can be in another
// item than its neighbours.
struct Walk {
  int b, hg, t_first, tiles_left, before_b;
  int n, req;            // length and request of sequence b
  int tiles_b;           // balanced mode: tiles of sequence b
  int lo, hi, ntiles;    // the item: tokens [lo, hi) of (b, head group hg)

  __device__ __forceinline__ void cut() {
    tiles_b = (n + kTile - 1) / kTile;
    ntiles = min(tiles_left, tiles_b - t_first);
    lo = t_first * kTile;
    hi = min(n, (t_first + ntiles) * kTile);
  }
  // false: the CTA has no work
  __device__ __forceinline__ bool start(const TcArgs& ta, const Share& sh, int n_hg) {
    const WsvdLatentDecodeParams& p = ta.k.p;
    if (ta.balanced) {
      if (sh.tiles_left <= 0) return false;
      b = sh.b, hg = sh.hg, t_first = sh.t_first, tiles_left = sh.tiles_left, before_b = sh.before_b;
      n = p.b_seq_len[b], req = p.b_req_idx[b];
      cut();
      return true;
    }
    // one fixed-length split; an empty one writes nothing
    const int split = blockIdx.x % ta.k.n_splits;
    hg = (blockIdx.x / ta.k.n_splits) % n_hg, b = blockIdx.x / (ta.k.n_splits * n_hg);
    t_first = 0, before_b = 0, tiles_b = 0;
    n = p.b_seq_len[b], req = p.b_req_idx[b];
    lo = split * ta.k.split_len;
    hi = min(n, lo + ta.k.split_len);
    ntiles = tiles_left = (hi - lo + kTile - 1) / kTile;
    return hi > lo;
  }
  // the next item of the share: the next head group, or the next sequence that has tokens
  __device__ __forceinline__ bool next(const WsvdLatentDecodeParams& p, int n_hg) {
    tiles_left -= ntiles;
    if (tiles_left <= 0) return false;
    t_first = 0;
    if (++hg == n_hg) {
      hg = 0;
      before_b += tiles_b;
      do {
        if (++b >= p.batch) return false;
        n = p.b_seq_len[b];
      } while (n <= 0);
      req = p.b_req_idx[b];
    }
    cut();
    return true;
  }
};

// ------------------------------------------------------------------ score MMAs (one warp)
template <class C>
__device__ __forceinline__ void score_role(const TcArgs& ta, const Share& sh, uint32_t sbase, uint32_t tmem) {
  const WsvdLatentDecodeParams& p = ta.k.p;
  const int n_hg = (p.n_q_heads + C::kG - 1) / C::kG;
  auto bar = [&](int i) { return sbase + C::kOffBar + 8u * i; };
  // descriptors: only the start-address field changes between k-steps, buffers and pairs
  const uint64_t adesc0 = smem_desc_sw128(sbase + C::kOffA), bdesc0 = smem_desc_sw128(sbase + C::kOffB);
  const uint32_t a_lo = (uint32_t)adesc0, b_lo = (uint32_t)bdesc0, d_hi = (uint32_t)(adesc0 >> 32);
  const bool issuer = elect_one();
  Walk w;
  bool ok = true;
  uint32_t T = 0, u = 0, item = 0;  // tiles, (tile, pair) units (unit u uses W buffer u % kWBufs) and items so far
  for (bool more = w.start(ta, sh, n_hg); more && ok; more = w.next(p, n_hg), ++item) {
    const int G = min(C::kG, p.n_q_heads - w.hg * C::kG), npairs = (G + 1) >> 1;
    ok = warp_wait(bar(C::kBarPq), item & 1);
    for (int t = 0; t < w.ntiles && ok; ++t, ++T) {
      const uint32_t buf = T % C::kABufs;
      ok = warp_wait(bar(C::kBarAFull + buf), (T / C::kABufs) & 1);
      for (int pr = 0; pr < npairs && ok; ++pr, ++u) {
        const uint32_t wb = u % C::kWBufs, use = u / C::kWBufs;
        if (use > 0) ok = warp_wait(bar(C::kBarWEmpty + wb), (use - 1) & 1);
        if (!ok) break;
        tc_fence_after();
        const uint32_t idesc = instr_desc_f16(kTile, kRkMax * min(2, G - 2 * pr));
        const uint32_t d_tmem = tmem + wb * 128;
        const uint32_t a_at = a_lo + buf * (kABufBytes >> 4), b_at = b_lo + pr * ((2 * kRkMax * 128) >> 4);
        if (issuer) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            umma_f16(d_tmem, join64(a_at + (((kk >> 2) * kAHalfBytes + (kk & 3) * 32) >> 4), d_hi),
                     join64(b_at + (((kk >> 2) * C::kBHalfBytes + (kk & 3) * 32) >> 4), d_hi), idesc, kk > 0);
          umma_commit(bar(C::kBarWFull + wb));
          if (pr == npairs - 1) umma_commit(bar(C::kBarAEmpty + buf));
        }
        __syncwarp();
      }
    }
  }
  // the releases of the last table buffers are arrivals that nobody else waits for: none may be on its way
  // when the CTA exits
  for (uint32_t t = T < C::kABufs ? 0 : T - C::kABufs; t < T && ok; ++t)
    ok = warp_wait(bar(C::kBarAEmpty + t % C::kABufs), (t / C::kABufs) & 1);
  if (!ok) atomicMax(&g_status, (unsigned)kTimeoutMma);
}

// ------------------------------------------------------------------ copies (one warp)
// Per tile, in this order, each as soon as its slot is free: the table tile (free when the score MMAs of the
// tile two before it are complete), the K rows (when every warp has copied the rows of the tile before to
// registers), the V rows (when the value MMAs of the tile two before are complete).  The warp runs on into
// the next item while the epilogue finishes the last one.
// A tensor copy needs token slots that are consecutive.  The warp checks that tile by tile: lane l holds the
// page entries of tokens 4l..4l+3 (fetched one tile ahead), and the warp votes.
//  - the tile's 128 slots are one run (a cache laid out sequence by sequence, a page of 128 or more): one copy
//    for K and one for V fetch all heads of the group;
//  - every aligned group of 64, or else of 16, tokens is a run (a paged cache): one copy per run and head.  A copy
//    costs this warp about 80 cycles whatever its size: 24 sequences of 500 to 4096 tokens, 32 heads, took 82 us in
//    one run, 118 us with pages of 64 copied by sixteens, 88 us by 64;
//  - else the epilogue's warps fetch their own tokens' rows.
template <class C>
__device__ __forceinline__ void copy_role(const TcArgs& ta, const Share& sh, uint32_t sbase, uint8_t* sm) {
  const WsvdLatentDecodeParams& p = ta.k.p;
  const int lane = threadIdx.x & 31;
  const int n_hg = (p.n_q_heads + C::kG - 1) / C::kG, gqa = p.n_q_heads / p.n_kv_heads;
  auto bar = [&](int i) { return sbase + C::kOffBar + 8u * i; };
  volatile int* mode = reinterpret_cast<volatile int*>(sm + C::kOffMode);
  const bool issuer = elect_one();
  const uint32_t box_bytes = ta.box_heads * C::kHeadBytes;
  const bool use_tma = ta.use_tma != 0;
  Walk w;
  bool ok = true;
  uint32_t T = 0;
  for (bool more = w.start(ta, sh, n_hg); more && ok; more = w.next(p, n_hg)) {
    const int h0 = w.hg * C::kG, G = min(C::kG, p.n_q_heads - h0);
    const int hk0 = h0 / gqa, nkv = (h0 + G - 1) / gqa - hk0 + 1;  // the group's KV heads
    const int32_t* page = p.req_to_token + (int64_t)w.req * p.rtt_stride;
    int pos = (p.pos_offset != nullptr ? p.pos_offset[w.b] : 0) + w.lo;  // RoPE position of the tile's first token
    if constexpr (C::kAny) {  // the position table alone
      for (int t = 0; t < w.ntiles && ok; ++t, ++T, pos += kTile) {
        const uint32_t buf = T % C::kABufs, au = T / C::kABufs;
        if (au > 0) ok = warp_wait(bar(C::kBarAEmpty + buf), (au - 1) & 1);
        if (ok && issuer) {
          mbar_expect_tx(bar(C::kBarAFull + buf), kABufBytes);
          tma_load_3d(sbase + C::kOffA + buf * kABufBytes, &ta.tmap_table, 0, pos, 0, bar(C::kBarAFull + buf));
        }
      }
      continue;
    }
    int ent[4];
    auto fetch_entries = [&](int t) {
      const int s0 = w.lo + t * kTile + 4 * lane;
#pragma unroll
      for (int j = 0; j < 4; ++j) ent[j] = s0 + j < w.hi ? page[s0 + j] : -1;
    };
    fetch_entries(0);
    for (int t = 0; t < w.ntiles && ok; ++t, ++T, pos += kTile) {
      // ---- position table
      const uint32_t buf = T % C::kABufs, au = T / C::kABufs;
      if (au > 0) ok = warp_wait(bar(C::kBarAEmpty + buf), (au - 1) & 1);
      if (!ok) break;
      if (issuer) {
        mbar_expect_tx(bar(C::kBarAFull + buf), kABufBytes);
        tma_load_3d(sbase + C::kOffA + buf * kABufBytes, &ta.tmap_table, 0, pos, 0, bar(C::kBarAFull + buf));
      }
      // ---- which way the rows come (entries past the end are -1 and match anything)
      const int first = __shfl_sync(0xffffffffu, ent[0], 0);
      bool good = use_tma;
#pragma unroll
      for (int j = 0; j < 4; ++j) good = good && (ent[j] < 0 || ent[j] == first + 4 * lane + j);
      const bool run = __all_sync(0xffffffffu, good);
      // not one run: two of 64 slots, or eight of 16?  Lane l copies run l / 4 of KV head l % 4.
      int len = 0, first_r = 0, groups = 0;  // length of a run, first slot of this lane's run (-1: past the end), runs that hold tokens
      if (!run) {
#pragma unroll
        for (int lg = 4; lg >= 2 && len == 0; lg -= 2) {  // a run spans 2^lg lanes' entries
          const int first_l = __shfl_sync(0xffffffffu, ent[0], lane & ~((1 << lg) - 1));
          good = use_tma;
#pragma unroll
          for (int j = 0; j < 4; ++j) good = good && (ent[j] < 0 || ent[j] == first_l + 4 * (lane & ((1 << lg) - 1)) + j);
          if (__all_sync(0xffffffffu, good)) {
            len = 4 << lg;
            groups = __popc(__ballot_sync(0xffffffffu, first_l >= 0)) >> lg;
            first_r = __shfl_sync(0xffffffffu, ent[0], ((lane >> 2) << lg) & 31);
            if (lane >= 4 * (32 >> lg)) first_r = -1;
          }
        }
      }
      if (issuer) mode[T & 3] = (int)(2 * T) + (!run && len == 0);
      if (t + 1 < w.ntiles) fetch_entries(t + 1);
      auto request = [&](const CUtensorMap* whole, const CUtensorMap* part, uint32_t dst, uint32_t full) {
        if (run) {
          if (issuer) {
            mbar_expect_tx(full, box_bytes);
            tma_load_3d(dst, whole, 0, first, hk0, full);
          }
        } else if (len != 0) {
          if (issuer) {
            mbar_expect_tx(full, (uint32_t)(groups * nkv * len) * C::kRowBytes);
          }
          __syncwarp();
          const int j = lane & 3;
          if (j < nkv && first_r >= 0)
            tma_load_3d(dst + j * C::kHeadBytes + (lane >> 2) * (len * C::kRowBytes), part + (len == 64 ? 0 : 2), 0, first_r, hk0 + j, full);
        } else if (issuer) {
          mbar_arrive(full);
        }
      };
      // ---- K rows, V rows
      const uint32_t ks = T % C::kKSlots, ku = T / C::kKSlots, vs = T % C::kVSlots, vu = T / C::kVSlots;
      if (ku > 0) ok = warp_wait(bar(C::kBarKEmpty + ks), (ku - 1) & 1);
      if (!ok) break;
      request(&ta.tmap_k, &ta.tmap_runs[0], sbase + C::kOffK + ks * C::kUnitBytes, bar(C::kBarKFull + ks));
      if (vu > 0) ok = warp_wait(bar(C::kBarVEmpty + vs), (vu - 1) & 1);
      if (!ok) break;
      request(&ta.tmap_v, &ta.tmap_runs[1], sbase + C::kOffV + vs * C::kUnitBytes, bar(C::kBarVFull + vs));
    }
  }
  // as in the score role: the releases of the last V slots
  for (uint32_t t = T < C::kVSlots ? 0 : T - C::kVSlots; t < T && ok && !C::kAny; ++t)
    ok = warp_wait(bar(C::kBarVEmpty + t % C::kVSlots), (t / C::kVSlots) & 1);
  if (!ok) atomicMax(&g_status, (unsigned)kTimeoutProducer);
}

// ------------------------------------------------------------------ value MMAs (one warp per pair of heads)
// One byte per warp of head g: bit 0 which of its two value accumulators this tile's sums go to, bit 1 whether
// they are added to it.  (It sits in the unused last word of the head's first ItemState.)
template <class C>
__device__ __forceinline__ volatile uint32_t* value_modes(uint8_t* sm, int g) {
  return reinterpret_cast<volatile uint32_t*>(sm + C::kOffItem + g * 128 + 60);
}

// The warp serves its two heads in turn: it waits for the digit planes of a head's four warps and issues the
// head's value MMAs (one per warp of 32 tokens, each into 8 columns of tensor memory of its own); two commits
// then tell the epilogue warps (D full) and the copying warp (V empty) when the MMAs have completed.  All lanes
// hold the same operands and flags: the instruction takes them from uniform registers, and when two lanes
// served a head each, one head's sums were now and then added to, or not, as the other's should have been.
template <class C>
__device__ __forceinline__ void value_role(const TcArgs& ta, const Share& sh, uint32_t sbase, uint8_t* sm,
                                           uint32_t tmem, int pair) {
  const WsvdLatentDecodeParams& p = ta.k.p;
  const int n_hg = (p.n_q_heads + C::kG - 1) / C::kG, gqa = p.n_q_heads / p.n_kv_heads;
  auto bar = [&](int i) { return sbase + C::kOffBar + 8u * i; };
  const uint32_t idesc = C::kF16 ? instr_desc_f16(64, 8) | (1u << 15) : instr_desc_i8(64, 8);
  const volatile int* mode = reinterpret_cast<const volatile int*>(sm + C::kOffMode);
  const uint64_t vdesc0 = C::kF16 ? smem_desc_mn_sw128(sbase + C::kOffV) : smem_desc_mn_sw64(sbase + C::kOffV), pdesc0 = smem_desc_k_plain(sbase + C::kOffPlanes);
  const uint32_t v_lo = (uint32_t)vdesc0, v_hi = (uint32_t)(vdesc0 >> 32), p_lo = (uint32_t)pdesc0, p_hi = (uint32_t)(pdesc0 >> 32);
  const bool issuer = elect_one();
  Walk w;
  bool ok = true, skipped = false;   // skipped: the pair was not there in the item before
  uint32_t T = 0, mine[2] = {0, 0};  // tiles so far, and those that each head took part in
  for (bool more = w.start(ta, sh, n_hg); more && ok; more = w.next(p, n_hg)) {
    const int h0 = w.hg * C::kG, G = min(C::kG, p.n_q_heads - h0);
    if (2 * pair >= G) {
      T += w.ntiles;
      skipped = true;
      continue;
    }
    // After tiles that passed this warp by the parity of V full says nothing, for the barrier may be phases behind.  The
    // planes, whose phases are this warp's own, are ready only when all tiles of the item before are done with.
    if (skipped) ok = warp_wait(bar(C::kBarPlanes + 2 * pair), mine[0] & 1);
    skipped = false;
    for (int t = 0; t < w.ntiles && ok; ++t, ++T) {
      const uint32_t vslot = T % C::kVSlots;
      // the V rows arrive long before the planes are ready: wait for them first, off the
      // critical path from "planes ready" to "D full"
      if constexpr (!C::kAny) ok = warp_wait(bar(C::kBarVFull + vslot), (T / C::kVSlots) & 1);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int g = 2 * pair + j;
        if (g >= G || !ok) break;
        ok = warp_wait(bar(C::kBarPlanes + g), mine[j] & 1);
        if (!ok) break;
        ++mine[j];
        tc_fence_after();
        const uint32_t how = C::kF16 ? *value_modes<C>(sm, g) : 0u;  // a byte per warp: which of its accumulators, added to or started
        // copied rows sit at the head's KV head, gathered ones at the head itself
        const int sub = C::kAny || (mode[T & 3] & 1) ? g : (h0 + g) / gqa - h0 / gqa;
        const uint32_t v_at = v_lo + ((vslot * C::kUnitBytes + sub * C::kHeadBytes) >> 4);
        const uint32_t d_tmem = tmem + C::kTmemD + 4 * C::kDCols * g;
        if (issuer) {
#pragma unroll
          for (int w4 = 0; w4 < 4; ++w4) {  // the 32 tokens of warp w4: 32 rows
            const uint32_t d = d_tmem + C::kDCols * w4 + ((how >> (8 * w4)) & 1) * 8;
            const uint32_t va = v_at + ((w4 * 32 * C::kRowBytes) >> 4), pa = p_lo + (((2 * g + (w4 >> 1)) * C::kPlaneBytes) >> 4);
            if constexpr (C::kF16) {  // 16 tokens an instruction
              umma_f16(d, join64(va, v_hi), join64(pa, p_hi), idesc, (how >> (8 * w4)) & 2);
              umma_f16(d, join64(va + (2048 >> 4), v_hi), join64(pa + (256 >> 4), p_hi), idesc, 1);
            } else {
              umma_i8(d, join64(va, v_hi), join64(pa, p_hi), idesc, 0);
            }
          }
          umma_commit(bar(C::kBarDFull + g));
          if constexpr (!C::kAny) umma_commit(bar(C::kBarVEmpty + vslot));
          if (!C::kAny && g == 0 && G < C::kG) mbar_arrive_n(bar(C::kBarVEmpty + vslot), C::kG - G);  // for the heads that are not there
        }
        __syncwarp();
      }
    }
  }
  if (!ok) atomicMax(&g_status, (unsigned)kTimeoutProducer);
}

// ------------------------------------------------------------------ epilogue (four warps per head)
// Where chunk ic (8 frequencies) of rank r of head g sits in either half of the B operand.
__device__ __forceinline__ uint32_t pq_off(int g, int r, int ic) {
  const int nrow = g * kRkMax + r;
  return nrow * 128 + ((ic ^ (nrow & 7)) << 4);
}

// Asks for what the [P;Q] build of an item needs from memory: the head's slice of wk goes, without passing
// through registers, to the places in the B operand that the thread which asked for it will overwrite with P
// and Q; the page entries of the first two tiles go to L1.
template <class C>
__device__ __forceinline__ void request_pq(const TcArgs& ta, uint32_t sbase, const Walk& w, int g, bool wk_vec) {
  const WsvdLatentDecodeParams& p = ta.k.p;
  const int gqa = p.n_q_heads / p.n_kv_heads, hk = (w.hg * C::kG + g) / gqa;
  const bool il = p.rope_layout == WSVD_ROPE_INTERLEAVED, wk_i8 = p.wk_dtype == WSVD_I8;
  const int tid = threadIdx.x & 127, ic = tid & 7;
  const int d0 = il ? ic * 16 : ic * 8, d1 = il ? ic * 16 + 8 : 64 + ic * 8;
  if (wk_vec) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = (tid + 128 * i) >> 3;
      if (r >= p.rank_k) continue;
      const uint32_t dst = sbase + C::kOffB + pq_off(g, r, ic);
      const int64_t at = (int64_t)r * p.wk_stride_r + (int64_t)hk * 128;
      if (wk_i8) {
        const int8_t* s = reinterpret_cast<const int8_t*>(p.wk) + at;
        cp_async8(dst, s + d0);
        cp_async8(dst + C::kBHalfBytes, s + d1);
      } else {
        const __half* s = reinterpret_cast<const __half*>(p.wk) + at;
        cp_async16(dst, s + d0);
        cp_async16(dst + C::kBHalfBytes, s + d1);
      }
    }
  }
  const int32_t* page = p.req_to_token + (int64_t)w.req * p.rtt_stride;
  const int s_first = w.lo + tid;
  if (s_first < w.hi) asm volatile("prefetch.global.L1 [%0];" ::"l"(page + s_first));
  if (s_first + kTile < w.hi) asm volatile("prefetch.global.L1 [%0];" ::"l"(page + s_first + kTile));
}

// B operand: P (cos coefficients) and Q (sin coefficients) of head g of the group, f16, rows n = g*64 + r, 64
// frequencies per row, 128-byte swizzle; rows r >= rank_k are zero.
template <class C>
__device__ __forceinline__ void build_pq(const TcArgs& ta, uint8_t* sm, int b, int h, int hk, int g, bool wk_vec) {
  const KArgs& a = ta.k;
  const WsvdLatentDecodeParams& p = a.p;
  const bool interleaved = p.rope_layout == WSVD_ROPE_INTERLEAVED, wk_i8 = p.wk_dtype == WSVD_I8;
  const int tid = threadIdx.x & 127;
  uint4 qv0, qv1;  // the 16 query values of this thread's chunk of 8 frequencies
  {
    const int ic = tid & 7;
    const __half* qp = reinterpret_cast<const __half*>(p.q) + (int64_t)b * p.q_stride_b + (int64_t)h * p.q_stride_h;
    qv0 = *reinterpret_cast<const uint4*>(qp + (interleaved ? ic * 16 : ic * 8));
    qv1 = *reinterpret_cast<const uint4*>(qp + (interleaved ? ic * 16 + 8 : 64 + ic * 8));
  }
  uint4 s0v = make_uint4(0u, 0u, 0u, 0u), s1v = s0v;  // int8 wk: the scales of the chunk's two sets of dimensions
  if (wk_vec && wk_i8) {
    const int ic = tid & 7;
    const __half* ws = reinterpret_cast<const __half*>(p.wk_scale) + (int64_t)hk * 128;
    s0v = *reinterpret_cast<const uint4*>(ws + (interleaved ? ic * 16 : ic * 8));
    s1v = *reinterpret_cast<const uint4*>(ws + (interleaved ? ic * 16 + 8 : 64 + ic * 8));
  }
  cp_async_wait_all();  // this thread's own pieces of wk
  // q * sm_scale * log2(e) (scores come out in the log2 domain): qlo[e] pairs with dimension
  // d0 and qhi[e] with its rotation partner d1 of frequency ic*8 + e
  float qlo[8], qhi[8];
  {
    const float qscale = a.sm_scale * 1.4426950408889634f;
    const __half* q0 = reinterpret_cast<const __half*>(&qv0);
    const __half* q1 = reinterpret_cast<const __half*>(&qv1);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      if (interleaved) {
        const __half* src = e < 4 ? q0 : q1;
        qlo[e] = __half2float(src[(2 * e) & 7]) * qscale;
        qhi[e] = __half2float(src[(2 * e + 1) & 7]) * qscale;
      } else {
        qlo[e] = __half2float(q0[e]) * qscale;
        qhi[e] = __half2float(q1[e]) * qscale;
      }
    }
  }
  const int64_t col = (int64_t)hk * 128;
  if (!C::kF16 && !C::kAny && wk_vec && !wk_i8 && !interleaved) {
    // Common case (int8 latents in whole 16-byte rows, f16 wk, half-split pairing): packed f16 arithmetic.  The operands are
    // rounded to f16 for the MMA anyway; forming them with one extra f16 rounding of a
    // product keeps the error of the scores within a few 1e-5.  This thread's chunk of 8
    // frequencies is the same for its four ranks, so q is converted once.
    const int ic = tid & 7;
    __half2 qa[4], qb[4], nqa[4];
    {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        qa[e] = __floats2half2_rn(qlo[2 * e], qlo[2 * e + 1]);
        qb[e] = __floats2half2_rn(qhi[2 * e], qhi[2 * e + 1]);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) nqa[e] = __hneg2(qa[e]);
    }
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int r = (tid + 128 * it) >> 3;
      const uint32_t off = pq_off(g, r, ic);
      uint4 u_lo = make_uint4(0u, 0u, 0u, 0u), u_hi = u_lo;
      if (r < p.rank_k) {
        u_lo = *reinterpret_cast<const uint4*>(sm + C::kOffB + off);
        u_hi = *reinterpret_cast<const uint4*>(sm + C::kOffB + C::kBHalfBytes + off);
      }
      const __half2* ua = reinterpret_cast<const __half2*>(&u_lo);  // U[d = ic*8 .. +7]
      const __half2* ub = reinterpret_cast<const __half2*>(&u_hi);  // U[64 + ic*8 .. +7]
      __align__(16) __half2 pv[4];
      __align__(16) __half2 qv[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        pv[e] = __hfma2(qa[e], ua[e], __hmul2(qb[e], ub[e]));   // P = q_i U_i + q_{i+64} U_{i+64}
        qv[e] = __hfma2(nqa[e], ub[e], __hmul2(qb[e], ua[e]));  // Q = q_{i+64} U_i - q_i U_{i+64}
      }
      *reinterpret_cast<uint4*>(sm + C::kOffB + off) = *reinterpret_cast<const uint4*>(pv);
      *reinterpret_cast<uint4*>(sm + C::kOffB + C::kBHalfBytes + off) = *reinterpret_cast<const uint4*>(qv);
    }
  } else if (wk_vec && wk_i8) {
    // int8 wk in vectors of eight; the columns' scales are this thread's for all four ranks.  fp32 throughout.
    const int ic = tid & 7;
    const __half* s0h = reinterpret_cast<const __half*>(&s0v);
    const __half* s1h = reinterpret_cast<const __half*>(&s1v);
#pragma unroll 2
    for (int it = 0; it < 4; ++it) {
      const int r = (tid + 128 * it) >> 3;
      const uint32_t off = pq_off(g, r, ic);
      uint2 b0 = make_uint2(0u, 0u), b1 = b0;
      if (r < p.rank_k) {
        b0 = *reinterpret_cast<const uint2*>(sm + C::kOffB + off);
        b1 = *reinterpret_cast<const uint2*>(sm + C::kOffB + C::kBHalfBytes + off);
      }
      __align__(16) __half pv[8];
      __align__(16) __half qv[8];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        // bytes of dimension d0 and d1 of four frequencies
        uint32_t w0, w1;
        if (interleaved) {
          const uint2 src = half == 0 ? b0 : b1;
          w0 = __byte_perm(src.x, src.y, 0x6420);
          w1 = __byte_perm(src.x, src.y, 0x7531);
        } else {
          w0 = half == 0 ? b0.x : b0.y;
          w1 = half == 0 ? b1.x : b1.y;
        }
        const __half* pair = half == 0 ? s0h : s1h;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int e = 4 * half + j;
          const float s0 = __half2float(interleaved ? pair[(2 * e) & 7] : s0h[e]);
          const float s1 = __half2float(interleaved ? pair[(2 * e + 1) & 7] : s1h[e]);
          const float u0 = (float)(int8_t)(w0 >> (8 * j)) * s0, u1 = (float)(int8_t)(w1 >> (8 * j)) * s1;
          pv[e] = __float2half_rn(qlo[e] * u0 + qhi[e] * u1);
          qv[e] = __float2half_rn(qhi[e] * u0 - qlo[e] * u1);
        }
      }
      *reinterpret_cast<uint4*>(sm + C::kOffB + off) = *reinterpret_cast<const uint4*>(pv);
      *reinterpret_cast<uint4*>(sm + C::kOffB + C::kBHalfBytes + off) = *reinterpret_cast<const uint4*>(qv);
    }
  } else
#pragma unroll 2
  for (int it = 0; it < 4; ++it) {
    const int task = tid + 128 * it;
    const int r = task >> 3, ic = task & 7;  // rank, chunk of 8 frequencies
    float u0[8], u1[8];
    if (r >= p.rank_k) {
#pragma unroll
      for (int e = 0; e < 8; ++e) u0[e] = u1[e] = 0.f;
    } else if (wk_vec) {
      // half layout: dims ic*8.. and 64+ic*8..; interleaved: 16 consecutive dims
      const uint4 a0 = *reinterpret_cast<const uint4*>(sm + C::kOffB + pq_off(g, r, ic));
      const uint4 a1 = *reinterpret_cast<const uint4*>(sm + C::kOffB + C::kBHalfBytes + pq_off(g, r, ic));
      const __half* h0p = reinterpret_cast<const __half*>(&a0);
      const __half* h1p = reinterpret_cast<const __half*>(&a1);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        if (interleaved) {
          const __half* src = e < 4 ? h0p : h1p;
          u0[e] = __half2float(src[(2 * e) & 7]);
          u1[e] = __half2float(src[(2 * e + 1) & 7]);
        } else {
          u0[e] = __half2float(h0p[e]);
          u1[e] = __half2float(h1p[e]);
        }
      }
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int i = ic * 8 + e;
        const int d0 = interleaved ? 2 * i : i, d1 = interleaved ? 2 * i + 1 : i + 64;
        if (p.wk_dtype == WSVD_I8) {
          const int8_t* w = reinterpret_cast<const int8_t*>(p.wk) + (int64_t)r * p.wk_stride_r + col;
          const __half* ws = reinterpret_cast<const __half*>(p.wk_scale) + col;
          u0[e] = (float)w[d0] * __half2float(ws[d0]);
          u1[e] = (float)w[d1] * __half2float(ws[d1]);
        } else {
          const __half* w = reinterpret_cast<const __half*>(p.wk) + (int64_t)r * p.wk_stride_r + col;
          u0[e] = __half2float(w[d0]);
          u1[e] = __half2float(w[d1]);
        }
      }
    }
    __align__(16) __half pv[8];
    __align__(16) __half qv[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      pv[e] = __float2half_rn(qlo[e] * u0[e] + qhi[e] * u1[e]);
      qv[e] = __float2half_rn(qhi[e] * u0[e] - qlo[e] * u1[e]);
    }
    const uint32_t off = pq_off(g, r, ic);
    *reinterpret_cast<uint4*>(sm + C::kOffB + off) = *reinterpret_cast<const uint4*>(pv);
    *reinterpret_cast<uint4*>(sm + C::kOffB + C::kBHalfBytes + off) = *reinterpret_cast<const uint4*>(qv);
  }
}

// What a head's warps know of an item lives in shared memory ([head][item parity], every warp of the head writes
// the same values): the registers are needed for the tile loop and the [P;Q] build, and state that is kept
// in registers across both comes back as reloads from local memory inside the tile loop.
enum ItemField { kItB, kItHg, kItLeft, kItBefore, kItN, kItReq, kItTilesB, kItLo, kItHi, kItTiles, kItT, kItUnits, kItMine, kItParts, kItFirst };

__device__ __forceinline__ void put_item(volatile int* st, const Walk& w, uint32_t T, uint32_t units, uint32_t mine) {
  if ((threadIdx.x & 31) == 0) {
    st[kItB] = w.b, st[kItHg] = w.hg, st[kItLeft] = w.tiles_left, st[kItBefore] = w.before_b, st[kItN] = w.n, st[kItReq] = w.req;
    st[kItTilesB] = w.tiles_b, st[kItLo] = w.lo, st[kItHi] = w.hi, st[kItTiles] = w.ntiles;
    st[kItT] = (int)T, st[kItUnits] = (int)units, st[kItMine] = (int)mine;
  }
  __syncwarp();
}
__device__ __forceinline__ Walk get_item(const volatile int* st) {
  Walk w;
  w.b = st[kItB], w.hg = st[kItHg], w.tiles_left = st[kItLeft], w.before_b = st[kItBefore], w.n = st[kItN], w.req = st[kItReq];
  w.tiles_b = st[kItTilesB], w.lo = st[kItLo], w.hi = st[kItHi], w.ntiles = st[kItTiles], w.t_first = 0;
  return w;
}

// Merges, projects and writes the output rows of a head whose last partial this CTA has delivered (or that it
// covered alone: the latent-space row is in shared memory then).  Run by the head's 128 threads.
// `seen`: for thread 0 of the head, the arrivals before this CTA's.
template <class C>
__device__ __forceinline__ void finish_head(const TcArgs& ta, uint8_t* sm, int g, const volatile int* st, unsigned int seen) {
  const KArgs& a = ta.k;
  const WsvdLatentDecodeParams& p = a.p;
  const int d = threadIdx.x & 127, Rv = p.rank_v;
  const int n_hg = (p.n_q_heads + C::kG - 1) / C::kG;
  struct { int b, hg, n_parts, c_first; } const f = {st[kItB], st[kItHg], st[kItParts], st[kItFirst]};
  const int h = f.hg * C::kG + g, hk = h / (p.n_q_heads / p.n_kv_heads);
  float* o_row = reinterpret_cast<float*>(sm + C::kOffPlanes + 2 * g * C::kPlaneBytes);
  int* verdict = reinterpret_cast<int*>(sm + C::kOffSum) + g * 8;  // the head's (max, sum) pairs were read before
  auto head_sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "r"(128) : "memory"); };
  if (f.n_parts > 1) {
    // the CTA that adds the head's last partial merges them all
    if (d == 0) {
      __threadfence();
      verdict[0] = seen + 1u == (unsigned int)f.n_parts;
    }
    head_sync();
    if (verdict[0] == 0) return;
    const int64_t slot0 = ((int64_t)f.b * n_hg + f.hg + f.c_first) * C::kG + g;
    // Eight partials at a time, their loads all in flight at once, each batch under a running maximum.  (A loop of one
    // partial after another cost a round trip to L2 each: with 16 CTAs on a head, half of the smallest call's time.)
    // (The maximum starts at the lowest finite value: a partial of -inf has weight 0 also where nothing has had any yet.)
    float m = -FLT_MAX, wsum = 0.f, osum = 0.f;
    for (int i0 = 0; i0 < f.n_parts; i0 += 8) {
      float ls[8], mo[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const bool on = i0 + i < f.n_parts;
        ls[i] = on ? __ldcg(a.lse + slot0 + (int64_t)(i0 + i) * C::kG) : -INFINITY;
        mo[i] = on && d < Rv ? __ldcg(a.mid_o + (slot0 + (int64_t)(i0 + i) * C::kG) * Rv + d) : 0.f;
      }
      float m_new = m;
#pragma unroll
      for (int i = 0; i < 8; ++i) m_new = fmaxf(m_new, ls[i]);
      const float keep = __expf(m - m_new);
      wsum *= keep;
      osum *= keep;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (i0 + i >= f.n_parts) continue;
        const float w = __expf(ls[i] - m_new);  // (a NaN stays one)
        wsum += w;
        osum = fmaf(w, mo[i], osum);
      }
      m = m_new;
    }
    if (d < Rv) o_row[d] = osum / wsum;
  }
  head_sync();
  // with peers the finished row is staged (second half of the head's plane area) and leaves as
  // 16-byte stores, one per thread per peer
  __half* stage = reinterpret_cast<__half*>(sm + C::kOffPlanes + 2 * g * C::kPlaneBytes + C::kPlaneBytes);
  __half* out = ta.has_peers ? stage
                             : reinterpret_cast<__half*>(p.out) + (int64_t)f.b * p.out_stride_b + (int64_t)h * p.out_stride_h;
  if (p.wv == nullptr) {
    if (d < Rv) out[d] = __float2half_rn(o_row[d]);
  } else {
    // out[d] = sum_r O_lat[r] U_v[r, hk*128 + d]: consecutive d in consecutive lanes, four sums and
    // 32 loads of U_v (L2) in flight
    const __half* w = reinterpret_cast<const __half*>(p.wv) + (int64_t)hk * p.head_dim + d;
    float y0 = 0.f, y1 = 0.f, y2 = 0.f, y3 = 0.f;
    int k = 0;
#pragma unroll 8
    for (; k + 4 <= Rv; k += 4) {
      y0 = fmaf(o_row[k], __half2float(__ldg(w + (int64_t)k * p.wv_stride_r)), y0);
      y1 = fmaf(o_row[k + 1], __half2float(__ldg(w + (int64_t)(k + 1) * p.wv_stride_r)), y1);
      y2 = fmaf(o_row[k + 2], __half2float(__ldg(w + (int64_t)(k + 2) * p.wv_stride_r)), y2);
      y3 = fmaf(o_row[k + 3], __half2float(__ldg(w + (int64_t)(k + 3) * p.wv_stride_r)), y3);
    }
    if constexpr (C::kAny)
      for (; k < Rv; ++k) y0 = fmaf(o_row[k], __half2float(__ldg(w + (int64_t)k * p.wv_stride_r)), y0);
    out[d] = __float2half_rn((y0 + y1) + (y2 + y3));
  }
  head_sync();  // o_row has been read (and the staged row is complete): the next item's planes may go there
  if (ta.has_peers) {
    const int chunks = (p.wv == nullptr ? Rv : p.head_dim) >> 3;
    const int64_t doff = (int64_t)f.b * ta.peers.out_stride_b + (int64_t)(h + ta.peers.head_offset) * ta.peers.out_stride_h;
    for (int idx = d; idx < chunks * ta.peers.n_peers; idx += 128) {
      const int peer = idx / chunks, c = idx - peer * chunks;
      *reinterpret_cast<uint4*>(ta.peers.out[peer] + doff + 8 * c) = reinterpret_cast<const uint4*>(stage)[c];
    }
    head_sync();
  }
}

template <class C>
__device__ __forceinline__ volatile int* item_state(uint8_t* sm, int g, uint32_t item) {
  return reinterpret_cast<volatile int*>(sm + C::kOffItem) + (g * 2 + (item & 1)) * 16;
}

// The rows of a warp's 32 tokens (lane l: slot of token l, -1: none), by asynchronous 16-byte copies.  kRowBytes / 16
// lanes share a row, so that a copy instruction touches a few lines of memory and not 32 (with one lane per row the
// load unit, not HBM, set the pace: f16 rows scattered over their slots took 354 us for 24 sequences of 32 heads against 170 us).
//  - whole 16-byte rows: piece c goes where the tensor copy would have put it;
//  - ANY: the 16-byte pieces that hold bytes of the row, each fetched only if it does (so never past the row by more than
//    the 16 bytes it ends in), go to the row's place in the area of raw rows.
template <class C>
__device__ __forceinline__ void fetch_rows_async(uint32_t dst, const uint8_t* base, int64_t stride_bytes, int slot, int bytes) {
  constexpr int kLanes = C::kRowBytes / 16;
  const int lane = threadIdx.x & 31, c = lane % kLanes, row0 = (threadIdx.x & 127) & ~31;
#pragma unroll
  for (int i = 0; i < kLanes; ++i) {
    const int r = i * (32 / kLanes) + lane / kLanes;
    const int sl = __shfl_sync(0xffffffffu, slot, r);
    const uint8_t* src = base + (int64_t)sl * stride_bytes;
    if constexpr (C::kAny) {
      const uintptr_t first = reinterpret_cast<uintptr_t>(src) & ~(uintptr_t)15;
      const int span = (int)(reinterpret_cast<uintptr_t>(src) & 15) + bytes;
      const uint32_t to = dst + (row0 + r) * C::kRawPitch;
      if (sl >= 0 && c * 16 < span) cp_async16(to + c * 16, reinterpret_cast<const void*>(first + c * 16));
      if (sl >= 0 && c == 0 && C::kRowBytes < span)
        cp_async16(to + C::kRowBytes, reinterpret_cast<const void*>(first + C::kRowBytes));
    } else {
      if (sl >= 0 && c * 16 < bytes) cp_async16(dst + C::row_off(row0 + r, c), src + c * 16);
    }
  }
}
// Shifts the row, `skip` (0..15) bytes into the words, to their start: by 8 and 4 bytes with selects, by the rest with
// funnel shifts.  Bytes past the row are whatever the pieces held: they meet zeros of W, or ranks nobody reads.
template <int kWordsOut>
__device__ __forceinline__ void shift_row(uint32_t (&w)[kWordsOut + 4], int skip) {
  const bool by8 = skip & 8, by4 = skip & 4;
#pragma unroll
  for (int i = 0; i < kWordsOut + 2; ++i) w[i] = by8 ? w[i + 2] : w[i];
#pragma unroll
  for (int i = 0; i < kWordsOut + 1; ++i) w[i] = by4 ? w[i + 1] : w[i];
#pragma unroll
  for (int i = 0; i < kWordsOut; ++i) w[i] = __funnelshift_r(w[i], w[i + 1], (skip & 3) * 8);
}

// One head's running sums over the tiles of an item, all in the log2 domain and fp32.
//  - Denominator: l_lane, this lane's tokens, under the warp's reference m_run: the warp's maximum of z (int8), or a value
//    that follows it only when it has grown by more than kSlackZ (f16: a weight may reach 2^kSlackZ, which fp32 does not mind).
//  - Values: acc, rank 16*q4 + lane (lanes 0..15), all four warps' tokens, under big_m.  int8: every tile's sums are folded
//    in.  f16: the sums of a warp's tokens stay in tensor memory, relative to 2^my_ref, until a weight would no longer fit.
//    Then the warp goes over to its other accumulator with a new reference and leaves the old one to be folded into
//    acc.  New references leave kSlackY bits of room, so that a few per item are enough.
struct HeadSums {
  float m_run, l_lane;
  float big_m, acc;
  float my_ref, scale;  // f16: scale = 2^(m_run - my_ref) * kPlaneScale
  uint32_t bufs;        // f16, bit w4: the accumulator warp w4 of the head is using
};
constexpr float kSlackZ = 8.f;
constexpr int kSlackY = 3;

// int8: fold in the value sums of the head's tile number tp: D[rank][8*w + 0..2] are the three digit-plane sums over
// the 32 tokens of warp w, whose weights were taken relative to refs[tp & 1][w].
template <class C>
__device__ __forceinline__ void fold_tile(HeadSums& hs, uint32_t d_addr, const float* refs, uint32_t tp) {
  uint32_t d[4][4];
#pragma unroll
  for (int w4 = 0; w4 < 4; ++w4) tmem_ld4(d_addr + 8 * w4 + 3 * (w4 & 1), d[w4]);
  const float4 rf = *reinterpret_cast<const float4*>(refs + (tp & 1) * 4);
  const float ref[4] = {rf.x, rf.y, rf.z, rf.w};
#pragma unroll
  for (int w4 = 0; w4 < 4; ++w4) tmem_wait_ld(d[w4]);
  float m_new = hs.big_m;
#pragma unroll
  for (int w4 = 0; w4 < 4; ++w4) m_new = fmaxf(m_new, ref[w4]);
  if (m_new > -INFINITY) {
    hs.acc *= fast_exp2(hs.big_m - m_new);  // big_m = -inf -> factor 0
#pragma unroll
    for (int w4 = 0; w4 < 4; ++w4) {
      if (ref[w4] > -INFINITY) {  // (a warp without tokens in this tile has reference -inf)
        // the two low digit sums are combined as integers (|d| <= 32 * 255 * 128 < 2^21)
        const float v = fmaf((float)(int32_t)d[w4][2], 65536.f, (float)((int32_t)d[w4][1] * 256 + (int32_t)d[w4][0]));
        hs.acc = fmaf(v, fast_exp2(ref[w4] - m_new) * (1.f / C::kPlaneScale), hs.acc);
      }
    }
    hs.big_m = m_new;
  }
}

// f16: fold in one accumulator of warp w4 of the head: D[rank][0..2] are its three sums, relative to 2^ref.
template <class C>
__device__ __forceinline__ void fold_values(HeadSums& hs, uint32_t d_addr, int w4, uint32_t buf, float ref) {
  uint32_t d[4];
  tmem_ld4(d_addr + 16 * w4 + 8 * buf + 4 * (w4 & 1), d);
  tmem_wait_ld(d);
  const float m_new = fmaxf(hs.big_m, ref);
  float v = fmaf(__uint_as_float(d[2]), 2.384185791015625e-7f, fmaf(__uint_as_float(d[1]), 4.8828125e-4f, __uint_as_float(d[0])));  // 2^-22, 2^-11
  if (isinf(__uint_as_float(d[0]))) v = __uint_as_float(d[0]);  // an infinite V times a lower term of zero is no NaN
  hs.acc = fmaf(v, fast_exp2(ref - m_new) * (1.f / C::kPlaneScale), hs.acc * fast_exp2(hs.big_m - m_new));
  hs.big_m = m_new;
}

// f16: what the head's warps have left behind with tile number tp (see HeadSums).
template <class C>
__device__ __forceinline__ void fold_left(HeadSums& hs, uint32_t d_addr, const float* refs, uint32_t tp) {
  const float4 rf = *reinterpret_cast<const float4*>(refs + (tp & 1) * 4);
  if (fmaxf(fmaxf(rf.x, rf.y), fmaxf(rf.z, rf.w)) > kNone) {
    const float ref[4] = {rf.x, rf.y, rf.z, rf.w};
    __syncwarp();
#pragma unroll 1
    for (int w4 = 0; w4 < 4; ++w4) {
      const float r = w4 == 0 ? ref[0] : w4 == 1 ? ref[1] : w4 == 2 ? ref[2] : ref[3];
      if (r > kNone) {
        fold_values<C>(hs, d_addr, w4, (hs.bufs >> w4) & 1, r);
        hs.bufs ^= 1u << w4;
      }
    }
  }
}

// int8 ANY, rarely: a token of the warp has a negative or NaN scale.  The weight of a negative scale takes its magnitude
// (returned: y with it), and the V row goes in as -v - 1, which an int8 holds for every v: what each rank then lacks is the
// sum of those weights, which is kept for the head's end as (reference, sum), together with any NaN, which the planes of
// the weights cannot hold.
// Eight sequences of up to 4096 tokens, 32 heads, rank 62: 64.1 us without any of this, 64.4 with it, 65.5 with the weights summed
// for every token instead of here.
__device__ __forceinline__ float odd_scales(float z, float sv, float y, float* kept) {
  const bool neg = sv < 0.f;
  if (neg) y = z + fast_log2(-sv);
  const float ref = warp_max_redux(neg ? y : -INFINITY);
  const float sum = warp_sum(y != y ? y : neg && y > -INFINITY ? fast_exp2(y - ref) : 0.f);
  if ((threadIdx.x & 31) == 0) {
    const float was = kept[4], m = fmaxf(was, ref);
    kept[0] = fmaf(kept[0], fast_exp2(was - m), sum * fast_exp2(ref - m));
    kept[4] = m;
  }
  return y;
}

// The tiles of an item, for one warp of a head that is there.
template <class C>
__device__ __forceinline__ bool run_tiles(const TcArgs& ta, uint8_t* sm, uint32_t item, HeadSums& hs) {
  const WsvdLatentDecodeParams& p = ta.k.p;
  const int tid = fresh_tid(), lane = tid & 31, g = tid >> 7, row = tid & 127, q4 = row >> 5;
  const uint32_t sbase = smem_u32(sm);
  auto bar = [&](int i) { return sbase + C::kOffBar + 8u * i; };
  const int gqa = p.n_q_heads / p.n_kv_heads, Rv = p.rank_v;
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(sm + C::kOffTmemSlot);
  const volatile int* st = item_state<C>(sm, g, item);
  const volatile int* mode = reinterpret_cast<const volatile int*>(sm + C::kOffMode);
  float* refs = reinterpret_cast<float*>(sm + C::kOffRef) + g * 8;  // [tile parity][warp], see Cfg
  // Digit planes: the two warps of half a tile share one 8-row block (the MMA's B operand has 8
  // rows): rows 0..2 hold the even warp's digits, rows 3..5 (f16: 4..6) the odd warp's.  Each warp's MMA
  // reads the whole block, so its other columns are the other warp's weights times this warp's V rows:
  // garbage that nobody reads.  The remaining rows are never written.
  const uint32_t my_planes = sbase + C::kOffPlanes + (2 * g + (q4 >> 1)) * C::kPlaneBytes + (q4 & 1) * (C::kF16 ? 64 : 48) +
                             (C::kF16 ? (lane >> 3) * 128 + (lane & 7) * 2 : (lane >> 4) * 128 + (lane & 15));
  const uint32_t d_addr = tmem + ((uint32_t)(q4 * 32) << 16) + C::kTmemD + 4 * C::kDCols * g;
  const int h0 = st[kItHg] * C::kG, G = min(C::kG, p.n_q_heads - h0), npairs = (G + 1) >> 1;
  bool ok = true;
  uint32_t own_buf = 0;  // this warp's accumulator
  const int hk = (h0 + g) / gqa;
  const int pr = g >> 1, sub = hk - h0 / gqa;  // sub: this head's KV head inside a unit
  const int lo = st[kItLo], hi = st[kItHi], ntiles = st[kItTiles];
  constexpr int kChunks = C::kRowBytes / 16;  // 16-byte chunks of a latent row
  int slot_c = -1, slot_n = -1;
  unsigned short sk_raw = 0, sv_raw = 0;
  const uint32_t T = st[kItT], ub = st[kItUnits], mine = st[kItMine];
  const int32_t* page = p.req_to_token + (int64_t)st[kItReq] * p.rtt_stride;
  const __half* ksc = reinterpret_cast<const __half*>(p.k_scale) + (int64_t)hk * p.ks_stride_h;
  const __half* vsc = reinterpret_cast<const __half*>(p.v_scale) + (int64_t)hk * p.vs_stride_h;
  // counts that stay the same when the last group is not full: its first head arrives for the missing
  // ones, and a pair that holds a single head arrives twice
  const uint32_t k_arrivals = g == 0 ? 1u + (C::kG - G) : 1u;
  const uint32_t w_arrivals = (G - 2 * pr) >= 2 ? 1u : 2u;
  // this lane's first token and its next one (the lines were asked for with the item's other loads)
  slot_c = lo + row < hi ? page[lo + row] : -1;
  slot_n = lo + kTile + row < hi ? page[lo + kTile + row] : -1;
  if constexpr (!C::kF16) {
    if (slot_c >= 0) {
      sk_raw = reinterpret_cast<const unsigned short*>(ksc)[(int64_t)slot_c * p.ks_stride_t];
      sv_raw = reinterpret_cast<const unsigned short*>(vsc)[(int64_t)slot_c * p.vs_stride_t];
    }
  }
  constexpr int kEsize = C::kRowBytes / 64;  // bytes of a latent
  constexpr int kWords = C::kRowBytes / 4;
  const uint8_t* k_base = reinterpret_cast<const uint8_t*>(p.latent_k) + kEsize * (int64_t)hk * p.k_stride_h;
  const uint8_t* v_base = reinterpret_cast<const uint8_t*>(p.latent_v) + kEsize * (int64_t)hk * p.v_stride_h;
  // ANY: this head's raw rows
  const uint32_t k_raw = sbase + C::kOffK + g * (kTile * C::kRawPitch), v_raw = k_raw + (C::kOffVRaw - C::kOffK);
  auto fetch_k = [&](uint32_t dst, int slot) { fetch_rows_async<C>(dst, k_base, p.k_stride_t * kEsize, slot, p.rank_k * kEsize); };
  auto fetch_v = [&](uint32_t dst, int slot) { fetch_rows_async<C>(dst, v_base, p.v_stride_t * kEsize, slot, Rv * kEsize); };
  auto read_raw = [&](uint32_t (&w)[kWords + 4], uint32_t raw, const uint8_t* base, int64_t stride, int slot) {
#pragma unroll
    for (int c = 0; c <= kChunks; ++c)
      asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                   : "=r"(w[4 * c]), "=r"(w[4 * c + 1]), "=r"(w[4 * c + 2]), "=r"(w[4 * c + 3])
                   : "r"(raw + row * C::kRawPitch + 16 * c));
    // (2^31 slots are a multiple of 16 bytes: a sign bit that marks the slot changes nothing here; no slot: any shift does)
    shift_row<kWords>(w, (int)((reinterpret_cast<uintptr_t>(base) + (int64_t)slot * stride) & 15));
  };
  bool k_ahead = false;  // the K rows of the tile that comes are on their way (gathered tiles)
  bool gathered = false; // the tile before was
  if constexpr (C::kAny) {
    fetch_k(k_raw, slot_c);
    cp_async_commit();
    fetch_v(v_raw, slot_c);
    cp_async_commit();
  }
  for (int t = 0; t < ntiles && ok; ++t) {
    const int s = lo + t * kTile + row;
    const bool valid = s < hi;
    const uint32_t Tt = T + t, u = ub + t * npairs + pr, wb = u % C::kWBufs, mt = mine + t;
    // ---- the next tile's scales and the page entry of the tile after it: requested a whole
    //      tile before they are used
    unsigned short sk_n = 0, sv_n = 0;
    if constexpr (!C::kF16) {  // (f16 latents have no scales: null pointers)
      if (slot_n >= 0) {
        sk_n = reinterpret_cast<const unsigned short*>(ksc)[(int64_t)slot_n * p.ks_stride_t];
        sv_n = reinterpret_cast<const unsigned short*>(vsc)[(int64_t)slot_n * p.vs_stride_t];
      }
    }
    int slot_t = slot_c;
    slot_c = slot_n;
    slot_n = -1;
    if (s + 2 * kTile < hi) slot_n = page[s + 2 * kTile];
    // ---- this warp's 32 K rows (lane = token) go from the ring slot to registers at once and
    //      the slot is handed back: its refill has the whole tile to arrive
    uint4 kreg[kChunks];
    bool gather = false;
    if constexpr (C::kAny) {
      // the K rows of this tile have been on their way for a tile (its V rows may still be); those of the next tile
      // take their place
      cp_async_wait_but_one();
      __syncwarp();
      uint32_t w[kWords + 4];
      read_raw(w, k_raw, k_base, p.k_stride_t * kEsize, slot_t);
#pragma unroll
      for (int c = 0; c < kChunks; ++c) kreg[c] = make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
      __syncwarp();
      if (lo + (t + 1) * kTile < hi) fetch_k(k_raw, slot_c);
      cp_async_commit();
    } else {
      const uint32_t kslot = Tt % C::kKSlots;
      ok = mbar_wait(bar(C::kBarKFull + kslot), (Tt / C::kKSlots) & 1);
      if (!ok) break;
      gather = mode[Tt & 3] & 1;
      // copied rows sit at the head's KV head, gathered ones at the head itself
      const uint32_t krows = sbase + C::kOffK + kslot * C::kUnitBytes + (gather ? g : sub) * C::kHeadBytes;
      if (gather) {
        if (!k_ahead) fetch_k(krows, slot_t);
        cp_async_wait_all();
        __syncwarp();
      }
#pragma unroll
      for (int c = 0; c < kChunks; ++c)
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(kreg[c].x), "=r"(kreg[c].y), "=r"(kreg[c].z), "=r"(kreg[c].w)
                     : "r"(krows + C::row_off(row, c)));
      __syncwarp();
      if (lane == 0) mbar_arrive_n(bar(C::kBarKEmpty + kslot), k_arrivals);
      if (gather) {
        // the copying warp's arrival says that every head's value MMAs on the V slot are complete
        ok = mbar_wait(bar(C::kBarVFull + Tt % C::kVSlots), (Tt / C::kVSlots) & 1);
        if (!ok) break;
        fetch_v(sbase + C::kOffV + (Tt % C::kVSlots) * C::kUnitBytes + g * C::kHeadBytes, slot_t);
        // K of the next tile, if that is known to be gathered too and the slot's last tile was (with one slot that
        // is this tile): then this head's rows of the slot are its own, and this warp has read them.  The copying warp may
        // be publishing the word at this moment: one read decides for all lanes, which fetch together or not at all.
        const int next_mode = __shfl_sync(0xffffffffu, lane == 0 ? mode[(Tt + 1) & 3] : 0, 0);
        k_ahead = (C::kKSlots == 1 || gathered) && lo + (t + 1) * kTile < hi && next_mode == (int)(2 * (Tt + 1)) + 1;
        if (k_ahead) fetch_k(sbase + C::kOffK + (Tt + 1) % C::kKSlots * C::kUnitBytes + g * C::kHeadBytes, slot_c);
      } else {
        k_ahead = false;
      }
      gathered = gather;
    }
    if constexpr (C::kF16) {
      if (C::kAny || gather) {  // what lies behind the row may be a NaN, which a zero of W does not silence (the rank is even)
#pragma unroll
        for (int c = 0; c < kChunks; ++c) {
          uint32_t* x = reinterpret_cast<uint32_t*>(&kreg[c]);
#pragma unroll
          for (int j = 0; j < 4; ++j) x[j] = 2 * (4 * c + j) < p.rank_k ? x[j] : 0u;
        }
      }
    }
    ok = mbar_wait(bar(C::kBarWFull + wb), (u / C::kWBufs) & 1);
    if (!ok) break;
    tc_fence_after();

    // int8 ANY: a negative or NaN scale among the warp's?  (Asked behind the wait for W, by which time the scales are here;
    // the answer has the dot to arrive.)
    bool odd = false;
    if constexpr (C::kAny && !C::kF16) odd = __any_sync(0xffffffffu, sv_raw > 0x7c00);
    // ---- score: dot of this token's K row with its row of W, 16 ranks at a time
    const uint32_t taddr = tmem + ((uint32_t)(q4 * 32) << 16) + wb * 128 + (g & 1) * kRkMax;
    float2 dot0 = make_float2(0.f, 0.f), dot1 = make_float2(0.f, 0.f);
    // two 16-column loads in flight alternately: the next chunk of W travels while this one is used
    uint32_t wa[16], wb16[16];
    auto mac16 = [&](const uint32_t (&wv)[16], int c) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float2 x01, x23;
        if constexpr (C::kF16) {
          const uint4 kq = kreg[(2 * c + (j >> 1)) % kChunks];
          const uint32_t h01 = j & 1 ? kq.z : kq.x, h23 = j & 1 ? kq.w : kq.y;
          x01 = __half22float2(*reinterpret_cast<const __half2*>(&h01));
          x23 = __half22float2(*reinterpret_cast<const __half2*>(&h23));
        } else {
          const uint4 kq = kreg[c % kChunks];
          cvt4((j == 0 ? kq.x : j == 1 ? kq.y : j == 2 ? kq.z : kq.w) ^ 0x80808080u, x01, x23);
        }
        dot0 = __ffma2_rn(x01, make_float2(__uint_as_float(wv[4 * j]), __uint_as_float(wv[4 * j + 1])), dot0);
        dot1 = __ffma2_rn(x23, make_float2(__uint_as_float(wv[4 * j + 2]), __uint_as_float(wv[4 * j + 3])), dot1);
      }
    };
    tmem_ld16(taddr, wa);
    tmem_wait_ld();
    tmem_ld16(taddr + 16, wb16);
    mac16(wa, 0);
    tmem_wait_ld();
    tmem_ld16(taddr + 32, wa);
    mac16(wb16, 1);
    tmem_wait_ld();
    tmem_ld16(taddr + 48, wb16);
    mac16(wa, 2);
    tmem_wait_ld();
    mac16(wb16, 3);
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive_n(bar(C::kBarWEmpty + wb), w_arrivals);  // this warp has read its rows of W
    const float2 dsum = __fadd2_rn(dot0, dot1);
    const float sk = __half2float(__ushort_as_half(sk_raw)), sv = __half2float(__ushort_as_half(sv_raw));
    const float z = valid ? (C::kF16 ? dsum.x + dsum.y : (dsum.x + dsum.y) * sk) : -INFINITY;
    sk_raw = sk_n;
    sv_raw = sv_n;

    // ---- softmax weights under the warp's reference, denominator (fp32, by the owner threads)
    // (int8 ANY: a NaN among the scores shows in the maximum, so that it reaches l_lane whatever the others are)
    const float mz_w = C::kAny && !C::kF16 ? warp_max_redux_nan(z) : warp_max_redux(z);
    float wgt, left;        // what the value MMA's operand is made of; what goes to refs
    uint32_t how = 0;       // f16: accumulator and whether to add to it
    if constexpr (C::kF16) {
      bool renew = mz_w > hs.m_run + kSlackZ;
      if (renew) {
        hs.l_lane *= fast_exp2(hs.m_run - mz_w);
        hs.m_run = mz_w;
      }
      const float e = fast_exp2(z - hs.m_run);  // masked tokens: 2^-inf = 0
      hs.l_lane += e;
      const float e_w = warp_max_redux(e);
      // does every weight fit under the reference of the value sums?
      left = kNone;
      how = t > 0 ? 2u : 0u;
      renew = renew || e_w * hs.scale > C::kPlaneScale || (t & (C::kRenewTiles - 1)) == C::kRenewTiles - 1;
      if (renew) {
        left = hs.my_ref;
        if (left > kNone) {
          how = 0u;
          own_buf ^= 1u;
        }
        // 2^k, the power of two that leaves the largest weight kSlackY bits of room (weights 2^-60 below the largest
        // of the softmax do not show in the result)
        const int k = max((int)((__float_as_uint(e_w) >> 23) & 0xff) - 126 + kSlackY, -60);
        hs.my_ref = hs.m_run + (float)k;
        hs.scale = C::kPlaneScale * __uint_as_float((uint32_t)(127 - k) << 23);
      }
      how |= own_buf;
      wgt = e * hs.scale;
    } else {
      // log2(0) = -inf: a zero scale drops the token's value.  (Whole rows: a negative or NaN scale does too.)
      float y = valid ? z + fast_log2(sv) : -INFINITY;
      if constexpr (C::kAny) {
        if (odd) {
          y = odd_scales(z, sv, y, reinterpret_cast<float*>(sm + C::kOffNeg) + g * 8 + q4);
          if (sv < 0.f) slot_t |= (int)0x80000000;  // (the sign is looked at when the V row is put into place)
        }
      }
      left = warp_max_redux(y);
      if (C::kAny ? !(mz_w == -INFINITY) : mz_w > -INFINITY) {
        const float m_new = fmaxf(hs.m_run, mz_w);
        hs.l_lane = fmaf(hs.l_lane, fast_exp2(hs.m_run - m_new), fast_exp2(z - m_new));  // 2^-inf = 0: m_run = -inf, masked tokens
        hs.m_run = m_new;
      }
      wgt = (y > -INFINITY ? fast_exp2(y - left) : 0.f) * C::kPlaneScale;  // <= kPlaneScale
    }

    // ---- the previous tile's value MMAs are complete: fold in its sums, or what the head's warps left behind.  This
    //      also orders this warp's reads of D and of the references (and, through the MMAs' completion,
    //      the MMAs' reads of its digit planes and V rows) before those of this tile are written.
    if (t > 0) {
      ok = mbar_wait(bar(C::kBarDFull + g), (mt - 1) & 1);
      if (!ok) break;
      tc_fence_after();
      if constexpr (C::kF16) fold_left<C>(hs, d_addr, refs, mt - 1);
      else fold_tile<C>(hs, d_addr, refs, mt - 1);
    }
    const uint32_t vrow = sbase + C::kOffV + (Tt % C::kVSlots) * C::kUnitBytes + (C::kAny || gather ? g : sub) * C::kHeadBytes;
    if constexpr (C::kAny) {
      // this head's own region: its value MMAs of the tile before are complete
      cp_async_wait_but_one();  // all but the next tile's K rows
      __syncwarp();
      uint32_t w[kWords + 4];
      read_raw(w, v_raw, v_base, p.v_stride_t * kEsize, slot_t);
      if constexpr (C::kF16) {  // no token: zeros (0 x NaN)
#pragma unroll
        for (int i = 0; i < kWords; ++i) w[i] = valid ? w[i] : 0u;
      } else if (__any_sync(0xffffffffu, slot_t < -1)) {  // (see odd_scales; what an int8 row without a token holds meets a weight of 0)
        const uint32_t flip = (uint32_t)(slot_t >> 31);
#pragma unroll
        for (int i = 0; i < kWords; ++i) w[i] ^= flip;
      }
#pragma unroll
      for (int c = 0; c < kChunks; ++c)
        asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(vrow + C::row_off(row, c)), "r"(w[4 * c]), "r"(w[4 * c + 1]),
                     "r"(w[4 * c + 2]), "r"(w[4 * c + 3])
                     : "memory");
      __syncwarp();
      if (lo + (t + 1) * kTile < hi) fetch_v(v_raw, slot_c);
      cp_async_commit();
    } else {
      if (gather) {
        cp_async_wait_all();
        __syncwarp();
      }
      if (C::kF16 && lo + (t + 1) * kTile > hi) {
        // the end of the sequence: what was copied behind it may be anything, and in f16 a NaN times a weight of
        // zero is a NaN
        ok = mbar_wait(bar(C::kBarVFull + Tt % C::kVSlots), (Tt / C::kVSlots) & 1);
        if (!ok) break;
        if (!valid) {
#pragma unroll
          for (int c = 0; c < kChunks; ++c)
            asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};" ::"r"(vrow + C::row_off(row, c)), "r"(0) : "memory");
        }
      }
    }

    // ---- this token's weight for the value MMA: three 8-bit digits, or three f16 terms (11 bits each, every remainder
    //      is exact: nothing that fp32 holds of the weight is lost)
    if constexpr (C::kF16) {
      const __half t0 = __float2half_rn(wgt);
      const float r1 = (wgt - __half2float(t0)) * 2048.f;
      const __half t1 = __float2half_rn(r1);
      const __half t2 = __float2half_rn((r1 - __half2float(t1)) * 2048.f);
      asm volatile("st.shared.u16 [%0], %1;" ::"r"(my_planes), "h"(__half_as_ushort(t0)) : "memory");
      asm volatile("st.shared.u16 [%0], %1;" ::"r"(my_planes + 16), "h"(__half_as_ushort(t1)) : "memory");
      asm volatile("st.shared.u16 [%0], %1;" ::"r"(my_planes + 32), "h"(__half_as_ushort(t2)) : "memory");
    } else {
      const uint32_t nq = __float2uint_rn(wgt);
      asm volatile("st.shared.u8 [%0], %1;" ::"r"(my_planes), "r"(nq) : "memory");
      asm volatile("st.shared.u8 [%0], %1;" ::"r"(my_planes + 16), "r"(nq >> 8) : "memory");
      asm volatile("st.shared.u8 [%0], %1;" ::"r"(my_planes + 32), "r"(nq >> 16) : "memory");
    }
    fence_proxy_async();
    tc_fence_before();
    if (lane == 0) {
      refs[(mt & 1) * 4 + q4] = left;
      if constexpr (C::kF16) reinterpret_cast<volatile uint8_t*>(value_modes<C>(sm, g))[q4] = (uint8_t)how;
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(C::kBarPlanes + g));
  }
  return ok;
}

template <class C>
__device__ __forceinline__ void epilogue_role(const TcArgs& ta, const Share& sh, uint8_t* sm, uint32_t sbase, uint32_t tmem) {
  const KArgs& a = ta.k;
  const WsvdLatentDecodeParams& p = a.p;
  const int n_hg = (p.n_q_heads + C::kG - 1) / C::kG, gqa = p.n_q_heads / p.n_kv_heads;
  const int Rv = p.rank_v;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = warp >> 2, q4 = warp & 3, row = q4 * 32 + lane;
  auto bar = [&](int i) { return sbase + C::kOffBar + 8u * i; };
  auto head_sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "r"(128) : "memory"); };
  const bool balanced = ta.balanced != 0, fused = balanced && ta.arrivals != nullptr;
  // vector loads of eight values of wk need rows aligned to them: 16 bytes for f16, 8 bytes for int8
  // (whose scales are then read as 16-byte vectors too)
  const bool wk_i8 = p.wk_dtype == WSVD_I8;
  const bool wk_vec = (p.wk_stride_r & 7) == 0 &&
                      (wk_i8 ? (reinterpret_cast<uintptr_t>(p.wk) & 7) == 0 && (reinterpret_cast<uintptr_t>(p.wk_scale) & 15) == 0
                             : (reinterpret_cast<uintptr_t>(p.wk) & 15) == 0);
  auto state = [&](uint32_t i) { return item_state<C>(sm, g, i); };
  bool ok = true;  // after a wait that timed out: tiles are skipped, results are NaN
  bool pending = false;  // the item before is still to be finished
  bool idle = false;     // this warp's head was not there in the item before
  unsigned int seen = 0;
  {
    Walk w;
    if (!w.start(ta, sh, n_hg)) return;
    if (g < p.n_q_heads - w.hg * C::kG) request_pq<C>(ta, sbase, w, g, wk_vec);
    put_item(state(0), w, 0, 0, 0);
  }
  for (uint32_t item = 0;; ++item) {
    volatile int* st = state(item);
    const int h0 = st[kItHg] * C::kG, G = min(C::kG, p.n_q_heads - h0), npairs = (G + 1) >> 1;
    const bool active = g < G;
    if (active) {
      const int hk = (h0 + g) / gqa;
      // The rows of this head in the B operand are free: this warp has seen W of the head's last tile, and
      // with it the completion of every score MMA that read them.
      build_pq<C>(ta, sm, st[kItB], h0 + g, hk, g, wk_vec);
      fence_proxy_async();
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(C::kBarPq));
    // A warp whose head is not there must not arrive for the next item before this one's phase is over.  Where its head
    // is there again, it must not start on the tiles before every other warp is through with the item that it sat out:
    // the parities of K full and W full, which it would wait for, say nothing while those barriers are phases behind.
    if ((!active || idle) && ok) ok = warp_wait(bar(C::kBarPq), item & 1);
    idle = !active;
    if (pending) finish_head<C>(ta, sm, g, state(item + 1), seen);  // the item before, while the first score MMAs of this one run
    pending = false;

    const float none = C::kF16 ? kNone : -INFINITY;
    HeadSums hs = {none, 0.f, none, 0.f, kNone, 0.f, 0u};
    if constexpr (C::kAny && !C::kF16) {
      float* kept = reinterpret_cast<float*>(sm + C::kOffNeg) + g * 8 + q4;
      if (lane == 0) kept[0] = 0.f, kept[4] = kNone;
    }
    if (active && ok) ok = run_tiles<C>(ta, sm, item, hs);

    // ---- the item's end.  What the next item needs is requested before the last value sums are waited for.
    bool more;
    int n_parts = 1;
    {
      Walk w = get_item(st);
      const uint32_t mine = st[kItMine] + (active ? w.ntiles : 0);
      const uint32_t T = st[kItT] + w.ntiles, units = st[kItUnits] + w.ntiles * npairs;
      if (fused && active) {  // the CTAs that share this (sequence, head group)
        const int64_t first = (int64_t)w.before_b * n_hg + (int64_t)w.hg * w.tiles_b;
        const int c_first = share_owner(first, sh.total, sh.shares);
        n_parts = share_owner(first + w.tiles_b - 1, sh.total, sh.shares) - c_first + 1;
        if (lane == 0) st[kItParts] = n_parts, st[kItFirst] = c_first;
      }
      more = w.next(p, n_hg);
      if (more) {
        if (g < p.n_q_heads - w.hg * C::kG) request_pq<C>(ta, sbase, w, g, wk_vec);
        put_item(state(item + 1), w, T, units, mine);
      }
    }
    if (active) {
      const uint32_t last = st[kItMine] + st[kItTiles] - 1;  // count of the head's last tile
      const int b = st[kItB], hg = st[kItHg], h = h0 + g;
      const uint32_t d_addr = tmem + ((uint32_t)(q4 * 32) << 16) + C::kTmemD + 4 * C::kDCols * g;
      float* refs = reinterpret_cast<float*>(sm + C::kOffRef) + g * 8;
      if (ok) {
        ok = warp_wait(bar(C::kBarDFull + g), last & 1);
        if (ok) {
          tc_fence_after();
          if constexpr (C::kF16) {
            fold_left<C>(hs, d_addr, refs, last);
          } else {
            fold_tile<C>(hs, d_addr, refs, last);
            tc_fence_before();
          }
        }
      }
      if (!ok) atomicMax(&g_status, (unsigned)kTimeoutEpilogue);

      // ---- the head's denominator: the four warps' (reference, sum) pairs under a common maximum; with them, f16, the
      //      references of the value accumulators in use
      const float l_w = warp_sum(hs.l_lane);
      float2* sums = reinterpret_cast<float2*>(sm + C::kOffSum) + g * 4;
      if (lane == 0) {
        sums[q4] = make_float2(hs.m_run, l_w);
        if constexpr (C::kF16) refs[((last + 1) & 1) * 4 + q4] = hs.my_ref;
      }
      head_sync();
      if (C::kF16 && ok) {
        const float4 rf = *reinterpret_cast<const float4*>(refs + ((last + 1) & 1) * 4);
        if (rf.x > kNone) fold_values<C>(hs, d_addr, 0, hs.bufs & 1, rf.x);
        if (rf.y > kNone) fold_values<C>(hs, d_addr, 1, (hs.bufs >> 1) & 1, rf.y);
        if (rf.z > kNone) fold_values<C>(hs, d_addr, 2, (hs.bufs >> 2) & 1, rf.z);
        if (rf.w > kNone) fold_values<C>(hs, d_addr, 3, (hs.bufs >> 3) & 1, rf.w);
        tc_fence_before();
      }
      float m_all = none;
#pragma unroll
      for (int w4 = 0; w4 < 4; ++w4) m_all = fmaxf(m_all, sums[w4].x);
      float l_tot = 0.f;  // (f16, ANY: a NaN in any warp's sum stays)
#pragma unroll
      for (int w4 = 0; w4 < 4; ++w4)
        if (C::kF16 || sums[w4].x > -INFINITY) l_tot = fmaf(sums[w4].y, fast_exp2(sums[w4].x - m_all), l_tot);
        else if (C::kAny) l_tot += sums[w4].y;  // 0, or a NaN
      const int64_t slot = balanced ? ((int64_t)b * n_hg + hg + blockIdx.x) * C::kG + g
                                    : ((int64_t)b * p.n_q_heads + h) * a.n_splits + blockIdx.x % a.n_splits;
      const int r = 16 * q4 + lane;
      // sum_s 2^z sv Lv / sum_s 2^z  =  acc * 2^(big_m - m_all) / l
      // (after a wait that timed out the item's result is poisoned: NaN here propagates through the
      // merge into the output row, so a time-out cannot pass for a valid result)
      const float sum = hs.big_m > none ? hs.acc * fast_exp2(hs.big_m - m_all) : 0.f;
      float o = C::kF16 || hs.big_m > none ? sum / l_tot : 0.f;
      if constexpr (C::kAny && !C::kF16) {
        const float4 kept = reinterpret_cast<const float4*>(sm + C::kOffNeg)[g * 2];
        if ((kept.x + kept.y) + (kept.z + kept.w) != 0.f) {  // (no sum is negative)
          const float4 ref = reinterpret_cast<const float4*>(sm + C::kOffNeg)[g * 2 + 1];
          const float k[4] = {kept.x, kept.y, kept.z, kept.w}, kr[4] = {ref.x, ref.y, ref.z, ref.w};
          float neg_tot = 0.f;
#pragma unroll
          for (int w4 = 0; w4 < 4; ++w4) neg_tot = fmaf(k[w4], m_all > -INFINITY ? fast_exp2(kr[w4] - m_all) : 1.f, neg_tot);
          o = neg_tot != neg_tot ? neg_tot : o + neg_tot / l_tot;
        }
        if (l_tot != l_tot) o = l_tot;
      }
      if (!ok) o = __int_as_float(0x7fc00000);
      if (!fused || n_parts > 1) {
        if (lane < 16 && r < Rv) a.mid_o[slot * Rv + r] = o;
        // natural-log lse, as the merge kernel expects (stage1.py:216)
        if (q4 == 0 && lane == 0) a.lse[slot] = m_all * 0.6931471805599453f + logf(l_tot);
      } else if (lane < 16 && r < Rv) {
        // this CTA covered the whole (sequence, head): no partials.  The latent-space row goes to shared
        // memory (the head's plane area: its value MMAs are complete).
        reinterpret_cast<float*>(sm + C::kOffPlanes + 2 * g * C::kPlaneBytes)[r] = o;
      }
      head_sync();  // the partial is out, the (max, sum) pairs and the references have been read
      if (fused) {
        // the counter's answer is needed only after the next item's [P;Q] build
        // (the fence is this thread's alone: it covers what the barrier above has shown it of the others' stores)
        if (n_parts > 1 && row == 0) {
          __threadfence();
          seen = atomicAdd(ta.arrivals + (int64_t)b * p.n_q_heads + h, 1u);
        }
        pending = true;
      }
    }
    if (!more) {
      if (pending) finish_head<C>(ta, sm, g, st, seen);
      break;
    }
  }
}

// ------------------------------------------------------------------ the kernel
template <class C>
__global__ void __launch_bounds__(C::kThreads, 1) stage1_tc_kernel(const __grid_constant__ TcArgs ta) {
  const KArgs& a = ta.k;
  const WsvdLatentDecodeParams& p = a.p;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t sbase = smem_u32(smem_raw);
  uint8_t* sm = smem_raw;
  if ((sbase & 1023u) != 0) {  // the swizzled operand tiles need a 1024-byte aligned base
    if (threadIdx.x == 0) atomicMax(&g_status, (unsigned)kBadSmemAlignment);
    return;
  }
  const int n_hg = (p.n_q_heads + C::kG - 1) / C::kG;
  const bool balanced = ta.balanced != 0, fused = balanced && ta.arrivals != nullptr;
  auto tiles_of = [&](int i) {
    const int n = i < p.batch ? p.b_seq_len[i] : 0;
    return n > 0 ? (n + kTile - 1) / kTile : 0;
  };
  // Balanced mode.  Up to 128 sequences: every warp works the shares out for itself, lane l from the lengths of sequences
  // 4l..4l+3 (requested here, before the set-up below).  More: block-wide sums.
  const bool by_warp = balanced && p.batch <= 128;
  int len4[4] = {0, 0, 0, 0};
  int mine = 0;
  if (by_warp) {
#pragma unroll
    for (int j = 0; j < 4; ++j) len4[j] = 4 * lane + j < p.batch ? p.b_seq_len[4 * lane + j] : 0;
    if (4 * lane < p.batch) asm volatile("prefetch.global.L1 [%0];" ::"l"(p.b_req_idx + 4 * lane));
  } else if (balanced) {
    for (int i = threadIdx.x; i < p.batch; i += C::kThreads) mine += tiles_of(i);
  }

  // ---- once per CTA: tensor memory, barriers, descriptor prefetch
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(sm + C::kOffTmemSlot);
  if (warp == C::kMmaWarp) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), kTmemCols);
    tmem_relinquish();
    tc_fence_before();
  } else if (warp == C::kLoadWarp) {
    if (lane < 4) reinterpret_cast<volatile int*>(sm + C::kOffMode)[lane] = -1;  // no tile (the epilogue looks ahead)
    for (int i = lane; i < C::kNumBars; i += 32) {
      uint32_t count = 1;                                                       // one copy, or one commit
      if (i >= C::kBarVEmpty && i < C::kBarKEmpty) count = C::kG;               // a commit per head, after its value MMAs on the slot
      else if (i >= C::kBarKEmpty && i < C::kBarAFull) count = 4 * C::kG;       // every warp that copies rows out of the slot
      else if (i >= C::kBarWEmpty && i < C::kBarDFull) count = 8;               // the warps of a pair of heads
      else if (i >= C::kBarPlanes && i < C::kBarPq) count = 4;                  // the head's four warps
      else if (i == C::kBarPq) count = 4 * C::kG;
      mbar_init(sbase + C::kOffBar + 8u * i, count);
    }
    fence_barrier_init();
  } else if (warp == C::kValWarp && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&ta.tmap_table)) : "memory");
    if (ta.use_tma) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&ta.tmap_k)) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&ta.tmap_v)) : "memory");
    }
  }

  Share sh = {};
  if (by_warp) {
    int tiles[4], sum = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      tiles[j] = len4[j] > 0 ? (len4[j] + kTile - 1) / kTile : 0;
      sum += tiles[j];
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    const int all_tiles = __shfl_sync(0xffffffffu, incl, 31);
    sh.total = (int64_t)all_tiles * n_hg;
    sh.shares = (int)min((int64_t)gridDim.x, sh.total);
    if ((int)blockIdx.x < sh.shares) {
      const int64_t begin = share_begin(blockIdx.x, sh.total, sh.shares);
      sh.tiles_left = (int)(share_begin(blockIdx.x + 1, sh.total, sh.shares) - begin);
      // the sequence that holds tile begin / n_hg of the batch (a sequence takes n_hg entries per tile)
      const int at = (begin >> 32) == 0 ? (int)((uint32_t)begin / (uint32_t)n_hg) : (int)(begin / n_hg);
      int excl = incl - sum, found = -1, before = 0, tiles_b = 1;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (at >= excl && at < excl + tiles[j]) found = 4 * lane + j, before = excl, tiles_b = tiles[j];
        excl += tiles[j];
      }
      const int src = __ffs(__ballot_sync(0xffffffffu, found >= 0)) - 1;
      sh.b = __shfl_sync(0xffffffffu, found, src);
      sh.before_b = __shfl_sync(0xffffffffu, before, src);
      tiles_b = __shfl_sync(0xffffffffu, tiles_b, src);
      const int rem = (int)(begin - (int64_t)sh.before_b * n_hg);
      sh.hg = rem / tiles_b;
      sh.t_first = rem % tiles_b;
    }
    if (blockIdx.x == 0 && warp == 0 && ta.prefix_out != nullptr) {
      int excl = incl - sum;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (4 * lane + j < p.batch) ta.prefix_out[4 * lane + j] = excl;
        excl += tiles[j];
      }
      if (lane == 0) ta.prefix_out[p.batch] = all_tiles, ta.prefix_out[p.batch + 1] = sh.shares;
    }
  } else if (balanced) {
    // Tiles per sequence -> block-wide sums -> this CTA's share [begin, end) of the tile list and the
    // (sequence, head group, tile) it starts at.  Scratch: the reference/sum area, unused until the
    // first tile.
    int* plan_sm = reinterpret_cast<int*>(sm + C::kOffRef);  // [0, 20): per-warp sums; [24], [25]: start sequence, tiles before it
    constexpr int kWarps = C::kThreads / 32;
    static_assert(C::kOffMode - C::kOffRef >= 26 * 4 && kWarps <= 24, "plan scratch");
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
    if (lane == 0) plan_sm[warp] = mine;
    __syncthreads();
    int all_tiles = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) all_tiles += plan_sm[w];
    __syncthreads();
    sh.total = (int64_t)all_tiles * n_hg;
    sh.shares = (int)min((int64_t)gridDim.x, sh.total);
    const bool has_share = (int)blockIdx.x < sh.shares;
    const int64_t begin = has_share ? share_begin(blockIdx.x, sh.total, sh.shares) : 0;
    if (has_share) sh.tiles_left = (int)(share_begin(blockIdx.x + 1, sh.total, sh.shares) - begin);
    if (has_share || (blockIdx.x == 0 && ta.prefix_out != nullptr)) {
      int carry = 0;
      for (int base = 0; base < p.batch; base += C::kThreads) {
        const int i = base + threadIdx.x;
        const int v = tiles_of(i);
        int incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int up = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += up;
        }
        if (lane == 31) plan_sm[warp] = incl;
        __syncthreads();
        int lower = 0, chunk = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
          const int x = plan_sm[w];
          if (w < warp) lower += x;
          chunk += x;
        }
        const int excl = carry + lower + incl - v;
        if (has_share && v > 0 && (int64_t)excl * n_hg <= begin && begin < (int64_t)(excl + v) * n_hg) {
          plan_sm[24] = i;
          plan_sm[25] = excl;
        }
        if (blockIdx.x == 0 && ta.prefix_out != nullptr && i < p.batch) ta.prefix_out[i] = excl;
        carry += chunk;
        __syncthreads();
      }
      if (blockIdx.x == 0 && ta.prefix_out != nullptr && threadIdx.x == 0) {
        ta.prefix_out[p.batch] = all_tiles;
        ta.prefix_out[p.batch + 1] = sh.shares;
      }
      if (has_share) {
        sh.b = plan_sm[24];
        sh.before_b = plan_sm[25];
        const int tiles_b = tiles_of(sh.b), rem = (int)(begin - (int64_t)sh.before_b * n_hg);
        sh.hg = rem / tiles_b;
        sh.t_first = rem % tiles_b;
      }
    }
  }
  // sequences without tokens belong to no share: their output rows are zeros
  if (fused) {
    const int n_out = p.wv != nullptr ? p.head_dim : p.rank_v;
    for (int bb = blockIdx.x; bb < p.batch; bb += gridDim.x) {
      if (p.b_seq_len[bb] > 0) continue;
      if (ta.has_peers) {
        for (int i = threadIdx.x; i < p.n_q_heads * n_out * ta.peers.n_peers; i += C::kThreads) {
          const int peer = i / (p.n_q_heads * n_out), j = i % (p.n_q_heads * n_out);
          ta.peers.out[peer][(int64_t)bb * ta.peers.out_stride_b +
                             (int64_t)(j / n_out + ta.peers.head_offset) * ta.peers.out_stride_h + j % n_out] =
              __float2half_rn(0.f);
        }
      } else {
        __half* orow = reinterpret_cast<__half*>(p.out) + (int64_t)bb * p.out_stride_b;
        for (int i = threadIdx.x; i < p.n_q_heads * n_out; i += C::kThreads)
          orow[(int64_t)(i / n_out) * p.out_stride_h + i % n_out] = __float2half_rn(0.f);
      }
    }
  }
  __syncthreads();  // barriers, tensor memory; the scratch area is handed back
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  // ---- register budgets.  With int8 latents the launch gives every thread 96 registers (640 threads); the tile loop of
  //      the epilogue needs more and the control warps far fewer, so the control warpgroup hands
  //      registers back to the pool and the four epilogue warpgroups take them.
  if (warp < C::kEpiWarps) {
    if constexpr (!C::kF16) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::kEpiRegs));
    epilogue_role<C>(ta, sh, sm, sbase, tmem);
  } else {
    if constexpr (!C::kF16) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::kCtlRegs));
    if (warp == C::kMmaWarp) score_role<C>(ta, sh, sbase, tmem);
    else if (warp == C::kLoadWarp) copy_role<C>(ta, sh, sbase, sm);
    else value_role<C>(ta, sh, sbase, sm, tmem, warp - C::kValWarp);
  }

  // ---- common exit
  tc_fence_before();
  if (ta.has_peers) __threadfence_system();  // this thread's peer stores are ordered before the count below
  __syncthreads();
  if (warp == C::kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(*tmem_slot, kTmemCols);
  }
  if (ta.has_peers) {
    // the group's barrier, run by whichever CTA finishes last
    volatile int* last = reinterpret_cast<volatile int*>(sm + C::kOffSum);
    if (threadIdx.x == 0) {
      const unsigned int done = atomicAdd(ta.peers.counter, 1u) + 1u;
      *last = done == gridDim.x;
      if (done == gridDim.x) *ta.peers.counter = 0u;  // ready for the next launch
    }
    __syncthreads();
    if (*last) peer_group_barrier(ta.peers, &g_status);
  }
}

}  // namespace tc

namespace tc {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      ptr = nullptr;
    return reinterpret_cast<EncodeTiledFn>(ptr);
  }();
  return fn;
}

// One latent tensor [T, Hkv, R] with element strides (st, sh) as a 3-D tensor map [Hkv][T][R], whatever the
// order of the strides; box = 64 ranks x `slots` token slots x `heads` KV heads, so that a head's rows sit
// together in shared memory.  The box is wider than the tensor when the rank is below 64, and may reach past
// the last head: the missing elements arrive as zeros.
bool encode_latent(CUtensorMap* map, const void* base, bool f16, int64_t st, int64_t sh, int64_t T, int Hkv, int R,
                   int heads, int slots) {
  EncodeTiledFn fn = encode_fn();
  if (!fn || T <= 0 || T > 0xffffffffll || st < 0 || sh < 0) return false;
  const int64_t size = f16 ? 2 : 1;
  cuuint64_t dims[3] = {(cuuint64_t)R, (cuuint64_t)T, (cuuint64_t)Hkv};
  cuuint64_t strides[2] = {(cuuint64_t)(st * size), (cuuint64_t)(sh * size)};
  cuuint32_t box[3] = {64, (cuuint32_t)slots, (cuuint32_t)heads};
  cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = fn(map, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 3,
                        const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        f16 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// The position table [2][rows][64] f16; box = one 128-position tile of both planes (cos tile, then
// sin tile), 128-byte swizzle (the K-major operand layout of the score MMA).  Rows past the table
// read as zeros.
bool encode_table(CUtensorMap* map, const void* table, int rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn || rows <= 0) return false;
  cuuint64_t dims[3] = {64, (cuuint64_t)rows, 2};
  cuuint64_t strides[2] = {128, (cuuint64_t)rows * 128};
  cuuint32_t box[3] = {64, (cuuint32_t)kTile, 2};
  cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(table), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

}  // namespace tc

namespace tc {
// The kernel's shared-memory size is an attribute of the function on a device: set once per device and process.  (Two
// threads that come first may both set it; a device past the array sets it on every call.)
template <class C>
cudaError_t allow_smem() {
  static std::atomic<bool> done[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 64 && done[dev].load(std::memory_order_acquire)) return cudaSuccess;
  e = cudaFuncSetAttribute(stage1_tc_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::kSmemBytes);
  if (e == cudaSuccess && dev < 64) done[dev].store(true, std::memory_order_release);
  return e;
}
}  // namespace tc

size_t rope_table_bytes(int rows) { return (size_t)rows * 256; }

cudaError_t launch_rope_table(void* table, int rows, const KArgs& a, cudaStream_t stream) {
  const int total = rows * 64;
  tc::rope_table_kernel<<<(total + 255) / 256, 256, 0, stream>>>(reinterpret_cast<__half*>(table), rows, a);
  return cudaGetLastError();
}

template <class C>
static cudaError_t launch_tc(const KArgs& a, const void* table, int table_rows, const Stage1Work& work, cudaStream_t stream) {
  cudaError_t e = tc::allow_smem<C>();
  if (e != cudaSuccess) return e;
  tc::TcArgs ta;
  ta.k = a;
  ta.table_rows = table_rows;
  ta.use_tma = 0;
  ta.box_heads = 1;
  memset(&ta.tmap_k, 0, sizeof(CUtensorMap));
  memset(&ta.tmap_v, 0, sizeof(CUtensorMap));
  memset(&ta.tmap_runs, 0, sizeof(ta.tmap_runs));
  if (!tc::encode_table(&ta.tmap_table, table, table_rows)) return cudaErrorInvalidValue;
  if (a.p.n_token_slots > 0 && !C::kAny) {
    // KV heads one group of query heads can touch (its first head is a multiple of the group's size)
    const int gqa = a.p.n_q_heads / a.p.n_kv_heads;
    const int heads = gqa == 1 ? C::kG : gqa == 2 ? C::kG / 2 : gqa % C::kG == 0 ? 1 : 2;
    auto encode = [&](CUtensorMap* m, bool is_k, int heads_in_box, int slots) {
      return tc::encode_latent(m, is_k ? a.p.latent_k : a.p.latent_v, C::kF16, is_k ? a.p.k_stride_t : a.p.v_stride_t,
                               is_k ? a.p.k_stride_h : a.p.v_stride_h, a.p.n_token_slots, a.p.n_kv_heads,
                               is_k ? a.p.rank_k : a.p.rank_v, heads_in_box, slots);
    };
    if (encode(&ta.tmap_k, true, heads, tc::kTile) && encode(&ta.tmap_v, false, heads, tc::kTile) &&
        encode(&ta.tmap_runs[0], true, 1, 64) && encode(&ta.tmap_runs[1], false, 1, 64) &&
        encode(&ta.tmap_runs[2], true, 1, 16) && encode(&ta.tmap_runs[3], false, 1, 16)) {
      ta.use_tma = 1;
      ta.box_heads = heads;
    }
  }
  ta.balanced = work.n_ctas > 0;
  ta.prefix_out = work.prefix;
  ta.arrivals = work.arrivals;
  ta.has_peers = work.arrivals != nullptr && work.peers != nullptr;
  if (ta.has_peers) ta.peers = *work.peers;
  else memset(&ta.peers, 0, sizeof(ta.peers));
  const int grid = work.n_ctas > 0 ? work.n_ctas : a.n_splits * ((a.p.n_q_heads + C::kG - 1) / C::kG) * a.p.batch;
  if (work.n_ctas > 0 && work.arrivals != nullptr) {
    e = cudaMemsetAsync(work.arrivals, 0, sizeof(unsigned int) * (size_t)a.p.batch * a.p.n_q_heads, stream);
    if (e != cudaSuccess) return e;
  }
  tc::stage1_tc_kernel<C><<<grid, C::kThreads, C::kSmemBytes, stream>>>(ta);
  return cudaGetLastError();
}

cudaError_t launch_stage1_tc(const KArgs& a, const void* table, int table_rows, const Stage1Work& work, bool any_rows,
                             cudaStream_t stream) {
  if (a.p.latent_dtype == WSVD_F16)
    return any_rows ? launch_tc<tc::Cfg<true, true>>(a, table, table_rows, work, stream)
                    : launch_tc<tc::Cfg<true, false>>(a, table, table_rows, work, stream);
  return any_rows ? launch_tc<tc::Cfg<false, true>>(a, table, table_rows, work, stream)
                  : launch_tc<tc::Cfg<false, false>>(a, table, table_rows, work, stream);
}

cudaError_t read_tc_status(unsigned int* out) {
  return cudaMemcpyFromSymbol(out, tc::g_status, sizeof(unsigned int));
}

cudaError_t reset_tc_status() {
  const unsigned int zero = 0;
  return cudaMemcpyToSymbol(tc::g_status, &zero, sizeof(unsigned int));
}

}  // namespace wsvd
