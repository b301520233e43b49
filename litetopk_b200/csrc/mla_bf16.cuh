// BF16 MLA attention over a per-tile list of KV rows (sm_100a): the kernel behind the DSv4 operators
// (attn_dsv4.cu) and the bf16 route of masked_mla_fp8 (attn_bf16.cu).
//
// Numerics are the reference bf16 kernel's (kernels/b200/dsa/litedsa_attention_sm100_dsv4.cuh:
// 2015-2157): base-2 online softmax over the list in rank order whose running max moves only when a
// row of a 32-row group overshoots it by more than 6, P stored as bf16 without pre-scale, fp32
// accumulation, optional sink in the output normaliser only.  Where the rows come from is a template
// parameter:
//   kRange   compressed-prefix entries [0, p / ratio) of one tensor, then the sliding window of
//            another: contiguous rows, tiled TMA loads, mask computed from the token position;
//   kRank    two contiguous runs of rows of one workspace per tile, mask from rank ranges
//            (range_mask32, litedsa_attention_sm100_dsv4.cuh:1824-1829), tiled TMA loads;
//   kGather  an index list per tile (rank ranges or membership bits), 16-byte cp.async row gather.
//
// Organisation: persistent clusters of 2 CTAs (64 query rows each), tcgen05 cta_group::2 kind::f16
// MMAs, 64-key blocks.  With kGather they are the reference's, so the running max takes the same course;
// kRange and kRank lay each of the two segments out in half blocks of 32 keys, so a block holds other
// keys and P can be rounded relative to another running max.  One block's
// chain of loads, QK^T, softmax and PV takes about 5000 cycles, its 44 MMAs about 1250, so four blocks
// or more have to be in flight.  To make room for them:
//   * a block's K tile BECOMES its V tile (as in the FP8 kernel, attn_fp8.cu): CTA c loads the rows of
//     its own 32 keys; once QK^T has read them the half of the value dims that is the peer's is dead,
//     and the peer keys' rows of this CTA's 256 dims are loaded there.  One 36 KB slot per block, five.
//   * 384 of Q's dims live in tensor memory (A operand from TMEM, rows duplicated in lanes 64-127 as
//     the 64-rows-per-CTA form wants); they pass through two ring slots on their way there.  The
//     other chunks stay in shared memory and are fetched as soon as the previous item's last QK^T is
//     complete (prefetched into L2 before).
//   * half of P lies in the block's own rope chunk, dead after QK^T, too (576 dims).
// Roles (17 warps, 24 with the gather):
//   warps 0-7   softmax, two groups of four on alternate blocks (TMEM lane x 32 columns per thread);
//   warp 8      QK^T issue of even blocks (leader CTA);
//   warps 9-10  TMA producers of Q / K and of V -- or, with the gather, relays of "K / V landed" from
//               the peer CTA to the leader, and in the leader PV issue (warp 9) and QK^T issue of odd blocks (warp 10);
//   warp 11     PV issue (leader CTA) -- or, with the gather, index-validity bits;
//   warps 12-15 Q into tensor memory; tile epilogue: O out of TMEM, x 1 / normaliser, bf16, TMA stores;
//   warp 16     QK^T issue of odd blocks (leader CTA) -- or, warps 16-23, KV row gather.
// No TMA multicast of any kind.  Every wait is bounded (common.cuh).
#pragma once
#include "common.cuh"
#include "tensor_map.cuh"

namespace lt {
namespace mla16 {

enum Source { kRange, kRank, kGather };
// The first of each kRunGroup tiles has the sign bit of its first row set if the list of one of them is not two runs.
constexpr int kRunGroup = 16;

constexpr int kSoftmaxWarps = 8, kGatherWarps = 8, kEpiWarps = 4;
constexpr int kWarpMma = 8, kWarpK = 9, kWarpV = 10, kWarpValid = 11, kWarpEpi0 = 12, kWarpGather0 = 16;
constexpr int kBlockKeys = 64, kOwnKeys = 32;
constexpr int kDV = 512;
constexpr int kSlots = 5;
constexpr int kQChunksTmem = 6, kQEntries = 2;        // 64-dim chunks of Q in tensor memory; ring entries they take
constexpr uint32_t kQChunkBytes = 64 * 128;           // 64 rows x 64 bf16
constexpr uint32_t kChunkBytes = kOwnKeys * 128;      // 32 keys x 64 bf16
constexpr uint32_t kPHalf = 64 * kOwnKeys * 2;        // 64 rows x 32 keys of P
constexpr uint32_t kStageBytes = 4 * 2048;            // output staging, one slice per epilogue warp
constexpr uint32_t kMiscBytes = 6144;

constexpr int threads_of(Source src) { return src == kGather ? 768 : 544; }

template <int kD>
struct Plan {
  static constexpr int kChunks = kD / 64;
  static constexpr int kQRes = kChunks - kQChunksTmem;              // chunks of Q kept in shared memory
  static constexpr uint32_t kSlot = kChunks * kChunkBytes;
  static constexpr bool kRopeP = kD == 576;                         // P's keys 0-31 in the rope chunk
  static constexpr uint32_t kPBuf = kRopeP ? kPHalf : 2 * kPHalf;   // per softmax group
  static constexpr uint32_t kOffKV = 0;
  static constexpr uint32_t kOffQ = kOffKV + kSlots * kSlot;
  static constexpr uint32_t kOffP = kOffQ + kQRes * kQChunkBytes;
  static constexpr uint32_t kOffStage = kOffP + 2 * kPBuf;
  static constexpr uint32_t kOffMisc = kOffStage + kStageBytes;
  static constexpr uint32_t kSmem = kOffMisc + kMiscBytes + 1024;   // + alignment slack
  static_assert(kSlot % 1024 == 0 && kOffQ % 1024 == 0 && kOffP % 1024 == 0, "swizzled tiles need 1024-byte alignment");
  static_assert(kQChunksTmem / kQEntries * kQChunkBytes <= kSlot, "Q passes through ring slots");
  static_assert(kSmem <= 232448, "shared-memory plan exceeds the 227 KB per-CTA limit");
};

constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kTmemO = 0;                        // 256 columns: O (64 rows x 512 dims per CTA)
constexpr uint32_t kTmemS0 = 256, kTmemS1 = 288;      // 32 columns each: S double buffer
constexpr uint32_t kTmemQ = 320;                      // 192 columns: 384 dims of Q (two bf16 per column)

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr float kMInit = -1e30f;
constexpr float kRescaleThreshold = 6.0f;

struct Misc {
  // in the leader CTA only: k_full / v_full (TMA bytes of both CTAs, or the leader's own cp.async
  // arrivals), k_peer / v_peer (gather: the peer's rows landed), q_res (TMA bytes of both CTAs),
  // s_free / p_ready (softmax warps of both CTAs).  Barriers per block are indexed by the running
  // block number modulo 8 (pv_done: modulo 4): with five slots everybody has looked at block kb's
  // barriers before block kb + 8 can touch them.
  uint64_t k_full[8], v_full[8], k_peer[8], v_peer[8], q_res, s_free[2], p_ready[2];
  // in every CTA
  uint64_t qk_done[8], pv_done[4], slot_free[kSlots], valid_ready[2], valid_free[2], m_pub[2];
  uint64_t q_land;                  // this CTA's Q chunks for tensor memory have landed in their slot
  uint64_t q_taken[2];              // they have been moved out of it, by parity of the item ordinal
  uint64_t qt_ready;                // leader CTA: they are in tensor memory in both CTAs
  uint64_t q_free;                  // all QK^T of the current item are complete
  uint64_t o_free;                  // leader CTA: the item's O has been read out of TMEM
  uint64_t epi_ready[2];            // the item's row scales are published, by parity of the item ordinal: with
                                    // items of one or two blocks the next item's can be complete before the
                                    // epilogue has looked at this one's
  uint32_t valid[2][2];             // 64 validity bits per stage (gather)
  uint32_t tmem_base;
  // for the tear-down of a launch that gives up: a wait of this block has; ring entries of Q that have been requested, items
  // whose resident chunks have, and at whose q_land each K warp has arrived; leader: blocks whose QK^T (per issuing warp) and PV have been issued
  uint32_t left, q_asked, q_res_asked, q_passed[kGatherWarps / 2], qk_end[2], pv_end;
  float xbuf[2][2][128];            // [group][parity][lane]: row-max exchange between key halves
  float mshare[2][64];              // [group][row]: running max after the group's latest block
  float fin_l[256];                 // end of item: row sums per thread,
  float fin_rm[128], fin_m[128];    // true maxima, last running max per (group, row)
  float oscale[2][64];              // [item parity][row]: 1 / normaliser, 0 for rows without a key
};
static_assert(sizeof(Misc) <= kMiscBytes, "Misc too large");

struct Params {
  float* lse;                // [ng, 128]
  float* max_logits;         // [ng, 128] or null
  const float* sink;         // natural-log units, indexed by packed row modulo sink_mod, or null
  int sink_mod;              // 128: one value per packed row; h_per_q: one per head
  int ng, G, h_per_q;
  float scale_log2;
  int epoch;                          // this launch's epoch for the bounded waits
  uint32_t wait_limit;       // of one wait, in ticks (BlockWaiter)
  // slices: every tile's blocks are cut into nsplit > 1 work items, each leaving its unnormalised
  // O (fp32 [ng * nsplit, 128, 512]) and (running max, row sum) for merge_slices
  int nsplit;
  float* part_o;
  float2* part_ml;
  // The device-side choice between the rank and the gather form of one call: the rank form runs if no group of tiles is
  // marked in `runs` (kGather: null: it always runs), the gather form if one is.
  const int4* runs;          // [ng]: (first row of run 0, its length, first row of run 1, its length); groups: see kRunGroup
  // kRange: token t of the call sits at pos0 + t
  int n_comp, pos0, window, ratio;
  // kGather: rows of kv (kv_pitch bytes apart) by index
  const uint8_t* kv;
  long long kv_pitch, idx_stride;
  const int32_t* indices;    // [ng, idx_stride]
  const uint32_t* memb;      // [ng, G, cap / 32] membership bits, or null (rank ranges)
  int s_kv, cap;
  // kRank, kGather without memb: rank < pref, or win_lo <= rank < win_hi; all < counts
  const int32_t* pref;       // [ng, G]
  const int32_t* win_lo;
  const int32_t* win_hi;
  const int32_t* counts;     // [ng] or null
  const int2* order;         // kOrdered: [ng] (tile, its counts clamped to cap) in the order in which they are dealt out
};

enum { kSiteQ = 101, kSiteKFull, kSiteQkDone, kSitePvDone, kSiteValidReady, kSiteValidFree,
       kSiteKFree, kSiteVFree, kSitePFree, kSiteEpi, kSiteQFree, kSiteMPub, kSiteRelayK, kSiteRelayV,
       kSiteSFree, kSiteOFree, kSitePReady };

// status block of the kernels of this translation unit (layout: see Waiter in common.cuh)
static __device__ int g_status[8];

// One work item: blocks [k0, k0 + nb) of a tile.  Half block 2 b + c (32 keys, the ones CTA c loads) is the
// unit in which a tile's keys are laid out.  kRange / kRank: the first nh0 half blocks walk len0 rows
// from row0, the others len1 rows from row1 -- a block may hold the end of one segment and the
// start of the other (128-key windows of two tokens are 129 keys: five half blocks, not three
// blocks).  kGather: len0 list entries.
struct Item {
  int tile, k0, nb, nh0, row0, len0, row1, len1;
};

// bits [0, x) of a 32-bit word (x may be negative or beyond 32)
__device__ __forceinline__ uint32_t low_bits(int x) {
  return x <= 0 ? 0u : (x >= 32 ? 0xffffffffu : ((1u << x) - 1u));
}
__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
  return e != 0;
}
__device__ __forceinline__ void commit_one(uint32_t a) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(a) : "memory");
}
// MMA loops, run by ONE elected thread under one branch: with an elect-predicated MMA in a warp-wide
// loop an MMA took 55-67 cycles to issue here, whatever the loop around it; this way it takes 21, and
// the tensor pipe (18-25 cycles per QK^T step at N = 64, 64 per PV step) is the limit.
// Four steps of one 64-dim chunk (16 dims each): A in tensor memory (two bf16 per column) / shared
// memory, B at k_lo; descriptors differ only in their low word (start address >> 4).
__device__ __forceinline__ void mma4_ts(uint32_t d, uint32_t q_tmem, uint32_t k_lo, uint32_t hi, uint32_t idesc,
                                        uint32_t accumulate_first) {
  asm volatile(
      "{\n\t.reg .pred pf, po;\n\t.reg .b32 qa, lo;\n\t.reg .b64 bd;\n\t"
      "setp.ne.b32 pf, %5, 0;\n\tsetp.eq.b32 po, 0, 0;\n\t"
      "mov.b64 bd, {%2, %3};\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], [%1], bd, %4, pf;\n\t"
      "add.u32 qa, %1, 8;\n\tadd.u32 lo, %2, 2;\n\tmov.b64 bd, {lo, %3};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [qa], bd, %4, po;\n\t"
      "add.u32 qa, %1, 16;\n\tadd.u32 lo, %2, 4;\n\tmov.b64 bd, {lo, %3};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [qa], bd, %4, po;\n\t"
      "add.u32 qa, %1, 24;\n\tadd.u32 lo, %2, 6;\n\tmov.b64 bd, {lo, %3};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [qa], bd, %4, po;\n\t}"
      ::"r"(d), "r"(q_tmem), "r"(k_lo), "r"(hi), "r"(idesc), "r"(accumulate_first) : "memory");
}
__device__ __forceinline__ void mma4_ss(uint32_t d, uint32_t q_lo, uint32_t k_lo, uint32_t hi, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred po;\n\t.reg .b32 alo, lo;\n\t.reg .b64 ad, bd;\n\t"
      "setp.eq.b32 po, 0, 0;\n\t"
      "mov.b64 ad, {%1, %3};\n\tmov.b64 bd, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], ad, bd, %4, po;\n\t"
      "add.u32 alo, %1, 2;\n\tadd.u32 lo, %2, 2;\n\tmov.b64 ad, {alo, %3};\n\tmov.b64 bd, {lo, %3};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], ad, bd, %4, po;\n\t"
      "add.u32 alo, %1, 4;\n\tadd.u32 lo, %2, 4;\n\tmov.b64 ad, {alo, %3};\n\tmov.b64 bd, {lo, %3};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], ad, bd, %4, po;\n\t"
      "add.u32 alo, %1, 6;\n\tadd.u32 lo, %2, 6;\n\tmov.b64 ad, {alo, %3};\n\tmov.b64 bd, {lo, %3};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], ad, bd, %4, po;\n\t}"
      ::"r"(d), "r"(q_lo), "r"(k_lo), "r"(hi), "r"(idesc) : "memory");
}
// four steps of 16 keys of P V into one N = 256 accumulator: keys 0-31 (P at p0_lo, V at v_lo), then keys
// 32-63 (p1_lo, four V chunks further); 2048 bytes per step
__device__ __forceinline__ void mma4_pv(uint32_t d, uint32_t p0_lo, uint32_t p1_lo, uint32_t v_lo, uint32_t p_hi,
                                        uint32_t v_hi, uint32_t idesc, uint32_t accumulate_first) {
  asm volatile(
      "{\n\t.reg .pred pf, po;\n\t.reg .b32 alo, lo;\n\t.reg .b64 ad, bd;\n\t"
      "setp.ne.b32 pf, %7, 0;\n\tsetp.eq.b32 po, 0, 0;\n\t"
      "mov.b64 ad, {%1, %4};\n\tmov.b64 bd, {%3, %5};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], ad, bd, %6, pf;\n\t"
      "add.u32 alo, %1, 128;\n\tadd.u32 lo, %3, 128;\n\tmov.b64 ad, {alo, %4};\n\tmov.b64 bd, {lo, %5};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], ad, bd, %6, po;\n\t"
      "add.u32 lo, %3, 1024;\n\tmov.b64 ad, {%2, %4};\n\tmov.b64 bd, {lo, %5};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], ad, bd, %6, po;\n\t"
      "add.u32 alo, %2, 128;\n\tadd.u32 lo, %3, 1152;\n\tmov.b64 ad, {alo, %4};\n\tmov.b64 bd, {lo, %5};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], ad, bd, %6, po;\n\t}"
      ::"r"(d), "r"(p0_lo), "r"(p1_lo), "r"(v_lo), "r"(p_hi), "r"(v_hi), "r"(idesc), "r"(accumulate_first) : "memory");
}
// S = Q K^T of one block: chunks 0-5 of Q in tensor memory, the others in shared memory
template <int kD>
__device__ __forceinline__ void mma_qk(uint32_t d, uint32_t q_tmem, uint32_t q_lo, uint32_t k_lo, uint32_t hi,
                                       uint32_t idesc) {
#pragma unroll 1
  for (int j = 0; j < kQChunksTmem; ++j) mma4_ts(d, q_tmem + 32 * j, k_lo + 256 * j, hi, idesc, j);
  k_lo += 256 * kQChunksTmem;
#pragma unroll 1
  for (int j = 0; j < kD / 64 - kQChunksTmem; ++j) mma4_ss(d, q_lo + 512 * j, k_lo + 256 * j, hi, idesc);
}
// O += P V of one block: two N = 256 halves (128 dims of each CTA, D column offset 128, V chunks 0-1 / 2-3)
__device__ __forceinline__ void mma_pv(uint32_t d, uint32_t v_lo, uint32_t p0_lo, uint32_t p1_lo, uint32_t p_hi,
                                       uint32_t v_hi, uint32_t idesc, uint32_t accumulate) {
#pragma unroll 1
  for (int i = 0; i < 2; ++i) mma4_pv(d + 128 * i, p0_lo, p1_lo, v_lo + 512 * i, p_hi, v_hi, idesc, accumulate);
}

template <int kD, Source kSrc, bool kSliced, bool kOrdered>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(threads_of(kSrc), 1)
mla_bf16_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kv0,
                const __grid_constant__ CUtensorMap map_kv1, const __grid_constant__ CUtensorMap map_out,
                const Params p) {
  using PL = Plan<kD>;
  constexpr int kChunks = PL::kChunks, kQRes = PL::kQRes;
  constexpr bool kTma = kSrc != kGather;
  constexpr int kWarpQkOdd = kTma ? kWarpGather0 : kWarpV;      // second QK^T warp: where the gather's peer has its V relay
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sbase = (raw + 1023u) & ~1023u;       // 128B-swizzle tiles need 1024-byte alignment
  uint8_t* sm = smem_raw + (sbase - raw);
  Misc& ms = *reinterpret_cast<Misc*>(sm + PL::kOffMisc);
  const BlockWaiter wt{&ms.left, p.wait_limit};
  pdl_trigger();
  // whether a list of the call is not two runs (grid-uniform)
  auto scattered = [&]() -> bool {
    int marked = 0;
    for (int i = threadIdx.x * kRunGroup; i < p.ng; i += blockDim.x * kRunGroup) marked |= __ldcg(&p.runs[i].x) < 0;
    return __syncthreads_or(marked) != 0;
  };
  if (kSrc == kGather && p.runs != nullptr) {
    pdl_wait();
    if (!scattered()) return;
  }

  // Persistent: each cluster walks items cid, cid + #clusters, ...  Every role runs the same item
  // loop; slots, buffers and barrier phases are indexed by the cluster-wide running block number kb,
  // so the next item's loads and first QK^T overlap the previous item's last softmax blocks and
  // its epilogue.  Ring entries: each item's Q chunks, then its blocks; entry of running block kb
  // of item ordinal it: kb + 2 it + 2.
  const uint32_t cta = cluster_ctarank();
  const int cid = blockIdx.x >> 1, ncl = gridDim.x >> 1;
  const int n_items = kSliced ? p.ng * p.nsplit : p.ng;
  // broadcast so the compiler knows the role index is warp-uniform
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  auto halves_of = [](int n) -> int { return (n + kOwnKeys - 1) / kOwnKeys; };
  auto tile_of = [&](int w) -> int { return kSliced ? w / p.nsplit : kOrdered ? __ldcg(&p.order[w].x) : w; };
  auto item_of = [&](int w) -> Item {
    Item t;
    t.row0 = t.row1 = t.len1 = 0;
    if (kOrdered) {
      const int2 v = __ldcg(p.order + w);
      t.tile = v.x; t.len0 = v.y;
    } else {
      t.tile = tile_of(w);
    }
    if (kOrdered) {
    } else if (kSrc == kRange) {
      const int p0 = p.pos0 + t.tile * p.G, plast = p0 + p.G - 1;
      t.len0 = min(plast / p.ratio, p.n_comp);
      t.row1 = max(0, p0 - p.window + 1);
      t.len1 = plast - t.row1 + 1;
    } else if (kSrc == kRank) {
      const int4 r = __ldcg(p.runs + t.tile);
      t.row0 = r.x; t.len0 = max(r.y, 0);
      t.row1 = r.z; t.len1 = max(r.w, 0);
    } else {
      t.len0 = min(max(p.counts ? __ldcg(p.counts + t.tile) : p.cap, 0), p.cap);
    }
    t.nh0 = halves_of(t.len0);
    t.k0 = 0;
    t.nb = max((t.nh0 + halves_of(t.len1) + 1) / 2, 1);     // an empty list: one fully masked block
    if (kSliced) {            // slice `part`; an empty one runs a block beyond the list: fully masked
      const int part = w - t.tile * p.nsplit, all = t.nb;
      t.k0 = part * all / p.nsplit;
      t.nb = (part + 1) * all / p.nsplit - t.k0;
      if (t.nb == 0) { t.nb = 1; t.k0 = all; }
    }
    return t;
  };

  if (threadIdx.x == 0) {
    mbar_init(&ms.q_res, 1);
    mbar_init(&ms.q_land, kQEntries + (kTma ? 0 : kGatherWarps / 2 - 1));      // gather: and the other K warps
    ms.left = ms.q_asked = ms.q_res_asked = ms.qk_end[0] = ms.qk_end[1] = ms.pv_end = 0;
    for (int i = 0; i < kGatherWarps / 2; ++i) ms.q_passed[i] = 0;
    mbar_init(&ms.qt_ready, 2 * kEpiWarps);
    mbar_init(&ms.q_free, 2);              // both QK^T warps
    mbar_init(&ms.o_free, 2 * kEpiWarps);
    for (int i = 0; i < 8; ++i) {
      mbar_init(&ms.k_full[i], kTma ? 1 : kGatherWarps / 2 * 32);     // gather: one async arrival per thread
      mbar_init(&ms.v_full[i], kTma ? 1 : kGatherWarps / 2 * 32);
      mbar_init(&ms.k_peer[i], 1);
      mbar_init(&ms.v_peer[i], 1);
      mbar_init(&ms.qk_done[i], 1);
    }
    for (int i = 0; i < 4; ++i) mbar_init(&ms.pv_done[i], 1);
    for (int i = 0; i < kSlots; ++i) mbar_init(&ms.slot_free[i], 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&ms.s_free[i], 8);         // 4 warps of one softmax group x 2 CTAs
      mbar_init(&ms.p_ready[i], 8);
      mbar_init(&ms.valid_ready[i], 1);
      mbar_init(&ms.valid_free[i], 4);
      mbar_init(&ms.m_pub[i], 4);
      mbar_init(&ms.epi_ready[i], kSoftmaxWarps);
      mbar_init(&ms.q_taken[i], 1);
    }
    fence_mbar_init();
    tma_prefetch_desc(&map_q);
    if (kTma) { tma_prefetch_desc(&map_kv0); tma_prefetch_desc(&map_kv1); }
    if (!kSliced) tma_prefetch_desc(&map_out);
  }
  __syncthreads();
  cluster_sync_all();
  if (warp == kWarpMma) {
    tmem_alloc_pair(&ms.tmem_base, kTmemCols);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, ms.tmem_base, 0);
  if (kSrc != kGather || p.runs == nullptr) pdl_wait();      // (the set-up overlaps the kernel before)
  if (kSrc == kRank && scattered()) {
    cluster_sync_all();
    if (warp == kWarpMma) tmem_dealloc_pair(tmem, kTmemCols);
    return;
  }

  // Requests half `e` of an item's Q chunks for tensor memory into ring slot `slot` (one thread); the
  // other chunks go into L2, for the fetch that follows the previous item's last QK^T.  (Nothing behind a wait that gave
  // up: the Q before could still be in flight.)
  const uint64_t pol_stream = l2_policy_evict_first();
  const int q_head = (64 * (int)cta) % p.h_per_q, q_tok0 = (64 * (int)cta) / p.h_per_q;
  auto request_q = [&](int w, int it, int e, int slot) {
    constexpr int kPer = kQChunksTmem / kQEntries;
    if (wt.aborting()) return;
    ms.q_asked = kQEntries * it + e + 1;
    const int qt = tile_of(w) * p.G + q_tok0;
    mbar_arrive_expect_tx(&ms.q_land, kPer * kQChunkBytes);
    for (int j = 0; j < kPer; ++j)
      tma_load_3d_hint(sbase + PL::kOffKV + slot * PL::kSlot + j * kQChunkBytes, &map_q, 64 * (kPer * e + j), q_head,
                       qt, &ms.q_land, pol_stream);
    if (e == 0)
      for (int j = kQChunksTmem; j < kChunks; ++j) tma_prefetch_3d(&map_q, 64 * j, q_head, qt);
  };

  if (warp < kSoftmaxWarps) {
    // ------------------------------------------------------------ softmax
    // Group g serves the blocks with kb % 2 == g; thread = TMEM lane tl: tile row r = tl % 64, keys
    // [32 h, +32) of the block with h = tl / 64.  The only state that crosses groups is the running
    // max, handed over right after a block's row maxima are known; the row sum is kept per thread
    // relative to the max of the group's latest block.
    const int g = warp >> 2;
    const int tl = ((warp & 3) << 5) | lane;
    const int r = tl & 63, h = tl >> 6;
    const int row = (int)cta * 64 + r;
    const int q = row / p.h_per_q;                // token of the tile this row belongs to
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const int capw = p.cap >> 5;
    const float c = p.scale_log2;
    const uint64_t c2 = pack2(c, c);
    const uint32_t a_s_free = mapa(smem_u32(&ms.s_free[g]), 0);
    const uint32_t a_p_ready = mapa(smem_u32(&ms.p_ready[g]), 0);
    const uint32_t scol = tmem + lane_base + (g ? kTmemS1 : kTmemS0);
    int kb0 = 0, it = 0;

    for (int w = cid; w < n_items; w += ncl) {
      const Item item = item_of(w);
      const int nb = item.nb;
      const size_t trow = (size_t)item.tile * p.G + q;            // (tile, token) of this row
      // list ranks this token may attend: rank < pref, or lo <= rank < hi
      int pref = 0, lo = 0, hi = 0;
      const uint32_t* mrow = nullptr;
      if (kSrc == kRange) {
        const int pq = p.pos0 + item.tile * p.G + q;
        pref = min(pq / p.ratio, p.n_comp);
        lo = item.len0 + max(pq - p.window + 1, 0) - item.row1;
        hi = item.len0 + pq + 1 - item.row1;
      } else if (kSrc == kGather && p.memb) {
        mrow = p.memb + trow * capw + h;
      } else {
        const int total = item.len0 + item.len1;
        const int cnt = p.counts ? min(max(__ldcg(p.counts + item.tile), 0), total) : total;
        pref = min(__ldcg(p.pref + trow), cnt);
        lo = __ldcg(p.win_lo + trow);
        hi = min(__ldcg(p.win_hi + trow), cnt);
      }
      float m_mine = kMInit;      // the running max my row sum is relative to
      float li = 0.f, real_m = -INFINITY;
      const int k_first = (g - kb0) & 1;          // first local block with (kb0 + k) % 2 == g
      uint32_t mk = 0u;
      if (mrow && k_first < nb) mk = __ldcs(mrow + 2 * (item.k0 + k_first));

      for (int k = k_first; k < nb; k += 2) {
        const int kb = kb0 + k;
        const uint32_t ph = (kb >> 1) & 1;
        uint32_t mk_next = 0u;
        if (kSrc == kGather && mrow && k + 2 < nb) mk_next = __ldcs(mrow + 2 * (item.k0 + k + 2));

        mbar_wait(&ms.qk_done[kb & 7], (kb >> 3) & 1, wt, kSiteQkDone, k);
        __syncwarp();      // lanes leave the wait loop one by one: re-converge before .aligned ops
        tc_fence_after();
        float sv[32];
        tmem_ld32(scol, sv);
        tmem_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(a_s_free);

        uint32_t vm;
        {
          const int hb = 2 * (item.k0 + k) + h;
          const bool seg0 = kSrc == kGather || hb < item.nh0;
          const int base = (seg0 ? hb : hb - item.nh0) * kOwnKeys;            // within the segment
          const int off = (seg0 ? 0 : item.len0) + base;                      // list rank of column 0
          if (kSrc == kGather && mrow)
            vm = mk;
          else
            vm = low_bits(pref - off) | (low_bits(hi - off) & ~low_bits(lo - off));
          if (kTma) vm &= low_bits((seg0 ? item.len0 : item.len1) - base);
        }
        if (!kTma) {
          mbar_wait(&ms.valid_ready[g], ph, wt, kSiteValidReady, k);
          vm &= ms.valid[g][h];
          __syncwarp();
          if (lane == 0) mbar_arrive(&ms.valid_free[g]);
          mk = mk_next;
        }

        if (vm != ~0u) {
#pragma unroll
          for (int j = 0; j < 32; ++j) sv[j] = ((vm >> j) & 1u) ? sv[j] : -INFINITY;
        }
        float mx[4] = {sv[0], sv[1], sv[2], sv[3]};
#pragma unroll
        for (int j = 4; j < 32; j += 4) {
          mx[0] = fmaxf(mx[0], sv[j]);
          mx[1] = fmaxf(mx[1], sv[j + 1]);
          mx[2] = fmaxf(mx[2], sv[j + 2]);
          mx[3] = fmaxf(mx[3], sv[j + 3]);
        }
        float cur = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * c;
        float* xb = ms.xbuf[g][ph];
        xb[tl] = cur;
        if (g == 0) asm volatile("bar.sync 1, 128;" ::: "memory");
        else asm volatile("bar.sync 2, 128;" ::: "memory");
        cur = fmaxf(cur, xb[tl ^ 64]);
        real_m = fmaxf(real_m, cur);
        // running max after block k-1 of this item comes from the other group
        float m_prev = kMInit;
        if (k > 0) {
          mbar_wait(&ms.m_pub[g ^ 1], ((kb - 1) >> 1) & 1, wt, kSiteMPub, k);
          m_prev = ms.mshare[g ^ 1][r];
        }
        const bool rescale = __any_sync(0xffffffffu, cur - m_prev > kRescaleThreshold);
        const float new_m = rescale ? fmaxf(cur, m_prev) : m_prev;
        if (h == 0) ms.mshare[g][r] = new_m;
        __syncwarp();
        if (lane == 0) mbar_arrive(&ms.m_pub[g]);
        li *= fast_exp2(m_mine - new_m);
        m_mine = new_m;

        const uint64_t nm2 = pack2(-new_m, -new_m);
        uint32_t pk[16];
        uint64_t l2 = 0;              // a pair of partial sums
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          float2 d = unpack2(fma2(pack2(sv[j], sv[j + 1]), c2, nm2));
          d.x = fast_exp2(d.x);
          d.y = fast_exp2(d.y);
          l2 = add2(l2, pack2(d.x, d.y));
          const __nv_bfloat162 b2 = __floats2bfloat162_rn(d.x, d.y);
          pk[j >> 1] = *reinterpret_cast<const uint32_t*>(&b2);
        }
        const float2 ls = unpack2(l2);
        li += ls.x + ls.y;
        // P: [64 rows][32 keys] per half, K-major core matrices (8-key group at 1024 * group + 16 * row).
        // Keys 0-31 go into the block's own rope chunk (576 dims); the other buffer was last read by
        // the PV of block kb - 2.
        uint32_t poff;
        if (PL::kRopeP && h == 0)
          poff = PL::kOffKV + (uint32_t)((kb + 2 * it + 2) % kSlots) * PL::kSlot + (kChunks - 1) * kChunkBytes;
        else
          poff = PL::kOffP + (uint32_t)g * PL::kPBuf + (PL::kRopeP ? 0 : h * kPHalf);
        if (kb >= 2) mbar_wait(&ms.pv_done[(kb - 2) & 3], ((kb - 2) >> 2) & 1, wt, kSitePFree, k);
        uint8_t* pdst = sm + poff + r * 16;
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<uint4*>(pdst + i * 1024) =
              make_uint4(pk[4 * i], pk[4 * i + 1], pk[4 * i + 2], pk[4 * i + 3]);

        if (rescale && k > 0) {
          // O holds blocks [0, k) relative to m_prev: bring it to new_m once PV(k-1) is complete
          mbar_wait(&ms.pv_done[(kb - 1) & 3], ((kb - 1) >> 2) & 1, wt, kSitePvDone, k);
          __syncwarp();
          tc_fence_after();
          const float f = fast_exp2(m_prev - new_m);
          float o[32];
#pragma unroll 1
          for (int cc = 0; cc < 8; ++cc) {
            const uint32_t ocol = tmem + lane_base + kTmemO + cc * 32;
            tmem_ld32(ocol, o);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 32; ++j) o[j] *= f;
            tmem_st32(ocol, o);
          }
          tmem_wait_st();
          tc_fence_before();
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(a_p_ready);
      }

      // end of item: merge the row sums (each relative to its own group's latest running max; the
      // previous item's sums have been read once every warp has arrived on its epi_ready)
      if (it > 0) mbar_wait(&ms.epi_ready[(it - 1) & 1], ((it - 1) >> 1) & 1, wt, kSiteEpi, it);
      ms.fin_l[g * 128 + tl] = li;
      if (h == 0) {
        ms.fin_rm[g * 64 + r] = real_m;
        ms.fin_m[g * 64 + r] = m_mine;
      }
      asm volatile("bar.sync 3, 256;" ::: "memory");
      if (g == 0 && h == 0) {
        const int last_g = (kb0 + nb - 1) & 1;      // group of the item's last block
        float m = ms.fin_m[last_g * 64 + r];        // running max after the last block
        float lsum = 0.f;
        real_m = -INFINITY;
        // fixed summation order (even local blocks first, whichever group served them), so an
        // item's result does not depend on the blocks its cluster processed before
        const int g_even = kb0 & 1;
#pragma unroll
        for (int gi = 0; gi < 2; ++gi) {
          const int gg = gi ^ g_even;
          const float f = fast_exp2(ms.fin_m[gg * 64 + r] - m);
          lsum += ms.fin_l[gg * 128 + r] * f;
          lsum += ms.fin_l[gg * 128 + 64 + r] * f;
          real_m = fmaxf(real_m, ms.fin_rm[gg * 64 + r]);
        }
        li = lsum;
        if (real_m == -INFINITY) { li = 0.f; m = -INFINITY; }
        if (kSliced) {
          p.part_ml[(size_t)w * 128 + row] = make_float2(m, li);
        } else {
          const size_t grow = (size_t)item.tile * 128 + row;
          float l = __logf(li) + m * kLn2;
          if (!(li > 0.f)) l = INFINITY;
          p.lse[grow] = l;
          if (p.max_logits) p.max_logits[grow] = real_m * kLn2;
          // the epilogue warps need 1 / normaliser per row; the sink joins it here only
          float denom = li;
          if (p.sink != nullptr && li > 0.f) denom += fast_exp2(__ldcg(p.sink + row % p.sink_mod) * kLog2e - m);
          ms.oscale[it & 1][r] = (li > 0.f) ? __fdividef(1.0f, denom) : 0.f;
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&ms.epi_ready[it & 1]);
      kb0 += nb;
      ++it;
    }
  } else if (warp < kWarpEpi0 || (kTma && warp == kWarpQkOdd)) {
   if (!kTma) asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
   // running position of an MMA-issuing warp: work item, block of the item, blocks of the item, item
   // ordinal, running block number, ring slot
   struct MmaCursor { int w, k, nb, it, kb, slot; };
   auto mma_next = [&](MmaCursor& c) {
     ++c.kb;
     if (++c.slot == kSlots) c.slot = 0;
     if (++c.k == c.nb) {
       c.w += ncl; c.k = 0; ++c.it;
       c.slot += kQEntries;                       // the next item's Q entries
       if (c.slot >= kSlots) c.slot -= kSlots;
       c.nb = c.w < n_items ? item_of(c.w).nb : 0;
     }
   };
   // the time-limit and abort check of a wait that has not been satisfied yet (warp-uniform answer)
   auto mma_idle = [&](uint32_t& since, int site, int kb) -> bool {
     return __any_sync(0xffffffffu, wt.gives_up(since, site, kb));
   };
   if (warp == kWarpMma || (warp == kWarpQkOdd && (kTma || cta == 0))) {
    // ------------------------------------------------------------ QK^T issue (leader CTA)
    // Three warps issue the MMAs, two QK^T, of even and odd blocks, and one PV: each waits for its own operands and the
    // tensor pipe takes what comes first.  (One warp polling for all needed 150-300 cycles per look and
    // could not look at all while its MMAs filled the queue.  With one for QK^T there were 600 cycles, 420 without the gather,
    // from its last MMA of a block to its first of the next, cursor, polls and commits, with the pipe idle as soon as it had
    // caught up: per 64-key block 1880 and 1450 cycles; native cache, 1184 tokens x 64 heads, top-2048 375 -> 354 us,
    // ranges, 1184 x 64 at 131072 159 -> 156.)
    if (cta == 0) {
      constexpr uint32_t idesc_qk = umma_idesc(1, 1, false, false, 128, kBlockKeys);
      const uint32_t a_qk_done = smem_u32(&ms.qk_done[0]), a_qk_done_peer = mapa(a_qk_done, 1);
      const uint32_t a_q_free = smem_u32(&ms.q_free), a_q_free_peer = mapa(a_q_free, 1);
      const uint64_t q_desc = umma_desc(sbase + PL::kOffQ, 16, 1024, kSwz128);
      static_assert(kChunkBytes >> 4 == 256 && kQChunkBytes >> 4 == 512, "strides of the MMA loops");
      // S of block kb goes into S buffer kb % 2
      auto issue_qk = [&](int kb, int slot) {
        if (!kTma) fence_proxy_async_smem();     // rows written by cp.async, read through the async proxy
        tc_fence_after();
        const uint64_t kd = umma_desc(sbase + PL::kOffKV + slot * PL::kSlot, 16, 1024, kSwz128);
        if (elect_one()) {
        mma_qk<kD>(tmem + ((kb & 1) ? kTmemS1 : kTmemS0), tmem + kTmemQ, (uint32_t)q_desc, (uint32_t)kd,
                   (uint32_t)(kd >> 32), idesc_qk);
        commit_one(a_qk_done + 8u * (uint32_t)(kb & 7));
        commit_one(a_qk_done_peer + 8u * (uint32_t)(kb & 7));
        }
        __syncwarp();
      };
      const int mine = warp == kWarpMma ? 0 : 1;
      MmaCursor c{cid, 0, cid < n_items ? item_of(cid).nb : 0, 0, 0, kQEntries};
      auto step = [&]() {
        const int it = c.it;
        mma_next(c);
        if (c.it != it && elect_one()) {      // this warp's QK^T of the item, if it had any
          commit_one(a_q_free);
          commit_one(a_q_free_peer);
        }
        __syncwarp();
      };
      bool aborted = false;
      uint32_t since = 0;
      while (c.w < n_items && !aborted) {
        // K rows landed on both CTAs, S buffer drained and, for an item's first block, Q in place.  Both warps stop at
        // every item's first block, whoever's it is: one that had none in an item could otherwise report two items
        // as read before the other has read one.
        const uint32_t ph = (c.kb >> 3) & 1;
        const bool own = (c.kb & 1) == mine;
        const bool ok = (c.k > 0 || (mbar_try_wait(&ms.qt_ready, c.it & 1) && mbar_try_wait(&ms.q_res, c.it & 1))) &&
                        (!own || (mbar_try_wait(&ms.k_full[c.kb & 7], ph) && (kTma || mbar_try_wait(&ms.k_peer[c.kb & 7], ph)) &&
                                  (c.kb < 2 || mbar_try_wait(&ms.s_free[c.kb & 1], ((c.kb >> 1) & 1) ^ 1))));
        if (__all_sync(0xffffffffu, ok)) {
          if (own) issue_qk(c.kb, c.slot);
          step();
          if (own && c.k != 0) step();      // the other warp's block
          since = 0;
        } else {
          aborted = mma_idle(since, kSiteKFull, c.kb);
        }
      }
      if (lane == 0) ms.qk_end[mine] = (c.kb + 1 - mine) / 2;      // of its own
    }
   } else if (warp == (kTma ? kWarpValid : kWarpK) && cta == 0) {
    // ------------------------------------------------------------ PV issue (leader CTA)
      constexpr uint32_t idesc_pv = umma_idesc(1, 1, false, true, 128, 256);
      const uint32_t a_pv_done = smem_u32(&ms.pv_done[0]), a_pv_done_peer = mapa(a_pv_done, 1);
      const uint32_t a_slot_free = smem_u32(&ms.slot_free[0]), a_slot_free_peer = mapa(a_slot_free, 1);
      auto issue_pv = [&](int k, int kb, int slot) {
        if (!kTma) fence_proxy_async_smem();
        tc_fence_after();
        const uint32_t kv = sbase + PL::kOffKV + slot * PL::kSlot;
        const uint32_t pb = sbase + PL::kOffP + (uint32_t)(kb & 1) * PL::kPBuf;
        const uint64_t vd = umma_desc(kv, kChunkBytes, 1024, kSwz128);
        const uint64_t p0 = umma_desc(PL::kRopeP ? kv + (kChunks - 1) * kChunkBytes : pb, 1024, 128, kSwzNone);
        const uint64_t p1 = umma_desc(PL::kRopeP ? pb : pb + kPHalf, 1024, 128, kSwzNone);
        if (elect_one()) {
        mma_pv(tmem + kTmemO, (uint32_t)vd, (uint32_t)p0, (uint32_t)p1, (uint32_t)(p0 >> 32), (uint32_t)(vd >> 32),
               idesc_pv, k ? 1u : 0u);
        commit_one(a_slot_free + 8u * (uint32_t)slot);
        commit_one(a_slot_free_peer + 8u * (uint32_t)slot);
        commit_one(a_pv_done + 8u * (uint32_t)(kb & 3));
        commit_one(a_pv_done_peer + 8u * (uint32_t)(kb & 3));
        }
        __syncwarp();
      };
      MmaCursor c{cid, 0, cid < n_items ? item_of(cid).nb : 0, 0, 0, kQEntries};
      bool aborted = false;
      uint32_t since = 0;
      while (c.w < n_items && !aborted) {
        // V rows landed on both CTAs, P written; an item's first PV overwrites O: the previous item
        // must have read it out
        const uint32_t ph = (c.kb >> 3) & 1;
        const bool ok = mbar_try_wait(&ms.v_full[c.kb & 7], ph) && (kTma || mbar_try_wait(&ms.v_peer[c.kb & 7], ph)) &&
                        (c.k > 0 || c.it == 0 || mbar_try_wait(&ms.o_free, (c.it - 1) & 1)) &&
                        mbar_try_wait(&ms.p_ready[c.kb & 1], (c.kb >> 1) & 1);
        if (__all_sync(0xffffffffu, ok)) {
          issue_pv(c.k, c.kb, c.slot);
          mma_next(c);
          since = 0;
        } else {
          aborted = mma_idle(since, kSitePReady, c.kb);
        }
      }
      if (lane == 0) ms.pv_end = c.kb;
   } else if (kTma && (warp == kWarpK || warp == kWarpV)) {
    // ------------------------------------------------------------ TMA producers (tiled loads, one lane)
    if (lane == 0) {
      const bool is_v = warp == kWarpV;
      const uint32_t a_k_full = mapa(smem_u32(&ms.k_full[0]), 0), a_v_full = mapa(smem_u32(&ms.v_full[0]), 0);
      int slot = 0, ring = 0, kb = 0, it = 0;
      auto advance = [&]() { if (++slot == kSlots) { slot = 0; ++ring; } };
      bool ok = true;
      for (int w = cid; w < n_items && ok; w += ncl, ++it) {
        const Item item = item_of(w);
        // the previous item's Q must have been moved on: with short items its bytes could still be in flight
        if (!is_v && it > 0) ok = mbar_wait(&ms.q_taken[(it - 1) & 1], ((it - 1) >> 1) & 1, wt, kSiteQFree, kb);
        for (int e = 0; e < kQEntries && ok; ++e) {
          if (!is_v) {
            if (ring > 0) ok = mbar_wait(&ms.slot_free[slot], (ring - 1) & 1, wt, kSiteQFree, kb);
            if (ok) request_q(w, it, e, slot);
          }
          advance();
        }
        if (!ok) break;
        for (int k = 0; k < item.nb; ++k, ++kb) {
          const int hb = 2 * (item.k0 + k) + (is_v ? (int)cta ^ 1 : (int)cta);
          const bool seg0 = hb < item.nh0;
          const int row0 = seg0 ? item.row0 + hb * kOwnKeys : item.row1 + (hb - item.nh0) * kOwnKeys;
          const CUtensorMap* m = seg0 ? &map_kv0 : &map_kv1;
          const uint32_t dst = sbase + PL::kOffKV + slot * PL::kSlot;
          if (!is_v) {
            // this CTA's 32 keys, all dims, once the slot's previous entry is dead
            if (ring > 0) ok = mbar_wait(&ms.slot_free[slot], (ring - 1) & 1, wt, kSiteKFree, kb);
            if (!ok) break;
            if (cta == 0) mbar_arrive_expect_tx(&ms.k_full[kb & 7], 2 * PL::kSlot);
            for (int j = 0; j < kChunks; ++j)
              tma_load_2d_pair(dst + j * kChunkBytes, m, 64 * j, row0, a_k_full + 8u * (uint32_t)(kb & 7));
          } else {
            // the peer's 32 keys, this CTA's 256 value dims, once QK^T has read the tile
            ok = mbar_wait(&ms.qk_done[kb & 7], (kb >> 3) & 1, wt, kSiteVFree, kb);
            if (!ok) break;
            if (cta == 0) mbar_arrive_expect_tx(&ms.v_full[kb & 7], 2 * 4 * kChunkBytes);
            for (int j = 0; j < 4; ++j)
              tma_load_2d_pair(dst + ((cta == 0 ? 4 : 0) + j) * kChunkBytes, m, 256 * (int)cta + 64 * j,
                               row0, a_v_full + 8u * (uint32_t)(kb & 7));
          }
          advance();
        }
      }
    }
   } else if (!kTma && (warp == kWarpK || warp == kWarpV)) {
    // ------------------------------------------------------------ "landed" relays to the leader CTA
    // The MMA warp lives in the leader CTA and can only wait on its own barriers: in the peer CTA
    // these warps forward "K rows landed" and "V rows landed".
    if (cta == 1) {
      const bool is_k = warp == kWarpK;
      const uint32_t a_peer0 = mapa(smem_u32(is_k ? &ms.k_peer[0] : &ms.v_peer[0]), 0);
      int kb = 0;
      for (int w = cid; w < n_items; w += ncl) {
        const int nb = item_of(w).nb;
        for (int k = 0; k < nb; ++k, ++kb) {
          const int s = kb & 7;
          mbar_wait(is_k ? &ms.k_full[s] : &ms.v_full[s], (kb >> 3) & 1, wt, is_k ? kSiteRelayK : kSiteRelayV, k);
          fence_proxy_async_smem();     // this CTA's cp.async writes -> the leader's MMA reads
          if (lane == 0) mbar_arrive_cluster_release(a_peer0 + 8u * (uint32_t)s);
        }
      }
    }
   } else if (!kTma && warp == kWarpValid) {
    // ------------------------------------------------------------ index-validity bits (warp kWarpValid)
    int kb = 0;
    for (int w = cid; w < n_items; w += ncl) {
      const Item item = item_of(w);
      const int32_t* idx_row = p.indices + (size_t)item.tile * p.idx_stride;
      auto load = [&](int k, int i) -> int {      // entry 32 i + lane of local block k; -1 beyond the list
        const int pos = (item.k0 + k) * kBlockKeys + 32 * i + lane;
        return pos < item.len0 ? __ldcs(idx_row + pos) : -1;
      };
      int cur[2], nxt[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) cur[i] = load(0, i);
      for (int k = 0; k < item.nb; ++k, ++kb) {
        const int s = kb & 1;
        const uint32_t ph = (kb >> 1) & 1;
#pragma unroll
        for (int i = 0; i < 2; ++i) nxt[i] = k + 1 < item.nb ? load(k + 1, i) : -1;
        uint32_t word = 0;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint32_t b = __ballot_sync(0xffffffffu, (unsigned)cur[i] < (unsigned)p.s_kv);
          if (lane == i) word = b;
        }
        if (kb >= 2) mbar_wait(&ms.valid_free[s], ph ^ 1, wt, kSiteValidFree, k);
        __syncwarp();
        if (lane < 2) ms.valid[s][lane] = word;
        __syncwarp();
        if (lane == 0) mbar_arrive(&ms.valid_ready[s]);
#pragma unroll
        for (int i = 0; i < 2; ++i) cur[i] = nxt[i];
      }
    }
   }
  } else if (warp < kWarpGather0) {
    if (!kTma) asm volatile("setmaxnreg.inc.sync.aligned.u32 176;");      // 80 x 2 + 48 + 48 x 2 + 176 = 480 = 80 x 6, as launched
    // ------------------------------------------------------------ epilogue warps
    // Bring the Q tiles in, then write out O: a warp reads the TMEM lanes of its quarter (warp % 4),
    // i.e. rows e_r of key half e_h, dims [256 e_h, +256) in 8 rounds of 32.  A round (32 rows x 64
    // bytes, 64-byte swizzle) is staged in the warp's own 2 KB slice and one lane hands the box to TMA.
    const int e_tid = (int)threadIdx.x - 32 * kWarpEpi0;
    const int e_tl = ((warp & 3) << 5) | lane, e_r = e_tl & 63, e_h = e_tl >> 6;
    const uint32_t e_lane = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t a_o_free = mapa(smem_u32(&ms.o_free), 0);
    const uint32_t a_qt_ready = mapa(smem_u32(&ms.qt_ready), 0), a_q_res = mapa(smem_u32(&ms.q_res), 0);
    const uint32_t stage_off = PL::kOffStage + (warp - kWarpEpi0) * 2048;
    uint8_t* st_row = sm + stage_off + (e_r & 31) * 64;
    const int sw = (e_r >> 1) & 3;
    // Q of item ordinal j (work item w, first ring entry n): once the previous item's QK^T are complete,
    // the resident chunks are fetched by TMA and the others moved from their slot to tensor memory
    // (chunk -> 32 columns; lane = row, duplicated in lanes 64-127)
    auto bring_q = [&](int w, int j, int n) {
      if (j > 0) mbar_wait(&ms.q_free, (j - 1) & 1, wt, kSiteQFree, j);
      if (e_tid == 0 && !wt.aborting()) {
        ms.q_res_asked = j + 1;
        const int qt = tile_of(w) * p.G + q_tok0;
        if (cta == 0) mbar_arrive_expect_tx(&ms.q_res, 2 * kQRes * kQChunkBytes);
        for (int i = 0; i < kQRes; ++i)
          tma_load_3d_pair_hint(sbase + PL::kOffQ + i * kQChunkBytes, &map_q, 64 * (kQChunksTmem + i), q_head, qt,
                                a_q_res, pol_stream);
      }
      mbar_wait(&ms.q_land, j & 1, wt, kSiteQ, j);
      __syncwarp();      // lanes leave the wait loop one by one: re-converge before .aligned ops
      tc_fence_after();
      constexpr int kPer = kQChunksTmem / kQEntries;
#pragma unroll 1
      for (int jc = 0; jc < kQChunksTmem; ++jc) {
        const uint8_t* qrow = sm + PL::kOffKV + (uint32_t)((n + jc / kPer) % kSlots) * PL::kSlot +
                              (jc % kPer) * kQChunkBytes + e_r * 128;
        uint32_t v[32];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const uint4 t = *reinterpret_cast<const uint4*>(qrow + ((u ^ (e_r & 7)) << 4));
          v[4 * u] = t.x; v[4 * u + 1] = t.y; v[4 * u + 2] = t.z; v[4 * u + 3] = t.w;
        }
        tmem_st32(tmem + e_lane + kTmemQ + 32 * jc, reinterpret_cast<const float*>(v));
      }
      tmem_wait_st();
      tc_fence_before();
      fence_proxy_async_smem();      // these reads -> the slot's next TMA write
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(a_qt_ready);
      asm volatile("bar.sync 4, 128;" ::: "memory");      // all four warps have read the slots
      if (e_tid < kQEntries) mbar_arrive(&ms.slot_free[(n + e_tid) % kSlots]);
      if (e_tid == 0) mbar_arrive(&ms.q_taken[j & 1]);
    };
    int kb0 = 0, it = 0;
    if (cid < n_items) bring_q(cid, 0, 0);
    for (int w = cid; w < n_items; w += ncl, ++it) {
      const Item item = item_of(w);
      const int kbl = kb0 + item.nb - 1;           // last block of the item
      if (w + ncl < n_items) bring_q(w + ncl, it + 1, kb0 + item.nb + kQEntries * (it + 1));
      // the row scales are published and the item's last PV has completed
      mbar_wait(&ms.epi_ready[it & 1], (it >> 1) & 1, wt, kSiteEpi, it);
      mbar_wait(&ms.pv_done[kbl & 3], (kbl >> 2) & 1, wt, kSiteEpi, item.nb);
      __syncwarp();
      tc_fence_after();
      const uint32_t ocol = tmem + e_lane + kTmemO;
      float o[32];
      // Behind the cluster's last item nothing is loaded any more, and with its PVs complete the ring is free for all of O:
      // one fence and one group of stores instead of eight rounds at the end of every launch.  (2 tokens x 64 heads, top-2048, in
      // slices 24.2 -> 21.9 us on a native cache, FP8 22.2 -> 20.1; ranges, 34 x 64 11.3 -> 10.5.)
      const bool last = w + ncl >= n_items;
      if (kSliced) {
        // a slice: unnormalised fp32 O to its slot (few slices exist, all of them in L2), a row's half per thread: in one
        // bulk copy through the ring, or directly
        float4* dst = reinterpret_cast<float4*>(p.part_o + ((size_t)w * 128 + 64 * cta + e_r) * kDV + 256 * e_h);
        const uint32_t row_off = PL::kOffKV + (64 * e_h + e_r) * 1024;
        float4* to = last ? reinterpret_cast<float4*>(sm + row_off) : dst;
        static_assert(128 * 1024 <= kSlots * PL::kSlot, "O of a slice fits into the ring");
#pragma unroll 1
        for (int cc = 0; cc < 8; ++cc) {
          tmem_ld32(ocol + cc * 32, o);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 8; ++j) to[part_unit(cc * 8 + j, e_r)] = make_float4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
        }
        tc_fence_before();
        if (last) {
          fence_proxy_async_smem();
          bulk_store_1d(dst, sbase + row_off, 1024);
          bulk_commit_group();
        }
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(a_o_free);
      } else if (last) {
        const float oscale = ms.oscale[it & 1][e_r];
        const uint32_t emask = oscale != 0.f ? 0xffffffffu : 0u;
        const int r0 = (int)cta * 64 + 32 * (warp & 1);
        const int out_head = r0 % p.h_per_q, out_tok = item.tile * p.G + r0 / p.h_per_q;
        const uint32_t all = PL::kOffKV + (warp - kWarpEpi0) * 16384;
        uint8_t* row_off = sm + all + (e_r & 31) * 64;
#pragma unroll 1
        for (int cc = 0; cc < 8; ++cc) {
          tmem_ld32(ocol + cc * 32, o);
          tmem_wait_ld();
          uint32_t w16[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const __nv_bfloat162 v2 = __floats2bfloat162_rn(o[2 * j] * oscale, o[2 * j + 1] * oscale);
            w16[j] = *reinterpret_cast<const uint32_t*>(&v2) & emask;      // rows without a key: zeros
          }
#pragma unroll
          for (int j = 0; j < 4; ++j)
            *reinterpret_cast<uint4*>(row_off + cc * 2048 + ((j ^ sw) << 4)) =
                make_uint4(w16[4 * j], w16[4 * j + 1], w16[4 * j + 2], w16[4 * j + 3]);
        }
        tc_fence_before();
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          for (int cc = 0; cc < 8; ++cc)
            tma_store_3d_hint(&map_out, sbase + all + cc * 2048, 256 * e_h + 32 * cc, out_head, out_tok, pol_stream);
          bulk_commit_group();
          mbar_arrive_cluster(a_o_free);
        }
      } else {
        const float oscale = ms.oscale[it & 1][e_r];
        const uint32_t emask = oscale != 0.f ? 0xffffffffu : 0u;
        // this warp's 32 rows of the tile = (token, head) pairs starting at row r0
        const int r0 = (int)cta * 64 + 32 * (warp & 1);
        const int out_head = r0 % p.h_per_q, out_tok = item.tile * p.G + r0 / p.h_per_q;
        // The last kHeld boxes are scaled, rounded and kept in registers, so that the next item's first PV may overwrite O
        // before they are handed over: a box's way through the warp's slice takes some 500 cycles, all eight 4000, by
        // which that PV was late.  With the gather the block's registers are redistributed for it (7 boxes; native cache,
        // 1184 tokens x 64 heads, top-2048 354 -> 343 us); the tiled forms lose more by that than they gain (items of
        // four blocks 52.5 -> 54 us) and hold the boxes for which their registers suffice: ranges 3 (1184 x 64 at 65536 100.0 -> 97.9; 4 would
        // spill), runs 2 (3 would spill).  Straight to memory from registers, a row per lane, O is free after 4000 cycles, too.
        constexpr int kHeld = kSrc == kRange ? 3 : kSrc == kRank ? 2 : 7;
        uint32_t wv[kHeld][16];
        auto pack = [&](int cc, uint32_t (&w)[16]) {
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            float x[16];
            tmem_ld16(ocol + 32 * cc + 16 * i, x);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const __nv_bfloat162 v2 = __floats2bfloat162_rn(x[2 * j] * oscale, x[2 * j + 1] * oscale);
              w[8 * i + j] = *reinterpret_cast<const uint32_t*>(&v2) & emask;      // rows without a key: zeros
            }
          }
        };
        auto put = [&](const uint32_t (&w)[16]) {      // once the slice's previous box has been read out of it
          if (lane == 0) bulk_wait_read_all();
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 4; ++j)
            *reinterpret_cast<uint4*>(st_row + ((j ^ sw) << 4)) = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
        };
        auto send = [&](int cc) {
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_3d_hint(&map_out, sbase + stage_off, 256 * e_h + 32 * cc, out_head, out_tok, pol_stream);
            bulk_commit_group();
          }
        };
#pragma unroll 1
        for (int cc = 0; cc < 7 - kHeld; ++cc) {
          pack(cc, wv[0]);
          put(wv[0]);
          send(cc);
        }
        pack(7 - kHeld, wv[0]);
        put(wv[0]);
#pragma unroll
        for (int cc = 0; cc < kHeld; ++cc) pack(8 - kHeld + cc, wv[cc]);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(a_o_free);
        send(7 - kHeld);
#pragma unroll
        for (int cc = 0; cc < kHeld; ++cc) {
          put(wv[cc]);
          send(8 - kHeld + cc);
        }
      }
      kb0 += item.nb;
    }
    if (kSliced || lane == 0) bulk_wait_all();   // boxes and rows written before the CTA retires
    tc_fence_before();
  } else if (!kTma) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
    // ------------------------------------------------------------ KV row gather (cp.async)
    // 16-byte copies written straight into the 128-byte-swizzled layout, completion reported to an mbarrier by an
    // asynchronous arrival.  Four warps fetch K rows (this CTA's 32 keys, all dims: warp pw rows [8 pw, 8 pw + 8)) as
    // soon as the slot's previous entry is dead, the other four V rows (the PEER's 32 keys, this CTA's 256
    // value dims) into the dead half of the slot as soon as the block's QK^T is complete.  (Eight warps that polled for both
    // in turn were late for either: see attn_fp8.cu.)  Entries without a valid index become zeros without a read.
    const int pw = (warp - kWarpGather0) & 3;
    const bool is_k = warp < kWarpGather0 + kGatherWarps / 2;
    const uint8_t* kvb = p.kv;
    const long long pitch = p.kv_pitch;
    const int cj = lane >> 3, cc = lane & 7;       // piece `lane` of 32: chunk cj, 16-byte unit cc
    // lane l holds the index of key 8 pw + l % 8 of the CTA's own (K) / the peer's (V) 32 keys, -1 if it has none;
    // loaded one block ahead
    const int key = kOwnKeys * ((int)cta ^ (is_k ? 0 : 1)) + 8 * pw + (lane & 7);
    auto load_idx = [&](const Item& t, int k) -> int {
      const int pos = (t.k0 + k) * kBlockKeys + key;
      return pos < t.len0 ? __ldcs(p.indices + (size_t)t.tile * p.idx_stride + pos) : -1;
    };
    Item nx = item_of(min(cid, n_items - 1));
    int idx = load_idx(nx, 0);
    int slot = 0, ring = 0, kb = 0, it = 0;        // ring entry = kSlots ring + slot
    auto advance = [&]() { if (++slot == kSlots) { slot = 0; ++ring; } };
    // the block's index, with the next block's (of the next item behind the last) on its way
    auto take_idx = [&](const Item& t, int k, int w) -> int {
      const int cur = (unsigned)idx < (unsigned)p.s_kv ? idx : -1;
      if (k + 1 < t.nb) idx = load_idx(t, k + 1);
      else if (w + ncl < n_items) idx = load_idx(nx, 0);
      return cur;
    };
    bool ok = true, go = true;                     // none of this lane's / this warp's waits has given up: then it leaves
    if (is_k) {
      for (int w = cid; go && w < n_items; w += ncl, ++it) {
        const Item t = nx;
        if (w + ncl < n_items) nx = item_of(w + ncl);
        // The item's Q entries, requested by warp 0.  Every warp goes through their slots' barriers and that of the
        // previous Q (whose bytes could, with short items, still be in flight), and Q counts as landed only when
        // all of them have: no warp is overtaken and tests a phase that is two ahead.
        if (it > 0) ok &= mbar_wait(&ms.q_taken[(it - 1) & 1], ((it - 1) >> 1) & 1, wt, kSiteQ, it);
        for (int e = 0; e < kQEntries; ++e) {
          if (ring > 0) ok &= mbar_wait(&ms.slot_free[slot], (ring - 1) & 1, wt, kSiteKFree, it);
          __syncwarp();
          if (pw == 0 && lane == 0 && ok) request_q(w, it, e, slot);
          __syncwarp();
          advance();
        }
        if (pw != 0 && lane == 0 && ok && !wt.aborting()) {
          ms.q_passed[pw] = it + 1;
          mbar_arrive(&ms.q_land);
        }
        for (int k = 0; k < t.nb; ++k, ++kb) {
          const int cur = take_idx(t, k, w);
          if (ring > 0) ok &= mbar_wait(&ms.slot_free[slot], (ring - 1) & 1, wt, kSiteKFree, k);
          const bool full = __all_sync(0xffffffffu, cur >= 0 && ok);
          const uint32_t kst = sbase + PL::kOffKV + slot * PL::kSlot + 8 * pw * 128;
          if (full) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {         // 1024 latent bytes per row: two instructions
              const int ri = __shfl_sync(0xffffffffu, cur, i >> 1);
              cp_async16(kst + (4 * (i & 1) + cj) * kChunkBytes + (i >> 1) * 128 + ((cc ^ (i >> 1)) << 4),
                         kvb + (size_t)ri * pitch + 512 * (i & 1) + 16 * lane);
            }
          } else {
            go = __all_sync(0xffffffffu, ok);
            if (!go) break;
#pragma unroll 1
            for (int i = 0; i < 16; ++i) {
              const int ri = __shfl_sync(0xffffffffu, cur, i >> 1);
              cp_async16_or_zero(kst + (4 * (i & 1) + cj) * kChunkBytes + (i >> 1) * 128 + ((cc ^ (i >> 1)) << 4),
                                 kvb + (size_t)max(ri, 0) * pitch + 512 * (i & 1) + 16 * lane, ri >= 0);
            }
          }
          if (kD == 576) {                         // 128 rope bytes: four rows in one instruction
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const int rw = 4 * i + cj, ri = __shfl_sync(0xffffffffu, cur, rw);
              cp_async16_or_zero(kst + 8 * kChunkBytes + rw * 128 + ((cc ^ rw) << 4),
                                 kvb + (size_t)max(ri, 0) * pitch + 1024 + 16 * cc, ri >= 0);
            }
          }
          cp_async_mbar_arrive_noinc(&ms.k_full[kb & 7]);
          advance();
        }
      }
    } else {
      const uint8_t* src = kvb + 512 * (int)cta + 16 * lane;
      for (int w = cid; go && w < n_items; w += ncl) {
        const Item t = nx;
        if (w + ncl < n_items) nx = item_of(w + ncl);
        for (int e = 0; e < kQEntries; ++e) advance();
        for (int k = 0; k < t.nb; ++k, ++kb) {
          const int cur = take_idx(t, k, w);
          ok &= mbar_wait(&ms.qk_done[kb & 7], (kb >> 3) & 1, wt, kSiteVFree, k);
          go = __all_sync(0xffffffffu, ok);
          if (!go) break;
          const uint32_t vst = sbase + PL::kOffKV + slot * PL::kSlot + ((cta == 0 ? 4 : 0) + cj) * kChunkBytes + 8 * pw * 128;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int ri = __shfl_sync(0xffffffffu, cur, i);
            cp_async16_or_zero(vst + i * 128 + ((cc ^ i) << 4), src + (size_t)max(ri, 0) * pitch, ri >= 0);
          }
          cp_async_mbar_arrive_noinc(&ms.v_full[kb & 7]);
          advance();
        }
      }
    }
  }

  // tear-down: nobody may still be reading TMEM of either CTA when it is released
  __syncthreads();
  if (ms.left != 0) {
    cp_async_wait_all();
    if (threadIdx.x == 0) {
      const unsigned long long t0 = globaltimer_ns();
      const uint32_t n = ms.q_asked, items = (n + kQEntries - 1) / kQEntries;
      if (n != 0) {               // the last Q requested: with the arrivals that are missing it counts as landed when it has
        for (uint32_t i = n; i < kQEntries * items; ++i) mbar_arrive(&ms.q_land);
        for (int i = 1; !kTma && i < kGatherWarps / 2; ++i)
          if (ms.q_passed[i] < items) mbar_arrive(&ms.q_land);
        mbar_drain(&ms.q_land, (items - 1) & 1);
      }
      if (cta == 0 && ms.q_res_asked != 0) mbar_drain(&ms.q_res, (ms.q_res_asked - 1) & 1);      // both CTAs' bytes
      for (int i = 0; i < 2; ++i) {      // block 2 (n - 1) + i was the warp's last
        const uint32_t kb = 2 * (ms.qk_end[i] - 1) + i;
        if (ms.qk_end[i] != 0) mbar_drain(&ms.qk_done[kb & 7], (kb >> 3) & 1);
      }
      if (ms.pv_end != 0) mbar_drain(&ms.pv_done[(ms.pv_end - 1) & 3], ((ms.pv_end - 1) >> 2) & 1);
      // K and V by TMA: the leader's barriers count the bytes of both CTAs, of which one may have asked for none.  No load
      // takes a tenth of this.
      while (kTma && globaltimer_ns() - t0 < 100000ull) {}
    }
  }
  __syncwarp();
  cluster_sync_all();
  if (warp == kWarpMma) tmem_dealloc_pair(tmem, kTmemCols);
  if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&g_status[3], 1);
  if (threadIdx.x == 0) wt.report(g_status, p.epoch);
}

// how many 2-CTA clusters of this kernel device `dev` (the current one) can hold at once
template <int kD, Source kSrc>
static int max_clusters(int dev) {
  static thread_local int cached_dev = -1, cached = 0;
  if (dev == cached_dev) return cached;
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int n = sms / 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(sms, 1, 1); cfg.blockDim = dim3(threads_of(kSrc), 1, 1); cfg.dynamicSmemBytes = Plan<kD>::kSmem;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = 2; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
  cfg.attrs = &at; cfg.numAttrs = 1;
  int q = 0;
  if (ensure_smem<mla_bf16_kernel<kD, kSrc, false, false>>(dev, Plan<kD>::kSmem) &&
      cudaOccupancyMaxActiveClusters(&q, mla_bf16_kernel<kD, kSrc, false, false>, &cfg) == cudaSuccess && q > 0)
    n = q;
  cudaGetLastError();
  cached_dev = dev; cached = n;
  return n;
}

// Tensor maps of q and out, addressed as (dim, head, token): row r of a tile is (token r / h, head
// r % h), which covers the dense packed layout and the in-place layout with padded head slots
// alike.  Strides in ELEMENTS, 0 = dense.  q in boxes of 64 dims x 64 rows, out in boxes of 32 dims x
// 32 rows (64 bytes wide, 64-byte swizzle).
struct QOutArgs {
  const void* q; void* out;
  int d, ng, h;
  int64_t q_row_stride, q_token_stride, q_head_stride, out_token_stride, out_head_stride;
  int64_t out_hs() const { return out_head_stride ? out_head_stride : kDV; }
  int64_t out_ts() const { return out_token_stride ? out_token_stride : h * out_hs(); }
};
inline bool make_q_out_maps(const QOutArgs& a, CUtensorMap* mq, CUtensorMap* mout) {
  const auto BF = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const uint64_t q_hs = (uint64_t)(a.q_head_stride ? a.q_head_stride : a.q_row_stride) * 2;
  const uint64_t q_ts = a.q_token_stride ? (uint64_t)a.q_token_stride * 2 : (uint64_t)a.h * q_hs;
  const uint64_t tokens = (uint64_t)a.ng * (128 / a.h);
  const uint32_t qb_h = (uint32_t)min(a.h, 64), ob_h = (uint32_t)min(a.h, 32);
  return make_map_3d(mq, a.q, BF, (uint64_t)a.d, (uint64_t)a.h, tokens, q_hs, q_ts, 64, qb_h, 64 / qb_h) &&
         make_map_3d(mout, a.out, BF, kDV, (uint64_t)a.h, tokens, (uint64_t)a.out_hs() * 2, (uint64_t)a.out_ts() * 2,
                     32, ob_h, 32 / ob_h, CU_TENSOR_MAP_SWIZZLE_64B);
}
// map of KV rows for the tiled loads: boxes of 64 dims x 32 rows; pitch in ELEMENTS
inline bool make_kv_map(CUtensorMap* m, const void* kv, int d, int64_t rows, int64_t pitch) {
  return make_map_2d(m, kv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (uint64_t)d, (uint64_t)rows, (uint64_t)pitch * 2, 64, kOwnKeys);
}

// Launch over p.ng tiles of p.nsplit slices (a merge has to follow when they are sliced).
template <int kD, Source kSrc, bool kSliced, bool kOrdered = false>
static int launch(const CUtensorMap& mq, const CUtensorMap& m0, const CUtensorMap& m1, const CUtensorMap& mout,
                  const Params& p, cudaStream_t stream) {
  const int dev = current_device();
  if (!ensure_smem<mla_bf16_kernel<kD, kSrc, kSliced, kOrdered>>(dev, Plan<kD>::kSmem)) return LITEDSA_ERR_CUDA;
  const int items = kSliced ? p.ng * p.nsplit : p.ng;
  return launch_pdl(mla_bf16_kernel<kD, kSrc, kSliced, kOrdered>, dim3(2 * min(items, max_clusters<kD, kSrc>(dev))),
                    threads_of(kSrc), Plan<kD>::kSmem, stream, mq, m0, m1, mout, p);
}

}  // namespace mla16
}  // namespace lt
