// Masked FP8 MLA prefill over a per-tile union list (sm_100a, tcgen05 + TMEM + TMA).
//
// What it computes is fixed by the reference operator masked_mla_fp8
// (kernels/b200/dsa/litedsa.cu:77-135, kernel
// kernels/b200/dsa/litedsa_attention_sm100.cuh:1832-2479): for every 128-row tile
// (G = 128 / h_per_q adjacent tokens x h_per_q heads), S = Q8 K8^T over the tile's union
// of KV rows, a per-row validity/membership mask, base-2 online softmax in blocks of
// 128 keys whose running max only moves when some row of a 32-row group overshoots it
// by more than 6, P quantised to e4m3 after a x7 pre-scale, O += P8 V8 (V = the first
// 512 bytes of the same KV rows), out = bf16(O * out_scale / l), lse, max_logits.
// Those numerics are reproduced exactly so the two implementations agree to rounding.
//
// How it is organised here (written from scratch, raw PTX, no CuTe):
//   * persistent: one cluster of 2 CTAs per SM pair walks work items cid, cid + #clusters, ...
//     (an item is a tile, or one of nsplit slices of a tile's key blocks); each CTA owns 64 query
//     rows.  Both GEMMs are single tcgen05 cta_group::2 instructions spanning the pair: QK^T
//     splits the 128 keys of a block across the CTAs (N split), PV splits the 512 value dims.
//   * a block's K tile BECOMES its V tile.  CTA c gathers the 576-byte rows of its own 64 keys
//     (column chunks 0-3 of 128 dims, rope chunk).  PV wants, per CTA, 256 value dims of all 128
//     keys: for its own keys they are already there (chunks 2c, 2c + 1), and once QK^T has read
//     the tile the other two chunks are dead -- the peer keys' rows of this CTA's 256 dims are
//     gathered into them.  Both CTAs then hold keys 0-63 in chunks 0-1 and keys 64-127 in chunks
//     2-3, which is what one pair-wide descriptor needs.  Against separate V tiles: 52 instead of
//     68 KB fetched per block and CTA, and 36 instead of 68 KB of shared memory per block, i.e.
//     four blocks in flight instead of two.
//   * 32 warps per CTA:
//       warps 0-15  softmax, two groups of eight warps on alternate key blocks (one TMEM lane and
//                   32 S columns per thread: short chains, and eight warps per scheduler to hide
//                   them);
//       warps 16-23 KV row gather with 16-byte cp.async copies written straight into the
//                   128-byte-swizzled tile layout: K rows (16-19), the peer's value halves (20-23);
//       warp 24     QK^T issue (leader CTA; whole warp polls, one elected lane issues);
//       warps 25-26 in the peer CTA: relay "K / V landed" to the leader's barriers; in the leader
//                   warp 25 issues PV;
//       warp 27     index-validity bits;
//       warps 28-31 Q tiles in (TMA, or bf16 rows quantised on the way) and tile epilogue: O out
//                   of TMEM, x out_scale / l, bf16, staged per warp and written with TMA tile
//                   stores while the softmax warps already work on the next item.
//   * Q and K tiles are four 128-byte-swizzled column chunks per 64 rows plus a compact
//     64-byte-swizzled chunk for the 64 rope bytes.
//   * the 512 latent dims of every Q tile are moved from shared memory into TENSOR MEMORY once
//     per item (by the epilogue warps) and the QK^T MMAs read them from there (A operand in
//     TMEM); only the rope chunk of Q stays in shared memory.
//   * completion is tracked with mbarriers only; every wait is bounded (common.cuh) and
//     reports through a status word instead of trapping.
//   * no TMA multicast of any kind; the pair is signalled with two plain commits.
#include "common.cuh"
#include "tensor_map.cuh"


namespace lt {

constexpr int kSoftmaxWarps = 16, kProducerWarps = 8;
constexpr int kWarpGather0 = 16, kWarpMma = 24, kWarpRelayK = 25, kWarpRelayV = 26, kWarpValid = 27, kWarpEpi0 = 28;
constexpr int kEpiWarps = 4;
constexpr int kAttnThreads = 1024;
constexpr int kBlockKeys = 128;                      // keys per softmax block (whole pair)
constexpr int kDQK = 576, kDV = 512;
constexpr int kChunkBytes = 64 * 128;                // 64 rows x 128 B (dims 128j .. 128j+127)
constexpr int kRopeChunkBytes = 64 * 64;             // 64 rows x 64 B (dims 512 .. 575), 64-byte swizzle
constexpr uint32_t kQLatent = 4 * kChunkBytes;       // 32768 (per CTA)
constexpr uint32_t kStageKV = kQLatent + kRopeChunkBytes;        // 64 keys x 576 B
constexpr uint32_t kPBytes = 64 * 128;               // 64 rows x 128 keys e4m3
constexpr uint32_t kMiscBytes = 10240;
constexpr uint32_t kStageBytes = 4 * 4096;           // staged epilogue: one 4 KB slice per epilogue warp
constexpr int kFillBatch = 6;                        // bf16 q: 32-byte loads in flight per thread while filling a Q tile
constexpr int kSlots = 5;                            // ring of 36 KB slots

// Shared-memory plan.  A ring of five slots carries, in order, each item's Q tile and its K tiles:
// Q only passes through on its way to tensor memory (latent dims) and to a fixed 4 KB buffer (rope
// chunk), so a landing area of its own would idle 19 blocks out of 20.  The entry number of running
// block kb of item ordinal it is kb + it + 1, that of the item's Q (its first block's kb) + it.
// What bounds the kernel is latency: a slot is held for a gather, a QK^T, a softmax chain and a PV,
// about 9000 cycles, so blocks in flight are the throughput.
struct Plan {
  static constexpr uint32_t kOffKV = 0;
  static constexpr uint32_t kOffRope = kOffKV + kSlots * kStageKV;
  static constexpr uint32_t kOffP = kOffRope + kRopeChunkBytes;
  static constexpr uint32_t kOffStage = kOffP + 2 * kPBytes;
  static constexpr uint32_t kOffMisc = kOffStage + kStageBytes;
  static constexpr uint32_t kSmem = kOffMisc + kMiscBytes + 1024;   // + alignment slack
  static_assert(kStageKV % 1024 == 0 && kOffP % 1024 == 0, "swizzled tiles need 1024-byte alignment");
  static_assert(kSmem <= 232448, "shared-memory plan exceeds the 227 KB per-CTA limit");
};

constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kTmemO = 0;                        // 256 columns: O (64 rows x 512 dims per CTA)
constexpr uint32_t kTmemS0 = 256, kTmemS1 = 320;      // 64 columns each: S double buffer
constexpr uint32_t kTmemQ = 384;                      // 128 columns: the 512 latent dims of Q (e4m3, 4 per column)

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr float kPScaleLog2 = 2.8073549220576042f;    // log2(7)
constexpr float kPScaleLn = kFp8LseOffset;            // ln(7)
constexpr float kMInit = -1e30f;
constexpr float kRescaleThreshold = 6.0f;

struct Misc {
  // in the leader CTA only: k_peer / v_peer (peer's K / V rows landed), s_free / p_ready (softmax
  // warps of both CTAs)
  uint64_t k_peer[8], v_peer[8], s_free[2], p_ready[2];
  // in every CTA, indexed by the running block number modulo 8 (pv_done: modulo 4): with five
  // slots everybody has looked at block kb's barriers before block kb + 8 can touch them
  uint64_t k_land[8], v_land[8], qk_done[8], pv_done[4];
  uint64_t slot_free[kSlots];       // the slot's entry is dead: block through its PV, or Q moved on
  uint64_t valid_ready[2], valid_free[2];
  uint64_t m_pub[2];                // running max of block k published by softmax group k%2
  uint64_t q_land;                  // every CTA: this CTA's Q tile has landed in its slot (e4m3 q);
                                    // its slot is free for the epilogue warps to fill (bf16 q)
  uint64_t q_taken;                 // every CTA: the item's Q has been moved out of its slot
  uint64_t qt_ready;                // leader CTA: Q's latent part is in tensor memory in both CTAs
  uint64_t q_free;                  // all QK^T of the current item are complete (Q reusable)
  uint64_t o_free;                  // leader CTA: the item's O has been read out of TMEM
  uint64_t epi_ready[2];            // the item's row scales are published (softmax warps), by parity of
                                    // the item ordinal: with items of one or two blocks the next item's can
                                    // be complete before the epilogue has looked at this one's
  uint32_t valid[2][4];             // 128 validity bits per stage
  uint32_t tmem_base;
  // for the tear-down of a launch that gives up: a wait of this block has; items whose Q has been requested from TMA
  // and at whose q_land each K warp has arrived; leader: blocks whose QK^T and PV have been issued
  uint32_t left, q_asked, q_passed[kProducerWarps / 2], qk_end, pv_end;
  float xbuf[2][2][2][128];         // [group][parity][column half][lane]: row-max exchange
  float mshare[2][128];             // [group][lane]: running max after the group's latest block
  float fin_l[512];                 // end of item: row sums per thread ...
  float fin_rm[128], fin_m[128];    // ... true maxima, last running max per (group, row)
  float oscale[2][64];              // [item parity][row]: out_scale / l, 0 for rows without a key
};
static_assert(sizeof(Misc) <= kMiscBytes, "Misc too large");

constexpr int kMaxOutputs = 8;
// tensor maps of the output destinations: this GPU's buffer and, in a sharded run, the
// peers' gathered buffers (peer-mapped addresses written with plain TMA tile stores)
struct OutMaps { CUtensorMap m[kMaxOutputs]; };

struct AttnParams {
  const uint32_t* memb;      // [ng, G, cap/32], or null when len_per_q replaces it
  const int32_t* len_per_q;  // [ng, G] per-token causal prefix bound on the union ranks, or null
  const float* sink;         // [128] per packed row (natural-log units), or null
  int q_group_div;           // this many consecutive tiles share one Q tile (KV split)
  const uint8_t* kv;         // [s_kv, kv_pitch] e4m3 rows (576 bytes used)
  long long kv_pitch;        // bytes between KV rows
  const int32_t* indices;    // [ng, idx_stride]
  const int32_t* counts;     // [ng] or null
  float* lse;                // [ng, 128]
  float* max_logits;         // [ng, 128] or null
  int ng, s_kv, cap, h_per_q, G;
  int n_out;                 // destinations of every output box (1 + peers that hold a copy)
  long long idx_stride;
  float scale_log2, out_scale;
  int epoch;                          // this launch's epoch for the bounded waits
  uint32_t wait_limit;       // of one wait, in ticks (BlockWaiter)
  // bf16 queries (dense packed layout), quantised to e4m3 on their way in: code = e4m3(q * q_inv);
  // null: q arrives as e4m3 through map_q / map_q_rope
  const uint4* q_bf16;
  float q_inv;
  // KV split inside the launch: nsplit > 1 slices per tile, each leaving its unnormalised O (fp32
  // [ng * nsplit, 128, 512]) and (running max, row sum) for merge_slices_kernel
  int nsplit;
  float* part_o;
  float2* part_ml;
};

// four e4m3 codes of two packed bf16 pairs, x inv (saturating): the arithmetic of quantize_e4m3
__device__ __forceinline__ uint32_t e4m3x4_of_bf16(uint32_t lo, uint32_t hi, float inv) {
  float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&lo));
  float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&hi));
  a.x *= inv; a.y *= inv; b.x *= inv; b.y *= inv;
  return (uint32_t)__nv_cvt_float2_to_fp8x2(a, __NV_SATFINITE, __NV_E4M3) |
         ((uint32_t)__nv_cvt_float2_to_fp8x2(b, __NV_SATFINITE, __NV_E4M3) << 16);
}

// One work item: nb blocks of a tile; ranks >= lim are masked.  A slice behind the first opens
// with the tile's block 0 (lead = 1), of which only the row maxima count: its running max then
// starts where the unsliced tile's does, and as long as that has not moved after block 0 its P are rounded
// to e4m3 relative to the same value.  Where it has, a 32-row group's P of the later slices differ from the
// unsliced tile's by their rounding (about 1 % of the output where every group is affected; the error
// against the exact result is the same).
template <bool kSliced>
struct ItemT {
  int tile, k0, nb, lim, lead;
  // the tile's block that local block k is, and whether only its maxima count
  __device__ __forceinline__ int block(int k) const { return !kSliced ? k : (k < lead ? 0 : k0 + k - lead); }
  __device__ __forceinline__ bool leads(int k) const { return kSliced && k < lead; }
};

// wait sites reported in the status word (kSiteAlign: the shared-memory base is not where the plan needs it)
enum { kSiteQ = 1, kSiteKLand, kSiteQkDone, kSitePvDone,
       kSiteSFree, kSitePReady, kSiteValidReady, kSiteValidFree, kSiteKFree,
       kSiteVFree, kSitePFree, kSiteEpi, kSiteRelayK, kSiteRelayV, kSiteMPub, kSiteQFree, kSiteOFree, kSiteSelfTest, kSiteAlign };

// status block of the FP8 attention kernels (layout: see Waiter in common.cuh)
__device__ int g_attn_status[8];

// kSliced: p.nsplit > 1 (the unsliced kernel carries none of the slices' block arithmetic)
template <bool kSliced>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kAttnThreads, 1)
masked_mla_fp8_kernel(const __grid_constant__ CUtensorMap map_q,
                      const __grid_constant__ CUtensorMap map_q_rope,
                      const __grid_constant__ OutMaps omaps, const AttnParams p) {
  using PL = Plan;
  using Item = ItemT<kSliced>;
  constexpr uint32_t kOffRope = PL::kOffRope, kOffKV = PL::kOffKV, kOffP = PL::kOffP, kOffMisc = PL::kOffMisc, kOffStage = PL::kOffStage;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sbase = (raw + 1023u) & ~1023u;       // 128B-swizzle tiles need 1024-byte alignment
  uint8_t* sm = smem_raw + (sbase - raw);
  Misc& ms = *reinterpret_cast<Misc*>(sm + kOffMisc);
  const BlockWaiter wt{&ms.left, p.wait_limit};

  // Persistent: each cluster walks items cid, cid + #clusters, ...  Every role runs the same
  // item loop; stages, buffers and barrier phases are indexed by the cluster-wide running
  // block number kb, so the next item's Q / K / V loads and first QK^T overlap the previous
  // item's last softmax blocks and its epilogue.
  const uint32_t cta = cluster_ctarank();
  const int cid = blockIdx.x >> 1, ncl = gridDim.x >> 1;
  const int n_items = kSliced ? p.ng * p.nsplit : p.ng;
  // broadcast so the compiler knows the role index is warp-uniform
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  auto item_of = [&](int w) -> Item {
    Item t;
    t.tile = kSliced ? w / p.nsplit : w;
    // live union entries of the tile; with per-token prefix bounds the block loop runs to the LAST
    // token's bound (litedsa_attention_sm100.cuh:1846-1851)
    const int c = p.len_per_q ? p.len_per_q[(size_t)t.tile * p.G + (p.G - 1)]
                              : (p.counts ? p.counts[t.tile] : p.cap);
    t.lim = min(max(c, 0), p.cap);
    t.k0 = t.lead = 0;
    t.nb = max((t.lim + kBlockKeys - 1) / kBlockKeys, 1);
    if (kSliced) {            // slice `part`; an empty slice runs one fully masked block
      const int part = w - t.tile * p.nsplit, nbt = t.nb;
      const int k1 = (part + 1) * nbt / p.nsplit;
      t.k0 = part * nbt / p.nsplit;
      t.lead = part > 0 ? 1 : 0;
      t.nb = max(k1 - t.k0, 1) + t.lead;
      t.lim = min(t.lim, k1 * kBlockKeys);
    }
    return t;
  };

  if (threadIdx.x == 0) {
    mbar_init(&ms.q_land, kProducerWarps / 2);              // the K warps
    ms.left = ms.q_asked = ms.qk_end = ms.pv_end = 0;
    for (int i = 0; i < kProducerWarps / 2; ++i) ms.q_passed[i] = 0;
    mbar_init(&ms.q_taken, 1);
    mbar_init(&ms.qt_ready, 2 * kEpiWarps);
    mbar_init(&ms.q_free, 1);
    mbar_init(&ms.o_free, 2 * kEpiWarps);
    for (int i = 0; i < 8; ++i) {
      mbar_init(&ms.k_peer[i], 1);
      mbar_init(&ms.v_peer[i], 1);
      mbar_init(&ms.k_land[i], kProducerWarps / 2 * 32);    // one async arrival per gather thread
      mbar_init(&ms.v_land[i], kProducerWarps / 2 * 32);
      mbar_init(&ms.qk_done[i], 1);
    }
    for (int i = 0; i < 4; ++i) mbar_init(&ms.pv_done[i], 1);
    for (int i = 0; i < kSlots; ++i) mbar_init(&ms.slot_free[i], 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&ms.s_free[i], 16);        // 8 warps of one softmax group x 2 CTAs
      mbar_init(&ms.p_ready[i], 16);
      mbar_init(&ms.valid_ready[i], 1);
      mbar_init(&ms.valid_free[i], 8);
      mbar_init(&ms.m_pub[i], 8);
      mbar_init(&ms.epi_ready[i], kSoftmaxWarps);
    }
    fence_mbar_init();
    if (p.q_bf16 == nullptr) {
      tma_prefetch_desc(&map_q);
      tma_prefetch_desc(&map_q_rope);
    }
    if (!kSliced)
      for (int d = 0; d < p.n_out; ++d) tma_prefetch_desc(&omaps.m[d]);
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
  const uint32_t tmem = ms.tmem_base;
  pdl_trigger();
  pdl_wait();

  // Registers: the block is launched with 64 per thread (8 warpgroups, 512 in sum); the softmax
  // warps need more for their 32 scores, the epilogue for its 32 + 16 outputs, the others less:
  // 80 x 4 + 40 x 2 + 40 + 72 = 512.  (With 64 everywhere a handful of values spilled, and with
  // nearly all of L1 used as shared memory a spill is a round trip to L2.)
  if (warp < kSoftmaxWarps) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 80;");
    // ------------------------------------------------------------ softmax
    // Two groups of eight warps work on alternate key blocks (group g: blocks with kb % 2 == g),
    // so two blocks are in flight and the latencies of one chain (TMEM load, exchanges,
    // fences) hide behind the other.  Within a group, thread = (TMEM lane tl, column half cs):
    // tile row r = tl % 64, keys [64 h + 32 cs, +32) of the block with h = tl / 64.  (64 columns
    // per thread in four warps made one block's chain 2.4 us, i.e. the kernel's pace.)  The only
    // state that crosses groups is the running max m, handed over through shared memory right
    // after each block's row maxima are known; the row sum l is kept per thread relative to the m
    // of the group's latest block and merged at the end of the item.
    const int g = warp >> 3;                      // softmax group = block parity it serves
    const int cs = (warp >> 2) & 1;
    const int tl = ((warp & 3) << 5) | lane;
    const int r = tl & 63, h = tl >> 6;
    const int row = (int)cta * 64 + r;            // row of the 128-row tile
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const int capw = p.cap >> 5;
    const float c = p.scale_log2;
    const uint64_t c2 = pack2(c, c);
    const uint32_t a_s_free = mapa(smem_u32(&ms.s_free[g]), 0);
    const uint32_t a_p_ready = mapa(smem_u32(&ms.p_ready[g]), 0);
    const uint32_t scol = tmem + lane_base + (g ? kTmemS1 : kTmemS0) + 32 * cs;
    const int key0 = 64 * h + 32 * cs;            // first of this thread's keys within a block
    int kb0 = 0, it = 0;

    for (int w = cid; w < n_items; w += ncl) {
      const Item item = item_of(w);
      const int nb = item.nb;
      const size_t trow = (size_t)item.tile * p.G + row / p.h_per_q;     // (tile, token) of this row
      const uint32_t* mrow = p.memb ? p.memb + trow * capw + (key0 >> 5) : nullptr;
      // per-token causal prefix: this row may attend union ranks < row_bound
      const int row_bound = p.len_per_q ? __ldcg(p.len_per_q + trow) : 0x7fffffff;
      float m_mine = kMInit;      // the running max my row sum is relative to
      float li = 0.f, real_m = -INFINITY;
      const int k_first = (g - kb0) & 1;          // first local block with (kb0 + k) % 2 == g
      uint32_t mk = ~0u;
      if (mrow && k_first < nb) mk = __ldcs(mrow + (size_t)item.block(k_first) * 4);

      for (int k = k_first; k < nb; k += 2) {
        const int kb = kb0 + k;
        const uint32_t ph = (kb >> 1) & 1;
        uint32_t mk_next = mk;
        if (mrow && k + 2 < nb) mk_next = __ldcs(mrow + (size_t)item.block(k + 2) * 4);

        mbar_wait(&ms.qk_done[kb & 7], (kb >> 3) & 1, wt, kSiteQkDone, k);
        __syncwarp();      // lanes leave the wait loop one by one: re-converge before .aligned ops
        tc_fence_after();
        float sv[32];
        tmem_ld32(scol, sv);
        tmem_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(a_s_free);

        mbar_wait(&ms.valid_ready[g], ph, wt, kSiteValidReady, k);
        uint32_t vm = ms.valid[g][key0 >> 5] & mk;
        if (p.len_per_q) {     // ranks of my 32 columns
          const int n = min(max(row_bound - (item.block(k) * kBlockKeys + key0), 0), 32);
          vm &= n >= 32 ? ~0u : ((1u << n) - 1u);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&ms.valid_free[g]);
        mk = mk_next;

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
        float (*xb)[128] = ms.xbuf[g][ph];
        xb[cs][tl] = cur;
        if (g == 0) asm volatile("bar.sync 1, 256;" ::: "memory");
        else asm volatile("bar.sync 2, 256;" ::: "memory");
        cur = fmaxf(fmaxf(xb[0][r], xb[1][r]), fmaxf(xb[0][r + 64], xb[1][r + 64]));
        if (!item.leads(k)) real_m = fmaxf(real_m, cur);
        // running max after block k-1 of this item comes from the other group
        float m_prev = kMInit;
        if (k > 0) {
          mbar_wait(&ms.m_pub[g ^ 1], ((kb - 1) >> 1) & 1, wt, kSiteMPub, k);
          m_prev = ms.mshare[g ^ 1][tl];
        }
        const bool rescale = __any_sync(0xffffffffu, cur - m_prev > kRescaleThreshold);
        const float new_m = rescale ? fmaxf(cur, m_prev) : m_prev;
        if (cs == 0) ms.mshare[g][tl] = new_m;
        __syncwarp();
        if (lane == 0) mbar_arrive(&ms.m_pub[g]);
        li *= fast_exp2(m_mine - new_m);
        m_mine = new_m;

        if (item.leads(k)) {
#pragma unroll
          for (int j = 0; j < 32; ++j) sv[j] = -INFINITY;      // only the maxima of this block count
        }
        const float nm = -new_m + kPScaleLog2;
        const uint64_t nm2 = pack2(nm, nm);
        uint32_t pk[8];
        uint64_t l0 = 0, l1 = 0;      // two pairs of partial sums
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          float2 d0 = unpack2(fma2(pack2(sv[j], sv[j + 1]), c2, nm2));
          float2 d1 = unpack2(fma2(pack2(sv[j + 2], sv[j + 3]), c2, nm2));
          d0.x = fast_exp2(d0.x);
          d0.y = fast_exp2(d0.y);
          d1.x = fast_exp2(d1.x);
          d1.y = fast_exp2(d1.y);
          l0 = add2(l0, pack2(d0.x, d0.y));
          l1 = add2(l1, pack2(d1.x, d1.y));
          const uint32_t lo = __nv_cvt_float2_to_fp8x2(d0, __NV_SATFINITE, __NV_E4M3);
          const uint32_t hi = __nv_cvt_float2_to_fp8x2(d1, __NV_SATFINITE, __NV_E4M3);
          pk[j >> 2] = lo | (hi << 16);
        }
        const float2 ls = unpack2(add2(l0, l1));
        li += ls.x + ls.y;
        // the P buffer was last read by the PV of block kb-2
        if (kb >= 2) mbar_wait(&ms.pv_done[(kb - 2) & 3], ((kb - 2) >> 2) & 1, wt, kSitePFree, k);
        uint8_t* pdst = sm + kOffP + g * kPBytes + (4 * h + 2 * cs) * 1024 + r * 16;
        *reinterpret_cast<uint4*>(pdst) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        *reinterpret_cast<uint4*>(pdst + 1024) = make_uint4(pk[4], pk[5], pk[6], pk[7]);

        if (rescale && k > 0) {
          // O holds blocks [0, k) relative to m_prev: bring it to new_m once PV(k-1) is complete
          // (each thread of the pair serving a TMEM lane takes half of the lane's columns)
          mbar_wait(&ms.pv_done[(kb - 1) & 3], ((kb - 1) >> 2) & 1, wt, kSitePvDone, k);
          __syncwarp();      // lanes leave the wait loop one by one: re-converge before .aligned ops
          tc_fence_after();
          const float f = fast_exp2(m_prev - new_m);
          float o[32];
#pragma unroll 1
          for (int cc = 0; cc < 4; ++cc) {
            const uint32_t ocol = tmem + lane_base + kTmemO + cs * 128 + cc * 32;
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

      // end of item: merge the row sums (each relative to its own group's latest running max)
      // (the previous item's sums must have been read: every warp has arrived on its epi_ready)
      if (it > 0) mbar_wait(&ms.epi_ready[(it - 1) & 1], ((it - 1) >> 1) & 1, wt, kSiteEpi, it);
      ms.fin_l[(g * 2 + cs) * 128 + tl] = li;
      if (cs == 0 && h == 0) {
        ms.fin_rm[g * 64 + r] = real_m;
        ms.fin_m[g * 64 + r] = m_mine;
      }
      asm volatile("bar.sync 3, 512;" ::: "memory");
      if (g == 0 && cs == 0 && h == 0) {
        const int last_g = (kb0 + nb - 1) & 1;      // group of the item's last block
        float m = ms.fin_m[last_g * 64 + r];       // running max after the last block
        float lsum = 0.f;
        real_m = -INFINITY;
        // fixed summation order (even local blocks first, whichever group served them), so an
        // item's result does not depend on the blocks its cluster processed before
        const int g_even = kb0 & 1;
#pragma unroll
        for (int gi = 0; gi < 2; ++gi) {
          const int gg = gi ^ g_even;
          const float f = fast_exp2(ms.fin_m[gg * 64 + r] - m);
#pragma unroll
          for (int hc = 0; hc < 4; ++hc)
            lsum += ms.fin_l[(gg * 2 + (hc & 1)) * 128 + (hc >> 1) * 64 + r] * f;
          real_m = fmaxf(real_m, ms.fin_rm[gg * 64 + r]);
        }
        li = lsum;
        if (real_m == -INFINITY) { li = 0.f; m = -INFINITY; }
        if (kSliced) {
          p.part_ml[(size_t)w * 128 + row] = make_float2(m, li);
        } else {
          const size_t grow = (size_t)item.tile * 128 + row;
          float l = __logf(li) - kPScaleLn + m * kLn2;
          if (!(li > 0.f)) l = INFINITY;
          p.lse[grow] = l;
          if (p.max_logits) p.max_logits[grow] = real_m * kLn2;
          // the epilogue warps need 1 / l per row; the sink joins the OUTPUT normaliser only (in l's
          // units: x 7, relative to m)
          float denom = li;
          if (p.sink != nullptr && li > 0.f) denom += fast_exp2(__ldcg(p.sink + row) * kLog2e - m + kPScaleLog2);
          ms.oscale[it & 1][r] = (li > 0.f) ? __fdividef(p.out_scale, denom) : 0.f;
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&ms.epi_ready[it & 1]);
      kb0 += nb;
      ++it;
    }
  } else if (warp < kWarpGather0 + kProducerWarps) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    // ------------------------------------------------------------ KV row gather (cp.async)
    // The union rows are fetched with 16-byte cp.async copies issued by all 256 threads of
    // these eight warps: fire-and-forget, any number of blocks in flight, destination written
    // directly in the 128-byte-swizzled tile layout, completion reported to an mbarrier by an
    // asynchronous arrival.  (These copies alone reach 17-20 TB/s from L2; TMA gather4 takes one request
    // of 512 bytes per ~8.5 ns and SM, half of that.)
    // Four warps fetch K rows (this CTA's 64 keys, all 576 bytes: warp pw rows [16 pw, 16 pw + 16), 18 copies
    // per lane) as soon as the slot's previous entry is dead, the other four V rows (the PEER's 64 keys,
    // this CTA's 256 value bytes, eight copies per lane) into the dead half of the slot as soon as the block's QK^T
    // is complete.  (Eight warps that polled for both in turn noticed a free slot 1500 cycles and a finished QK^T
    // 1200 cycles late, out of the 11400 that a slot was held for; five slots make that the kernel's
    // pace.)  Entries without a valid index become zeros without a read: all of them read from row 0, the padded
    // blocks of all SMs met at one L2 slice (1.2 instead of 18 TB/s).
    const int pw = (warp - kWarpGather0) & 3;
    const uint8_t* kvb = p.kv;
    const long long pitch = p.kv_pitch;
    // lane l holds the index of key 16 pw + l % 16 of the CTA's own (K) / the peer's (V) 64 keys, -1 if it is out of
    // range; a block's are loaded a block ahead, so that nothing waits for a cold line
    const bool is_k = warp < kWarpGather0 + kProducerWarps / 2;
    const int key = (64 * (int)cta + 16 * pw + (lane & 15)) ^ (is_k ? 0 : 64);
    auto load_idx = [&](const Item& t, int k) -> int {
      return __ldcs(p.indices + (size_t)t.tile * p.idx_stride + (size_t)t.block(k) * kBlockKeys + key);
    };
    Item nx = item_of(min(cid, n_items - 1));
    int idx = load_idx(nx, 0);
    int slot = 0, ring = 0, kb = 0, it = 0;        // entry = 5 ring + slot
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
      const uint64_t pol_stream = l2_policy_evict_first();
      const int cj = lane >> 3, cc = lane & 7;     // latent piece `lane`: chunk cj, 16-byte slot cc
      for (int w = cid; go && w < n_items; w += ncl, ++it) {
        const Item t = nx;
        if (w + ncl < n_items) nx = item_of(w + ncl);
        // The item's Q entry, in front of its K entries.  Every warp goes through its slot's barrier and that of
        // the previous Q (whose bytes could, with short items, still be in flight), and it counts as landed
        // only when all of them have: no warp is overtaken and tests a phase that is two ahead.
        if (it > 0) ok &= mbar_wait(&ms.q_taken, (it - 1) & 1, wt, kSiteQ, it);
        if (ring > 0) ok &= mbar_wait(&ms.slot_free[slot], (ring - 1) & 1, wt, kSiteKFree, it);
        __syncwarp();
        // (nothing behind a wait of any warp that gave up: the Q before could still be in flight)
        if (lane == 0 && ok && !wt.aborting()) {
          ms.q_passed[pw] = it + 1;
          if (pw != 0 || p.q_bf16 != nullptr) {
            mbar_arrive(&ms.q_land);               // bf16 q: the epilogue warps fill the slot
          } else {
            ms.q_asked = it + 1;
            mbar_arrive_expect_tx(&ms.q_land, kStageKV);
            // this CTA's 64 rows of the tile = (token, head) pairs starting at row 64 cta
            const int qh = (64 * (int)cta) % p.h_per_q;
            const int qt = t.tile / p.q_group_div * p.G + (64 * (int)cta) / p.h_per_q;
            const uint32_t dst = sbase + kOffKV + slot * kStageKV;
            for (int c = 0; c < 4; ++c)
              tma_load_3d_hint(dst + c * kChunkBytes, &map_q, 128 * c, qh, qt, &ms.q_land, pol_stream);
            tma_load_3d_hint(dst + kQLatent, &map_q_rope, 512, qh, qt, &ms.q_land, pol_stream);
          }
        }
        __syncwarp();
        advance();
        for (int k = 0; k < t.nb; ++k, ++kb) {
          const int cur = take_idx(t, k, w);
          if (ring > 0) ok &= mbar_wait(&ms.slot_free[slot], (ring - 1) & 1, wt, kSiteKFree, k);
          const bool full = __all_sync(0xffffffffu, cur >= 0 && ok);
          const uint32_t kst = sbase + kOffKV + slot * kStageKV;
          const uint32_t kdst = kst + cj * kChunkBytes + 16 * pw * 128;
          // rope bytes: compact 64-byte rows, 64-byte swizzle (16-byte unit ^ ((row / 2) % 4))
          const uint32_t rdst = kst + kQLatent + (16 * pw + (lane >> 2)) * 64 + (((lane & 3) ^ ((lane >> 3) & 3)) << 4);
          if (full) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int ri = __shfl_sync(0xffffffffu, cur, i);
              cp_async16(kdst + i * 128 + ((cc ^ (i & 7)) << 4), kvb + (size_t)ri * pitch + 16 * lane);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const int ri = __shfl_sync(0xffffffffu, cur, 8 * i + (lane >> 2));
              cp_async16(rdst + i * 512, kvb + (size_t)ri * pitch + 512 + 16 * (lane & 3));
            }
          } else {
            go = __all_sync(0xffffffffu, ok);
            if (!go) break;
#pragma unroll 1
            for (int i = 0; i < 16; ++i) {
              const int ri = __shfl_sync(0xffffffffu, cur, i);
              cp_async16_or_zero(kdst + i * 128 + ((cc ^ (i & 7)) << 4), kvb + (size_t)max(ri, 0) * pitch + 16 * lane, ri >= 0);
            }
#pragma unroll 1
            for (int i = 0; i < 2; ++i) {
              const int ri = __shfl_sync(0xffffffffu, cur, 8 * i + (lane >> 2));
              cp_async16_or_zero(rdst + i * 512, kvb + (size_t)max(ri, 0) * pitch + 512 + 16 * (lane & 3), ri >= 0);
            }
          }
          cp_async_mbar_arrive_noinc(&ms.k_land[kb & 7]);
          advance();
        }
      }
    } else {
      // lane: rows 16 pw + 2 i + lane / 16 of the peer's keys, 16-byte piece lane % 16 of this CTA's 256 value bytes
      const int pc = lane & 15, r2 = lane >> 4;
      const uint8_t* src = kvb + 256 * cta + 16 * pc;
      for (int w = cid; go && w < n_items; w += ncl) {
        const Item t = nx;
        if (w + ncl < n_items) nx = item_of(w + ncl);
        advance();                                 // the item's Q
        for (int k = 0; k < t.nb; ++k, ++kb) {
          const int cur = take_idx(t, k, w);
          ok &= mbar_wait(&ms.qk_done[kb & 7], (kb >> 3) & 1, wt, kSiteVFree, k);
          const bool full = __all_sync(0xffffffffu, cur >= 0 && ok);
          // the dead half of the K tile: chunks 2-3 in CTA 0, chunks 0-1 in CTA 1
          const uint32_t vst = sbase + kOffKV + slot * kStageKV + (cta == 0 ? 2 * kChunkBytes : 0) + (pc >> 3) * kChunkBytes +
                               (16 * pw + r2) * 128;
          if (full) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int ri = __shfl_sync(0xffffffffu, cur, 2 * i + r2);
              cp_async16(vst + i * 256 + (((pc & 7) ^ ((2 * i + r2) & 7)) << 4), src + (size_t)ri * pitch);
            }
          } else {
            go = __all_sync(0xffffffffu, ok);
            if (!go) break;
#pragma unroll 1
            for (int i = 0; i < 8; ++i) {
              const int ri = __shfl_sync(0xffffffffu, cur, 2 * i + r2);
              cp_async16_or_zero(vst + i * 256 + (((pc & 7) ^ ((2 * i + r2) & 7)) << 4), src + (size_t)max(ri, 0) * pitch, ri >= 0);
            }
          }
          cp_async_mbar_arrive_noinc(&ms.v_land[kb & 7]);
          advance();
        }
      }
    }
  } else if (warp < kWarpEpi0) {
   asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
   // running position of an MMA-issuing warp: work item, block of the item, blocks of the item, item
   // ordinal, running block number, ring slot
   struct MmaCursor { int w, k, nb, it, kb, slot; };
   auto mma_next = [&](MmaCursor& c) {
     ++c.kb;
     if (++c.slot == kSlots) c.slot = 0;
     if (++c.k == c.nb) {
       c.w += ncl; c.k = 0; ++c.it;
       if (++c.slot == kSlots) c.slot = 0;       // the next item's Q entry
       c.nb = c.w < n_items ? item_of(c.w).nb : 0;
     }
   };
   // the time-limit and abort check of a wait that has not been satisfied yet (warp-uniform answer)
   auto mma_idle = [&](uint32_t& since, int site, int kb) -> bool {
     return __any_sync(0xffffffffu, wt.gives_up(since, site, kb));
   };
   if (warp == kWarpMma) {
    // ------------------------------------------------------------ MMA issue (leader CTA only)
    if (cta == 0) {   // the whole warp runs this loop; one elected lane issues
      constexpr uint32_t idesc_qk = umma_idesc(0, 0, false, false, 128, 128);
      const uint32_t a_qk_done0 = smem_u32(&ms.qk_done[0]), a_qk_done0_peer = mapa(a_qk_done0, 1);
      const uint32_t a_q_free_peer = mapa(smem_u32(&ms.q_free), 1);
      // S = Q K^T of block kb into S buffer kb%2
      // (the K / V rows were written by cp.async (generic proxy) and are read by the tensor core
      // through the async proxy: a cross-proxy fence sits between "landed" and the MMA)
      // descriptor high words: 128-byte swizzle (8-row groups 1024 B apart) for the four latent
      // chunks, 64-byte swizzle (8-row groups 512 B apart) for the compact rope chunk
      const uint32_t hi128 = (uint32_t)(umma_desc(0, 16, 1024, kSwz128) >> 32);
      const uint32_t hi64 = (uint32_t)(umma_desc(0, 16, 512, kSwz64) >> 32);
      const uint32_t a_rope_lo = (uint32_t)umma_desc(sbase + kOffRope, 16, 512, kSwz64);
      auto issue_qk = [&](int kb, int slot) {
        fence_proxy_async_smem();
        tc_fence_after();
        const uint32_t d = tmem + ((kb & 1) ? kTmemS1 : kTmemS0);
        const uint32_t b_lo = (uint32_t)umma_desc(sbase + kOffKV + slot * kStageKV, 16, 1024, kSwz128);
        mma_f8_pair_qk18(d, idesc_qk, tmem + kTmemQ, b_lo, hi128, hi64, a_rope_lo);
        mma_commit_pair_elect(a_qk_done0 + 8u * (uint32_t)(kb & 7));
        mma_commit_pair_elect(a_qk_done0_peer + 8u * (uint32_t)(kb & 7));
      };
      // Two warps issue the MMAs, this one QK^T and the next one PV: each waits for its own operands and
      // the tensor pipe takes what comes first.  One flat loop over a cursor whose every decision is a
      // vote: the compiler then keeps the MMA operands in uniform registers (nested loops with
      // breaks: 53 cycles to issue an MMA instead of 23).
      MmaCursor c{cid, 0, cid < n_items ? item_of(cid).nb : 0, 0, 0, 1};
      bool aborted = false;
      uint32_t since = 0;
      while (c.w < n_items && !aborted) {
        // K rows landed on both CTAs, S buffer drained and, for an item's first block, Q in place
        const uint32_t ph = (c.kb >> 3) & 1;
        const bool ok = (c.k > 0 || mbar_try_wait(&ms.qt_ready, c.it & 1)) && mbar_try_wait(&ms.k_land[c.kb & 7], ph) &&
                        mbar_try_wait(&ms.k_peer[c.kb & 7], ph) &&
                        (c.kb < 2 || mbar_try_wait(&ms.s_free[c.kb & 1], ((c.kb >> 1) & 1) ^ 1));
        if (__all_sync(0xffffffffu, ok)) {
          issue_qk(c.kb, c.slot);
          if (c.k == c.nb - 1) {      // Q is no longer needed once these MMAs complete
            mma_commit_pair_elect(smem_u32(&ms.q_free));
            mma_commit_pair_elect(a_q_free_peer);
          }
          mma_next(c);
          since = 0;
        } else {
          aborted = mma_idle(since, kSiteKLand, c.kb);
        }
      }
      if (lane == 0) ms.qk_end = c.kb;
    }
   } else if (warp == kWarpRelayK && cta == 0) {
      // ---------------------------------------------------------- PV issue (leader CTA)
      constexpr uint32_t idesc_pv = umma_idesc(0, 0, false, true, 128, 256);
      const uint32_t a_pv_done0 = smem_u32(&ms.pv_done[0]), a_pv_done0_peer = mapa(a_pv_done0, 1);
      const uint32_t a_slot_free0 = smem_u32(&ms.slot_free[0]), a_slot_free0_peer = mapa(a_slot_free0, 1);
      auto issue_pv = [&](int k, int kb, int slot) {
        fence_proxy_async_smem();
        tc_fence_after();
        const uint64_t ad = umma_desc(sbase + kOffP + (kb & 1) * kPBytes, 1024, 128, kSwzNone);
        const uint64_t bd = umma_desc(sbase + kOffKV + slot * kStageKV, kChunkBytes, 1024, kSwz128);
        mma_f8_pair_pv8(tmem + kTmemO, idesc_pv, (uint32_t)ad, (uint32_t)bd, (uint32_t)(ad >> 32),
                        (uint32_t)(bd >> 32), k ? 1u : 0u);
        mma_commit_pair_elect(a_slot_free0 + 8u * (uint32_t)slot);
        mma_commit_pair_elect(a_slot_free0_peer + 8u * (uint32_t)slot);
        mma_commit_pair_elect(a_pv_done0 + 8u * (uint32_t)(kb & 3));
        mma_commit_pair_elect(a_pv_done0_peer + 8u * (uint32_t)(kb & 3));
      };
      MmaCursor c{cid, 0, cid < n_items ? item_of(cid).nb : 0, 0, 0, 1};
      bool aborted = false;
      uint32_t since = 0;
      while (c.w < n_items && !aborted) {
        // V rows landed on both CTAs, P written; an item's first PV overwrites O: the previous item
        // must have read it out
        const uint32_t ph = (c.kb >> 3) & 1;
        const bool ok = mbar_try_wait(&ms.v_land[c.kb & 7], ph) && mbar_try_wait(&ms.v_peer[c.kb & 7], ph) &&
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
  } else if (warp == kWarpRelayK || warp == kWarpRelayV) {
    // ------------------------------------------------------------ "landed" relays to the leader CTA
    // The MMA thread lives in the leader CTA and can only wait on its own barriers: in the
    // peer CTA these warps forward "K rows landed" and "V rows landed".
    if (cta == 1) {
      const bool is_k = warp == kWarpRelayK;
      const uint32_t a_peer0 = mapa(smem_u32(is_k ? &ms.k_peer[0] : &ms.v_peer[0]), 0);
      int kb = 0;
      for (int w = cid; w < n_items; w += ncl) {
        const int nb = item_of(w).nb;
        for (int k = 0; k < nb; ++k, ++kb) {
          const int s = kb & 7;
          mbar_wait(is_k ? &ms.k_land[s] : &ms.v_land[s], (kb >> 3) & 1, wt, is_k ? kSiteRelayK : kSiteRelayV, k);
          fence_proxy_async_smem();     // this CTA's cp.async writes -> the leader's MMA reads
          if (lane == 0) mbar_arrive_cluster_release(a_peer0 + 8u * (uint32_t)s);
        }
      }
    }
  } else {
    // ------------------------------------------------------------ index-validity bits (warp kWarpValid)
    static_assert(kWarpValid == kWarpRelayV + 1 && kWarpValid + 1 == kWarpEpi0, "role layout");
    int kb = 0;
    for (int w = cid; w < n_items; w += ncl) {
      const Item item = item_of(w);
      const int32_t* idx_row = p.indices + (size_t)item.tile * p.idx_stride;
      int4 cur = __ldcs(reinterpret_cast<const int4*>(idx_row + (size_t)item.block(0) * kBlockKeys) + lane);
      for (int k = 0; k < item.nb; ++k, ++kb) {
        const int s = kb & 1;
        const uint32_t ph = (kb >> 1) & 1;
        int4 nxt = cur;
        if (k + 1 < item.nb) nxt = __ldcs(reinterpret_cast<const int4*>(idx_row + (size_t)item.block(k + 1) * kBlockKeys) + lane);
        const int rank0 = item.block(k) * kBlockKeys + lane * 4;
        auto ok = [&](int idx, int rk) -> uint32_t {
          return (idx >= 0 && idx < p.s_kv && rk < item.lim) ? 1u : 0u;
        };
        const uint32_t nib = ok(cur.x, rank0) | (ok(cur.y, rank0 + 1) << 1) |
                             (ok(cur.z, rank0 + 2) << 2) | (ok(cur.w, rank0 + 3) << 3);
        if (kb >= 2) mbar_wait(&ms.valid_free[s], ph ^ 1, wt, kSiteValidFree, k);
        __syncwarp();
        const uint32_t nib_hi = __shfl_down_sync(0xffffffffu, nib, 1);
        if ((lane & 1) == 0)
          reinterpret_cast<uint8_t*>(&ms.valid[s][0])[lane >> 1] = (uint8_t)(nib | (nib_hi << 4));
        __syncwarp();
        if (lane == 0) mbar_arrive(&ms.valid_ready[s]);
        cur = nxt;
      }
    }
   }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 72;");
    // ------------------------------------------------------------ epilogue warps
    // O out of TMEM, x out_scale / l, bf16, TMA tile stores -- while the softmax warps already
    // work on the next tile.  A warp reads the TMEM lanes of its quarter (warp % 4): rows r of
    // key half h, dims [256h, 256h + 256) in 8 rounds of 32 dims.  Two rounds are staged as one
    // box of 32 rows x 128 bytes in the warp's 4 KB slice (128-byte swizzle: the 16-byte stores
    // of eight consecutive rows hit distinct banks) and one lane hands the box to TMA:
    // full-line asynchronous writes, no barrier wider than the warp.
    const int ew = warp - kWarpEpi0, e_tid = (int)threadIdx.x - 32 * kWarpEpi0;
    const int e_tl = ((warp & 3) << 5) | lane, e_r = e_tl & 63, e_h = e_tl >> 6;
    const uint32_t e_ocol = tmem + ((uint32_t)((warp & 3) * 32) << 16) + kTmemO;
    const uint32_t a_o_free = mapa(smem_u32(&ms.o_free), 0);
    const uint32_t a_qt_ready = mapa(smem_u32(&ms.qt_ready), 0);
    const uint64_t pol_stream = l2_policy_evict_first();
    // These warps also bring the Q tiles in: from the ring slot where TMA has put the item's 64 rows
    // -- or, bf16 q, where fill_q puts them: loaded, quantised and stored in the same swizzled layout
    // by these 128 threads (one pass over q instead of the quantise kernel's read and write and this
    // kernel's read) -- transfer_q moves the latent part into tensor memory, where the QK^T MMAs read
    // it: lane = row (e_r, duplicated in lanes 64-127 as the 64-rows-per-CTA form of the
    // instruction wants), chunk j -> 32 columns, and the rope chunk into its fixed buffer.  Order:
    // move Q(t + 1) once item t's last QK^T is complete, then write out O(t).
    auto fill_q = [&](int w, int j, int n) {
      mbar_wait(&ms.q_land, j & 1, wt, kSiteQ, j);         // the slot is ours
      __syncwarp();
      const int qtile = item_of(w).tile / p.q_group_div;
      const uint32_t qoff = kOffKV + (uint32_t)(n % kSlots) * kStageKV, rope = qoff + kQLatent;
      {
        const uint4* src = p.q_bf16 + ((size_t)qtile * 128 + 64 * cta) * (kDQK / 8);
#pragma unroll 1
        for (int i = 0; i < 18; i += kFillBatch) {      // 64 rows x 36 units of 16 codes = 18 units per thread
          uint4 a[kFillBatch], b[kFillBatch];
#pragma unroll
          for (int u = 0; u < kFillBatch; ++u) {
            const int unit = (i + u) * 128 + e_tid;
            a[u] = __ldcs(src + 2 * unit);
            b[u] = __ldcs(src + 2 * unit + 1);
          }
#pragma unroll
          for (int u = 0; u < kFillBatch; ++u) {
            const int unit = (i + u) * 128 + e_tid, row = unit / 36, c = unit - 36 * row;
            const uint4 v = make_uint4(e4m3x4_of_bf16(a[u].x, a[u].y, p.q_inv), e4m3x4_of_bf16(a[u].z, a[u].w, p.q_inv),
                                       e4m3x4_of_bf16(b[u].x, b[u].y, p.q_inv), e4m3x4_of_bf16(b[u].z, b[u].w, p.q_inv));
            const uint32_t off = c < 32 ? qoff + (c >> 3) * kChunkBytes + row * 128 + (((c & 7) ^ (row & 7)) << 4)
                                        : rope + row * 64 + (((c - 32) ^ ((row >> 1) & 3)) << 4);
            *reinterpret_cast<uint4*>(sm + off) = v;
          }
        }
        asm volatile("bar.sync 4, 128;" ::: "memory");
      }
    };
    auto transfer_q = [&](int j, int n) {
      if (j > 0) mbar_wait(&ms.q_free, (j - 1) & 1, wt, kSiteQFree, j);
      if (p.q_bf16 == nullptr) mbar_wait(&ms.q_land, j & 1, wt, kSiteQ, j);
      __syncwarp();      // lanes leave the wait loop one by one: re-converge before .aligned ops
      tc_fence_after();
      const int slot = n % kSlots;
      const uint8_t* qtile = sm + kOffKV + slot * kStageKV;
      const uint8_t* qrow = qtile + e_r * 128;
      {                              // rope chunk: 4 KB, 32 bytes per thread
        const uint4* src = reinterpret_cast<const uint4*>(qtile + kQLatent) + 2 * e_tid;
        uint4* dst = reinterpret_cast<uint4*>(sm + kOffRope) + 2 * e_tid;
        dst[0] = src[0];
        dst[1] = src[1];
      }
#pragma unroll 1
      for (int j4 = 0; j4 < 4; ++j4) {
        uint32_t v[32];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const uint4 t = *reinterpret_cast<const uint4*>(qrow + j4 * kChunkBytes + ((u ^ (e_r & 7)) << 4));
          v[4 * u] = t.x; v[4 * u + 1] = t.y; v[4 * u + 2] = t.z; v[4 * u + 3] = t.w;
        }
        tmem_st32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + kTmemQ + 32 * j4, reinterpret_cast<const float*>(v));
      }
      tmem_wait_st();
      tc_fence_before();
      fence_proxy_async_smem();      // rope -> the MMAs' reads; these reads -> the slot's next TMA write
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(a_qt_ready);
      asm volatile("bar.sync 4, 128;" ::: "memory");      // all four warps have read the slot
      if (e_tid == 0) {
        mbar_arrive(&ms.slot_free[slot]);
        mbar_arrive(&ms.q_taken);
      }
    };
    int kb0 = 0, it = 0;
    if (cid < n_items) {
      if (p.q_bf16 != nullptr) fill_q(cid, 0, 0);
      transfer_q(0, 0);
    }
    for (int w = cid; w < n_items; w += ncl, ++it) {
      const Item item = item_of(w);
      const int tile = item.tile;
      const int kbl = kb0 + item.nb - 1;           // last block of the item
      if (w + ncl < n_items) {
        const int n = kb0 + item.nb + it + 1;      // entry number of the next item's Q
        if (p.q_bf16 != nullptr) fill_q(w + ncl, it + 1, n);
        transfer_q(it + 1, n);
      }
      // the row scales are published and the item's last PV has completed
      mbar_wait(&ms.epi_ready[it & 1], (it >> 1) & 1, wt, kSiteEpi, it);
      mbar_wait(&ms.pv_done[kbl & 3], (kbl >> 2) & 1, wt, kSiteEpi, item.nb);
      __syncwarp();      // lanes leave the wait loop one by one: re-converge before .aligned ops
      tc_fence_after();
      // Behind the cluster's last item nothing is loaded any more, and with its PVs complete the ring is free for all of O.
      const bool last = w + ncl >= n_items;
      if (kSliced) {
        // a slice: unnormalised fp32 O to its slot (few slices exist, all of them in L2), a row's half per thread: in one
        // bulk copy through the ring, or directly
        float4* dst = reinterpret_cast<float4*>(p.part_o + ((size_t)w * 128 + 64 * cta + e_r) * kDV + 256 * e_h);
        const uint32_t row_off = kOffKV + (64 * e_h + e_r) * 1024;
        float4* to = last ? reinterpret_cast<float4*>(sm + row_off) : dst;
        static_assert(128 * 1024 <= kSlots * kStageKV, "O of a slice fits into the ring");
        float o[32];
#pragma unroll 1
        for (int cc = 0; cc < 8; ++cc) {
          tmem_ld32(e_ocol + cc * 32, o);
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
        kb0 += item.nb;
        continue;
      }
      const float oscale = ms.oscale[it & 1][e_r];
      const uint32_t emask = oscale != 0.f ? 0xffffffffu : 0u;
      // this warp's 32 rows of the tile = (token, head) pairs starting at row r0
      const int r0 = (int)cta * 64 + 32 * (warp & 1);
      const int out_head = r0 % p.h_per_q, out_tok = tile * p.G + r0 / p.h_per_q;
      float o[32];
      tmem_ld32(e_ocol, o);
#pragma unroll 1
      for (int cc = 0; cc < 8; ++cc) {
        tmem_wait_ld();
        uint32_t wv[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          __nv_bfloat162 v2 = __floats2bfloat162_rn(o[2 * j] * oscale, o[2 * j + 1] * oscale);
          wv[j] = *reinterpret_cast<uint32_t*>(&v2) & emask;    // rows without a valid key: zeros
        }
        if (cc < 7) {
          tmem_ld32(e_ocol + (cc + 1) * 32, o);
        } else {
          // O has been read: the next item's first PV may overwrite it
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(a_o_free);
        }
        {
          // two rounds make one box of 32 rows x 128 bytes (128-byte swizzle) in the warp's 4 KB
          // slice; before the first of them the previous box must have been read out
          if ((cc & 1) == 0 && !last) {
            if (lane == 0) bulk_wait_read_all();
            __syncwarp();
          }
          const uint32_t slice = last ? kOffKV + (uint32_t)ew * 16384 + (cc >> 1) * 4096 : kOffStage + (uint32_t)ew * 4096;
          uint8_t* st_row = sm + slice + (e_r & 31) * 128;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            *reinterpret_cast<uint4*>(st_row + (((4 * (cc & 1) + j) ^ (e_r & 7)) << 4)) =
                make_uint4(wv[4 * j], wv[4 * j + 1], wv[4 * j + 2], wv[4 * j + 3]);
          if (last ? cc == 7 : (cc & 1) != 0) {
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              for (int x = last ? 0 : cc >> 1; x <= cc >> 1; ++x)
                for (int d = 0; d < p.n_out; ++d)
                  tma_store_3d_hint(&omaps.m[d], sbase + slice - 4096 * ((cc >> 1) - x), 256 * e_h + 64 * x, out_head, out_tok, pol_stream);
              bulk_commit_group();
            }
          }
        }
      }
      kb0 += item.nb;
    }
    if (kSliced || lane == 0) bulk_wait_all();   // output boxes and rows written before the CTA retires
    tc_fence_before();
  }

  // tear-down: nobody may still be reading TMEM of either CTA when it is released
  __syncthreads();
  if (ms.left != 0) {
    cp_async_wait_all();
    if (threadIdx.x == 0) {
      if (ms.q_asked != 0) {      // the last Q requested: with the arrivals of the warps that have left it counts as landed when it has
        for (int i = 0; i < kProducerWarps / 2; ++i)
          if (ms.q_passed[i] < ms.q_asked) mbar_arrive(&ms.q_land);
        mbar_drain(&ms.q_land, (ms.q_asked - 1) & 1);
      }
      if (ms.qk_end != 0) mbar_drain(&ms.qk_done[(ms.qk_end - 1) & 7], ((ms.qk_end - 1) >> 3) & 1);
      if (ms.pv_end != 0) mbar_drain(&ms.pv_done[(ms.pv_end - 1) & 3], ((ms.pv_end - 1) >> 2) & 1);
    }
  }
  __syncwarp();
  cluster_sync_all();
  if (warp == kWarpMma) tmem_dealloc_pair(tmem, kTmemCols);
  if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&g_attn_status[3], 1);
  if (threadIdx.x == 0) wt.report(g_attn_status, p.epoch);
}

// how many 2-CTA clusters of this kernel device `dev` (the current one) can hold at once
static int max_clusters(int dev) {
  static thread_local int cached_dev = -1, cached = 0;
  if (dev == cached_dev) return cached;
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int n = sms / 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(sms, 1, 1); cfg.blockDim = dim3(kAttnThreads, 1, 1); cfg.dynamicSmemBytes = Plan::kSmem;
  cudaLaunchAttribute at; at.id = cudaLaunchAttributeClusterDimension; at.val.clusterDim.x = 2; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
  cfg.attrs = &at; cfg.numAttrs = 1;
  int q = 0;
  if (ensure_smem<masked_mla_fp8_kernel<false>>(dev, Plan::kSmem) &&
      cudaOccupancyMaxActiveClusters(&q, masked_mla_fp8_kernel<false>, &cfg) == cudaSuccess && q > 0)
    n = q;
  cudaGetLastError();
  cached_dev = dev; cached = n;
  return n;
}

static int launch_fp8_t(const CUtensorMap& map_q, const CUtensorMap& map_q_rope, const OutMaps& omaps,
                        const AttnParams& p, cudaStream_t stream) {
  const int dev = current_device();
  const bool sliced = p.nsplit > 1;
  if (!(sliced ? ensure_smem<masked_mla_fp8_kernel<true>>(dev, Plan::kSmem)
               : ensure_smem<masked_mla_fp8_kernel<false>>(dev, Plan::kSmem)))
    return LITEDSA_ERR_CUDA;
  return launch_pdl(sliced ? masked_mla_fp8_kernel<true> : masked_mla_fp8_kernel<false>, dim3(2 * min(p.ng * p.nsplit, max_clusters(dev))), kAttnThreads,
                    Plan::kSmem, stream, map_q, map_q_rope, omaps, p);
}

static int launch_fp8(const Fp8Args& a, void* const* outs, int n_out, cudaStream_t stream) {
  CUtensorMap map_q, map_q_rope;
  OutMaps omaps;
  // q and out are addressed as (dim, head, token): row r of a tile is (token r / h, head r % h),
  // which covers the dense packed layout and the in-place layout with padded head slots alike.
  // out is stored as boxes of 32 rows x 64 dims (128 bytes wide, 128-byte swizzle); only the
  // destinations in use are encoded, the unused slots repeat the first map
  const int h = a.h_per_q, G = 128 / h;
  const int qdiv = a.q_group_div > 0 ? a.q_group_div : 1;
  const uint64_t q_hs = a.q_head_stride ? (uint64_t)a.q_head_stride : (uint64_t)a.q_row_stride;
  const uint64_t q_ts = a.q_token_stride ? (uint64_t)a.q_token_stride : (uint64_t)h * q_hs;
  const uint64_t o_hs = (a.out_head_stride ? (uint64_t)a.out_head_stride : (uint64_t)kDV) * 2;
  const uint64_t o_ts = a.out_token_stride ? (uint64_t)a.out_token_stride * 2 : (uint64_t)h * o_hs;
  const uint32_t ob_h = (uint32_t)min(h, 32);
  for (int d = 0; d < n_out; ++d)
    if (!make_map_3d(&omaps.m[d], outs[d], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, kDV, (uint64_t)h,
                     (uint64_t)a.ng * G, o_hs, o_ts, 64, ob_h, 32 / ob_h, CU_TENSOR_MAP_SWIZZLE_128B))
      return LITEDSA_ERR_CUDA;
  for (int d = n_out; d < kMaxOutputs; ++d) omaps.m[d] = omaps.m[0];
  // Q per CTA: four boxes of 128 bytes x 64 rows (128-byte swizzle) and the rope box of 64 bytes
  // x 64 rows (64-byte swizzle)
  const uint32_t qb_h = (uint32_t)min(h, 64);
  if (a.q_is_bf16) {
    map_q = map_q_rope = omaps.m[0];       // not used by the kernel
  } else if (!make_map_3d(&map_q, a.q8, CU_TENSOR_MAP_DATA_TYPE_UINT8, kDQK, (uint64_t)h,
                   (uint64_t)(a.ng / qdiv) * G, q_hs, q_ts, 128, qb_h, 64 / qb_h) ||
      !make_map_3d(&map_q_rope, a.q8, CU_TENSOR_MAP_DATA_TYPE_UINT8, kDQK, (uint64_t)h,
                   (uint64_t)(a.ng / qdiv) * G, q_hs, q_ts, 64, qb_h, 64 / qb_h, CU_TENSOR_MAP_SWIZZLE_64B))
    return LITEDSA_ERR_CUDA;
  AttnParams p;
  p.memb = a.memb_qm; p.len_per_q = a.topk_length_per_q; p.sink = a.attn_sink; p.q_group_div = qdiv;
  p.indices = a.indices; p.counts = a.topk_length;
  p.kv = reinterpret_cast<const uint8_t*>(a.kv8); p.kv_pitch = a.kv_row_stride;
  p.n_out = n_out; p.lse = a.lse;
  p.max_logits = a.max_logits;
  p.ng = a.ng; p.s_kv = a.s_kv; p.cap = a.topk; p.h_per_q = a.h_per_q; p.G = 128 / a.h_per_q;
  p.idx_stride = a.indices_row_stride;
  p.scale_log2 = a.sm_scale * kLog2e; p.out_scale = a.out_scale;
  p.epoch = next_launch_epoch(); p.wait_limit = wait_limit_ticks();
  p.q_bf16 = a.q_is_bf16 ? reinterpret_cast<const uint4*>(a.q8) : nullptr; p.q_inv = a.q_inv;
  p.nsplit = a.nsplit; p.part_o = a.part_o; p.part_ml = reinterpret_cast<float2*>(a.part_ml);
  return launch_fp8_t(map_q, map_q_rope, omaps, p, stream);
}

// Host-side argument rules shared by every FP8 attention entry point: the reference
// launcher's shape rules (kernels/b200/dsa/litedsa.cu:82-98) plus the alignment TMA needs.
// No CUDA call is made here.
int check_fp8_args(const Fp8Args& a) {
  if (!a.q8 || !a.kv8 || !a.indices || !a.lse) return LITEDSA_ERR_ARG;
  if (!a.memb_qm && !a.topk_length_per_q) return LITEDSA_ERR_ARG;   // one of the two masks
  if (a.ng <= 0 || a.s_kv <= 0 || a.topk <= 0 || a.topk % 128 != 0) return LITEDSA_ERR_SHAPE;
  if (a.h_per_q <= 0 || 128 % a.h_per_q != 0 || 128 / a.h_per_q > 16) return LITEDSA_ERR_SHAPE;
  if (a.q_group_div < 1 || a.ng % a.q_group_div != 0) return LITEDSA_ERR_SHAPE;
  // TMA needs 16-byte aligned bases and row pitches
  if (a.q_row_stride < kDQK || a.kv_row_stride < kDQK || a.q_row_stride % 16 || a.kv_row_stride % 16)
    return LITEDSA_ERR_UNSUPPORTED;
  if (((uintptr_t)a.q8 | (uintptr_t)a.kv8 | (uintptr_t)a.indices) & 15) return LITEDSA_ERR_UNSUPPORTED;
  if (a.indices_row_stride < a.topk || a.indices_row_stride % 4) return LITEDSA_ERR_UNSUPPORTED;
  // in-place addressing: TMA wants 16-byte multiples for every pitch
  if (a.q_token_stride < 0 || a.q_head_stride < 0 || a.out_token_stride < 0 || a.out_head_stride < 0)
    return LITEDSA_ERR_SHAPE;
  if ((a.q_head_stride && (a.q_head_stride < kDQK || a.q_head_stride % 16)) || a.q_token_stride % 16 ||
      (a.out_head_stride && (a.out_head_stride < kDV || a.out_head_stride % 8)) || a.out_token_stride % 8)
    return LITEDSA_ERR_UNSUPPORTED;
  return LITEDSA_OK;
}

int run_fp8(const Fp8Args& a, void* const* outs, int n_outs, void* stream) {
  int rc = check_fp8_args(a);
  if (rc != LITEDSA_OK) return rc;
  if (!outs || n_outs < 1 || n_outs > kMaxOutputs) return n_outs < 1 || n_outs > kMaxOutputs ? LITEDSA_ERR_SHAPE : LITEDSA_ERR_ARG;
  for (int d = 0; d < n_outs; ++d) {
    if (!outs[d]) return LITEDSA_ERR_ARG;
    if ((uintptr_t)outs[d] & 15) return LITEDSA_ERR_UNSUPPORTED;
  }
  return launch_fp8(a, outs, n_outs, reinterpret_cast<cudaStream_t>(stream));
}

}  // namespace lt

#include "attn_fp8_r64.cuh"

// Masked FP8 MLA prefill; replaces the reference operator
//   masked_mla_fp8(q, kv, indices, sm_scale, out_scale, topk_length, memb_qm, h_per_q,
//                  out, max_logits, lse)            (kernels/b200/dsa/litedsa.cu:77-135)
// with the same argument order and meaning; tensor shapes and strides are integers.
extern "C" int litedsa_masked_mla_fp8(const void* q8, const void* kv8, const int32_t* indices,
                                      float sm_scale, float out_scale,
                                      const int32_t* topk_length, const uint32_t* memb_qm,
                                      int h_per_q, void* out, float* max_logits, float* lse,
                                      int ng, int s_kv, int topk, int64_t q_row_stride,
                                      int64_t kv_row_stride, int64_t indices_row_stride,
                                      void* stream) {
  using namespace lt;
  if (!memb_qm || !out) return LITEDSA_ERR_ARG;
  Fp8Args a{q8, kv8, indices, sm_scale, out_scale, topk_length, memb_qm, h_per_q, max_logits, lse,
            ng, s_kv, topk, q_row_stride, kv_row_stride, indices_row_stride, nullptr, nullptr, 1};
  void* outs[1] = {out};
  return run_fp8(a, outs, 1, stream);
}

// The operator with the optional modes of the reference kernel's parameter block that its
// binding leaves switched off (litedsa.cu:127-132): attn_sink [128] per packed row joins the
// output normaliser (litedsa_attention_sm100.cuh:2127-2133); topk_length_per_q [ng, G] bounds
// each token to a causal prefix of the union ranks and may replace memb_qm (:1378-1385,
// :1988-1996); q_group_div consecutive tiles share one Q tile (KV split, :1383-1385, :1909).
// q_token_stride / q_head_stride / out_token_stride / out_head_stride (ELEMENTS, 0 = dense packed)
// address q and out in place inside [T, H_padded, d] tensors that hold h_per_q real heads per
// token, which removes the pack / unpack copies around the kernel
// (kernels/b200/dsa/DSV4_ZEROCOPY_PLAN.md:12-22, 50-76).
extern "C" int litedsa_masked_mla_fp8_ex(const void* q8, const void* kv8, const int32_t* indices,
                                         float sm_scale, float out_scale,
                                         const int32_t* topk_length, const uint32_t* memb_qm,
                                         int h_per_q, void* out, float* max_logits, float* lse,
                                         int ng, int s_kv, int topk, int64_t q_row_stride,
                                         int64_t kv_row_stride, int64_t indices_row_stride,
                                         const float* attn_sink, const int32_t* topk_length_per_q,
                                         int q_group_div, int64_t q_token_stride,
                                         int64_t q_head_stride, int64_t out_token_stride,
                                         int64_t out_head_stride, void* stream) {
  using namespace lt;
  if (!out) return LITEDSA_ERR_ARG;
  Fp8Args a{q8, kv8, indices, sm_scale, out_scale, topk_length, memb_qm, h_per_q, max_logits, lse,
            ng, s_kv, topk, q_row_stride, kv_row_stride, indices_row_stride, attn_sink,
            topk_length_per_q, q_group_div, q_token_stride, q_head_stride, out_token_stride,
            out_head_stride};
  void* outs[1] = {out};
  return run_fp8(a, outs, 1, stream);
}

// The same operator with the all-gather of a sharded run folded into its epilogue: every
// output box is written to n_outs destinations with plain TMA tile stores -- outs[0] is
// this GPU's buffer, outs[1..] are the peers' copies (peer-mapped device addresses of the
// slot this rank owns in each peer's gathered buffer).  The reference has no multi-GPU path.
extern "C" int litedsa_masked_mla_fp8_multi(const void* q8, const void* kv8, const int32_t* indices,
                                            float sm_scale, float out_scale,
                                            const int32_t* topk_length, const uint32_t* memb_qm,
                                            int h_per_q, void* const* outs, int n_outs,
                                            float* max_logits, float* lse, int ng, int s_kv,
                                            int topk, int64_t q_row_stride, int64_t kv_row_stride,
                                            int64_t indices_row_stride, void* stream) {
  using namespace lt;
  if (!memb_qm || !outs) return LITEDSA_ERR_ARG;
  Fp8Args a{q8, kv8, indices, sm_scale, out_scale, topk_length, memb_qm, h_per_q, max_logits, lse,
            ng, s_kv, topk, q_row_stride, kv_row_stride, indices_row_stride, nullptr, nullptr, 1};
  return run_fp8(a, outs, n_outs, stream);
}

// Synchronous read (and optional reset) of the device status block of the FP8 attention
// kernels on the current device: out[0] = first wait site that expired since the last reset
// (0 = none), out[1] = block, out[2] = iteration, out[3] = launches completed since the reset.
extern "C" int litedsa_attn_status(int* out4_host, int reset) {
  using namespace lt;
  if (out4_host &&
      cudaMemcpyFromSymbol(out4_host, g_attn_status, sizeof(int) * 4) != cudaSuccess)
    return LITEDSA_ERR_CUDA;
  if (reset) {
    const int z[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (cudaMemcpyToSymbol(g_attn_status, z, sizeof(z)) != cudaSuccess) return LITEDSA_ERR_CUDA;
  }
  return (out4_host && out4_host[0] != 0) ? LITEDSA_ERR_TIMEOUT : LITEDSA_OK;
}

// Self-test of the bounded wait, for test suites: a one-warp kernel waits with the given
// limit on an mbarrier that nobody arrives on.  The wait must give up, record its site
// (kSiteSelfTest) in the same status block the attention kernels use, and the kernel must
// return normally.  Synchronous.  Returns LITEDSA_ERR_TIMEOUT when the wait expired as it
// should, LITEDSA_OK if it (wrongly) succeeded.  Nothing hangs or faults.
namespace lt {
__global__ void wait_selftest_kernel(int epoch, unsigned long long limit_ns, int* returned) {
  __shared__ uint64_t bar;
  const Waiter wt{g_attn_status, epoch, limit_ns};
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
  }
  __syncwarp();
  const bool ok = mbar_wait(&bar, 0, wt, kSiteSelfTest, 7);
  if (threadIdx.x == 0) *returned = ok ? 1 : 2;
}
}  // namespace lt
extern "C" int litedsa_selftest_wait_timeout(uint64_t limit_ns, int* returned_device) {
  using namespace lt;
  if (!returned_device || limit_ns == 0 || limit_ns > 1000000000ull) return LITEDSA_ERR_ARG;
  wait_selftest_kernel<<<1, 32>>>(next_launch_epoch(), limit_ns, returned_device);
  if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) return LITEDSA_ERR_CUDA;
  int st[4] = {0, 0, 0, 0};
  if (cudaMemcpyFromSymbol(st, g_attn_status, sizeof(st)) != cudaSuccess) return LITEDSA_ERR_CUDA;
  return st[0] != 0 ? LITEDSA_ERR_TIMEOUT : LITEDSA_OK;
}
