// The FP8 attention kernel for tiles of 64 query rows: one CTA per tile (part of attn_fp8.cu).
//
// What it computes is masked_mla_fp8's operation on 64-row tiles (64 / h tokens x h heads) with the same
// quantisation points; only blocks are 64 keys instead of 128 and the rule that moves a row's running max is
// another one, so that it, and with it the rounding of P to e4m3, takes another course.  sparse_prefill uses it for calls of many tokens (the
// rule and its reasons: use_rows64 in prefill.cu): a union of half as many lists is shorter -- 8 tokens
// that share 70 % of their lists attend 3.1 k keys together, 4 of them 1.9 k -- and with 64 heads a tile
// is a single token that needs no membership mask at all.
//
// How it is organised:
//   * persistent, one CTA of 32 warps per SM, walking tiles blockIdx, blockIdx + #CTAs, ...
//   * tcgen05.mma.ws with M = 64: the form that spreads 64 rows over all 128 TMEM lanes (lanes 0-63 the
//     first half of an instruction's columns, lanes 64-127 the second), which plain M = 64 does not (half
//     the rate).  A block's 64 K rows are also its V rows: nothing is fetched twice and nothing crosses CTAs.
//     Measured cycles per K step of 32 bytes: QK^T (N = 64, A in TMEM) 28, although its K rows are 16 shared-memory
//      wavefronts of 128 bytes; PV (N = 256) 80, the wavefronts of both operands.  So 830 per block of 64 x 64.
//   * six 36 KB slots in a ring hold the blocks in flight (and each item's Q on its way to TMEM).
//   * warps 0-15   softmax, four groups of four warps on every fourth block each (TMEM lane x 32 columns per
//                  thread); the running max is handed from group to group, row sums are merged by the
//                  epilogue, so no group ever waits for another at the end of a tile;
//     warps 16-23  KV row gather (16-byte cp.async; entries without a key are filled with zeros);
//     warps 24, 27 QK^T issue, even and odd blocks;   warp 25  PV issue;   warp 26  index-validity bits;
//     warps 28-31  Q tiles in, tile epilogue.
//   * every wait is bounded (common.cuh).
// What bounds it inside a tile is latency x slots: stamps per role show a slot held 6100 cycles (copies 1700, QK^T and its queue
// 700, softmax 2500, wait for PV 700, PV 330), six of them 1015 per block, against 830 of the MMAs; the shared-memory pipe is 87 %
// busy beside.  Between tiles 2.3 to 3 us pass: Q's entry takes a turn of the ring, and its slot stays until the output
// staged in it has left.  Long runs are at the power limit.  With the union, e4m3 queries, three quarters
// of the lists shared, us on 128-row tiles and here: 8192 tokens x 64 heads, top-2048 1430 / 1237; 16384 x 32, top-1024 of 65535 1065 / 875; 16384 x 16,
// top-2048 of 131072 1597 / 1181; 4096 x 64, top-256 183 / 144.
#pragma once

namespace lt {
namespace r64 {

constexpr int kGroups = 4, kGroupWarps = 4, kGatherWarps = 8;
constexpr int kSlots = 6;
constexpr int kWarpGather0 = 16, kWarpQk = 24, kWarpPv = 25, kWarpValid = 26, kWarpQkOdd = 27, kWarpEpi0 = 28;
constexpr int kThreads = 1024, kRows = 64, kBlockKeys = 64;
constexpr uint32_t kSlot = kStageKV;                  // 64 rows x 576 B, laid out as in attn_fp8.cu
// By how much (log2) a row's maximum passes the running max before that moves: see the softmax warps.
constexpr float kRescale = 5.5f;

// Six slots, Q's rope chunk and the rest: P (64 rows x 64 keys e4m3) lies in the rope chunk of its own block's
// slot, which is dead once QK^T has read it and of the same 4 KB; an item's output is staged in the slot of the
// next item's Q, which has moved on to tensor memory by then (behind the last item an entry without a Q follows).
struct Plan {
  static constexpr uint32_t kOffKV = 0;
  static constexpr uint32_t kOffRope = kOffKV + kSlots * kSlot;
  static constexpr uint32_t kOffMisc = kOffRope + kRopeChunkBytes;
  static constexpr uint32_t kMiscBytes = 7168;
  static constexpr uint32_t kSmem = kOffMisc + kMiscBytes;
  static_assert(kSlot % 1024 == 0, "swizzled tiles need 1024-byte alignment");
  static_assert(kSmem <= 232448, "shared-memory plan exceeds the 227 KB per-CTA limit");
};
constexpr uint32_t kTmemO = 0;                        // 256 columns: lanes 0-63 dims 0-127 and 256-383, lanes 64-127 the others
constexpr uint32_t kTmemS = 256;                      // 32 columns per group: lanes 0-63 keys 0-31, lanes 64-127 keys 32-63
constexpr uint32_t kTmemQ = 384;                      // 128 columns: Q's latent dims, rows repeated in lanes 64-127

struct Misc {
  // by running block number modulo 8 (everybody has looked at block kb's before block kb + 8 can touch them)
  uint64_t k_land[8], qk_done[8], p_ready[8], pv_done[8];
  uint64_t slot_free[kSlots];       // the slot's entry is dead: block through its PV, or Q moved on and output staged
  uint64_t s_free[kGroups], valid_ready[kGroups], valid_free[kGroups];
  uint64_t m_pub[kGroups];          // running max after the group's latest block published
  uint64_t q_codes;                 // bf16 q: the item's codes are in q_codes
  uint64_t q_land;                  // the item's Q tile has landed in its slot
  uint64_t q_taken;                 // the item's Q has been moved out of its slot
  uint64_t qt_ready;                // Q's latent dims are in tensor memory
  uint64_t q_free;                  // all QK^T of the current item are complete
  uint64_t o_free;                  // the item's O has been read out of TMEM
  uint64_t fin_ready, fin_free;     // the item's row sums are published / have been read
  uint32_t valid[kGroups][2];       // 64 validity bits
  uint32_t tmem_base;
  // for the tear-down of a launch that gives up: a wait of this block has; items whose Q has been requested and at
  // whose q_land each gather warp has arrived; blocks whose QK^T (per issuing warp) and PV have been issued
  uint32_t left, q_asked, q_passed[kGatherWarps], qk_end[2], pv_end;
  float xbuf[kGroups][128];         // [group][lane]: row-max exchange between the key halves
  float mshare[kGroups][64];        // [group][row]: running max after the group's latest block
  float fin_l[kGroups][128], fin_m[kGroups][64];     // end of item: row sums per thread, relative to the group's last running max
};
static_assert(sizeof(Misc) <= Plan::kMiscBytes, "Misc too large");

struct Params {
  const uint32_t* memb;      // [ng, G, cap / 32], or null: every list entry is every row's
  const int32_t* indices;    // [ng, cap], -1 up to the next multiple of 64
  const int32_t* counts;     // [ng]
  const int2* order;         // [ng] (tile, keys) in the order in which they are dealt out, or null: as they come
  const uint8_t* kv;         // [s_kv, kv_pitch] e4m3 rows (576 bytes used)
  long long kv_pitch;
  float* lse;                // [ng, 64]
  int ng, s_kv, cap, h_per_q, G;
  float scale_log2, out_scale;
  int epoch;
  uint32_t wait_limit;       // of one wait, in ticks (BlockWaiter)
  // bf16 queries, quantised by the epilogue warps an item ahead into q_codes [2][CTAs][64, 576] (map_q and
  // map_q_rope are of that then); null: e4m3
  const uint4* q_bf16;
  uint8_t* q_codes;
  float q_inv;
};

// the whole K loop of one 64-key block, one elected lane of a converged warp issues (as in common.cuh)
#define LT_WS_TS(AINC, BINC, PRED)                                             \
  "add.u32 qa, %2, " #AINC ";\n\tadd.u32 blo, %3, " #BINC ";\n\tmov.b64 bd, {blo, %4};\n\t" \
  "@pe tcgen05.mma.ws.cta_group::1.kind::f8f6f4 [%0], [qa], bd, %1, " #PRED ";\n\t"
#define LT_WS_SS(INC, PRED)                                                    \
  "add.u32 alo, %6, " #INC ";\n\tadd.u32 blo, %3, 2048 + " #INC ";\n\t"           \
  "mov.b64 ad, {alo, %5};\n\tmov.b64 bd, {blo, %5};\n\t"                       \
  "@pe tcgen05.mma.ws.cta_group::1.kind::f8f6f4 [%0], ad, bd, %1, " #PRED ";\n\t"
__device__ __forceinline__ void mma_qk18(uint32_t d_tmem, uint32_t idesc, uint32_t q_tmem, uint32_t b_lo, uint32_t hi128,
                                         uint32_t hi64, uint32_t a_rope_lo) {
  asm volatile(
      "{\n\t.reg .pred pz, po, pe;\n\t.reg .b32 qa, alo, blo;\n\t.reg .b64 ad, bd;\n\t"
      "setp.ne.b32 pz, 0, 0;\n\tsetp.eq.b32 po, 0, 0;\n\telect.sync _|pe, 0xffffffff;\n\t"
      LT_WS_TS(0, 0, pz) LT_WS_TS(8, 2, po) LT_WS_TS(16, 4, po) LT_WS_TS(24, 6, po)
      LT_WS_TS(32, 512, po) LT_WS_TS(40, 514, po) LT_WS_TS(48, 516, po) LT_WS_TS(56, 518, po)
      LT_WS_TS(64, 1024, po) LT_WS_TS(72, 1026, po) LT_WS_TS(80, 1028, po) LT_WS_TS(88, 1030, po)
      LT_WS_TS(96, 1536, po) LT_WS_TS(104, 1538, po) LT_WS_TS(112, 1540, po) LT_WS_TS(120, 1542, po)
      LT_WS_SS(0, po) LT_WS_SS(2, po)
      "}"
      ::"r"(d_tmem), "r"(idesc), "r"(q_tmem), "r"(b_lo), "r"(hi128), "r"(hi64), "r"(a_rope_lo)
      : "memory");
}
//   P V: two N = 256 halves (D column offset 128, two 128-dim chunks of V each) x two 32-key steps
#define LT_WS_PV(DOFF, AINC, BINC, PRED)                                \
  "add.u32 dd, %0, " #DOFF ";\n\tadd.u32 alo, %2, " #AINC ";\n\tadd.u32 blo, %3, " #BINC ";\n\t" \
  "mov.b64 ad, {alo, %4};\n\tmov.b64 bd, {blo, %5};\n\t"                  \
  "@pe tcgen05.mma.ws.cta_group::1.kind::f8f6f4 [dd], ad, bd, %1, " #PRED ";\n\t"
__device__ __forceinline__ void mma_pv4(uint32_t d_tmem, uint32_t idesc, uint32_t a_lo, uint32_t b_lo, uint32_t a_hi,
                                        uint32_t b_hi, uint32_t accumulate_first) {
  asm volatile(
      "{\n\t.reg .pred pf, po, pe;\n\t.reg .b32 alo, blo, dd;\n\t.reg .b64 ad, bd;\n\t"
      "setp.ne.b32 pf, %6, 0;\n\tsetp.eq.b32 po, 0, 0;\n\telect.sync _|pe, 0xffffffff;\n\t"
      LT_WS_PV(0, 0, 0, pf) LT_WS_PV(0, 128, 256, po) LT_WS_PV(128, 0, 1024, pf) LT_WS_PV(128, 128, 1280, po)
      "}"
      ::"r"(d_tmem), "r"(idesc), "r"(a_lo), "r"(b_lo), "r"(a_hi), "r"(b_hi), "r"(accumulate_first)
      : "memory");
}
__device__ __forceinline__ void commit_elect(uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred pe;\n\telect.sync _|pe, 0xffffffff;\n\t"
      "@pe tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
      ::"r"(smem_u32(bar)) : "memory");
}
// kWide: the cache is too large for row offsets in 32 bits of 16-byte units (64 GB); their products in 64 bits take 1 %
// of the time (8192 tokens x 64 heads 1271 -> 1295 us)
template <bool kWide, bool kOrdered>
__global__ void __launch_bounds__(kThreads, 1)
masked_mla_fp8_r64_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_q_rope,
                          const __grid_constant__ CUtensorMap map_out, const Params p) {
  constexpr uint32_t kOffRope = Plan::kOffRope, kOffKV = Plan::kOffKV, kOffMisc = Plan::kOffMisc;
  extern __shared__ __align__(1024) uint8_t sm[];
  const uint32_t sbase = smem_u32(sm);
  Misc& ms = *reinterpret_cast<Misc*>(sm + kOffMisc);
  const BlockWaiter wt{&ms.left, p.wait_limit};
  // The plan fills the shared memory, so the base cannot be rounded up: swizzled tiles on another one would be
  // read wrongly without any error.
  if ((sbase & 1023u) != 0) {
    pdl_wait();
    if (threadIdx.x == 0) Waiter{g_attn_status, p.epoch, 0}.fail(kSiteAlign, (int)(sbase & 1023u));
    return;
  }

  const int cid = blockIdx.x, ncta = gridDim.x, ng = p.ng;
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  // item i: its tile (x) and that one's keys (y), and the key blocks of these, 0 past the last one.  Every role loads the next
  // item's a tile ahead: a dependent load at the change of tiles would hold up all of them.
  auto item_at = [&](int i) -> int2 {
    if (i >= ng) return make_int2(0, -1);
    return kOrdered ? __ldcg(p.order + i) : make_int2(i, min(max(p.counts[i], 0), p.cap));
  };
  struct Next { int tile, nb; };
  auto next_at = [&](int i) -> Next {
    const int2 v = item_at(i);
    return {v.x, v.y >= 0 ? max((v.y + kBlockKeys - 1) / kBlockKeys, 1) : 0};
  };
  // the tile of item i, `known` where that has to be loaded
  auto tile_at = [&](int i, int known) -> int { return kOrdered ? known : i; };

  if (threadIdx.x == 0) {
    for (int i = 0; i < 8; ++i) {
      mbar_init(&ms.k_land[i], kGatherWarps / 2 * 32);      // one async arrival per thread of the block's gather set
      mbar_init(&ms.qk_done[i], 1);
      mbar_init(&ms.p_ready[i], kGroupWarps);
      mbar_init(&ms.pv_done[i], 1);
    }
    for (int i = 0; i < kSlots; ++i) mbar_init(&ms.slot_free[i], 1);
    for (int i = 0; i < kGroups; ++i) {
      mbar_init(&ms.s_free[i], kGroupWarps);
      mbar_init(&ms.valid_ready[i], 1);
      mbar_init(&ms.valid_free[i], kGroupWarps);
      mbar_init(&ms.m_pub[i], kGroupWarps);
    }
    mbar_init(&ms.q_codes, 1);
    mbar_init(&ms.q_land, kGatherWarps);
    mbar_init(&ms.q_taken, 1);
    mbar_init(&ms.qt_ready, kEpiWarps);
    mbar_init(&ms.q_free, 2);                       // both QK^T warps
    mbar_init(&ms.o_free, kEpiWarps);
    mbar_init(&ms.fin_ready, kGroups * kGroupWarps);
    mbar_init(&ms.fin_free, kEpiWarps);
    ms.left = ms.q_asked = 0;
    for (int i = 0; i < kGatherWarps; ++i) ms.q_passed[i] = 0;
    fence_mbar_init();
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_q_rope);
    tma_prefetch_desc(&map_out);
  }
  if (warp == kWarpQk) {
    tmem_alloc_cta(&ms.tmem_base, kTmemCols);
    tmem_relinquish_cta();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = ms.tmem_base;
  pdl_trigger();
  pdl_wait();

  // registers: 72 x 4 + 48 x 2 + 48 + 80 = 512 = 64 x 8, as launched
  if (warp < kWarpGather0) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 72;");
    // ------------------------------------------------------------ softmax
    // Group g serves the blocks with kb % 4 == g; thread = (TMEM lane tl, all 32 columns): row r = tl % 64, keys
    // [32 h, +32) of the block with h = tl / 64.  (Two groups of eight warps with 16 columns per thread take as
    // long for a block, 1900 cycles: waits and exchanges, not arithmetic, are most of it.)  Block kb always
    // waits for block kb - 1's running max, also over the end of an item: that keeps every barrier's phases in step.
    // The largest weight of a row is exact in e4m3 if the running max is its own.  With the 128-row kernel's rule (it moves
    // when a row of the warp's 32 passes it by more than 6) and 64 keys at a time it less often was: error against 64
    // bits over the 128-row form's, 13 shapes, N(0, s) queries: s = 1 0.96-1.01, s = 2.5 1.00-1.10, s = 4 0.99-1.13.  So
    // when it moves it also covers the maxima of the block behind (0.96-1.01, 0.92-1.01, 0.88-1.01: fewer
    // moves, so it costs nothing), and it moves at 5.5: 0.95-1.00, 0.84-0.97, 0.83-0.97, for about 1 % of the time
    // (4096 tokens x 64 heads, top-512: 212 -> 215 us; at 5.25 217).  The maxima of the block behind stay in their
    // group's xbuf until they have been read: the group's next block comes behind this block's running max.
    const int g = warp >> 2;
    const int tl = ((warp & 3) << 5) | lane;
    const int r = tl & 63, h = tl >> 6;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const int capw = p.cap >> 5;
    const float c = p.scale_log2;
    const uint64_t c2 = pack2(c, c);
    const uint32_t scol = tmem + lane_base + kTmemS + 32 * g;
    int kb0 = 0, it = 0;
    Next next = next_at(cid);
    // this thread's membership words: two per block of its token
    const uint32_t* mrow = p.memb ? p.memb + ((size_t)tile_at(cid, next.tile) * p.G + r / p.h_per_q) * capw + h : nullptr;
    uint32_t mk_next = ~0u;
    if (mrow) mk_next = __ldcs(mrow + 2 * g);      // (cap >= 256: a group's first word exists even if its block does not)

    for (int i = cid; i < ng; i += ncta, ++it) {
      const Next cur = next;
      const int nb = cur.nb;
      next = next_at(i + ncta);
      float m_mine = kMInit;      // the running max my row sum is relative to
      float li = 0.f;

      for (int k = (g - kb0) & (kGroups - 1); k < nb; k += kGroups) {
        const int kb = kb0 + k;
        const uint32_t mk = mk_next;
        if (mrow && k + kGroups < nb) mk_next = __ldcs(mrow + 2 * (k + kGroups));

        mbar_wait(&ms.qk_done[kb & 7], (kb >> 3) & 1, wt, kSiteQkDone, k);
        __syncwarp();      // lanes leave the wait loop one by one: re-converge before .aligned ops
        tc_fence_after();
        float sv[32];
        tmem_ld32(scol, sv);
        mbar_wait(&ms.valid_ready[g], (kb >> 2) & 1, wt, kSiteValidReady, k);
        const uint32_t vm = ms.valid[g][h] & mk;
        __syncwarp();
        tmem_wait_ld();
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
        ms.xbuf[g][tl] = cur;
        asm volatile("bar.sync %0, 128;" ::"r"(1 + g) : "memory");
        cur = fmaxf(cur, ms.xbuf[g][tl ^ 64]);
        // S and the validity bits have been read, the maxima published: the group's next block may come
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&ms.s_free[g]);
          mbar_arrive(&ms.valid_free[g]);
        }
        float m_prev = kMInit;
        if (kb > 0) {
          mbar_wait(&ms.m_pub[(g + 3) & 3], ((kb - 1) >> 2) & 1, wt, kSiteMPub, k);
          if (k > 0) m_prev = ms.mshare[(g + 3) & 3][r];
        }
        const bool rescale = __any_sync(0xffffffffu, cur - m_prev > kRescale);
        if (rescale && k + 1 < nb) {
          const int g2 = (g + 1) & 3;
          mbar_wait(&ms.s_free[g2], ((kb + 1) >> 2) & 1, wt, kSiteMPub, k);
          cur = fmaxf(cur, fmaxf(ms.xbuf[g2][r], ms.xbuf[g2][r + 64]));
          __syncwarp();
        }
        const float new_m = rescale ? fmaxf(cur, m_prev) : m_prev;
        if (h == 0) ms.mshare[g][r] = new_m;
        __syncwarp();
        if (lane == 0) mbar_arrive(&ms.m_pub[g]);
        li *= fast_exp2(m_mine - new_m);
        m_mine = new_m;

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
        // P into the slot's rope chunk: [16-key group][row][16 B]
        const uint32_t slot = (uint32_t)(kb + it + 1) % kSlots;
        uint8_t* pdst = sm + kOffKV + slot * kSlot + kQLatent + 2 * h * 1024 + r * 16;
        *reinterpret_cast<uint4*>(pdst) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        *reinterpret_cast<uint4*>(pdst + 1024) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
        const float2 ls = unpack2(add2(l0, l1));
        li += ls.x + ls.y;

        if (rescale && k > 0) {
          // O holds blocks [0, k) relative to m_prev: bring it to new_m once PV(k-1) is complete
          mbar_wait(&ms.pv_done[(kb - 1) & 7], ((kb - 1) >> 3) & 1, wt, kSitePvDone, k);
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
        if (lane == 0) mbar_arrive(&ms.p_ready[kb & 7]);
      }

      if (mrow && i + ncta < ng) {
        mrow += (kOrdered ? (ptrdiff_t)(next.tile - cur.tile) : (ptrdiff_t)ncta) * p.G * capw;
        mk_next = __ldcs(mrow + 2 * ((g - kb0 - nb) & (kGroups - 1)));
      }
      // end of item: row sums, each relative to its own group's latest running max, for the epilogue
      if (it > 0) mbar_wait(&ms.fin_free, (it - 1) & 1, wt, kSiteEpi, it);
      ms.fin_l[g][tl] = li;
      if (h == 0) ms.fin_m[g][r] = m_mine;
      __syncwarp();
      if (lane == 0) mbar_arrive(&ms.fin_ready);
      kb0 += nb;
    }
  } else if (warp < kWarpGather0 + kGatherWarps) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
    // ------------------------------------------------------------ KV row gather (cp.async)
    // Two sets of four warps take the ring's entries in turn (even and odd ones: with an even number of slots a
    // set also sees every earlier entry of its slots, so a slot's barrier is never tested more than one phase
    // behind).  Warp pw of a set fetches rows [16 pw, 16 pw + 16) of its blocks, 18 copies per lane; its first
    // warp requests the items' Q.  (One set for all entries: 770 cycles to issue a block's copies and 550 until
    // the next block's could start.)
    static_assert(kSlots % 2 == 0, "two sets of gather warps");
    const int set = (warp - kWarpGather0) >> 2, pw = (warp - kWarpGather0) & 3;
    const uint64_t pol_stream = l2_policy_evict_first();
    const size_t unit = kWide ? (size_t)p.kv_pitch : 16;
    const uint32_t pitch16 = (uint32_t)(p.kv_pitch >> 4);
    const int cj = lane >> 3, cc = lane & 7;       // latent piece `lane`: chunk cj, 16-byte slot cc
    const uint8_t* kv_lat = p.kv + 16 * lane;
    const uint8_t* kv_rope = p.kv + 512 + 16 * (lane & 3);
    const int own_key = 16 * pw + (lane & 15);
    int slot = set, ring = 0, e = 0, it = 0;
    Next next = next_at(cid);
    auto first_k = [&](int e0) -> int { return (set - e0 - 1) & 1; };      // first own block of an item whose Q is entry e0
    int kidx = __ldcs(p.indices + (size_t)tile_at(cid, next.tile) * p.cap + first_k(0) * kBlockKeys + own_key);
    auto advance = [&]() { slot += 2; if (slot >= kSlots) { slot -= kSlots; ++ring; } };
    bool ok = true, go = true;                     // none of this lane's / this warp's waits has given up: then it leaves
    for (int i = cid; go && i < ng + ncta; i += ncta, ++it) {      // behind the last item: an entry to stage its output in
      const int tile = tile_at(i, next.tile), nb = next.nb;
      next = next_at(i + ncta);
      const int32_t* idx = p.indices + (size_t)tile * p.cap + own_key;
      auto next_tile_idx = [&]() -> int {
        return i + ncta < ng ? __ldcs((kOrdered ? p.indices + (size_t)next.tile * p.cap + own_key : idx + (size_t)ncta * p.cap) +
                                     first_k(e + nb + 1) * kBlockKeys) : 0;
      };
      // With short items the previous Q could still be on its way.  Every warp goes through every item's barrier
      // and a Q counts as landed only when all of them have -- those of its set also through its slot's
      // barrier --, so that none is overtaken and tests a phase that is two ahead.
      if (it > 0) ok &= mbar_wait(&ms.q_taken, (it - 1) & 1, wt, kSiteQ, it);
      if (p.q_bf16 != nullptr && i < ng) ok &= mbar_wait(&ms.q_codes, it & 1, wt, kSiteQ, it);
      const bool q_mine = (e & 1) == set;
      if (q_mine && ring > 0) ok &= mbar_wait(&ms.slot_free[slot], (ring - 1) & 1, wt, kSiteKFree, it);
      __syncwarp();
      // (nothing behind a wait of any warp that gave up: the Q before could still be in flight)
      if (lane == 0 && ok && !wt.aborting()) {
        ms.q_passed[warp - kWarpGather0] = it + 1;
        if (!q_mine || pw != 0 || i >= ng) {
          mbar_arrive(&ms.q_land);
        } else {
          ms.q_asked = it + 1;
          mbar_arrive_expect_tx(&ms.q_land, kSlot);
          const uint32_t dst = sbase + kOffKV + slot * kSlot;
          const int z = p.q_bf16 != nullptr ? (it & 1) * ncta + cid : tile * p.G;
          for (int x = 0; x < 4; ++x)
            tma_load_3d_hint(dst + x * kChunkBytes, &map_q, 128 * x, 0, z, &ms.q_land, pol_stream);
          tma_load_3d_hint(dst + kQLatent, &map_q_rope, 512, 0, z, &ms.q_land, pol_stream);
        }
      }
      __syncwarp();
      if (q_mine) advance();
      int k = first_k(e);
      if (k >= nb) kidx = next_tile_idx();
      for (; k < nb; k += 2) {
        // this lane's row as an offset in 16-byte units (kWide: in rows); entries without a key become zeros.
        // (Indices are loaded a block ahead: nothing waits for a cold line.)
        const bool has = (unsigned)kidx < (unsigned)p.s_kv;
        const uint32_t row = has ? (kWide ? (uint32_t)kidx : (uint32_t)kidx * pitch16) : 0xffffffffu;
        kidx = k + 2 < nb ? __ldcs(idx + (k + 2) * kBlockKeys) : next_tile_idx();
        if (ring > 0) ok &= mbar_wait(&ms.slot_free[slot], (ring - 1) & 1, wt, kSiteKFree, k);
        const bool full = __all_sync(0xffffffffu, has && ok);
        const uint32_t kst = sbase + kOffKV + slot * kSlot;
        const uint32_t kdst = kst + cj * kChunkBytes + 16 * pw * 128;
        // rope bytes: compact 64-byte rows, 64-byte swizzle (16-byte unit ^ ((row / 2) % 4))
        const uint32_t rdst = kst + kQLatent + (16 * pw + (lane >> 2)) * 64 + (((lane & 3) ^ ((lane >> 3) & 3)) << 4);
        if (full) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const uint32_t o = __shfl_sync(0xffffffffu, row, i);
            cp_async16(kdst + i * 128 + ((cc ^ (i & 7)) << 4), kv_lat + (size_t)o * unit);
          }
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const uint32_t o = __shfl_sync(0xffffffffu, row, 8 * i + (lane >> 2));
            cp_async16(rdst + i * 512, kv_rope + (size_t)o * unit);
          }
        } else {
          go = __all_sync(0xffffffffu, ok);
          if (!go) break;
#pragma unroll 1
          for (int i = 0; i < 16; ++i) {
            const uint32_t o = __shfl_sync(0xffffffffu, row, i);
            const bool rd = o != 0xffffffffu;
            cp_async16_or_zero(kdst + i * 128 + ((cc ^ (i & 7)) << 4), rd ? kv_lat + (size_t)o * unit : p.kv, rd);
          }
#pragma unroll 1
          for (int i = 0; i < 2; ++i) {
            const uint32_t o = __shfl_sync(0xffffffffu, row, 8 * i + (lane >> 2));
            const bool rd = o != 0xffffffffu;
            cp_async16_or_zero(rdst + i * 512, rd ? kv_rope + (size_t)o * unit : p.kv, rd);
          }
        }
        cp_async_mbar_arrive_noinc(&ms.k_land[(e - it + k) & 7]);      // e - it: running number of the item's first block
        advance();
      }
      e += nb + 1;
    }
  } else if (warp < kWarpEpi0) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
    // running position of an MMA-issuing warp: item, block of its tile, its blocks, item ordinal, running block, slot
    struct Cursor { int i, k, nb, it, kb, slot, nb_next; };
    auto next = [&](Cursor& c) {
      ++c.kb;
      if (++c.slot == kSlots) c.slot = 0;
      if (++c.k == c.nb) {
        c.i += ncta; c.k = 0; ++c.it;
        if (++c.slot == kSlots) c.slot = 0;       // the next item's Q entry
        c.nb = c.nb_next;
        c.nb_next = next_at(c.i + ncta).nb;
      }
    };
    // the time-limit and abort check of a wait that has not been satisfied yet (warp-uniform answer)
    auto idle = [&](uint32_t& since, int site, int kb) -> bool {
      return __any_sync(0xffffffffu, wt.gives_up(since, site, kb));
    };
    if (warp == kWarpQk || warp == kWarpQkOdd) {
      // ---------------------------------------------------------- QK^T issue (every decision a vote: see attn_fp8.cu)
      // Two warps on alternate blocks: between two blocks a warp spends some 700 cycles on its cursor and its
      // polls among busy neighbours, and the tensor pipe's queue is shorter than that.  (One warp: 1600 cycles per block.)
      constexpr uint32_t idesc_qk = umma_idesc(0, 0, false, false, 64, 64);
      const uint32_t hi128 = (uint32_t)(umma_desc(0, 16, 1024, kSwz128) >> 32);
      const uint32_t hi64 = (uint32_t)(umma_desc(0, 16, 512, kSwz64) >> 32);
      const uint32_t a_rope_lo = (uint32_t)umma_desc(sbase + kOffRope, 16, 512, kSwz64);
      Cursor c{cid, 0, next_at(cid).nb, 0, 0, 1, next_at(cid + ncta).nb};
      auto step = [&]() {
        const int it = c.it;
        next(c);
        if (c.it != it) commit_elect(&ms.q_free);      // this warp's QK^T of the item, if it had any
      };
      const int mine = warp == kWarpQkOdd ? 1 : 0;
      bool aborted = false;
      uint32_t since = 0;
      while (c.i < ng && !aborted) {
        // K rows landed, S buffer drained and, at an item's first block, Q in place, waited for one after the other and
        // suspended.  (One barrier per lane, all tested by one instruction in a loop, took issue slots and power from the
        // warps beside: 1184 tokens x 64 heads, top-2048 189.3 -> 181.1 us, top-512 71.8 -> 68.3; long runs at the power
        // limit, 8192 x 64, top-2048, bf16 queries 1533 -> 1482.)  Both warps stop at every item's first block, whoever's it is: a warp
        // that had none in an item could otherwise report two items as read before the other has read one.
        const bool own = (c.kb & 1) == mine;
        const bool ok = (c.k > 0 || mbar_try_wait(&ms.qt_ready, c.it & 1)) &&
                        (!own || (mbar_try_wait(&ms.k_land[c.kb & 7], (c.kb >> 3) & 1) &&
                                  (c.kb < kGroups || mbar_try_wait(&ms.s_free[c.kb & (kGroups - 1)], ((c.kb >> 2) & 1) ^ 1))));
        if (__all_sync(0xffffffffu, ok)) {
          if (own) {
            fence_proxy_async_smem();      // cp.async writes -> the tensor core's reads
            tc_fence_after();
            mma_qk18(tmem + kTmemS + 32 * (c.kb & (kGroups - 1)), idesc_qk, tmem + kTmemQ,
                     (uint32_t)umma_desc(sbase + kOffKV + c.slot * kSlot, 16, 1024, kSwz128), hi128, hi64, a_rope_lo);
            commit_elect(&ms.qk_done[c.kb & 7]);
          }
          step();
          if (own && c.k != 0) step();      // the other warp's block
          since = 0;
        } else {
          aborted = idle(since, kSiteKLand, c.kb);
        }
      }
      if (lane == 0) ms.qk_end[mine] = (c.kb + 1 - mine) / 2;      // of its own
    } else if (warp == kWarpPv) {
      // ---------------------------------------------------------- PV issue
      constexpr uint32_t idesc_pv = umma_idesc(0, 0, false, true, 64, 256);
      Cursor c{cid, 0, next_at(cid).nb, 0, 0, 1, next_at(cid + ncta).nb};
      bool aborted = false;
      uint32_t since = 0;
      while (c.i < ng && !aborted) {
        // P written (its QK^T has read the K rows that are V here, so they have landed); an item's first PV
        // overwrites O: the previous item must have been read out
        const bool ok = (c.k > 0 || c.it == 0 || mbar_try_wait(&ms.o_free, (c.it - 1) & 1)) &&
                        mbar_try_wait(&ms.p_ready[c.kb & 7], (c.kb >> 3) & 1);
        if (__all_sync(0xffffffffu, ok)) {
          fence_proxy_async_smem();
          tc_fence_after();
          const uint64_t ad = umma_desc(sbase + kOffKV + c.slot * kSlot + kQLatent, 1024, 128, kSwzNone);
          const uint64_t bd = umma_desc(sbase + kOffKV + c.slot * kSlot, kChunkBytes, 1024, kSwz128);
          mma_pv4(tmem + kTmemO, idesc_pv, (uint32_t)ad, (uint32_t)bd, (uint32_t)(ad >> 32), (uint32_t)(bd >> 32), c.k ? 1u : 0u);
          commit_elect(&ms.slot_free[c.slot]);
          commit_elect(&ms.pv_done[c.kb & 7]);
          next(c);
          since = 0;
        } else {
          aborted = idle(since, kSitePReady, c.kb);
        }
      }
      if (lane == 0) ms.pv_end = c.kb;
    } else if (warp == kWarpValid) {
      // ---------------------------------------------------------- index-validity bits
      int kb = 0;
      int2 next = item_at(cid);
      const int32_t* idx = p.indices + (size_t)tile_at(cid, next.x) * p.cap + lane;
      int i0 = __ldcs(idx), i1 = __ldcs(idx + 32);
      for (int i = cid; i < ng; i += ncta) {
        const int lim = next.y, nb = max((lim + kBlockKeys - 1) / kBlockKeys, 1);
        next = item_at(i + ncta);
        for (int k = 0; k < nb; ++k, ++kb) {
          const int s = kb & (kGroups - 1), rank = k * kBlockKeys + lane;
          const uint32_t w0 = __ballot_sync(0xffffffffu, (unsigned)i0 < (unsigned)p.s_kv && rank < lim);
          const uint32_t w1 = __ballot_sync(0xffffffffu, (unsigned)i1 < (unsigned)p.s_kv && rank + 32 < lim);
          idx += kBlockKeys;
          if (k + 1 == nb) idx = p.indices + (size_t)tile_at(i + ncta, next.x) * p.cap + lane;
          if (k + 1 < nb || i + ncta < ng) {
            i0 = __ldcs(idx);
            i1 = __ldcs(idx + 32);
          }
          if (kb >= kGroups) mbar_wait(&ms.valid_free[s], ((kb >> 2) & 1) ^ 1, wt, kSiteValidFree, k);
          __syncwarp();
          if (lane == 0) {
            ms.valid[s][0] = w0;
            ms.valid[s][1] = w1;
            mbar_arrive(&ms.valid_ready[s]);
          }
          __syncwarp();
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 80;");
    // ------------------------------------------------------------ Q in, epilogue (see attn_fp8.cu)
    const int ew = warp - kWarpEpi0, e_tid = (int)threadIdx.x - 32 * kWarpEpi0;
    const uint64_t pol_stream = l2_policy_evict_first();
    const int e_r = e_tid & 63, e_h = e_tid >> 6;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t e_ocol = tmem + lane_base + kTmemO;
    // bf16 q: item j's codes into q_codes, an item ahead.  (Straight into the Q's ring slot, which is free only when
    // the item before it ends, the loads' latency held up each item by some 6000 cycles.)
    // (behind: the item behind that)
    auto quantise_q = [&](int tile, int j, bool ahead, int behind) {
      const uint4* src = p.q_bf16 + (size_t)tile * kRows * (kDQK / 8);
      uint4* dst = reinterpret_cast<uint4*>(p.q_codes + (size_t)((j & 1) * ncta + cid) * kSlot);
      // The Q of the item behind that into L2 -- with short items only, whose pace these loads' latency bounds (1184 tokens x 64
      // heads, top-256 82.3 -> 78.0 us; top-2048 199.5 -> 202.6).
      if (ahead && e_tid == 0 && behind < ng)
        l2_prefetch_1d(p.q_bf16 + (size_t)tile_at(behind, item_at(behind).x) * kRows * (kDQK / 8), kRows * kDQK * 2);
      // 64 rows x 36 units of 16 codes = 18 units per thread, six under way: a unit's registers take the next one's loads as
      // soon as its codes are on their way
      uint4 a[kFillBatch], b[kFillBatch];
      auto load = [&](int u, int unit) {
        a[u] = __ldcs(src + 2 * unit);
        b[u] = __ldcs(src + 2 * unit + 1);
      };
#pragma unroll
      for (int u = 0; u < kFillBatch; ++u) load(u, u * 128 + e_tid);
#pragma unroll 1
      for (int i = 0; i < 18; i += kFillBatch) {
#pragma unroll
        for (int u = 0; u < kFillBatch; ++u) {
          const int unit = (i + u) * 128 + e_tid;
          dst[unit] = make_uint4(e4m3x4_of_bf16(a[u].x, a[u].y, p.q_inv), e4m3x4_of_bf16(a[u].z, a[u].w, p.q_inv),
                                 e4m3x4_of_bf16(b[u].x, b[u].y, p.q_inv), e4m3x4_of_bf16(b[u].z, b[u].w, p.q_inv));
          if (i + kFillBatch < 18) load(u, unit + kFillBatch * 128);
        }
      }
      __threadfence();
      asm volatile("fence.proxy.async;" ::: "memory");      // these stores -> the TMA loads of the codes
      asm volatile("bar.sync 5, 128;" ::: "memory");
      if (e_tid == 0) mbar_arrive(&ms.q_codes);
    };
    auto transfer_q = [&](int j, int n) {
      if (j > 0) mbar_wait(&ms.q_free, (j - 1) & 1, wt, kSiteQFree, j);
      mbar_wait(&ms.q_land, j & 1, wt, kSiteQ, j);
      __syncwarp();
      tc_fence_after();
      const uint8_t* qtile = sm + kOffKV + (n % kSlots) * kSlot;
      const uint8_t* qrow = qtile + e_r * 128;
      // rope chunk: 4 KB, 32 bytes per thread
      reinterpret_cast<uint4*>(sm + kOffRope)[e_tid] = reinterpret_cast<const uint4*>(qtile + kQLatent)[e_tid];
      reinterpret_cast<uint4*>(sm + kOffRope)[e_tid + 128] = reinterpret_cast<const uint4*>(qtile + kQLatent)[e_tid + 128];
#pragma unroll 1
      for (int j4 = 0; j4 < 4; ++j4) {
        uint32_t v[32];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const uint4 t = *reinterpret_cast<const uint4*>(qrow + j4 * kChunkBytes + ((u ^ (e_r & 7)) << 4));
          v[4 * u] = t.x; v[4 * u + 1] = t.y; v[4 * u + 2] = t.z; v[4 * u + 3] = t.w;
        }
        tmem_st32(tmem + lane_base + kTmemQ + 32 * j4, reinterpret_cast<const float*>(v));
      }
      tmem_wait_st();
      tc_fence_before();
      fence_proxy_async_smem();      // rope -> the MMAs' reads; these reads -> the slot's next TMA write
      __syncwarp();
      if (lane == 0) mbar_arrive(&ms.qt_ready);
      asm volatile("bar.sync 5, 128;" ::: "memory");      // all warps have read the slot
      if (e_tid == 0) mbar_arrive(&ms.q_taken);
    };
    // the slot of entry n is dead (its TMA reads included)
    auto release = [&](int n) {
      if (lane == 0) bulk_wait_read_all();
      __syncwarp();
      asm volatile("bar.sync 5, 128;" ::: "memory");
      if (e_tid == 0) mbar_arrive(&ms.slot_free[n % kSlots]);
    };
    int kb0 = 0, it = 0;
    Next next = next_at(cid);
    if (p.q_bf16 != nullptr) quantise_q(tile_at(cid, next.tile), 0, false, 0);
    transfer_q(0, 0);
    release(0);
    for (int i = cid; i < ng; i += ncta, ++it) {
      const int tile = tile_at(i, next.tile), nb = next.nb, kbl = kb0 + nb - 1;           // last block of the item
      next = next_at(i + ncta);
      const int n = kb0 + nb + it + 1;             // entry number of the next item's Q
      if (i + ncta < ng) {
        if (p.q_bf16 != nullptr) quantise_q(tile_at(i + ncta, next.tile), it + 1, nb <= 12, i + 2 * ncta);
        transfer_q(it + 1, n);
      } else {
        mbar_wait(&ms.q_land, (it + 1) & 1, wt, kSiteQ, it + 1);      // an empty entry
      }
      // row sums of the groups, in the order of the item's first blocks (whichever group served them), so that
      // a tile's result does not depend on what its CTA processed before
      mbar_wait(&ms.fin_ready, it & 1, wt, kSiteEpi, it);
      __syncwarp();
      const float m = ms.fin_m[kbl & (kGroups - 1)][e_r];
      float li = 0.f;
#pragma unroll
      for (int j = 0; j < kGroups; ++j) {
        const int gg = (kb0 + j) & (kGroups - 1);
        li += (ms.fin_l[gg][e_r] + ms.fin_l[gg][e_r + 64]) * fast_exp2(ms.fin_m[gg][e_r] - m);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&ms.fin_free);
      if (e_h == 0) p.lse[(size_t)tile * kRows + e_r] = li > 0.f ? __logf(li) - kPScaleLn + m * kLn2 : INFINITY;
      const float oscale = li > 0.f ? __fdividef(p.out_scale, li) : 0.f;
      const bool no_key = oscale == 0.f, some_no_key = __any_sync(0xffffffffu, no_key);
      const uint64_t os2 = pack2(oscale, oscale);
      mbar_wait(&ms.pv_done[kbl & 7], (kbl >> 3) & 1, wt, kSiteEpi, nb);
      __syncwarp();
      tc_fence_after();
      // this warp's 32 rows of the tile = (token, head) pairs starting at row r0
      const int r0 = 32 * (warp & 1);
      const int out_head = r0 % p.h_per_q, out_tok = tile * p.G + r0 / p.h_per_q;
      const uint32_t stage = kOffKV + (uint32_t)(n % kSlots) * kSlot + (uint32_t)ew * 8192;
      // Four boxes of 32 rows x 64 dims (128-byte swizzle) leave through the warp's two 4 KB pieces of the slot; each
      // is in registers before it waits until the one before last has been read out
#pragma unroll 1
      for (int x = 0; x < 4; ++x) {
        uint32_t wv[32];
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {      // 64 columns, scaled and rounded
          float o[32];
          tmem_ld32(e_ocol + 64 * x + 32 * cc, o);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float2 v = unpack2(mul2(pack2(o[2 * j], o[2 * j + 1]), os2));
            const __nv_bfloat162 v2 = __floats2bfloat162_rn(v.x, v.y);
            wv[16 * cc + j] = *reinterpret_cast<const uint32_t*>(&v2);
          }
        }
        if (some_no_key) {      // rows without a valid key: zeros, whatever O holds
#pragma unroll
          for (int j = 0; j < 32; ++j) wv[j] = no_key ? 0u : wv[j];
        }
        if (x == 3) {           // O has been read: the next item's first PV may overwrite it
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ms.o_free);
        }
        if (x >= 2 && lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        __syncwarp();
        const uint32_t piece = stage + (x & 1) * 4096;
        uint8_t* st_row = sm + piece + lane * 128;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          *reinterpret_cast<uint4*>(st_row + ((j ^ (lane & 7)) << 4)) = make_uint4(wv[4 * j], wv[4 * j + 1], wv[4 * j + 2], wv[4 * j + 3]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          // dims 256 (x / 2) + 128 e_h + 64 (x % 2)
          tma_store_3d_hint(&map_out, sbase + piece, 256 * (x >> 1) + 128 * e_h + 64 * (x & 1), out_head, out_tok, pol_stream);
          bulk_commit_group();
        }
      }
      release(n);
      kb0 += nb;
    }
    if (lane == 0) bulk_wait_all();   // output boxes written before the CTA retires
    tc_fence_before();
  }

  __syncthreads();
  if (ms.left != 0) {
    cp_async_wait_all();
    if (threadIdx.x == 0) {
      if (ms.q_asked != 0) {      // the last Q requested: with the arrivals of the warps that have left it counts as landed when it has
        for (int i = 0; i < kGatherWarps; ++i)
          if (ms.q_passed[i] < ms.q_asked) mbar_arrive(&ms.q_land);
        mbar_drain(&ms.q_land, (ms.q_asked - 1) & 1);
      }
      for (int i = 0; i < 2; ++i) {      // block 2 (n - 1) + i was the warp's last
        const uint32_t kb = 2 * (ms.qk_end[i] - 1) + i;
        if (ms.qk_end[i] != 0) mbar_drain(&ms.qk_done[kb & 7], (kb >> 3) & 1);
      }
      if (ms.pv_end != 0) mbar_drain(&ms.pv_done[(ms.pv_end - 1) & 7], ((ms.pv_end - 1) >> 3) & 1);
    }
  }
  __syncwarp();
  if (warp == kWarpQk) tmem_dealloc_cta(tmem, kTmemCols);
  if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&g_attn_status[3], 1);
  if (threadIdx.x == 0) wt.report(g_attn_status, p.epoch);
}
#undef LT_WS_TS
#undef LT_WS_SS
#undef LT_WS_PV

}  // namespace r64

// One launch over the 64-row tiles of dense q [T, h, 576] (ng = T h / 64).  a.nsplit, sinks, strides of q / out and
// further destinations are not supported here.  With one token per tile every list entry is every row's.  q_codes:
// rows64_scratch() bytes, used with bf16 queries.  order: see Params.
int64_t rows64_scratch(int ng) { return (int64_t)2 * min(ng, sm_count()) * r64::kSlot; }
int run_fp8_rows64(const Fp8Args& a, void* out, void* q_codes, const int2* order, void* stream) {
  Fp8Args c = a;
  if (a.h_per_q == r64::kRows) c.memb_qm = reinterpret_cast<const uint32_t*>(a.indices);      // none there, and none read
  const int rc = check_fp8_args(c);
  if (rc != LITEDSA_OK) return rc;
  if (a.h_per_q > r64::kRows || a.topk < 256 || ((uintptr_t)out & 15)) return LITEDSA_ERR_UNSUPPORTED;
  CUtensorMap map_q, map_q_rope, map_out;
  const int h = a.h_per_q, G = r64::kRows / h;
  const uint64_t tokens = (uint64_t)a.ng * G;
  const uint32_t ob_h = (uint32_t)min(h, 32);
  const int ncta = min(a.ng, sm_count());
  if (!make_map_3d(&map_out, out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, kDV, (uint64_t)h, tokens, kDV * 2, (uint64_t)h * kDV * 2,
                   64, ob_h, 32 / ob_h, CU_TENSOR_MAP_SWIZZLE_128B))
    return LITEDSA_ERR_CUDA;
  // Q: boxes of 64 rows x 128 bytes (128-byte swizzle) and the rope box of 64 rows x 64 bytes (64-byte swizzle)
  const void* q = a.q_is_bf16 ? q_codes : a.q8;
  const uint32_t qh = a.q_is_bf16 ? (uint32_t)r64::kRows : (uint32_t)h;
  const uint64_t qz = a.q_is_bf16 ? (uint64_t)2 * ncta : tokens;
  if (!make_map_3d(&map_q, q, CU_TENSOR_MAP_DATA_TYPE_UINT8, kDQK, qh, qz, kDQK, (uint64_t)qh * kDQK, 128, qh, r64::kRows / qh) ||
      !make_map_3d(&map_q_rope, q, CU_TENSOR_MAP_DATA_TYPE_UINT8, kDQK, qh, qz, kDQK, (uint64_t)qh * kDQK, 64, qh, r64::kRows / qh,
                   CU_TENSOR_MAP_SWIZZLE_64B))
    return LITEDSA_ERR_CUDA;
  r64::Params p;
  p.memb = G > 1 ? a.memb_qm : nullptr; p.indices = a.indices; p.counts = a.topk_length; p.order = order;
  p.kv = reinterpret_cast<const uint8_t*>(a.kv8); p.kv_pitch = a.kv_row_stride;
  p.lse = a.lse;
  p.ng = a.ng; p.s_kv = a.s_kv; p.cap = a.topk; p.h_per_q = h; p.G = G;
  p.scale_log2 = a.sm_scale * kLog2e; p.out_scale = a.out_scale;
  p.epoch = next_launch_epoch(); p.wait_limit = wait_limit_ticks();
  p.q_bf16 = a.q_is_bf16 ? reinterpret_cast<const uint4*>(a.q8) : nullptr; p.q_inv = a.q_inv;
  p.q_codes = reinterpret_cast<uint8_t*>(q_codes);
  const bool wide = (int64_t)a.s_kv * (a.kv_row_stride >> 4) >= 0xffffffffll;
  const int dev = current_device();
  auto launch = [&](auto is_wide, auto is_ordered) -> int {
    constexpr auto kern = r64::masked_mla_fp8_r64_kernel<decltype(is_wide)::value, decltype(is_ordered)::value>;
    if (!ensure_smem<kern>(dev, r64::Plan::kSmem)) return LITEDSA_ERR_CUDA;
    return launch_pdl(kern, dim3((unsigned)ncta), r64::kThreads, r64::Plan::kSmem, reinterpret_cast<cudaStream_t>(stream), map_q, map_q_rope,
                      map_out, p);
  };
  using Yes = std::true_type;
  using No = std::false_type;
  return order != nullptr ? (wide ? launch(Yes{}, Yes{}) : launch(No{}, Yes{})) : (wide ? launch(Yes{}, No{}) : launch(No{}, No{}));
}

}  // namespace lt
