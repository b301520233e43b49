// The step before the union: index logits and top-k selection (sm_100a).
//
// The reference repository no longer carries its indexer ("The repository-local LiteTopK
// indexer and standalone MS MARCO top-k kernels have been removed", README.md:3-6); what its
// attention path consumes is the result, `topk_indices [T, k] i32` with -1 padding
// (kernels/b200/dsa/litedsa.cu:31-33).  This file produces that tensor from the published
// formulation of the DeepSeek-V3.2 lightning indexer in its FP8 form:
//
//   logit[t, s] = k_scale[s] * sum_h  weights[t, h] * relu( q8[t, h, :] . k8[s, :] )     (s <= pos(t))
//   topk_idx[t, :] = the k positions s <= pos(t) with the largest logits (all of them and -1
//                    padding when fewer than k exist)
//
// with q8 [T, Hi, 128] and k8 [S, 128] e4m3 codes, weights [T, Hi] fp32 (head weight x query
// scale x softmax scale), k_scale [S] fp32 and pos(t) = q_pos0 + t.  Nothing here has a
// counterpart in the reference to be checked against; the CPU oracle restates the formula.
//
// index_logits_kernel (tensor-bound): the product is computed TRANSPOSED, keys on the M axis,
// so that the head sum of a (token, key) pair is a sum along one accumulator row.  One CTA owns
// 512 / Hi tokens: their q rows are the B operand of four N = 128 accumulators (512 TMEM columns);
// the K tiles (128 keys x 128 bytes, TMA, four stages) are the A operand and are streamed once per
// CTA, up to the causal bound of its last token.  While the tensor core fills one accumulator,
// sixteen warps (accumulator x lane quarter) drain the others: tcgen05.ld, relu, multiply by the head
// weight, add; then x k_scale, causal mask, and 128 consecutive fp32 logits per token leave each warp
// as coalesced stores.  The drain paces the kernel (2070 cycles per key tile, of which the MMAs need
// 1024): 4096 tokens x 32768 keys x 64 heads 934 us; 966 with two N = 256 accumulators, weights from shared
// memory and the warps of a scheduler in two phases instead of four.
//
// topk_select (memory-bound): exact selection per token row.  Rows up to 32768 entries go
// through persistent CTAs that prefetch the next row with a bulk copy while the current one
// is processed from registers (value-linear histogram, exact ranking of the threshold bin);
// longer rows through a radix select over the order-preserving integer image of the logits.
// Ties at the k-th value are resolved towards the smaller position, so the selected set is
// deterministic; the order inside a row is not specified.
#include "common.cuh"
#include "tensor_map.cuh"

namespace lt {
namespace idx {

// ------------------------------------------------------------------ index logits
constexpr int kThreads = 576;             // TMA and MMA warps + 16 drain warps
constexpr int kDrainWarp0 = 2;
constexpr int kKeyTile = 128;             // keys per MMA (M)
constexpr int kCols = 128;                // (token, head) columns per accumulator (N)
constexpr int kAccs = 4;                  // accumulators: all 512 TMEM columns
constexpr int kDim = 128;                 // index head dim = bytes per row
constexpr int kStages = 4;
constexpr uint32_t kQTile = kCols * kDim;       // 16 KB
constexpr uint32_t kKTile = kKeyTile * kDim;    // 16 KB
constexpr uint32_t kOffQ = 0;
constexpr uint32_t kOffK = kOffQ + kAccs * kQTile;
constexpr uint32_t kOffW = kOffK + kStages * kKTile;
constexpr uint32_t kOffBar = kOffW + kAccs * kCols * 4;
constexpr uint32_t kSmem = kOffBar + 256 + 1024;   // + alignment slack

struct Bars {
  uint64_t q_full, k_full[kStages], k_free[kStages], acc_full[kAccs], acc_free[kAccs];
  uint32_t tmem_base;
};
static_assert(sizeof(Bars) <= 256, "barrier block too large");

struct LogitParams {
  const float* weights;     // [T, Hi]
  const float* k_scale;     // [S] or null (1.0)
  float* logits;            // [T, ld]
  int T, Hi, S, q_pos0;
  int live_tiles;           // key tiles up to the last token's causal bound
  int tiles_per_split;      // of these, blockIdx.y owns tiles [y * this, (y + 1) * this)
  long long ld;
  int epoch;
  unsigned long long wait_limit_ns;
};

enum { kSiteQFull = 1, kSiteKFull, kSiteKFree, kSiteAccFull, kSiteAccFree };

// packed fp32 pair fma (one issue slot for two lanes of work)
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)),
        "l"(reinterpret_cast<unsigned long long&>(c)));
  return d;
}

__device__ int g_status[8];

__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
  return e != 0;
}

// accs: accumulators in use, a CTA's tokens are accs * 128 / HI (a run-time number costs spills)
template <int HI, int accs>
__global__ void __launch_bounds__(kThreads, 1)
index_logits_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                    const LogitParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sbase = (raw + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (sbase - raw);
  float* wsm = reinterpret_cast<float*>(sm + kOffW);
  Bars& bar = *reinterpret_cast<Bars*>(sm + kOffBar);
  const Waiter wt{g_status, p.epoch, p.wait_limit_ns};

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  constexpr int tpa = kCols / HI;               // tokens per accumulator
  const int tok0 = blockIdx.x * accs * tpa;     // first token of this CTA
  const int tok_end = min(p.T, tok0 + accs * tpa);
  // key tiles up to the causal bound of the CTA's last token, and this CTA's share [j0, j0 + n)
  const int pos_max = p.q_pos0 + tok_end - 1;
  const int all_tiles = (p.S + kKeyTile - 1) / kKeyTile;
  const int causal_tiles = min(all_tiles, pos_max / kKeyTile + 1);
  const int j0 = blockIdx.y * p.tiles_per_split, j_end = min(j0 + p.tiles_per_split, p.live_tiles);
  const int n_tiles = max(min(j_end, causal_tiles) - j0, 0);

  if (threadIdx.x == 0) {
    mbar_init(&bar.q_full, 1);
    for (int i = 0; i < kStages; ++i) { mbar_init(&bar.k_full[i], 1); mbar_init(&bar.k_free[i], 1); }
    for (int i = 0; i < kAccs; ++i) { mbar_init(&bar.acc_full[i], 1); mbar_init(&bar.acc_free[i], 4); }
    fence_mbar_init();
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_k);
  }
  pdl_trigger();
  pdl_wait();
  // head weights of the CTA's tokens: column c of accumulator a is row tok0 * Hi + 128 a + c.
  // Halved: the drain computes relu(x) as (x + |x|) / 2 with the division folded in here.
  for (int i = threadIdx.x; i < kAccs * kCols; i += kThreads) {
    const long long r = (long long)tok0 * HI + i;
    wsm[i] = r < (long long)p.T * HI ? 0.5f * __ldcg(p.weights + r) : 0.f;
  }
  __syncthreads();
  if (warp == 0) {
    tmem_alloc_cta(&bar.tmem_base, 512);
    tmem_relinquish_cta();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bar.tmem_base;

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0 && n_tiles > 0) {
      const uint64_t pol_keep = l2_policy_evict_last(), pol_stream = l2_policy_evict_first();
      mbar_arrive_expect_tx(&bar.q_full, accs * kQTile);
      for (int a = 0; a < accs; ++a)
        tma_load_2d_hint(sbase + kOffQ + a * kQTile, &map_q, 0, tok0 * HI + a * kCols, &bar.q_full, pol_stream);
      for (int j = 0; j < n_tiles; ++j) {
        const int s = j % kStages;
        if (j >= kStages && !mbar_wait(&bar.k_free[s], ((j / kStages) & 1) ^ 1, wt, kSiteKFree, j)) break;
        mbar_arrive_expect_tx(&bar.k_full[s], kKTile);
        tma_load_2d_hint(sbase + kOffK + s * kKTile, &map_k, 0, (j0 + j) * kKeyTile, &bar.k_full[s], pol_keep);
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issue (one elected thread)
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc(0, 0, false, false, kKeyTile, kCols);
      bool ok = n_tiles > 0 && mbar_wait(&bar.q_full, 0, wt, kSiteQFull, 0);
      for (int j = 0; j < n_tiles && ok; ++j) {
        const int s = j % kStages;
        ok = mbar_wait(&bar.k_full[s], (j / kStages) & 1, wt, kSiteKFull, j);
        if (!ok) break;
        const uint64_t ad = umma_desc(sbase + kOffK + s * kKTile, 16, 1024, kSwz128);
        for (int a = 0; a < accs && ok; ++a) {
          // accumulator a still holds tile j-1 until its four warps have read it
          if (j > 0) ok = mbar_wait(&bar.acc_free[a], (j - 1) & 1, wt, kSiteAccFree, j);
          if (!ok) break;
          tc_fence_after();
          const uint64_t bd = umma_desc(sbase + kOffQ + a * kQTile, 16, 1024, kSwz128);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            mma_f8_cta(tmem + a * kCols, ad + 2 * kk, bd + 2 * kk, idesc, kk ? 1u : 0u);
          mma_commit_cta(&bar.acc_full[a]);
        }
        mma_commit_cta(&bar.k_free[s]);     // all accumulators have read the K tile
      }
    }
    __syncwarp();
  } else if (warp < kDrainWarp0 + 4 * accs) {
    // ---------------------------------------------------------------- accumulator drain
    // Sixteen warps: accumulator a, TMEM lane quarter q4.  The four warps of one scheduler (one lane
    // quarter) serve four accumulators, which are filled in turn, so that they are in different phases:
    // with two accumulators of 256 columns the warps waited, multiplied and reduced in lockstep.
    // relu(x) * w is computed as (x + |x|) * (w / 2): an add with an absolute-value operand and a
    // packed fma, both on the fma pipe (a max would go to the half-rate integer pipe).
    // The accumulator is read as 16 x 256-bit fragments: lane l gets columns 8 i + 2 (l % 4) + {0, 1}
    // of rows l / 4 and l / 4 + 8, so it needs a quarter of the weights and keeps them in registers.
    // (With one key row per lane every lane needs every weight; as 16-byte broadcasts from shared
    // memory those take 1024 of its cycles per key tile, beside 1024 for the MMAs' operands.)
    const int a = (warp - kDrainWarp0) >> 2, q4 = warp & 3;
    // the key row whose sums this lane ends up with (below)
    const int krow = 32 * q4 + 16 * ((lane >> 1) & 1) + 8 * (lane & 1) + (lane >> 2);
    const uint32_t tcol = tmem + ((uint32_t)(32 * q4) << 16) + a * kCols;
    const int t_base = tok0 + a * tpa;
    float2 w[kCols / 8];                                // columns 8 i + 2 (lane % 4) + {0, 1}
#pragma unroll
    for (int i = 0; i < kCols / 8; ++i)
      w[i] = *reinterpret_cast<const float2*>(wsm + a * kCols + 8 * i + 2 * (lane & 3));
    // Key tiles beyond the causal bound of the CTA's last token are not computed: their entries
    // are -inf for every token of the CTA (this warp's tokens and key rows).  Written first,
    // while the tensor core fills the first accumulators: those of the CTA's own range, and its share of
    // the tiles beyond every token's bound.
    auto fill = [&](int ja, int jb) {
      for (int j = ja; j < jb; ++j) {
        const int s_key = j * kKeyTile + krow;
        if (s_key < p.S) {
#pragma unroll
          for (int tt = 0; tt < tpa; ++tt)
            if (t_base + tt < p.T) p.logits[(long long)(t_base + tt) * p.ld + s_key] = -INFINITY;
        }
      }
    };
    fill(j0 + n_tiles, j_end);
    const long long dead = all_tiles - p.live_tiles;
    fill(p.live_tiles + (int)(dead * blockIdx.y / gridDim.y), p.live_tiles + (int)(dead * (blockIdx.y + 1) / gridDim.y));
    // tiles below this one lie inside the cache and inside every token's causal bound
    const int j_plain = min(p.S, p.q_pos0 + tok0 + 1) / kKeyTile - j0;
    const bool all_toks = t_base + tpa <= p.T;
    auto scale_of = [&](int j) -> float {
      const int s_key = (j0 + j) * kKeyTile + krow;
      return (p.k_scale && s_key < p.S) ? __ldcg(p.k_scale + s_key) : 1.f;
    };
    float* out = p.logits + (long long)t_base * p.ld + (long long)j0 * kKeyTile + krow;
    float ks_next = n_tiles > 0 ? scale_of(0) : 1.f;    // fetched a tile ahead
    for (int j = 0; j < n_tiles; ++j, out += kKeyTile) {
      const float ks = ks_next;
      if (j + 1 < n_tiles) ks_next = scale_of(j + 1);
      const bool landed = mbar_wait(&bar.acc_full[a], j & 1, wt, kSiteAccFull, j);
      if (!__all_sync(0xffffffffu, landed)) break;
      tc_fence_after();
      // step m: 32 columns (chunk m / 2) of 16 rows (half m % 2).  One packed chain per row, carried
      // over the chunks of a token (a chunk never straddles two tokens).
      float acc[tpa];
      float x[2][16];
      float2 sum[2][2];                                 // [row half][row l / 4, + 8]
      tmem_ld_16x256b_x4(tcol, x[0]);
#pragma unroll
      for (int m = 0; m < kCols / 16; ++m) {
        const int c = m >> 1, rh = m & 1;
        tmem_wait_ld();
        if (m + 1 < kCols / 16) {
          tmem_ld_16x256b_x4(tcol + 32 * ((m + 1) >> 1) + ((uint32_t)(16 * ((m + 1) & 1)) << 16), x[(m + 1) & 1]);
        } else {
          tc_fence_before();                            // everything has been read
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar.acc_free[a]);
        }
        const float* xc = x[m & 1];
        if ((32 * c) % HI == 0) sum[rh][0] = sum[rh][1] = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          sum[rh][0] = fma2(make_float2(xc[4 * i] + fabsf(xc[4 * i]), xc[4 * i + 1] + fabsf(xc[4 * i + 1])),
                            w[4 * c + i], sum[rh][0]);
          sum[rh][1] = fma2(make_float2(xc[4 * i + 2] + fabsf(xc[4 * i + 2]), xc[4 * i + 3] + fabsf(xc[4 * i + 3])),
                            w[4 * c + i], sum[rh][1]);
        }
        if (rh == 1 && (32 * (c + 1)) % HI == 0) {
          // the four lanes of a row group hold a quarter of the columns each; two exchanges leave
          // lane l with the whole sum of row 16 (l / 2 % 2) + 8 (l % 2) + l / 4
          float v[2];
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const float lo = sum[r][0].x + sum[r][0].y, hi = sum[r][1].x + sum[r][1].y;
            v[r] = ((lane & 1) ? hi : lo) + __shfl_xor_sync(0xffffffffu, (lane & 1) ? lo : hi, 1);
          }
          acc[(32 * c) / HI] = ((lane & 2) ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, (lane & 2) ? v[0] : v[1], 2);
        }
      }
      // scale, causal mask, store: the lanes of a warp hold 32 consecutive keys
      if (j < j_plain && all_toks) {
#pragma unroll
        for (int tt = 0; tt < tpa; ++tt) out[tt * p.ld] = acc[tt] * ks;
      } else {
        const int s_key = (j0 + j) * kKeyTile + krow;
#pragma unroll
        for (int tt = 0; tt < tpa; ++tt) {
          const int t = t_base + tt;
          if (t < p.T && s_key < p.S) out[tt * p.ld] = s_key <= p.q_pos0 + t ? acc[tt] * ks : -INFINITY;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    tmem_dealloc_cta(tmem, 512);
  }
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) atomicAdd(&g_status[3], 1);
}

template <int N> struct Int { static constexpr int value = N; };

// How many key ranges the grid splits every token group's keys into.  A CTA occupies an SM by
// itself (all of TMEM) and works about one unit of time per key tile -- less with fewer accumulators in use -- after a start-up
// worth about four (TMEM and barrier set-up, the 64 KB of Q, the first K tile), so the launch takes
// waves(ctas_x * splits) * (4 + tiles per split): few tokens need many splits to fill the SMs (36
// tokens of 32 heads are 3 CTAs: 867 -> 22 us against 100K keys), many tokens a few so that the
// last wave is full.  The tiles beyond every token's position are only filled with -inf, at about a 90th of
// a unit per tile and token of the CTA, and shared out among the same CTAs.  (A CTA per range of the
// whole cache paid the start-up for each of them: 150 tokens of 128 heads at position 0 of 131072
// 507 us; with ranges of the live tiles alone 20.)
static int pick_splits(int ctas_x, int live, int dead, int tok_per_cta, int accs, int sms) {
  int best = 1;
  long long best_cost = -1;
  for (int n = 1; n <= 64 && n <= live + dead; ++n) {
    const int per = (live + n - 1) / n;
    const long long ranges = dead > 0 ? n : (live + per - 1) / per;      // CTAs with something to do
    const long long waves = (ctas_x * ranges + sms - 1) / sms;
    const long long cost = waves * (90LL * 4 + 18LL * (accs + 1) * per + (long long)((dead + n - 1) / n) * tok_per_cta);
    if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = n; }
  }
  return best;
}

// ------------------------------------------------------------------ top-k selection
constexpr int kBins = 2048;
constexpr int kMaxSmemRow = 49152;       // keys of a row held in shared memory (192 KB)
constexpr int kCandCap = 4096;           // keys of the threshold bin kept in shared memory

struct SelParams {
  const float* logits;      // [T, ld]
  const int32_t* lengths;   // [T] valid prefix per row, or null: min(S, q_pos0 + t + 1)
  int32_t* out;             // [T, k]
  int T, S, k, q_pos0;
  long long ld;
  int epoch;
  unsigned long long wait_limit_ns;
};

// order-preserving map fp32 -> u32 (NaN sorts lowest, -0 and +0 share one key) and its inverse
__device__ __forceinline__ uint32_t okey(float f) {
  if (f != f) return 0u;
  const uint32_t b = f == 0.f ? 0u : __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float okey_inv(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

struct SelShared {
  uint32_t hist[kBins];
  uint32_t cand[kCandCap];
  uint32_t wa[32], wb[32];
  uint32_t sel_bin, sel_rem, n_cand, kth, ties;
};

// block-wide max / min of two values (all threads get the result); ends with a barrier
template <int NT>
__device__ __forceinline__ void block_max_min(SelShared& sh, uint32_t& vmax, uint32_t& vmin) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    vmax = max(vmax, __shfl_xor_sync(0xffffffffu, vmax, off));
    vmin = min(vmin, __shfl_xor_sync(0xffffffffu, vmin, off));
  }
  if (lane == 0) { sh.wa[wid] = vmax; sh.wb[wid] = vmin; }
  __syncthreads();
  uint32_t a = lane < NT / 32 ? sh.wa[lane] : 0u, b = lane < NT / 32 ? sh.wb[lane] : 0xffffffffu;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    a = max(a, __shfl_xor_sync(0xffffffffu, a, off));
    b = min(b, __shfl_xor_sync(0xffffffffu, b, off));
  }
  vmax = a; vmin = b;
  __syncthreads();
}

// Block-wide: given hist[0 .. kBins) and `rem`, find the bin b with count(bins > b) < rem <=
// count(bins >= b); returns b and the rank inside the bin (rem - count(bins > b)).  Thread i
// owns kBins / NT consecutive bins.  Ends with a barrier; hist may be reused afterwards.
template <int NT>
__device__ __forceinline__ uint32_t find_bin(SelShared& sh, uint32_t rem, uint32_t* rem_out) {
  constexpr int BPT = kBins / NT;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  uint32_t h[BPT], mine = 0;
#pragma unroll
  for (int i = 0; i < BPT; ++i) { h[i] = sh.hist[BPT * tid + i]; mine += h[i]; }
  uint32_t incl = mine;                      // inclusive suffix sum within the warp (towards higher lanes)
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t v = __shfl_down_sync(0xffffffffu, incl, off);
    if (lane + off < 32) incl += v;
  }
  if (lane == 0) sh.wa[wid] = incl;
  __syncthreads();
  // suffix sum over the warp totals (every warp computes it; NT / 32 <= 32 entries)
  uint32_t wt = lane < NT / 32 ? sh.wa[lane] : 0u, wsuf = wt;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t v = __shfl_down_sync(0xffffffffu, wsuf, off);
    if (lane + off < 32) wsuf += v;
  }
  const uint32_t above_warps = __shfl_sync(0xffffffffu, wsuf - wt, wid);   // totals of the higher warps
  uint32_t above = above_warps + incl - mine;                             // + higher lanes of my warp
  if (above < rem && rem <= above + mine) {  // the crossing is in my bins: walk them from the top
    int b = BPT - 1;
#pragma unroll
    for (int i = BPT - 1; i > 0; --i)
      if (b == i && above + h[i] < rem) { above += h[i]; b = i - 1; }
    sh.sel_bin = (uint32_t)(BPT * tid + b);
    sh.sel_rem = rem - above;
  }
  __syncthreads();
  *rem_out = sh.sel_rem;
  const uint32_t bsel = sh.sel_bin;
  __syncthreads();
  return bsel;
}

// Block-wide exact radix select over m keys get(0 .. m): the rem-th largest key and how many
// keys equal to it belong to the top rem.  Digits of up to 11 bits, most significant first,
// starting at the highest bit in which kmax and kmin (the range of the keys) differ.
template <int NT, class Get>
__device__ __forceinline__ uint32_t radix_kth(SelShared& sh, Get get, int m, uint32_t kmax, uint32_t kmin,
                                              uint32_t rem, uint32_t* ties_out) {
  const int tid = threadIdx.x;
  const int top = kmax == kmin ? -1 : 31 - __clz(kmax ^ kmin);
  uint32_t prefix_mask = top < 0 ? 0xffffffffu : (top >= 31 ? 0u : ~((2u << top) - 1u));
  uint32_t prefix = kmax & prefix_mask;
  int hi = top;                              // highest bit not yet decided
#pragma unroll 1
  while (hi >= 0) {
    const int bits = min(11, hi + 1);
    const int shift = hi + 1 - bits;
    const uint32_t dmask = (1u << bits) - 1u;
    for (int i = tid; i < kBins; i += NT) sh.hist[i] = 0;
    __syncthreads();
    for (int i = tid; i < m; i += NT) {
      const uint32_t u = get(i);
      if ((u & prefix_mask) == prefix) atomicAdd(&sh.hist[(u >> shift) & dmask], 1u);
    }
    __syncthreads();
    const uint32_t b = find_bin<NT>(sh, rem, &rem);
    prefix |= b << shift;
    prefix_mask |= dmask << shift;
    hi = shift - 1;
  }
  *ties_out = rem;
  return prefix;
}

// Block-wide ordered emission: out[slot] = i for every selected position i, ascending, where
// selected = key > kth, or key == kth and fewer than `ties` equal keys precede it.  Warp w owns
// a contiguous segment of the row; slot = #greater before i + min(#equal before i, ties).
template <int NT, class Get>
__device__ __forceinline__ void emit_ordered(SelShared& sh, Get key_at, int n, uint32_t kth, uint32_t ties,
                                             int32_t* out, int k) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int seg = (((n + NT / 32 - 1) / (NT / 32)) + 31) & ~31;
  const int s0 = min(wid * seg, n), s1 = min(s0 + seg, n);
  uint32_t cgt = 0, ceq = 0;
  for (int i = s0 + lane; i < s1; i += 32) {
    const uint32_t u = key_at(i);
    cgt += u > kth;
    ceq += u == kth;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    cgt += __shfl_xor_sync(0xffffffffu, cgt, off);
    ceq += __shfl_xor_sync(0xffffffffu, ceq, off);
  }
  __syncthreads();
  if (lane == 0) { sh.wa[wid] = cgt; sh.wb[wid] = ceq; }
  __syncthreads();
  uint32_t gt_run = 0, eq_run = 0;
  for (int w = 0; w < wid; ++w) { gt_run += sh.wa[w]; eq_run += sh.wb[w]; }
  const uint32_t lt_mask = (1u << lane) - 1u;
  for (int i0 = s0; i0 < s1; i0 += 32) {
    const int i = i0 + lane;
    const uint32_t u = i < s1 ? key_at(i) : 0u;
    const bool gt = i < s1 && u > kth, eq = i < s1 && u == kth;
    const uint32_t bg = __ballot_sync(0xffffffffu, gt), be = __ballot_sync(0xffffffffu, eq);
    const uint32_t gt_before = gt_run + __popc(bg & lt_mask);
    const uint32_t eq_before = eq_run + __popc(be & lt_mask);
    if (gt || (eq && eq_before < ties)) {
      const uint32_t slot = gt_before + min(eq_before, ties);
      if (slot < (uint32_t)k) out[slot] = i;
    }
    gt_run += __popc(bg);
    eq_run += __popc(be);
  }
}

// One CTA per row, rows of any length and alignment: the exact bitwise radix select over the
// row's order-preserving keys (kept in shared memory when they fit, re-read from memory by
// every pass otherwise) and the ordered emission.  This is the path for logits tensors whose
// rows are not 16-byte aligned; aligned rows go through the streaming kernels below, which fall
// back to the same two steps whenever their fast path does not apply.
constexpr int kGenericThreads = 1024;
template <bool kSmemRow>
__global__ void __launch_bounds__(kGenericThreads)
topk_select_kernel(const SelParams p) {
  constexpr int NT = kGenericThreads;
  extern __shared__ __align__(16) uint32_t rowkeys[];
  __shared__ SelShared sh;
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x, tid = threadIdx.x;
  const int n = p.lengths ? min(max(p.lengths[t], 0), p.S) : min(p.S, max(p.q_pos0 + t + 1, 0));
  int32_t* out = p.out + (long long)t * p.k;
  const float* row = p.logits + (long long)t * p.ld;
  if (n <= p.k) {            // everything valid is selected
    for (int i = tid; i < p.k; i += NT) out[i] = i < n ? i : -1;
    return;
  }
  uint32_t kmax = 0u, kmin = 0xffffffffu;
  for (int i = tid; i < n; i += NT) {
    const uint32_t u = okey(__ldcg(row + i));
    if (kSmemRow) rowkeys[i] = u;
    kmax = max(kmax, u);
    kmin = min(kmin, u);
  }
  block_max_min<NT>(sh, kmax, kmin);         // barrier: the shared-memory row is complete
  auto key_at = [&](int i) -> uint32_t { return kSmemRow ? rowkeys[i] : okey(__ldcg(row + i)); };
  uint32_t ties = 0;
  const uint32_t kth = radix_kth<NT>(sh, key_at, n, kmax, kmin, (uint32_t)p.k, &ties);
  emit_ordered<NT>(sh, key_at, n, kth, ties, out, p.k);
}

constexpr int kSurvCap = 8192;           // survivors of the sampled filter kept in shared memory

// block-wide float max / min (NaN operands are ignored); all threads get the result
template <int NT>
__device__ __forceinline__ void block_fmax_fmin(float* red_a, float* red_b, float& vmax, float& vmin) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, off));
    vmin = fminf(vmin, __shfl_xor_sync(0xffffffffu, vmin, off));
  }
  if (lane == 0) { red_a[wid] = vmax; red_b[wid] = vmin; }
  __syncthreads();
  float a = lane < NT / 32 ? red_a[lane] : -INFINITY, b = lane < NT / 32 ? red_b[lane] : INFINITY;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, off));
    b = fminf(b, __shfl_xor_sync(0xffffffffu, b, off));
  }
  vmax = a; vmin = b;
  __syncthreads();
}

// Block-wide, second half of a row for the streaming kernels.  The m_s survivors of the filter
// sit in shared memory (values sval, positions spos).  fast: the filter kept at least k and at
// most kSurvCap entries.  Steps: exact selection among the survivors (value-linear histogram,
// threshold bin, its keys ranked by counting), then every survivor >= the k-th value is written
// out (thread i owns a contiguous run of survivor slots; one block-wide exclusive scan).  When
// the fast path does not apply -- or stops applying: infinite values, a single value, more
// threshold-bin keys than threads (ties share a bin) -- the row is finished exactly from memory:
// bitwise radix select and ordered emission.  One such row
// costs about 30 us, and of 4096 rows of 30K logits one has a tie to be cut: cut among the survivors
// (260 -> 229 us on such data).
template <int NT, class PosT>
__device__ __forceinline__ void finish_row(SelShared& sh, float* red_a, float* red_b, uint32_t* eq_total,
                                           const float* sval, const PosT* spos, uint32_t m_s, bool fast,
                                           const float* row, int n, int k, int32_t* out) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  uint32_t kth = 0, ties = 0, tie_end = 0xffffffffu;      // tie_end: last position selected among the tied
  if (fast) {
    float vmax = -INFINITY, vmin = INFINITY, chk = 0.f;
    for (uint32_t i = tid; i < m_s; i += NT) {
      const float v = sval[i];
      vmax = fmaxf(vmax, v); vmin = fminf(vmin, v); chk = fmaf(v, 0.f, chk);
    }
    const bool any_odd = __syncthreads_or(chk != chk);
    block_fmax_fmin<NT>(red_a, red_b, vmax, vmin);
    const float range = vmax - vmin;
    if (!any_odd && range > 0.f && range <= 3.0e38f) {
      const float sc = 2047.f / range;
      auto bin_of = [&](float v) -> uint32_t {
        return __float_as_uint(fmaf(v - vmin, sc, 8388608.f)) & 0xFFFu;
      };
      for (int i = tid; i < kBins; i += NT) sh.hist[i] = 0;
      __syncthreads();
      for (uint32_t i = tid; i < m_s; i += NT) atomicAdd(&sh.hist[bin_of(sval[i])], 1u);
      __syncthreads();
      uint32_t rem = 0;
      const uint32_t b = find_bin<NT>(sh, (uint32_t)k, &rem);
      for (uint32_t i = tid; i < m_s; i += NT) {
        const float v = sval[i];
        if (bin_of(v) == b) {
          const uint32_t c = atomicAdd(&sh.n_cand, 1u);
          if (c < (uint32_t)NT) sh.cand[c] = okey(v);
        }
      }
      __syncthreads();
      const uint32_t m = sh.n_cand;
      if (m <= (uint32_t)NT) {
        if (tid < (int)m) {
          const uint32_t mine = sh.cand[tid];
          uint32_t gtc = 0, eqc = 0;
          for (uint32_t j = 0; j < m; ++j) {
            const uint32_t o = sh.cand[j];
            gtc += o > mine;
            eqc += o == mine;
          }
          if (gtc < rem && rem <= gtc + eqc) { sh.kth = mine; sh.ties = rem - gtc; *eq_total = eqc; }
        }
        __syncthreads();
        kth = sh.kth; ties = sh.ties;
        if (ties != *eq_total) {                  // the tie at the k-th value must be cut by position
          const float kv = okey_inv(kth);
          __syncthreads();
          if (tid == 0) sh.n_cand = 0;
          __syncthreads();
          for (uint32_t i = tid; i < m_s; i += NT)
            if (sval[i] == kv) sh.cand[atomicAdd(&sh.n_cand, 1u)] = spos[i];
          __syncthreads();
          const uint32_t me = sh.n_cand;          // equal values share the threshold bin: at most its m keys
          if (tid < (int)me) {
            const uint32_t mine = sh.cand[tid];
            uint32_t r = 0;
            for (uint32_t j = 0; j < me; ++j) r += sh.cand[j] < mine;
            if (r + 1 == ties) sh.kth = mine;
          }
          __syncthreads();
          tie_end = sh.kth;
        }
      } else {
        fast = false;
      }
      __syncthreads();
    } else {
      fast = false;
    }
  }
  if (fast) {
    const float kv = okey_inv(kth);
    auto emit = [&](auto selected) {
      const uint32_t per = (m_s + NT - 1) / NT;
      const uint32_t i0 = min((uint32_t)tid * per, m_s), i1 = min(i0 + per, m_s);
      uint32_t cnt = 0;
      for (uint32_t i = i0; i < i1; ++i) cnt += selected(i);
      uint32_t inc = cnt;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t a = __shfl_up_sync(0xffffffffu, inc, off);
        if (lane >= off) inc += a;
      }
      if (lane == 31) sh.wa[wid] = inc;
      __syncthreads();
      uint32_t wtot = lane < NT / 32 ? sh.wa[lane] : 0u, ws = wtot;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t a = __shfl_up_sync(0xffffffffu, ws, off);
        if (lane >= off) ws += a;
      }
      uint32_t o = __shfl_sync(0xffffffffu, ws - wtot, wid) + inc - cnt;
      for (uint32_t i = i0; i < i1; ++i)
        if (selected(i)) {
          if (o < (uint32_t)k) out[o] = (int32_t)spos[i];
          ++o;
        }
    };
    if (tie_end == 0xffffffffu) emit([&](uint32_t i) { return sval[i] >= kv; });
    else emit([&](uint32_t i) { return sval[i] > kv || (sval[i] == kv && (uint32_t)spos[i] <= tie_end); });
  } else {
    auto key_mem = [&](int i) -> uint32_t { return okey(__ldcg(row + i)); };
    uint32_t kmax = 0u, kmin = 0xffffffffu;
    for (int i = tid; i < n; i += NT) {
      const uint32_t u = key_mem(i);
      kmax = max(kmax, u);
      kmin = min(kmin, u);
    }
    block_max_min<NT>(sh, kmax, kmin);
    kth = radix_kth<NT>(sh, key_mem, n, kmax, kmin, (uint32_t)k, &ties);
    emit_ordered<NT>(sh, key_mem, n, kth, ties, out, k);
  }
}

// Block-wide: a filter threshold from 2048 samples smp[4] per thread of a row of n entries.
// With q = k / n the expected number of samples above the k-th value is 2048 q; four standard
// deviations and a few bins above that, the sample rank r gives a value that at least k
// elements of the row exceed (probability of the opposite about 3e-5 per row; that case and
// every other surprise take the exact path).  -inf when no useful threshold exists.
template <int NT>
__device__ __forceinline__ float sampled_threshold(SelShared& sh, float* red_a, float* red_b,
                                                   const float (&smp)[4], int n, int k) {
  float smax = fmaxf(fmaxf(smp[0], smp[1]), fmaxf(smp[2], smp[3]));
  float smin = fminf(fminf(smp[0], smp[1]), fminf(smp[2], smp[3]));
  block_fmax_fmin<NT>(red_a, red_b, smax, smin);
  const float srange = smax - smin;
  const float qf = (float)k / (float)n, mean = 2048.f * qf;
  const uint32_t r = (uint32_t)ceilf(mean + 4.f * sqrtf(mean * (1.f - qf)) + 8.f);
  float t_lo = -INFINITY;
  if (srange > 0.f && srange <= 3.0e38f && r < 2048u) {
    const float sc = 2047.f / srange;
    for (int i = threadIdx.x; i < kBins; i += NT) sh.hist[i] = 0;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (smp[i] == smp[i]) atomicAdd(&sh.hist[__float_as_uint(fmaf(smp[i] - smin, sc, 8388608.f)) & 0xFFFu], 1u);
    __syncthreads();
    uint32_t rem_s = 0;
    const uint32_t b = find_bin<NT>(sh, r, &rem_s);
    if (b > 1u) t_lo = smin + (float)(b - 2u) / sc;       // two bins below: rounding-safe lower edge
  }
  return t_lo;
}

// Rows of at most 512 * EPT entries, 16-byte aligned: persistent CTAs, one row at a time.
// The row arrives in shared memory by ONE bulk copy (no registers, no threads involved), is
// moved into REGISTERS as fp32 values -- thread i owns the 16-byte quads i, i + 512, ... -- and
// the next row's copy is issued at once, so it lands while this row is being processed.
// Selection without sorting and without touching most elements more than once:
//   1. 2048 evenly spaced samples of the row give a threshold that, with overwhelming
//      probability, a little more than k elements exceed;
//   2. one compare per element builds the survivors' positional masks (block-wide scan);
//   3. the ~1.3 k survivors' positions go to shared memory, their values are re-read;
//   4. among them: value-linear histogram (bin = the low bits of fma(v - min, 2047 / range,
//      2^23): no float-to-int conversion), suffix scan, the few keys of the threshold bin ranked
//      exactly by counting;
//   5. survivors >= the k-th value are written out (block-wide scan of per-thread counts).
// The output order is fixed but not ascending.  Whatever the fast path does not cover -- too
// few or too many survivors, infinite values, a single value, more threshold-bin keys than
// threads -- is finished by the
// exact bitwise radix select and the ordered emission over the row re-read from memory.
constexpr int kStreamThreads = 512;
enum { kSiteSelRow = 11 };

template <int EPT>
__global__ void __launch_bounds__(kStreamThreads, 1)
topk_select_stream_kernel(const SelParams p) {
  constexpr int NT = kStreamThreads, NQ = EPT / 4;
  extern __shared__ __align__(16) float rowbuf[];      // the row | survivor values | survivor positions
  float* sval = rowbuf + ((p.S + 3) & ~3);
  uint16_t* spos = reinterpret_cast<uint16_t*>(sval + kSurvCap);
  __shared__ SelShared sh;
  __shared__ __align__(8) uint64_t row_bar;
  __shared__ float red_a[NT / 32], red_b[NT / 32];
  __shared__ uint32_t eq_total;
  const Waiter wt{g_status, p.epoch, p.wait_limit_ns};
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  auto len_of = [&](int t) -> int {
    return p.lengths ? min(max(p.lengths[t], 0), p.S) : min(p.S, max(p.q_pos0 + t + 1, 0));
  };
  // rows that need a selection are fetched; the others are written directly
  auto fetch = [&](int t) {       // thread 0 only
    const int n = len_of(t);
    if (n > p.k) {
      const uint32_t bytes = (uint32_t)(((n + 3) & ~3) * 4);
      mbar_arrive_expect_tx(&row_bar, bytes);
      bulk_load_1d(smem_u32(rowbuf), p.logits + (long long)t * p.ld, bytes, &row_bar);
    }
  };
  if (tid == 0) {
    mbar_init(&row_bar, 1);
    fence_mbar_init();
  }
  __syncthreads();
  pdl_trigger();
  pdl_wait();
  if (tid == 0 && (int)blockIdx.x < p.T) fetch(blockIdx.x);
  uint32_t phase = 0;

  for (int t = blockIdx.x; t < p.T; t += gridDim.x) {
    const int n = len_of(t);
    int32_t* out = p.out + (long long)t * p.k;
    const int t_next = t + gridDim.x;
    if (n <= p.k) {            // everything valid is selected; no copy was issued for this row
      for (int i = tid; i < p.k; i += NT) out[i] = i < n ? i : -1;
      if (tid == 0 && t_next < p.T) fetch(t_next);
      continue;
    }
    const bool landed = mbar_wait(&row_bar, phase, wt, kSiteSelRow, t);
    phase ^= 1;
    // ---- registers: quad q of this thread holds positions 4 * (q * NT + tid) .. + 3.  Quads
    // [0, nfull) are entirely below n for every thread; the next one may be cut; the rest is empty.
    float vr[EPT];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const float4 v = 4 * (q * NT + tid) < n ? reinterpret_cast<const float4*>(rowbuf)[q * NT + tid]
                                              : make_float4(0.f, 0.f, 0.f, 0.f);
      vr[4 * q] = v.x; vr[4 * q + 1] = v.y; vr[4 * q + 2] = v.z; vr[4 * q + 3] = v.w;
    }
    const int nfull = n / (4 * NT);                 // block-uniform
    // 2048 samples of the row, evenly spaced over its positions (read while the row is still
    // in shared memory): they place the threshold of the filter below
    float smp[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) smp[i] = rowbuf[(int)(((long long)(4 * tid + i) * n) >> 11)];
    auto live = [&](int q, int c) -> bool { return q < nfull || 4 * (q * NT + tid) + c < n; };
    fence_proxy_async_smem();      // these reads are ordered before the next bulk write
    if (tid == 0) sh.n_cand = 0;
    const bool all_landed = __syncthreads_and(landed);
    if (tid == 0 && t_next < p.T) fetch(t_next);
    if (!all_landed) continue;     // a wait ran out: the status word says so (block-uniform decision)

    const float* row = p.logits + (long long)t * p.ld;
    bool fast = true;                // block-uniform: the fast path still applies

    // ---- 1. a threshold from the sample; short rows skip the filter: everything survives
    float t_lo = -INFINITY;
    if (n > kSurvCap / 2) t_lo = sampled_threshold<NT>(sh, red_a, red_b, smp, n, p.k);

    // ---- 2. filter: one 4-bit mask per quad (kept for the extraction below), survivor count,
    // block-wide exclusive scan
    unsigned long long selm = 0ull;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      uint32_t m4;
      if (q < nfull) {
        m4 = (uint32_t)(vr[4 * q] >= t_lo) | ((uint32_t)(vr[4 * q + 1] >= t_lo) << 1) |
             ((uint32_t)(vr[4 * q + 2] >= t_lo) << 2) | ((uint32_t)(vr[4 * q + 3] >= t_lo) << 3);
      } else {
        m4 = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c) m4 |= (uint32_t)(live(q, c) && vr[4 * q + c] >= t_lo) << c;
      }
      selm |= (unsigned long long)m4 << (4 * q);
    }
    const uint32_t nsel = __popcll(selm);
    uint32_t slot = 0, m_s = 0;
    {
      const uint32_t cnt = nsel;
      uint32_t inc = cnt;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t a = __shfl_up_sync(0xffffffffu, inc, off);
        if (lane >= off) inc += a;
      }
      if (lane == 31) sh.wa[wid] = inc;
      __syncthreads();
      uint32_t wtot = lane < NT / 32 ? sh.wa[lane] : 0u, ws = wtot;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t a = __shfl_up_sync(0xffffffffu, ws, off);
        if (lane >= off) ws += a;
      }
      slot = __shfl_sync(0xffffffffu, ws - wtot, wid) + inc - cnt;
      m_s = __shfl_sync(0xffffffffu, ws, NT / 32 - 1);
      __syncthreads();
    }
    if (m_s < (uint32_t)p.k || m_s > (uint32_t)kSurvCap) fast = false;   // too few (threshold too high) / too many

    if (fast) {
      // ---- 3. survivors: values and positions out of the registers into shared memory; about
      // one element in ten survives, so most quads are skipped on their mask nibble
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const uint32_t m4 = (uint32_t)(selm >> (4 * q)) & 15u;
        if (m4) {
#pragma unroll
          for (int c = 0; c < 4; ++c)
            if (m4 & (1u << c)) {
              sval[slot] = vr[4 * q + c];
              spos[slot] = (uint16_t)(4 * (q * NT + tid) + c);
              ++slot;
            }
        }
      }
      __syncthreads();
    }
    finish_row<NT>(sh, red_a, red_b, &eq_total, sval, spos, m_s, fast, row, n, p.k, out);
    __syncthreads();               // sh.* is reused by the next row
  }
}


// Rows of any length, 16-byte aligned: persistent CTAs; a row streams through two 64 KB
// shared-memory buffers (bulk copies, two chunks in flight, running across rows), its 2048
// samples are read from memory first.  Per chunk a thread filters 32 elements straight out of
// shared memory (count, block-wide scan, survivors appended to the list); after the last chunk
// the survivors are finished like in the register kernel above.
constexpr int kChunk = 16384;            // floats per chunk
enum { kSiteSelChunk = 12 };

// Block-wide: append the elements >= t_lo of one chunk (positions start .. start + kChunk - 1 of
// the row, cut at n) to the survivor list, m_run entries long so far.  `release` runs on thread 0
// once every thread has read the chunk out of its buffer.  fast turns false when the list is full
// or a wait ran out.
template <int NT, class Release>
__device__ __forceinline__ void filter_chunk(SelShared& sh, const float* chunk, int start, int n, float t_lo,
                                             bool landed, float* sval, uint32_t* spos, uint32_t& m_run,
                                             bool& fast, Release release) {
  constexpr int NQ = kChunk / 4 / NT;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const float4* buf = reinterpret_cast<const float4*>(chunk);
  // this thread's NQ quads of the chunk: positions start + 4 * (q * NT + tid) .. + 3
  float4 v[NQ];
  uint32_t cnt = 0;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const int pos = start + 4 * (q * NT + tid);
    v[q] = pos < n ? buf[q * NT + tid] : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
    if (pos + 3 >= n) {      // the row's last quad may be cut: entries beyond n never survive
      if (pos + 1 >= n) v[q].y = NAN;
      if (pos + 2 >= n) v[q].z = NAN;
      if (pos + 3 >= n) v[q].w = NAN;
      if (pos >= n) v[q].x = NAN;
    }
    cnt += (v[q].x >= t_lo) + (v[q].y >= t_lo) + (v[q].z >= t_lo) + (v[q].w >= t_lo);
  }
  fence_proxy_async_smem();    // these reads are ordered before the next bulk write of the buffer
  // block-wide exclusive scan of the counts (its barrier also frees the buffer)
  uint32_t inc = cnt;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t a = __shfl_up_sync(0xffffffffu, inc, off);
    if (lane >= off) inc += a;
  }
  if (lane == 31) sh.wa[wid] = inc;
  const bool all_landed = __syncthreads_and(landed);
  if (tid == 0) release();
  uint32_t wtot = lane < NT / 32 ? sh.wa[lane] : 0u, ws = wtot;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t a = __shfl_up_sync(0xffffffffu, ws, off);
    if (lane >= off) ws += a;
  }
  uint32_t slot = m_run + __shfl_sync(0xffffffffu, ws - wtot, wid) + inc - cnt;
  const uint32_t total = __shfl_sync(0xffffffffu, ws, NT / 32 - 1);
  if (!all_landed || m_run + total > (uint32_t)kSurvCap) fast = false;   // block-uniform
  if (fast) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const uint32_t pos = (uint32_t)(start + 4 * (q * NT + tid));
      if (v[q].x >= t_lo) { sval[slot] = v[q].x; spos[slot] = pos; ++slot; }
      if (v[q].y >= t_lo) { sval[slot] = v[q].y; spos[slot] = pos + 1; ++slot; }
      if (v[q].z >= t_lo) { sval[slot] = v[q].z; spos[slot] = pos + 2; ++slot; }
      if (v[q].w >= t_lo) { sval[slot] = v[q].w; spos[slot] = pos + 3; ++slot; }
    }
  }
  m_run += total;
  __syncthreads();             // sh.wa is reused by the next chunk's scan
}

__global__ void __launch_bounds__(kStreamThreads, 1)
topk_select_chunked_kernel(const SelParams p) {
  constexpr int NT = kStreamThreads;
  extern __shared__ __align__(16) float cbuf[];       // 2 chunks | survivor values | survivor positions
  float* sval = cbuf + 2 * kChunk;
  uint32_t* spos = reinterpret_cast<uint32_t*>(sval + kSurvCap);
  __shared__ SelShared sh;
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ float red_a[NT / 32], red_b[NT / 32];
  __shared__ uint32_t eq_total;
  const Waiter wt{g_status, p.epoch, p.wait_limit_ns};
  const int tid = threadIdx.x;
  auto len_of = [&](int t) -> int {
    return p.lengths ? min(max(p.lengths[t], 0), p.S) : min(p.S, max(p.q_pos0 + t + 1, 0));
  };
  auto chunks_of = [&](int n) -> int { return (n + kChunk - 1) / kChunk; };
  // fetch cursor (thread 0): next (row, chunk) to request and its running chunk number
  int tf = blockIdx.x, cf = 0;
  uint32_t gf = 0;
  auto skip_short = [&]() { while (tf < p.T && len_of(tf) <= p.k) tf += gridDim.x; };
  auto fetch_next = [&]() {       // thread 0 only
    if (tf >= p.T) return;
    const int n = len_of(tf);
    const int start = cf * kChunk;
    const uint32_t bytes = (uint32_t)(min(kChunk, ((n + 3) & ~3) - start) * 4);
    uint64_t* b = &bar[gf & 1];
    mbar_arrive_expect_tx(b, bytes);
    bulk_load_1d(smem_u32(cbuf + (gf & 1) * kChunk), p.logits + (long long)tf * p.ld + start, bytes, b);
    ++gf;
    if (++cf == chunks_of(n)) { cf = 0; tf += gridDim.x; skip_short(); }
  };
  pdl_trigger();
  pdl_wait();
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_mbar_init();
    skip_short();
    fetch_next();
    fetch_next();
  }
  __syncthreads();
  uint32_t gc = 0;                 // running number of the next chunk to consume

  for (int t = blockIdx.x; t < p.T; t += gridDim.x) {
    const int n = len_of(t);
    int32_t* out = p.out + (long long)t * p.k;
    if (n <= p.k) {            // everything valid is selected; nothing was fetched for this row
      for (int i = tid; i < p.k; i += NT) out[i] = i < n ? i : -1;
      continue;
    }
    const float* row = p.logits + (long long)t * p.ld;
    // 2048 evenly spaced samples, read from memory while the first chunk lands
    float smp[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) smp[i] = __ldcg(row + (int)(((long long)(4 * tid + i) * n) >> 11));
    if (tid == 0) sh.n_cand = 0;
    float t_lo = -INFINITY;
    if (n > kSurvCap / 2) t_lo = sampled_threshold<NT>(sh, red_a, red_b, smp, n, p.k);
    else __syncthreads();

    bool fast = true;
    uint32_t m_run = 0;
    const int nch = chunks_of(n);
    for (int c = 0; c < nch; ++c, ++gc) {
      const bool landed = mbar_wait(&bar[gc & 1], (gc >> 1) & 1, wt, kSiteSelChunk, c);
      filter_chunk<NT>(sh, cbuf + (gc & 1) * kChunk, c * kChunk, n, t_lo, landed, sval, spos, m_run, fast,
                       [&]() { fetch_next(); });
    }
    if (m_run < (uint32_t)p.k) fast = false;       // the threshold was too high
    finish_row<NT>(sh, red_a, red_b, &eq_total, sval, spos, m_run, fast, row, n, p.k, out);
    __syncthreads();               // sh.* is reused by the next row
  }
}

// Few long rows: one CLUSTER per row, so that the SMs a row-per-CTA launch would leave idle share
// the row.  CTA r filters the r-th of the row's equal segments (every CTA draws the same 2048
// samples of the whole row, hence the same threshold); the survivors are then appended to the
// leader's list through distributed shared memory in segment order and the leader finishes the
// row like the kernels above.  Latency-bound: one CTA needs 27 us for a 100K-entry row.
__global__ void __launch_bounds__(kStreamThreads, 1)
topk_select_cluster_kernel(const SelParams p, int nc) {
  constexpr int NT = kStreamThreads;
  extern __shared__ __align__(16) float cbuf[];       // 2 chunks | survivor values | survivor positions
  float* sval = cbuf + 2 * kChunk;
  uint32_t* spos = reinterpret_cast<uint32_t*>(sval + kSurvCap);
  __shared__ SelShared sh;
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ float red_a[NT / 32], red_b[NT / 32];
  __shared__ uint32_t eq_total, seg_cnt[8];           // seg_cnt: leader CTA, survivors per segment
  const Waiter wt{g_status, p.epoch, p.wait_limit_ns};
  pdl_trigger();
  pdl_wait();
  const int tid = threadIdx.x, rank = (int)cluster_ctarank(), t = blockIdx.x / nc;
  const int n = p.lengths ? min(max(p.lengths[t], 0), p.S) : min(p.S, max(p.q_pos0 + t + 1, 0));
  int32_t* out = p.out + (long long)t * p.k;
  const float* row = p.logits + (long long)t * p.ld;
  if (n <= p.k) {              // everything valid is selected (uniform over the cluster)
    if (rank == 0)
      for (int i = tid; i < p.k; i += NT) out[i] = i < n ? i : -1;
    return;
  }
  const int seg = (((n + nc - 1) / nc) + 3) & ~3;
  const int s0 = min(rank * seg, n), s1 = min(s0 + seg, n);
  const int nch = (s1 - s0 + kChunk - 1) / kChunk;
  auto fetch = [&](int c) {    // thread 0 only; whole 16-byte quads
    const int start = s0 + c * kChunk;
    const uint32_t bytes = (uint32_t)(min(kChunk, ((s1 + 3) & ~3) - start) * 4);
    mbar_arrive_expect_tx(&bar[c & 1], bytes);
    bulk_load_1d(smem_u32(cbuf + (c & 1) * kChunk), row + start, bytes, &bar[c & 1]);
  };
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_mbar_init();
    if (nch > 0) fetch(0);
    if (nch > 1) fetch(1);
    sh.n_cand = 0;
  }
  float smp[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) smp[i] = __ldcg(row + (int)(((long long)(4 * tid + i) * n) >> 11));
  __syncwarp();
  cluster_sync_all();          // barriers initialised; every CTA of the cluster runs (remote stores below)
  float t_lo = -INFINITY;
  if (n > kSurvCap / 2) t_lo = sampled_threshold<NT>(sh, red_a, red_b, smp, n, p.k);

  bool fast = true;
  uint32_t m_run = 0;
  for (int c = 0; c < nch; ++c) {
    const bool landed = mbar_wait(&bar[c & 1], (c >> 1) & 1, wt, kSiteSelChunk, c);
    filter_chunk<NT>(sh, cbuf + (c & 1) * kChunk, s0 + c * kChunk, s1, t_lo, landed, sval, spos, m_run, fast,
                     [&]() { if (c + 2 < nch) fetch(c + 2); });
  }
  // a segment that did not fit says so with a count no list can hold
  if (tid == 0)
    st_cluster_u32(mapa(smem_u32(&seg_cnt[rank]), 0), fast ? m_run : (uint32_t)kSurvCap + 1u);
  __syncwarp();
  cluster_sync_all();
  uint32_t before = 0, m_s = 0;
  for (int i = 0; i < nc; ++i) {
    const uint32_t c = ld_cluster_u32(mapa(smem_u32(&seg_cnt[i]), 0));
    if (i < rank) before += c;
    m_s += c;
  }
  if (m_s > (uint32_t)kSurvCap) fast = false;            // uniform over the cluster from here on
  else if (rank > 0) {
    const uint32_t dv = mapa(smem_u32(sval), 0), dp = mapa(smem_u32(spos), 0);
    for (uint32_t i = tid; i < m_run; i += NT) {
      st_cluster_u32(dv + 4 * (before + i), __float_as_uint(sval[i]));
      st_cluster_u32(dp + 4 * (before + i), spos[i]);
    }
  }
  __syncwarp();
  cluster_sync_all();
  if (rank > 0) return;
  if (m_s < (uint32_t)p.k) fast = false;                 // the threshold was too high
  finish_row<NT>(sh, red_a, red_b, &eq_total, sval, spos, m_s, fast, row, n, p.k, out);
}

constexpr size_t kChunkDyn = (size_t)2 * kChunk * 4 + (size_t)kSurvCap * 8;

// how many clusters of nc (2 .. 8) CTAs of topk_select_cluster_kernel device `dev` holds at once
static int row_clusters(int dev, int nc, int sms) {
  static thread_local int cached_dev = -1, cached[9];
  if (dev != cached_dev) {
    for (int i = 2; i <= 8; ++i) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3((unsigned)(sms / i * i)); cfg.blockDim = dim3(kStreamThreads);
      cfg.dynamicSmemBytes = kChunkDyn;
      cudaLaunchAttribute at;
      at.id = cudaLaunchAttributeClusterDimension;
      at.val.clusterDim.x = (unsigned)i; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
      cfg.attrs = &at; cfg.numAttrs = 1;
      int n = 0;
      if (!ensure_smem<topk_select_cluster_kernel>(dev, kChunkDyn) ||
          cudaOccupancyMaxActiveClusters(&n, topk_select_cluster_kernel, &cfg) != cudaSuccess)
        n = 0;
      cudaGetLastError();
      cached[i] = n;
    }
    cached_dev = dev;
  }
  return cached[nc];
}

}  // namespace idx
}  // namespace lt

// Index logits of T query tokens at positions q_pos0 .. q_pos0 + T - 1 against S keys.
//   q_idx8  [T, Hi, 128] e4m3 codes, dense; Hi in {32, 64, 128}
//   k_idx8  [S, 128] e4m3 codes, rows k_row_stride bytes apart (multiple of 16)
//   weights [T, Hi] fp32;  k_scale [S] fp32 or null (1.0)
//   logits  [T, logits_row_stride] fp32: the first S entries of every row are written, those beyond
//           the token's position (s > q_pos0 + t) as -inf
// No counterpart in the reference (its indexer was removed); asynchronous on `stream`.
extern "C" int litedsa_index_logits_fp8(const void* q_idx8, const void* k_idx8, const float* weights,
                                        const float* k_scale, float* logits, int T, int Hi, int S,
                                        int q_pos0, long long k_row_stride,
                                        long long logits_row_stride, void* stream) {
  using namespace lt;
  using namespace lt::idx;
  if (!q_idx8 || !k_idx8 || !weights || !logits) return LITEDSA_ERR_ARG;
  if (T <= 0 || S <= 0 || q_pos0 < 0) return LITEDSA_ERR_SHAPE;
  if (Hi != 32 && Hi != 64 && Hi != 128) return LITEDSA_ERR_UNSUPPORTED;
  if (logits_row_stride < S || k_row_stride < kDim || k_row_stride % 16) return LITEDSA_ERR_SHAPE;
  if (((uintptr_t)q_idx8 | (uintptr_t)k_idx8) & 15) return LITEDSA_ERR_UNSUPPORTED;
  if ((long long)T * Hi > 0x7fffffffLL) return LITEDSA_ERR_UNSUPPORTED;
  CUtensorMap map_q, map_k;
  if (!make_map_2d(&map_q, q_idx8, CU_TENSOR_MAP_DATA_TYPE_UINT8, kDim, (uint64_t)T * Hi, kDim, kDim, kCols) ||
      !make_map_2d(&map_k, k_idx8, CU_TENSOR_MAP_DATA_TYPE_UINT8, kDim, (uint64_t)S,
                   (uint64_t)k_row_stride, kDim, kKeyTile))
    return LITEDSA_ERR_CUDA;
  LogitParams p;
  p.weights = weights; p.k_scale = k_scale; p.logits = logits;
  p.T = T; p.Hi = Hi; p.S = S; p.q_pos0 = q_pos0; p.ld = logits_row_stride;
  p.epoch = next_launch_epoch(); p.wait_limit_ns = wait_limit_ns();
  const int dev = current_device();
  // The tokens are dealt to as few CTAs as hold them, evenly: the drain of a key tile, which paces a CTA, takes as long as its
  // accumulators are many (36 tokens of 32 heads: three CTAs of three accumulators each, not of four, four and one:
  // 100003 keys 24.4 -> 20.8 us; two tokens of 64 heads, one accumulator, 65536 keys 12.0 -> 8.1).
  const int groups = (T + kCols / Hi - 1) / (kCols / Hi), ctas_x = (groups + kAccs - 1) / kAccs;
  const int accs = (groups + ctas_x - 1) / ctas_x, tok_per_cta = accs * (kCols / Hi);
  // the tiles that do work: up to the last token's causal bound
  const int all_tiles = (S + kKeyTile - 1) / kKeyTile;
  const int live_tiles = (int)min((long long)all_tiles, ((long long)q_pos0 + T - 1) / kKeyTile + 1);
  const int dead_tiles = all_tiles - live_tiles;
  const int splits = pick_splits(ctas_x, live_tiles, dead_tiles, tok_per_cta, accs, sm_count());
  p.live_tiles = live_tiles;
  p.tiles_per_split = (live_tiles + splits - 1) / splits;
  const int grid_y = dead_tiles > 0 ? splits : (live_tiles + p.tiles_per_split - 1) / p.tiles_per_split;
  auto go = [&](auto hi, auto use) -> int {
    constexpr auto* kern = index_logits_kernel<decltype(hi)::value, decltype(use)::value>;
    if (!ensure_smem<index_logits_kernel<decltype(hi)::value, decltype(use)::value>>(dev, kSmem)) return LITEDSA_ERR_CUDA;
    return launch_pdl(kern, dim3(ctas_x, grid_y), kThreads, kSmem, reinterpret_cast<cudaStream_t>(stream), map_q, map_k, p);
  };
  auto with_accs = [&](auto hi) -> int {
    return accs == 1 ? go(hi, Int<1>()) : accs == 2 ? go(hi, Int<2>()) : accs == 3 ? go(hi, Int<3>()) : go(hi, Int<4>());
  };
  return Hi == 32 ? with_accs(Int<32>()) : Hi == 64 ? with_accs(Int<64>()) : with_accs(Int<128>());
}

// Exact top-k per row of `logits`: topk_idx[t, :] = the k positions i < len(t) with the largest
// values (order inside a row unspecified), ties at the k-th value resolved towards smaller
// positions; rows with len(t) <= k list 0 .. len(t) - 1 and are padded with -1.  len(t) = lengths[t], or
// min(S, q_pos0 + t + 1) when lengths is null (causal).  NaN sorts below every number.
// The output is what the union operator takes as topk_indices
// (kernels/b200/dsa/litedsa.cu:31-33).  No allocation; asynchronous on `stream`.
extern "C" int litedsa_topk_select(const float* logits, const int32_t* lengths, int32_t* topk_idx,
                                   int T, int S, int k, int q_pos0, long long logits_row_stride,
                                   void* stream) {
  using namespace lt::idx;
  if (!logits || !topk_idx) return LITEDSA_ERR_ARG;
  if (T <= 0 || S <= 0 || k <= 0 || logits_row_stride < S) return LITEDSA_ERR_SHAPE;
  SelParams p;
  p.logits = logits; p.lengths = lengths; p.out = topk_idx;
  p.T = T; p.S = S; p.k = k; p.q_pos0 = q_pos0; p.ld = logits_row_stride;
  p.epoch = lt::next_launch_epoch(); p.wait_limit_ns = lt::wait_limit_ns();
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  // aligned rows up to 32768 entries live in registers, longer ones stream through shared memory;
  // unaligned ones are kept in shared memory up to 49152 entries and re-read from memory beyond
  const size_t smem = (((size_t)S + 3) & ~(size_t)3) * 4;      // whole 16-byte quads
  const int dev = lt::current_device();
  const bool aligned = (logits_row_stride & 3) == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0;
  const int sms = lt::sm_count(), grid = T < sms ? T : sms;
  // Few long rows: the largest clusters of which the chip holds one per row at once, if every CTA gets at
  // least 8192 entries.  Below 24576 entries the cluster synchronisations cost more than the shorter
  // filter saves (20000 entries, k = 2048: 11.9 us, one CTA per row 10.3; 32768: 12.2 and 12.3; 131072:
  // 14.1 and 28.8).  What counts is how many clusters fit, not how many SMs there are: 18 clusters of eight are
  // 144 CTAs but more than the chip's GPCs hold, and the second wave made 18 rows of 32768 entries take
  // 20.3 us.  Sizes that are no powers of two fit where the next power does not: 36 rows of 100003 entries in clusters of three
  // 16.2 us, of two 18.2.
  int nc = aligned ? 8 : 1;
  while (nc > 1 && (S <= 24576 || S < 8192 * nc || T > row_clusters(dev, nc, sms))) --nc;
  if (nc > 1) {
    if (!lt::ensure_smem<topk_select_cluster_kernel>(dev, kChunkDyn)) return LITEDSA_ERR_CUDA;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(T * nc)); cfg.blockDim = dim3(kStreamThreads);
    cfg.dynamicSmemBytes = kChunkDyn; cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)nc; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = 2;
    return lt::launch_result(cudaLaunchKernelEx(&cfg, topk_select_cluster_kernel, (const SelParams)p, nc));
  }
  if (aligned && S <= kStreamThreads * 64) {
    const bool small = S <= kStreamThreads * 32;
    const size_t dyn = smem + (size_t)kSurvCap * 6;      // + survivor values (fp32) and positions (u16)
    if (!(small ? lt::ensure_smem<topk_select_stream_kernel<32>>(dev, dyn) : lt::ensure_smem<topk_select_stream_kernel<64>>(dev, dyn)))
      return LITEDSA_ERR_CUDA;
    return lt::launch_pdl(small ? topk_select_stream_kernel<32> : topk_select_stream_kernel<64>, dim3(grid),
                          kStreamThreads, dyn, st, p);
  }
  if (aligned) {
    if (!lt::ensure_smem<topk_select_chunked_kernel>(dev, kChunkDyn)) return LITEDSA_ERR_CUDA;
    return lt::launch_pdl(topk_select_chunked_kernel, dim3(grid), kStreamThreads, kChunkDyn, st, p);
  }
  if (S <= kMaxSmemRow) {
    if (!lt::ensure_smem<topk_select_kernel<true>>(dev, smem)) return LITEDSA_ERR_CUDA;
    return lt::launch_pdl(topk_select_kernel<true>, dim3(T), kGenericThreads, smem, st, p);
  }
  return lt::launch_pdl(topk_select_kernel<false>, dim3(T), kGenericThreads, 0, st, p);
}

// Status block of the index-logits kernel (same layout as litedsa_attn_status).
extern "C" int litedsa_index_status(int* out4_host, int reset) {
  using namespace lt::idx;
  if (out4_host && cudaMemcpyFromSymbol(out4_host, g_status, sizeof(int) * 4) != cudaSuccess)
    return LITEDSA_ERR_CUDA;
  if (reset) {
    const int z[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (cudaMemcpyToSymbol(g_status, z, sizeof(z)) != cudaSuccess) return LITEDSA_ERR_CUDA;
  }
  return (out4_host && out4_host[0] != 0) ? LITEDSA_ERR_TIMEOUT : LITEDSA_OK;
}
