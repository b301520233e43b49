// The whole path of one chunk of query tokens behind one call: union of the tiles' top-k lists,
// masked attention over it, and -- for chunks of few tokens -- the merge of the tiles' slices.
//
// What one call costs beyond its kernels matters for small chunks: as separate operators (each
// with its own checks, output allocations and ctypes call) two tokens took 70 us of host time
// around 38 us of kernels.  Here the intermediate tensors live in one caller-owned workspace.
//
// Few tiles leave most of the chip idle while each of them walks its union list serially (one
// cluster of two SMs per tile, about 1.3 us per 128-key block).  Such tiles are cut into slices
// (pick_slices) that run as separate work items of the attention kernel; every slice leaves its
// unnormalised fp32 O with its running max and row sum, and merge_slices_kernel brings them to a
// common max, normalises and rounds once -- the same fp32 accumulation as the unsliced tile, in
// another order.  The reference leaves KV splits to its callers
// (kernels/b200/dsa/litedsa_attention_sm100.cuh:1383-1385).
#include "common.cuh"

namespace lt {
namespace prefill {

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

// out = out_scale * sum_j O_j 2^(m_j - M) / (sum_j l_j 2^(m_j - M) + sink), lse = ln(sum) + M ln 2 - lse_off
// (the sink joins the output's normaliser only; row r of a tile = token r / h, head r % h).
// A warp has kPieces of a row's four 128-dim pieces, lane i unit i (4 dims) of each, as part_unit() has swapped them.  Latency-
// bound at the sizes it runs at (2 KB per slice and row): the loads of eight (two) slices are under way with that of the
// maxima, before a weight is known.  One piece per warp for few tiles, else four (merge_slices).  (A warp per row that went from slice to
// slice: 2 tokens x 64 heads in five slices 20.3 -> 18.6 us, in eight of a native cache 20.6 -> 18.3.)
template <int kPieces>
__global__ void __launch_bounds__(256)
merge_slices_kernel(const float* __restrict__ part_o, const float2* __restrict__ part_ml, int nsplit, int n_rows, int h,
                    float out_scale, float lse_off, const float* __restrict__ sink, int sink_mod,
                    __nv_bfloat16* __restrict__ out, long long out_ts, long long out_hs, float* __restrict__ lse) {
  constexpr int kPer = 4 / kPieces, kBatch = 8 / kPieces;
  const int w = (int)(blockIdx.x * 8 + (threadIdx.x >> 5)), lane = threadIdx.x & 31;
  const int row = w / kPer, c0 = w % kPer * kPieces;
  if (row >= n_rows) return;
  pdl_wait();
  const int tile = row >> 7, r = row & 127;
  const size_t p0 = (size_t)tile * nsplit * 128 + r;            // slice j of the row: p0 + 128 j
  float2 ml = make_float2(-INFINITY, 0.f);
  if (lane < nsplit) ml = __ldcg(part_ml + p0 + (size_t)lane * 128);
  const float4* src = reinterpret_cast<const float4*>(part_o + p0 * 512) + 32 * c0 + lane;
  float4 v[kBatch][kPieces];
  auto fetch = [&](int j0) {
#pragma unroll
    for (int u = 0; u < kBatch; ++u)
#pragma unroll
      for (int c = 0; c < kPieces; ++c)
        if (j0 + u < nsplit) v[u][c] = __ldcg(src + (size_t)(j0 + u) * (128 * 128) + 32 * c);
  };
  fetch(0);
  float m = ml.y > 0.f ? ml.x : -INFINITY;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
  const float f = ml.y > 0.f ? fast_exp2(ml.x - m) : 0.f;       // slices without a key weigh nothing
  float l = ml.y * f;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) l += __shfl_xor_sync(0xffffffffu, l, off);
  float denom = l;
  if (sink != nullptr && l > 0.f) denom += fast_exp2(__ldcg(sink + r % sink_mod) * kLog2e - m);
  float4 acc[kPieces];
#pragma unroll
  for (int c = 0; c < kPieces; ++c) acc[c] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int j0 = 0; j0 < nsplit; j0 += kBatch) {
    if (j0 > 0) fetch(j0);
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const float fj = j0 + u < nsplit ? __shfl_sync(0xffffffffu, f, j0 + u) : 0.f;
      if (fj == 0.f) continue;                                  // warp-uniform; whatever the slice holds
#pragma unroll
      for (int c = 0; c < kPieces; ++c) {
        acc[c].x = fmaf(v[u][c].x, fj, acc[c].x);
        acc[c].y = fmaf(v[u][c].y, fj, acc[c].y);
        acc[c].z = fmaf(v[u][c].z, fj, acc[c].z);
        acc[c].w = fmaf(v[u][c].w, fj, acc[c].w);
      }
    }
  }
  const float os = l > 0.f ? __fdividef(out_scale, denom) : 0.f;
  uint2* dst = reinterpret_cast<uint2*>(out + (row / h) * out_ts + (row % h) * out_hs) + 32 * c0 + part_unit(lane, r);
#pragma unroll
  for (int c = 0; c < kPieces; ++c) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(acc[c].x * os, acc[c].y * os), b = __floats2bfloat162_rn(acc[c].z * os, acc[c].w * os);
    dst[32 * c] = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
  }
  if (lane == 0 && c0 == 0) lse[row] = l > 0.f ? __logf(l) + m * kLn2 - lse_off : INFINITY;
}

// Slices of a tile of `blocks` key blocks that are worth what they cost when nothing else runs: what each costs grows with
// their number, the time that they save does less and less.
static int most_slices(int blocks) {
  int n = 1;
  while (n < kMaxSlices && (n + 1) * (n + 1) <= 4 * blocks) ++n;
  return n;
}

// How many slices a tile is cut into when a launch has `tiles` tiles of G lists of k entries: no more than there are clusters
// for.  A union is not known on the host; neighbouring tokens share about three quarters of their lists, so it is taken as
// k (3 + G) / 4 entries.  Slices cost a launch for the merge, fp32 partial results, which grow with their number, and, FP8, a
// block each for the running max; a block of an unsliced tile takes 1.1 us (bf16: bf16_slices).  FP8: tiles of ten blocks and more; with
// a few tiles in slices of two to three blocks, with many of four.  Slices that shorten a tile by less than 4 + 0.08 tiles n blocks even
// when only half of the lists is shared are not made (128 heads, 37 tiles of 12 blocks: 30.5 us in two slices, 25.6 whole).  us, whole / in n:
// 2 tokens x 64 heads, top-2048 30.4, five 18.7, eight 18.0; 8 x 64 30.6, five 19.6, eight 19.2; 18 x 64 31.5, five 21.0, eight 22.3;
// top-1024 20.8, three 19.5, five 18.3; 36 x 64, top-2048 31.7, two 27.7, four 25.3; 68 x 64 33.3, two 30.4, top-1024 22.0 and 24.5;
// 16 x 8, top-1024, half shared 81.5, eight 28.7, twelve 26.5, nine tenths shared 35.1, 22.1, 21.8.
static int pick_slices(int tiles, int G, int k, bool bf16) {
  const int blocks = (int)((int64_t)k * (3 + G) / 4 / (bf16 ? 64 : 128));
  if (bf16) return bf16_slices(tiles, blocks);
  if (blocks < 10) return 1;
  const int few = min(most_slices(blocks), 48 / tiles);
  const int n = min(min(sm_count() / 2 / tiles, max(blocks / 4, few)), kMaxSlices);
  if (n < 2) return 1;
  const double half = (double)k * (1 + G) / 2 / 128;
  return half - (half / n + 1.0) >= 4.0 + 0.08 * tiles * n ? n : 1;
}

// In which order the tiles are dealt out to the CTAs (64-row tiles) or clusters (a native cache).  Unions of several lists differ in
// size, and a CTA that has every 148th tile as they come can have more to do than the others: with half to nine tenths of the lists
// shared, 16384 tokens x 32 heads 4 % more than the mean, 8192 x 16 10 %, 8192 x 8 22 %.  A block of this kernel takes eight rounds
// of tiles, sorts them by their key blocks (a counting sort) and deals them out to and fro: 1 to 2 %.  Not all tiles at once, so
// that neighbours, whose tokens attend much the same keys, still run at about the same time.  A tile's result does not depend on
// its place.
constexpr int kMostBlocks = 1024;      // of 64 keys: 65536
static int order_window(int ncta) { return ncta * max(min(8, 2048 / ncta), 1); }      // at most 2048 tiles
__global__ void __launch_bounds__(1024)
order_tiles_kernel(const int32_t* __restrict__ counts, int ng, int cap, int ncta, int window, int2* __restrict__ order) {
  __shared__ int place[kMostBlocks], warp_sum[32];
  const int tid = threadIdx.x, lane = tid & 31, base = blockIdx.x * window, m = min(window, ng - base);
  pdl_trigger();
  place[tid] = 0;
  __syncthreads();
  pdl_wait();
  int live[2], bin[2];      // of tiles tid and tid + 1024; the largest come first
#pragma unroll
  for (int u = 0; u < 2; ++u) live[u] = tid + 1024 * u < m ? min(max(__ldcg(counts + base + tid + 1024 * u), 0), cap) : 0;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    bin[u] = kMostBlocks - min(max((live[u] + 63) / 64, 1), kMostBlocks);
    if (tid + 1024 * u < m) atomicAdd(&place[bin[u]], 1);
  }
  __syncthreads();
  const int n = place[tid];
  int sum = n;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, sum, off);
    if (lane >= off) sum += v;
  }
  if (lane == 31) warp_sum[tid >> 5] = sum;
  __syncthreads();
  int before = lane < (tid >> 5) ? warp_sum[lane] : 0;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) before += __shfl_xor_sync(0xffffffffu, before, off);
  place[tid] = before + sum - n;
  __syncthreads();
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    if (tid + 1024 * u >= m) break;
    const int at = atomicAdd(&place[bin[u]], 1), round = at / ncta, c = at - round * ncta;
    const bool back = (round + 1) * ncta <= m && ((round ^ blockIdx.x) & 1);
    order[base + round * ncta + (back ? ncta - 1 - c : c)] = make_int2(base + tid + 1024 * u, live[u]);
  }
}

// workspace layout: all offsets are multiples of 256 bytes
struct Layout { int64_t counts, u, memb, part_o, part_ml, q_codes, order, total; };
// The launch costs 1.5 to 3 us, whatever there is to gain: for long jobs, longer ones with two lists per tile, whose unions differ
// less.  As they come / ordered, us: half to nine tenths of the lists shared 8192 x 8, top-1024 296 / 261; 8192 x 16 345 / 325; 4096 x
// 16, bf16 queries 197 / 184; 16384 x 32 933 / 925; below the line, with it none: 4096 x 16, top-512 111 / 106, 2048 x 32, top-1024
// 132 / 130.  Seven tenths shared by all: 8192 x 16, top-2048 637 / 641, top-512 226 / 227; below the line 1776 x 16, top-256 32 / 34.
// Native cache, half to nine tenths shared: 4096 x 8, top-512 241 / 196; 2048 x 16, top-1024 256 / 215; 2048 x 32 263 / 242; 2050 x 64,
// top-1984 616 / 605; three quarters shared by all 174 / 175, 193 / 195, and 583 / 585.
static bool ordered(int ng, int G, int cap, bool rows64, bool kv_bf16) {
  const int ncta = rows64 ? sm_count() : sm_count() / 2;
  if (G == 1 || ng <= ncta || !(rows64 || kv_bf16)) return false;
  return (int64_t)ng * cap >= (int64_t)(rows64 ? (G > 2 ? 400 : 1000) : (G > 2 ? 280 : 700)) * 64 * ncta;
}
static Layout layout_of(int ng, int G, int cap, int nsplit, bool rows64, bool kv_bf16) {
  auto up = [](int64_t b) { return (b + 255) & ~(int64_t)255; };
  Layout l;
  l.counts = 0;
  l.u = up(4 * (int64_t)ng);
  l.memb = l.u + up(4 * (int64_t)ng * cap);
  l.part_o = l.memb + (rows64 && G == 1 ? 0 : up(4 * (int64_t)ng * G * (cap / 32)));      // one token per tile: none
  l.part_ml = l.part_o + (nsplit > 1 ? up((int64_t)ng * nsplit * 128 * 512 * 4) : 0);
  l.q_codes = l.part_ml + (nsplit > 1 ? up((int64_t)ng * nsplit * 128 * 8) : 0);
  l.order = l.q_codes + (rows64 ? rows64_scratch(ng) : 0);
  l.total = l.order + (nsplit == 1 && ordered(ng, G, cap, rows64, kv_bf16) ? up(8 * (int64_t)ng) : 0);
  return l;
}

static int check_shape(int T, int h, int k, int policy_tokens) {
  if (h <= 0 || 128 % h != 0 || 128 / h > 16 || T <= 0 || T % (128 / h) != 0 || k <= 0) return LITEDSA_ERR_SHAPE;
  if (policy_tokens < T) return LITEDSA_ERR_SHAPE;
  if ((int64_t)(128 / h) * k > 65536) return LITEDSA_ERR_UNSUPPORTED;      // 16-bit ranks (union_qm)
  return LITEDSA_OK;
}

// Whether a job of `tokens` tokens runs on 64-row tiles (attn_fp8_r64.cuh) instead of 128-row ones: with an FP8
// cache, up to 64 heads, lists of a tile of 256 entries and more, a tile for every other SM and at least ten key
// blocks per SM.  Fewer tiles run faster as slices of 128-row ones: 40 tiles of 16 heads, top-2048, 48 us against 56.  (Of the line of
// ten blocks that no longer holds: 148 tiles of 64 heads, top-512, 21.1 / 16.4 us, 296 of top-256 22.3 / 18.3, 60 of top-1024 23.2 / 18.3.  It was drawn when
// both forms took the 23 us of a call's launches there; such calls keep the rounding that 128-row tiles give them.)
// 128-row / 64-row tiles, half and nine tenths of the lists shared, e4m3 queries, us (bf16 queries: much the same, but
// 69 / 68 at 222 tiles and nine tenths, 90 / 79 with top-256):
//   74 tiles of 64 rows: 64 heads, top-2048    34 / 28 and 31 / 28;    16 heads 65 / 58 and 41 / 37
//   222: 32 heads, top-2048                    106 / 75 and 65 / 63
//   1184: 64 heads, top-256 59 / 46 both, top-2048 249 / 183 and 199 / 184;    32 heads, top-2048 392 / 266 and
//         231 / 217;    16 heads 690 / 430 and 306 / 261;    8 heads 1322 / 754 and 449 / 347
// The more of the lists is shared, the less there is to gain: of 402 calls above the line (74 to 1200 tiles, sharing 30 to 97 %, both query
// types) four were slower, by 1 to 3 %, all of 32 heads with 95 % shared and more; 0.75 of the time in the mean.  How
// much is shared is not known on the host.
static bool use_rows64(int tokens, int h, int k, bool kv_bf16) {
  if (kv_bf16 || h > 64 || (int64_t)(128 / h) * k % 128 != 0) return false;
  const int64_t tiles = (int64_t)tokens * h / 64, list = (int64_t)(64 / h) * k;
  return list >= 256 && tiles >= sm_count() / 2 && tiles * list >= (int64_t)10 * 64 * sm_count();
}

}  // namespace prefill

// What the slices save (0.75 us a block) has to be more than the merge and the items cost.  us, whole / in n slices: 2 tokens x 64
// heads at 131072 (18.5 blocks) 21.3, two 18.5, four 14.5, eight 13.1; at 65536 (10.5) 14.9, two 15.2, six 12.5; 8 x 16 at 40000 (7.5)
// 13.1, five 12.3, at 32768 (6.5) 12.4 and 12.4; 16 x 64 at 131072 22.0, four 16.3, eight 15.5; 40 x 64 22.8, three 19.5; 70 x 64 23.4,
// two 24.0.  Unions on a native cache: 2 x 64, top-2048 43.7, five 21.2, twelve 18.4; 18 x 64 44.6, four 25.1, eight 22.8, top-1024 28.1, four
// 19.9, eight 20.1; 68 x 64, top-2048 50.4, two 38.6, top-1024 30.4 and 27.8; 40 x 64, top-512 19.7, three 19.8.
int bf16_slices(int tiles, int blocks) {
  const int n = min(prefill::most_slices(blocks), sm_count() / 2 / tiles);
  return n >= 2 && 0.75 * blocks * (n - 1) / n >= 4.0 + 0.045 * tiles * n ? n : 1;
}

int merge_slices(const float* part_o, const float2* part_ml, int nsplit, int ng, int h, float out_scale, float lse_off,
                 const float* sink, int sink_mod, void* out, int64_t out_token_stride, int64_t out_head_stride,
                 float* lse, cudaStream_t stream) {
  // One piece per warp makes blocks of 256 threads (57 registers), of which an SM holds four: nine tiles are all of them at once.  The line is
  // where both forms take the same time, at 11 tiles.  Calls with their merge, four pieces / one, us, top-2048, native cache and ranges at 131072: 1 tile
  // 18.4 / 17.0, 19.2 / 17.6, 13.8 / 12.3; 9 tiles 20.4 / 20.1, 24.1 / 22.0, 17.5 / 15.4; 10 tiles 21.3 / 20.7, 24.4 / 23.7, 17.0 / 16.6; 12 tiles 22.1 /
  // 22.3, 25.3 / 25.3, 17.3 / 17.5; 18 tiles 24.3 / 24.9, 27.7 / 28.4, 17.9 / 18.7; 34 tiles 30.4 / 32.2, 38.5 / 40.2, 23.5 / 25.3.
  const bool few = ng * 64 <= 5 * sm_count();
  return launch_pdl(few ? prefill::merge_slices_kernel<1> : prefill::merge_slices_kernel<4>, dim3(ng * (few ? 64 : 16)), 256, 0, stream,
                    part_o, part_ml, nsplit, ng * 128, h, out_scale, lse_off, sink, sink_mod, reinterpret_cast<__nv_bfloat16*>(out),
                    (long long)out_token_stride, (long long)out_head_stride, lse);
}
}  // namespace lt

namespace lt {
namespace prefill {

// rows of a tile and length of its list; the slices of a tile
struct Route { int ng, G, cap, ns; bool rows64; };
static Route route_of(int T, int h, int k, bool kv_bf16, int policy_tokens, bool by_job) {
  Route r;
  r.rows64 = by_job && use_rows64(policy_tokens, h, k, kv_bf16);
  r.G = (r.rows64 ? 64 : 128) / h;
  r.ng = T / r.G;
  r.cap = r.rows64 ? (r.G * k + 127) / 128 * 128 : r.G * k;
  r.ns = r.rows64 ? 1 : pick_slices(policy_tokens / r.G, r.G, k, kv_bf16);
  return r;
}

static int64_t workspace(int T, int h, int k, int kv_is_bf16, int policy_tokens, bool by_job) {
  if (check_shape(T, h, k, policy_tokens) != LITEDSA_OK) return 0;
  const Route r = route_of(T, h, k, kv_is_bf16 != 0, policy_tokens, by_job);
  return layout_of(r.ng, r.G, r.cap, r.ns, r.rows64, kv_is_bf16 != 0).total;
}

static int run(const void* q, int q_is_bf16, const void* kv, int kv_is_bf16, const int32_t* topk_idx, double sm_scale,
               double q_scale, double kv_scale, void* out, float* lse, int T, int h, int k, int s_kv,
               int64_t kv_row_stride, int64_t seq_space, int policy_tokens, bool by_job, void* workspace,
               int64_t workspace_bytes, void* stream) {
  if (!q || !kv || !topk_idx || !out || !lse || !workspace) return LITEDSA_ERR_ARG;
  int rc = check_shape(T, h, k, policy_tokens);
  if (rc != LITEDSA_OK) return rc;
  if (kv_is_bf16 && !q_is_bf16) return LITEDSA_ERR_UNSUPPORTED;
  if (!kv_is_bf16 && q_is_bf16 && !((float)q_scale > 0.f)) return LITEDSA_ERR_SHAPE;
  if (((uintptr_t)workspace & 255) || ((uintptr_t)q & 15) || ((uintptr_t)out & 15) || ((uintptr_t)topk_idx & 15))
    return LITEDSA_ERR_UNSUPPORTED;
  const Route r = route_of(T, h, k, kv_is_bf16 != 0, policy_tokens, by_job);
  const int G = r.G, ng = r.ng, cap = r.cap, ns = r.ns;
  const Layout l = layout_of(ng, G, cap, ns, r.rows64, kv_is_bf16 != 0);
  if (workspace_bytes < l.total) return LITEDSA_ERR_SHAPE;
  char* ws = reinterpret_cast<char*>(workspace);
  int32_t* counts = reinterpret_cast<int32_t*>(ws + l.counts);
  int32_t* u = reinterpret_cast<int32_t*>(ws + l.u);
  uint32_t* memb = r.rows64 && G == 1 ? nullptr : reinterpret_cast<uint32_t*>(ws + l.memb);
  // what the 128-row form of the call refuses (8 heads: lists of more than 2048 entries) is refused in either form
  if (r.rows64) {
    const int G2 = 128 / h;
    rc = check_union(T, k, T / G2, G2 * k, G2, seq_space);
    if (rc != LITEDSA_OK) return rc;
  }
  // fill 2: lists padded to whole 128-key blocks, nothing written beyond
  rc = run_union(topk_idx, u, counts, memb, nullptr, nullptr, T, k, ng, cap, G, 0, 0, 1, seq_space, 2, stream);
  if (rc != LITEDSA_OK) return rc;
  // tiles in order of their size
  int2* order = nullptr;
  if (ns == 1 && ordered(ng, G, cap, r.rows64, kv_is_bf16 != 0)) {
    order = reinterpret_cast<int2*>(ws + l.order);
    const int ncta = r.rows64 ? sm_count() : sm_count() / 2, window = order_window(ncta);
    rc = launch_pdl(order_tiles_kernel, dim3((ng + window - 1) / window), 1024, 0, reinterpret_cast<cudaStream_t>(stream), counts, ng, cap,
                    ncta, window, order);
    if (rc != LITEDSA_OK) return rc;
  }
  if (kv_is_bf16 && (ns > 1 || order != nullptr)) {
    float* part_o = reinterpret_cast<float*>(ws + l.part_o);
    float2* part_ml = reinterpret_cast<float2*>(ws + l.part_ml);
    rc = run_bf16_union(q, kv, u, (float)sm_scale, counts, memb, h, out, lse, ng, s_kv, cap, kv_row_stride, ns, part_o, part_ml, order, stream);
    if (rc != LITEDSA_OK || ns == 1) return rc;
    return merge_slices(part_o, part_ml, ns, ng, h, 1.f, 0.f, nullptr, 1, out, (int64_t)h * 512, 512, lse,
                        reinterpret_cast<cudaStream_t>(stream));
  }
  if (kv_is_bf16)
    return litedsa_masked_mla_bf16(q, kv, u, (float)sm_scale, counts, memb, h, out, nullptr, lse, ng, s_kv, cap, 576, 576,
                                   kv_row_stride, cap, nullptr, stream);
  // one rounding to fp32 of the whole product, as a caller of the operators makes it
  Fp8Args a{q, kv, u, (float)(sm_scale * q_scale * kv_scale), (float)kv_scale, counts, memb, h, nullptr, lse,
            ng, s_kv, cap, 576, kv_row_stride, cap, nullptr, nullptr, 1};
  a.q_is_bf16 = q_is_bf16 != 0;
  a.q_inv = 1.0f / (float)q_scale;
  if (r.rows64) return run_fp8_rows64(a, out, ws + l.q_codes, order, stream);
  a.nsplit = ns;
  a.part_o = reinterpret_cast<float*>(ws + l.part_o);
  a.part_ml = ws + l.part_ml;
  void* outs[1] = {out};
  rc = run_fp8(a, outs, 1, stream);
  if (rc != LITEDSA_OK || ns == 1) return rc;
  return merge_slices(a.part_o, reinterpret_cast<const float2*>(a.part_ml), ns, ng, h, a.out_scale, kFp8LseOffset,
                      nullptr, 1, out, (int64_t)h * 512, 512, lse, reinterpret_cast<cudaStream_t>(stream));
}

}  // namespace prefill
}  // namespace lt

// Bytes of workspace litedsa_sparse_prefill needs (0: the shape is not supported).
extern "C" int64_t litedsa_sparse_prefill_workspace(int T, int h, int k, int kv_is_bf16, int policy_tokens) {
  return lt::prefill::workspace(T, h, k, kv_is_bf16, policy_tokens, false);
}
extern "C" int64_t litedsa_sparse_prefill_job_workspace(int T, int h, int k, int kv_is_bf16, int job_tokens) {
  return lt::prefill::workspace(T, h, k, kv_is_bf16, job_tokens, true);
}

// union_qm + masked attention of T query tokens in one call; see include/litedsa_b200.h.
extern "C" int litedsa_sparse_prefill(const void* q, int q_is_bf16, const void* kv, int kv_is_bf16,
                                      const int32_t* topk_idx, double sm_scale, double q_scale, double kv_scale,
                                      void* out, float* lse, int T, int h, int k, int s_kv,
                                      int64_t kv_row_stride, int64_t seq_space, int policy_tokens,
                                      void* workspace, int64_t workspace_bytes, void* stream) {
  return lt::prefill::run(q, q_is_bf16, kv, kv_is_bf16, topk_idx, sm_scale, q_scale, kv_scale, out, lse, T, h, k, s_kv,
                          kv_row_stride, seq_space, policy_tokens, false, workspace, workspace_bytes, stream);
}

// The same, the rows of a tile chosen by the size of the job; see include/litedsa_b200.h.
extern "C" int litedsa_sparse_prefill_job(const void* q, int q_is_bf16, const void* kv, int kv_is_bf16,
                                          const int32_t* topk_idx, double sm_scale, double q_scale, double kv_scale,
                                          void* out, float* lse, int T, int h, int k, int s_kv, int64_t kv_row_stride,
                                          int64_t seq_space, int job_tokens, void* workspace, int64_t workspace_bytes,
                                          void* stream) {
  return lt::prefill::run(q, q_is_bf16, kv, kv_is_bf16, topk_idx, sm_scale, q_scale, kv_scale, out, lse, T, h, k, s_kv,
                          kv_row_stride, seq_space, job_tokens, true, workspace, workspace_bytes, stream);
}

// litedsa_masked_mla_fp8 on bf16 queries, quantised inside the attention kernel.
extern "C" int litedsa_masked_mla_fp8_bf16q(const void* q_bf16, float q_scale, const void* kv8, const int32_t* indices,
                                            float sm_scale, float out_scale, const int32_t* topk_length,
                                            const uint32_t* memb_qm, int h_per_q, void* out, float* max_logits,
                                            float* lse, int ng, int s_kv, int topk, int64_t kv_row_stride,
                                            int64_t indices_row_stride, void* stream) {
  using namespace lt;
  if (!memb_qm || !out) return LITEDSA_ERR_ARG;
  if (!(q_scale > 0.f)) return LITEDSA_ERR_SHAPE;
  Fp8Args a{q_bf16, kv8, indices, sm_scale, out_scale, topk_length, memb_qm, h_per_q, max_logits, lse,
            ng, s_kv, topk, 576, kv_row_stride, indices_row_stride, nullptr, nullptr, 1};
  a.q_is_bf16 = true;
  a.q_inv = 1.0f / q_scale;
  void* outs[1] = {out};
  return run_fp8(a, outs, 1, stream);
}
