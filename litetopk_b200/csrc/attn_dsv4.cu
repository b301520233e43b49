// DeepSeek-V4 style packed BF16 attention over two contiguous key ranges (sm_100a): host side and the
// classification of index lists.  The kernel is mla_bf16.cuh.
//
// Every query token at position p attends to the compressed-prefix entries
// [0, p / ratio) of a small compressed KV and to the raw sliding window
// [p - window + 1, p]; G = 128 / h adjacent tokens are packed into one 128-row tile.
// The reference's DSv4 operator (kernels/b200/dsa/litedsa_dsv4.cu:50-121, kernel
// kernels/b200/dsa/litedsa_attention_sm100_dsv4.cuh:1849-2485) expresses the same mask as
// two ranges per token in the rank space of a gathered union list and gathers rows with TMA
// gather4.  Here both key segments are contiguous in memory, so K and V tiles come from plain
// tiled TMA loads, no index list exists, and the mask is a few comparisons per thread and block.
#include "mla_bf16.cuh"

namespace lt {
namespace dsv4 {

using namespace mla16;

// One warp per tile: is the tile's gathered index list (its first counts[tile] entries) two contiguous ascending runs of
// valid rows?  runs[tile] = (first row of run 0, its length, first row of run 1, its length), and a mark if one of a
// block's tiles is not (kRunGroup): nothing has to be cleared beforehand.  Latency-bound, so sixteen loads of a lane are in
// flight (2048 lists of 641 entries: 10 us with one after the other, and a launch to clear a word, 1.5, before it).
__global__ void __launch_bounds__(32 * kRunGroup)
classify_runs_kernel(const int32_t* __restrict__ indices, long long idx_stride, int topk,
                     const int32_t* __restrict__ counts, int ng, int s_kv, int4* __restrict__ runs) {
  const int tile = (int)(blockIdx.x * kRunGroup + (threadIdx.x >> 5)), lane = threadIdx.x & 31;
  pdl_trigger();
  pdl_wait();
  int scattered = 0;
  int4 r = make_int4(0, 0, 0, 0);
  if (tile < ng) {
    const int32_t* row = indices + (size_t)tile * idx_stride;
    const int cnt = min(max(counts ? __ldcg(counts + tile) : topk, 0), topk);
    int breaks = 0, first_break = 0x7fffffff, bad = 0;
    for (int j0 = lane; j0 < cnt; j0 += 32 * 8) {
      int v[8], next[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int j = j0 + 32 * u;
        v[u] = j < cnt ? __ldcg(row + j) : 0;
        next[u] = j + 1 < cnt ? __ldcg(row + j + 1) : v[u] + 1;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        bad |= v[u] < 0 || v[u] >= s_kv;
        if (next[u] != v[u] + 1) {
          ++breaks;
          first_break = min(first_break, j0 + 32 * u);
        }
      }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      breaks += __shfl_xor_sync(0xffffffffu, breaks, off);
      first_break = min(first_break, __shfl_xor_sync(0xffffffffu, first_break, off));
      bad |= __shfl_xor_sync(0xffffffffu, bad, off);
    }
    r.y = breaks ? first_break + 1 : cnt;
    r.w = cnt - r.y;
    if (cnt > 0) r.x = __ldcg(row);
    if (r.w > 0) r.z = __ldcg(row + r.y);
    scattered = bad || breaks > 1;
  }
  scattered = __syncthreads_or(scattered);
  if (threadIdx.x == 0 && scattered) r.x |= (int)0x80000000;
  if (lane == 0 && tile < ng) runs[tile] = r;
}


// most blocks a tile of the call can have: its last tile has the longest prefix
static int most_blocks(int ng, int G, int n_comp, int pos0, int window, int ratio) {
  const int64_t last = (int64_t)pos0 + (int64_t)ng * G - 1;
  const int64_t pref = min(last / ratio, (int64_t)n_comp);
  const int64_t halves = (pref + kOwnKeys - 1) / kOwnKeys + (min(last + 1, (int64_t)window + G - 1) + kOwnKeys - 1) / kOwnKeys;
  return (int)((halves + 1) / 2);
}
static int64_t slice_bytes(int ng, int nsplit) {
  return nsplit < 2 ? 0 : (int64_t)ng * nsplit * 128 * (512 * 4 + 8);
}

static Params base_params(int ng, int h, float sm_scale, float* lse, const float* sink, int sink_mod) {
  Params p = {};
  p.lse = lse; p.sink = sink; p.sink_mod = sink_mod;
  p.ng = ng; p.G = 128 / h; p.h_per_q = h; p.nsplit = 1;
  p.window = p.ratio = 1;
  p.scale_log2 = sm_scale * kLog2e;
  p.epoch = next_launch_epoch(); p.wait_limit = wait_limit_ticks();
  return p;
}

}  // namespace dsv4

// Rank mode of the range kernel for the reference operator's argument list (see
// litedsa_dsv4_masked_mla_bf16): classifies every tile's index list on the device, then enqueues
// the range kernel gated on "every tile is two contiguous runs".  workspace: 16 + 16 * ng bytes
// (runs[ng] from byte 16); the caller enqueues the gather kernel behind it, gated on the
// opposite value, so exactly one of the two does the work -- no host synchronisation.
int dsv4_rank_enqueue(const void* q, const void* kv, const int32_t* indices, const int32_t* pref,
                      const int32_t* win_lo, const int32_t* win_hi, const int32_t* counts,
                      float sm_scale, int h_per_q, void* out, float* lse, const float* attn_sink,
                      int ng, int s_kv, int topk, int d, int64_t q_row_stride, int64_t kv_row_stride,
                      int64_t indices_row_stride, int64_t q_token_stride, int64_t q_head_stride,
                      int64_t out_token_stride, int64_t out_head_stride, void* workspace,
                      cudaStream_t stream) {
  using namespace dsv4;
  int4* runs = reinterpret_cast<int4*>(reinterpret_cast<char*>(workspace) + 16);
  const int rc = launch_pdl(classify_runs_kernel, dim3((unsigned)(ng + kRunGroup - 1) / kRunGroup), 32 * kRunGroup, 0, stream, indices,
                            (long long)indices_row_stride, topk, counts, ng, s_kv, runs);
  if (rc != LITEDSA_OK) return rc;
  CUtensorMap mq, mkv, mout;
  const QOutArgs a{q, out, d, ng, h_per_q, q_row_stride, q_token_stride, q_head_stride, out_token_stride, out_head_stride};
  if (!make_q_out_maps(a, &mq, &mout) || !make_kv_map(&mkv, kv, d, s_kv, kv_row_stride)) return LITEDSA_ERR_CUDA;
  Params p = base_params(ng, h_per_q, sm_scale, lse, attn_sink, 128);
  p.runs = runs; p.pref = pref; p.win_lo = win_lo; p.win_hi = win_hi; p.counts = counts;
  return d == 576 ? launch<576, kRank, false>(mq, mkv, mkv, mout, p, stream)
                  : launch<512, kRank, false>(mq, mkv, mkv, mout, p, stream);
}

}  // namespace lt

// Bytes of workspace with which litedsa_dsv4_c128a_bf16_ws runs this shape in slices (0: it does not).
extern "C" int64_t litedsa_dsv4_workspace(int ng, int h_per_q, int n_comp, int pos0, int window, int ratio) {
  using namespace lt::dsv4;
  if (ng <= 0 || h_per_q <= 0 || 128 % h_per_q || n_comp < 0 || pos0 < 0 || window <= 0 || ratio <= 0) return 0;
  return slice_bytes(ng, lt::bf16_slices(ng, most_blocks(ng, 128 / h_per_q, n_comp, pos0, window, ratio)));
}

// DSv4 packed BF16 attention over (compressed prefix, sliding window).  Replaces the
// reference operator dsv4_masked_mla_bf16 (kernels/b200/dsa/litedsa_dsv4.cu:50-55) for
// callers whose two key ranges are contiguous: instead of a gathered union index list plus
// per-token rank ranges it takes the two KV tensors and the first query position.
extern "C" int litedsa_dsv4_c128a_bf16(const void* q, const void* kv_comp, const void* kv_raw,
                                       int ng, int h_per_q, int n_comp, int s_raw, int pos0,
                                       int window, int ratio, float sm_scale,
                                       const float* attn_sink, void* out, float* lse,
                                       int64_t q_row_stride, int64_t kc_row_stride,
                                       int64_t kr_row_stride, int64_t q_token_stride,
                                       int64_t q_head_stride, int64_t out_token_stride,
                                       int64_t out_head_stride, void* stream) {
  return litedsa_dsv4_c128a_bf16_ws(q, kv_comp, kv_raw, ng, h_per_q, n_comp, s_raw, pos0, window, ratio, sm_scale,
                                    attn_sink, 128, out, lse, q_row_stride, kc_row_stride, kr_row_stride,
                                    q_token_stride, q_head_stride, out_token_stride, out_head_stride, nullptr, 0,
                                    stream);
}

// The same with one sink per head (sink_len == h_per_q) or per packed row (128), and with a workspace
// for calls of few tiles, whose key blocks are then cut into slices that run in parallel.
extern "C" int litedsa_dsv4_c128a_bf16_ws(const void* q, const void* kv_comp, const void* kv_raw, int ng,
                                          int h_per_q, int n_comp, int s_raw, int pos0, int window, int ratio,
                                          float sm_scale, const float* attn_sink, int sink_len, void* out,
                                          float* lse, int64_t q_row_stride, int64_t kc_row_stride,
                                          int64_t kr_row_stride, int64_t q_token_stride, int64_t q_head_stride,
                                          int64_t out_token_stride, int64_t out_head_stride, void* workspace,
                                          int64_t workspace_bytes, void* stream) {
  using namespace lt;
  using namespace lt::dsv4;
  constexpr int kD = 576;
  if (!q || !kv_raw || !out || !lse) return LITEDSA_ERR_ARG;
  if (n_comp > 0 && !kv_comp) return LITEDSA_ERR_ARG;
  if (ng <= 0 || s_raw <= 0 || n_comp < 0 || pos0 < 0 || window <= 0 || ratio <= 0)
    return LITEDSA_ERR_SHAPE;
  if (h_per_q <= 0 || 128 % h_per_q != 0 || 128 / h_per_q > 16) return LITEDSA_ERR_SHAPE;
  const int G = 128 / h_per_q;
  if (attn_sink && sink_len != 128 && sink_len != h_per_q) return LITEDSA_ERR_SHAPE;
  if ((int64_t)pos0 + (int64_t)ng * G > s_raw) return LITEDSA_ERR_SHAPE;   // queries sit inside the cache
  if (window + G - 1 > 32768) return LITEDSA_ERR_UNSUPPORTED;
  // strides are in ELEMENTS (bf16); TMA needs 16-byte aligned bases and pitches
  if (q_row_stride < kD || kr_row_stride < kD || (q_row_stride % 8) || (kr_row_stride % 8) ||
      (n_comp > 0 && (kc_row_stride < kD || (kc_row_stride % 8))))
    return LITEDSA_ERR_UNSUPPORTED;
  if (((uintptr_t)q | (uintptr_t)kv_raw | (uintptr_t)kv_comp | (uintptr_t)out) & 15)
    return LITEDSA_ERR_UNSUPPORTED;
  if (q_token_stride < 0 || q_head_stride < 0 || out_token_stride < 0 || out_head_stride < 0)
    return LITEDSA_ERR_SHAPE;
  if ((q_head_stride && (q_head_stride < kD || q_head_stride % 8)) || q_token_stride % 8 ||
      (out_head_stride && (out_head_stride < kDV || out_head_stride % 8)) || out_token_stride % 8)
    return LITEDSA_ERR_UNSUPPORTED;
  CUtensorMap mq, mc, mr, mout;
  const QOutArgs a{q, out, kD, ng, h_per_q, q_row_stride, q_token_stride, q_head_stride, out_token_stride, out_head_stride};
  // without compressed rows the first segment is empty and its map never used
  if (!make_q_out_maps(a, &mq, &mout) || !make_kv_map(&mr, kv_raw, kD, s_raw, kr_row_stride) ||
      !(n_comp > 0 ? make_kv_map(&mc, kv_comp, kD, n_comp, kc_row_stride) : make_kv_map(&mc, kv_raw, kD, 1, kr_row_stride)))
    return LITEDSA_ERR_CUDA;
  Params p = base_params(ng, h_per_q, sm_scale, lse, attn_sink, sink_len);
  p.n_comp = n_comp; p.pos0 = pos0; p.window = window; p.ratio = ratio;
  if (workspace) {
    if ((uintptr_t)workspace & 255) return LITEDSA_ERR_UNSUPPORTED;
    const int ns = bf16_slices(ng, most_blocks(ng, G, n_comp, pos0, window, ratio));
    if (ns > 1 && workspace_bytes >= slice_bytes(ng, ns)) {
      p.nsplit = ns;
      p.part_o = reinterpret_cast<float*>(workspace);
      p.part_ml = reinterpret_cast<float2*>(p.part_o + (size_t)ng * ns * 128 * kDV);
    }
  }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (p.nsplit == 1) return launch<kD, kRange, false>(mq, mc, mr, mout, p, st);
  const int rc = launch<kD, kRange, true>(mq, mc, mr, mout, p, st);
  if (rc != LITEDSA_OK) return rc;
  return merge_slices(p.part_o, p.part_ml, p.nsplit, ng, h_per_q, 1.f, 0.f, attn_sink, sink_len, out,
                      a.out_ts(), a.out_hs(), lse, st);
}

// Status word of the DSv4 kernel (same meaning as litedsa_attn_status).
extern "C" int litedsa_dsv4_status(int* out4_host, int reset) {
  using namespace lt::dsv4;
  if (out4_host && cudaMemcpyFromSymbol(out4_host, g_status, sizeof(int) * 4) != cudaSuccess)
    return LITEDSA_ERR_CUDA;
  if (reset) {
    const int z[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (cudaMemcpyToSymbol(g_status, z, sizeof(z)) != cudaSuccess) return LITEDSA_ERR_CUDA;
  }
  return (out4_host && out4_host[0] != 0) ? LITEDSA_ERR_TIMEOUT : LITEDSA_OK;
}
