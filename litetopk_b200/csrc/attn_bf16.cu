// Masked BF16 MLA prefill over a per-tile union list of gathered KV rows (sm_100a): host side and the
// dequantisation of packed cache rows.  The kernel is mla_bf16.cuh.
//
// Two operators of the reference end up here:
//   * dsv4_masked_mla_bf16(q, kv, indices, pref, win_lo, win_hi, counts, sm_scale, h_per_q,
//     out, lse, attn_sink)  (kernels/b200/dsa/litedsa_dsv4.cu:50-121, kernel
//     kernels/b200/dsa/litedsa_attention_sm100_dsv4.cuh:1849-2485): bf16 q / KV rows of 512
//     dims gathered through an ascending index list; row r of a tile attends the union
//     ranks [0, pref) and [win_lo, win_hi) of its token (range_mask32, :1824-1829);
//   * masked_mla_fp8 on a cache whose per-128 scales differ and whose rope part is bf16
//     (the DeepSeek-V3.2 cache row): such a cache has no single-scale all-e4m3 form, so it is
//     dequantised once into a bf16 [s_kv, 576] workspace (litedsa_dequant_kv656) and attended
//     here with the query-major membership mask of union_qm
//     (kernels/b200/dsa/litedsa_union.cuh:147-171) at bf16 accuracy -- the same "flat
//     dequantised workspace" route the reference's own bf16 operator takes
//     (litedsa_dsv4.cu:40-48).
//
#include "mla_bf16.cuh"

namespace lt {
namespace b16 {

using namespace mla16;

struct Args {
  const void* q; const void* kv; const int32_t* indices; const int32_t* counts;
  const uint32_t* memb; const int32_t* pref; const int32_t* win_lo; const int32_t* win_hi;
  const float* sink; void* out; float* max_logits; float* lse;
  int ng, s_kv, topk, d, h_per_q;
  int64_t q_row_stride, kv_row_stride, idx_row_stride;     // ELEMENTS
  float sm_scale;
  // in-place addressing of q / out inside [T, H_padded, d] tensors (ELEMENTS, 0 = dense packed)
  int64_t q_token_stride, q_head_stride, out_token_stride, out_head_stride;
  const int4* runs = nullptr;     // run only if a tile's list is not two runs (see Params)
  // nsplit > 1 (d = 576): every tile's blocks are cut into slices whose fp32 results go to part_o / part_ml
  int nsplit = 1;
  float* part_o = nullptr;
  float2* part_ml = nullptr;
  const int2* order = nullptr;    // d = 576, unsliced (see Params)
};

// argument rules shared by both entry points (no CUDA call)
static int check(const Args& a) {
  if (!a.q || !a.kv || !a.indices || !a.out || !a.lse) return LITEDSA_ERR_ARG;
  if (!a.memb && !(a.pref && a.win_lo && a.win_hi)) return LITEDSA_ERR_ARG;
  if (a.ng <= 0 || a.s_kv <= 0 || a.topk <= 0 || a.topk % 64 != 0) return LITEDSA_ERR_SHAPE;
  if (a.h_per_q <= 0 || 128 % a.h_per_q != 0 || 128 / a.h_per_q > 16) return LITEDSA_ERR_SHAPE;
  if (a.d != 512 && a.d != 576) return LITEDSA_ERR_SHAPE;
  if (a.memb && a.topk % 128 != 0) return LITEDSA_ERR_SHAPE;        // whole mask words per tile row
  // strides in ELEMENTS (bf16); TMA / 16-byte copies need 16-byte aligned bases and pitches
  if (a.q_row_stride < a.d || a.kv_row_stride < a.d || (a.q_row_stride % 8) || (a.kv_row_stride % 8))
    return LITEDSA_ERR_UNSUPPORTED;
  if (((uintptr_t)a.q | (uintptr_t)a.kv | (uintptr_t)a.out) & 15) return LITEDSA_ERR_UNSUPPORTED;
  if (a.idx_row_stride < a.topk) return LITEDSA_ERR_UNSUPPORTED;
  if (a.q_token_stride < 0 || a.q_head_stride < 0 || a.out_token_stride < 0 || a.out_head_stride < 0)
    return LITEDSA_ERR_SHAPE;
  if ((a.q_head_stride && (a.q_head_stride < a.d || a.q_head_stride % 8)) || a.q_token_stride % 8 ||
      (a.out_head_stride && (a.out_head_stride < kDV || a.out_head_stride % 8)) || a.out_token_stride % 8)
    return LITEDSA_ERR_UNSUPPORTED;
  return LITEDSA_OK;
}

static int run(const Args& a, void* stream) {
  const int rc = check(a);
  if (rc != LITEDSA_OK) return rc;
  CUtensorMap mq, mout;
  const QOutArgs qo{a.q, a.out, a.d, a.ng, a.h_per_q, a.q_row_stride, a.q_token_stride, a.q_head_stride,
                    a.out_token_stride, a.out_head_stride};
  if (!make_q_out_maps(qo, &mq, &mout)) return LITEDSA_ERR_CUDA;
  Params p = {};
  p.lse = a.lse; p.max_logits = a.max_logits; p.sink = a.sink; p.sink_mod = 128;
  p.ng = a.ng; p.G = 128 / a.h_per_q; p.h_per_q = a.h_per_q; p.nsplit = 1;
  p.scale_log2 = a.sm_scale * kLog2e;
  p.epoch = next_launch_epoch(); p.wait_limit = wait_limit_ticks();
  p.runs = a.runs;
  p.kv = reinterpret_cast<const uint8_t*>(a.kv); p.kv_pitch = a.kv_row_stride * 2;
  p.indices = a.indices; p.idx_stride = a.idx_row_stride;
  p.memb = a.memb; p.s_kv = a.s_kv; p.cap = a.topk;
  p.pref = a.pref; p.win_lo = a.win_lo; p.win_hi = a.win_hi; p.counts = a.counts;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (a.nsplit > 1) {
    p.nsplit = a.nsplit; p.part_o = a.part_o; p.part_ml = a.part_ml;
    return launch<576, kGather, true>(mq, mq, mq, mout, p, st);
  }
  if (a.order != nullptr) {
    p.order = a.order;
    return launch<576, kGather, false, true>(mq, mq, mq, mout, p, st);
  }
  return a.d == 576 ? launch<576, kGather, false>(mq, mq, mq, mout, p, st)
                    : launch<512, kGather, false>(mq, mq, mq, mout, p, st);
}

// One warp per cache row: 512 e4m3 codes x their per-128 fp32 scale -> bf16, the 64 bf16 rope
// values copied behind them.
__global__ void __launch_bounds__(256) dequant_kv656_kernel(const uint8_t* __restrict__ in,
                                                             uint8_t* __restrict__ out, int s_kv,
                                                             long long out_pitch) {
  const int warps_per_block = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  for (int row = blockIdx.x * warps_per_block + (threadIdx.x >> 5); row < s_kv;
       row += gridDim.x * warps_per_block) {
    const uint8_t* src = in + (size_t)row * 656;
    uint8_t* dst = out + (size_t)row * out_pitch;
    // lane: codes [8 lane, +8) (chunk lane / 16) and [256 + 8 lane, +8) (chunk 2 + lane / 16):
    // two coalesced 256-byte loads in, two coalesced 512-byte stores out
    const uint2 c0 = __ldcs(reinterpret_cast<const uint2*>(src) + lane);
    const uint2 c1 = __ldcs(reinterpret_cast<const uint2*>(src) + 32 + lane);
    const float s0 = __ldg(reinterpret_cast<const float*>(src + 512) + (lane >> 4));
    const float s1 = __ldg(reinterpret_cast<const float*>(src + 512) + 2 + (lane >> 4));
    const uint32_t w[4] = {c0.x, c0.y, c1.x, c1.y};
    uint32_t o[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float sc = j < 2 ? s0 : s1;
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const __nv_fp8x2_storage_t two = (__nv_fp8x2_storage_t)((w[j] >> (16 * hh)) & 0xffffu);
        const __half2_raw hr = __nv_cvt_fp8x2_to_halfraw2(two, __NV_E4M3);
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hr));
        __nv_bfloat162 b2 = __floats2bfloat162_rn(f.x * sc, f.y * sc);
        o[2 * j + hh] = *reinterpret_cast<uint32_t*>(&b2);
      }
    }
    uint4* d4 = reinterpret_cast<uint4*>(dst);
    d4[lane] = make_uint4(o[0], o[1], o[2], o[3]);
    d4[32 + lane] = make_uint4(o[4], o[5], o[6], o[7]);
    // rope: 128 bytes = 8 x 16
    if (lane < 8)
      reinterpret_cast<uint4*>(dst + 1024)[lane] = __ldcs(reinterpret_cast<const uint4*>(src + 528) + lane);
  }
}

}  // namespace b16

// the union form on dense packed operands of 576 dims, in nsplit slices or in an order (prefill.cu)
int run_bf16_union(const void* q, const void* kv, const int32_t* indices, float sm_scale, const int32_t* counts,
                    const uint32_t* memb, int h, void* out, float* lse, int ng, int s_kv, int cap, int64_t kv_row_stride,
                    int nsplit, float* part_o, float2* part_ml, const int2* order, void* stream) {
  b16::Args a{q, kv, indices, counts, memb, nullptr, nullptr, nullptr, nullptr, out, nullptr, lse,
              ng, s_kv, cap, 576, h, 576, kv_row_stride, cap, sm_scale, 0, 0, 0, 0};
  a.nsplit = nsplit; a.part_o = part_o; a.part_ml = part_ml; a.order = order;
  return b16::run(a, stream);
}
}  // namespace lt

// The reference's DSv4 operator with its own argument list
//   dsv4_masked_mla_bf16(q, kv, indices, pref, win_lo, win_hi, counts, sm_scale, h_per_q,
//                        out, lse, attn_sink)        (kernels/b200/dsa/litedsa_dsv4.cu:50-121)
// tensor shapes and strides passed as integers.  d = 512 as in the reference, or 576.  The four
// trailing strides (ELEMENTS, 0 = dense packed) address q and out in place inside
// [T, H_padded, d] tensors with h_per_q real heads per token: the zero-copy form the reference
// planned for this operator (kernels/b200/dsa/DSV4_ZEROCOPY_PLAN.md:50-76).
extern "C" int litedsa_dsv4_masked_mla_bf16(const void* q, const void* kv, const int32_t* indices,
                                            const int32_t* pref, const int32_t* win_lo,
                                            const int32_t* win_hi, const int32_t* counts,
                                            float sm_scale, int h_per_q, void* out, float* lse,
                                            const float* attn_sink, int ng, int s_kv, int topk,
                                            int d, int64_t q_row_stride, int64_t kv_row_stride,
                                            int64_t indices_row_stride, int64_t q_token_stride,
                                            int64_t q_head_stride, int64_t out_token_stride,
                                            int64_t out_head_stride, void* workspace,
                                            int64_t workspace_bytes, void* stream) {
  using namespace lt::b16;
  if (!pref || !win_lo || !win_hi || !counts) return LITEDSA_ERR_ARG;
  Args a{q, kv, indices, counts, nullptr, pref, win_lo, win_hi, attn_sink, out, nullptr, lse,
         ng, s_kv, topk, d, h_per_q, q_row_stride, kv_row_stride, indices_row_stride, sm_scale,
         q_token_stride, q_head_stride, out_token_stride, out_head_stride};
  const int rc = check(a);
  if (rc != LITEDSA_OK) return rc;
  // With a workspace the device decides: when every tile's index list is two contiguous runs
  // of rows (the packed prefix + window pattern this operator exists for) the range kernel
  // reads K and V with tiled TMA loads and the gather kernel returns at once; otherwise the
  // range kernel returns at once and the gather kernel does the work.
  if (workspace != nullptr) {
    if (workspace_bytes < 16 + 16 * (int64_t)ng || ((uintptr_t)workspace & 15)) return LITEDSA_ERR_SHAPE;
    const int rc2 = lt::dsv4_rank_enqueue(q, kv, indices, pref, win_lo, win_hi, counts, sm_scale, h_per_q, out,
                                          lse, attn_sink, ng, s_kv, topk, d, q_row_stride, kv_row_stride,
                                          indices_row_stride, q_token_stride, q_head_stride,
                                          out_token_stride, out_head_stride, workspace,
                                          reinterpret_cast<cudaStream_t>(stream));
    if (rc2 != LITEDSA_OK) return rc2;
    a.runs = reinterpret_cast<const int4*>(reinterpret_cast<const char*>(workspace) + 16);
  }
  return run(a, stream);
}

// masked_mla_fp8's bf16 twin: the same union list + query-major membership mask
// (kernels/b200/dsa/litedsa.cu:77-80 argument order, minus out_scale) over bf16 q and a bf16
// KV workspace, for caches that have no single-scale all-e4m3 form.
extern "C" int litedsa_masked_mla_bf16(const void* q, const void* kv, const int32_t* indices,
                                       float sm_scale, const int32_t* topk_length,
                                       const uint32_t* memb_qm, int h_per_q, void* out,
                                       float* max_logits, float* lse, int ng, int s_kv, int topk,
                                       int d, int64_t q_row_stride, int64_t kv_row_stride,
                                       int64_t indices_row_stride, const float* attn_sink,
                                       void* stream) {
  using namespace lt::b16;
  if (!memb_qm) return LITEDSA_ERR_ARG;
  Args a{q, kv, indices, topk_length, memb_qm, nullptr, nullptr, nullptr, attn_sink, out, max_logits,
         lse, ng, s_kv, topk, d, h_per_q, q_row_stride, kv_row_stride, indices_row_stride, sm_scale,
         0, 0, 0, 0};
  return run(a, stream);
}

// Packed 656-byte cache rows (512 e4m3 codes | 4 fp32 per-128 scales | 64 bf16 rope) ->
// bf16 rows [s_kv, 576] (latent = code x its chunk's scale, rope copied); out_pitch = bytes
// between output rows (>= 1152, multiple of 16).
extern "C" int litedsa_dequant_kv656(const void* kv656, void* kv_bf16, int s_kv, int64_t out_pitch,
                                     void* stream) {
  using namespace lt::b16;
  if (!kv656 || !kv_bf16) return LITEDSA_ERR_ARG;
  if (s_kv <= 0 || out_pitch < 1152 || out_pitch % 16) return LITEDSA_ERR_SHAPE;
  if (((uintptr_t)kv656 | (uintptr_t)kv_bf16) & 15) return LITEDSA_ERR_UNSUPPORTED;
  const int blocks = min(148 * 8, (s_kv + 7) / 8);
  dequant_kv656_kernel<<<blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const uint8_t*>(kv656), reinterpret_cast<uint8_t*>(kv_bf16), s_kv, out_pitch);
  return cudaGetLastError() == cudaSuccess ? LITEDSA_OK : LITEDSA_ERR_CUDA;
}

// Status block of the bf16 gather kernel (same meaning and use as litedsa_attn_status).
extern "C" int litedsa_bf16_status(int* out4_host, int reset) {
  using namespace lt::b16;
  if (out4_host && cudaMemcpyFromSymbol(out4_host, g_status, sizeof(int) * 4) != cudaSuccess)
    return LITEDSA_ERR_CUDA;
  if (reset) {
    const int z[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (cudaMemcpyToSymbol(g_status, z, sizeof(z)) != cudaSuccess) return LITEDSA_ERR_CUDA;
  }
  return (out4_host && out4_host[0] != 0) ? LITEDSA_ERR_TIMEOUT : LITEDSA_OK;
}
