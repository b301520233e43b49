// Per-tile union of the top-k index lists of the G tokens that share one 128-row
// attention tile, plus the query-major membership bitmask.
//
// Contract (what every LIVE output word must equal), stated by the reference at
// kernels/b200/dsa/litedsa_union.cuh:4-25 and implemented there at :34-184:
//   counts[g]        number of distinct positions p, 0 <= p < seq_space, in the tile
//   u_phys[g, r]     physical slot of the r-th smallest such position (r < count)
//   memb_qm[g,q,w]   bit b set  <=>  rank 32*w+b is in token q's own list
// Only the algorithmic idea "a position bitmap makes sort + dedup a scan" is shared
// with the reference; this kernel is laid out for B200 differently:
//   * small CTAs, several resident per SM, so one tile's barrier phases overlap another
//     tile's loads, instead of one 1024-thread CTA per SM slot;
//   * the tile's indices are read from HBM ONCE with 16-byte loads and stay in
//     registers for the second (rank) pass;
//   * a per-word exclusive rank table makes the rank lookup one popcount;
//   * the sorted list is staged in shared memory and leaves the SM as 16-byte coalesced stores.
// Integer-only work: no tensor cores, no TMA.  It moves the index lists and the union once (65536
// tokens of 16 heads, top-2048 of 131072: 0.8 GB, 120 us), and is bound by the instructions and
// shared-memory cycles per candidate: insert (one atomic), rank (two loads), membership (one atomic),
// list entry (one store; expanding the list from the bitmap instead was 5 % slower).
#include "common.cuh"

namespace lt {


struct UnionParams {
  const int32_t* idx;       // [T, k]
  int32_t* u_phys;          // [ng, cap]
  int32_t* counts;          // [ng]
  uint32_t* memb;           // [ng, G, cap/32], or null: no membership words (one list per tile needs none)
  const int32_t* req_pg;    // [ng] or null (identity table)
  const int32_t* btab;      // [nreq, bt_stride] or null
  int bt_stride, bt_blocks, bsz;
  uint32_t bsz_mul;         // ceil(2^32 / bsz), or 0: divide
  int kq;                   // k / 4: 16-byte loads per token row
  uint32_t kq_mul;          // ceil(2^32 / kq), or 0: divide
  int k, G, cap, s_words;   // s_words = seq_space / 32
  int quads_per_thread;     // 16-byte bitmap quads a thread counts: 1 or odd (conflict-free reads)
  int window;               // list entries staged in shared memory; later ones are written directly
  int fill_tail;            // 1: also write -1 / 0 beyond the live prefixes; 2: -1 up to the next multiple of 128, 128 entries at least
};

// Shared-memory carve-up (bytes): bitmap | rank table (u16) | qm accumulator | list window
__host__ __device__ inline size_t union_smem_bytes(int s_words, int rank_shift, int G, int cap, int window) {
  return (size_t)s_words * 4 + (size_t)(s_words >> rank_shift) * 2 + (size_t)G * (cap / 32) * 4 + (size_t)window * 4;
}

// n / d through a multiply-high when the host proved it exact (n * d < 2^32, d > 1)
__device__ __forceinline__ int fast_div(int n, int d, uint32_t mul) {
  return mul ? (int)__umulhi((uint32_t)n, mul) : n / d;
}
inline uint32_t fast_div_mul(int64_t n_max, int d) {
  if (d <= 1 || n_max * d >= (int64_t(1) << 32)) return 0;
  return (uint32_t)(((int64_t(1) << 32) + d - 1) / d);
}

// NT threads per tile; VPT int4 loads cached per thread (0: nothing cached, the second pass re-reads
// the tile).  RS: the rank table holds one entry per (1 << RS) bitmap words.  BT: block table.
template <int NT, int VPT, int RS, bool BT>
__global__ void __launch_bounds__(NT)
union_qm_kernel(const UnionParams p) {
  constexpr int NW = NT / 32;
  extern __shared__ __align__(16) uint32_t smem[];
  __shared__ int warp_tot[NW];

  const int g = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int s_words = p.s_words, cap = p.cap, capw = cap >> 5, total = p.G * p.k;
  const uint32_t S = (uint32_t)s_words << 5;
  uint32_t* bm = smem;                                          // s_words % 32 == 0: all parts are 16-byte aligned
  uint16_t* rtab = reinterpret_cast<uint16_t*>(bm + s_words);
  uint32_t* qm_s = reinterpret_cast<uint32_t*>(rtab + (s_words >> RS));
  int32_t* list_s = reinterpret_cast<int32_t*>(qm_s + (size_t)p.G * capw);

  // ---- clear the bitmap and the membership words (own memory: before the wait for the previous kernel)
  {
    uint4* b4 = reinterpret_cast<uint4*>(bm);
    for (int i = tid; i < (s_words >> 2); i += NT) b4[i] = make_uint4(0, 0, 0, 0);
    uint4* q4 = reinterpret_cast<uint4*>(qm_s);
    for (int i = tid; p.memb && i < (p.G * capw >> 2); i += NT) q4[i] = make_uint4(0, 0, 0, 0);
  }
  pdl_trigger();
  pdl_wait();
  // issue the tile's loads while the clear drains
  const int4* src = reinterpret_cast<const int4*>(p.idx + (size_t)g * total);
  const int nquad = total >> 2;
  int4 v[VPT > 0 ? VPT : 1];
  if (VPT > 0) {
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int qd = i * NT + tid;
      v[i] = qd < nquad ? __ldcg(src + qd) : make_int4(-1, -1, -1, -1);
    }
  }
  __syncthreads();

  // ---- insert
  auto insert = [&](int pos) {
    if ((uint32_t)pos < S) atomicOr(&bm[pos >> 5], 1u << (pos & 31));
  };
  if (VPT > 0) {
#pragma unroll
    for (int i = 0; i < VPT; ++i) { insert(v[i].x); insert(v[i].y); insert(v[i].z); insert(v[i].w); }
  } else {
    for (int qd = tid; qd < nquad; qd += NT) {
      const int4 t = __ldcg(src + qd);
      insert(t.x); insert(t.y); insert(t.z); insert(t.w);
    }
  }
  __syncthreads();

  // ---- rank of every word: each thread counts a run of quads; warp scan, then a scan of the warp totals
  const int nq_bm = s_words >> 2;
  const int q0 = min(tid * p.quads_per_thread, nq_bm), q1 = min(q0 + p.quads_per_thread, nq_bm);
  const uint4* b4 = reinterpret_cast<const uint4*>(bm);
  int mine = 0;
  for (int i = q0; i < q1; ++i) {
    const uint4 b = b4[i];
    mine += __popc(b.x) + __popc(b.y) + __popc(b.z) + __popc(b.w);
  }
  int incl = mine;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += t;
  }
  if (lane == 31) warp_tot[wid] = incl;
  __syncthreads();
  const int wt = lane < NW ? warp_tot[lane] : 0;
  int wincl = wt;
#pragma unroll
  for (int off = 1; off < NW; off <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, wincl, off);
    if (lane >= off) wincl += t;
  }
  const int live = __shfl_sync(0xffffffffu, wincl, NW - 1);     // <= G * k <= cap
  int r0 = __shfl_sync(0xffffffffu, wincl - wt, wid) + incl - mine;
  if (tid == 0) p.counts[g] = live;
  for (int i = q0; i < q1; ++i) {
    const uint4 b = b4[i];
    if (RS == 0) {
      const int r1 = r0 + __popc(b.x), r2 = r1 + __popc(b.y), r3 = r2 + __popc(b.z);
      reinterpret_cast<uint2*>(rtab)[i] = make_uint2((uint32_t)r0 | (uint32_t)r1 << 16, (uint32_t)r2 | (uint32_t)r3 << 16);
      r0 = r3 + __popc(b.w);
    } else {
      static_assert(RS == 0 || RS == 2, "one rank per word or per quad");
      rtab[i] = (uint16_t)r0;
      r0 += __popc(b.x) + __popc(b.y) + __popc(b.z) + __popc(b.w);
    }
  }
  __syncthreads();

  // ---- every candidate looks up its rank, sets its token's membership bit and writes its own entry of
  // the sorted list (duplicates write the same value)
  const int32_t* bt_row = BT ? p.btab + (size_t)p.req_pg[g] * p.bt_stride : nullptr;
  int32_t* out_row = p.u_phys + (size_t)g * cap;
  auto mark = [&](int pos, uint32_t* row) {
    if ((uint32_t)pos < S) {
      const int w = pos >> 5;
      int r = rtab[w >> RS];
      if (RS)
        for (int x = (w >> RS) << RS; x < w; ++x) r += __popc(bm[x]);
      r += __popc(bm[w] & ((1u << (pos & 31)) - 1u));
      if (p.memb) atomicOr(row + (r >> 5), 1u << (r & 31));
      int phys = pos;
      if (BT) {
        const int blk = fast_div(pos, p.bsz, p.bsz_mul);
        phys = blk < p.bt_blocks ? bt_row[blk] * p.bsz + (pos - blk * p.bsz) : -1;
      }
      if (r < p.window) list_s[r] = phys;
      else out_row[r] = phys;
    }
  };
  if (VPT > 0) {
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      // k % 4 == 0: the four candidates of one 16-byte load belong to one token (loads past the tile
      // are all -1)
      uint32_t* row = qm_s + fast_div(i * NT + tid, p.kq, p.kq_mul) * capw;
      mark(v[i].x, row); mark(v[i].y, row); mark(v[i].z, row); mark(v[i].w, row);
    }
  } else {
    for (int qd = tid; qd < nquad; qd += NT) {
      const int4 t = __ldcg(src + qd);
      uint32_t* row = qm_s + fast_div(qd, p.kq, p.kq_mul) * capw;
      mark(t.x, row); mark(t.y, row); mark(t.z, row); mark(t.w, row);
    }
  }
  __syncthreads();

  // ---- staged list -> global, 16-byte stores; the last quad is padded with -1
  {
    const int end = p.fill_tail == 1 ? cap : (p.fill_tail == 2 ? max(128, ((live + 127) >> 7) << 7) : (live + 3) & ~3);
    for (int i = tid; i < end >> 2; i += NT) {
      const int b = i << 2;
      if (b >= p.window && b + 3 < live) continue;              // written above (window % 4 == 0)
      if (b >= p.window && b < live) {                          // the last quad, partly written above
        for (int e = live; e < b + 4; ++e) out_row[e] = -1;
        continue;
      }
      int4 o = make_int4(-1, -1, -1, -1);
      if (b < live) {
        o = reinterpret_cast<const int4*>(list_s)[i];
        if (b + 1 >= live) o.y = -1;
        if (b + 2 >= live) o.z = -1;
        if (b + 3 >= live) o.w = -1;
      }
      reinterpret_cast<int4*>(out_row)[i] = o;
    }
  }

  // ---- live mask words, max(4, roundup4(ceil(live / 32))) per token (whole rows when fill_tail is 1;
  // the words beyond are still zero)
  {
    const int c4 = capw >> 2;
    const int per_row = p.fill_tail == 1 ? c4 : max(1, (live + 127) >> 7);
    const int runs = (per_row + 31) >> 5;                       // warp-wide pieces of a row
    uint4* dst = reinterpret_cast<uint4*>(p.memb + (size_t)g * p.G * capw);
    const uint4* s4 = reinterpret_cast<const uint4*>(qm_s);
    for (int c = wid; p.memb && c < p.G * runs; c += NW) {
      const int q = c / runs, j = 32 * (c - q * runs) + lane;
      if (j < per_row) dst[q * c4 + j] = s4[q * c4 + j];
    }
  }
}

template <int NT, int VPT, int RS>
static int launch_union_rs(const UnionParams& p, int ng, size_t smem, cudaStream_t stream) {
  const int dev = current_device();
  if (!(p.btab ? ensure_smem<union_qm_kernel<NT, VPT, RS, true>>(dev, smem) : ensure_smem<union_qm_kernel<NT, VPT, RS, false>>(dev, smem)))
    return LITEDSA_ERR_CUDA;
  return launch_pdl(p.btab ? union_qm_kernel<NT, VPT, RS, true> : union_qm_kernel<NT, VPT, RS, false>, dim3(ng), NT, smem,
                    stream, p);
}
template <int NT, int VPT>
static int launch_union(const UnionParams& p, int rank_shift, int ng, size_t smem, cudaStream_t stream) {
  return rank_shift ? launch_union_rs<NT, VPT, 2>(p, ng, smem, stream) : launch_union_rs<NT, VPT, 0>(p, ng, smem, stream);
}

// Shared memory (227 KB per CTA on sm_100): the whole list is staged if two CTAs fit on an SM then,
// else its first 8192 entries (a union is usually well below G * k); one rank per bitmap word if
// that fits, else one per quad.
constexpr size_t kUnionSmemLimit = 220 * 1024;
struct UnionSmem { int window, rank_shift; size_t bytes; };
static UnionSmem union_smem(int s_words, int G, int cap) {
  UnionSmem m{cap, 0, 0};
  if (union_smem_bytes(s_words, 0, G, cap, cap) > 110 * 1024) m.window = cap < 8192 ? cap : 8192;
  if (union_smem_bytes(s_words, 0, G, cap, m.window) > kUnionSmemLimit) m.window = cap < 1024 ? cap : 1024;
  if (union_smem_bytes(s_words, 0, G, cap, m.window) > kUnionSmemLimit) m.rank_shift = 2;
  m.bytes = union_smem_bytes(s_words, m.rank_shift, G, cap, m.window);
  return m;
}

// The shapes that a union of G lists of k entries takes: no CUDA call.
int check_union(int T, int k, int ng, int cap, int G, int64_t seq_space) {
  if (ng <= 0 || G <= 0 || k <= 0 || T != ng * G) return LITEDSA_ERR_SHAPE;
  if (cap < G * k || cap % 128 != 0) return LITEDSA_ERR_SHAPE;
  if (G > 16 || (int64_t)G * (cap / 32) > 16 * 1024) return LITEDSA_ERR_SHAPE;
  if (seq_space <= 0 || seq_space > (1 << 20)) return LITEDSA_ERR_SHAPE;
  if ((seq_space + 31) / 32 % 32 != 0) return LITEDSA_ERR_SHAPE;   // 1024-position aligned
  if (k % 4 != 0) return LITEDSA_ERR_UNSUPPORTED;    // 16-byte row loads
  if (cap > 65536) return LITEDSA_ERR_UNSUPPORTED;   // 16-bit rank table
  if (union_smem((int)((seq_space + 31) / 32), G, cap).bytes > kUnionSmemLimit) return LITEDSA_ERR_UNSUPPORTED;
  return LITEDSA_OK;
}

// Checks and launch behind litedsa_union_qm and litedsa_sparse_prefill; fill as UnionParams::fill_tail.
int run_union(const int32_t* topk_indices, int32_t* u_phys, int32_t* counts, uint32_t* memb_qm, const int32_t* req_pg,
              const int32_t* block_table, int T, int k, int ng, int cap, int G, int bt_rows, int bt_blocks,
              int block_size, int64_t seq_space, int fill, void* stream) {
  // same argument checks as the reference launcher (litedsa.cu:43-59)
  if (!topk_indices || !u_phys || !counts || (!memb_qm && G != 1)) return LITEDSA_ERR_ARG;
  const int rc = check_union(T, k, ng, cap, G, seq_space);
  if (rc == LITEDSA_ERR_SHAPE) return rc;
  const int s_words = (int)((seq_space + 31) / 32);
  if ((block_table != nullptr) != (req_pg != nullptr)) return LITEDSA_ERR_ARG;
  if (block_table && (block_size <= 0 || bt_blocks <= 0 || bt_rows <= 0)) return LITEDSA_ERR_SHAPE;
  if (rc != LITEDSA_OK) return rc;

  UnionParams p;
  p.idx = topk_indices; p.u_phys = u_phys; p.counts = counts; p.memb = memb_qm;
  p.req_pg = req_pg; p.btab = block_table;
  p.bt_stride = bt_blocks; p.bt_blocks = bt_blocks; p.bsz = block_table ? block_size : 1;
  p.bsz_mul = fast_div_mul(int64_t(s_words) * 32, p.bsz);
  p.kq = k / 4; p.kq_mul = fast_div_mul(int64_t(G) * (k / 4), k / 4);
  p.k = k; p.G = G; p.cap = cap; p.s_words = s_words; p.fill_tail = fill;
  const UnionSmem m = union_smem(s_words, G, cap);
  p.window = m.window;
  const int rank_shift = m.rank_shift;
  const size_t smem = m.bytes;

  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int quads = G * k / 4;
  // At most one tile per SM and more than 256 loads or bitmap quads in it: 1024 threads shorten the
  // tile's own chain of phases.  Otherwise 256 threads (512 for tiles that need more registers),
  // several tiles per SM.  (65536 tokens of 16 heads, top-2048 of 131072: 610 us with one CTA of 1024
  // threads per SM, 440 with two of 512; 16384 x 32 heads, top-1024 of 65536: 72 -> 55.)
  const bool small = quads <= 256 && s_words <= 1024;
  const int nt = ng <= sm_count() && !small ? 1024 : (quads <= 2048 ? 256 : 512);
  const int qpt = (s_words / 4 + nt - 1) / nt;
  p.quads_per_thread = qpt == 1 ? 1 : (qpt | 1);
  const int vpt = (quads + nt - 1) / nt;
  if (nt == 1024) {
    if (vpt <= 1) return launch_union<1024, 1>(p, rank_shift, ng, smem, st);
    if (vpt <= 4) return launch_union<1024, 4>(p, rank_shift, ng, smem, st);
    return launch_union<1024, 0>(p, rank_shift, ng, smem, st);
  }
  if (nt == 256) {
    if (vpt <= 1) return launch_union<256, 1>(p, rank_shift, ng, smem, st);
    if (vpt <= 4) return launch_union<256, 4>(p, rank_shift, ng, smem, st);
    return launch_union<256, 8>(p, rank_shift, ng, smem, st);
  }
  if (vpt <= 8) return launch_union<512, 8>(p, rank_shift, ng, smem, st);
  return launch_union<512, 0>(p, rank_shift, ng, smem, st);
}

}  // namespace lt

// C-ABI entry point; argument order and meaning follow the reference operator
// union_qm(topk_indices, u_phys, counts, memb_qm, req_pg, block_table, block_size, seq_space)
// (kernels/b200/dsa/litedsa.cu:31-75), with tensor shapes passed as integers.
extern "C" int litedsa_union_qm(const int32_t* topk_indices, int32_t* u_phys, int32_t* counts,
                                uint32_t* memb_qm, const int32_t* req_pg,
                                const int32_t* block_table, int T, int k, int ng, int cap, int G,
                                int bt_rows, int bt_blocks, int block_size, int64_t seq_space,
                                int fill_tail, void* stream) {
  if (!topk_indices || !u_phys || !counts || !memb_qm) return LITEDSA_ERR_ARG;
  if (cap != G * k) return LITEDSA_ERR_SHAPE;
  return lt::run_union(topk_indices, u_phys, counts, memb_qm, req_pg, block_table, T, k, ng, cap, G, bt_rows, bt_blocks,
                       block_size, seq_space, fill_tail != 0 ? 1 : 0, stream);
}
