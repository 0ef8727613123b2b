// Declarations of the decode kernel (hkv_decode.cu): launch parameters, the per-request view of the unit
// stream, and the log-sum-exp merge of a split sequence.
#pragma once

#include <cuda_bf16.h>

#include "hkv_common.cuh"

namespace hkv {

constexpr int kMaxRows = 64;     // G * qlmax: more rows than one pass serves are handled by several passes over the cache
constexpr float NEG_BIG = -1.0e30f;
constexpr float TAU = 8.0f;      // lazy rescale threshold (log2 domain): P stays below 2^8, inside f16's range

struct DecodeParams {
  const __nv_bfloat16* q;
  const uint8_t* kd;
  const uint8_t* ksf;
  const uint8_t* vd;
  const uint8_t* vsf;
  long long dsh, ssh;                                // byte strides between kv heads (codes, scales)
  unsigned dst;                                      // byte stride between positions of a page (row-copy layout only)
  unsigned dsp, ssp;                                 // byte strides between pages (codes, scales), < 2^31
  const int* bt;
  const int* seq_lens;
  const int* qsl;
  const float* gk;
  const float* gv;
  uint8_t* ws;
  __nv_bfloat16* out;
  int MP, B, KVH, G, qlmax, PS;
  const float* signs;                                // +-1 per channel when the keys were written rotated, else null
  float rot_scale;                                   // head_dim^-0.5 rounded to fp32
  int row0;                                          // first query row (of the G * ql rows of a request and kv head) of this pass
  int max_len;                                       // MP * PS, capped at INT_MAX
  int early_meta;                                    // seq_lens / query_start_loc are read before the launch dependency
  float scale_log2, v_scale;
};

// one request as the unit stream sees it; all fields are warp-uniform
struct ReqInfo {
  int U, L, ql, q0;                                    // units per kv head, context length, query tokens, first query row
};
template <int LOG_UT>
__device__ __forceinline__ ReqInfo load_req(const DecodeParams& p, int b) {
  ReqInfo r;
  r.q0 = __ldg(p.qsl + b);
  int ql = __ldg(p.qsl + b + 1) - r.q0;
  ql = (ql < 0 || ql > p.qlmax || p.G * ql <= p.row0) ? 0 : ql;     // (no rows in this pass: the request is skipped)
  r.ql = ql;
  // (a length beyond the block table's reach is cut there, so that bad metadata can never read past a table row)
  r.L = ql > 0 ? min(max(__ldg(p.seq_lens + b), 0), p.max_len) : 0;
  r.U = ql > 0 ? max(1, (r.L + (1 << LOG_UT) - 1) >> LOG_UT) : 0;
  return r;
}

// a split sequence as the ticket round at the end of a partition needs it
struct SplitSeq {
  int h, U, q0, R;                                   // kv head, units of the whole sequence, first query token, rows of this pass
  long long seq0;                                    // stream position of the sequence (its cost slots come first)
};

// ------------------------------------------------------------------------------------------------------- combine
// Log-sum-exp merge of P pieces of one split sequence by the whole CTA (NT threads) that drew their last ticket: all pieces
// of the sequence, or a group of them (kGroup below). w_i = 2^(lse_i - max), result sum w_i part_i / sum w_i, accumulated in
// partition order, so it does not depend on which CTA merges. (Reference: hz4::combine_rg, kv_fp4_serving.py:518-558.)
//
// What bounds it is the latency of its loads from L2: nobody else works on the sequence by then. Up to eight pieces (FEW) are
// loaded with their log-sum-exps in one round trip per eight rows (four at head_dim 256). For more, the weights of all pieces
// come first, in one round trip through shared memory, and a thread then has sixteen partials in flight whatever they weigh.
// Launches back to back (`microbench decode --iters 2000 --batch B --min-len L --max-len L ..`), before (rounds of four pieces
// under a running maximum, partitions of any size) -> now, with the two steps below and kMinPer: one request of 6453 tokens,
// 8 kv heads x 128, 51 -> 26 pieces a head, 24.4 -> 14.7 us (15.9 with the 51 pieces); of 32768 tokens, 2 x 256, 147 -> 129
// pieces, 101 -> 26.5; eight of 131072, 8 x 128, 7 pieces, 236 both.
struct Pieces {
  const float* lse;                                  // [slot][RP]
  const float* part;                                 // [slot][RP][D]
  int first_slot, first, step, n;                    // piece 0 lies in first_slot, piece i in slot 0 of partition first + i * step
  __device__ __forceinline__ int slot(int i) const { return i == 0 ? first_slot : 2 * (first + i * step); }
};
// where the merged rows go: the output (row 0 of the (request, kv head) group's first query token; rows of the next token are
// tok_stride elements further), or back into the partial of the first piece, which only this CTA reads any more
struct MergeOut {
  __nv_bfloat16* row0;                               // null: to `part` and `lse`
  long long tok_stride;
  float v_scale;
  int first_row, G;                                  // row r of the pass is row first_row + r of the group
  float* part;
  float* lse;
};
template <int D>
__device__ __forceinline__ void merge_store(const MergeOut& o, int row, int ch, float4 a, float total) {
  const float inv = total > 0.0f ? (o.row0 ? o.v_scale : 1.0f) / total : 0.0f;
  a.x *= inv; a.y *= inv; a.z *= inv; a.w *= inv;
  if (o.row0) {
    const int t = (o.first_row + row) / o.G, gq = o.first_row + row - t * o.G;
    const __nv_bfloat162 lo = __floats2bfloat162_rn(a.x, a.y), hi = __floats2bfloat162_rn(a.z, a.w);
    *reinterpret_cast<uint2*>(o.row0 + t * o.tok_stride + (long long)gq * D + ch) =
        make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
  } else {
    *reinterpret_cast<float4*>(o.part + (size_t)row * D + ch) = a;
  }
}
// sm: RP + cap floats of shared memory
template <int D, int RP, int NT>
__device__ __forceinline__ void merge_pieces(const Pieces& pc, int R, const MergeOut& o, float* sm, int cap) {
  constexpr int C4 = D / 4;                          // threads of a row, four channels each
  // (six in the sixteen-row kernel at head_dim 256, whose registers are the tightest: with eight it takes 255 and spills. 96
  // requests of 0.5k to 16k tokens, 2 kv heads, group 8 x 2 query tokens: 96.6 us with eight, 93.9 with six, 97.9 with four)
  constexpr int FEW = D == 256 && RP == 16 ? 6 : 8, GRP = 16;
  const float ninf = -__int_as_float(0x7f800000);
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const int P = pc.n, lane = threadIdx.x & 31;
  auto fma4 = [](float4& a, const float4& v, float w) {
    a.x = fmaf(v.x, w, a.x);
    a.y = fmaf(v.y, w, a.y);
    a.z = fmaf(v.z, w, a.z);
    a.w = fmaf(v.w, w, a.w);
  };
  auto load = [&](int i, int row, int ch) {
    return __ldcg(reinterpret_cast<const float4*>(pc.part + ((size_t)pc.slot(i) * RP + row) * D + ch));
  };
  if (P <= FEW && o.row0) {
    constexpr int IT = 2, RB = IT * NT / C4;         // items of a thread, rows at a time
    for (int rb = 0; rb < R; rb += RB) {
      float ls[IT][FEW];
      float4 v[IT][FEW];
#pragma unroll
      for (int it = 0; it < IT; ++it) {
        const int idx = threadIdx.x + it * NT, row = rb + idx / C4, ch = idx % C4 * 4;
#pragma unroll
        for (int i = 0; i < FEW; ++i) {
          const bool on = i < P && row < R;
          ls[it][i] = on ? __ldcg(pc.lse + pc.slot(i) * RP + row) : ninf;
          v[it][i] = on ? load(i, row, ch) : zero;
        }
      }
#pragma unroll
      for (int it = 0; it < IT; ++it) {
        const int idx = threadIdx.x + it * NT, row = rb + idx / C4, ch = idx % C4 * 4;
        if (row >= R) continue;
        float m = ls[it][0], tot = 0.0f;
#pragma unroll
        for (int i = 1; i < FEW; ++i) m = fmaxf(m, ls[it][i]);
        float4 a = zero;
#pragma unroll
        for (int i = 0; i < FEW; ++i) {
          if (ls[it][i] == ninf) continue;           // an empty piece: its partial is garbage and must not be used
          const float w = exp2f(ls[it][i] - m);
          tot += w;
          fma4(a, v[it][i], w);
        }
        merge_store<D>(o, row, ch, a, tot);
      }
    }
    return;
  }
  const int fit = max(1, min(R, cap / P));           // rows whose weights fit the shared memory
  float* const sum = sm;
  float* const wt = sm + RP;                         // [row][piece]; -0: an empty piece, whose partial is garbage, not to be used
  for (int rb = 0; rb < R; rb += fit) {
    const int nr = min(fit, R - rb);
    __syncthreads();                                 // the shared memory's last use is over
#pragma unroll 4
    for (int i = threadIdx.x; i < nr * P; i += NT) {
      const int k = i / nr, r = i - k * nr;
      wt[r * P + k] = __ldcg(pc.lse + pc.slot(k) * RP + rb + r);
    }
    __syncthreads();
    for (int r = threadIdx.x >> 5; r < nr; r += NT / 32) {
      float m = ninf, s = 0.0f;
      for (int k = lane; k < P; k += 32) m = fmaxf(m, wt[r * P + k]);
#pragma unroll
      for (int x = 16; x > 0; x >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, x));
      for (int k = lane; k < P; k += 32) {
        const float x = wt[r * P + k], w = x == ninf ? -0.0f : exp2f(x - m);
        wt[r * P + k] = w;
        s += w;
      }
#pragma unroll
      for (int x = 16; x > 0; x >>= 1) s += __shfl_xor_sync(0xffffffffu, s, x);
      if (lane == 0) {
        sum[r] = s;
        if (!o.row0) o.lse[rb + r] = s > 0.0f ? m + log2f(s) : ninf;
      }
    }
    __syncthreads();
    for (int item = threadIdx.x; item < nr * C4; item += NT) {
      const int r = item / C4, ch = item % C4 * 4;
      const float* w = wt + r * P;
      float4 a = zero;
      for (int k0 = 0; k0 < P; k0 += GRP) {
        float4 v[GRP];
        float wg[GRP];
#pragma unroll
        for (int i = 0; i < GRP; ++i) {              // (a weight that underflowed to zero still carries a NaN or an infinity)
          wg[i] = k0 + i < P ? w[k0 + i] : -0.0f;
          v[i] = __float_as_int(wg[i]) >= 0 ? load(k0 + i, rb + r, ch) : zero;
        }
#pragma unroll
        for (int i = 0; i < GRP; ++i) fma4(a, v[i], wg[i]);
      }
      merge_store<D>(o, rb + r, ch, a, sum[r]);
    }
  }
}

// Tickets. A sequence in more than kGroupFrom pieces is merged in two steps: groups of kGroup neighbouring pieces by the CTA
// that finishes the group's last piece, then the groups by the CTA that merges the last of them. One CTA alone reads 129 pieces
// at what one SM gets from L2 (the launch above: 40.9 us), the groups are read by as many SMs (26.5 us). The line, one request,
// in one step / in two: 8 x 128, 26 pieces (6453 tokens) 14.7 / 16.7 us, 48 pieces 16.6 / 17.4, 54 pieces 21.3 / 21.6; 2 x 256,
// 17 pieces 18.6 / 20.8, 31 pieces 20.3 / 21.4, 33 pieces 21.0 / 21.2, 48 pieces 23.2 / 22.0; sixteen rows there, 33 pieces
// 31.4 / 29.6. The counters lie in tickets[last partition of the group / of the sequence]: finished pieces of a group in the low
// 16 bits, merged groups of the sequence in the high ones. They are zero between launches. (No other split sequence ends in
// such a partition, so no other one counts there.)
constexpr int kGroup = 16, kGroupFrom = 32;
struct Group {
  int first, last;                                   // partitions
};
__device__ __forceinline__ Group group_of(int part, int first, int last) {
  if (last - first + 1 <= kGroupFrom) return {first, last};
  const int g0 = first + (part - first) / kGroup * kGroup;
  return {g0, min(g0 + kGroup - 1, last)};
}
// counts a finished piece of its group; true for the last one
__device__ __forceinline__ bool draw_piece(int* tickets, Group g) {
  __threadfence();
  const int n = g.last - g.first + 1;
  const bool win = (atomicAdd(tickets + g.last, 1) & 0xffff) == n - 1;
  if (win) atomicSub(tickets + g.last, n);
  return win;
}
// counts a merged group of the sequence; true for the last one
__device__ __forceinline__ bool draw_group(int* tickets, int first, int last) {
  __threadfence();
  const int n = (last - first) / kGroup + 1;
  const bool win = (atomicAdd(tickets + last, 0x10000) >> 16) == n - 1;
  if (win) atomicSub(tickets + last, n << 16);
  return win;
}

}  // namespace hkv
