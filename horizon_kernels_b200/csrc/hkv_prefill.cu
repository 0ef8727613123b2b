// Prefill attention over the FP4 cache: requests with many query tokens (fresh prompts, chunks of long prompts, prompts
// with a cached prefix) in three kinds of launches.
//
//   tile_kernel     cached tokens -> 16-bit operand tiles of 128 keys, written once, in the byte order in which the
//                   tensor core reads them from shared memory (128-byte swizzle; values transposed), so that
//                   attend_kernel fetches a tile with plain contiguous bulk copies and needs no tensor map
//   attend_kernel   flash attention on tcgen05: scores and output accumulate in tensor memory, probabilities are
//                   handed to the value product through tensor memory
//   merge_kernel    joins the parts of row tiles whose keys were divided among CTAs (only when there are any)
//
// Replaces the reference's library attention over dequantised tokens (backend.py:438-543).
//
// Device times on a B200 (ncu, one launch alone; write launch included in the totals): a fresh prompt of 6144 tokens, 32
// query heads over 8 kv heads, head_dim 128: tile 12 us, attend 308 us (1.0 PFLOP/s), merge 9 us; the layer step 366 us
// against 16.5 ms with torch matmuls and eager softmax passes, whose fp32 score matrices went through memory. 2048 tokens
// over 30000 cached, 16 heads over 2, head_dim 256: tile 28 us, attend 683 us (1.54 PFLOP/s), merge 10 us; the step 0.84
// ms (the power cap lowers the clock) against 15.0 ms.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "hkv_common.cuh"

namespace hkv {

int record_cuda(cudaError_t e);

constexpr int kPfReqs = 32;            // requests per launch (the tables below are kernel arguments, at most 4 KB)
constexpr int kPfCtas = 160;           // CTAs per launch
constexpr int kKeys = 128;             // keys per tile
constexpr int kPieceCost = 3;          // cost of starting and ending a piece, in key tiles (of about 1 us)
constexpr int kMinPiece = 2;           // no piece of a divided row tile is shorter, in key tiles
constexpr int kStageBytes = 32768;
constexpr int kStages = 5;
constexpr int kPfThreads = 320;        // 8 softmax warps, the MMA warp, the copy warp
constexpr uint32_t kQBytes = 65536;    // query operands: 256 rows x 128 or 128 rows x 256 channels, 16 bits

// rows of the tensor-core tiles: a "piece row tile" has NT sub-tiles of 128 rows; row r of a sub-tile is query head
// r % G of token r / G, so that a sub-tile covers 128 / G consecutive tokens and its causal edge is short
template <int D>
struct PfShape {
  static constexpr int NT = D == 128 ? 2 : 1;
  static constexpr int ROWS = NT * 128;
  static constexpr int COLS = D == 128 ? 128 : 64;      // score columns of a softmax thread
  static constexpr int OCOL = 256;                      // tensor-memory column of the output accumulators
  static constexpr int PCOL = D == 128 ? 64 : 0;        // probabilities, from the thread's first score column
  static constexpr int PHALF = D == 128 ? 32 : 64;      // columns from the first 64 keys' probabilities to the others'
};

struct PfReq {
  int q0, ql, L;
  int tile0;                           // first key tile of the request in the operand scratch
};
struct PfStart {                       // where a CTA's share of the key tiles begins (the next CTA's start ends it)
  int kt, rt;
  short h, req;
};
struct PfSplit {                       // a row tile in parts: the last part of CTA c1, all of the CTAs between, the first of c2
  short c1, c2, slot1, pad;
};

struct PrefillParams {
  const void* q;
  void* out;
  const uint8_t* tiles;
  float* part_o;                       // [CTA][2][ROWS][D]
  float* part_ml;                      // [CTA][2][2][ROWS]: running maximum (log2 domain), sum
  float* state_o;                      // chunked contexts: [token][head][D], then the same tables per row
  float* state_ml;
  int* status;
  float c, vs;                         // score scale x log2(e) (> 0), output scale
  uint32_t q_flip;                     // 0x80008000 when the score scale is negative
  int q_cvt, out_f32, k_bf16;
  int KVH, G, tok;                     // tok: query tokens per sub-tile (128 / G)
  int n_req;
  int kt_lo, kt_hi;                    // key tiles of this launch's chunk
  int first_chunk;
  PfReq req[kPfReqs];
  PfStart start[kPfCtas + 1];
  PfSplit split[kPfCtas];
};
static_assert(sizeof(PrefillParams) <= 4096, "kernel arguments");

// one past the last key tile (of the chunk) that a row tile sees; at least one tile, so that rows without any visible
// key still get their zero output
__host__ __device__ inline int pf_hi(const PfReq& r, int rt, int piece_tok, int kt_hi) {
  const int t_end = min(r.ql, (rt + 1) * piece_tok);
  const int vis = max(1, min(r.L, r.L - r.ql + t_end));
  return min((vis + kKeys - 1) / kKeys, kt_hi);
}
__host__ __device__ inline int pf_row_tiles(const PfReq& r, int piece_tok) { return (r.ql + piece_tok - 1) / piece_tok; }

struct Walk {
  int req, h, rt, kt;
  __host__ __device__ bool same_tile(const PfStart& e) const { return req == e.req && h == e.h && rt == e.rt; }
  // the next row tile that has keys in this chunk
  __host__ __device__ void advance(const PfReq* r, int n_req, int KVH, int piece_tok, int kt_lo, int kt_hi) {
    kt = kt_lo;
    do {
      if (++rt >= pf_row_tiles(r[req], piece_tok)) {
        rt = 0;
        if (++h >= KVH) { h = 0; ++req; }
      }
    } while (req < n_req && pf_hi(r[req], rt, piece_tok, kt_hi) <= kt_lo);
  }
};

// ------------------------------------------------------------------------------------------------------- tile_kernel
struct TileParams {
  const uint8_t* kd;
  const uint8_t* ksf;
  const uint8_t* vd;
  const uint8_t* vsf;
  long long dsp, dst, dsh, ssp, sst, ssh;
  const int* bt;
  uint8_t* tiles;
  int MP, PS, KVH, n_req;
  int kt_lo, n_tiles;                  // first key tile of the chunk; key tiles of the launch
  int row[kPfReqs];                    // block-table rows
  int L[kPfReqs];
  int tile0[kPfReqs];
};

template <int BF16>
__device__ __forceinline__ uint32_t operand_pair(uint32_t h2) {       // f16x2 -> the key operand's type (exact)
  if (!BF16) return h2;
  const __half2 h = u32_as_h2(h2);
  const __nv_bfloat162 b = __floats2bfloat162_rn(__low2float(h), __high2float(h));
  return *reinterpret_cast<const uint32_t*>(&b);
}

// One CTA = one key tile of one kv head and side: 128 x D values of 4 (K8: 8) bits in, 16 bits out. Keys: D / 64 images
// of 128 rows (keys) x 128 bytes; values: 2 images of D rows (channels) x 128 bytes (64 keys). Byte b of row r lies at
// r * 128 + (b ^ ((r & 7) << 4)): the 128-byte swizzle. HBM-bound on its output; every value is converted once per
// launch, whereas converting inside attend_kernel would repeat it for every row tile (128 times in the chunk above).
template <int D, int BF16, int K8>
__global__ void __launch_bounds__(128) tile_kernel(const __grid_constant__ TileParams p) {
  constexpr int NB = D / 16;
  pdl_wait();                                     // the cache may come from the preceding launch
  pdl_launch_dependents();
  const int side = blockIdx.z, h = blockIdx.y, gt = blockIdx.x, tid = threadIdx.x;
  int r = 0;
  while (r + 1 < p.n_req && p.tile0[r + 1] <= gt) ++r;
  const int n_t = (r + 1 < p.n_req ? p.tile0[r + 1] : p.n_tiles) - p.tile0[r];
  const int pos0 = (p.kt_lo + gt - p.tile0[r]) * kKeys, L = p.L[r];
  const int* bt = p.bt + (long long)p.row[r] * p.MP;
  const size_t image = (size_t)kKeys * D * 2;
  // request r's tiles: [head][tile][K, V]
  uint8_t* dst = p.tiles + ((size_t)p.tile0[r] * p.KVH + (size_t)h * n_t + (gt - p.tile0[r])) * 2 * image + side * image;
  if (side == 0) {
#pragma unroll 4
    for (int it = tid; it < kKeys * NB; it += 128) {
      const int blk4 = it & 3, key = (it >> 2) & 127, kb = it >> 9;   // four lanes write the 128 bytes of an image row
      const int blk = kb * 4 + blk4, pos = pos0 + key;
      uint32_t o[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] = 0;
      if (pos < L && pos / p.PS < p.MP) {
        const long long page = __ldg(bt + pos / p.PS), off = pos % p.PS;
        if (K8) {
          const uint4 w8 = *reinterpret_cast<const uint4*>(p.kd + page * p.dsp + off * p.dst + h * p.dsh + blk * 16);
          const uint32_t ws[4] = {w8.x, w8.y, w8.z, w8.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint32_t lo, hi;
            e4m3x4_to_f16x2(ws[i], lo, hi);
            o[2 * i] = operand_pair<BF16>(lo);
            o[2 * i + 1] = operand_pair<BF16>(hi);
          }
        } else {
          const uint2 w = *reinterpret_cast<const uint2*>(p.kd + page * p.dsp + off * p.dst + h * p.dsh + blk * 8);
          const __half2 s2 = __low2half2(u32_as_h2(e4m3x2_to_f16x2(p.ksf[page * p.ssp + off * p.sst + h * p.ssh + blk])));
          uint32_t a[4], b[4];
          e2m1x8_to_f16x2(w.x, a);
          e2m1x8_to_f16x2(w.y, b);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            o[i] = operand_pair<BF16>(hmul2h(a[i], s2));
            o[4 + i] = operand_pair<BF16>(hmul2h(b[i], s2));
          }
        }
      }
      uint8_t* rowp = dst + (size_t)kb * 16384 + key * 128;
      *reinterpret_cast<uint4*>(rowp + (((blk4 * 2) ^ (key & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
      *reinterpret_cast<uint4*>(rowp + (((blk4 * 2 + 1) ^ (key & 7)) << 4)) = make_uint4(o[4], o[5], o[6], o[7]);
    }
  } else {
    // eight keys x sixteen channels per thread; eight lanes write the 128 bytes (64 keys) of a channel's row
    for (int it = tid; it < 16 * NB; it += 128) {
      const int c = it & 7, rest = it >> 3, kb = rest & 1, blk = rest >> 1;
      uint32_t e[8][8];                           // [key][channel pair]
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int pos = pos0 + kb * 64 + c * 8 + k;
        uint2 w = make_uint2(0, 0);
        uint32_t sb = 0;
        if (pos < L && pos / p.PS < p.MP) {
          const long long page = __ldg(bt + pos / p.PS), off = pos % p.PS;
          w = *reinterpret_cast<const uint2*>(p.vd + page * p.dsp + off * p.dst + h * p.dsh + blk * 8);
          sb = p.vsf[page * p.ssp + off * p.sst + h * p.ssh + blk];
        }
        const __half2 s2 = __low2half2(u32_as_h2(e4m3x2_to_f16x2(sb)));
        uint32_t a[4], b[4];
        e2m1x8_to_f16x2(w.x, a);
        e2m1x8_to_f16x2(w.y, b);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          e[k][i] = hmul2h(a[i], s2);
          e[k][4 + i] = hmul2h(b[i], s2);
        }
      }
      uint8_t* img = dst + (size_t)kb * D * 128;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int d = blk * 16 + 2 * i + half;
          const uint32_t sel = half ? 0x7632 : 0x5410;
          const uint4 v = make_uint4(__byte_perm(e[0][i], e[1][i], sel), __byte_perm(e[2][i], e[3][i], sel),
                                     __byte_perm(e[4][i], e[5][i], sel), __byte_perm(e[6][i], e[7][i], sel));
          *reinterpret_cast<uint4*>(img + d * 128 + ((c ^ (d & 7)) << 4)) = v;
        }
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------- rotated queries
// bf16 query rows -> bf16(FWHT(q * signs) * D^-0.5), butterflies in fp32 in the reference's stage order (rotate_q,
// kv_fp4_ref.py:76-92, bit for bit) -> the compute type. One warp per row: a lane holds D / 32 adjacent channels, the
// first stages stay inside the lane, the others exchange between lanes.
template <int D>
__global__ void __launch_bounds__(256) rotate_kernel(const __nv_bfloat16* q, const float* signs, uint32_t* out, long long rows,
                                                     float scale, int to_bf16) {
  constexpr int V = D / 32;
  pdl_wait();
  pdl_launch_dependents();
  const long long row = (long long)blockIdx.x * 8 + threadIdx.x / 32;
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  float x[V];
#pragma unroll
  for (int i = 0; i < V; ++i) x[i] = __bfloat162float(q[row * D + lane * V + i]) * __ldg(signs + lane * V + i);
#pragma unroll
  for (int s = 1; s < V; s *= 2)
#pragma unroll
    for (int i = 0; i < V; ++i)
      if (!(i & s)) {
        const float a = x[i], b = x[i | s];
        x[i] = a + b;
        x[i | s] = a - b;
      }
#pragma unroll
  for (int s = 1; s < 32; s *= 2)
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const float o = __shfl_xor_sync(0xffffffffu, x[i], s);
      x[i] = (lane & s) ? o - x[i] : x[i] + o;
    }
#pragma unroll
  for (int i = 0; i < V; i += 2) {
    const __nv_bfloat162 b = __floats2bfloat162_rn(x[i] * scale, x[i + 1] * scale);
    const uint32_t w = *reinterpret_cast<const uint32_t*>(&b);
    out[(row * D + lane * V + i) / 2] = to_bf16 ? w : pack_f16x2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  }
}

// ----------------------------------------------------------------------------------------------------- attend_kernel
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr) {
  // K-major operand, 128-byte swizzle: 8-row groups 1024 bytes apart, descriptor version 1
  return (uint64_t)((smem_addr >> 4) & 0x3FFF) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void umma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc)
               : "memory");
}
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(acc)
               : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

#define HKV_R32(x) "=r"((x)[0]), "=r"((x)[1]), "=r"((x)[2]), "=r"((x)[3]), "=r"((x)[4]), "=r"((x)[5]), "=r"((x)[6]), \
  "=r"((x)[7]), "=r"((x)[8]), "=r"((x)[9]), "=r"((x)[10]), "=r"((x)[11]), "=r"((x)[12]), "=r"((x)[13]), "=r"((x)[14]), \
  "=r"((x)[15]), "=r"((x)[16]), "=r"((x)[17]), "=r"((x)[18]), "=r"((x)[19]), "=r"((x)[20]), "=r"((x)[21]), \
  "=r"((x)[22]), "=r"((x)[23]), "=r"((x)[24]), "=r"((x)[25]), "=r"((x)[26]), "=r"((x)[27]), "=r"((x)[28]), \
  "=r"((x)[29]), "=r"((x)[30]), "=r"((x)[31])
#define HKV_RW32(x) "+r"((x)[0]), "+r"((x)[1]), "+r"((x)[2]), "+r"((x)[3]), "+r"((x)[4]), "+r"((x)[5]), "+r"((x)[6]), \
  "+r"((x)[7]), "+r"((x)[8]), "+r"((x)[9]), "+r"((x)[10]), "+r"((x)[11]), "+r"((x)[12]), "+r"((x)[13]), "+r"((x)[14]), \
  "+r"((x)[15]), "+r"((x)[16]), "+r"((x)[17]), "+r"((x)[18]), "+r"((x)[19]), "+r"((x)[20]), "+r"((x)[21]), \
  "+r"((x)[22]), "+r"((x)[23]), "+r"((x)[24]), "+r"((x)[25]), "+r"((x)[26]), "+r"((x)[27]), "+r"((x)[28]), \
  "+r"((x)[29]), "+r"((x)[30]), "+r"((x)[31])
#define HKV_I16(x) "r"((x)[0]), "r"((x)[1]), "r"((x)[2]), "r"((x)[3]), "r"((x)[4]), "r"((x)[5]), "r"((x)[6]), \
  "r"((x)[7]), "r"((x)[8]), "r"((x)[9]), "r"((x)[10]), "r"((x)[11]), "r"((x)[12]), "r"((x)[13]), "r"((x)[14]), \
  "r"((x)[15])

// 32 columns of this thread's lane; tm_ready() must stand between the load and the first use
__device__ __forceinline__ void tm_ld32(uint32_t* x, uint32_t addr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
      "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : HKV_R32(x)
      : "r"(addr));
}
__device__ __forceinline__ void tm_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// keeps the uses of loaded registers behind the wait (an empty statement that passes them through)
__device__ __forceinline__ void tm_ready(uint32_t* x) { asm volatile("" : HKV_RW32(x)); }
__device__ __forceinline__ void tm_st16(uint32_t addr, const uint32_t* x) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::HKV_I16(x),
      "r"(addr)
      : "memory");
}

__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

struct PfShared {
  uint64_t full[kStages], empty[kStages];
  uint64_t q_full[2], s_full[2], p_full[2], o_done[2];
  uint64_t pair[4];                    // head_dim 256: the two warps that share 32 rows exchange maxima and sums
  uint64_t drain;
  uint32_t tmem;
  int abort;
};
constexpr int kPfSmem = (int)kQBytes + kStages * kStageBytes + 2048 + 512;
static_assert(sizeof(PfShared) <= 512 && kPfSmem <= 232448, "shared memory");

// bounded wait: gives up when it runs out or when another role of the CTA has given up
__device__ __forceinline__ bool pf_wait_slow(uint32_t bar, uint32_t parity, volatile int* abort) {
  const long long t0 = clock64();
  while (!mbar_try_wait_u32(bar, parity)) {
    if (*abort) return false;
    if (clock64() - t0 > kWaitCycles) {
      *abort = 1;
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ bool pf_wait(uint32_t bar, uint32_t parity, volatile int* abort) {
  if (mbar_try_wait_u32(bar, parity)) return true;
  return pf_wait_slow(bar, parity, abort);
}

__device__ __forceinline__ void store_out(const PrefillParams& p, long long elem, const float* v) {   // 8 values
  if (p.out_f32) {
    float4* o = reinterpret_cast<float4*>((float*)p.out + elem);
    o[0] = make_float4(v[0], v[1], v[2], v[3]);
    o[1] = make_float4(v[4], v[5], v[6], v[7]);
  } else {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&b);
    }
    *reinterpret_cast<uint4*>((__nv_bfloat16*)p.out + elem) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// One persistent CTA per SM. The key tiles of all row tiles form one stream that the host cuts into equal shares (with
// kPieceCost per piece), so that a chunk of 2048 tokens over 30k keys and four short prompts both occupy every SM to
// the end; a row tile whose keys were divided leaves unnormalised fp32 parts for merge_kernel.
//
// head_dim 128: two sub-tiles of 128 rows; while one has its scores exponentiated the tensor core works on the other.
//   tensor memory: S0 S1 O0 O1, 128 columns each.
// head_dim 256: one sub-tile (its output takes 256 columns), two score buffers; each score tile is shared by two
//   softmax warpgroups, 64 columns each, which agree on the row maximum through shared memory.
// Bound: tensor pipe and ex2 unit (16 per clock and SM: 1024 clocks per 128 x 128 scores, as long as the two products of
// head_dim 128, half as long as those of head_dim 256, which therefore reaches 0.92 of the burst peak and the other 0.60).
// The 16-bit probabilities overwrite their own scores in tensor memory. The running maximum moves only when a score
// exceeds it by 2^8 (the probabilities then stay below 2^8, inside f16), so the output is rarely rescaled.
template <int D>
__global__ void __launch_bounds__(kPfThreads, 1) attend_kernel(const __grid_constant__ PrefillParams p) {
  using S = PfShape<D>;
  constexpr int COLS = S::COLS;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* ring = smem + kQBytes;
  float* xch = reinterpret_cast<float*>(smem + kQBytes + kStages * kStageBytes);      // [2 turns][2 halves][128 rows]
  PfShared& sh = *reinterpret_cast<PfShared*>(smem + kQBytes + kStages * kStageBytes + 2048);
  volatile int* abort = &sh.abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int piece_tok = S::NT * p.tok;

  if (tid == 0) {
    sh.abort = (smem_u32(smem) & 1023) ? 1 : 0;        // the swizzled operands need 1024-byte alignment
    for (int i = 0; i < kStages; ++i) { mbar_init(&sh.full[i], 1); mbar_init(&sh.empty[i], 1); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sh.q_full[i], S::NT == 2 ? 128 : 256);
      mbar_init(&sh.s_full[i], 1);
      mbar_init(&sh.p_full[i], S::NT == 2 ? 128 : 256);
      mbar_init(&sh.o_done[i], 1);
    }
    for (int i = 0; i < 4; ++i) mbar_init(&sh.pair[i], 64);
    mbar_init(&sh.drain, 1);
    fence_barrier_init();
  }
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&sh.tmem)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh.tmem;
  pdl_wait();
  pdl_launch_dependents();

  const PfStart first = p.start[blockIdx.x], last = p.start[blockIdx.x + 1];
  Walk w{first.req, first.h, first.rt, first.kt};
  const uint32_t full0 = smem_u32(&sh.full[0]), empty0 = smem_u32(&sh.empty[0]), q_full0 = smem_u32(&sh.q_full[0]),
                 s_full0 = smem_u32(&sh.s_full[0]), p_full0 = smem_u32(&sh.p_full[0]), o_done0 = smem_u32(&sh.o_done[0]);

  if (warp == 9) {
    // ------------------------------------------------------------------------------------------------ copy warp
    if (elect_one()) {
      constexpr uint32_t IMAGE = kKeys * D * 2;
      constexpr int PER = IMAGE / kStageBytes;            // stages per operand tile: 1 or 2
      uint32_t fill = 0;
      bool ok = *abort == 0;
      while (ok && (!w.same_tile(last) || w.kt < last.kt)) {
        const PfReq r = p.req[w.req];
        const int hi = w.same_tile(last) ? last.kt : pf_hi(r, w.rt, piece_tok, p.kt_hi);
        const int n_t = min(p.kt_hi, (r.L + kKeys - 1) / kKeys) - p.kt_lo;
        const uint8_t* src = p.tiles + ((size_t)r.tile0 * p.KVH + (size_t)w.h * n_t - p.kt_lo) * 2 * IMAGE;
        auto fetch = [&](const uint8_t* from) {
          for (int i = 0; ok && i < PER; ++i) {
            const uint32_t st = fill % kStages, turn = fill / kStages;
            if (turn > 0) ok = pf_wait(empty0 + 8 * st, (turn - 1) & 1, abort);
            if (!ok) return;
            mbar_expect_tx_u32(full0 + 8 * st, kStageBytes);
            bulk_g2s_u32(smem_u32(ring) + st * kStageBytes, from + i * kStageBytes, kStageBytes, full0 + 8 * st);
            ++fill;
          }
        };
        fetch(src + (size_t)w.kt * 2 * IMAGE);
        for (int kt = w.kt; ok && kt < hi; ++kt) {
          if (kt + 1 < hi) fetch(src + (size_t)(kt + 1) * 2 * IMAGE);
          fetch(src + (size_t)kt * 2 * IMAGE + IMAGE);
        }
        if (w.same_tile(last)) break;
        w.advance(p.req, p.n_req, p.KVH, piece_tok, p.kt_lo, p.kt_hi);
      }
      if (!ok) {                       // nothing of this CTA's may still be on its way when it ends
        for (uint32_t f = fill > kStages ? fill - kStages : 0; f < fill; ++f)
          mbar_wait_bounded_u32(full0 + 8 * (f % kStages), (f / kStages) & 1);
      }
    }
  } else if (warp == 8) {
    // ------------------------------------------------------------------------------------------------- MMA warp
    if (elect_one()) {
      const uint32_t base = (1u << 4) | ((128u / 16) << 24);
      const uint32_t id_qk = base | ((128u / 8) << 17) | (p.k_bf16 ? (1u << 7) | (1u << 10) : 0u);
      const uint32_t id_pv = base | ((uint32_t)(D / 8) << 17);
      const uint32_t q_smem = smem_u32(smem), ring_a = smem_u32(ring);
      uint32_t use = 0, g = 0, piece = 0;                 // stages consumed, key tiles done, pieces done
      bool ok = *abort == 0;
      auto stage_wait = [&](uint32_t n) { return pf_wait(full0 + 8 * (n % kStages), (n / kStages) & 1, abort); };
      auto stage_addr = [&](uint32_t n) { return ring_a + (n % kStages) * kStageBytes; };
      // scores of a sub-tile: K tile in stages n (and n + 1)
      auto qk = [&](int sub, uint32_t n, uint32_t col) {
#pragma unroll
        for (int kb = 0; kb < D / 64; ++kb) {
          const uint64_t a = umma_desc(q_smem + sub * 32768 + kb * 16384);
          const uint64_t b = umma_desc(stage_addr(n + kb / 2) + (kb & 1) * 16384);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_ss(tmem + col, a + 2 * k, b + 2 * k, id_qk, kb + k > 0);
        }
      };
      auto pv = [&](uint32_t pcol, uint32_t n, uint32_t ocol, bool acc) {
#pragma unroll
        for (int kb = 0; kb < 2; ++kb) {
          const uint64_t b = umma_desc(D == 128 ? stage_addr(n) + kb * 16384 : stage_addr(n + kb));
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_ts(tmem + ocol, tmem + pcol + S::PCOL + kb * S::PHALF + k * 8, b + 2 * k, id_pv, acc || kb + k > 0);
        }
      };
      while (ok && (!w.same_tile(last) || w.kt < last.kt)) {
        const int hi = w.same_tile(last) ? last.kt : pf_hi(p.req[w.req], w.rt, piece_tok, p.kt_hi);
        const int n = hi - w.kt;
        if constexpr (D == 128) {
          ok = stage_wait(use);
          for (int t = 0; ok && t < 2; ++t) {
            ok = pf_wait(q_full0 + 8 * t, piece & 1, abort);
            if (!ok) break;
            tc_fence_after();
            qk(t, use, t * 128);
            umma_commit(s_full0 + 8 * t);
          }
          if (ok) umma_commit(empty0 + 8 * (use % kStages));
          ++use;
          for (int j = 0; ok && j < n; ++j, ++g) {
            const bool more = j + 1 < n;
            const uint32_t kst = use, vst = use + (more ? 1 : 0);
            use = vst + 1;
            for (int t = 0; ok && t < 2; ++t) {
              if (t == 0) ok = stage_wait(vst);
              ok = ok && pf_wait(p_full0 + 8 * t, g & 1, abort);
              if (!ok) break;
              tc_fence_after();
              pv(t * 128, vst, S::OCOL + t * 128, j > 0);
              umma_commit(o_done0 + 8 * t);
              if (more) {
                if (t == 0) ok = stage_wait(kst);
                if (!ok) break;
                qk(t, kst, t * 128);
                umma_commit(s_full0 + 8 * t);
              }
            }
            if (ok) {
              if (more) umma_commit(empty0 + 8 * (kst % kStages));
              umma_commit(empty0 + 8 * (vst % kStages));
            }
          }
        } else {
          ok = pf_wait(q_full0, piece & 1, abort) && stage_wait(use) && stage_wait(use + 1);
          if (ok) {
            tc_fence_after();
            qk(0, use, (g & 1) * 128);
            umma_commit(s_full0 + 8 * (g & 1));
            umma_commit(empty0 + 8 * (use % kStages));
            umma_commit(empty0 + 8 * ((use + 1) % kStages));
          }
          use += 2;
          for (int j = 0; ok && j < n; ++j, ++g) {
            if (j + 1 < n) {
              ok = stage_wait(use) && stage_wait(use + 1);
              if (!ok) break;
              qk(0, use, ((g + 1) & 1) * 128);
              umma_commit(s_full0 + 8 * ((g + 1) & 1));
              umma_commit(empty0 + 8 * (use % kStages));
              umma_commit(empty0 + 8 * ((use + 1) % kStages));
              use += 2;
            }
            ok = stage_wait(use) && stage_wait(use + 1) && pf_wait(p_full0 + 8 * (g & 1), (g >> 1) & 1, abort);
            if (!ok) break;
            tc_fence_after();
            pv((g & 1) * 128, use, S::OCOL, j > 0);
            umma_commit(o_done0 + 8 * (g & 1));
            umma_commit(empty0 + 8 * (use % kStages));
            umma_commit(empty0 + 8 * ((use + 1) % kStages));
            use += 2;
          }
        }
        ++piece;
        if (w.same_tile(last)) break;
        w.advance(p.req, p.n_req, p.KVH, piece_tok, p.kt_lo, p.kt_hi);
      }
      if (!ok) {                       // no product of this CTA's may still be running when its tensor memory is given back
        umma_commit(smem_u32(&sh.drain));
        mbar_wait_bounded_u32(smem_u32(&sh.drain), 0);
      }
    }
  } else {
    // -------------------------------------------------------------------------------------------- softmax warps
    const int wg = warp >> 2, quad = warp & 3;
    const int row = quad * 32 + lane;                     // of the sub-tile, = tensor-memory lane
    const int sub = D == 128 ? wg : 0;
    const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16);
    const uint32_t o_addr = lane_base + S::OCOL + wg * 128;
    const uint32_t pair_bar = smem_u32(&sh.pair[quad]);
    const uint32_t q_bar = q_full0 + 8 * sub;
    uint32_t turn = 0, g = 0;                             // exchanges done, key tiles done
    bool ok = *abort == 0;

    auto load_q = [&](const Walk& x) {
      // this warpgroup's (head_dim 256: both warpgroups') rows, 16 bytes per lane and load, whole rows per half warp or warp
      constexpr int LPR = D / 8;                          // lanes per row
      constexpr int NTH = D == 128 ? 128 : 256;
      const PfReq r = p.req[x.req];
      const int t = D == 128 ? (tid & 127) : tid;
      const int ch = t % LPR;
      uint8_t* qs = smem + sub * 32768 + (ch >> 3) * 16384;
      const int tok0 = x.rt * piece_tok + sub * p.tok;
      const int HQ = p.KVH * p.G;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint4 v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int rr = t / LPR + (half * 8 + i) * (NTH / LPR);
          const int tk = rr / p.G, token = tok0 + tk;
          v[i] = make_uint4(0, 0, 0, 0);
          if (tk < p.tok && token < r.ql) {
            const long long e = ((long long)(r.q0 + token) * HQ + x.h * p.G + (rr - tk * p.G)) * D + ch * 8;
            v[i] = *reinterpret_cast<const uint4*>((const uint16_t*)p.q + e);
          }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int rr = t / LPR + (half * 8 + i) * (NTH / LPR);
          uint32_t u[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            u[k] ^= p.q_flip;
            if (p.q_cvt) u[k] = pack_f16x2(__uint_as_float(u[k] << 16), __uint_as_float(u[k] & 0xffff0000u));
          }
          *reinterpret_cast<uint4*>(qs + rr * 128 + (((ch & 7) ^ (rr & 7)) << 4)) = make_uint4(u[0], u[1], u[2], u[3]);
        }
      }
      fence_proxy_async();
      mbar_arrive_u32(q_bar);
    };
    // head_dim 256: this thread's value and that of the thread that holds the row's other columns
    auto exchange = [&](float mine, float& other) {
      float* buf = xch + (turn & 1) * 256;
      buf[wg * 128 + row] = mine;
      mbar_arrive_u32(pair_bar);
      const bool good = __all_sync(0xffffffffu, pf_wait(pair_bar, turn & 1, abort));
      other = *(volatile float*)&buf[(wg ^ 1) * 128 + row];
      ++turn;
      return good;
    };

    // the value product of key tile n has completed (head_dim 256: the scores of tile n + 1 precede it, so two barriers take
    // turns, lest a wait meet a phase two behind)
    auto o_wait = [&](uint32_t n) {
      return __all_sync(0xffffffffu, D == 128 ? pf_wait(o_done0 + 8 * wg, n & 1, abort)
                                              : pf_wait(o_done0 + 8 * (n & 1), (n >> 1) & 1, abort));
    };

    bool first_piece = true;
    if (ok && (!w.same_tile(last) || w.kt < last.kt)) load_q(w);
    while (ok && (!w.same_tile(last) || w.kt < last.kt)) {
      const PfReq r = p.req[w.req];
      const bool cut = w.same_tile(last);                 // the row tile goes on in the next CTA
      const int tile_hi = pf_hi(r, w.rt, piece_tok, p.kt_hi);
      const int hi = cut ? last.kt : tile_hi;
      const int tk = row / p.G, gq = row - tk * p.G;
      const int token = w.rt * piece_tok + sub * p.tok + tk;
      const bool live = tk < p.tok && token < r.ql;
      const int lim = live ? max(0, min(r.L, r.L - r.ql + token + 1)) : 0;      // keys this row sees
      // tiles below this one are seen whole by every live row of the sub-tile (rows that do not exist may take any value)
      const int whole = max(0, min(r.L, r.L - r.ql + w.rt * piece_tok + sub * p.tok + 1)) / kKeys;
      float m = -INFINITY;
      unsigned long long l2 = 0;                          // two partial sums
      for (int kt = w.kt; kt < hi; ++kt, ++g) {
        const uint32_t sb = D == 128 ? (uint32_t)wg : (g & 1);
        const uint32_t ph = D == 128 ? (g & 1) : ((g >> 1) & 1);
        const uint32_t s_addr = lane_base + sb * 128 + (D == 128 ? 0 : wg * 64);
        ok = __all_sync(0xffffffffu, pf_wait(s_full0 + 8 * sb, ph, abort));
        if (!ok) break;
        tc_fence_after();
        const bool edge = kt >= whole;
        const int rel = lim - kt * kKeys - (D == 128 ? 0 : wg * 64);
        auto mask = [&](uint32_t* x, int col, int n) {    // scores of keys past the row's last one
#pragma unroll
          for (int i = 0; i < n; ++i)
            if (col + i >= rel) x[i] = 0xff800000u;
        };
        uint32_t s[COLS];
#pragma unroll
        for (int i = 0; i < COLS; i += 32) tm_ld32(s + i, s_addr + i);
        tm_wait_ld();
#pragma unroll
        for (int i = 0; i < COLS; i += 32) tm_ready(s + i);
        if (edge) mask(s, 0, COLS);
        float mx[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) mx[i] = __uint_as_float(s[i]);
#pragma unroll
        for (int i = 4; i < COLS; ++i) mx[i & 3] = fmaxf(mx[i & 3], __uint_as_float(s[i]));
        float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.c;
        if constexpr (D == 256) {
          float other;
          ok = exchange(top, other);
          if (!ok) break;
          top = fmaxf(top, other);
        }
        const bool move = top > m + 8.0f;
        if (__any_sync(0xffffffffu, move)) {
          const float m_new = move ? (top == INFINITY ? 0.0f : top) : m;
          const float al = move ? fast_exp2(m - m_new) : 1.0f;
          m = m_new;
          l2 = fma2(l2, pack2(al, al), 0ull);
          if (kt > w.kt) {
            // the last value product must have left the accumulator; the next waits for this warp's probabilities
            ok = o_wait(g - 1);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int i = 0; i < 128; i += 32) {
              uint32_t o[32];
              tm_ld32(o, o_addr + i);
              tm_wait_ld();
              tm_ready(o);
#pragma unroll
              for (int k = 0; k < 32; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * al);
              tm_st16(o_addr + i, o);
              tm_st16(o_addr + i + 16, o + 16);
            }
          }
        }
        const float mu = m == -INFINITY ? 0.0f : -m;
        const unsigned long long c2 = pack2(p.c, p.c), m2 = pack2(mu, mu);
        auto probs = [&](const uint32_t* x, uint32_t addr) {        // 32 scores -> 32 probabilities in 16 columns
          uint32_t ph16[16];
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            float a, b;
            unpack2(fma2(pack2(__uint_as_float(x[2 * k]), __uint_as_float(x[2 * k + 1])), c2, m2), a, b);
            a = fast_exp2(a);
            b = fast_exp2(b);
            l2 = add2(l2, pack2(a, b));
            ph16[k] = pack_f16x2(a, b);
          }
          tm_st16(addr, ph16);
        };
        if constexpr (D == 128) {
          // the second half of the scores stays in registers and its probabilities go over the columns it came from; the
          // first half is read once more (128 scores, their maximum and the packed results do not fit 168 registers)
          uint32_t r[64];
          tm_ld32(r, s_addr);
          tm_ld32(r + 32, s_addr + 32);
          probs(s + 64, s_addr + S::PCOL + 32);
          probs(s + 96, s_addr + S::PCOL + 48);
          tm_wait_ld();
          tm_ready(r);
          tm_ready(r + 32);
          if (edge) mask(r, 0, 64);
          probs(r, s_addr + S::PCOL);
          probs(r + 32, s_addr + S::PCOL + 16);
        } else {
          probs(s, s_addr + S::PCOL);
          probs(s + 32, s_addr + S::PCOL + 16);
        }
        tc_wait_st();
        tc_fence_before();
        mbar_arrive_u32(p_full0 + 8 * sb);
      }
      if (!ok) break;
      // the next piece's queries go in while the last value product runs (its scores have left the query operands)
      const Walk done = w;
      if (!cut) w.advance(p.req, p.n_req, p.KVH, piece_tok, p.kt_lo, p.kt_hi);
      if (!cut && (!w.same_tile(last) || w.kt < last.kt)) load_q(w);
      float l, l_hi;
      unpack2(l2, l, l_hi);
      l += l_hi;
      if constexpr (D == 256) {
        float other;
        ok = exchange(l, other);
        if (!ok) break;
        l += other;
      }
      ok = o_wait(g - 1);
      if (!ok) break;
      tc_fence_after();
      const bool divided = cut || done.kt > p.kt_lo;
      const int HQ = p.KVH * p.G;
      const int col0 = D == 128 ? 0 : wg * 128;
      float wo = 0.0f, wn = 1.0f, inv = 0.0f;
      long long st_row = 0;
      bool finish = true;
      float* part = nullptr;
      if (divided) {
        const long long slot = (long long)blockIdx.x * 2 + (first_piece ? 0 : 1);
        part = p.part_o + (slot * S::ROWS + sub * 128 + row) * D + col0;
        if (D == 128 || wg == 0) {
          p.part_ml[(slot * 2) * S::ROWS + sub * 128 + row] = m;
          p.part_ml[(slot * 2 + 1) * S::ROWS + sub * 128 + row] = l;
        }
      } else if (p.state_o != nullptr && live) {
        st_row = (long long)token * HQ + done.h * p.G + gq;
        float mo = -INFINITY, lo = 0.0f;
        if (!p.first_chunk) {
          mo = p.state_ml[2 * st_row];
          lo = p.state_ml[2 * st_row + 1];
        }
        const float mm = fmaxf(mo, m), ms = mm == -INFINITY ? 0.0f : mm;
        wo = fast_exp2(mo - ms);
        wn = fast_exp2(m - ms);
        l = l * wn + lo * wo;
        m = mm;
        finish = tile_hi == (max(1, min(r.L, r.L - r.ql + min(r.ql, (done.rt + 1) * piece_tok))) + kKeys - 1) / kKeys;
      }
      inv = p.vs / fmaxf(l, 1e-30f);
      if (l != l) inv = l;
      const long long out_row = ((long long)(r.q0 + token) * HQ + done.h * p.G + gq) * D + col0;
#pragma unroll
      for (int i = 0; i < 128; i += 32) {
        uint32_t o[32];
        tm_ld32(o, o_addr + i);
        tm_wait_ld();
        tm_ready(o);
        if (divided) {
#pragma unroll
          for (int k = 0; k < 32; k += 4) *reinterpret_cast<uint4*>(part + i + k) = make_uint4(o[k], o[k + 1], o[k + 2], o[k + 3]);
        } else if (live) {
          float f[32];
#pragma unroll
          for (int k = 0; k < 32; ++k) f[k] = __uint_as_float(o[k]);
          if (p.state_o != nullptr) {
            float* so = p.state_o + st_row * D + col0 + i;
#pragma unroll
            for (int k = 0; k < 32; ++k) {
              f[k] *= wn;
              if (!p.first_chunk) f[k] += so[k] * wo;
            }
            if (!finish) {
#pragma unroll
              for (int k = 0; k < 32; ++k) so[k] = f[k];
            }
          }
          if (finish) {
#pragma unroll
            for (int k = 0; k < 32; ++k) f[k] *= inv;
#pragma unroll
            for (int k = 0; k < 32; k += 8) store_out(p, out_row + i + k, f + k);
          }
        }
      }
      if (D == 256 && !divided && p.state_o != nullptr) {
        // both threads of a row have read its old maximum and sum before one of them writes the new ones
        float other;
        ok = exchange(0.0f, other);
        if (!ok) break;
      }
      if (!divided && live && p.state_o != nullptr && !finish && (D == 128 || wg == 0)) {
        p.state_ml[2 * st_row] = m;
        p.state_ml[2 * st_row + 1] = l;
      }
      tc_fence_before();               // the accumulator has been read: the next piece's first arrival lets it be overwritten
      first_piece = false;
      if (cut) break;
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 8) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
  if (tid == 0 && *abort && p.status != nullptr) atomicExch(p.status, HKV_ERR_DEVICE_WAIT);
}

// ------------------------------------------------------------------------------------------------------ merge_kernel
// parts of a divided row tile (and the state of earlier chunks) -> output or state; a thread has eight channels of a row
template <int D>
__global__ void __launch_bounds__(256) merge_kernel(const __grid_constant__ PrefillParams p) {
  using S = PfShape<D>;
  constexpr int LPR = D / 8;
  pdl_wait();
  pdl_launch_dependents();
  const PfSplit sp = p.split[blockIdx.x];
  const PfStart t = p.start[sp.c2];                       // the row tile: the last of its CTAs begins inside it
  const PfReq r = p.req[t.req];
  const int piece_tok = S::NT * p.tok;
  const int prow = blockIdx.y * (256 / LPR) + threadIdx.x / LPR, ch = (threadIdx.x % LPR) * 8;
  const int row = prow & 127, tk = row / p.G;
  const int token = t.rt * piece_tok + (prow >> 7) * p.tok + tk;
  if (tk >= p.tok || token >= r.ql) return;               // (a row's lanes agree)
  const int HQ = p.KVH * p.G;
  const long long st_row = (long long)token * HQ + t.h * p.G + (row - tk * p.G);
  const bool state = p.state_o != nullptr;
  float m = -INFINITY, l = 0.0f, acc[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) acc[k] = 0.0f;
  auto add = [&](float mi, float li, const float* o) {
    const float mm = fmaxf(m, mi), ms = mm == -INFINITY ? 0.0f : mm;
    const float a = fast_exp2(m - ms), b = fast_exp2(mi - ms);
    l = l * a + li * b;
    const float4 x = *reinterpret_cast<const float4*>(o), y = *reinterpret_cast<const float4*>(o + 4);
    const float v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] = acc[k] * a + v[k] * b;
    m = mm;
  };
  if (state && !p.first_chunk) add(p.state_ml[2 * st_row], p.state_ml[2 * st_row + 1], p.state_o + st_row * D + ch);
  for (int c = sp.c1; c <= sp.c2; ++c) {
    const long long slot = (long long)c * 2 + (c == sp.c1 ? sp.slot1 : 0);
    add(p.part_ml[slot * 2 * S::ROWS + prow], p.part_ml[(slot * 2 + 1) * S::ROWS + prow],
        p.part_o + (slot * S::ROWS + prow) * D + ch);
  }
  const int end = (max(1, min(r.L, r.L - r.ql + min(r.ql, (t.rt + 1) * piece_tok))) + kKeys - 1) / kKeys;
  if (state && end > p.kt_hi) {
    float* so = p.state_o + st_row * D + ch;
    __syncwarp(__activemask());                           // a row's lanes have read its state
#pragma unroll
    for (int k = 0; k < 8; ++k) so[k] = acc[k];
    if (ch == 0) {
      p.state_ml[2 * st_row] = m;
      p.state_ml[2 * st_row + 1] = l;
    }
    return;
  }
  float inv = p.vs / fmaxf(l, 1e-30f);
  if (l != l) inv = l;
#pragma unroll
  for (int k = 0; k < 8; ++k) acc[k] *= inv;
  store_out(p, ((long long)(r.q0 + token) * HQ + t.h * p.G + (row - tk * p.G)) * D + ch, acc);
}

// ---------------------------------------------------------------------------------------------------------- the plan
// Cuts the key tiles of the launch into at most n_cta shares of equal cost; returns the CTAs used. Greedy: a CTA takes
// row tiles in order until its share is full, and divides the one that does not fit when both parts are long enough.
static int plan(PrefillParams& p, int piece_tok, int n_cta, int* n_split) {
  long long total = 0;
  Walk w0{0, 0, -1, 0};
  w0.advance(p.req, p.n_req, p.KVH, piece_tok, p.kt_lo, p.kt_hi);      // the first row tile with keys in the chunk
  for (int r = 0; r < p.n_req; ++r) {
    long long head = 0;
    const int n_rt = pf_row_tiles(p.req[r], piece_tok);
    for (int rt = 0; rt < n_rt; ++rt) {
      const int n = pf_hi(p.req[r], rt, piece_tok, p.kt_hi) - p.kt_lo;
      if (n > 0) head += kPieceCost + n;
    }
    total += head * p.KVH;
  }
  long long cap = (total + n_cta - 1) / n_cta;
  if (cap < kPieceCost + 4) cap = kPieceCost + 4;
  for (;; cap += cap / 64 + 1) {
    Walk w = w0;
    int c = 0;
    *n_split = 0;
    int part_c1 = -1, part_slot1 = 0, pieces = 0;         // the divided row tile being cut; pieces of the current CTA
    long long room = cap;
    bool fits = true;
    auto begin = [&]() { p.start[c] = PfStart{w.kt, w.rt, (short)w.h, (short)w.req}; room = cap; pieces = 0; };
    if (w.req < p.n_req) begin();
    while (w.req < p.n_req) {
      const int hi = pf_hi(p.req[w.req], w.rt, piece_tok, p.kt_hi);
      const int n = hi - w.kt;
      if (kPieceCost + n <= room) {                       // the rest of the row tile
        if (part_c1 >= 0) {
          p.split[(*n_split)++] = PfSplit{(short)part_c1, (short)c, (short)part_slot1, 0};
          part_c1 = -1;
        }
        room -= kPieceCost + n;
        ++pieces;
        w.advance(p.req, p.n_req, p.KVH, piece_tok, p.kt_lo, p.kt_hi);
        if (w.req >= p.n_req) break;
        continue;
      }
      long long u = room - kPieceCost;
      if (n - u < kMinPiece) u = n - kMinPiece;
      if (u >= kMinPiece) {
        if (part_c1 < 0) { part_c1 = c; part_slot1 = pieces == 0 ? 0 : 1; }
        w.kt += (int)u;
      } else if (pieces == 0) {                           // (cannot happen: cap holds kPieceCost + 2 * kMinPiece)
        fits = false;
        break;
      }
      if (++c >= n_cta) { fits = false; break; }
      begin();
    }
    if (!fits) continue;
    p.start[c + 1] = PfStart{p.kt_lo, 0, 0, (short)p.n_req};
    return c + 1;
  }
}

static size_t a256(size_t x) { return align_up(x, 256); }

// requests of one launch: as many as fit the chunk; a longer context alone, chunk by chunk
struct PfGroup {
  int n, tiles;
  bool chunked;
};
static PfGroup next_group(const int32_t* rows, int n_rows, int chunk_tiles) {
  PfGroup g{0, 0, false};
  for (int i = 0; i < n_rows && g.n < kPfReqs; ++i) {
    const int t = (rows[4 * i + 3] + kKeys - 1) / kKeys;
    if (t > chunk_tiles) {
      if (g.n == 0) g = PfGroup{1, chunk_tiles, true};
      break;
    }
    if (g.tiles + t > chunk_tiles) break;
    g.tiles += t;
    ++g.n;
  }
  return g;
}

static int prefill_ctas() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1)
    n = 148;
  return n < kPfCtas ? n : kPfCtas;
}

struct PfScratch {
  size_t tiles, part_o, part_ml, state_o, state_ml, rot, total;
};
static PfScratch prefill_scratch(const int32_t* rows, int n_rows, int n_tok, int KVH, int G, int D, int chunk_tiles, int rot) {
  int max_tiles = 0;
  size_t state_rows = 0;
  for (int i = 0; i < n_rows;) {
    const PfGroup g = next_group(rows + 4 * i, n_rows - i, chunk_tiles);
    if (g.tiles > max_tiles) max_tiles = g.tiles;
    if (g.chunked) {
      const size_t n = (size_t)(rows[4 * i + 2] - rows[4 * i + 1]) * KVH * G;
      if (n > state_rows) state_rows = n;
    }
    i += g.n;
  }
  const size_t rws = D == 128 ? 256 : 128, n_cta = prefill_ctas();
  PfScratch s;
  s.tiles = 0;
  s.part_o = a256(s.tiles + (size_t)max_tiles * KVH * 2 * kKeys * D * 2);
  s.part_ml = a256(s.part_o + n_cta * 2 * rws * D * 4);
  s.state_o = a256(s.part_ml + n_cta * 2 * 2 * rws * 4);
  s.state_ml = a256(s.state_o + state_rows * D * 4);
  s.rot = a256(s.state_ml + state_rows * 8);
  s.total = a256(s.rot + (rot ? (size_t)n_tok * KVH * G * D * 2 : 0));
  return s;
}

static int chunk_tiles_of(int64_t chunk) {
  const int64_t t = chunk / kKeys;
  return t < 1 ? 1 : t > (1 << 23) ? (1 << 23) : (int)t;
}

static int check_rows(const int32_t* rows, int n_rows, int n_tok, int KVH, int G, int D) {
  if (!rows) return HKV_ERR_NULL;
  if (D != 128 && D != 256) return HKV_ERR_UNSUPPORTED;
  if (KVH < 1 || KVH > 1024 || G < 1 || G > 128) return HKV_ERR_UNSUPPORTED;
  for (int i = 0; i < n_rows; ++i) {
    const int32_t* r = rows + 4 * i;
    if (r[0] < 0 || r[1] < 0 || r[2] <= r[1] || r[2] > n_tok || r[3] < 1 || r[3] > 0x3fffff00) return HKV_ERR_RANGE;
  }
  return HKV_OK;
}

}  // namespace hkv

extern "C" size_t hkv_prefill_scratch_bytes(const int32_t* rows, int n_rows, int n_tokens, int KVH, int G, int D, int64_t chunk,
                                            int rotated) {
  using namespace hkv;
  if (n_rows < 1 || check_rows(rows, n_rows, n_tokens, KVH, G, D) != HKV_OK) return 0;
  return prefill_scratch(rows, n_rows, n_tokens, KVH, G, D, chunk_tiles_of(chunk), rotated).total;
}

extern "C" int hkv_prefill(const void* q, int q_ready, const void* kd, const void* ksf, const void* vd, const void* vsf,
                           const int64_t strides[6], int PS, const int32_t* block_tables, int n_tables, int MP,
                           const int32_t* rows, int n_rows, int n_tokens, int KVH, int G, int D, float qk_scale, float out_scale,
                           int k_f16, const float* signs, int k8, int64_t chunk, void* scratch, size_t scratch_bytes, void* out,
                           int out_f32, void* workspace, void* stream) {
  using namespace hkv;
  if (n_rows == 0) return HKV_OK;
  if (n_rows < 0) return HKV_ERR_RANGE;
  int rc = check_rows(rows, n_rows, n_tokens, KVH, G, D);
  if (rc != HKV_OK) return rc;
  if (k8 && D != 256) return HKV_ERR_UNSUPPORTED;
  if (!q || !kd || !ksf || !vd || !vsf || !strides || !block_tables || !scratch || !out) return HKV_ERR_NULL;
  if (signs && (k8 || q_ready)) return HKV_ERR_UNSUPPORTED;
  if (PS < 1) return HKV_ERR_UNSUPPORTED;
  if (((uintptr_t)kd | (uintptr_t)vd | (uintptr_t)strides[0] | (uintptr_t)strides[1] | (uintptr_t)strides[2]) & 7) return HKV_ERR_ALIGN;
  if (k8 && (((uintptr_t)kd | (uintptr_t)strides[0] | (uintptr_t)strides[1] | (uintptr_t)strides[2]) & 15)) return HKV_ERR_ALIGN;
  if (((uintptr_t)q | (uintptr_t)out) & 15 || ((uintptr_t)scratch & 255)) return HKV_ERR_ALIGN;
  for (int i = 0; i < n_rows; ++i)
    if (rows[4 * i] >= n_tables || (int64_t)rows[4 * i + 3] > (int64_t)MP * PS) return HKV_ERR_RANGE;
  const int ct = chunk_tiles_of(chunk);
  const PfScratch sc = prefill_scratch(rows, n_rows, n_tokens, KVH, G, D, ct, signs != nullptr);
  if (scratch_bytes < sc.total) return HKV_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  uint8_t* base = (uint8_t*)scratch;

  PrefillParams p = {};
  p.q = q;
  p.q_cvt = k_f16 && !q_ready;
  if (signs) {
    const long long n = (long long)n_tokens * KVH * G;
    const float scale = (float)(1.0 / sqrt((double)D));
    void (*k)(const __nv_bfloat16*, const float*, uint32_t*, long long, float, int) = D == 128 ? rotate_kernel<128> : rotate_kernel<256>;
    rc = record_cuda(launch_pdl(k, dim3((unsigned)((n + 7) / 8)), dim3(256), 0, st, (const __nv_bfloat16*)q, signs,
                                (uint32_t*)(base + sc.rot), n, scale, k_f16 ? 0 : 1));
    if (rc != HKV_OK) return rc;
    p.q = base + sc.rot;
    p.q_cvt = 0;
  }
  const float c = qk_scale * 1.4426950408889634f;
  p.q_flip = c < 0.0f ? 0x80008000u : 0u;
  p.c = fmaxf(fabsf(c), 1e-37f);                          // (zero: masked scores would become 0 * -inf)
  p.vs = out_scale;
  p.out = out;
  p.out_f32 = out_f32;
  p.k_bf16 = !k_f16;
  p.KVH = KVH;
  p.G = G;
  p.tok = 128 / G;
  p.tiles = base + sc.tiles;
  p.part_o = (float*)(base + sc.part_o);
  p.part_ml = (float*)(base + sc.part_ml);
  p.status = workspace ? &((Header*)workspace)->status : nullptr;
  const int piece_tok = (D == 128 ? 2 : 1) * p.tok, n_cta = prefill_ctas();

  TileParams t = {};
  t.kd = (const uint8_t*)kd; t.ksf = (const uint8_t*)ksf; t.vd = (const uint8_t*)vd; t.vsf = (const uint8_t*)vsf;
  t.dsp = strides[0]; t.dst = strides[1]; t.dsh = strides[2];
  t.ssp = strides[3]; t.sst = strides[4]; t.ssh = strides[5];
  t.bt = block_tables; t.tiles = base + sc.tiles;
  t.MP = MP; t.PS = PS; t.KVH = KVH;
  void (*tk)(const TileParams);
  if (k8) tk = k_f16 ? tile_kernel<256, 0, 1> : tile_kernel<256, 1, 1>;
  else if (D == 128) tk = k_f16 ? tile_kernel<128, 0, 0> : tile_kernel<128, 1, 0>;
  else tk = k_f16 ? tile_kernel<256, 0, 0> : tile_kernel<256, 1, 0>;
  void (*ak)(const PrefillParams) = D == 128 ? attend_kernel<128> : attend_kernel<256>;
  void (*mk)(const PrefillParams) = D == 128 ? merge_kernel<128> : merge_kernel<256>;
  rc = record_cuda(cudaFuncSetAttribute((const void*)ak, cudaFuncAttributeMaxDynamicSharedMemorySize, kPfSmem));
  if (rc != HKV_OK) return rc;

  for (int i = 0; i < n_rows;) {
    const PfGroup g = next_group(rows + 4 * i, n_rows - i, ct);
    int base_tile = 0, all_tiles = 0;
    p.n_req = t.n_req = g.n;
    for (int k = 0; k < g.n; ++k) {
      const int32_t* r = rows + 4 * (i + k);
      const int n_t = (r[3] + kKeys - 1) / kKeys;
      p.req[k] = PfReq{r[1], r[2] - r[1], r[3], base_tile};
      t.row[k] = r[0];
      t.L[k] = r[3];
      t.tile0[k] = base_tile;
      base_tile += n_t;
      all_tiles = n_t > all_tiles ? n_t : all_tiles;
    }
    p.state_o = g.chunked ? (float*)(base + sc.state_o) : nullptr;
    p.state_ml = g.chunked ? (float*)(base + sc.state_ml) : nullptr;
    for (int lo = 0; lo < all_tiles; lo += ct) {          // (one turn unless chunked)
      p.first_chunk = lo == 0;
      p.kt_lo = t.kt_lo = lo;
      p.kt_hi = g.chunked ? (lo + ct < all_tiles ? lo + ct : all_tiles) : all_tiles;
      t.n_tiles = g.chunked ? p.kt_hi - lo : base_tile;
      int n_split = 0;
      const int used = plan(p, piece_tok, n_cta, &n_split);
      rc = record_cuda(launch_pdl(tk, dim3((unsigned)t.n_tiles, (unsigned)KVH, 2), dim3(128), 0, st, t));
      if (rc == HKV_OK) rc = record_cuda(launch_pdl(ak, dim3((unsigned)used), dim3(kPfThreads), kPfSmem, st, p));
      if (rc == HKV_OK && n_split > 0)
        rc = record_cuda(launch_pdl(mk, dim3((unsigned)n_split, 16), dim3(256), 0, st, p));
      if (rc != HKV_OK) return rc;
      if (!g.chunked) break;
    }
    i += g.n;
  }
  return HKV_OK;
}
