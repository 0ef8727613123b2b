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
// Layer steps on a B200 (write launch included): a fresh prompt of 6144 tokens, 32 query heads over 8 kv heads, head_dim 128:
// 372 us against 16.5 ms with torch matmuls and eager softmax passes, whose fp32 score matrices went through memory. 2048
// tokens over 30000 cached, 16 heads over 2, head_dim 256: 0.91 ms (1.14 PFLOP/s; a plain bf16 GEMM sustains 1.37 at the
// board's 1000 W) against 15.0 ms.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "hkv_common.cuh"

namespace hkv {

int record_cuda(cudaError_t e);
int noalloc_workspace(void** ws);

constexpr int kPfReqs = 32;            // requests per launch (the tables below are kernel arguments, at most 4 KB)
constexpr int kPfCtas = 160;           // CTAs per launch
constexpr int kKeys = 128;             // keys per tile
constexpr int kPieceCost = 3;          // cost of starting and ending a piece, in key tiles (of about 1 us)
constexpr int kMinPiece = 2;           // no piece of a divided row tile is shorter, in key tiles
constexpr int kStageBytes = 32768;
constexpr int kStages = 5;
constexpr uint32_t kQBytes = 65536;    // query operands of 128 rows: two buffers at head_dim 128, one at 256

// A row tile has 128 rows; row r is query head r % G of token r / G, so that it covers 128 / G consecutive tokens and its
// causal edge is short.
template <int D>
struct PfShape {
  static constexpr int SETS = D == 128 ? 3 : 2;         // score tiles in flight, each with its softmax warpgroup
  static constexpr int OCOL = SETS * 128;               // tensor-memory column of the output accumulator
  static constexpr int NQ = D == 128 ? 2 : 1;           // query buffers
  static constexpr int SOFT = 4 * SETS;                 // softmax warps
  static constexpr int THREADS = 32 * (SOFT + 8);       // + the MMA warp, the copy warp, two idle ones; four end warps
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
  float* part_o;                       // [CTA][2][128][D]
  float* part_ml;                      // [CTA][2][2][128]: running maximum (log2 domain), sum
  float* state_o;                      // chunked contexts: [token][head][D], then the same tables per row
  float* state_ml;
  int* status;                         // of the workspace, or of the built-in one
  float c, vs;                         // score scale x log2(e) (> 0), output scale
  int out_f32, k_bf16;
  int KVH, G, tok;                     // tok: query tokens per row tile (128 / G)
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
__host__ __device__ inline int pf_hi(const PfReq& r, int rt, int tok, int kt_hi) {
  const int t_end = min(r.ql, (rt + 1) * tok);
  const int vis = max(1, min(r.L, r.L - r.ql + t_end));
  return min((vis + kKeys - 1) / kKeys, kt_hi);
}
__host__ __device__ inline int pf_row_tiles(const PfReq& r, int tok) { return (r.ql + tok - 1) / tok; }

struct Walk {
  int req, h, rt, kt;
  __host__ __device__ bool same_tile(const PfStart& e) const { return req == e.req && h == e.h && rt == e.rt; }
  // the next row tile that has keys in this chunk
  __host__ __device__ void advance(const PfReq* r, int n_req, int KVH, int tok, int kt_lo, int kt_hi) {
    kt = kt_lo;
    do {
      if (++rt >= pf_row_tiles(r[req], tok)) {
        rt = 0;
        if (++h >= KVH) { h = 0; ++req; }
      }
    } while (req < n_req && pf_hi(r[req], rt, tok, kt_hi) <= kt_lo);
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
  uint32_t k_flip;                     // 0x80008000 when the score scale is negative: the keys carry its sign
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
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] ^= p.k_flip;
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
// kv_fp4_ref.py:76-92, bit for bit). One warp per row: a lane holds D / 32 adjacent channels, the
// first stages stay inside the lane, the others exchange between lanes.
template <int D>
__global__ void __launch_bounds__(256) rotate_kernel(const __nv_bfloat16* q, const float* signs, uint32_t* out, long long rows,
                                                     float scale) {
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
    out[(row * D + lane * V + i) / 2] = *reinterpret_cast<const uint32_t*>(&b);
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

__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
struct PfShared {
  uint64_t full[kStages], empty[kStages];
  uint64_t q_full[2], q_free[2];       // query operands written / read for the last time in a piece
  uint64_t s_full[3], p_full[3];       // [set] scores, probabilities
  uint64_t o_done[3];                  // [set] value product of the set's tile has left the tensor pipe
  uint64_t told[12];                   // [set][quad] running maxima of 32 rows
  uint64_t ml_full, ml_free;           // a piece's maxima and sums written / read
  uint64_t o_free;                     // a piece's output has left the accumulator
  uint64_t drain;
  uint32_t tmem;
  int abort;
};
constexpr int kAux = (3 + 2) * 128 * 4;          // sums [set][128], running maxima [piece & 1][128]
constexpr int kPfSmem = (int)kQBytes + kStages * kStageBytes + kAux + (int)sizeof(PfShared);
static_assert(kPfSmem <= 232448, "shared memory");

// bounded wait: gives up when it runs out or when another role of the CTA has given up
template <long long LIMIT>
__device__ __forceinline__ bool pf_wait_slow(uint32_t bar, uint32_t parity, volatile int* abort) {
  const long long t0 = clock64();
  while (!mbar_try_wait_u32(bar, parity)) {
    if (*abort) return false;
    if (clock64() - t0 > LIMIT) {
      *abort = 1;
      return false;
    }
  }
  return true;
}
template <long long LIMIT>
__device__ __forceinline__ bool pf_wait(uint32_t bar, uint32_t parity, volatile int* abort) {
  if (mbar_try_wait_u32(bar, parity)) return true;
  return pf_wait_slow<LIMIT>(bar, parity, abort);
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
// Roles: a copy warp streams key and value tiles through a ring; one thread issues all products; SETS warpgroups take the
// score tiles in turn (a thread has a whole row of 128 scores); four end warps fetch the queries of the pieces to come and
// write the outputs of the pieces that are done. Tensor memory: SETS score tiles of 128 columns, the output (head_dim
// columns). Scores run SETS - 1 tiles ahead of the value products, across pieces too.
//
// Why so: a score tile is 1024 clocks of exponentials (ex2: 16 per clock and SM) and twice that again in latencies (loads
// from tensor memory, barriers, contention) before its value product can start, while the tensor pipe needs 1024 clocks
// (head_dim 128) or 2048 for both products. Two 128-row sub-tiles with one score buffer each left the tensor pipe idle 45 %
// of the time (3590 clocks for both against 2048; here 1450 a tile before the maximum was exact) and 9000 clocks between pieces (here about 3000; short
// prompts gain most, a step of four prompts with 48 decode requests went from 128 to 117 us); 64-key steps with two buffers
// each paid twice for the score product, which reads its 128 query rows from shared memory whatever the number of keys.
// The 16-bit probabilities go over the scores they came from. A thread tells the next tile's thread of its row the running
// maximum as soon as it knows it, and rescales the output, where the maximum has moved, after its probabilities are written:
// the wait for the value product before it then passes behind the exponentials. The maximum is the exact one: the largest
// probability is 1 and loses nothing to the rounding to f16. One that lags by up to 2^14 hardly ever rescales, but its
// largest probability is any number: the error against 64 bits (before the output's own rounding) was 1.9e-4 where this has
// 6.5e-5 (a prompt of 6144 tokens, head_dim 128) and 2.0e-4 where this has 8.3e-5 (2048 tokens over 30000, head_dim 256);
// the torch path before had 8.0e-5 and 1.06e-4. With the lag the steps took 361 and 862 us, now 372 and 915; with the rescaling
// before the exponentials 1.6 and 1.3 times as long.
// A walk over the CTA's key tiles, piece by piece. A step to the next row tile of a request costs a few instructions: every
// role takes it at every piece, two of them in a single thread.
struct Tiles {
  const PrefillParams& p;
  PfStart last;
  int req, h, rt, kt, hi;              // hi: end of the current piece
  PfReq r;
  int n_rt;                            // row tiles of the request
  uint32_t piece;
  bool first, end;                     // first tile of its piece; nothing left
  __device__ __forceinline__ explicit Tiles(const PrefillParams& p_) : p(p_), last(p_.start[blockIdx.x + 1]), piece(0) {
    const PfStart s = p_.start[blockIdx.x];
    req = s.req;
    h = s.h;
    rt = s.rt;
    kt = s.kt;
    enter_request();
    enter();
  }
  __device__ __forceinline__ void enter_request() {
    if (req < p.n_req) {
      r = p.req[req];
      n_rt = pf_row_tiles(r, p.tok);
    }
  }
  __device__ __forceinline__ bool cut() const { return rt == last.rt && h == last.h && req == last.req; }   // goes on in the next CTA
  __device__ __forceinline__ int tile_hi() const { return pf_hi(r, rt, p.tok, p.kt_hi); }
  __device__ __forceinline__ void enter() {
    first = true;
    const bool c = cut();
    end = c && kt >= last.kt;
    hi = c ? last.kt : tile_hi();
  }
  __device__ __forceinline__ void next_piece() {
    if (cut()) {
      end = true;
      return;
    }
    kt = p.kt_lo;
    do {
      if (++rt >= n_rt) {
        rt = 0;
        if (++h >= p.KVH) {
          h = 0;
          ++req;
          enter_request();
        }
      }
    } while (req < p.n_req && tile_hi() <= p.kt_lo);      // (no keys in this chunk)
    ++piece;
    enter();
  }
  __device__ __forceinline__ void next() {
    first = false;
    if (++kt == hi) next_piece();
  }
};

// LOSE (the self-test of the give-up path): the copy warp stops after three stages, and waits run out after a millisecond.
template <int D, bool LOSE>
__global__ void __launch_bounds__(PfShape<D>::THREADS, 1) attend_kernel(const __grid_constant__ PrefillParams p) {
  using S = PfShape<D>;
  constexpr int SETS = S::SETS, SOFT = S::SOFT, NQ = S::NQ;
  constexpr uint32_t IMAGE = kKeys * D * 2;
  constexpr int PER = IMAGE / kStageBytes;                // ring stages per operand tile: 1 or 2
  constexpr long long LIMIT = LOSE ? 1ll << 21 : kWaitCycles;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* ring = smem + kQBytes;
  uint8_t* aux = smem + kQBytes + kStages * kStageBytes;
  volatile float* xl = reinterpret_cast<float*>(aux);               // [set][128]: sums of a piece
  volatile float* xm = reinterpret_cast<float*>(aux) + 3 * 128;     // [piece & 1][128]: running maxima (log2 domain)
  PfShared& sh = *reinterpret_cast<PfShared*>(aux + kAux);
  volatile int* abort = &sh.abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    sh.abort = (smem_u32(smem) & 1023) ? 1 : 0;        // the swizzled operands need 1024-byte alignment
    for (int i = 0; i < kStages; ++i) { mbar_init(&sh.full[i], 1); mbar_init(&sh.empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&sh.q_full[i], 128); mbar_init(&sh.q_free[i], 1); }
    for (int i = 0; i < 3; ++i) { mbar_init(&sh.s_full[i], 1); mbar_init(&sh.p_full[i], 128); mbar_init(&sh.o_done[i], 1); }
    for (int i = 0; i < 12; ++i) mbar_init(&sh.told[i], 32);
    mbar_init(&sh.ml_full, SETS * 128);
    mbar_init(&sh.ml_free, 128);
    mbar_init(&sh.o_free, 128);
    mbar_init(&sh.drain, 1);
    fence_barrier_init();
  }
  if (warp == SOFT) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&sh.tmem)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh.tmem;
  pdl_wait();
  pdl_launch_dependents();

  const uint32_t full0 = smem_u32(&sh.full[0]), empty0 = smem_u32(&sh.empty[0]), q_full0 = smem_u32(&sh.q_full[0]),
                 q_free0 = smem_u32(&sh.q_free[0]), s_full0 = smem_u32(&sh.s_full[0]), p_full0 = smem_u32(&sh.p_full[0]),
                 o_done0 = smem_u32(&sh.o_done[0]), told0 = smem_u32(&sh.told[0]), ml_full = smem_u32(&sh.ml_full),
                 ml_free = smem_u32(&sh.ml_free), o_free = smem_u32(&sh.o_free);
  auto all_wait = [&](uint32_t bar, uint32_t phase) { return (bool)__all_sync(0xffffffffu, pf_wait<LIMIT>(bar, phase & 1, abort)); };

  if (warp == SOFT + 1) {
    // ------------------------------------------------------------------------------------------------ copy warp
    if (elect_one()) {
      Tiles k(p), v(p);
      uint32_t fill = 0, st = 0, turn = 0;
      bool ok = *abort == 0;
      auto fetch = [&](Tiles& x, int side) {
        const PfReq& r = x.r;
        const int n_t = min(p.kt_hi, (r.L + kKeys - 1) / kKeys) - p.kt_lo;
        const uint8_t* from = p.tiles + ((size_t)r.tile0 * p.KVH + (size_t)x.h * n_t + (x.kt - p.kt_lo)) * 2 * IMAGE + side * IMAGE;
        for (int i = 0; ok && i < PER; ++i) {
          if (LOSE && fill == 3) ok = false;
          else if (turn > 0) ok = pf_wait<LIMIT>(empty0 + 8 * st, (turn - 1) & 1, abort);
          if (!ok) return;
          mbar_expect_tx_u32(full0 + 8 * st, kStageBytes);
          bulk_g2s_u32(smem_u32(ring) + st * kStageBytes, from + i * kStageBytes, kStageBytes, full0 + 8 * st);
          ++fill;
          if (++st == kStages) { st = 0; ++turn; }
        }
        x.next();
      };
      for (int i = 0; ok && i < SETS - 1 && !k.end; ++i) fetch(k, 0);
      while (ok && !v.end) {
        if (!k.end) fetch(k, 0);
        if (ok) fetch(v, 1);
      }
      // nothing of this CTA's may still be on its way when it ends (another role may give up at any time)
      for (uint32_t f = fill > kStages ? fill - kStages : 0; f < fill; ++f)
        mbar_wait_bounded_u32(full0 + 8 * (f % kStages), (f / kStages) & 1);
    }
  } else if (warp == SOFT) {
    // ------------------------------------------------------------------------------------------------- MMA warp
    if (elect_one()) {
      const uint32_t base = (1u << 4) | ((128u / 16) << 24);
      const uint32_t id_qk = base | ((uint32_t)(kKeys / 8) << 17) | (p.k_bf16 ? (1u << 7) | (1u << 10) : 0u);
      const uint32_t id_pv = base | ((uint32_t)(D / 8) << 17);
      const uint32_t q_smem = smem_u32(smem), ring_a = smem_u32(ring);
      Tiles k(p), v(p);
      uint32_t use = 0;                                   // ring stages handed out, in the copy warp's order
      uint32_t sk = 0, sv = 0, tv = 0;                    // score tile (of SETS) of the next score and value product; turn of the latter
      bool ok = *abort == 0;
      auto stage_wait = [&](uint32_t n) { return pf_wait<LIMIT>(full0 + 8 * (n % kStages), (n / kStages) & 1, abort); };
      auto stage_addr = [&](uint32_t n) { return ring_a + (n % kStages) * kStageBytes; };
      auto stages_done = [&](uint32_t n) {
        for (int i = 0; i < PER; ++i) umma_commit(empty0 + 8 * ((n + i) % kStages));
      };
      auto scores = [&](uint32_t n) {                     // of the next key tile, which lies in stage n (and n + 1)
        const uint32_t qb = k.piece % NQ;
        if (k.first) ok = pf_wait<LIMIT>(q_full0 + 8 * qb, (k.piece / NQ) & 1, abort);
        ok = ok && stage_wait(n) && (PER == 1 || stage_wait(n + 1));
        if (!ok) return;
        tc_fence_after();
#pragma unroll
        for (int kb = 0; kb < D / 64; ++kb) {
          const uint64_t a = umma_desc(q_smem + qb * 32768 + kb * 16384);
          const uint64_t b = umma_desc(stage_addr(n + kb / 2) + (kb & 1) * 16384);
#pragma unroll
          for (int i = 0; i < 4; ++i) umma_ss(tmem + sk * 128, a + 2 * i, b + 2 * i, id_qk, kb + i > 0);
        }
        umma_commit(s_full0 + 8 * sk);
        stages_done(n);
        if (k.kt + 1 == k.hi) umma_commit(q_free0 + 8 * qb);
        if (++sk == SETS) sk = 0;
        k.next();
      };
      auto values = [&](uint32_t n) {
        // (the accumulator holds the piece before until the end warps have read it)
        ok = stage_wait(n) && (PER == 1 || stage_wait(n + 1)) &&
             (!v.first || v.piece == 0 || pf_wait<LIMIT>(o_free, (v.piece - 1) & 1, abort)) && pf_wait<LIMIT>(p_full0 + 8 * sv, tv & 1, abort);
        if (!ok) return;
        tc_fence_after();
#pragma unroll
        for (int kb = 0; kb < 2; ++kb) {
          const uint64_t b = umma_desc(PER == 1 ? stage_addr(n) + kb * 16384 : stage_addr(n + kb));
#pragma unroll
          for (int i = 0; i < 4; ++i)
            umma_ts(tmem + S::OCOL, tmem + sv * 128 + 64 + kb * 32 + i * 8, b + 2 * i, id_pv, !v.first || kb + i > 0);
        }
        umma_commit(o_done0 + 8 * sv);
        stages_done(n);
        if (++sv == SETS) { sv = 0; ++tv; }
        v.next();
      };
      for (int i = 0; ok && i < SETS - 1 && !k.end; ++i) { scores(use); use += PER; }
      while (ok && !v.end) {
        if (k.end) {
          values(use);
          use += PER;
          continue;
        }
        // (a single query buffer is only refilled once the scores of the piece are done: the value product does not wait)
        const bool later = NQ == 1 && k.first;
        if (later) values(use + PER);
        if (ok) scores(use);
        if (ok && !later) values(use + PER);
        use += 2 * PER;
      }
      // no product of this CTA's may still be running when its tensor memory is given back
      umma_commit(smem_u32(&sh.drain));
      mbar_wait_bounded_u32(smem_u32(&sh.drain), 0);
    }
  } else if (warp >= SOFT + 4) {
    // ------------------------------------------------------------------------------------------------ end warps
    const int row = tid - (SOFT + 4) * 32, quad = warp & 3;              // row of the tile, = tensor-memory lane
    const uint32_t inv_g = 65536u / p.G + 1;              // floor(row / G) = row * inv_g >> 16 for rows below 128
    const int HQ = p.KVH * p.G;
    Tiles x(p), y(p);                                  // the piece to write out; the piece to fetch queries of
    uint32_t g = 0;
    bool ok = *abort == 0;
    // queries of piece y: 16 bytes per lane and copy, whole rows per half warp or warp; rows that do not exist are zero
    auto load_q = [&]() {
      constexpr int LPR = D / 8, RSTEP = 128 / LPR;
      const PfReq r = y.r;
      const int ch = row % LPR, tok0 = y.rt * p.tok;
      const uint32_t qs = smem_u32(smem) + (y.piece % NQ) * 32768 + (ch >> 3) * 16384;
      const uint16_t* q = (const uint16_t*)p.q + ((long long)(r.q0 + tok0) * HQ + y.h * p.G) * D + ch * 8;
      if (y.piece >= NQ && !pf_wait<LIMIT>(q_free0 + 8 * (y.piece % NQ), (y.piece / NQ - 1) & 1, abort)) return false;
#pragma unroll 4
      for (int rr = row / LPR; rr < 128; rr += RSTEP) {
        const int tk = (int)((uint32_t)rr * inv_g >> 16);
        const uint32_t dst = qs + rr * 128 + (((ch & 7) ^ (rr & 7)) << 4);
        if (tk < p.tok && tok0 + tk < r.ql) cp_async<16>(dst, q + ((long long)tk * HQ + (rr - tk * p.G)) * D);
        else asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(dst), "r"(0u) : "memory");
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      fence_proxy_async();
      mbar_arrive_u32(q_full0 + 8 * (y.piece % NQ));
      return true;
    };
    for (int i = 0; ok && i < NQ && !y.end; ++i) {
      ok = __all_sync(0xffffffffu, load_q());
      y.next_piece();
    }
    while (ok && !x.end) {
      if (!y.end) {
        ok = __all_sync(0xffffffffu, load_q());
        if (!ok) break;
        y.next_piece();
      }
      const PfReq r = x.r;
      const int tile_hi = x.tile_hi();
      g += x.hi - x.kt;
      const bool divided = x.cut() || x.kt > p.kt_lo;
      const int tk = (int)((uint32_t)row * inv_g >> 16), token = x.rt * p.tok + tk;
      const bool live = tk < p.tok && token < r.ql;
      const int head = x.h * p.G + (row - tk * p.G);
      ok = all_wait(ml_full, x.piece);
      if (!ok) break;
      float l = xl[row], m = xm[(x.piece & 1) * 128 + row];
      for (int i = 1; i < SETS; ++i) l += xl[i * 128 + row];
      mbar_arrive_u32(ml_free);
      float wo = 0.0f, wn = 1.0f;
      const long long st_row = (long long)token * HQ + head;
      bool finish = true;
      float* part = nullptr;
      if (divided) {
        const long long slot = (long long)blockIdx.x * 2 + (x.piece == 0 ? 0 : 1);
        part = p.part_o + (slot * 128 + row) * D;
        p.part_ml[slot * 256 + row] = m;
        p.part_ml[slot * 256 + 128 + row] = l;
      } else if (p.state_o != nullptr && live) {
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
        finish = tile_hi == (max(1, min(r.L, r.L - r.ql + min(r.ql, (x.rt + 1) * p.tok))) + kKeys - 1) / kKeys;
        if (!finish) {
          p.state_ml[2 * st_row] = m;
          p.state_ml[2 * st_row + 1] = l;
        }
      }
      float inv = p.vs / fmaxf(l, 1e-30f);
      if (l != l) inv = l;
      const long long out_row = ((long long)(r.q0 + token) * HQ + head) * D;
      ok = all_wait(o_done0 + 8 * ((g - 1) % SETS), (g - 1) / SETS);
      if (!ok) break;
      tc_fence_after();
      const uint32_t o_addr = tmem + ((uint32_t)(quad * 32) << 16) + S::OCOL;
      if (!divided && p.state_o == nullptr && !p.out_f32) {
        // the usual output: 16 bits, 64 columns at a time; the accumulator is free before the last ones are stored
#pragma unroll 1
        for (int i = 0; i < D; i += 64) {
          uint32_t u[32];
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            uint32_t o[32];
            tm_ld32(o, o_addr + i + 32 * k);
            tm_wait_ld();
            tm_ready(o);
#pragma unroll
            for (int n = 0; n < 16; ++n) {
              const __nv_bfloat162 b = __floats2bfloat162_rn(__uint_as_float(o[2 * n]) * inv, __uint_as_float(o[2 * n + 1]) * inv);
              u[16 * k + n] = *reinterpret_cast<const uint32_t*>(&b);
            }
          }
          if (i + 64 == D) {
            tc_fence_before();
            mbar_arrive_u32(o_free);
          }
          if (live) {
            uint4* dst = reinterpret_cast<uint4*>((__nv_bfloat16*)p.out + out_row + i);
#pragma unroll
            for (int n = 0; n < 8; ++n) dst[n] = make_uint4(u[4 * n], u[4 * n + 1], u[4 * n + 2], u[4 * n + 3]);
          }
        }
        x.next_piece();
        continue;
      }
#pragma unroll 1
      for (int i = 0; i < D; i += 32) {
        uint32_t o[32];
        tm_ld32(o, o_addr + i);
        tm_wait_ld();
        tm_ready(o);
        if (i + 32 == D) {
          tc_fence_before();
          mbar_arrive_u32(o_free);
        }
        if (divided) {
#pragma unroll
          for (int k = 0; k < 32; k += 4) *reinterpret_cast<uint4*>(part + i + k) = make_uint4(o[k], o[k + 1], o[k + 2], o[k + 3]);
        } else if (live) {
          float f[32];
#pragma unroll
          for (int k = 0; k < 32; ++k) f[k] = __uint_as_float(o[k]);
          if (p.state_o != nullptr) {
            float* so = p.state_o + st_row * D + i;
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
      x.next_piece();
    }
  } else if (warp < SOFT) {
    // -------------------------------------------------------------------------------------------- softmax warps
    const int set = warp >> 2, quad = warp & 3;
    const int row = quad * 32 + lane;                     // of the tile, = tensor-memory lane
    const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16), s_addr = lane_base + set * 128;
    const uint32_t s_bar = s_full0 + 8 * set, my_word = told0 + 8 * (set * 4 + quad);
    const int before = set == 0 ? SETS - 1 : set - 1;     // the set of the tile before
    const uint32_t word_before = told0 + 8 * (before * 4 + quad);
    Tiles x(p);
    uint32_t g = set, turn = 0;                           // the set's next tile in the CTA's stream; its tiles done
    uint32_t g0 = 0;                                      // first tile of the piece
    const int tk = row / p.G;
    bool ok = *abort == 0;
    while (ok && !x.end) {
      const PfReq& r = x.r;
      const int token = x.rt * p.tok + tk;
      const int lim = tk < p.tok && token < r.ql ? max(0, min(r.L, r.L - r.ql + token + 1)) : 0;      // keys this row sees
      // keys below this one are seen by every live row of the tile (rows that do not exist may take any value)
      const int whole = max(0, min(r.L, r.L - r.ql + x.rt * p.tok + 1));
      const uint32_t g_end = g0 + (x.hi - x.kt);
      volatile float* top_now = xm + (x.piece & 1) * 128 + row;
      float m = -INFINITY;                                // the running maximum as this thread knows it
      unsigned long long l2 = 0;                          // two partial sums
      bool any_tile = false;
      for (; g < g_end; g += SETS, ++turn) {
        const int key = (x.kt + (int)(g - g0)) * kKeys;
        const bool head = g == g0;
        ok = all_wait(s_bar, turn);
        if (!ok) break;
        tc_fence_after();
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        uint32_t s0[32];
        auto load = [&](int c) {                          // 32 scores
          tm_ld32(s0, s_addr + 32 * c);
          tm_wait_ld();
          tm_ready(s0);
          if (key + 32 * c + 32 > whole) {
            const int rel = lim - key - 32 * c;
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (i >= rel) s0[i] = 0xff800000u;
          }
        };
        // (rolled loops, and no register to spare: unrolled, the code of all roles leaves the instruction cache, and a register
        // spilled in here costs an L2 access, since the L1 cache is all shared memory; each made the launch 8 to 15 % longer. At
        // head_dim 256 the compiler spills 24 bytes of the 128 registers that 512 threads leave, in all)
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          load(c);
#pragma unroll
          for (int i = 0; i < 32; i += 2)
            mx[i / 2 & 3] = fmaxf(mx[i / 2 & 3], fmaxf(__uint_as_float(s0[i]), __uint_as_float(s0[i + 1])));
        }
        const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.c;
        // (also at the head of a piece: no barrier may get two phases ahead of its reader)
        if (g > 0) ok = all_wait(word_before, (g - 1) / SETS);
        if (!ok) break;
        const float m_old = m, m_in = head ? -INFINITY : *top_now;
        const bool move = top > m_in;
        m = move ? (top == INFINITY ? 0.0f : top) : m_in;
        if (move || head) *top_now = m;
        mbar_arrive_u32(my_word);
        if (__any_sync(0xffffffffu, m != m_old)) {
          const float al = m == m_old ? 1.0f : fast_exp2(m_old - m);
          l2 = mul2(l2, pack2(al, al));
        }
        const float al_o = move && !head ? fast_exp2(m_in - m) : 1.0f;
        const float mu = m == -INFINITY ? 0.0f : -m;
        const unsigned long long c2 = pack2(p.c, p.c), m2 = pack2(mu, mu);
        // from the last 32 scores (still in registers) to the first, so that the probabilities of a part, 16 columns, go over
        // scores that have been read: columns 64 .. 127 in the end
#pragma unroll 1
        for (int c = 3;; --c) {
          uint32_t ph16[16];
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            float a, b;
            unpack2(fma2(pack2(__uint_as_float(s0[2 * k]), __uint_as_float(s0[2 * k + 1])), c2, m2), a, b);
            a = fast_exp2(a);
            b = fast_exp2(b);
            l2 = add2(l2, pack2(a, b));
            ph16[k] = pack_f16x2(a, b);
          }
          tm_st16(s_addr + 64 + 16 * c, ph16);
          if (c == 0) break;
          load(c - 1);
        }
        if (__any_sync(0xffffffffu, al_o != 1.0f)) {
          // the output of the tiles before this one, all of whose value products must have been added first; 64 columns at a
          // time and in packed pairs (32 at a time and one by one, a step at head_dim 256 took 2 % longer)
          ok = all_wait(o_done0 + 8 * before, (g - 1) / SETS);
          if (!ok) {
            tc_wait_st();
            break;
          }
          tc_fence_after();
          const unsigned long long al2 = pack2(al_o, al_o);
#pragma unroll 1
          for (int i = 0; i < D; i += 64) {
            uint32_t o[2][32];
            tm_ld32(o[0], lane_base + S::OCOL + i);
            tm_ld32(o[1], lane_base + S::OCOL + i + 32);
            tm_wait_ld();
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              tm_ready(o[u]);
#pragma unroll
              for (int k = 0; k < 32; k += 2) {
                float a, b;
                unpack2(mul2(pack2(__uint_as_float(o[u][k]), __uint_as_float(o[u][k + 1])), al2), a, b);
                o[u][k] = __float_as_uint(a);
                o[u][k + 1] = __float_as_uint(b);
              }
              tm_st16(lane_base + S::OCOL + i + 32 * u, o[u]);
              tm_st16(lane_base + S::OCOL + i + 32 * u + 16, o[u] + 16);
            }
          }
        }
        tc_wait_st();
        tc_fence_before();
        mbar_arrive_u32(p_full0 + 8 * set);
        any_tile = true;
      }
      if (!ok) break;
      // the set's sum under the piece's last maximum, for the end warps, which have read those of the piece before
      float l = 0.0f, l_hi;
      if (any_tile) {
        unpack2(l2, l, l_hi);
        l += l_hi;
        if (g_end > g - SETS + 1) {                       // another set has the last tile
          const uint32_t gl = g_end - 1;
          ok = all_wait(told0 + 8 * (gl % SETS * 4 + quad), gl / SETS);
          if (!ok) break;
          const float m_end = *top_now;
          if (m_end != m) l *= fast_exp2(m - m_end);
        }
      }
      if (x.piece > 0) ok = all_wait(ml_free, x.piece - 1);
      if (!ok) break;
      xl[set * 128 + row] = l;
      mbar_arrive_u32(ml_full);
      g0 = g_end;
      x.next_piece();
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == SOFT) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
  if (tid == 0 && *abort) atomicExch(p.status, HKV_ERR_DEVICE_WAIT);
}

// ------------------------------------------------------------------------------------------------------ merge_kernel
// parts of a divided row tile (and the state of earlier chunks) -> output or state; a thread has eight channels of a row
template <int D>
__global__ void __launch_bounds__(256) merge_kernel(const __grid_constant__ PrefillParams p) {
  constexpr int LPR = D / 8;
  pdl_wait();
  pdl_launch_dependents();
  const PfSplit sp = p.split[blockIdx.x];
  const PfStart t = p.start[sp.c2];                       // the row tile: the last of its CTAs begins inside it
  const PfReq r = p.req[t.req];
  const int row = blockIdx.y * (256 / LPR) + threadIdx.x / LPR, ch = (threadIdx.x % LPR) * 8;
  const int tk = row / p.G, token = t.rt * p.tok + tk;
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
    add(p.part_ml[slot * 256 + row], p.part_ml[slot * 256 + 128 + row], p.part_o + (slot * 128 + row) * D + ch);
  }
  const int end = (max(1, min(r.L, r.L - r.ql + min(r.ql, (t.rt + 1) * p.tok))) + kKeys - 1) / kKeys;
  if (state && end > p.kt_hi) {
    float* so = p.state_o + st_row * D + ch;
    // a row's lanes (they agree on the return above) have read its state
    __syncwarp(LPR == 32 ? 0xffffffffu : 0xffffu << (threadIdx.x & 16));
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
static int plan(PrefillParams& p, int n_cta, int* n_split) {
  long long total = 0;
  Walk w0{0, 0, -1, 0};
  w0.advance(p.req, p.n_req, p.KVH, p.tok, p.kt_lo, p.kt_hi);      // the first row tile with keys in the chunk
  for (int r = 0; r < p.n_req; ++r) {
    long long head = 0;
    const int n_rt = pf_row_tiles(p.req[r], p.tok);
    for (int rt = 0; rt < n_rt; ++rt) {
      const int n = pf_hi(p.req[r], rt, p.tok, p.kt_hi) - p.kt_lo;
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
      const int hi = pf_hi(p.req[w.req], w.rt, p.tok, p.kt_hi);
      const int n = hi - w.kt;
      if (kPieceCost + n <= room) {                       // the rest of the row tile
        if (part_c1 >= 0) {
          p.split[(*n_split)++] = PfSplit{(short)part_c1, (short)c, (short)part_slot1, 0};
          part_c1 = -1;
        }
        room -= kPieceCost + n;
        ++pieces;
        w.advance(p.req, p.n_req, p.KVH, p.tok, p.kt_lo, p.kt_hi);
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
  const size_t n_cta = prefill_ctas();
  PfScratch s;
  s.tiles = 0;
  s.part_o = a256(s.tiles + (size_t)max_tiles * KVH * 2 * kKeys * D * 2);
  s.part_ml = a256(s.part_o + n_cta * 2 * 128 * D * 4);
  s.state_o = a256(s.part_ml + n_cta * 2 * 2 * 128 * 4);
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

static int prefill_impl(const void* q, int q_f16, const void* kd, const void* ksf, const void* vd, const void* vsf,
                           const int64_t strides[6], int PS, const int32_t* block_tables, int n_tables, int MP,
                           const int32_t* rows, int n_rows, int n_tokens, int KVH, int G, int D, float qk_scale, float out_scale,
                           const float* signs, int k8, int64_t chunk, void* scratch, size_t scratch_bytes, void* out,
                           int out_f32, void* workspace, void* stream, bool lose) {
  using namespace hkv;
  if (n_rows == 0) return HKV_OK;
  if (n_rows < 0) return HKV_ERR_RANGE;
  int rc = check_rows(rows, n_rows, n_tokens, KVH, G, D);
  if (rc != HKV_OK) return rc;
  if (k8 && D != 256) return HKV_ERR_UNSUPPORTED;
  if (!q || !kd || !ksf || !vd || !vsf || !strides || !block_tables || !scratch || !out) return HKV_ERR_NULL;
  if (signs && (k8 || q_f16)) return HKV_ERR_UNSUPPORTED;
  if (PS < 1) return HKV_ERR_UNSUPPORTED;
  if (((uintptr_t)kd | (uintptr_t)vd | (uintptr_t)strides[0] | (uintptr_t)strides[1] | (uintptr_t)strides[2]) & 7) return HKV_ERR_ALIGN;
  if (k8 && (((uintptr_t)kd | (uintptr_t)strides[0] | (uintptr_t)strides[1] | (uintptr_t)strides[2]) & 15)) return HKV_ERR_ALIGN;
  if (((uintptr_t)q | (uintptr_t)out) & 15 || (((uintptr_t)scratch | (uintptr_t)workspace) & 255)) return HKV_ERR_ALIGN;
  for (int i = 0; i < n_rows; ++i)
    if (rows[4 * i] >= n_tables || (int64_t)rows[4 * i + 3] > (int64_t)MP * PS) return HKV_ERR_RANGE;
  const int ct = chunk_tiles_of(chunk);
  const PfScratch sc = prefill_scratch(rows, n_rows, n_tokens, KVH, G, D, ct, signs != nullptr);
  if (scratch_bytes < sc.total) return HKV_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  uint8_t* base = (uint8_t*)scratch;

  PrefillParams p = {};
  p.q = q;
  if (signs) {
    const long long n = (long long)n_tokens * KVH * G;
    const float scale = (float)(1.0 / sqrt((double)D));
    void (*k)(const __nv_bfloat16*, const float*, uint32_t*, long long, float) = D == 128 ? rotate_kernel<128> : rotate_kernel<256>;
    rc = record_cuda(launch_pdl(k, dim3((unsigned)((n + 7) / 8)), dim3(256), 0, st, (const __nv_bfloat16*)q, signs,
                                (uint32_t*)(base + sc.rot), n, scale));
    if (rc != HKV_OK) return rc;
    p.q = base + sc.rot;
  }
  const float c = qk_scale * 1.4426950408889634f;
  p.c = fmaxf(fabsf(c), 1e-37f);                          // (zero: masked scores would become 0 * -inf)
  p.vs = c != c ? c : out_scale;                          // (fmaxf drops a NaN: the output takes it instead)
  p.out = out;
  p.out_f32 = out_f32;
  p.k_bf16 = !q_f16;                                      // (the cached values are exact in both types)
  p.KVH = KVH;
  p.G = G;
  p.tok = 128 / G;
  p.tiles = base + sc.tiles;
  p.part_o = (float*)(base + sc.part_o);
  p.part_ml = (float*)(base + sc.part_ml);
  if (!workspace) {
    rc = noalloc_workspace(&workspace);
    if (rc != HKV_OK) return rc;
  }
  p.status = &((Header*)workspace)->status;
  const int n_cta = prefill_ctas();

  TileParams t = {};
  t.kd = (const uint8_t*)kd; t.ksf = (const uint8_t*)ksf; t.vd = (const uint8_t*)vd; t.vsf = (const uint8_t*)vsf;
  t.dsp = strides[0]; t.dst = strides[1]; t.dsh = strides[2];
  t.ssp = strides[3]; t.sst = strides[4]; t.ssh = strides[5];
  t.bt = block_tables; t.tiles = base + sc.tiles;
  t.MP = MP; t.PS = PS; t.KVH = KVH;
  t.k_flip = c < 0.0f ? 0x80008000u : 0u;
  void (*tk)(const TileParams);
  if (k8) tk = q_f16 ? tile_kernel<256, 0, 1> : tile_kernel<256, 1, 1>;
  else if (D == 128) tk = q_f16 ? tile_kernel<128, 0, 0> : tile_kernel<128, 1, 0>;
  else tk = q_f16 ? tile_kernel<256, 0, 0> : tile_kernel<256, 1, 0>;
  void (*ak)(const PrefillParams) = lose ? (D == 128 ? attend_kernel<128, true> : attend_kernel<256, true>)
                                         : D == 128 ? attend_kernel<128, false> : attend_kernel<256, false>;
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
      const int used = plan(p, n_cta, &n_split);
      rc = record_cuda(launch_pdl(tk, dim3((unsigned)t.n_tiles, (unsigned)KVH, 2), dim3(128), 0, st, t));
      if (rc == HKV_OK) rc = record_cuda(launch_pdl(ak, dim3((unsigned)used), dim3(D == 128 ? PfShape<128>::THREADS : PfShape<256>::THREADS), kPfSmem, st, p));
      if (rc == HKV_OK && n_split > 0)
        rc = record_cuda(launch_pdl(mk, dim3((unsigned)n_split, D == 128 ? 8 : 16), dim3(256), 0, st, p));
      if (rc != HKV_OK) return rc;
      if (!g.chunked) break;
    }
    i += g.n;
  }
  return HKV_OK;
}

extern "C" int hkv_prefill(const void* q, int q_f16, const void* kd, const void* ksf, const void* vd, const void* vsf,
                           const int64_t strides[6], int PS, const int32_t* block_tables, int n_tables, int MP,
                           const int32_t* rows, int n_rows, int n_tokens, int KVH, int G, int D, float qk_scale, float out_scale,
                           const float* signs, int k8, int64_t chunk, void* scratch, size_t scratch_bytes, void* out,
                           int out_f32, void* workspace, void* stream) {
  return prefill_impl(q, q_f16, kd, ksf, vd, vsf, strides, PS, block_tables, n_tables, MP, rows, n_rows, n_tokens, KVH, G, D, qk_scale,
                      out_scale, signs, k8, chunk, scratch, scratch_bytes, out, out_f32, workspace, stream, false);
}

extern "C" int hkv_selftest_prefill_timeout(const void* q, int q_f16, const void* kd, const void* ksf, const void* vd,
                                            const void* vsf, const int64_t strides[6], int PS, const int32_t* block_tables,
                                            int n_tables, int MP, const int32_t* rows, int n_rows, int n_tokens, int KVH, int G,
                                            int D, float qk_scale, float out_scale, const float* signs, int k8, int64_t chunk,
                                            void* scratch, size_t scratch_bytes, void* out, int out_f32, void* workspace,
                                            void* stream) {
  return prefill_impl(q, q_f16, kd, ksf, vd, vsf, strides, PS, block_tables, n_tables, MP, rows, n_rows, n_tokens, KVH, G, D, qk_scale,
                      out_scale, signs, k8, chunk, scratch, scratch_bytes, out, out_f32, workspace, stream, true);
}
