// Chunked gated-delta-rule backward for sm_100a, part 2: everything that is local to one chunk.
// Reference: chunk_gated_delta_rule_bwd (flash_qla/ops/gated_delta_rule/chunk/__init__.py:89-182); the
// math is the decomposed form of tests/ref_gdr.py:263-557 / chunk/blackwell/bwd_sm12x.py (dv_local,
// dq/dk/dw/dg, WY backward), the fused original is chunk/hopper/fused_bwd.py:388-882.
//
// The backward is two kernels:
//  bwd_scan_kernel   (chunk_bwd_scan.cu) one CTA per (sequence, v-head), chunks in reverse order, dS resident
//                    in tensor memory; writes du^T [chunk][Hv][128 v][64 tokens], the state gradient
//                    leaving every chunk dh^T [chunk][Hv][128 v][128 k] and dh0.
//  bwd_chunk_kernel  (this file) persistent CTAs walk the (chunk, k-head) items and loop over the v-heads of the
//                    GQA group, so that dq and dk leave already reduced over the group: the sixteen remaining
//                    products of a chunk, the triangular-inverse backward, dbeta, and dg with its chunk-local
//                    reverse cumulative sum.
//
// Every product is a tcgen05.mma with M = 64 (the 64 tokens of the chunk; such an accumulator occupies 16
// lanes of each 32-lane partition of tensor memory, so two accumulators share a column range: "bank" 0 at
// lane offset 0, bank 1 at lane offset 16), operands are TMA-written or thread-written 128B-swizzled
// shared-memory tiles read K-major or MN-major as the product needs, so no tile is ever transposed.
// Accumulators are read back as 16 x 256 bit fragments: warp (mt, half) gets rows 16 mt .. 16 mt + 15 and half of the
// columns in the mma.sync accumulator layout: thread 4 g + c holds rows g, g + 8 and column pairs 8 nt + 2 c.
//
// One step = one (chunk, v-head).  Products in issue order, with the tensor-memory area they go to and the accumulator
// whose readers must be done with it:
//   dO v_new^T -> P0    du h^T -> W0    du V^T -> R0    dO h^T -> T0    x = A^T du -> W1    Q K^T -> P1    K K^T -> R1
//   | ds, dw written |  dw K^T -> P0    v_new dh^T -> T1
//   | dA written |      M1 = A^T dA -> P1    ds K -> Q0
//   | M1 written |      M1 A^T -> R0    ds^T Q -> Q1    y = A^T dw -> W0
//   | dL written |      (beta dL) K, (beta dL)^T K -> added to Q1
// What a step computes splits in a serial chain (ds -> dw K^T -> dA -> M1 -> dL, five accumulators through registers
// and back) and the rest, which nothing in the step waits for.  Three groups of eight warps:
//   chain warps 0-7:    ds, dA, M1, beta .* dL; sums of the 64 x 64 products (dg, dbeta).  The row products that dbeta and
//                       dg need, x . v, y . k and (dL K) . k, are row and column sums of A .* (du V^T), A .* (dw K^T) and
//                       dL .* (K K^T), which the chain holds in registers anyway.
//   q side, warps 8-15: sum(h .* dh), dw, dq and its row product;   k side, warps 16-23: dv, dk and its row product.
//                       dq and dk gather in tensor memory: these warps put the scaled dO h^T and v_new dh^T there and the
//                       products ds K, ds^T Q, (beta dL) K, (beta dL)^T K of all heads of the group add to them.
//   warp 24: TMA producer + gate vectors, warp 25: MMA issuer, warp 26: adds up the partial sums and forms the reverse
//                       cumulative sum of dg (done by a warp of the k side it made that warp late for the next step).
// Tiles are refilled for the next step as soon as their last product has read them (v_new dh^T for dO, v_new, V, h, dh;
// M1 A^T for du, whose tile holds M1 meanwhile; the last product for Q, K, A), so that the next step's first products
// run while the sides finish this one.
// What bounds it: HBM.  A step moves 216 KB (8 heads of a group share q, k, dq, dk: then 152 KB), 6 to 9 k cycles at the
// rate of a copy; the tensor pipe needs 4.7k.  Measured for 512 chunks of 32 heads: 1177 us with one set of 16 epilogue
// warps doing everything in turn (30k warp instructions per step, sm__inst_executed), 660 to 690 us now (20k).
// Rows beyond the end of a sequence hold the next sequence's tokens (TMA does not know about sequences);
// they never contribute because du, beta, rho and the ds rows of such tokens are exactly zero.
#include "chunk_params.cuh"
#include "warp_pieces.cuh"

namespace qla {
namespace {

constexpr int kGroupWarps = 8;  // chain warps 0..7, q-side warps 8..15, k-side warps 16..23
constexpr int kProducerWarp = 3 * kGroupWarps, kMmaWarp = kProducerWarp + 1, kReduceWarp = kMmaWarp + 1;
constexpr int kThreads = 32 * (kReduceWarp + 1);
// partial sums per parity: dg rows of the q side [2][64], of the k side [2][64], of the chain [2][64], dbeta rows of the
// chain [2][64], dg columns [4][64], dbeta columns [4][64], share of the chunk's last token [16]
constexpr int kRedQ = 0, kRedK = 128, kRedRow = 256, kRedBRow = 384, kRedCol = 512, kRedBCol = 768, kRedLast = 1024, kRedFloats = 1040;

// ---- shared-memory map (offsets from a 1024-byte aligned base; every tile 128B-swizzled)
constexpr uint32_t kOffQ = 0;        // [64][128] as two [64][64] halves
constexpr uint32_t kOffK = 16384;
constexpr uint32_t kOffA = 32768;    // [64][64]
constexpr uint32_t kOffDO = 40960;
constexpr uint32_t kOffVn = 57344;
constexpr uint32_t kOffV = 73728;    // V, then dv on its way out
constexpr uint32_t kOffDu = 90112;   // du^T [128 v][64 tokens], then M1 [64][64]
constexpr uint32_t kOffH = 106496;   // h [128 k][128 v] as two [128][64] halves
constexpr uint32_t kOffDh = 139264;  // dh^T [128 v][128 k] as two [128][64] halves
constexpr uint32_t kOffDw = 172032;  // dw [64][128], written by the output warps; then dq on its way out
constexpr uint32_t kOffX = 188416;   // [64][64]: ds
constexpr uint32_t kOffY = 196608;   // [64][64]: dA, then beta .* dL
constexpr uint32_t kOffDk = 204800;  // dk on its way out
constexpr uint32_t kSmemBytes = 221184 + 1024;
constexpr uint32_t kEarlyBytes = 3 * 16384 + 2 * 32768;  // dO, v_new, V, h, dh^T

// ---- tensor-memory columns; bank 1 = the same columns at lane offset 16
constexpr uint32_t kBank1 = 16u << 16;
constexpr uint32_t kColT = 0;      // dO h^T | v_new dh^T
constexpr uint32_t kColW = 128;    // du h^T, then y = A^T dw | x = A^T du
constexpr uint32_t kColP = 256;    // dO v_new^T, then dw K^T | Q K^T, then M1
constexpr uint32_t kColR = 320;    // du V^T, then M1 A^T | K K^T
constexpr uint32_t kColQ = 384;    // ds K | ds^T Q + (beta dL) K + (beta dL)^T K   (summed over the heads of the group)

enum Bar {
  kEarlyFull = 0, kEarlyFree, kDuFull, kDuFree, kLateFull, kLateFree,  // tiles
  kC45, kC3, kCT1, kCB, kCL1, kCT2, kC12, kC13, kCY, kC4,              // products
  kL1Ready, kDaReady, kM1Ready, kDlReady,                              // operands written by the epilogue warps
  kQ0Ready, kQ1Ready, kDvReady, kDqReady, kDkReady, kStFree, kRedReady, kNumBars
};

// The products of a step in issue order.  The issuer walks this table (constant memory, indexed by a uniform counter): all
// roles share the SM's instruction cache, and with the sixteen products written out forward and backward of 4 x 8192 tokens of
// 32 heads took 1995 to 2020 us against 1950.
struct Product {
  uint32_t bars;    // barrier waited for | << 8, << 16: barriers that the completion arrives on (kNoBar: none)
  uint32_t a, b;    // low words of the shared-memory descriptors: tile offset >> 4 (the CTA's base is added), leading offset
  uint32_t idesc;   // without the element type
  uint32_t d;       // accumulator
  uint32_t steps;   // descriptor step per 16 of K: a | b << 16 (16-byte units)
  uint32_t jumps;   // from the first to the second 64 of K, the same
  uint32_t flags;
};
constexpr uint32_t kNoBar = 255, kAdd = 1, kK128 = 2, kAfterStep = 4;
// An operand tile, its rows K-major (64 columns of K contiguous; the second half of a 128-wide tile `half` bytes behind) or
// MN-major (halves = 64 of M or N, `half` apart; 16 of K are 16 rows of 128 bytes).
struct Operand {
  uint32_t lo, step, jump, major;
};
constexpr Operand kmaj(uint32_t off, uint32_t half) { return {(off >> 4) | (1u << 16), 2, half >> 4, ptx::kMajorK}; }
constexpr Operand mnmaj(uint32_t off, uint32_t half) { return {(off >> 4) | ((half >> 4) << 16), 128, 512, ptx::kMajorMN}; }
constexpr Product product(uint32_t wait, uint32_t done1, uint32_t done2, uint32_t d, Operand a, Operand b, uint32_t n, uint32_t flags) {
  return {wait | (done1 << 8) | (done2 << 16), a.lo, b.lo, ptx::mma_idesc(64, n, 0, a.major, b.major), d, a.step | (b.step << 16),
          a.jump | (b.jump << 16), flags};
}
constexpr int kNumProducts = 16;
__constant__ const Product kProducts[kNumProducts] = {
    product(kEarlyFull, kC45, kNoBar, kColP, kmaj(kOffDO, 8192), kmaj(kOffVn, 8192), 64, kK128),                        // dO v_new^T
    product(kDuFull, kC3, kNoBar, kColW, mnmaj(kOffDu, 8192), kmaj(kOffH, 16384), 128, kK128 | kAfterStep),             // du h^T
    product(kNoBar, kNoBar, kNoBar, kColR, mnmaj(kOffDu, 8192), kmaj(kOffV, 8192), 64, kK128),                          // du V^T
    product(kNoBar, kCT1, kNoBar, kColT, kmaj(kOffDO, 8192), kmaj(kOffH, 16384), 128, kK128),                           // dO h^T
    product(kLateFull, kNoBar, kNoBar, kColW + kBank1, mnmaj(kOffA, 8192), kmaj(kOffDu, 8192), 128, 0),                 // x = A^T du
    product(kNoBar, kNoBar, kNoBar, kColP + kBank1, kmaj(kOffQ, 8192), kmaj(kOffK, 8192), 64, kK128),                   // Q K^T
    product(kNoBar, kCB, kNoBar, kColR + kBank1, kmaj(kOffK, 8192), kmaj(kOffK, 8192), 64, kK128),                      // K K^T
    product(kL1Ready, kCL1, kNoBar, kColP, kmaj(kOffDw, 8192), kmaj(kOffK, 8192), 64, kK128),                           // dw K^T
    product(kNoBar, kCT2, kEarlyFree, kColT + kBank1, kmaj(kOffVn, 8192), mnmaj(kOffDh, 16384), 128, kK128),            // v_new dh^T
    product(kDaReady, kC12, kNoBar, kColP + kBank1, mnmaj(kOffA, 8192), mnmaj(kOffY, 8192), 64, 0),                     // M1 = A^T dA
    product(kQ0Ready, kNoBar, kNoBar, kColQ, kmaj(kOffX, 8192), mnmaj(kOffK, 8192), 128, kAdd),                         // + ds K
    product(kM1Ready, kC13, kDuFree, kColR, kmaj(kOffDu, 8192), kmaj(kOffA, 8192), 64, 0),                              // M1 A^T
    product(kQ1Ready, kNoBar, kNoBar, kColQ + kBank1, mnmaj(kOffX, 8192), mnmaj(kOffQ, 8192), 128, kAdd),               // + ds^T Q
    product(kNoBar, kCY, kNoBar, kColW, mnmaj(kOffA, 8192), mnmaj(kOffDw, 8192), 128, 0),                               // y = A^T dw
    product(kDlReady, kNoBar, kNoBar, kColQ + kBank1, kmaj(kOffY, 8192), mnmaj(kOffK, 8192), 128, kAdd),                // + (beta dL) K
    product(kNoBar, kC4, kLateFree, kColQ + kBank1, mnmaj(kOffY, 8192), mnmaj(kOffK, 8192), 128, kAdd),                 // + (beta dL)^T K
};

struct ChunkCoord {
  int seq, seq_start, seq_end, local_chunk;
};

// chunk index -> sequence (binary search over the exclusive scan of chunks per sequence)
__device__ __forceinline__ ChunkCoord locate_chunk(int chunk, const int32_t* cu, const int32_t* chunk_offsets,
                                                       int num_seqs, int seq_len) {
  ChunkCoord c;
  if (cu != nullptr) {
    int lo = 0, hi = num_seqs - 1;
#pragma unroll 1
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (chunk_offsets[mid] <= chunk) lo = mid; else hi = mid - 1;
    }
    c.seq = lo;
    c.seq_start = cu[lo];
    c.seq_end = cu[lo + 1];
    c.local_chunk = chunk - chunk_offsets[lo];
  } else {
    const int per = (seq_len + kChunk - 1) / kChunk;
    c.seq = chunk / per;
    c.local_chunk = chunk % per;
    c.seq_start = c.seq * seq_len;
    c.seq_end = c.seq_start + seq_len;
  }
  return c;
}

__device__ __forceinline__ float quad_sum(float x) {  // over the four lanes that share a row
  x += __shfl_xor_sync(0xffffffffu, x, 1);
  x += __shfl_xor_sync(0xffffffffu, x, 2);
  return x;
}
// Column sums: v[i] summed over the eight lanes 4 g + c of a column quad; lane (g, c) is left with the sum of v[g].
__device__ __forceinline__ float column_sum(const float (&v)[8], int g) {
  float a[4], b[2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    a[i] = ((g & 4) ? v[i + 4] : v[i]) + __shfl_xor_sync(0xffffffffu, (g & 4) ? v[i] : v[i + 4], 16);
#pragma unroll
  for (int i = 0; i < 2; ++i)
    b[i] = ((g & 2) ? a[i + 2] : a[i]) + __shfl_xor_sync(0xffffffffu, (g & 2) ? a[i] : a[i + 2], 8);
  return ((g & 1) ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, (g & 1) ? b[0] : b[1], 4);
}
// The value itself, but unknown to the compiler: conditions on loop-invariant values (a ragged chunk, the first or last head,
// an element type) are otherwise hoisted by copying the loop body for each of their outcomes.
__device__ __forceinline__ int opaque(int x) {
  asm volatile("" : "+r"(x));
  return x;
}
__device__ __forceinline__ void warp_arrive(uint64_t* bar, int lane) {
  __syncwarp();
  if (lane == 0) ptx::mbar_arrive(bar);
}

template <typename T>
__device__ __forceinline__ uint32_t pack2(float a, float b);
template <>
__device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float a, float b) {
  __nv_bfloat162 x = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&x);
}
template <>
__device__ __forceinline__ uint32_t pack2<__half>(float a, float b) {
  __half2 x = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&x);
}

template <typename T>
__device__ __forceinline__ F2 widen(uint32_t raw);  // two 16-bit values
template <>
__device__ __forceinline__ F2 widen<__nv_bfloat16>(uint32_t raw) {
  return f2(raw << 16, raw & 0xffff0000u);
}
template <>
__device__ __forceinline__ F2 widen<__half>(uint32_t raw) {
  const float2 v = __half22float2(*reinterpret_cast<__half2*>(&raw));
  return f2(v.x, v.y);
}
template <typename T>
__device__ __forceinline__ uint32_t pack2(F2 x) {
  const float2 v = unpack(x);
  return pack2<T>(v.x, v.y);
}
__device__ __forceinline__ float sum2(F2 x) {
  const float2 v = unpack(x);
  return v.x + v.y;
}

// One warp adds up the partial sums of a step: dg (rows + columns + the last token's share) with its chunk-local reverse
// cumulative sum, and dbeta, 32 tokens at a time from the end; `e` is the element of token `lane`.
__device__ __forceinline__ void reduce_step(const float* rr, float* dg_out, float* dbeta_out, int64_t e, int heads, int valid) {
  const int lane = threadIdx.x & 31;
  float last = lane < 2 * kGroupWarps ? rr[kRedLast + lane] : 0.f, tail = 0.f;
#pragma unroll
  for (int off = 8; off > 0; off >>= 1) last += __shfl_xor_sync(0xffffffffu, last, off);
  last = __shfl_sync(0xffffffffu, last, 0);
#pragma unroll 1
  for (int t = lane + 32; t >= 0; t -= 32) {
    float dg = 0.f, db = rr[kRedBRow + t] + rr[kRedBRow + 64 + t];
#pragma unroll
    for (int m = 0; m < 6; ++m) dg += rr[kRedQ + 64 * m + t];  // q side, k side, chain
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      dg += rr[kRedCol + 64 * m + t];
      db += rr[kRedBCol + 64 * m + t];
    }
    if (t == valid - 1) dg += last;
    if (t >= valid) dg = 0.f;  // rows of the next sequence: they must not enter the suffix sum
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {  // dg_raw[c] = sum_{c' >= c} dg_cum[c']
      const float n = __shfl_down_sync(0xffffffffu, dg, off);
      if (lane + off < 32) dg += n;
    }
    dg += tail;
    tail = __shfl_sync(0xffffffffu, dg, 0);
    if (t < valid) {
      const int64_t at = e + static_cast<int64_t>(t - lane) * heads;
      dg_out[at] = dg;
      dbeta_out[at] = db;
    }
  }
}

// kTrace: a separate instantiation whose CTA 0 stamps clock64() at the phase boundaries of its fourth step into
// the buffer registered with qla_set_trace_buffer (events 0..19 chain warp 0, 20..39 the MMA issuer, 40..59 output warp 8).
template <typename T, bool kTrace>
__global__ void __launch_bounds__(kThreads, 1)
bwd_chunk_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                 const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_vn,
                 const __grid_constant__ CUtensorMap tm_do, const __grid_constant__ CUtensorMap tm_a,
                 const __grid_constant__ CUtensorMap tm_h, const __grid_constant__ CUtensorMap tm_dh,
                 const __grid_constant__ CUtensorMap tm_du, const __grid_constant__ CUtensorMap tm_dq,
                 const __grid_constant__ CUtensorMap tm_dk, const __grid_constant__ CUtensorMap tm_dv, const BwdParams p,
                 const int total_items) {
  constexpr uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? ptx::kFmtBF16 : ptx::kFmtF16;
  grid_dep_wait();    // earlier kernels of the stream have completed (see launch_dependent)
  grid_dep_launch();  // the next one may be scheduled; it waits the same way
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int group = p.num_v_heads / p.num_k_heads;
  const int real_chunks = p.cu_seqlens != nullptr ? p.chunk_offsets[p.num_seqs] : 0x7fffffff;

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (ptx::smem_u32(smem_raw) & 1023u)) & 1023u);
  __shared__ uint64_t bars[kNumBars];
  __shared__ uint32_t tmem_base_s;
  __shared__ __align__(16) float sG[2][64];  // log2(e) x cumulative gates of the step (parity), padded rows = last valid
  __shared__ __align__(16) float sB[2][64];  // beta, 0 on padded rows
  __shared__ float red[2 * kRedFloats];
  // what the producer found out about the step (parity): first token, tokens of the sequence, k-head, v-head, whether it
  // is the first / last head of its group
  struct StepInfo {
    int t0, valid, hk, hv, first, last;
  };
  __shared__ StepInfo info[2];

  if (tid < kNumBars) {  // (a thread each)
    const int b = tid;
    int count = 1;  // tcgen05.commit, the producer's expect_tx arrival, or one thread
    if (b == kEarlyFull) count = 33;
    else if (b == kEarlyFree) count = 2 * kGroupWarps + 2;
    else if (b == kLateFree) count = 2 * kGroupWarps + 1;
    else if (b == kL1Ready) count = 2 * kGroupWarps;
    else if (b == kRedReady) count = 3 * kGroupWarps;
    else if (b == kDaReady || b == kM1Ready || b == kDlReady || (b >= kQ0Ready && b <= kDkReady)) count = kGroupWarps;
    ptx::mbar_init(&bars[b], count);
    ptx::fence_mbar_init();
    if (tid == 0) ptx::mbar_wait_setup(p.status, bars, 128);  // (+ 128 in the recorded barrier index: this kernel)
  }
  if (warp == kProducerWarp) {
    ptx::tmem_alloc(&tmem_base_s, 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem = tmem_base_s;
  const uint32_t bar0 = ptx::smem_u32(&bars[0]);
  auto ba = [&](int b) { return bar0 + 8u * static_cast<uint32_t>(b); };
  // A wait that gives up (bounded, status word set) does not leave the loop on the spot: a branch out of the middle of these
  // loops makes the compiler lay out a copy of the rest, and the instruction cache is short already (12 % misses).  The
  // remaining waits of the step fail at once, its accesses are in bounds as ever, and the loop ends behind it.
  auto wait = [&](int b, uint32_t parity) { return ptx::mbar_wait_addr(ba(b), parity); };
  // steps of this CTA: items blockIdx.x, + gridDim.x, .. of the chunks there are, times the heads of a group
  const int items = static_cast<int>(min(static_cast<int64_t>(total_items), static_cast<int64_t>(real_chunks) * p.num_k_heads));
  const int steps = items > static_cast<int>(blockIdx.x)
                        ? (items - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x) * group
                        : 0;
  auto trace = [&](int step, int ev) {  // (warp-uniform: a lane-dependent branch before an MMA costs more than the stamp)
    if (kTrace && p.trace != nullptr && blockIdx.x == 0 && step == 8) p.trace[ev] = clock64();
  };

  if (warp == kProducerWarp) {
    // =========================================================== producer: TMA + gate vectors
    bool ok = true;
    int item = blockIdx.x, hh = 0;
    auto locate = [&](int it) {
      const int chunk = it / p.num_k_heads;
      StepInfo x;
      const ChunkCoord cc = locate_chunk(chunk, p.cu_seqlens, p.chunk_offsets, p.num_seqs, p.seq_len);
      x.t0 = cc.seq_start + cc.local_chunk * kChunk;
      x.valid = min(kChunk, cc.seq_end - x.t0);
      x.hk = it - chunk * p.num_k_heads;
      x.hv = x.hk * group;
      x.first = chunk;  // (replaced below)
      x.last = 0;
      return x;
    };
    StepInfo next = locate(steps > 0 ? item : 0);
    int next_chunk = next.first;
#pragma unroll 1
    for (int step = 0; ok && step < steps; ++step) {
      const int ph = step & 1, beta_dtype = opaque(p.beta_dtype);
      const StepInfo cur = next;
      const int chunk = next_chunk, hv = cur.hv, t0 = cur.t0, valid = cur.valid;
      const bool first = opaque(hh) == 0, last = opaque(hh) == group - 1;
      // gates and description of this step into its parity slot (the previous readers finished two steps ago: kLateFree)
      const int64_t last_tok = static_cast<int64_t>(t0) + valid - 1;
#pragma unroll 1
      for (int c = lane; c < kChunk; c += 32) {
        const bool okc = c < valid;
        const int64_t tok = okc ? static_cast<int64_t>(t0) + c : last_tok;
        sG[ph][c] = 1.4426950408889634f * p.g_cumsum[tok * p.num_v_heads + hv];
        sB[ph][c] = okc ? load_scalar(p.beta, beta_dtype, tok * p.num_v_heads + hv) : 0.f;
      }
      const int row = (chunk * p.num_v_heads + hv) * kHeadDim;  // row of the [chunks * Hv * 128, width] views
      if (opaque(step) > 0) ok &= wait(kEarlyFree, ph ^ 1);
      if (lane == 0) {
        info[ph] = StepInfo{t0, valid, cur.hk, hv, first, last};  // (the reducing warp was the last to read the slot)
        uint64_t* full = &bars[kEarlyFull];
        ptx::mbar_expect_tx(full, kEarlyBytes);
        ptx::tma_load_4d(smem + kOffDO, &tm_do, full, 0, hv, t0, 0);
        ptx::tma_load_4d(smem + kOffVn, &tm_vn, full, 0, hv, t0, 0);
        ptx::tma_load_4d(smem + kOffH, &tm_h, full, 0, 0, row, 0);
        ptx::tma_load_4d(smem + kOffV, &tm_v, full, 0, hv, t0, 0);
        ptx::tma_load_4d(smem + kOffDh, &tm_dh, full, 0, 0, row, 0);
      }
      __syncwarp();
      ptx::mbar_arrive(&bars[kEarlyFull]);  // 32 arrivals (gates written) + the expect_tx arrival
      if (opaque(step) > 0) ok &= wait(kDuFree, ph ^ 1);
      if (lane == 0) {
        ptx::mbar_expect_tx(&bars[kDuFull], 16384);
        ptx::tma_load_3d(smem + kOffDu, &tm_du, &bars[kDuFull], 0, 0, row);
      }
      __syncwarp();
      if (opaque(step) > 0) ok &= wait(kLateFree, ph ^ 1);
      if (lane == 0) {
        uint64_t* full = &bars[kLateFull];
        ptx::mbar_expect_tx(full, first ? 8192 + 32768 : 8192);
        ptx::tma_load_3d(smem + kOffA, &tm_a, full, 0, hv, t0);
        if (first) {
          ptx::tma_load_4d(smem + kOffQ, &tm_q, full, 0, cur.hk, t0, 0);
          ptx::tma_load_4d(smem + kOffK, &tm_k, full, 0, cur.hk, t0, 0);
        }
      }
      __syncwarp();
      // the tiles of the NEXT step into L2, so that its demand loads (issued when this step's buffers are
      // released) find them there
      if (last) {
        hh = 0;
        item += gridDim.x;
        if (step + 1 < steps) {
          next = locate(item);
          next_chunk = next.first;
        }
      } else {
        ++hh;
        ++next.hv;
      }
      if (step + 1 < steps) {
        const int t2 = next.t0, hv2 = next.hv;
        if (lane == 0) {
          const int row2 = (next_chunk * p.num_v_heads + hv2) * kHeadDim;
          ptx::tma_prefetch_l2_4d(&tm_do, 0, hv2, t2, 0);
          ptx::tma_prefetch_l2_4d(&tm_vn, 0, hv2, t2, 0);
          ptx::tma_prefetch_l2_4d(&tm_h, 0, 0, row2, 0);
          ptx::tma_prefetch_l2_4d(&tm_v, 0, hv2, t2, 0);
          ptx::tma_prefetch_l2_4d(&tm_dh, 0, 0, row2, 0);
          ptx::tma_prefetch_l2_3d(&tm_du, 0, 0, row2);
          ptx::tma_prefetch_l2_3d(&tm_a, 0, hv2, t2);
          if (last) {
            ptx::tma_prefetch_l2_4d(&tm_q, 0, next.hk, t2, 0);
            ptx::tma_prefetch_l2_4d(&tm_k, 0, next.hk, t2, 0);
          }
        }
        __syncwarp();
#pragma unroll 1
        for (int c = lane; c < next.valid; c += 32) {
          const int64_t e = (static_cast<int64_t>(t2) + c) * p.num_v_heads + hv2;
          ptx::prefetch_l2(p.g_cumsum + e);
          ptx::prefetch_l2(static_cast<const uint8_t*>(p.beta) + e * (beta_dtype == QLA_DT_F32 ? 4 : 2));
        }
        __syncwarp();
      }
    }
  } else if (warp == kMmaWarp) {
    // =========================================================== MMA issuer (whole warp, converged)
    bool ok = tmem == 0;  // the CTA owns all 512 columns: the allocation starts at column 0
    if (!ok) ptx::record_wait_failure(p.status, kStatusBadTmemBase, 0);
    const uint32_t base = ptx::smem_u32(smem) >> 4;
    constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);  // see smem_desc_sw128
#pragma unroll 1
    for (int step = 0; ok && step < steps; ++step) {
      const uint32_t ph = step & 1;
      trace(step, 20);
#pragma unroll 1
      for (int j = 0; j < kNumProducts; ++j) {
        // (the readers of T0, T1 and W1 of the previous step have released the early tiles)
        const Product pr = kProducts[j];
        const uint32_t w = pr.bars;
        if ((pr.flags & kAfterStep) && opaque(step) > 0) ok = ptx::mbar_wait_nocall(ba(kLateFree), ph ^ 1, ok);  // y and the sums of the previous step read
        if ((w & 255u) != kNoBar) {
          ok = ptx::mbar_wait_nocall(ba(w & 255u), ph, ok);
          ptx::tc_fence_after_sync();
        }
        trace(step, 21 + j);
        const uint32_t alo = pr.a + base, blo = pr.b + base, idesc = (fmt << 7) | (fmt << 10) | pr.idesc;
        ptx::umma_ss_k64_steps(pr.d, alo, blo, kDescHi, idesc, (pr.flags & kAdd) != 0, pr.steps & 0xffffu, pr.steps >> 16);
        if (pr.flags & kK128)
          ptx::umma_ss_k64_steps(pr.d, alo + (pr.jumps & 0xffffu), blo + (pr.jumps >> 16), kDescHi, idesc, true, pr.steps & 0xffffu,
                                 pr.steps >> 16);
        if (((w >> 8) & 255u) != kNoBar) ptx::umma_commit(&bars[(w >> 8) & 255u]);
        if ((w >> 16) != kNoBar) ptx::umma_commit(&bars[w >> 16]);
      }
    }
    ptx::report_issuer(p.status, ok, 128 + kNumBars);
  } else if (warp == kReduceWarp) {
    // =========================================================== sums of a step
    // It releases the slot of a step (partial sums, description) as one of the arrivals that let the next step's early tiles
    // be replaced: two steps later they have been.
    bool ok = true;
    if (lane == 0) ptx::mbar_arrive(&bars[kEarlyFree]);
#pragma unroll 1
    for (int step = 0; ok && step < steps; ++step) {
      const uint32_t ph = step & 1;
      ok &= wait(kRedReady, ph);
      const int t0 = info[ph].t0, valid = info[ph].valid, hv = info[ph].hv;
      reduce_step(red + ph * kRedFloats, p.dg, p.dbeta, (static_cast<int64_t>(t0) + lane) * p.num_v_heads + hv, p.num_v_heads, valid);
      ok &= wait(kEarlyFree, ph);  // (so that the arrival below counts for the next phase)
      warp_arrive(&bars[kEarlyFree], lane);
    }
  } else {
    // =========================================================== the three groups of epilogue warps
    const int g = lane >> 2, c4 = lane & 3;
    const int mt = warp & 3, half = (warp >> 2) & 1;  // rows 16 mt .., half of the columns
    const int r0 = mt * 16 + g, r1 = r0 + 8;          // the two rows this thread owns in every fragment
    const uint32_t tq = tmem + (static_cast<uint32_t>(mt * 32) << 16);  // bank 0 of this warp's partition
    const uint32_t sm = ptx::smem_u32(smem);
    // Fragments of 16 x 16 columns go to and come from 128B-swizzled tiles with one stmatrix / ldmatrix of four 8 x 8
    // matrices (rows +0 / +8 of two column groups): lane i names row i % 16 of column group i / 16.
    const uint32_t mrow = static_cast<uint32_t>(mt * 16 + (lane & 15)) * 128, mcol = lane >> 4, msw = lane & 7;
    auto frag_addr = [&](uint32_t tile, int c16) { return tile + mrow + (((c16 + mcol) ^ msw) << 4); };
    bool ok = true;

    // ---- both sides: columns 64 half + 8 nt + 2 c4 + {0, 1} of the 128-wide products
    const int ow = warp & (kGroupWarps - 1);
    const uint32_t tw = tq + 64 * half;
    const uint32_t h8 = 8192u * half;  // this warp's half of a [64][128] tile
    const uint32_t s_dw = sm + kOffDw + h8, s_dv = sm + kOffV + h8, s_dk = sm + kOffDk + h8;
    const uint32_t s_q = sm + kOffQ + h8, s_k = sm + kOffK + h8;
    // 32 of the warp's 64 columns at a time (part 0 / 1): accumulators as pairs of neighbouring columns, pair
    // 2 nt + (row r1), and their rounded values into a tile
    auto load_w = [&](uint32_t col, int part, uint32_t (&r)[16]) { ptx::tmem_ld_frag4(tw + col + 32 * part, r); };
    auto store_w = [&](uint32_t tile, int part, const F2 (&x)[8]) {
#pragma unroll
      for (int j = 0; j < 2; ++j)
        ptx::stmatrix_x4(frag_addr(tile, 4 * part + 2 * j), pack2<T>(x[4 * j]), pack2<T>(x[4 * j + 1]), pack2<T>(x[4 * j + 2]),
                         pack2<T>(x[4 * j + 3]));
    };
    // Ragged tail chunk: the rows of the sequence among this warp's 16 x 64 block of the tile, copied by the warp itself.
    auto copy_rows = [&](const uint8_t* tile, void* base, int heads, int head, int t0, int valid) {
      __syncwarp();
#pragma unroll 1
      for (int i = 0; i < 4; ++i) {
        const int row = mt * 16 + 4 * i + (lane >> 3);
        if (row < valid)
          *reinterpret_cast<uint4*>(static_cast<T*>(base) + (static_cast<int64_t>(t0 + row) * heads + head) * kHeadDim +
                                    64 * half + 8 * (lane & 7)) =
              *reinterpret_cast<const uint4*>(tile + h8 + ptx::sw128_offset(row, lane & 7));
      }
      __syncwarp();
    };
    // A tile leaves through a TMA store (`send`) once all eight warps have written their part; the group's first warp issues it.
    // Every step arrives once on each of the three barriers, also when there is nothing to send.
    auto stored = [&](int bar, uint32_t ph, bool send, const CUtensorMap* tm, uint32_t off, int head, int t0) {
      ptx::fence_proxy_async_smem();
      warp_arrive(&bars[bar], lane);
      bool done = true;
      if (opaque(ow) == 0) {
        done = wait(bar, ph);
        if (send && lane == 0) {
          ptx::tma_store_4d(tm, smem + off, 0, head, t0, 0);
          ptx::tma_store_commit();
        }
        __syncwarp();
      }
      return done;
    };
    if (warp < kGroupWarps) {
      // --------------------------------------------------------- chain warps: columns 32 half + 8 nt + 2 c4 + {0, 1}
      const uint32_t tx = tq + 32 * half;
      const int dr = r0 - 32 * half - 2 * c4;  // row - column of (r0, nt = 0, e = 0)
      const uint32_t s_ds = sm + kOffX, s_da = sm + kOffY, s_m1 = sm + kOffDu, s_a = sm + kOffA;
      auto load = [&](uint32_t col, uint32_t (&r)[16]) { ptx::tmem_ld_frag4(tx + col, r); };
      auto store = [&](uint32_t tile, const float (&x)[16]) {
#pragma unroll
        for (int j = 0; j < 2; ++j)
          ptx::stmatrix_x4(frag_addr(tile, 4 * half + 2 * j), pack2<T>(x[8 * j], x[8 * j + 1]), pack2<T>(x[8 * j + 2], x[8 * j + 3]),
                           pack2<T>(x[8 * j + 4], x[8 * j + 5]), pack2<T>(x[8 * j + 6], x[8 * j + 7]));
        ptx::fence_proxy_async_smem();
        ptx::tc_fence_before_sync();
      };
#pragma unroll 1
        for (int step = 0; ok && step < steps; ++step) {
          const uint32_t ph = step & 1;
          ok &= wait(kEarlyFull, ph);
          if (warp == 0) trace(step, 0);
          const int valid = info[ph].valid;
          // decay factors exp(min(g_row - g_col, 0)) of this thread's 16 (row, column) pairs (element
          // i = 4 nt + 2 (row r1) + e), exp(g_col) and beta of its eight columns
          const float g0 = sG[ph][r0], g1 = sG[ph][r1], be0 = sB[ph][r0], be1 = sB[ph][r1];
          float gw[16], ecol[8], bcol[8];
#pragma unroll
          for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const float gc = sG[ph][32 * half + 8 * nt + 2 * c4 + e];
              gw[4 * nt + e] = ptx::ex2(fminf(g0 - gc, 0.f));
              gw[4 * nt + 2 + e] = ptx::ex2(fminf(g1 - gc, 0.f));
              ecol[2 * nt + e] = ptx::ex2(gc);
              bcol[2 * nt + e] = sB[ph][32 * half + 8 * nt + 2 * c4 + e];
            }
          const int dv0 = r0 < valid ? dr : -1, dv1 = r1 < valid ? dr + 8 : -1;  // ds: rows of the sequence only
          float dg_row0 = 0.f, dg_row1 = 0.f, db_row0 = 0.f, db_row1 = 0.f, dg_col[8], db_col[8];

          // ---- ds = s G .* (dO v_new^T);  then ds .* (Q K^T) into dg
          ok &= wait(kC45, ph);
          ptx::tc_fence_after_sync();
          if (warp == 0) trace(step, 1);
          {
            uint32_t r[16];
            float ds[16];
            load(kColP, r);
            ptx::tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i)
              ds[i] = (8 * (i >> 2) + (i & 1) <= ((i & 2) ? dv1 : dv0)) ? __uint_as_float(r[i]) * (p.scale * gw[i]) : 0.f;
            store(s_ds, ds);
            warp_arrive(&bars[kL1Ready], lane);
            if (warp == 0) trace(step, 2);
            ok &= wait(kCB, ph);
            ptx::tc_fence_after_sync();
            load(kColP + kBank1, r);
            ptx::tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const float t = ds[i] * __uint_as_float(r[i]);
              (i & 2 ? dg_row1 : dg_row0) += t;
              const int c = 2 * (i >> 2) + (i & 1);
              dg_col[c] = (i & 2) ? dg_col[c] - t : -t;
            }
          }
          if (warp == 0) trace(step, 3);
          // ---- dA = beta_d (gamma_d (dw K^T) + du V^T), strictly lower;  column sums of A .* that without beta: dbeta,
          //      and of A .* beta gamma (dw K^T): dg
          ok &= wait(kCL1, ph);
          ptx::tc_fence_after_sync();
          if (warp == 0) trace(step, 4);
          {
            uint32_t r1a[16], r2a[16];
            float a1[16], a2[16];
            load(kColP, r1a);
            load(kColR, r2a);
            ptx::tmem_wait_ld();
            float da[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int c = 2 * (i >> 2) + (i & 1);
              a1[i] = ecol[c] * __uint_as_float(r1a[i]);
              a2[i] = a1[i] + __uint_as_float(r2a[i]);
              da[i] = (8 * (i >> 2) + (i & 1) < dr + ((i & 2) ? 8 : 0)) ? bcol[c] * a2[i] : 0.f;
            }
            store(s_da, da);
            warp_arrive(&bars[kDaReady], lane);
            if (warp == 0) trace(step, 5);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              uint32_t m[4];
              mm::ldsm_x4(m, frag_addr(s_a, 4 * half + 2 * j));
#pragma unroll
              for (int x = 0; x < 4; ++x) {  // matrix x: column group 2 j + x / 2, rows +8 (x & 1)
                const float2 a = unpack(widen<T>(m[x]));
                const int i = 8 * j + 4 * (x >> 1) + 2 * (x & 1), c = 2 * (2 * j + (x >> 1));
                dg_col[c] += bcol[c] * (a.x * a1[i]);
                dg_col[c + 1] += bcol[c + 1] * (a.y * a1[i + 1]);
                db_col[c] = (x & 1) ? db_col[c] + a.x * a2[i] : a.x * a2[i];
                db_col[c + 1] = (x & 1) ? db_col[c + 1] + a.y * a2[i + 1] : a.y * a2[i + 1];
              }
            }
          }
          // ---- M1 = A^T dA as the next operand, in the du tile (every product that reads du is done)
          ok &= wait(kC12, ph);
          ptx::tc_fence_after_sync();
          if (warp == 0) trace(step, 6);
          {
            uint32_t r[16];
            float x[16];
            load(kColP + kBank1, r);
            ptx::tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) x[i] = __uint_as_float(r[i]);
            store(s_m1, x);
            warp_arrive(&bars[kM1Ready], lane);
          }
          if (warp == 0) trace(step, 7);
          // ---- dL = -(M1 A^T) .* G, strictly lower; beta .* dL over dA;  u = dL .* (K K^T): dbeta += row sums of u,
          //      dg += row sums - column sums of beta .* u
          ok &= wait(kC13, ph);
          ptx::tc_fence_after_sync();
          if (warp == 0) trace(step, 8);
          {
            uint32_t r[16], kk[16];
            float dl[16], lb[16];
            load(kColR, r);
            load(kColR + kBank1, kk);
            ptx::tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              dl[i] = (8 * (i >> 2) + (i & 1) < dr + ((i & 2) ? 8 : 0)) ? -__uint_as_float(r[i]) * gw[i] : 0.f;
              lb[i] = ((i & 2) ? be1 : be0) * dl[i];
            }
            store(s_da, lb);
            warp_arrive(&bars[kDlReady], lane);
            if (warp == 0) trace(step, 9);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const float k2 = __uint_as_float(kk[i]);
              const float t = lb[i] * k2;
              (i & 2 ? dg_row1 : dg_row0) += t;
              dg_col[2 * (i >> 2) + (i & 1)] -= t;
              (i & 2 ? db_row1 : db_row0) += dl[i] * k2;
            }
          }
          // ---- partial sums
          float* rr = red + ph * kRedFloats;
          const float s0 = quad_sum(dg_row0), s1 = quad_sum(dg_row1), b0 = quad_sum(db_row0), b1 = quad_sum(db_row1);
          if (c4 == 0) {
            rr[kRedRow + half * 64 + r0] = s0;
            rr[kRedRow + half * 64 + r1] = s1;
            rr[kRedBRow + half * 64 + r0] = b0;
            rr[kRedBRow + half * 64 + r1] = b1;
          }
          const int col = mt * 64 + 32 * half + 8 * (g >> 1) + 2 * c4 + (g & 1);
          rr[kRedCol + col] = column_sum(dg_col, g);
          rr[kRedBCol + col] = column_sum(db_col, g);
          warp_arrive(&bars[kRedReady], lane);
          if (warp == 0) trace(step, 10);
        }
    } else if (warp < 2 * kGroupWarps) {
      // --------------------------------------------------------- q side: dw, dq
#pragma unroll 1
        for (int step = 0; ok && step < steps; ++step) {
          const uint32_t ph = step & 1;
          ok &= wait(kEarlyFull, ph);
          const int t0 = info[ph].t0, valid = info[ph].valid, hk = info[ph].hk, hv = info[ph].hv;
          const bool first_head = info[ph].first, last_head = info[ph].last;
          if (kTrace && ow == 0) trace(step, 40);
          const float gam0 = ptx::ex2(sG[ph][r0]), gam1 = ptx::ex2(sG[ph][r1]);
          float dg_last;
          // ---- sum(h .* dh): 16 rows of h per warp against the transposed 16 columns of dh^T.  (As the diagonal of an
          //      mma.sync product it took 3400 cycles instead of these instructions' 700: it queues behind the tcgen05 products.)
          {
            F2 s[2] = {0, 0};
            const uint32_t hrow = sm + kOffH + static_cast<uint32_t>(16 * ow + (lane & 15)) * 128;
            const uint32_t dcol = sm + kOffDh + (ow >> 2) * 16384 + (8 * (lane >> 4) + (lane & 7)) * 128 +
                                  (((2 * (ow & 3) + ((lane >> 3) & 1)) ^ msw) << 4);
#pragma unroll 2
            for (int v = 0; v < 8; ++v) {  // 16 v at a time: matrices (k +0, v +0), (k +8, v +0), (k +0, v +8), (k +8, v +8)
              uint32_t a[4], b[4];
              mm::ldsm_x4(a, hrow + (v >> 2) * 16384 + (((2 * (v & 3) + (lane >> 4)) ^ msw) << 4));
              mm::ldsm_x4_trans(b, dcol + v * 2048);
#pragma unroll
              for (int i = 0; i < 4; ++i) s[i & 1] = fma2(widen<T>(a[i]), widen<T>(b[i]), s[i & 1]);
            }
            dg_last = ptx::ex2(sG[ph][valid - 1]) * (sum2(s[0]) + sum2(s[1]));
          }
          if (opaque(ow) == 0) {  // the stores of the previous step have read the dw tile
            if (lane == 0) {
              ptx::tma_store_wait_read();
              ptx::mbar_arrive(&bars[kStFree]);
            }
            __syncwarp();
          }
          ok &= wait(kStFree, ph);

          // ---- dw = -du h^T
          ok &= wait(kC3, ph);
          ptx::tc_fence_after_sync();
          if (kTrace && ow == 0) trace(step, 42);
#pragma unroll 1
          for (int part = 0; part < 2; ++part) {
            uint32_t r[16];
            load_w(kColW, part, r);
            ptx::tmem_wait_ld();
            F2 x[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = f2(-__uint_as_float(r[2 * i]), -__uint_as_float(r[2 * i + 1]));
            store_w(s_dw, part, x);
          }
          ptx::fence_proxy_async_smem();
          ptx::tc_fence_before_sync();
          warp_arrive(&bars[kL1Ready], lane);
          if (kTrace && ow == 0) trace(step, 43);

          // ---- dO h^T: dq += s gamma .* that, dg += q . that
          float dg0, dg1;
          ok &= wait(kCT1, ph);
          ok &= wait(kLateFull, ph);
          ptx::tc_fence_after_sync();
          if (kTrace && ow == 0) trace(step, 44);
          {
            const F2 f[2] = {f2(p.scale * gam0, p.scale * gam0), f2(p.scale * gam1, p.scale * gam1)};
            F2 s[2] = {0, 0};
#pragma unroll 1
            for (int part = 0; part < 2; ++part) {
              uint32_t r[16], y[16], m[8];
              load_w(kColT, part, r);
              if (opaque(first_head)) {
#pragma unroll
                for (int i = 0; i < 16; ++i) y[i] = 0;
              } else {
                load_w(kColQ, part, y);
              }
              mm::ldsm_x4(reinterpret_cast<uint32_t(&)[4]>(m[0]), frag_addr(s_q, 4 * part));
              mm::ldsm_x4(reinterpret_cast<uint32_t(&)[4]>(m[4]), frag_addr(s_q, 4 * part + 2));
              ptx::tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const F2 x = f2(r[2 * i], r[2 * i + 1]);
                s[i & 1] = fma2(x, widen<T>(m[i]), s[i & 1]);
                const float2 v = unpack(fma2(f[i & 1], x, f2(y[2 * i], y[2 * i + 1])));
                r[2 * i] = __float_as_uint(v.x);
                r[2 * i + 1] = __float_as_uint(v.y);
              }
              ptx::tmem_st_frag4(tw + kColQ + 32 * part, r);
            }
            ptx::tmem_wait_st();
            ptx::tc_fence_before_sync();
            warp_arrive(&bars[kQ0Ready], lane);
            dg0 = p.scale * gam0 * sum2(s[0]);
            dg1 = p.scale * gam1 * sum2(s[1]);
          }
          ptx::tc_fence_before_sync();
          warp_arrive(&bars[kEarlyFree], lane);  // T0
          dg0 = quad_sum(dg0);
          dg1 = quad_sum(dg1);
          if (kTrace && ow == 0) trace(step, 45);

          // ---- dq, complete with the ds K of all heads
          ok &= wait(kCY, ph);
          ptx::tc_fence_after_sync();
          if (kTrace && ow == 0) trace(step, 50);
          float* rr = red + ph * kRedFloats;  // (dO h^T of the next step may be done before the chain has added to this one's
          if (c4 == 0) {
            rr[kRedQ + half * 64 + r0] = dg0;
            rr[kRedQ + half * 64 + r1] = dg1;
          }
#pragma unroll
          for (int off = 16; off > 0; off >>= 1) dg_last += __shfl_xor_sync(0xffffffffu, dg_last, off);
          if (lane == 0) rr[kRedLast + ow] = dg_last;
          warp_arrive(&bars[kRedReady], lane);  // sums, the products behind it are not)
          if (opaque(last_head)) {
#pragma unroll 1
            for (int part = 0; part < 2; ++part) {
              uint32_t r[16];
              load_w(kColQ, part, r);
              ptx::tmem_wait_ld();
              F2 x[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) x[i] = f2(r[2 * i], r[2 * i + 1]);
              store_w(s_dw, part, x);  // (dw has been read)
            }
            ptx::tc_fence_before_sync();
            if (opaque(valid) < kChunk) copy_rows(smem + kOffDw, p.dq, p.num_k_heads, hk, t0, valid);
          }
          warp_arrive(&bars[kLateFree], lane);  // Q rows, Q0
          ok &= stored(kDqReady, ph, last_head && valid == kChunk, &tm_dq, kOffDw, hk, t0);
          if (kTrace && ow == 0) trace(step, 51);

        }
      if (ow == 0 && lane == 0) ptx::tma_store_wait_all();
    } else {
      // --------------------------------------------------------- k side: dv, dk
#pragma unroll 1
        for (int step = 0; ok && step < steps; ++step) {
          const uint32_t ph = step & 1;
          ok &= wait(kEarlyFull, ph);
          const int t0 = info[ph].t0, valid = info[ph].valid, hk = info[ph].hk, hv = info[ph].hv;
          const bool first_head = info[ph].first, last_head = info[ph].last;
          const float gl = sG[ph][valid - 1], g0 = sG[ph][r0], g1 = sG[ph][r1];
          const float gam0 = ptx::ex2(g0), gam1 = ptx::ex2(g1);
          const float rho0 = (r0 < valid) ? ptx::ex2(gl - g0) : 0.f, rho1 = (r1 < valid) ? ptx::ex2(gl - g1) : 0.f;
          const float be0 = sB[ph][r0], be1 = sB[ph][r1];
          float dg_last = 0.f;
          if (kTrace && ow == 0) trace(step, 41);
          float dg0, dg1;
          // ---- dv = beta .* x through the V tile (its product is done) or row by row
          ok &= wait(kCB, ph);
          ptx::tc_fence_after_sync();
          if (kTrace && ow == 0) trace(step, 46);
          {
            const F2 f[2] = {f2(be0, be0), f2(be1, be1)};
#pragma unroll 1
            for (int part = 0; part < 2; ++part) {
              uint32_t r[16];
              load_w(kColW + kBank1, part, r);
              ptx::tmem_wait_ld();
              F2 x[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) x[i] = mul2(f[i & 1], f2(r[2 * i], r[2 * i + 1]));
              store_w(s_dv, part, x);
            }
            if (opaque(valid) < kChunk) copy_rows(smem + kOffV, p.dv, p.num_v_heads, hv, t0, valid);
            ok &= stored(kDvReady, ph, valid == kChunk, &tm_dv, kOffV, hv, t0);
          }
          if (kTrace && ow == 0) trace(step, 47);

          // ---- v_new dh^T: dk += rho .* that, dg -= k . that
          ok &= wait(kCT2, ph);
          ok &= wait(kLateFull, ph);  // (K rows)
          ptx::tc_fence_after_sync();
          if (kTrace && ow == 0) trace(step, 48);
          {
            const F2 f[2] = {f2(rho0, rho0), f2(rho1, rho1)};
            F2 s[2] = {0, 0};
#pragma unroll 1
            for (int part = 0; part < 2; ++part) {
              uint32_t r[16], y[16], m[8];
              load_w(kColT + kBank1, part, r);
              if (opaque(first_head)) {
#pragma unroll
                for (int i = 0; i < 16; ++i) y[i] = 0;
              } else {
                load_w(kColQ + kBank1, part, y);
              }
              mm::ldsm_x4(reinterpret_cast<uint32_t(&)[4]>(m[0]), frag_addr(s_k, 4 * part));
              mm::ldsm_x4(reinterpret_cast<uint32_t(&)[4]>(m[4]), frag_addr(s_k, 4 * part + 2));
              ptx::tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const F2 x = f2(r[2 * i], r[2 * i + 1]);
                s[i & 1] = fma2(x, widen<T>(m[i]), s[i & 1]);
                const float2 v = unpack(fma2(f[i & 1], x, f2(y[2 * i], y[2 * i + 1])));
                r[2 * i] = __float_as_uint(v.x);
                r[2 * i + 1] = __float_as_uint(v.y);
              }
              ptx::tmem_st_frag4(tw + kColQ + kBank1 + 32 * part, r);
            }
            ptx::tmem_wait_st();
            // the dv store must have read the V tile before that is released below, and (through the products that wait
            // here) the dk store of the previous step its tile before the next dk is written
            if (opaque(ow) == 0 && lane == 0) ptx::tma_store_wait_read();
            ptx::tc_fence_before_sync();
            warp_arrive(&bars[kQ1Ready], lane);
            const float s0 = rho0 * sum2(s[0]), s1 = rho1 * sum2(s[1]);
            dg0 = -quad_sum(s0);
            dg1 = -quad_sum(s1);
            dg_last += s0 + s1;
          }
          // ---- this warp's partial sums
          float* rr = red + ph * kRedFloats;
          if (c4 == 0) {
            rr[kRedK + half * 64 + r0] = dg0;
            rr[kRedK + half * 64 + r1] = dg1;
          }
#pragma unroll
          for (int off = 16; off > 0; off >>= 1) dg_last += __shfl_xor_sync(0xffffffffu, dg_last, off);
          if (lane == 0) rr[kRedLast + kGroupWarps + ow] = dg_last;
          warp_arrive(&bars[kRedReady], lane);
          // this warp no longer reads the early tiles or their accumulators
          ptx::tc_fence_before_sync();
          warp_arrive(&bars[kEarlyFree], lane);
          if (kTrace && ow == 0) trace(step, 49);

          // ---- y = A^T dw: dk += (beta gamma) .* y, and with the products of the 64 x 64 gradients dk is complete
          ok &= wait(kC4, ph);
          ptx::tc_fence_after_sync();
          if (kTrace && ow == 0) trace(step, 52);
          {
            const float e0 = be0 * gam0, e1 = be1 * gam1;
            const F2 f[2] = {f2(e0, e0), f2(e1, e1)};
#pragma unroll 1
            for (int part = 0; part < 2; ++part) {
              uint32_t r[16], y[16];
              load_w(kColW, part, y);
              load_w(kColQ + kBank1, part, r);
              ptx::tmem_wait_ld();
              F2 x[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) x[i] = fma2(f[i & 1], f2(y[2 * i], y[2 * i + 1]), f2(r[2 * i], r[2 * i + 1]));
              if (opaque(last_head)) {
                store_w(s_dk, part, x);
              } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                  const float2 v = unpack(x[i]);
                  r[2 * i] = __float_as_uint(v.x);
                  r[2 * i + 1] = __float_as_uint(v.y);
                }
                ptx::tmem_st_frag4(tw + kColQ + kBank1 + 32 * part, r);
              }
            }
            ptx::tmem_wait_st();
            ptx::tc_fence_before_sync();
            warp_arrive(&bars[kLateFree], lane);  // Q, K, A and this step's accumulators
            if (opaque(last_head) && valid < kChunk) copy_rows(smem + kOffDk, p.dk, p.num_k_heads, hk, t0, valid);
          }
          ok &= stored(kDkReady, ph, last_head && valid == kChunk, &tm_dk, kOffDk, hk, t0);
          if (kTrace && ow == 0) trace(step, 53);

          if (kTrace && ow == 0) trace(step, 54);
        }
      if (ow == 0 && lane == 0) ptx::tma_store_wait_all();
    }
  }

  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == kProducerWarp) ptx::tmem_dealloc(tmem, 512);
}

}  // namespace

int launch_chunk_bwd(const BwdParams& p, int64_t total_tokens, int total_chunks_upper, bool is_bf16,
                     cudaStream_t stream) {
  int rc;
  CUtensorMap tm_q, tm_k, tm_v, tm_vn, tm_do, tm_a, tm_h, tm_dh, tm_du, tm_dq, tm_dk, tm_dv;
  const uint64_t state_rows = static_cast<uint64_t>(total_chunks_upper) * p.num_v_heads * kHeadDim;
  if ((rc = make_tmap_halves(&tm_q, p.q, total_tokens, p.num_k_heads, 64, is_bf16)) != QLA_OK) return rc;
  if ((rc = make_tmap_halves(&tm_k, p.k, total_tokens, p.num_k_heads, 64, is_bf16)) != QLA_OK) return rc;
  if ((rc = make_tmap_halves(&tm_v, p.v, total_tokens, p.num_v_heads, 64, is_bf16)) != QLA_OK) return rc;
  if ((rc = make_tmap_halves(&tm_vn, p.v_new, total_tokens, p.num_v_heads, 64, is_bf16)) != QLA_OK) return rc;
  if ((rc = make_tmap_halves(&tm_do, p.d_o, total_tokens, p.num_v_heads, 64, is_bf16)) != QLA_OK) return rc;
  if ((rc = make_tmap_3d(&tm_a, p.A, total_tokens, p.num_v_heads, 64, 64, 64, true, is_bf16)) != QLA_OK) return rc;
  if ((rc = make_tmap_halves(&tm_h, p.h, state_rows, 1, 128, is_bf16)) != QLA_OK) return rc;
  if ((rc = make_tmap_halves(&tm_dh, p.dh, state_rows, 1, 128, is_bf16)) != QLA_OK) return rc;
  if ((rc = make_tmap_3d(&tm_du, p.du, state_rows, 1, kChunk, 128, 64, true, is_bf16)) != QLA_OK) return rc;
  if ((rc = make_tmap_halves(&tm_dq, p.dq, total_tokens, p.num_k_heads, 64, is_bf16)) != QLA_OK) return rc;
  if ((rc = make_tmap_halves(&tm_dk, p.dk, total_tokens, p.num_k_heads, 64, is_bf16)) != QLA_OK) return rc;
  if ((rc = make_tmap_halves(&tm_dv, p.dv, total_tokens, p.num_v_heads, 64, is_bf16)) != QLA_OK) return rc;
  const int total_items = total_chunks_upper * p.num_k_heads;
  int dev = 0, sms = 0;
  QLA_CHECK_CUDA(cudaGetDevice(&dev));
  QLA_CHECK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const unsigned grid = static_cast<unsigned>(total_items < sms ? total_items : sms);
#define QLA_LAUNCH_BWD_CHUNK(T, TR)                                                                         \
  do {                                                                                                     \
    if ((rc = ensure_dynamic_smem<bwd_chunk_kernel<T, TR>>(kSmemBytes)) != QLA_OK) return rc;              \
    QLA_CHECK_CUDA(launch_dependent(bwd_chunk_kernel<T, TR>, dim3(grid), dim3(kThreads), kSmemBytes, stream, tm_q, tm_k, tm_v, \
                                    tm_vn, tm_do, tm_a, tm_h, tm_dh, tm_du, tm_dq, tm_dk, tm_dv, p, total_items)); \
  } while (0)
  const bool traced = p.trace != nullptr;
  if (is_bf16) {
    if (traced) QLA_LAUNCH_BWD_CHUNK(__nv_bfloat16, true); else QLA_LAUNCH_BWD_CHUNK(__nv_bfloat16, false);
  } else {
    if (traced) QLA_LAUNCH_BWD_CHUNK(__half, true); else QLA_LAUNCH_BWD_CHUNK(__half, false);
  }
#undef QLA_LAUNCH_BWD_CHUNK
  QLA_CHECK_CUDA(cudaGetLastError());
  return QLA_OK;
}

void launch_info_bwd_chunk_kernel(int* block_threads, size_t* dynamic_smem_bytes) {
  *block_threads = kThreads;
  *dynamic_smem_bytes = kSmemBytes;
}

}  // namespace qla
