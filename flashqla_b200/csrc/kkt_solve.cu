// Chunk preparation for the prefill path: chunk-local cumulative gates and the gated WY matrix
//   A = (I + StrictLower(diag(beta) * (G .* K K^T)))^-1,   G[c,d] = exp(g_c - g_d),
// one 64x64 unit-lower-triangular inverse per (chunk, v-head), stored in the input dtype as
// A[token, v-head, 64].  Reference: chunk_local_cumsum (flash_qla/ops/utils/cumsum.py:17-168) and
// kkt_solve (chunk/hopper/kkt_solve.py:18-342; the gated form is chunk/blackwell/kkt_solve.py:118-136
// and tests/ref_gdr.py:42-104).  It also produces, per v-head, the chunk operand
//   Wt = A diag(beta gamma) K      (the "w" of tests/ref_gdr.py:107-147, stored negated)
// that lets the scan kernel form Vd = A diag(beta) V - Wt S0 with a single state-dependent product.
//
// Persistent CTAs of 128 threads walk items of 128 consecutive tokens (two chunks) x the v-heads of a k-head.  Two warps own a
// chunk: warp 2 ci + part has rows 32 part .. + 31, which are its tensor-memory quadrant; the two chunks share the K tile
// and run independently.  K K^T is one tcgen05 product per chunk, of whose M = 128 rows only the chunk's own lanes are written.
// Per head, in 16 x 16 blocks of N = -L and X = (I + L)^-1, kept as fragments of mma.sync:
//   1  N from K K^T and the gates; the two diagonal blocks of a warp are inverted by fp32 forward substitution, one per
//      half-warp, lane = column
//   2  X10 = X11 N10 X00 and X32 = X33 N32 X22: split TF32 products, to fp32 precision
//   3  X[2:4][0:2] = X[2:4][2:4] N[2:4][0:2] X[0:2][0:2]: TF32 products, one block column per warp
//   4  Wt = (-A diag(beta gamma)) K: a tcgen05 product, read back and stored through a swizzled tile (TMA); for a scan that forms
//      Wt itself its operand is stored instead, and A diag(beta) in place of A
// A product of three factors stays in registers: with T^T as the accumulator of the first product, its fragments ARE the B
// fragments of the second, because k may be numbered as one likes (slot c stands for k = 2c, slot c + 4 for 2c + 1).  Every
// block leaves as soon as its warp has it, in both 16-bit forms, by stmatrix.  Beside the chain the part 0 warp forms the
// next head's gates, and the next item's K is in L2 when it starts and in shared memory when this one has been multiplied.
//
// What bounds it: the writes (402 of 536 MB for 32768 tokens, 32 v-heads; without any arithmetic they take 102 us) and, beside them,
// a chain of dependent phases of some 1700 instructions per warp and head, 7 cycles each with three CTAs per SM.  Two warps per chunk
// instead of four, 16 x 16 blocks whose substitution does not waste half of its lanes, products in registers instead of through
// shared memory and items in a loop: 10.1 k -> 7.0 k warp instructions per 128 tokens and head, 32768 tokens of 16 / 32 heads
// 184 -> 140 us, 540 k packed tokens of 8 / 8 heads 836 -> 584, 32768 of 32 / 32 heads 197 -> 154.  Four warps per chunk (the emission of
// blocks and the gates on the other two): 161 us, with 9.0 k instructions.
#include <algorithm>
#include <cmath>

#include "chunk_params.cuh"

namespace qla {


namespace {

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

// Single TF32 in the last level, like the reference's fp32-tile gemm there (chunk/hopper/kkt_solve.py:181-183): against an
// fp64 inverse the error of that block is 1.70e-3 relative rms instead of 1.68e-3 with 3xTF32 (the 16-bit rounding of A
// dominates both), and o / final state do not move in the fourth digit.  The level below would lose precision by it.

// A 16 x 16 block of floats, element (r, col) at 16 r + (col ^ swz(r)): conflict-free for float2 fragments and for single values
// by lane = column.  17 rows from block to block: the two half-warps that invert neighbouring blocks read other banks.
constexpr int kBlock = 17 * 16;
__device__ __forceinline__ constexpr int swz(int r) { return ((r & 2) << 2) | (r & 4); }

// ---- shared memory (offsets from a 1024-byte aligned base): the K tile of both chunks, 32 KiB, as two [128][64] halves (columns
// 0..63 | 64..127), SW128; then per chunk
struct Area {
  static constexpr uint32_t kAw = 0;    // 8 KiB: -A diag(beta gamma), 16 bit, [64][64] SW128; kW: later columns 0..63 of Wt
  static constexpr uint32_t kX = 8192;  // 6 fp32 blocks X00, X11, X10, X22, X33, X32; later (8 KiB) A, 16 bit, [64][64] SW128;
                                        // kW: later columns 64..127 of Wt
  static constexpr uint32_t kN = kX + 6 * kBlock * 4;  // 4 blocks N20, N21, N30, N31 as fragments [s][lane] float4, TF32
  static constexpr uint32_t kBytes = kX + 11264;
  static constexpr size_t kSmem = 32768 + 2 * kBytes, kSmemOver = 2 * kBytes;  // (kOver: the K tile lies where the areas are)
  static_assert(kN + 4096 <= kBytes && kBytes % 1024 == 0, "shared-memory map");
};
constexpr int kCtasPerSm = 3, kCtasPerSmOver = 4;
constexpr int kKktThreads = 128;

// Fragments of a block, one array for all uses: value e of the pair [s][h] of lane 4 g + c is element (g + 8 h, 8 s + 2 c + e), which
// is the accumulator of two m16n8 products, the A operand of two k-steps and (of the transposed block) their B operand, if slot
// c of a k-step stands for k = 2 c and slot c + 4 for 2 c + 1.
using Frag = F2[2][2];  // [s][h]
// What a lane needs to know to find its values: element offsets in a block, and its address in a 16-bit tile.
struct LaneMap {
  int n;        // 16 g + (2 c ^ swz(g))
  int t;        // 32 c + (g ^ swz(2 c))
  uint32_t at;  // stmatrix: row lane % 16, 16-byte piece lane / 16 of a swizzled tile
  __device__ explicit LaneMap(int lane) {
    const int g = lane >> 2, c = lane & 3;
    n = 16 * g + ((2 * c) ^ swz(g));
    t = 32 * c + (g ^ swz(2 * c));
    at = ptx::sw128_offset(lane & 15, lane >> 4);
  }
  // ... of block (R, C) of a tile (the two bits that C and the lane put into the piece's number do not meet)
  __device__ __forceinline__ uint32_t tile(int R, int C) const { return (at ^ (C << 5)) + R * 2048; }
};
__device__ __forceinline__ void load_n(Frag& f, const float* blk, const LaneMap& m) {
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int h = 0; h < 2; ++h) f[s][h] = *reinterpret_cast<const F2*>(blk + (m.n ^ (8 * s)) + 128 * h);
}
__device__ __forceinline__ void load_t(Frag& f, const float* blk, const LaneMap& m) {  // of the transposed block
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float* x = blk + (m.t ^ (8 * h)) + 128 * s;
      f[s][h] = f2(x[0], x[16]);
    }
}
__device__ __forceinline__ void store_n(float* blk, const Frag& f, const LaneMap& m) {
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int h = 0; h < 2; ++h) *reinterpret_cast<F2*>(blk + (m.n ^ (8 * s)) + 128 * h) = f[s][h];
}
__device__ __forceinline__ void load_f(Frag& f, const float* frag, int lane) {
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(frag + 128 * s + 4 * lane);
    f[s][0] = x.x;
    f[s][1] = x.y;
  }
}
__device__ __forceinline__ void clear(Frag& f) { f[0][0] = f[0][1] = f[1][0] = f[1][1] = 0; }
__device__ __forceinline__ F2 cut_tf32(F2 x) { return x & 0xffffe000ffffe000ull; }
// Rounded to TF32 (11 significant bits), to nearest, ties away from zero, two values per instruction: the part behind the
// cut, added once more, carries where it is half a unit or more.  (cvt.rna.tf32.f32 takes 22 cycles and the time of
// four instructions; Veltkamp's splitting takes one instruction less than this, 482 instead of 498 us for 540 k packed tokens
// of 8 / 8 heads, but makes NaN of values beyond 4e34.)
__device__ __forceinline__ F2 nearest_tf32(F2 x) { return cut_tf32(add2(x, fma2(cut_tf32(x), f2(-1.f, -1.f), x))); }
__device__ __forceinline__ void round_tf32(Frag& f) {
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int h = 0; h < 2; ++h) f[s][h] = nearest_tf32(f[s][h]);
}
// acc += A B^T for fragments of A and B that hold TF32 values.
__device__ __forceinline__ void product_tf32(Frag& acc, const Frag& a, const Frag& b) {
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int t = 0; t < 2; ++t)
      asm("{\n.reg .b32 a0, a1, a2, a3, b0, b1;\n.reg .f32 c0, c1, c2, c3;\n"
          "mov.b64 {a0, a2}, %2;\nmov.b64 {a1, a3}, %3;\nmov.b64 {b0, b1}, %4;\nmov.b64 {c0, c1}, %0;\nmov.b64 {c2, c3}, %1;\n"
          "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {c0, c1, c2, c3}, {a0, a1, a2, a3}, {b0, b1}, {c0, c1, c2, c3};\n"
          "mov.b64 %0, {c0, c1};\nmov.b64 %1, {c2, c3};\n}\n"
          : "+l"(acc[t][0]), "+l"(acc[t][1]) : "l"(a[s][0]), "l"(a[s][1]), "l"(b[s][t]));
}
// A B^T of fp32 operands, to fp32 precision: each as a sum of two TF32 values (the upper one rounded to nearest, so that the
// lower one, which has 12 bits, is cut by one: 2^-23 of the operand), the product of the small parts left out (2^-24).
__device__ __forceinline__ void split_tf32(const Frag& x, Frag& hi, Frag& lo) {
  const F2 minus = f2(-1.f, -1.f);
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      hi[s][h] = nearest_tf32(x[s][h]);
      lo[s][h] = cut_tf32(fma2(hi[s][h], minus, x[s][h]));
    }
}
__device__ __forceinline__ void product_3xtf32(Frag& out, const Frag& a, const Frag& b) {
  Frag ah, al, bh, bl, small;
  split_tf32(a, ah, al);
  split_tf32(b, bh, bl);
  clear(out);
  clear(small);
  product_tf32(out, ah, bh);
  product_tf32(small, al, bh);
  product_tf32(small, ah, bl);
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int h = 0; h < 2; ++h) out[s][h] = add2(out[s][h], small[s][h]);
}
// A finished block, as 16-bit registers for the A tile: A, or with `beta` A diag(beta), the product of the rounded A rounded once
// more, as a scan that reads A forms it.  -A diag(beta gamma) goes to its tile (`aw_at` is this lane's stmatrix address there).
// bg, beta: factors of the block's columns.
template <typename T, bool kBeta>
__device__ __forceinline__ void emit(uint32_t (&av)[4], uint32_t aw_at, const Frag& f, const float* bg, const float* beta, int lane) {
  uint32_t aw[4];
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const F2 b = *reinterpret_cast<const F2*>(bg + 8 * s + 2 * (lane & 3));
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float lo, hi;
      unpack(mul2(f[s][h], b), lo, hi);
      aw[2 * s + h] = pack2<T>(lo, hi);
      unpack(f[s][h], lo, hi);
      av[2 * s + h] = pack2<T>(lo, hi);
      if (kBeta) {
        const T* a = reinterpret_cast<const T*>(&av[2 * s + h]);
        const float2 b2 = *reinterpret_cast<const float2*>(beta + 8 * s + 2 * (lane & 3));
        av[2 * s + h] = pack2<T>(Cvt<T>::to_f32(a[0]) * b2.x, Cvt<T>::to_f32(a[1]) * b2.y);
      }
    }
  }
  ptx::stmatrix_x4(aw_at, aw[0], aw[1], aw[2], aw[3]);
}
__device__ __forceinline__ void chunk_sync(int ci) {  // the two warps that own one chunk
  asm volatile("bar.sync %0, 64;" ::"r"(ci + 1) : "memory");
}

// kW: A and w are written.  Otherwise A diag(beta) and -A diag(beta gamma), for a scan that forms Wt from it.
// kOver (not with kW or the norms, which read the K tile later): an item's K tile lies where the two chunks' areas are, which nothing uses before
// K K^T.  The next item's K comes when both chunks are through with this one, which exposes its latency (about 1 us of 6 to 12), and four
// CTAs are resident instead of three: 32768 tokens of 16 / 32 heads 114 -> 105 us, 540 k packed tokens of 8 / 8 heads 510-524 -> 482 (with five, 91
// registers, 133 and 600).
template <typename T, bool kW, bool kOver>
__global__ void __launch_bounds__(kKktThreads, kOver ? kCtasPerSmOver : kCtasPerSm) kkt_solve_kernel(const __grid_constant__ CUtensorMap tm_k,
                                                                                   const __grid_constant__ CUtensorMap tm_q,
                                                                                   const __grid_constant__ CUtensorMap tm_a,
                                                                                   const __grid_constant__ CUtensorMap tm_w,
                                                                                   const KktParams p) {
  grid_dep_wait();    // earlier kernels of the stream have completed (see launch_dependent)
  grid_dep_launch();  // the next one may be scheduled; it waits the same way
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int group = p.num_v_heads / p.num_k_heads;
  // Warps 2 ci, 2 ci + 1 own chunk ci: rows 0..31 (part 0) and 32..63 (part 1), which are their tensor-memory quadrants.  The
  // two chunks of a CTA share the K tile and run independently of each other.
  const int ci = warp >> 1, part = warp & 1;

  // ---- work items: 128 tokens x (some of) the v-heads of a k-head.  Heads vary fastest: CTAs that run together read and write
  // the same rows.
  const unsigned columns = static_cast<unsigned>(p.num_k_heads * p.head_splits);
  const unsigned total_items = columns * static_cast<unsigned>(p.cu_seqlens != nullptr ? p.pair_offsets[p.num_seqs] : p.num_pairs);
  struct Item {
    int tok0, t0, valid;  // first token, first token of the chunk and number of its tokens (<= 0: there is no such chunk)
    int hk, hv0, hv1, split;
  };
  __shared__ Item s_item[2][2];  // [turn][chunk]: this item and the next
  int pair = static_cast<int>(blockIdx.x / columns), column = static_cast<int>(blockIdx.x % columns);
  const int step_pair = static_cast<int>(gridDim.x / columns), step_column = static_cast<int>(gridDim.x % columns);
  auto locate = [&]() {
    Item x;
    x.hk = p.head_splits == 1 ? column : column / p.head_splits;
    x.split = column - x.hk * p.head_splits;
    x.hv0 = x.hk * group + x.split * p.heads_per_cta;
    x.hv1 = min(x.hv0 + p.heads_per_cta, (x.hk + 1) * group);
    int seq_end;
    if (p.cu_seqlens != nullptr) {
      // the last sequence that starts at or before this pair, 32 candidates at a time
      int lo = 0, hi = p.num_seqs - 1;
      while (hi > lo) {
        const int step = (hi - lo) / 32 + 1, at = lo + lane * step;
        const bool below = at <= hi && p.pair_offsets[at] <= pair;
        const int last = __popc(__ballot_sync(0xffffffffu, below)) - 1;
        hi = min(hi, lo + last * step + step - 1);
        lo += last * step;
      }
      seq_end = p.cu_seqlens[lo + 1];
      x.tok0 = p.cu_seqlens[lo] + (pair - p.pair_offsets[lo]) * 128;
    } else {
      const int per_seq = (p.seq_len + 127) / 128;
      const int b = p.num_seqs == 1 ? 0 : pair / per_seq;
      seq_end = (b + 1) * p.seq_len;
      x.tok0 = b * p.seq_len + (pair - b * per_seq) * 128;
    }
    x.t0 = x.tok0 + ci * kChunk;
    x.valid = min(kChunk, seq_end - x.t0);
    return x;
  };
  if (blockIdx.x >= total_items) return;

  extern __shared__ __align__(1024) uint8_t smem[];  // (the compiler pads what is in front of it to that alignment)
  using M = Area;
  constexpr int kTmemColumns = kW ? 128 : 64;  // K K^T, and Wt over it
  static_assert(!kOver || !kW, "Wt is formed from the K tile");
  uint8_t *sK = smem, *area = smem + (kOver ? 0 : 32768) + ci * M::kBytes;
  float* sX = reinterpret_cast<float*>(area + M::kX);
  float* sN = reinterpret_cast<float*>(area + M::kN);
  // exponents (log2) of L: -L[c][d] = -sign(beta_c) (k_c . k_d) 2^(row[c] + col[d]); the sign is that of beta
  struct alignas(16) Gates {
    float row[64];  // g log2(e) + log2(|beta| / |k_c|)
    float col[64];  // -(g log2(e)) - log2 |k_d|     (|k| = 1 without in-kernel norm)
    float bg[64];   // -beta * gamma
    float beta[kW ? 4 : 64];  // (kW: not used)
  };
  constexpr int kGateBuffers = kW ? 2 : 1;
  __shared__ Gates s_gates[2][kGateBuffers];  // of the two chunks; kW: the head's and the next one's
  __shared__ uint64_t bar_k, bar_q, bar_kk[2], bar_w[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ unsigned k_released;  // times that a chunk was through with what the K tile holds
  const bool norm = !kOver && p.rnorm != nullptr;

  auto load_k = [&](const Item& x) {
    ptx::mbar_expect_tx(&bar_k, 32768);
    ptx::tma_load_4d(sK, &tm_k, &bar_k, 0, x.hk, x.tok0, 0);
  };
  // Q is only wanted for its row norms.  Its tile visits the memory of the K tile when that has been multiplied, and (kW) with a
  // CTA's first item both chunks' areas, which nothing uses yet: one short prompt does not wait for a second copy.
  auto load_q = [&](const Item& x, uint8_t* to) {
    ptx::mbar_expect_tx(&bar_q, 32768);
    ptx::tma_load_4d(to, &tm_q, &bar_q, 0, x.hk, x.tok0, 0);
  };
  if (tid == 0) {
    ptx::mbar_init(&bar_k, 1);
    ptx::mbar_init(&bar_q, 1);
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      ptx::mbar_init(&bar_kk[x], 1);
      ptx::mbar_init(&bar_w[x], 1);
    }
    ptx::fence_mbar_init();
    ptx::mbar_wait_setup(p.status, &bar_k, 0);
    k_released = 0;
  }
  // Gates: the part 0 warp of a chunk, two tokens per lane.  They are requested and activated one head ahead, and made public
  // when 1 / |k| is known too.
  float gv[2], bv[2], gin[2], lrk[2] = {0.f, 0.f};  // lrk: log2 of 1 / |k_t|
  auto fetch_gates = [&](const Item& x, int hv) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      gv[r] = bv[r] = gin[r] = 0.f;
      if (lane + 32 * r >= x.valid) continue;
      const int64_t idx = (static_cast<int64_t>(x.t0) + lane + 32 * r) * p.num_v_heads + hv;
      bv[r] = load_scalar(p.beta, p.beta_dtype, idx);
      if (p.A_in != nullptr) gin[r] = p.g_cumsum[idx];
      else gv[r] = load_scalar(p.g, p.gate_dtype, idx);
    }
  };
  float gc2[2];  // cumulative log decay, in log2
  auto activate = [&](const Item& x, int hv) {
    float sum[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const bool in = lane + 32 * r < x.valid;
      if (in && p.beta_out != nullptr) {  // logits in: the activated value is what every later stage reads
        bv[r] = 1.f / (1.f + __expf(-bv[r]));
        p.beta_out[(static_cast<int64_t>(x.t0) + lane + 32 * r) * p.num_v_heads + hv] = bv[r];
      }
      if (in && p.A_log != nullptr) {  // gate activation of the layer (recurrent op: recurrent_fused.py:346-487)
        const float y = gv[r] + p.dt_bias[hv];
        gv[r] = -expf(p.A_log[hv]) * (y <= 20.f ? log1pf(expf(y)) : y);
      }
      sum[r] = gv[r];
    }
#pragma unroll
    for (int off = 1; off < 32; off <<= 1)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float n = __shfl_up_sync(0xffffffffu, sum[r], off);
        if (lane >= off) sum[r] += n;
      }
    sum[1] += __shfl_sync(0xffffffffu, sum[0], 31);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int t = lane + 32 * r;
      if (p.A_in != nullptr) sum[r] = gin[r];  // gates are cumulative already
      else if (t < x.valid) p.g_cumsum[(static_cast<int64_t>(x.t0) + t) * p.num_v_heads + hv] = sum[r];
      gc2[r] = sum[r] * 1.4426950408889634f;  // exponents are formed in the log2 domain
    }
  };
  auto publish = [&](Gates& gt) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int t = lane + 32 * r;
      const float er = gc2[r] + (ptx::lg2(fabsf(bv[r])) + lrk[r]);  // (beta = 0: -inf, every power below is 0)
      gt.row[t] = er;
      gt.col[t] = lrk[r] - gc2[r];
      gt.bg[t] = copysignf(ptx::ex2(er), -bv[r]);
      if (!kW) gt.beta[t] = bv[r];
    }
  };
  if (part == 0) {
    const Item first = locate();
    if (lane == 0) {
      s_item[0][ci] = first;
      if (ci == 0) {
        load_k(first);
        if (kW && norm && first.split == 0) load_q(first, smem + 32768);
      }
    }
    fetch_gates(first, first.hv0);
    activate(first, first.hv0);
    if (!norm) publish(s_gates[ci][0]);
  }
  if (warp == 1) {
    ptx::tmem_alloc(&tmem_base_s, kTmemColumns);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem = tmem_base_s;
  const uint32_t a_k = ptx::smem_u32(&bar_k), a_q = ptx::smem_u32(&bar_q), a_kk = ptx::smem_u32(&bar_kk[ci]), a_w = ptx::smem_u32(&bar_w[ci]);
  const uint32_t quad = tmem + (static_cast<uint32_t>(warp * 32) << 16);
  constexpr uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? ptx::kFmtBF16 : ptx::kFmtF16;

  const uint32_t low_off = ci == 0 ? 0u : ~0u, high_off = ~low_off;  // lanes that are not this chunk's
  const LaneMap lm(lane);
  int uses = 0;  // phases of bar_w waited for
  int kk_turn = 0;  // and the parity of bar_kk's next one
  int buf = 0;   // buffer of the gates
  int q_turn = 0;  // parity of bar_q's next phase
#pragma unroll 1
  for (unsigned item = blockIdx.x, turn = 0; item < total_items; item += gridDim.x, turn ^= 1) {
  const bool more = item + gridDim.x < total_items;
  const Item &cur = s_item[turn][ci], &nxt = s_item[turn ^ 1][ci];
  // The next item (for the warp that forms the gates): its K tile goes to L2 now and to shared memory as soon as this item's
  // last product has read K.
  auto locate_next = [&]() {
    if (!more) return;
    pair += step_pair;
    column += step_column;
    if (column >= static_cast<int>(columns)) {
      column -= static_cast<int>(columns);
      ++pair;
    }
    const Item x = locate();
    if (lane == 0) {
      s_item[turn ^ 1][ci] = x;
      if (ci == 0) {
        ptx::tma_prefetch_l2_4d(&tm_k, 0, x.hk, x.tok0, 0);
        if (norm && x.split == 0) ptx::tma_prefetch_l2_4d(&tm_q, 0, x.hk, x.tok0, 0);
      }
    }
    __syncwarp();
  };
  // One thread per chunk says when the chunk is through with K (after its last product); the second one to do so loads the next
  // item's.  With the norms the Q tile visits the same memory in between, and each chunk says so a second time.
  // kOver: both chunks' products have read the K tile
  auto cta_sync = [&]() { asm volatile("bar.sync 3, 128;" ::: "memory"); };
  const bool q_first = kW && norm && cur.split == 0 && item == blockIdx.x, q_norms = norm && cur.split == 0 && !q_first;
  auto release_k = [&]() {
    unsigned before;
    asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;" : "=r"(before) : "r"(ptx::smem_u32(&k_released)) : "memory");
    if (before == 1 && q_norms) load_q(cur, sK);
    if (before == (q_norms ? 3 : 1)) {
      k_released = 0;
      if (more) load_k(nxt);
    }
  };
  auto row_norm = [&](const uint8_t* tile) {  // 1 / |row tid|: half rows, then their sum
    float sum[2] = {0.f, 0.f};
#pragma unroll
    for (int half = 0; half < 2; ++half) {
#pragma unroll 2
      for (int c16 = 0; c16 < 8; ++c16) {
        const uint4 raw = *reinterpret_cast<const uint4*>(tile + half * 16384 + ptx::sw128_offset(tid, c16));
        const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
        for (int x = 0; x < 8; ++x) sum[half] += Cvt<T>::to_f32(e[x]) * Cvt<T>::to_f32(e[x]);
      }
    }
    return rsqrtf(sum[0] + sum[1] + p.norm_eps);
  };
  // 1 / |q| of this item's rows, once Q has come to where K was; then the next item's K may come
  auto finish_q = [&](const uint8_t* tile) {
    if (ptx::mbar_wait_addr(a_q, q_turn)) {
      const float rq = row_norm(tile);
      if ((tid & 63) < cur.valid) p.rnorm[((static_cast<int64_t>(cur.tok0) + tid) * p.num_k_heads + cur.hk) * 2] = rq;
    }
    q_turn ^= 1;
    if (q_first) {
      __syncthreads();  // (the tile lies in both chunks' areas)
      return;
    }
    chunk_sync(ci);
    if (part == 0 && lane == 0) release_k();
  };
  const int t0 = cur.t0, valid = cur.valid, hv0 = cur.hv0, hv1 = cur.hv1;
  const int g = lane >> 2, c = lane & 3;
  const bool full = valid == kChunk;
  const uint32_t aw_tile = ptx::smem_u32(area + M::kAw), a_tile = ptx::smem_u32(area + M::kX);
  auto zero_above = [&](uint8_t* tile) {  // the blocks above the diagonal: (0, 1..3) part 0, (1, 2), (1, 3), (2, 3) part 1
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      const uint32_t at = part == 0 ? lm.tile(0, 1 + x) : lm.tile(1 + x / 2, x == 0 ? 2 : 3);
      *reinterpret_cast<uint4*>(tile + at) = make_uint4(0, 0, 0, 0);
    }
  };
  if (valid <= 0) {  // no second chunk: nothing to do but to get its next one under way
    if (part == 0) {
      locate_next();
      ptx::mbar_wait_addr(a_k, turn);  // (or two such items in a row would release the tile under the other chunk)
    }
    if (kOver) cta_sync();
    if (part == 0) {
      if (lane == 0) release_k();
      if (more) {
        fetch_gates(nxt, nxt.hv0);
        activate(nxt, nxt.hv0);
        if (!norm) publish(s_gates[ci][buf % kGateBuffers]);
      }
    }
    if (q_norms || q_first) finish_q(q_first ? smem + 32768 : sK);
    chunk_sync(ci);
  } else {
  // K K^T of this chunk (an M = 128 product with the rows of both chunks, of which only this chunk's lanes are written), read
  // again for every head or, with Wt in its place (kW), kept in registers: this warp's blocks (R, R), (R + 1, R + 1), (R + 1, R) with R = 2 part, and for part 1 (2, 0),
  // (2, 1), (3, 0), (3, 1).  Products are issued by a converged warp (one elected lane inside ptx::umma_*): operand arithmetic
  // then stays on the uniform datapath and an instruction costs its time on the tensor pipe.
  if (part == 1) {
    ptx::mbar_wait_addr(a_k, turn);
    ptx::tc_fence_after_sync();
    constexpr uint32_t idesc = ptx::mma_idesc(128, 64, fmt, ptx::kMajorK, ptx::kMajorK);
    const uint64_t d_k = ptx::smem_desc_sw128(ptx::smem_u32(sK), 16, 1024);
    ptx::umma_ss_k64_lanes<2, 2>(tmem, d_k, d_k + ci * (8192 >> 4), idesc, low_off, high_off, false);
    ptx::umma_ss_k64_lanes<2, 2>(tmem, d_k + (16384 >> 4), d_k + (16384 >> 4) + ci * (8192 >> 4), idesc, low_off, high_off, true, a_kk);
  } else {
    locate_next();
    if (!kOver && lane == 0) ptx::tma_store_wait_read();  // the last store has read its tiles
  }
  // In-kernel L2 norm of q and k (reference: l2norm before the kernels, flash_qla/utils/math.py:14-21 via
  // chunk/__init__.py:332-334): 1/sqrt(|row|^2 + eps), a row per thread.  Everything downstream uses the RAW tiles and
  // folds the factors in: K K^T[c][d] r_c r_d (in the exponents), r_k into beta gamma for w; the scan folds r_k
  // into rho, r_q into s gamma and both into Pg.
  if (norm) {
    Gates& gt = s_gates[ci][buf % kGateBuffers];
    if (ptx::mbar_wait_addr(a_k, turn)) {
      const float rk = row_norm(sK);
      gt.row[tid & 63] = ptx::lg2(rk);  // (for the warp that forms the gates)
      if ((tid & 63) < valid && cur.split == 0) p.rnorm[((static_cast<int64_t>(cur.tok0) + tid) * p.num_k_heads + cur.hk) * 2 + 1] = rk;
    }
    if (q_first) finish_q(smem + 32768);
    else chunk_sync(ci);
    if (part == 0) {
      lrk[0] = gt.row[lane];
      lrk[1] = gt.row[lane + 32];
      __syncwarp();
      publish(gt);
    }
  }
  chunk_sync(ci);
  ptx::mbar_wait_addr(a_kk, kk_turn);
  kk_turn ^= 1;
  if (kOver) cta_sync();
  ptx::tc_fence_after_sync();
  uint32_t kk_own[kW ? 3 : 1][8], kk_left[kW ? 4 : 1][8];
  const uint32_t high = quad + (16u << 16);
  if (kW) {
    ptx::tmem_ld_frag2(quad + part * 32, kk_own[0]);
    ptx::tmem_ld_frag2(high + part * 32 + 16, kk_own[kW ? 1 : 0]);
    ptx::tmem_ld_frag2(high + part * 32, kk_own[kW ? 2 : 0]);
    if (part == 1) {
#pragma unroll
      for (int x = 0; x < 4; ++x) ptx::tmem_ld_frag2(((x >> 1) ? high : quad) + 16 * (x & 1), kk_left[kW ? x : 0]);
    }
    ptx::tmem_wait_ld();
  } else if (!kOver && part == 0 && lane == 0) {
    release_k();
  }
#pragma unroll 1
  for (int hv = hv0; hv < hv1; ++hv, ++uses, buf ^= 1) {
    const Gates& gt = s_gates[ci][buf % kGateBuffers];
    const bool last = hv + 1 == hv1;
    if (part == 0 && (!last || more)) fetch_gates(last ? nxt : cur, last ? nxt.hv0 : hv + 1);
    // (not kW: activated early too, while the other warp forms N of four blocks more, but made public when this head's gates have been read)
    auto activate_next = [&]() {
      if (part == 0 && (!last || more)) activate(last ? nxt : cur, last ? nxt.hv0 : hv + 1);
    };
    auto publish_next = [&]() {
      if (part == 0 && (last ? more && !norm : true)) publish(s_gates[ci][(buf ^ 1) % kGateBuffers]);
    };
    if (hv > hv0) {  // the store of the previous head has read its tiles
      if (part == 0 && lane == 0) ptx::tma_store_wait_read();
      chunk_sync(ci);
    }
    uint32_t av[5][4];
    if (!kW || p.A_in == nullptr) {
      // ---- 1: blocks of N = -L = -beta_c exp(g_c - g_d) (k_c . k_d).  Entries on and above the diagonal are formed too; they may
      // overflow, but nothing reads them.
      float* own = sX + 3 * part * kBlock;
      Frag off;  // N of block (R + 1, R)
      {
        F2 er[2][2], sg[2][2];
#pragma unroll
        for (int rb = 0; rb < 2; ++rb)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int r = 32 * part + 16 * rb + 8 * h + g;
            const float e = gt.row[r], sign = copysignf(1.f, gt.bg[r]);  // -sign(beta)
            er[rb][h] = f2(e, e);
            sg[rb][h] = f2(sign, sign);
          }
        auto build = [&](Frag& n, const uint32_t (&kept)[8], int rb, int col0) {
          uint32_t x[8];
          if (kW) {
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = kept[i];
          } else {
            ptx::tmem_ld_frag2((rb ? high : quad) + col0, x);
          }
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            const F2 col = *reinterpret_cast<const F2*>(&gt.col[col0 + 8 * s + 2 * c]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              float lo, hi;
              unpack(add2(er[rb][h], col), lo, hi);
              n[s][h] = mul2(f2(ptx::ex2(lo), ptx::ex2(hi)), sg[rb][h]);
            }
          }
          if (!kW) ptx::tmem_wait_ld();
#pragma unroll
          for (int s = 0; s < 2; ++s)
#pragma unroll
            for (int h = 0; h < 2; ++h)
              n[s][h] = mul2(n[s][h], f2(__uint_as_float(x[4 * s + 2 * h]), __uint_as_float(x[4 * s + 2 * h + 1])));
        };
        Frag n;
        build(n, kk_own[0], 0, 32 * part);
        store_n(own, n, lm);
        build(n, kk_own[kW ? 1 : 0], 1, 32 * part + 16);
        store_n(own + kBlock, n, lm);
        build(off, kk_own[kW ? 2 : 0], 1, 32 * part);
        if (part == 1) {
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            build(n, kk_left[kW ? x : 0], x >> 1, 16 * (x & 1));
            round_tf32(n);
#pragma unroll
            for (int s = 0; s < 2; ++s)
              *reinterpret_cast<ulonglong2*>(sN + 256 * x + 128 * s + 4 * lane) = make_ulonglong2(n[s][0], n[s][1]);
          }
        }
      }
      __syncwarp();
      {
        // the two diagonal blocks, one per half-warp: x_i = e_i + sum_j<i N_ij x_j, lane = column, two terms per instruction, even
        // and odd j in partial sums; the lanes of a half-warp read the same row of N.
        const int col = lane & 15;
        float* blk = own + (lane >> 4) * kBlock;
        F2 xp[8];
        float x_even = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          F2 acc = f2(i == col ? 1.f : 0.f, 0.f), acc_b = f2(0.f, 0.f);
          float tail = 0.f;  // N[i][i - 1], odd i
#pragma unroll
          for (int j4 = 0; j4 < i; j4 += 4) {
            const ulonglong2 l = *reinterpret_cast<const ulonglong2*>(blk + 16 * i + (j4 ^ swz(i)));
            float unused;
            if (j4 + 1 < i) acc = fma2(l.x, xp[j4 / 2], acc);
            else unpack(l.x, tail, unused);
            if (j4 + 3 < i) acc_b = fma2(l.y, xp[j4 / 2 + 1], acc_b);
            else if (j4 + 2 < i) unpack(l.y, tail, unused);
          }
          float lo, hi;
          unpack(add2(acc, acc_b), lo, hi);
          const float x = (i & 1) ? fmaf(tail, x_even, lo + hi) : lo + hi;
          if (i & 1) xp[i / 2] = f2(x_even, x);
          else x_even = x;
        }
        __syncwarp();  // the blocks have been read
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float lo, hi;
          unpack(xp[i], lo, hi);
          blk[32 * i + (col ^ swz(2 * i))] = lo;
          blk[32 * i + 16 + (col ^ swz(2 * i + 1))] = hi;
        }
        __syncwarp();
      }
      if (!kW && q_norms && hv == hv0) finish_q(sK);  // (Q has been under way since K K^T)
      // ---- 2: X[R + 1][R] = X[R + 1][R + 1] N[R + 1][R] X[R][R]; the diagonal blocks leave beside it
      {
        const float *bg = &gt.bg[32 * part], *beta = &gt.beta[kW ? 0 : 32 * part];
        const int R = 2 * part;
        Frag d0t, d0, d1, t, y;
        load_t(d0t, own, lm);
        load_n(d1, own + kBlock, lm);
        load_n(d0, own, lm);
        product_3xtf32(t, d0t, off);  // T^T = X[R][R]^T N^T
        emit<T, !kW>(av[0], aw_tile + lm.tile(R, R), d0, bg, beta, lane);
        emit<T, !kW>(av[1], aw_tile + lm.tile(R + 1, R + 1), d1, bg + 16, beta + 16, lane);
        product_3xtf32(y, d1, t);
        store_n(own + 2 * kBlock, y, lm);
        emit<T, !kW>(av[2], aw_tile + lm.tile(R + 1, R), y, bg, beta, lane);
        if (kW || hv == hv0) zero_above(area + M::kAw);
        activate_next();
        if (kW) publish_next();
      }
      chunk_sync(ci);
      // ---- 3: column block m = part of the lower left quarter, X[2:4][m] = X[2:4][2:4] (N[2:4][0:2] X[0:2][m])
      {
        const float *bg = &gt.bg[16 * part], *beta = &gt.beta[kW ? 0 : 16 * part];
        Frag a, b2, b3, x22, x32, x33, t2, t3, y2, y3;
        load_t(a, sX + (part ? 1 : 2) * kBlock, lm);  // X11^T | X10^T
        load_f(b2, sN + 256, lane);
        load_f(b3, sN + 768, lane);
        load_n(x22, sX + 3 * kBlock, lm);
        load_n(x32, sX + 5 * kBlock, lm);
        load_n(x33, sX + 4 * kBlock, lm);
        clear(t2);
        clear(t3);
        round_tf32(a);
        product_tf32(t2, a, b2);  // T_j^T = X[0:2][m]^T N[j][0:2]^T, j = 2, 3
        product_tf32(t3, a, b3);
        if (part == 0) {
          load_t(a, sX, lm);  // X00^T
          load_f(b2, sN, lane);
          load_f(b3, sN + 512, lane);
          round_tf32(a);
          product_tf32(t2, a, b2);
          product_tf32(t3, a, b3);
        }
        round_tf32(x22);
        round_tf32(x32);
        round_tf32(x33);
        round_tf32(t2);
        round_tf32(t3);
        clear(y2);
        clear(y3);
        product_tf32(y2, x22, t2);
        product_tf32(y3, x32, t2);
        product_tf32(y3, x33, t3);
        emit<T, !kW>(av[3], aw_tile + lm.tile(2, part), y2, bg, beta, lane);
        emit<T, !kW>(av[4], aw_tile + lm.tile(3, part), y3, bg, beta, lane);
      }
    } else {
      // A comes from an earlier call: a row per thread (what lies in its upper right quarter is not looked at)
      const int row = 32 * part + lane;
      const T* arow = static_cast<const T*>(p.A_in) + ((static_cast<int64_t>(t0) + row) * p.num_v_heads + hv) * 64;
#pragma unroll 1
      for (int j = 0; j < 64; j += 8) {
        const uint4 raw = row < valid && (j < 32 || part == 1) ? *reinterpret_cast<const uint4*>(arow + j) : make_uint4(0, 0, 0, 0);
        const T* e = reinterpret_cast<const T*>(&raw);
        uint32_t aw[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const float* bg = &gt.bg[j + 2 * x];
          aw[x] = pack2<T>(Cvt<T>::to_f32(e[2 * x]) * bg[0], Cvt<T>::to_f32(e[2 * x + 1]) * bg[1]);
        }
        *reinterpret_cast<uint4*>(area + M::kAw + ptx::sw128_offset(row, j >> 3)) = make_uint4(aw[0], aw[1], aw[2], aw[3]);
      }
      activate_next();
      publish_next();
    }
    ptx::fence_proxy_async_smem();
    ptx::tc_fence_before_sync();
    chunk_sync(ci);  // the operand tile is complete, the fp32 blocks have been read
    // ---- 4: Wt = (-A diag(beta gamma)) K.  An M = 128 product over the operand tiles of both chunks, of which only this
    // chunk's 64 lanes are written: a row of Wt then lies in the quadrant of the warp that owns it (M = 64 would
    // spread a chunk over all four).
    if (kW && part == 1) {
      ptx::tc_fence_after_sync();
      constexpr uint32_t idesc = ptx::mma_idesc(128, 128, fmt, ptx::kMajorK, ptx::kMajorMN);
      const uint64_t da = ptx::smem_desc_sw128(aw_tile - ci * 8192u, 16, 1024);
      const uint64_t db = ptx::smem_desc_sw128(ptx::smem_u32(sK) + ci * 8192u, 16384, 1024);
      ptx::umma_ss_k64_lanes<2, 128>(tmem, da, db, idesc, low_off, high_off, false, a_w);
    }
    if (!kW) {
      if (full && part == 0 && lane == 0) {
        ptx::tma_store_3d(&tm_w, area + M::kAw, 0, hv, t0);
        ptx::tma_store_commit();
      }
      __syncwarp();
      publish_next();
    }
    if (!kW || p.A_in == nullptr) {
      const int R = 2 * part;
      auto put = [&](int r, int col, const uint32_t (&x)[4]) { ptx::stmatrix_x4(a_tile + lm.tile(r, col), x[0], x[1], x[2], x[3]); };
      put(R, R, av[0]);
      put(R + 1, R + 1, av[1]);
      put(R + 1, R, av[2]);
      put(2, part, av[3]);
      put(3, part, av[4]);
      zero_above(area + M::kX);
      ptx::fence_proxy_async_smem();
      chunk_sync(ci);
      if (full) {
        if (part == 0 && lane == 0) {
          ptx::tma_store_3d(&tm_a, area + M::kX, 0, hv, t0);
          ptx::tma_store_commit();
        }
      } else {  // ragged tail: the next sequence owns the rows behind it
        const int64_t first = (static_cast<int64_t>(t0) * p.num_v_heads + hv) * 64;
        for (int x = 32 * part + lane; x < valid * 8; x += 64) {
          const int64_t to = first + static_cast<int64_t>(x >> 3) * p.num_v_heads * 64 + (x & 7) * 8;
          const uint32_t from = ptx::sw128_offset(x >> 3, x & 7);
          *reinterpret_cast<uint4*>(static_cast<T*>(p.A) + to) = *reinterpret_cast<const uint4*>(area + M::kX + from);
          if (!kW) *reinterpret_cast<uint4*>(static_cast<T*>(p.aw) + to) = *reinterpret_cast<const uint4*>(area + M::kAw + from);
        }
        chunk_sync(ci);  // (the tile is overwritten)
      }
    }
    if (!kW) continue;
    ptx::mbar_wait_addr(a_w, uses & 1);  // (a wait that gives up is reported there)
    ptx::tc_fence_after_sync();
    if (last && part == 0 && lane == 0) release_k();
    // a row of Wt per thread, into the swizzled tiles of the two halves: columns 0..63 over the operand, 64..127 over the A tile
    const uint32_t row_at = ptx::sw128_offset(32 * part + lane, 0);
#pragma unroll 1
    for (int kb = 0; kb < 128; kb += 32) {
      uint32_t r[32];
      ptx::tmem_ld32(quad + kb, r);
      ptx::tmem_wait_ld();
      if (kb == 64) {
        if (part == 0 && lane == 0) ptx::tma_store_wait_read();  // the A tile has been read
        chunk_sync(ci);
      }
      const uint32_t to = row_at + (kb >> 6) * 8192;
#pragma unroll
      for (int e = 0; e < 32; e += 8)
        *reinterpret_cast<uint4*>(area + M::kAw + (to ^ ((((kb & 32) + e) >> 3) << 4))) =
            make_uint4(pack2<T>(__uint_as_float(r[e]), __uint_as_float(r[e + 1])),
                       pack2<T>(__uint_as_float(r[e + 2]), __uint_as_float(r[e + 3])),
                       pack2<T>(__uint_as_float(r[e + 4]), __uint_as_float(r[e + 5])),
                       pack2<T>(__uint_as_float(r[e + 6]), __uint_as_float(r[e + 7])));
    }
    ptx::fence_proxy_async_smem();
    ptx::tc_fence_before_sync();
    chunk_sync(ci);
    if (full) {
      if (part == 0 && lane == 0) {
        ptx::tma_store_4d(&tm_w, area + M::kAw, 0, hv, t0, 0);
        ptx::tma_store_commit();
      }
    } else {
      T* wrow = static_cast<T*>(p.w) + (static_cast<int64_t>(t0) * p.num_v_heads + hv) * kHeadDim;
      for (int x = 32 * part + lane; x < valid * 16; x += 64)
        *reinterpret_cast<uint4*>(wrow + static_cast<int64_t>(x >> 4) * p.num_v_heads * kHeadDim + (x & 15) * 8) =
            *reinterpret_cast<const uint4*>(area + M::kAw + (x & 8) * 1024 + ptx::sw128_offset(x >> 4, x & 7));
    }
  }
  if (kOver) {  // the areas are free for the next K when both chunks say so (their writes are fenced above)
    if (part == 0 && lane == 0) ptx::tma_store_wait_read();
    chunk_sync(ci);
    if (part == 0 && lane == 0) release_k();
  }
  }  // valid
  if (kW && valid > 0 && q_norms) finish_q(sK);
  }  // items

  if (part == 0 && lane == 0) ptx::tma_store_wait_read();  // shared memory stays allocated until the last stores have read it
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) ptx::tmem_dealloc(tmem, kTmemColumns);
}

// pair_offsets[n] = sum_{m<n} ceil(len_m / 128), chunk_offsets[n] = sum_{m<n} ceil(len_m / 64): one warp, 32
// sequences at a time (a single thread took 80 ns per sequence).
__global__ void chunk_tables_kernel(const int32_t* cu, int n, int32_t* pair_offsets, int32_t* chunk_offsets) {
  grid_dep_wait();
  grid_dep_launch();
  const int lane = threadIdx.x;
  int po = 0, co = 0;
  for (int i0 = 0; i0 < n; i0 += 32) {
    const int i = i0 + lane;
    const int len = i < n ? cu[i + 1] - cu[i] : 0;
    int p = (len + 127) / 128, c = (len + 63) / 64;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int pn = __shfl_up_sync(0xffffffffu, p, off), cn = __shfl_up_sync(0xffffffffu, c, off);
      if (lane >= off) {
        p += pn;
        c += cn;
      }
    }
    if (i < n) {
      pair_offsets[i + 1] = po + p;
      chunk_offsets[i + 1] = co + c;
    }
    po += __shfl_sync(0xffffffffu, p, 31);
    co += __shfl_sync(0xffffffffu, c, 31);
  }
  if (lane == 0) pair_offsets[0] = chunk_offsets[0] = 0;
}

}  // namespace

int launch_chunk_tables(const int32_t* cu, int n, int32_t* pair_offsets, int32_t* chunk_offsets,
                        cudaStream_t stream) {
  QLA_CHECK_CUDA(launch_dependent(chunk_tables_kernel, dim3(1), dim3(32), 0, stream, cu, n, pair_offsets, chunk_offsets));
  QLA_CHECK_CUDA(cudaGetLastError());
  return QLA_OK;
}

template <typename T, bool kW, bool kOver = false>
static int launch_kkt(const KktParams& p, const CUtensorMap& tm_k, const CUtensorMap& tm_q, const CUtensorMap& tm_a, const CUtensorMap& tm_w, unsigned grid,
                      cudaStream_t stream) {
  constexpr size_t smem = kOver ? Area::kSmemOver : Area::kSmem;
  const int rc = ensure_dynamic_smem<kkt_solve_kernel<T, kW, kOver>>(smem);
  if (rc != QLA_OK) return rc;
  QLA_CHECK_CUDA(launch_dependent(kkt_solve_kernel<T, kW, kOver>, dim3(grid), dim3(kKktThreads), smem, stream, tm_k, tm_q, tm_a, tm_w, p));
  QLA_CHECK_CUDA(cudaGetLastError());
  return QLA_OK;
}

int launch_kkt_solve(const KktParams& params, const void* k, const void* q, int64_t total_tokens, int pairs_upper, bool is_bf16, cudaStream_t stream) {
  KktParams p = params;
  const bool with_w = p.aw == nullptr;
  CUtensorMap tm_k, tm_q, tm_a, tm_w;
  int rc = make_tmap_halves(&tm_k, k, total_tokens, p.num_k_heads, 128, is_bf16);
  if (rc != QLA_OK) return rc;
  // q is only read for the in-kernel L2 norm (p.rnorm set); otherwise the map is made over k and unused
  rc = make_tmap_halves(&tm_q, p.rnorm != nullptr ? q : k, total_tokens, p.num_k_heads, 128, is_bf16);
  if (rc != QLA_OK) return rc;
  // A leaves through a [64 tokens][64] tile; in rebuild mode (A given) the map is made but unused
  rc = make_tmap_3d(&tm_a, p.A, total_tokens, p.num_v_heads, 64, kChunk, 64, true, is_bf16);
  if (rc != QLA_OK) return rc;
  rc = with_w ? make_tmap_halves(&tm_w, p.w, total_tokens, p.num_v_heads, kChunk, is_bf16)
              : make_tmap_3d(&tm_w, p.aw, total_tokens, p.num_v_heads, 64, kChunk, 64, true, is_bf16);
  if (rc != QLA_OK) return rc;
  const int group = p.num_v_heads / p.num_k_heads;
  int slots = 0, dev = 0;
  QLA_CHECK_CUDA(cudaGetDevice(&dev));
  QLA_CHECK_CUDA(cudaDeviceGetAttribute(&slots, cudaDevAttrMultiProcessorCount, dev));
  const bool over = !with_w && p.rnorm == nullptr;
  slots *= over ? kCtasPerSmOver : kCtasPerSm;
  // Work items: the v-heads of a k-head stay together, which reads K once, unless the rounds of resident CTAs come out shorter
  // with fewer heads per item.  Getting an item under way costs about as much as 0.6 heads.
  double best = 0;
  for (int per = 1; per <= group; ++per) {
    const int splits = (group + per - 1) / per;
    const double rounds = std::ceil(static_cast<double>(pairs_upper) * p.num_k_heads * splits / slots) * (per + 0.6);
    if (per == 1 || rounds <= best) {
      best = rounds;
      p.heads_per_cta = per;
      p.head_splits = splits;
    }
  }
  const int64_t items = static_cast<int64_t>(pairs_upper) * p.num_k_heads * p.head_splits;
  QLA_CHECK_SUPPORTED(items < (int64_t(1) << 31), "too many chunks and heads");
  p.num_pairs = pairs_upper;
  const unsigned grid = static_cast<unsigned>(std::min<int64_t>(items, slots));
#define QLA_LAUNCH_KKT(T)                                                                              \
  return with_w  ? launch_kkt<T, true>(p, tm_k, tm_q, tm_a, tm_w, grid, stream)                        \
         : over  ? launch_kkt<T, false, true>(p, tm_k, tm_q, tm_a, tm_w, grid, stream)                 \
                 : launch_kkt<T, false>(p, tm_k, tm_q, tm_a, tm_w, grid, stream)
  if (is_bf16) QLA_LAUNCH_KKT(__nv_bfloat16);
  QLA_LAUNCH_KKT(__half);
#undef QLA_LAUNCH_KKT
}

void launch_info_kkt_solve_kernel(bool over, int* block_threads, size_t* dynamic_smem_bytes) {
  *block_threads = kKktThreads;
  *dynamic_smem_bytes = over ? Area::kSmemOver : Area::kSmem;
}

}  // namespace qla
