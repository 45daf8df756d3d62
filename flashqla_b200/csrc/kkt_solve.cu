// Chunk preparation for the prefill path: chunk-local cumulative gates and the gated WY matrix
//   A = (I + StrictLower(diag(beta) * (G .* K K^T)))^-1,   G[c,d] = exp(g_c - g_d),
// one 64x64 unit-lower-triangular inverse per (chunk, v-head), stored in the input dtype as
// A[token, v-head, 64].  Reference: chunk_local_cumsum (flash_qla/ops/utils/cumsum.py:17-168) and
// kkt_solve (chunk/hopper/kkt_solve.py:18-342; the gated form is chunk/blackwell/kkt_solve.py:118-136
// and tests/ref_gdr.py:42-104).
//
// One CTA (256 threads) owns 128 consecutive tokens (two chunks) of one k-head and loops over the
// v-heads that share it, so K is fetched once per group.  K K^T for both chunks is a single
// tcgen05.mma (M = N = K = 128, operands straight from the TMA-written 128B-swizzled tile,
// accumulator in tensor memory); a thread owns half of row t of the product (TMEM lane t, 32 of its chunk's 64
// columns) and reads it from tensor memory, 16 columns at a time, when it builds L.  It also produces, per v-head,
// the chunk operand
//   Wt = A diag(beta gamma) K      (the "w" of tests/ref_gdr.py:107-147, stored negated)
// that lets the scan kernel form Vd = A diag(beta) V - Wt S0 with a single state-dependent product:
// one more tcgen05.mma per chunk (the [128][64] tile of -A diag(beta gamma) rows times that chunk's K rows read
// MN-major) leaves row t of Wt in TMEM lane t; the rows leave through a swizzled staging tile and TMA stores
// (row by row for a ragged tail).  Both products share 128 columns: K K^T is formed again for every further head.
// The inverse of the unit-lower-triangular I + L is
// blocked: the two 32 x 32 diagonal blocks by fp32 forward substitution (one warp per block, one lane per column), then
// X21 = -X22 (L21 X11) with mma.sync m16n8k8 TF32 products on fp32 shared-memory tiles.
//
// What bounds it: instruction issue, and a chain of a dozen short dependent phases per head whose latencies the warps of
// an SM hide for each other.  Four warps per chunk (24 per SM), code that fits the instruction cache (97 % hits), two fp32
// values per instruction (add / mul / fma .f32x2) where a phase is elementwise, exponents that carry |beta| and the
// norms, and no causal mask: what lies on or above
// the diagonal of L is never read.
#include "chunk_params.cuh"

namespace qla {


namespace {

// The inverse is formed IN PLACE: every block of X = (I + L)^-1 overwrites the block of L it was computed from, and
// the products L21 X11 pass through the (never used) upper-right 32 x 32 block of the same tile.  One fp32 tile
// per chunk keeps a CTA at 67 KiB of shared memory and 128 tensor-memory columns: three CTAs per SM.
constexpr int kLStride = 68;  // floats per L row: 16-byte aligned rows, conflict-free float4 stores
constexpr int kXStride = kLStride;
// The 32 x 32 products are single TF32, like the reference's fp32-tile gemm there (chunk/hopper/kkt_solve.py:181-183):
// against an fp64 inverse the error of that block is 1.70e-3 relative rms instead of 1.68e-3 with 3xTF32 (the 16-bit
// rounding of A dominates both), and o / final state do not move in the fourth digit.
constexpr int kTStride = kLStride;  // the products live in columns 32..63 of rows 0..31 of the chunk's tile

__device__ __forceinline__ uint32_t to_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// One warp: C[16 x 16] = A[16 x K] * B[K x 16] on fp32 shared-memory tiles (row-major, strides in floats), products
// k = first .. K - 1 in steps of 8.  A fragments come by ldmatrix: an 8 x 8 matrix of 16-bit values is an 8 x 4 one of
// 32-bit values, thread 4 g + c receiving element (g, c).
__device__ __forceinline__ void warp_gemm_tf32(float (&acc)[2][4], const float* A, const float* B, int stride, int K,
                                               int first) {
  const int lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[nt][e] = 0.f;
  // matrices of ldmatrix.x4: rows 0..7 | 8..15 of columns k0..k0+3, the same of columns k0+4..k0+7
  uint32_t a_addr = ptx::smem_u32(A + ((lane & 7) + (lane & 8)) * stride + (lane >> 4) * 4 + first);
  const float* b = B + (first + c) * stride + g;
#pragma unroll 1
  for (int k0 = first; k0 < K; k0 += 8) {
    uint32_t a[4];
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(a_addr) : "memory");
    const float b00 = b[0], b10 = b[4 * stride], b01 = b[8], b11 = b[4 * stride + 8];
#pragma unroll
    for (int e = 0; e < 4; ++e) a[e] = to_tf32(__uint_as_float(a[e]));
    mma_tf32(acc[0], a, to_tf32(b00), to_tf32(b10));
    mma_tf32(acc[1], a, to_tf32(b01), to_tf32(b11));
    a_addr += 32;
    b += 8 * stride;
  }
}
// Two fp32 values per instruction.
using F2 = unsigned long long;
__device__ __forceinline__ F2 f2(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack(F2 x, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(x)); }
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// Store a warp's 16 x 8*NT accumulator tile, negated or not, to a row-major fp32 tile.
template <int NT>
__device__ __forceinline__ void store_tile(float* D, int ldd, const float (&acc)[NT][4], float sign) {
  const int lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    *reinterpret_cast<float2*>(D + g * ldd + nt * 8 + 2 * c) = make_float2(sign * acc[nt][0], sign * acc[nt][1]);
    *reinterpret_cast<float2*>(D + (g + 8) * ldd + nt * 8 + 2 * c) = make_float2(sign * acc[nt][2], sign * acc[nt][3]);
  }
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
__device__ __forceinline__ void chunk_sync(int ci) {  // the four warps that own one chunk
  asm volatile("bar.sync %0, 128;" ::"r"(ci + 1) : "memory");
}
constexpr int kKktThreads = 256;

// K tile 32 KiB + one fp32 L / X tile per chunk (later the Aw, A and w staging tiles)
constexpr size_t kKktSmemBytes = 1024 + 32768 + 2 * 64 * kLStride * sizeof(float);

template <typename T>
__global__ void __launch_bounds__(kKktThreads, 3) kkt_solve_kernel(const __grid_constant__ CUtensorMap tm_k,
                                                                const __grid_constant__ CUtensorMap tm_q,
                                                                const __grid_constant__ CUtensorMap tm_a,
                                                                const __grid_constant__ CUtensorMap tm_w,
                                                                const KktParams p) {
  grid_dep_wait();    // earlier kernels of the stream have completed (see launch_dependent)
  grid_dep_launch();  // the next one may be scheduled; it waits the same way
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int hk = blockIdx.y;
  const int group = p.num_v_heads / p.num_k_heads;

  // ---- which 128 tokens
  int seq_start, seq_end, local_pair;
  if (p.cu_seqlens != nullptr) {
    const int pair = blockIdx.x;
    if (pair >= p.pair_offsets[p.num_seqs]) return;
    int lo = 0, hi = p.num_seqs - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (p.pair_offsets[mid] <= pair) lo = mid; else hi = mid - 1;
    }
    seq_start = p.cu_seqlens[lo];
    seq_end = p.cu_seqlens[lo + 1];
    local_pair = pair - p.pair_offsets[lo];
  } else {
    const int pairs_per_seq = (p.seq_len + 127) / 128;
    const int b = blockIdx.x / pairs_per_seq;
    local_pair = blockIdx.x % pairs_per_seq;
    seq_start = b * p.seq_len;
    seq_end = seq_start + p.seq_len;
  }
  const int tok0 = seq_start + local_pair * 128;

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* sK = smem_raw + ((1024u - (ptx::smem_u32(smem_raw) & 1023u)) & 1023u);
  float* sL = reinterpret_cast<float*>(sK + 32768);  // [2][64][kLStride]: L, then X in place
  uint8_t* sAw = reinterpret_cast<uint8_t*>(sL);     // 16 KiB [128 tokens][64] tile -A diag(beta gamma) (SW128), overlays L once solved
  uint8_t* sAst = sAw + 16384;                       // 16 KiB [128 tokens][64] staging tile of A for the TMA store (SW128)
  uint8_t* sW = sAw;                                 // 32 KiB staging tile of w (two [128][64] halves, SW128), once both are consumed
  __shared__ __align__(16) float s_bg[128];          // -beta * gamma per token
  // exponents (log2) of L: -L[c][d] = -sign(beta_c) (k_c . k_d) 2^(s_row[c] + s_col[d]); the sign is that of s_bg[c]
  __shared__ __align__(16) float s_row[128];         // g log2(e) + log2(|beta| / |k_c|)
  __shared__ __align__(16) float s_col[128];         // -(g log2(e)) - log2 |k_d|     (|k| = 1 without in-kernel norm)
  __shared__ float s_norm[2][128][2];                // [column half][token][k | q]: partial squared norms
  __shared__ float s_part[kKktThreads / 32];
  __shared__ uint64_t bar_tma, bar_mma;
  __shared__ uint32_t tmem_base_s;

  if (tid == 0) {
    ptx::mbar_init(&bar_tma, 1);
    ptx::mbar_init(&bar_mma, 1);
    ptx::fence_mbar_init();
    ptx::mbar_wait_setup(p.status, &bar_tma, 0);
    ptx::mbar_expect_tx(&bar_tma, p.rnorm != nullptr ? 65536 : 32768);
    ptx::tma_load_3d(sK, &tm_k, &bar_tma, 0, hk, tok0);           // columns 0..63 of 128 tokens
    ptx::tma_load_3d(sK + 16384, &tm_k, &bar_tma, 64, hk, tok0);  // columns 64..127
    if (p.rnorm != nullptr) {  // the Q tile visits the (still unused) X area, only for its row norms
      ptx::tma_load_3d(sK + 32768, &tm_q, &bar_tma, 0, hk, tok0);
      ptx::tma_load_3d(sK + 32768 + 16384, &tm_q, &bar_tma, 64, hk, tok0);
    }
  }
  // Warp w: TMEM quadrant w % 4, i.e. rows 32 (w & 1) .. + 31 of chunk (w >> 1) & 1, column half w >> 2.
  const int ci = (warp >> 1) & 1, ch = warp >> 2, c = (warp & 1) * 32 + lane, row = ci * 64 + c;
  const int64_t tok = static_cast<int64_t>(tok0) + row;
  const bool valid = tok < seq_end;
  // gate / beta of the first v-head are requested before anything waits, those of the next head at the
  // top of every head iteration: their global-memory latency hides behind the work in between
  float gv_n = 0.f, bv_n = 0.f, gin_n = 0.f;
  auto fetch_gates = [&](int hv) {
    gv_n = bv_n = gin_n = 0.f;
    if (ch == 0 && valid) {
      const int64_t idx = tok * p.num_v_heads + hv;
      bv_n = load_scalar(p.beta, p.beta_dtype, idx);
      if (p.A_in != nullptr) gin_n = p.g_cumsum[idx];
      else gv_n = load_scalar(p.g, p.gate_dtype, idx);
    }
  };
  fetch_gates(hk * group);
  if (warp == 0) {
    ptx::tmem_alloc(&tmem_base_s, 128);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem = tmem_base_s;
  const uint32_t a_tma = ptx::smem_u32(&bar_tma), a_mma = ptx::smem_u32(&bar_mma);

  const int wl = (warp & 1) + 2 * ch;  // warp within the chunk
  const uint32_t quad = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);

  constexpr uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? ptx::kFmtBF16 : ptx::kFmtF16;
  // Products are issued by warp 0 as a converged warp (one elected lane inside ptx::umma_*): operand
  // arithmetic then stays on the uniform datapath and an instruction costs its time on the tensor pipe.
  const uint64_t d_k = ptx::smem_desc_sw128(ptx::smem_u32(sK), 16, 1024);
  auto issue_kkt = [&]() {
    ptx::umma_ss_k128_rolled<2, 1024 - 6, 2, 1024 - 6>(tmem, d_k, d_k, ptx::mma_idesc(128, 128, fmt, ptx::kMajorK, ptx::kMajorK),
                                                       false, a_mma);
  };
  bool ok = true;
  if (warp == 0) {
    ok = ptx::mbar_wait_addr(a_tma, 0);
    if (ok) issue_kkt();
    else ptx::umma_commit(&bar_mma);
  }
  // In-kernel L2 norm of q and k (reference: l2norm before the kernels, flash_qla/utils/math.py:14-21 via
  // chunk/__init__.py:332-334): 1/sqrt(|row|^2 + eps) of the K and Q rows, half a row per thread, while the
  // product runs.  Everything downstream uses the RAW tiles and folds the factors in: K K^T[c][d] r_c r_d
  // (in the exponents), r_k into beta gamma for w; the scan folds r_k into rho, r_q into s gamma and both into Pg.
  float lrk = 0.f;  // log2 of 1 / |k_t|
  if (p.rnorm != nullptr) {
    const bool got = ptx::mbar_wait_addr(a_tma, 0);
    float sk = 0.f, sq = 0.f;
    if (got) {
#pragma unroll 2
      for (int c16 = 0; c16 < 8; ++c16) {
        const uint32_t off = ch * 16384 + ptx::sw128_offset(row, c16);
        const uint4 kv = *reinterpret_cast<const uint4*>(sK + off);
        const uint4 qv = *reinterpret_cast<const uint4*>(sK + 32768 + off);
        const T* ke = reinterpret_cast<const T*>(&kv);
        const T* qe = reinterpret_cast<const T*>(&qv);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float a = Cvt<T>::to_f32(ke[e]), b = Cvt<T>::to_f32(qe[e]);
          sk += a * a;
          sq += b * b;
        }
      }
    }
    s_norm[ch][row][0] = sk;
    s_norm[ch][row][1] = sq;
    __syncthreads();
    const float rk = rsqrtf(s_norm[0][row][0] + s_norm[1][row][0] + p.norm_eps);
    if (ch == 0) {
      lrk = ptx::lg2(rk);
      const float rq = rsqrtf(s_norm[0][row][1] + s_norm[1][row][1] + p.norm_eps);
      if (valid) *reinterpret_cast<float2*>(p.rnorm + (tok * p.num_k_heads + hk) * 2) = make_float2(rq, rk);
    }
  }
  // (every thread gets here; also orders the last reads of the Q tile before the head loop reuses that memory)
  ok = __syncthreads_and(ok) != 0;

  float* Lc = sL + ci * 64 * kLStride;  // this chunk's tile; the inverse X is formed in place
  float* Tc = Lc + 32;                  // products: rows 0..31, columns 32..63
  const bool full_pair = tok0 + 128 <= seq_end;
  int mma_uses = 0;  // phases of bar_mma waited for
#pragma unroll 1
  for (int hv = hk * group; ok && hv < (hk + 1) * group; ++hv) {
    float gv = gv_n, bv = bv_n;
    const float gin = gin_n;
    if (hv + 1 < (hk + 1) * group) fetch_gates(hv + 1);
    // K K^T again, over the w product of the previous head (which has been read)
    if (warp == 0 && hv > hk * group) {
      ptx::tc_fence_after_sync();
      issue_kkt();
    }
    // the previous head's w tile lies where L is built next: its store must have read it by now
    if (tid == 0) ptx::tma_store_wait_read();
    if (ch == 0) {
      if (valid && p.beta_out != nullptr) {  // logits in: the activated value is what every later stage reads
        bv = 1.f / (1.f + __expf(-bv));
        p.beta_out[tok * p.num_v_heads + hv] = bv;
      }
      if (valid && p.A_log != nullptr) {  // gate activation of the layer (recurrent op: recurrent_fused.py:346-487)
        const float x = gv + p.dt_bias[hv];
        gv = -expf(p.A_log[hv]) * (x <= 20.f ? log1pf(expf(x)) : x);
      }
      // inclusive scan over the 64 tokens of the chunk (two warps)
      float gcs = gv;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const float n = __shfl_up_sync(0xffffffffu, gcs, off);
        if (lane >= off) gcs += n;
      }
      if (lane == 31) s_part[warp] = gcs;
      asm volatile("bar.sync 3, 128;" ::: "memory");  // warps 0-3
      if (warp & 1) gcs += s_part[warp - 1];
      if (p.A_in != nullptr) gcs = gin;  // gates are cumulative already
      else if (valid) p.g_cumsum[tok * p.num_v_heads + hv] = gcs;
      const float gc2 = gcs * 1.4426950408889634f;  // exponents are formed in the log2 domain
      const float er = gc2 + (ptx::lg2(fabsf(bv)) + lrk);  // (beta = 0: -inf, every power below is 0)
      s_row[row] = er;
      s_col[row] = lrk - gc2;
      s_bg[row] = copysignf(ptx::ex2(er), -bv);
    }
    ok = __syncthreads_and(warp != 0 || ptx::mbar_wait_addr(a_mma, mma_uses & 1)) != 0;  // (one warp polls)
    ++mma_uses;
    if (!ok) continue;
    ptx::tc_fence_after_sync();

    if (p.A_in != nullptr) {
      // A comes from an earlier call: this thread's half row straight into the X tile
      const T* arow = static_cast<const T*>(p.A_in) + (tok * p.num_v_heads + hv) * 64 + ch * 32;
#pragma unroll 1
      for (int j = 0; j < 32; j += 8) {
        uint4 raw = valid ? *reinterpret_cast<const uint4*>(arow + j) : make_uint4(0, 0, 0, 0);
        const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
        for (int x = 0; x < 8; ++x) Lc[c * kXStride + ch * 32 + j + x] = Cvt<T>::to_f32(e[x]);
      }
    } else {
      // -L[c][d] = -beta_c exp(g_c - g_d) (k_c . k_d), 16 columns at a time, the entries on and above the diagonal
      // included: they may overflow, but nothing reads them.  The warps that own rows 0..31 have nothing to do in
      // columns 32..63.
      if (ch == 0 || (warp & 1)) {
        const float er = s_row[row];
        const float sign = copysignf(1.f, s_bg[row]);  // -sign(beta)
        const F2 er2 = f2(er, er), sign2 = f2(sign, sign);
#pragma unroll 1
        for (int d16 = ch * 32; d16 < ch * 32 + 32; d16 += 16) {
          uint32_t kk[16];
          ptx::tmem_ld16(quad + ci * 64 + d16, kk);
          const ulonglong2* col = reinterpret_cast<const ulonglong2*>(s_col + ci * 64 + d16);
          F2 e[8];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const ulonglong2 cv = col[j];
            e[2 * j] = add2(er2, cv.x);
            e[2 * j + 1] = add2(er2, cv.y);
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float lo, hi;
            unpack(e[j], lo, hi);
            e[j] = mul2(f2(ptx::ex2(lo), ptx::ex2(hi)), sign2);
          }
          ptx::tmem_wait_ld();
          ulonglong2* dst = reinterpret_cast<ulonglong2*>(Lc + c * kLStride + d16);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            dst[j] = make_ulonglong2(mul2(e[2 * j], f2(__uint_as_float(kk[4 * j]), __uint_as_float(kk[4 * j + 1]))),
                                     mul2(e[2 * j + 1], f2(__uint_as_float(kk[4 * j + 2]), __uint_as_float(kk[4 * j + 3]))));
        }
      }
      chunk_sync(ci);
      // ---- blocked inverse of I + L for this chunk (four warps)
      if (ch == 0) {
        // the two 32 x 32 diagonal blocks, one per warp: lane = column.  x_i = e_i + sum_j<i (-L)_ij x_j, two terms per
        // instruction, even and odd j in partial sums; every lane reads the same row of L.
        float* Lb = Lc + (c & 32) * (kLStride + 1);
        F2 xp[16];
        float x_even = 0.f;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          F2 acc = f2(i == lane ? 1.f : 0.f, 0.f), acc_b = f2(0.f, 0.f);
          float tail = 0.f;  // -L[i][i - 1], odd i
#pragma unroll
          for (int j4 = 0; j4 < i; j4 += 4) {
            const ulonglong2 l = *reinterpret_cast<const ulonglong2*>(Lb + i * kLStride + j4);
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
        __syncwarp();  // the whole block has been read
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float lo, hi;
          unpack(xp[i], lo, hi);
          Lb[2 * i * kLStride + lane] = lo;
          Lb[(2 * i + 1) * kLStride + lane] = hi;
        }
      }
      chunk_sync(ci);
      {
        // X[32:64, 0:32] = X[32:64, 32:64] ((-L)[32:64, 0:32] X[0:32, 0:32]); 16 rows and 16 columns per warp.  X[0:32, 0:32]
        // is lower triangular: its columns 16.. begin in row 16; so is X[32:64, 32:64]: its rows 0..15 end at column 15.
        const int r = wl & 1, R0 = 32 + 16 * r, n0 = 16 * (wl >> 1);
        float acc[2][4];
        warp_gemm_tf32(acc, Lc + R0 * kLStride, Lc + n0, kLStride, 32, n0);
        store_tile<2>(Tc + r * 16 * kTStride + n0, kTStride, acc, 1.f);
        chunk_sync(ci);
        warp_gemm_tf32(acc, Lc + R0 * kXStride + 32, Tc + n0, kTStride, 16 * (r + 1), 0);
        store_tile<2>(Lc + R0 * kXStride + n0, kXStride, acc, 1.f);
      }
    }  // A_in
    // ---- w = -A diag(beta gamma) K.  Row t of the [128][64] tile holds -A[t][:] .* (beta gamma) of t's own
    // chunk; one tcgen05.mma per chunk multiplies 64 rows with that chunk's 64 K rows (read MN-major).  The same pass
    // writes A itself (16-bit) into a staging tile for one TMA store.
    // The upper triangle of X is exactly zero (forward substitution yields exact zeros inside the diagonal blocks),
    // and rows / columns of tokens past the sequence end carry beta = 0, so no mask is applied here.
    __syncthreads();
    {
      // The staging tiles overlay the fp32 tile they are built from: every thread first takes its half row into
      // registers (both 16-bit forms), and writes after a barrier.  Columns 32..63 of rows 0..31 hold the scratch
      // products, not zeros: they are skipped.
      const float* xr = Lc + c * kXStride + ch * 32;
      const float* bg = s_bg + ci * 64 + ch * 32;
      const bool zero = ch == 1 && (warp & 1) == 0;
      uint32_t aw[16], av[16];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        ulonglong2 x = *reinterpret_cast<const ulonglong2*>(xr + j * 4);
        if (zero) x = make_ulonglong2(0, 0);
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(bg + j * 4);
        float lo, hi;
        unpack(mul2(x.x, b.x), lo, hi);
        aw[2 * j] = pack2<T>(lo, hi);
        unpack(mul2(x.y, b.y), lo, hi);
        aw[2 * j + 1] = pack2<T>(lo, hi);
        unpack(x.x, lo, hi);
        av[2 * j] = pack2<T>(lo, hi);
        unpack(x.y, lo, hi);
        av[2 * j + 1] = pack2<T>(lo, hi);
      }
      __syncthreads();
      T* arow = static_cast<T*>(p.A) + (tok * p.num_v_heads + hv) * 64 + ch * 32;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t off = ptx::sw128_offset(row, ch * 4 + j);  // row = token within the pair
        *reinterpret_cast<uint4*>(sAw + off) = make_uint4(aw[4 * j], aw[4 * j + 1], aw[4 * j + 2], aw[4 * j + 3]);
        if (p.A_in == nullptr) {
          const uint4 a4 = make_uint4(av[4 * j], av[4 * j + 1], av[4 * j + 2], av[4 * j + 3]);
          if (full_pair) *reinterpret_cast<uint4*>(sAst + off) = a4;
          else if (valid) *reinterpret_cast<uint4*>(arow + j * 8) = a4;  // ragged tail: the next sequence owns the rest
        }
      }
    }
    ptx::fence_proxy_async_smem();
    ptx::tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) {
      if (lane == 0 && p.A_in == nullptr && full_pair) {
        ptx::tma_store_3d(&tm_a, sAst, 0, hv, tok0);
        ptx::tma_store_commit();
      }
      __syncwarp();
      ptx::tc_fence_after_sync();
      // two M = 64 products into the same 128 columns: row r of chunk 0 lands in lane (r % 16) + 32 (r / 16), the
      // rows of chunk 1 in the 16 lanes above them
      const uint32_t idesc = ptx::mma_idesc(64, 128, fmt, ptx::kMajorK, ptx::kMajorMN);
      const uint64_t da = ptx::smem_desc_sw128(ptx::smem_u32(sAw), 16, 1024);
      const uint64_t db = ptx::smem_desc_sw128(ptx::smem_u32(sK), 16384, 1024);
      ptx::umma_ss_k64<2, 128>(tmem, da, db, idesc, false);                                            // chunk 0: K rows 0..63
      ptx::umma_ss_k64<2, 128>(tmem + (16u << 16), da + (8192 >> 4), db + (8192 >> 4), idesc, false, a_mma);  // chunk 1: rows 64..127
      // the w rows are staged where the A tile sits: its store has to have read it before anybody passes
      // the barrier below
      if (lane == 0) ptx::tma_store_wait_read();
      __syncwarp();
    }
    ok = __syncthreads_and(warp != 0 || ptx::mbar_wait_addr(a_mma, mma_uses & 1)) != 0;  // (one warp polls)
    ++mma_uses;
    if (!ok) continue;
    ptx::tc_fence_after_sync();
    {
      // Half a row of w per thread: lane l of quadrant q holds row 16 q + (l & 15) of chunk l >> 4.  A full
      // pair goes through a swizzled staging tile and two TMA stores (whole 128-byte lines per token row); a ragged
      // tail is written row by row, only by lanes with a valid token.  tcgen05.ld is warp-collective: every lane
      // runs the loop.
      const int tp = (lane >> 4) * 64 + (warp & 3) * 16 + (lane & 15);  // token within the pair
      const bool valid_w = static_cast<int64_t>(tok0) + tp < seq_end;
      T* wrow = static_cast<T*>(p.w) + ((static_cast<int64_t>(tok0) + tp) * p.num_v_heads + hv) * kHeadDim + ch * 64;
      uint8_t* half = sW + ch * 16384;
#pragma unroll 1
      for (int kb = 0; kb < 64; kb += 32) {
        uint32_t r[32];
        ptx::tmem_ld32(quad + ch * 64 + kb, r);
        ptx::tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 32; e += 8) {
          const uint4 val = make_uint4(pack2<T>(__uint_as_float(r[e]), __uint_as_float(r[e + 1])),
                                       pack2<T>(__uint_as_float(r[e + 2]), __uint_as_float(r[e + 3])),
                                       pack2<T>(__uint_as_float(r[e + 4]), __uint_as_float(r[e + 5])),
                                       pack2<T>(__uint_as_float(r[e + 6]), __uint_as_float(r[e + 7])));
          if (full_pair) *reinterpret_cast<uint4*>(half + ptx::sw128_offset(tp, (kb + e) >> 3)) = val;
          else if (valid_w) *reinterpret_cast<uint4*>(wrow + kb + e) = val;
        }
      }
    }
    ptx::fence_proxy_async_smem();
    ptx::tc_fence_before_sync();
    __syncthreads();  // s_g / s_bg are rewritten for the next head; the w tile is complete
    if (tid == 0 && full_pair) {
      ptx::tma_store_3d(&tm_w, sW, 0, hv, tok0);
      ptx::tma_store_3d(&tm_w, sW + 16384, 64, hv, tok0);
      ptx::tma_store_commit();
    }
  }
  if (tid == 0) ptx::tma_store_wait_read();  // shared memory stays allocated until the last store has read it

  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) ptx::tmem_dealloc(tmem, 128);
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

int launch_kkt_solve(const KktParams& p, const void* k, const void* q, int64_t total_tokens, int pairs_upper,
                     bool is_bf16, cudaStream_t stream) {
  CUtensorMap tm_k, tm_q, tm_a, tm_w;
  int rc = make_tmap_3d(&tm_k, k, total_tokens, p.num_k_heads, kHeadDim, 128, 64, true, is_bf16);
  if (rc != QLA_OK) return rc;
  // q is only read for the in-kernel L2 norm (p.rnorm set); otherwise the map is made over k and unused
  rc = make_tmap_3d(&tm_q, p.rnorm != nullptr ? q : k, total_tokens, p.num_k_heads, kHeadDim, 128, 64, true, is_bf16);
  if (rc != QLA_OK) return rc;
  // A leaves through a [128 tokens][64] staging tile; in rebuild mode (A given) the map is made but unused
  rc = make_tmap_3d(&tm_a, p.A, total_tokens, p.num_v_heads, 64, 128, 64, true, is_bf16);
  if (rc != QLA_OK) return rc;
  // w leaves through two [128 tokens][64] staging tiles per (pair, head)
  rc = make_tmap_3d(&tm_w, p.w, total_tokens, p.num_v_heads, kHeadDim, 128, 64, true, is_bf16);
  if (rc != QLA_OK) return rc;
  const size_t smem = kKktSmemBytes;
  dim3 grid(pairs_upper, p.num_k_heads);
  if (is_bf16) {
    if ((rc = ensure_dynamic_smem<kkt_solve_kernel<__nv_bfloat16>>(smem)) != QLA_OK) return rc;
    QLA_CHECK_CUDA(launch_dependent(kkt_solve_kernel<__nv_bfloat16>, grid, dim3(kKktThreads), smem, stream, tm_k, tm_q, tm_a, tm_w, p));
  } else {
    if ((rc = ensure_dynamic_smem<kkt_solve_kernel<__half>>(smem)) != QLA_OK) return rc;
    QLA_CHECK_CUDA(launch_dependent(kkt_solve_kernel<__half>, grid, dim3(kKktThreads), smem, stream, tm_k, tm_q, tm_a, tm_w, p));
  }
  QLA_CHECK_CUDA(cudaGetLastError());
  return QLA_OK;
}

void launch_info_kkt_solve_kernel(int* block_threads, size_t* dynamic_smem_bytes) {
  *block_threads = kKktThreads;
  *dynamic_smem_bytes = kKktSmemBytes;
}

}  // namespace qla
