// Chunked gated-delta-rule forward for sm_100a: the serial scan over 64-token chunks of one
// (sequence, v-head) with the recurrent state resident in tensor memory.
// Reference: fused_gdr_fwd (flash_qla/ops/gated_delta_rule/chunk/hopper/fused_fwd.py:19-656; the gated-A
// variant chunk/blackwell/fused_fwd.py:383-393) and the state-only pass fused_gdr_h
// (chunk/hopper/prepare_h.py:13-556); math as in tests/ref_gdr.py:107-260.
//
// Per chunk (S0 = state entering the chunk, g = chunk-local cumulative gate, gL its last value):
//   Vd = A diag(beta) (V - exp(g) .* (K S0)) = Ab V - Wt S0           (= "v_new")
//        Ab = A diag(beta),  Wt = A diag(beta exp(g)) K  (both state independent; Wt comes, negated,
//        from the preparation kernel)
//   O  = s exp(g) .* (Q S0) + (s G .* Q K^T) Vd                      G[c,d] = exp(g_c - g_d), c >= d
//   S1 = exp(gL) S0 + K^T (exp(gL - g) .* Vd)
//
// Everything is computed TRANSPOSED so that each tcgen05.mma has M = 128 (the V dimension on the 128
// TMEM lanes) and every dependent operand can stay in tensor memory:
//   MMAu  D2[128,64]  = V^T Ab^T           (SS)  state independent part of Vd^T
//   MMA2  D2[128,64] += S0^T_bf16 (-Wt)^T  (TS)  D2 = Vd^T
//   MMAq  Dq[128,64]  = S0^T_bf16 Q^T      (TS)  (Q S0)^T for the output, off the chain, two buffers
//   MMA3  S^T[128,128] += V'^T K           (TS, B operand MN-major straight from the K tile)
//   MMA4  D4[128,64]  = Vd^T Pg^T          (TS)  Pg = s G .* P is a swizzled smem tile; off the chain;
//                                                O^T = s gamma .* Dq + D4 in the output epilogue
//   MMA0  D0[64,64]   = Q K^T              (SS, M = 64)  P of the next chunk; state independent
// (all but MMA0 with M = 128: V' and Vd, 16 bit, are written back over the columns of D2 they were read from.)
// Between two state updates only  MMA2 -> (V' = rho .* Vd) -> MMA3 -> (16-bit copy of the state)  are
// serial; the other products are issued into the two gaps and complete in their shadow.
//
// What bounds it: that chain (1.4 us per chunk with the SM to itself: 1700 cycles of products in order, and hand-offs between
// 20 warps that share its issue slots), and with every SM busy the memory behind it (42 - 48 bytes per ns and SM; bulk copies alone 46 - 53).
// Shared memory moves 72 KB of TMA writes and 112 KB of operand reads per chunk at 128 bytes a cycle.  Operands
// that a thread produces therefore go to tensor memory (Vd as a shared-memory tile cost 48 KB per chunk), and Q K^T is
// not stacked on other rows to fill M = 128.  All roles share the SM's instruction cache (32 KB; 94 % of its requests hit),
// so that code which is not needed costs even where it is not executed often: see kState16.
// Thread v of a chain warpgroup owns TMEM lane v = column v of the state: it reads Vd^T rows
// with tcgen05.ld, applies the gates, and writes the bf16 operand of the next MMA back with
// tcgen05.st.  The fp32 state never leaves tensor memory between chunks.
//
// Warp roles (640 threads): warps 0-7 the chain (two warpgroups: tokens 0..31 | 32..63 of Vd, columns 0..63 | 64..127
// of the state conversion), warp 8 TMA producer + gate vectors, warp 9 MMA issuer, warps 10, 11 A diag(beta) of the
// next chunk, warps 12-15 the output, warps 16-19 Pg.  Two smem stages of {Wt,Q}, {K} and {V,A}, each reloaded as soon as its last
// product has read it (with the whole stage waiting for MMA3, and Q K^T behind MMA4: 512 chains of 32 chunks, 8 / 8 heads,
// 306 us, now 287; with the output norm 379 -> 366; kWIn has stages of its own, see its map), a four-deep ring of gate
// vectors; all waits are bounded mbarrier waits that raise a status word instead of hanging.
#include "chunk_params.cuh"

namespace qla {


namespace {

// ---- tensor-memory column map (512 columns)
constexpr uint32_t kColS = 0;      // fp32 state S^T, 128 columns
constexpr uint32_t kColSbf = 128;  // bf16 copy of S^T (A operand of MMA2), 64 columns
constexpr uint32_t kColD2 = 192;   // Vd^T; either half of 32 columns is overwritten by its V' (16 columns, A of MMA3), Vd (16, A of MMA4)
constexpr uint32_t kColDq = 256;   // (Q S0)^T, two buffers of 64 columns (chunk parity): read one chunk late
constexpr uint32_t kColD4 = 384;   // Vd^T Pg^T
constexpr uint32_t kColD0 = 448;   // Q K^T (M = 64: 16 lanes of every quadrant)

// ---- shared-memory map (offsets from a 1024-byte aligned base)
constexpr uint32_t kStageWQ = 0;         // 32 KiB: -Wt tile, then Q tile, each as two [64][64] halves (8 KiB), SW128
constexpr uint32_t kStageK = 32768;      // 16 KiB: K tile as two [64][64] halves (columns 0..63 | 64..127), SW128
constexpr uint32_t kStageV = 49152;      // 16 KiB: V tile, same form
constexpr uint32_t kStageA = 65536;      // 8 KiB: A tile [64][64], SW128; scaled in place to A diag(beta)
constexpr uint32_t kStageBytes = 73728;  // 72 KiB, multiple of 1024
constexpr uint32_t kOffPg = 2 * kStageBytes;         // 2 x 8 KiB Pg tiles, SW128 (chunk parity)
constexpr uint32_t kOffO = kOffPg + 2 * 8192;        // 2 x 16 KiB output tiles (chunk parity) as two [64][64] halves, SW128
constexpr uint32_t kOffVn = kOffO + 16384;           // kAux: the v_new tile in place of the second output tile,
constexpr uint32_t kOffH = kOffO + 2 * 16384;        // and 16 KiB for half of the h tile ([64 k][128 v] as two halves)
constexpr uint32_t kSmemBytes = kOffO + 2 * 16384 + 1024, kSmemBytesAux = kSmemBytes + 16384;

// kWIn (Wt formed by the kernel itself): {Q, V, A} in two stages, {K, -A diag(beta gamma)} in three, because Wt of a chunk is
// formed one chunk ahead; one Wt tile.
constexpr uint32_t kQvV = 16384, kQvA = 32768, kQvBytes = 40960;  // Q tile, V tile, A tile
constexpr uint32_t kOffKa = 2 * kQvBytes, kKaAw = 16384, kKaBytes = 24576;  // K tile, operand tile of Wt
constexpr int kKaStages = 3;
constexpr uint32_t kOffWt = kOffKa + kKaStages * kKaBytes;    // 16 KiB: Wt^T [128 k][64 tokens], SW128
constexpr uint32_t kOffPgWIn = kOffWt + 16384;
constexpr uint32_t kOffOWIn = kOffPgWIn + 2 * 8192;
constexpr uint32_t kSmemBytesWIn = kOffOWIn + 2 * 16384 + 1024;

struct alignas(16) Gates {
  // g * log2(e) in the two roles it plays for the aux warps, which form s exp(g_c - g_d) r_q[c] r_k[d] as
  // ex2(g2row[c] + log2 s - g2col[d]); r_q, r_k = 1 / |q_t|, 1 / |k_t| with in-kernel L2 norm, else 1
  float g2row[64];   // g log2(e) + log2 r_q
  float g2col[64];   // g log2(e) - log2 r_k
  float sgamma[64];  // scale * exp(g) * r_q
  float rho[64];
  float beta[64];
  float egl;
  int valid;  // number of valid tokens in the chunk
  int pad[2];
};
constexpr int kGateRing = 4;

enum Bar {
  kFull0 = 0, kFull1, kEmpty0, kEmpty1,
  kPDone, kPgReady, kD2Done, kVdReady, kVdStored, kSDone, kSbfReady, kSScaled, kAbReady0, kAbReady1,
  kD4Done, kORead, kOFree, kOReady, kONormed, kVnRead, kVnReady, kHRead, kHReady, kHFree, kGate0, kGate1, kGate2, kGate3,
  kD0Read,  // Q K^T has been read from its columns, which the next chunk's (kWIn: Wt of the next chunk) takes
  // kWIn: {K, operand of Wt} stages (kFull*, kEmpty* are those of {Q, V, A}), Wt in tensor memory, read from there, written to its tile
  kKaFull0, kKaFull1, kKaFull2, kKaEmpty0, kKaEmpty1, kKaEmpty2, kWDone, kWRead, kWReady,
  // otherwise: {V, A} and K of a stage (kFull*, kEmpty* are those of {Wt, Q})
  kVaFull0, kVaFull1, kVaEmpty0, kVaEmpty1, kKFull0, kKFull1, kKEmpty0, kKEmpty1,
  kNumBars
};

constexpr int kThreads = 640;

// One arrival per warp: every lane has finished (and fenced) its own writes, the warp converges, and
// lane 0 signals the barrier.
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
__device__ __forceinline__ uint32_t pack2(F2 x) {
  const float2 y = unpack(x);
  return pack2<T>(y.x, y.y);
}

// Gated RMS norm of an output tile (two 128B-swizzled [64][64] halves at shared address `so`), in place: rows first + 16 y +
// 0..7 (y = 0..3) by the four warps that call it, 16 threads per row with eight values each; `z` is the gate row of the
// tile's first token, `stride` elements from token to token.  The gate is requested before the tile is waited for.  With the
// four output warps doing all rows a chunk took 3.0 us (1.4 without the norm) and 777 tokens of 32 heads 46 us of scan; with
// the Pg warps doing half 39.5, with the Pg warps doing all 44.  One copy of the code for both callers.
// A chunk's norm is bound by instruction issue beside the other roles (2000 of its 2950 cycles; the rest is the latency of the
// gate), not by how many warps share it.  Pairs of values per instruction and the gate as z * (1 / (1 + 2^(-z log2 e))) without
// the scaling of tiny operands that a division brings: 777 tokens of 32 heads 45.3 -> 43.9 us of scan, 32768 tokens of 2 / 4 heads
// 57.7 -> 53.9 (with the pairs in the chain below).  Four rows at once, or the gate held a chunk ahead, were slower (more code).
template <typename T>
static __device__ __noinline__ bool norm_rows(uint32_t so, const T* z, int stride, const float* weight, float eps, int valid,
                                              int first, uint32_t bar, uint32_t parity) {
  const int tl = threadIdx.x & 127, row0 = first + (tl >> 4), col = (tl & 15) * 8;
  uint4 zr[4];
#pragma unroll
  for (int y = 0; y < 4; ++y) {
    zr[y] = make_uint4(0, 0, 0, 0);
    if (row0 + 16 * y < valid) zr[y] = *reinterpret_cast<const uint4*>(z + static_cast<int64_t>(row0 + 16 * y) * stride + col);
  }
  const float4 w0 = *reinterpret_cast<const float4*>(weight + col), w1 = *reinterpret_cast<const float4*>(weight + col + 4);
  const float wv[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
  if (!ptx::mbar_wait_addr(bar, parity)) return false;
  if (valid <= 0) return true;
  uint32_t cell = so + (tl & 8) * 1024 + ptx::sw128_offset(row0, tl & 7);
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass, cell += 4096) {  // two rows at a time: half the code, and code is what is short here
    F2 x[2][4];
    float ss[2];
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      uint4 raw;
      asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(raw.x), "=r"(raw.y), "=r"(raw.z), "=r"(raw.w)
                   : "r"(cell + 2048u * y) : "memory");
      const T* e = reinterpret_cast<const T*>(&raw);
      F2 sum = f2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        x[y][i] = f2(Cvt<T>::to_f32(e[2 * i]), Cvt<T>::to_f32(e[2 * i + 1]));
        sum = fma2(x[y][i], x[y][i], sum);
      }
      ss[y] = unpack(sum).x + unpack(sum).y;
    }
#pragma unroll
    for (int off = 1; off < 16; off <<= 1)
#pragma unroll
      for (int y = 0; y < 2; ++y) ss[y] += __shfl_xor_sync(0xffffffffu, ss[y], off);
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      const float rstd = rsqrtf(ss[y] * (1.f / kHeadDim) + eps);
      const T* ze = reinterpret_cast<const T*>(&zr[y]);
      uint32_t out[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const F2 zf = f2(Cvt<T>::to_f32(ze[2 * i]), Cvt<T>::to_f32(ze[2 * i + 1]));
        const float2 l = unpack(mul2(zf, f2(-1.4426950408889634f, -1.4426950408889634f)));
        const F2 silu = mul2(zf, f2(ptx::rcp(1.f + ptx::ex2(l.x)), ptx::rcp(1.f + ptx::ex2(l.y))));
        const float2 r = unpack(mul2(mul2(mul2(x[y][i], f2(rstd, rstd)), f2(wv[2 * i], wv[2 * i + 1])), silu));
        out[i] = pack2<T>(r.x, r.y);
      }
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(cell + 2048u * y), "r"(out[0]), "r"(out[1]),
                   "r"(out[2]), "r"(out[3]) : "memory");
    }
    zr[0] = zr[2];
    zr[1] = zr[3];
  }
  return true;
}

// kAux: the launch stores h and / or v_new (training forward, backward recomputation).  A separate
// instantiation, so that the plain inference forward does not carry that code in its instruction stream:
// the loops below are shaped for a small per-chunk code footprint (rolled 32-column groups, every product
// issued from one place, the slow path of a wait as a call).
// kNorm: the output tile passes through the gated RMS norm that follows the op in a GDN layer
// (o <- o * rsqrt(mean_v(o^2) + eps) * weight[v] * silu(z[t, h, v])) before it is stored.
// kState16: h0 / final_state are bf16 (state pools); its own instantiation, like kNorm: the code of the plain
// forward must stay small (it is the instruction cache, not the work, that a few extra branches in the
// unrolled state loops cost: +20 % on the whole scan when they were part of the plain kernel).
// kWIn: in place of A and w come A diag(beta) (rounded as this kernel rounds it otherwise) and -A diag(beta gamma) (as the preparation
// kernel does for w): Wt, the product of the latter with K, is formed here, one chunk ahead of its use.  Operands and
// orders are the same, so that results are the same bits.  It saves the write and the read of 128 bytes per token and head: 32768
// tokens of 16 / 32 heads 140 + 226 -> 114 + 225 us (preparation + scan), 540 k packed tokens of 8 / 8 heads 584 + 1141 -> 501 + 1015.
// (With A diag(beta) scaled here from A the preparation took 6 % less and the scan 9 % more.)
template <typename T, bool kStateOnly, bool kAux, bool kTrace, bool kNorm = false, bool kState16 = false, bool kWIn = false>
__global__ void __launch_bounds__(kThreads, 1)
chunk_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                 const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_a,
                 const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_o,
                 const __grid_constant__ CUtensorMap tm_vn, const __grid_constant__ CUtensorMap tm_h, const FwdParams p) {
  constexpr uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? ptx::kFmtBF16 : ptx::kFmtF16;
  grid_dep_wait();    // earlier kernels of the stream have completed (see launch_dependent)
  grid_dep_launch();  // the next one may be scheduled; it waits the same way
  // (the shuffle tells the compiler that the role is the same for the whole warp: addresses, descriptors and loop
  // counters of the single-warp roles then live in uniform registers)
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  // A "dual" launch carries two passes over the same sequences in one grid: the CTAs of the second half run
  // the transition-matrix pass of context parallelism (start from the identity, V treated as zero) with their
  // own chunk limits and output rows (chunk_limit_b, seq_map_b, final_state_b).
  const bool pass_b = p.dual && blockIdx.x >= static_cast<unsigned>(p.num_seqs) * p.num_v_heads;
  const unsigned cta = pass_b ? blockIdx.x - static_cast<unsigned>(p.num_seqs) * p.num_v_heads : blockIdx.x;
  const bool zero_v = p.zero_v || pass_b, init_identity = p.init_identity || pass_b;
  const int32_t* chunk_limit = pass_b ? p.chunk_limit_b : p.chunk_limit;
  const int32_t* seq_map = pass_b ? p.seq_map_b : p.seq_map;
  void* final_state = pass_b ? p.final_state_b : p.final_state;
  const int hv = cta % p.num_v_heads;
  const int slot = cta / p.num_v_heads;
  const int seq = p.seq_order ? p.seq_order[slot] : slot;  // CTAs start in grid order: the caller's order of sequences
  const int hk = hv / (p.num_v_heads / p.num_k_heads);

  int seq_start, seq_end;
  if (p.cu_seqlens != nullptr) {
    seq_start = p.cu_seqlens[seq];
    seq_end = p.cu_seqlens[seq + 1];
  } else {
    seq_start = seq * p.seq_len;
    seq_end = seq_start + p.seq_len;
  }
  int nchunks = (seq_end - seq_start + kChunk - 1) / kChunk;
  int first_chunk = 0;
  if (chunk_limit != nullptr) {
    const int lim = chunk_limit[seq * p.num_v_heads + hv];
    if (lim <= 0) return;  // nothing asked of this (sequence, head); uniform for the whole CTA
    if (lim < nchunks) first_chunk = nchunks - lim;
  }
  // warm-up inside the scan: `lead` chunks of the interval in front (same sequence) are run first from a zero
  // state; nothing of them is stored (their own interval's CTA computes them exactly)
  const int lead = (p.lead != nullptr && !pass_b) ? p.lead[seq * p.num_v_heads + hv] : 0;
  first_chunk -= lead;
  const int nproc = nchunks - first_chunk;
  int out_row = seq_map ? seq_map[seq] : seq;
  if (p.final_map != nullptr && !pass_b && out_row >= 0) out_row = p.final_map[out_row];
  const int64_t chunk_base =
      p.chunk_offsets ? p.chunk_offsets[seq] : static_cast<int64_t>(seq) * ((p.seq_len + kChunk - 1) / kChunk);

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // align up with pointer arithmetic on the shared array so that the compiler keeps the address space
  uint8_t* smem = smem_raw + ((1024u - (ptx::smem_u32(smem_raw) & 1023u)) & 1023u);
  __shared__ uint64_t bars[kNumBars];
  __shared__ uint32_t tmem_base_s;
  // Gate vectors live in their own ring (indexed by chunk, not by stage) with a barrier per slot: the compute
  // warpgroups read them long after the stage's tiles were consumed, and the stage must not wait for that.  Slot
  // reuse needs no barrier of its own: chunk i + 2 is only written after MMA3 of chunk i has finished, which needs
  // both warpgroups to have left chunk i - 1 and MMA4 of chunk i - 2 (the last use of its Pg) to have been issued.
  __shared__ Gates gate_ring[kGateRing];
  constexpr uint32_t kPgTiles = kWIn ? kOffPgWIn : kOffPg, kOTiles = kWIn ? kOffOWIn : kOffO;

  if (tid < kNumBars) {  // (a thread each: one after the other they were 3 us of a CTA's start: scan of 64 tokens 9.8 -> 6.9 us)
    const int b = tid;
    int count = 1;  // k*Full*, k*Empty*, kGate*, kPDone, kD2Done, kSDone, kD4Done, kWDone, kOFree: one commit / one thread
    if (b == kAbReady0 || b == kAbReady1) count = 2;
    else if (b == kPgReady || b == kORead || b == kOReady || b == kVnRead || b == kVnReady || b == kHRead ||
             b == kHReady || b == kWRead || b == kWReady || b == kD0Read)
      count = 4;
    else if (b == kVdReady || b == kVdStored || b == kSbfReady || b == kSScaled || b == kONormed) count = 8;
    ptx::mbar_init(&bars[b], count);
    ptx::fence_mbar_init();
    if (tid == 0) ptx::mbar_wait_setup(p.status, bars, 0);
  }
  if (!kStateOnly && warp >= 12) {  // the block of Pg above the diagonal (rows 0..31, columns 32..63) of both tiles
    for (int x = tid - 384; x < 2 * 32 * 4; x += 128)
      *reinterpret_cast<uint4*>(smem + kPgTiles + (x >> 7) * 8192 + ptx::sw128_offset((x >> 2) & 31, 4 + (x & 3))) =
          make_uint4(0, 0, 0, 0);
    ptx::fence_proxy_async_smem();
  }
  if (warp == 8) {
    ptx::tmem_alloc(&tmem_base_s, 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem = tmem_base_s;
  const uint32_t bar0 = ptx::smem_u32(&bars[0]);
  // (barrier index, parity) -> warp-uniform verdict
  auto wait = [&](int b, uint32_t parity) { return ptx::mbar_wait_addr(bar0 + 8u * static_cast<uint32_t>(b), parity); };

  // phase trace: one warp per role of one CTA stamps clock64() for chunks kTraceFirstChunk.. (off when p.trace is
  // NULL).  The whole warp stores (one address): a branch on the lane in the MMA issuer makes every product behind
  // it several times slower to issue, and the trace would show that instead of the kernel.
  // the traced CTA is chosen by the host through the last slot of the phase region (0 by default)
  const bool tracing = kTrace && p.trace != nullptr &&
                       static_cast<long long>(blockIdx.x) == p.trace[kTraceRoles * kTraceChunks * kTraceEvents - 1];
  auto trace = [&](int role, int i, int ev) {
    if (kTrace && tracing && i >= kTraceFirstChunk && i < kTraceFirstChunk + kTraceChunks)
      p.trace[(role * kTraceChunks + (i - kTraceFirstChunk)) * kTraceEvents + ev] = clock64();
  };

  // per-CTA residency record (start, end in ns, SM id) after the phase trace, when the buffer is large enough
  const long long cta_slot = kTraceRoles * kTraceChunks * kTraceEvents + 3ll * blockIdx.x;
  const bool cta_trace = kTrace && p.trace != nullptr && cta_slot + 3 <= p.trace_count;
  if (cta_trace && tid == 0) {
    unsigned sm;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
    p.trace[cta_slot] = static_cast<long long>(ptx::global_timer_ns());
    p.trace[cta_slot + 2] = sm;
  }

  constexpr int kTileDone = kNorm ? kONormed : kOReady;  // the output tile is what is to be stored
  auto stage_ptr = [&](int s) { return smem + s * kStageBytes; };
  auto gates_of = [&](int i) { return &gate_ring[i & (kGateRing - 1)]; };

  if (warp == 8) {
    // =========================================================== TMA producer, gate vectors
    // Tiles are not prefetched into L2.  A tensor prefetch costs the SM's copy engine and the fabric what a load costs: tiles of 128 CTAs
    // by bulk copies, four loaded and three stored per chunk, take 292 us without prefetches and 378 with the tiles requested four chunks
    // ahead.  Here, without and with: 4 x 8192 tokens of 32 heads with h and v_new 362 and 470 us, 540 k packed tokens of 8 / 8
    // heads 957 and 1020, 32768 tokens of 16 / 32 heads 215 and 226, few chains (one prompt of 777 tokens) equal.
    // Tiles are reloaded as their last product has read them.  kWIn: {Q, V, A} of chunk i behind MMAq of chunk i - 2, {K, operand of Wt}
    // of chunk i + 1 behind MMA3 of chunk i - 2.  Otherwise {Wt, Q} of chunk i behind MMAq and K behind MMA3 of chunk i - 2, {V, A} of chunk i + 1
    // behind MMAu of chunk i - 1.  Gate vectors of chunk i follow when MMA3 of chunk i - 2 is through: the last readers of their ring
    // slot (the output of chunk i - 4, which MMA4 of chunk i - 3 waited for) have left it.  Their scalars are requested a chunk before.
    constexpr int kPrefetchAhead = 4;
    const float log2e = 1.4426950408889634f;
    struct Scalars {
      float g[2], b[2], gl;
      float2 rn[2];  // (1 / |q|, 1 / |k|)
    };
    auto fetch = [&](int i, Scalars& x) {
      const int t0 = seq_start + (first_chunk + i) * kChunk;
      const int valid = min(kChunk, seq_end - t0);
      const int64_t row = static_cast<int64_t>(t0) * p.num_v_heads + hv;
      x.gl = p.g_cumsum[row + (valid - 1) * p.num_v_heads];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int c = min(lane + 32 * r, valid - 1);  // rows past the end repeat the last gate
        const int64_t at = row + c * p.num_v_heads;
        x.g[r] = p.g_cumsum[at];
        if (!kWIn) x.b[r] = load_scalar(p.beta, p.beta_dtype, at);
        x.rn[r] = make_float2(1.f, 1.f);
        if (p.rnorm != nullptr)
          x.rn[r] = *reinterpret_cast<const float2*>(p.rnorm + ((static_cast<int64_t>(t0) + c) * p.num_k_heads + hk) * 2);
      }
    };
    auto token_of = [&](int c) { return seq_start + (first_chunk + c) * kChunk; };
    auto load_early = [&](int c, int slot) {  // what a chunk needs first
      if (lane == 0 && kWIn) {
        uint8_t* st = smem + kOffKa + slot * kKaBytes;
        uint64_t* full = &bars[kKaFull0 + slot];
        ptx::mbar_expect_tx(full, kKaBytes);
        ptx::tma_load_4d(st, &tm_k, full, 0, hk, token_of(c), 0);
        ptx::tma_load_3d(st + kKaAw, &tm_w, full, 0, hv, token_of(c));
      } else if (lane == 0 && !zero_v) {
        uint8_t* st = stage_ptr(slot);
        uint64_t* full = &bars[kVaFull0 + slot];
        ptx::mbar_expect_tx(full, 8192 + 16384);
        ptx::tma_load_3d(st + kStageA, &tm_a, full, 0, hv, token_of(c));
        ptx::tma_load_4d(st + kStageV, &tm_v, full, 0, hv, token_of(c), 0);
      }
      __syncwarp();
    };
    Scalars cur = {};
    if (nproc > 0) {
      load_early(0, 0);
      fetch(0, cur);
    }
    int slot = 1, phase = 1;  // of chunk i + 1's early tiles: ring slot, and parity of its last release
#pragma unroll 1
    for (int i = 0; i < nproc; ++i) {
      const int s = i & 1;
      trace(0, i, 9);
      if (i >= 2 && !wait(kEmpty0 + s, ((i >> 1) - 1) & 1)) break;
      if (lane == 0) {
        uint64_t* full = &bars[kFull0 + s];
        if (kWIn) {
          uint8_t* st = smem + s * kQvBytes;
          ptx::mbar_expect_tx(full, (kStateOnly ? 0 : 16384) + (zero_v ? 0 : 16384 + 8192));
          if (!zero_v) {
            ptx::tma_load_3d(st + kQvA, &tm_a, full, 0, hv, token_of(i));
            ptx::tma_load_4d(st + kQvV, &tm_v, full, 0, hv, token_of(i), 0);
          }
          if (!kStateOnly) ptx::tma_load_4d(st, &tm_q, full, 0, hk, token_of(i), 0);
        } else {
          uint8_t* st = stage_ptr(s) + kStageWQ;
          ptx::mbar_expect_tx(full, kStateOnly ? 16384 : 32768);
          if (!kStateOnly) ptx::tma_load_4d(st + 16384, &tm_q, full, 0, hk, token_of(i), 0);
          ptx::tma_load_4d(st, &tm_w, full, 0, hv, token_of(i), 0);
        }
      }
      __syncwarp();
      if (!kWIn) {
        if (i >= 2 && !wait(kKEmpty0 + s, ((i >> 1) - 1) & 1)) break;
        if (lane == 0) {
          uint64_t* full = &bars[kKFull0 + s];
          ptx::mbar_expect_tx(full, 16384);
          ptx::tma_load_4d(stage_ptr(s) + kStageK, &tm_k, full, 0, hk, token_of(i), 0);
        }
        __syncwarp();
      }
      trace(0, i, 10);
      if (i + 1 < nproc) {
        if (kWIn) {
          if (i >= kKaStages - 1 && !wait(kKaEmpty0 + slot, phase)) break;
        } else if (i >= 1 && !zero_v && !wait(kVaEmpty0 + slot, phase)) {
          break;
        }
        load_early(i + 1, slot);
      }
      const int valid = min(kChunk, seq_end - token_of(i));
      Gates* gs = gates_of(i);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int c = lane + 32 * r;
        const bool ok = c < valid;
        const float g2 = cur.g[r] * log2e;
        gs->g2row[c] = g2 + ptx::lg2(cur.rn[r].x);
        gs->g2col[c] = g2 - ptx::lg2(cur.rn[r].y);
        gs->sgamma[c] = p.scale * ptx::ex2(g2) * cur.rn[r].x;
        gs->rho[c] = ok ? ptx::ex2((cur.gl - cur.g[r]) * log2e) * cur.rn[r].y : 0.f;
        if (!kWIn) gs->beta[c] = ok ? cur.b[r] : 0.f;
      }
      gs->egl = ptx::ex2(cur.gl * log2e);
      gs->valid = valid;
      warp_arrive(&bars[kGate0 + (i & 3)], lane);
      if (i + 1 < nproc) {
        if (++slot == (kWIn ? kKaStages : 2)) {
          slot = 0;
          phase ^= 1;
        }
        fetch(i + 1, cur);  // (used behind the next chunk's copies)
      }
      if (i + kPrefetchAhead < nproc) {  // the scalars of a chunk to come
        const int64_t ahead = token_of(i + kPrefetchAhead);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int64_t tk = min(ahead + lane + 32 * r, static_cast<int64_t>(seq_end) - 1);
          ptx::prefetch_l2(p.g_cumsum + tk * p.num_v_heads + hv);
          if (!kWIn) ptx::prefetch_l2(static_cast<const uint8_t*>(p.beta) + (tk * p.num_v_heads + hv) * (p.beta_dtype == QLA_DT_F32 ? 4 : 2));
          if (p.rnorm != nullptr) ptx::prefetch_l2(p.rnorm + (tk * p.num_k_heads + hk) * 2);
        }
      }
      __syncwarp();
      trace(0, i, 11);
    }
  } else if (warp == 9) {
    // =========================================================== MMA issuer (whole warp, converged)
    // Every lane runs this loop and all waits; the tcgen05.mma / commit instructions are issued by one
    // elected lane inside the ptx::umma_* blocks.  Keeping the warp converged keeps descriptors and
    // addresses on the uniform datapath, which is what makes a product cost no more than its time on
    // the tensor pipe.  The loop is software pipelined over i = -1 .. nproc - 1:
    //   [MMA2(i)] [MMAq(i), MMA0(i+1)] [MMA3(i)] [MMA4(i), MMAu(i+1)]           (MMA0 of the first chunk behind its MMAu)
    //   [MMA2(i)] [MMAq(i), MMAw(i+1)] [MMA3(i)] [MMA4(i), MMAu(i+1), MMA0(i+1)]  kWIn
    // Between two state updates only MMA2 -> (chain: V') -> MMA3 -> (both warpgroups: 16-bit state copy)
    // are serial; the other products sit in the two gaps and complete in their shadow.
    // The warp's own time counts: with an election per product, one wait after the other and D0 released behind the arithmetic of Pg
    // a chunk took it 2900 cycles.  Products in one block each, waits of one place together, D0 read first: one prompt of 777 tokens
    // 43.1 -> 41.8 us, 32768 tokens of 16 / 32 heads 215 -> 205, 540 k packed tokens of 8 / 8 heads 957 -> 936.
    {
      const uint32_t id_n64 = ptx::mma_idesc(128, 64, fmt, ptx::kMajorK, ptx::kMajorK);
      const uint32_t id_mn128 = ptx::mma_idesc(128, 128, fmt, ptx::kMajorK, ptx::kMajorMN);
      const uint32_t id_u = ptx::mma_idesc(128, 64, fmt, ptx::kMajorMN, ptx::kMajorK);
      // operand descriptors of stage 0; stage 1 is kStageBytes further (added to the address field)
      const uint64_t d_w = ptx::smem_desc_sw128(ptx::smem_u32(smem + kStageWQ), 16, 1024);      // -Wt, K-major; Q 16 KiB on
      const uint64_t d_k = ptx::smem_desc_sw128(ptx::smem_u32(smem + kStageK), 16, 1024);      // K tile, K-major
      const uint64_t d_kmn = ptx::smem_desc_sw128(ptx::smem_u32(smem + kStageK), 8192, 1024);  // K tile, MN-major
      const uint64_t d_a = ptx::smem_desc_sw128(ptx::smem_u32(smem + kStageA), 16, 1024);
      const uint64_t d_v = ptx::smem_desc_sw128(ptx::smem_u32(smem + kStageV), 8192, 1024);    // V tile, MN-major
      const uint64_t d_pg = ptx::smem_desc_sw128(ptx::smem_u32(smem + kPgTiles), 16, 1024);
      const uint32_t id_p = ptx::mma_idesc(64, 64, fmt, ptx::kMajorK, ptx::kMajorK);
      constexpr int kHalf = (8192 >> 4) - 3 * 2;  // from k-step 3 to k-step 4 of a 128-wide tile
      // The CTA owns all 512 columns, so the allocation starts at column 0 of lane 0: tensor-memory
      // addresses are compile-time constants here (checked once; a value loaded from shared memory would
      // have to be moved to a uniform register for every instruction).  Barrier addresses for the commits
      // that the product blocks issue themselves.
      constexpr uint32_t tmem0 = 0;
      auto bar_addr = [&](int b) { return bar0 + 8u * static_cast<uint32_t>(b); };
      bool ok = tmem == tmem0;
      if (!ok) ptx::record_wait_failure(p.status, kStatusBadTmemBase, 0);
      if constexpr (kWIn) {
        // The same order with MMAw(i + 1) in gap 1: D0 = K^T (-A diag(beta gamma))^T, which the Pg warps turn into the Wt tile while
        // MMA3, MMA4 and MMAu run.  D0 is Q K^T of a chunk and Wt of the next one by turns.
        const uint64_t q_desc = ptx::smem_desc_sw128(ptx::smem_u32(smem), 16, 1024);
        const uint64_t v_desc = ptx::smem_desc_sw128(ptx::smem_u32(smem + kQvV), 8192, 1024);
        const uint64_t k_desc = ptx::smem_desc_sw128(ptx::smem_u32(smem + kOffKa), 16, 1024);
        const uint64_t kmn_desc = ptx::smem_desc_sw128(ptx::smem_u32(smem + kOffKa), 8192, 1024);
        const uint64_t a_desc = ptx::smem_desc_sw128(ptx::smem_u32(smem + kQvA), 16, 1024);
        const uint64_t w_desc = ptx::smem_desc_sw128(ptx::smem_u32(smem + kOffWt), 8192, 1024);  // MN-major
        const uint64_t aw_desc = ptx::smem_desc_sw128(ptx::smem_u32(smem + kOffKa + kKaAw), 16, 1024);
        const uint32_t id_w = ptx::mma_idesc(128, 64, fmt, ptx::kMajorK, ptx::kMajorMN);
        int slot = 0, phase = 0, slot_i = 0;  // of chunk i + 1 in the {K, operand of Wt} ring; slot of chunk i
#pragma unroll 1
        for (int i = -1; ok && i < nproc; ++i) {
          const int ph = i & 1, j = i + 1;
          const uint64_t ka_i = static_cast<uint64_t>(slot_i * (kKaBytes >> 4)), ka_j = static_cast<uint64_t>(slot * (kKaBytes >> 4));
          if (i >= 0) {
            trace(0, i, 0);
            if (!(ok = ptx::mbar_wait_nocall2(bar_addr(kSbfReady), ph, bar_addr(kWReady), ph))) break;
            trace(0, i, 2);
            ptx::tc_fence_after_sync();
            ptx::umma_ts_k128<128, 128>(tmem0 + kColD2, tmem0 + kColSbf, w_desc, id_w, kStateOnly ? !zero_v : true,
                                               bar_addr(kD2Done));
            trace(0, i, 3);
            if (!kStateOnly)
              ptx::umma_ts_k128<2, kHalf>(tmem0 + kColDq + ph * 64, tmem0 + kColSbf,
                                                 q_desc + static_cast<uint64_t>(ph * (kQvBytes >> 4)), id_n64, false,
                                                 bar_addr(kEmpty0 + ph));
          }
          if (j < nproc) {
            if (kStateOnly || i < 0 ? !(ok = ptx::mbar_wait_nocall(bar_addr(kKaFull0 + slot), phase, true))
                                    : !(ok = ptx::mbar_wait_nocall2(bar_addr(kKaFull0 + slot), phase, bar_addr(kD0Read), ph)))
              break;
            ptx::tc_fence_after_sync();
            ptx::umma_ss_k64<128, 2>(tmem0 + kColD0, kmn_desc + ka_j, aw_desc + ka_j, id_u, false, bar_addr(kWDone));
          }
          if (i >= 0) {
            trace(0, i, 4);
            if (!(ok = ptx::mbar_wait_nocall2(bar_addr(kVdReady), ph, bar_addr(kSScaled), ph))) break;
            trace(0, i, 6);
            ptx::tc_fence_after_sync();
            ptx::umma_ts_k64_halves<128>(tmem0 + kColS, tmem0 + kColD2, kmn_desc + ka_i, id_mn128, true, bar_addr(kSDone),
                                         bar_addr(kKaEmpty0 + slot_i));
            trace(0, i, 7);
            if (kStateOnly) ptx::umma_commit(&bars[kEmpty0 + ph]);
            if (!kStateOnly) {
              if (!(ok = ptx::mbar_wait_nocall3(bar_addr(kVdStored), ph, bar_addr(kPgReady), ph, bar_addr(i > 0 ? kORead : kVdStored),
                                                i > 0 ? ph ^ 1 : ph)))
                break;
              ptx::tc_fence_after_sync();
              ptx::umma_ts_k64_halves<2>(tmem0 + kColD4, tmem0 + kColD2 + 16, d_pg + static_cast<uint64_t>(ph * (8192 >> 4)),
                                         id_n64, false, bar_addr(kD4Done));
            }
          }
          if (j < nproc) {
            const uint64_t qv = static_cast<uint64_t>((j & 1) * (kQvBytes >> 4));
            if (!(ok = ptx::mbar_wait_nocall(bar_addr(kFull0 + (j & 1)), (j >> 1) & 1, true))) break;
            ptx::tc_fence_after_sync();
            if (!zero_v) ptx::umma_ss_k64<128, 2>(tmem0 + kColD2, v_desc + qv, a_desc + qv, id_u, false);
            if (!kStateOnly) {
              if (!(ok = ptx::mbar_wait_nocall(bar_addr(kWRead), j & 1, true))) break;
              ptx::tc_fence_after_sync();
              ptx::umma_ss_k128<2, kHalf, 2, kHalf>(tmem0 + kColD0, q_desc + qv, k_desc + ka_j, id_p, false, bar_addr(kPDone));
            }
          }
          if (i >= 0) trace(0, i, 8);
          slot_i = slot;
          if (++slot == kKaStages) {
            slot = 0;
            phase ^= 1;
          }
        }
      } else
#pragma unroll 1
      for (int i = -1; ok && i < nproc; ++i) {
        const int ph = i & 1;
        const uint64_t so = static_cast<uint64_t>((i & 1) * (kStageBytes >> 4));
        if (i >= 0) {
          trace(0, i, 0);
          // MMA2: D2 += S0^T_bf16 (-Wt)^T on top of MMAu's product
          if (!(ok = ptx::mbar_wait_nocall(bar_addr(kSbfReady), ph, true))) break;
          trace(0, i, 2);
          ptx::tc_fence_after_sync();
          ptx::umma_ts_k128<2, kHalf>(tmem0 + kColD2, tmem0 + kColSbf, d_w + so, id_n64,
                                             kStateOnly ? !zero_v : true, bar_addr(kD2Done));
          if (kStateOnly) ptx::umma_commit(&bars[kEmpty0 + ph]);
          trace(0, i, 3);
          // gap 1 (the chain computes V'): MMAq: Dq[i & 1] = S0^T_bf16 Q^T; the output of chunk i - 2, which read that
          // buffer, was waited for in front of MMA4(i - 1)
          if (!kStateOnly)
            ptx::umma_ts_k128<2, kHalf>(tmem0 + kColDq + ph * 64, tmem0 + kColSbf, d_w + so + (16384 >> 4), id_n64,
                                               false, bar_addr(kEmpty0 + ph));
          // MMA0(i + 1): D0 = Q K^T, once the Pg warps have read that of chunk i.  (In gap 2 its 384 cycles stood between two MMA2.)
          if (!kStateOnly && i + 1 < nproc) {
            const int sj = (i + 1) & 1;
            const uint64_t sn = static_cast<uint64_t>(sj * (kStageBytes >> 4));
            if (!(ok = ptx::mbar_wait_nocall3(bar_addr(kD0Read), ph, bar_addr(kFull0 + sj), ((i + 1) >> 1) & 1, bar_addr(kKFull0 + sj),
                                              ((i + 1) >> 1) & 1)))
              break;
            ptx::tc_fence_after_sync();
            ptx::umma_ss_k128<2, kHalf, 2, kHalf>(tmem0 + kColD0, d_w + sn + (16384 >> 4), d_k + sn, id_p, false,
                                                         bar_addr(kPDone));
          }
          trace(0, i, 4);
          // MMA3: S^T += V'^T K   (B = K tile read MN-major: 64-column halves are 8 KiB apart)
          if (!(ok = ptx::mbar_wait_nocall2(bar_addr(kVdReady), ph, bar_addr(kSScaled), ph))) break;
          trace(0, i, 6);
          ptx::tc_fence_after_sync();
          ptx::umma_ts_k64_halves<128>(tmem0 + kColS, tmem0 + kColD2, d_kmn + so, id_mn128, true, bar_addr(kSDone),
                                       bar_addr(kKEmpty0 + ph));
          trace(0, i, 7);
          // gap 2 (both warpgroups convert the state).  MMA4: D4 = Vd^T Pg^T, once the output of chunk i - 1 has read D4
          if (!kStateOnly) {
            if (!(ok = ptx::mbar_wait_nocall3(bar_addr(kVdStored), ph, bar_addr(kPgReady), ph, bar_addr(i > 0 ? kORead : kVdStored),
                                              i > 0 ? ph ^ 1 : ph)))
              break;
            ptx::tc_fence_after_sync();
            ptx::umma_ts_k64_halves<2>(tmem0 + kColD4, tmem0 + kColD2 + 16, d_pg + static_cast<uint64_t>(ph * (8192 >> 4)),
                                       id_n64, false, bar_addr(kD4Done));
          }
        }
        // (kAux: v_new of this chunk has been read out of D2)
        if (kAux && i >= 0 && p.v_new != nullptr && !(ok = ptx::mbar_wait_nocall(bar_addr(kVnRead), ph, true))) break;
        // the state-independent products of the next chunk.  MMAu(i + 1): D2 = V^T (A diag(beta))^T; A operand = V tile
        // read MN-major, B operand = the A tile scaled in place (D2: MMA3 and MMA4 precede in the pipe).
        // The first chunk's MMA0 too: there is no gap 1 in front of it.
        if (i + 1 < nproc) {
          const int j = i + 1, sj = j & 1;
          const uint64_t sn = static_cast<uint64_t>(sj * (kStageBytes >> 4));
          if (!zero_v) {
            if (!(ok = ptx::mbar_wait_nocall2(bar_addr(kVaFull0 + sj), (j >> 1) & 1, bar_addr(kAbReady0 + sj), (j >> 1) & 1))) break;
            ptx::tc_fence_after_sync();
            ptx::umma_ss_k64<128, 2>(tmem0 + kColD2, d_v + sn, d_a + sn, id_u, false, bar_addr(kVaEmpty0 + sj));
          }
          if (kStateOnly || i < 0) {
            if (!(ok = ptx::mbar_wait_nocall(bar_addr(kFull0 + sj), (j >> 1) & 1, true))) break;
            if (!(ok = ptx::mbar_wait_nocall(bar_addr(kKFull0 + sj), (j >> 1) & 1, true))) break;
            ptx::tc_fence_after_sync();
          }
          if (!kStateOnly && i < 0)
            ptx::umma_ss_k128<2, kHalf, 2, kHalf>(tmem0 + kColD0, d_w + sn + (16384 >> 4), d_k + sn, id_p, false,
                                                         bar_addr(kPDone));
        }
        if (i >= 0) trace(0, i, 8);
      }
      ptx::report_issuer(p.status, ok, kNumBars);
    }
  } else if (warp >= 16) {
    // =========================================================== Pg = s * G .* P
    // Rows 16 q .. 16 q + 15 per warp (q = TMEM quadrant: the rows of an M = 64 accumulator), in the fragment layout of
    // 8 x 8 matrices, which stmatrix writes to the swizzled tile.  Warps 16, 17 have no causal entry in columns 32..63;
    // that part of their rows is zeroed once at start-up.
    const uint32_t tm = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const float log2_scale = __log2f(p.scale);
    const int p_row = (warp & 3) * 16 + (lane >> 2), p_cols = warp < 18 ? 32 : 64;
    // kWIn: Wt of chunk j, from the accumulator (lane = column k) to its tile [k][token]
    auto form_w = [&](int j) {
      if (!wait(kWDone, j & 1)) return false;
      ptx::tc_fence_after_sync();
      uint32_t x[2][32];
      ptx::tmem_ld32(tm + kColD0, x[0]);
      ptx::tmem_ld32(tm + kColD0 + 32, x[1]);
      ptx::tmem_wait_ld();
      ptx::tc_fence_before_sync();  // (kStateOnly: kWReady below is what the product that overwrites the columns waits for)
      if (!kStateOnly) warp_arrive(&bars[kWRead], lane);
      // (MMA2 of chunk j - 1, which read the tile, precedes this chunk's product in the pipe)
      const uint32_t at = ptx::sw128_offset((warp & 3) * 32 + lane, 0);
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < 4; ++e)
        {
          uint32_t y[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) y[c] = pack2<T>(__uint_as_float(x[h][8 * e + 2 * c]), __uint_as_float(x[h][8 * e + 2 * c + 1]));
          *reinterpret_cast<uint4*>(smem + kOffWt + (at ^ ((4 * h + e) << 4))) = make_uint4(y[0], y[1], y[2], y[3]);
        }
      ptx::fence_proxy_async_smem();
      warp_arrive(&bars[kWReady], lane);
      return true;
    };
    // kNorm: these warps have time to spare behind their tile and take half of the rows of the output tile's norm
    auto norm_half = [&](int j) {
      const int t0 = seq_start + (first_chunk + j) * kChunk;
      const int valid = j < lead ? 0 : min(kChunk, seq_end - t0);
      const T* z = static_cast<const T*>(p.norm_gate) + (static_cast<int64_t>(t0) * p.num_v_heads + hv) * kHeadDim;
      const bool fine = norm_rows<T>(ptx::smem_u32(smem + kOTiles + (j & 1) * 16384), z, p.num_v_heads * kHeadDim, p.norm_weight,
                                     p.norm_eps, valid, 8, bar0 + 8u * kOReady, j & 1);
      ptx::fence_proxy_async_smem();
      warp_arrive(&bars[kONormed], lane);
      return fine;
    };
    const bool begun = !kWIn || nproc == 0 || form_w(0);
#pragma unroll 1
    for (int i = 0; begun && (!kStateOnly || kWIn || (kAux && p.h != nullptr)) && i < nproc; ++i) {
      const int ph = i & 1;
      if (!kStateOnly) {
        if (warp == 16) trace(2, i, 8);
        if (!wait(kGate0 + (i & 3), (i >> 2) & 1)) break;
        const Gates* gs = gates_of(i);
        // s * exp(g_c - g_d) = 2^((g2_c + log2 s) - g2_d); above the diagonal the exponent may overflow, the
        // select below discards those entries
        const float gr0 = gs->g2row[p_row] + log2_scale, gr1 = gs->g2row[p_row + 8] + log2_scale;
        const float* gcol = gs->g2col + 2 * (lane & 3);
        if (!wait(kPDone, ph)) break;
        ptx::tc_fence_after_sync();
        if (warp == 16) trace(2, i, 9);
        // (tile i & 1 was last read by MMA4 of chunk i - 2: see the wait at the end)
        const uint32_t pg = ptx::smem_u32(smem + kPgTiles) + ph * 8192;
        // all of D0 first: the product that takes its columns next (kWIn: Wt of the next chunk) does not wait for the arithmetic
        uint32_t pr[16], pr1[16];
        ptx::tmem_ld_frag4(tm + kColD0, pr);
        ptx::tmem_ld_frag4(tm + kColD0 + 32, pr1);
        ptx::tmem_wait_ld();
        ptx::tc_fence_before_sync();
        warp_arrive(&bars[kD0Read], lane);
#pragma unroll 1
        for (int db = 0; db < p_cols; db += 32) {
          uint32_t m[8];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 gc = *reinterpret_cast<const float2*>(gcol + db + 8 * j);
            const int d = db + 8 * j + 2 * (lane & 3);
            const float x0 = ptx::ex2(gr0 - gc.x) * __uint_as_float(pr[4 * j]);
            const float x1 = ptx::ex2(gr0 - gc.y) * __uint_as_float(pr[4 * j + 1]);
            const float y0 = ptx::ex2(gr1 - gc.x) * __uint_as_float(pr[4 * j + 2]);
            const float y1 = ptx::ex2(gr1 - gc.y) * __uint_as_float(pr[4 * j + 3]);
            m[2 * j] = pack2<T>(d <= p_row ? x0 : 0.f, d + 1 <= p_row ? x1 : 0.f);
            m[2 * j + 1] = pack2<T>(d <= p_row + 8 ? y0 : 0.f, d + 1 <= p_row + 8 ? y1 : 0.f);
          }
          // matrices (columns 8 j, rows 0..7), (8 j, rows 8..15), (8 (j + 1), ..), ..: lane -> row of matrix lane / 8
          const int r = (warp & 3) * 16 + (lane & 15), c16 = (db >> 3) + (lane >> 4);
          ptx::stmatrix_x4(pg + ptx::sw128_offset(r, c16), m[0], m[1], m[2], m[3]);
          ptx::stmatrix_x4(pg + ptx::sw128_offset(r, c16 + 2), m[4], m[5], m[6], m[7]);
#pragma unroll
          for (int x = 0; x < 16; ++x) pr[x] = pr1[x];
        }
        ptx::fence_proxy_async_smem();
        // Before announcing this tile, make sure MMA4 of the previous chunk has finished: the next iteration overwrites the
        // tile it read.  Waiting HERE (MMA4 of this chunk cannot be issued before the arrival below) keeps this warp at
        // most one phase behind the D4Done barrier; behind the arrival it could fall two behind and wait forever.
        if (i > 0 && !wait(kD4Done, (i - 1) & 1)) break;
        warp_arrive(&bars[kPgReady], lane);
        if (kWIn && i + 1 < nproc && !form_w(i + 1)) break;
        if (kNorm && i > 0 && !norm_half(i - 1)) break;
        if (kNorm && i == nproc - 1 && !norm_half(i)) break;
      }
      if (kWIn && kStateOnly && i + 1 < nproc && !form_w(i + 1)) break;
      if (warp == 16) trace(2, i, 10);
      if (kAux && p.h != nullptr) {
        // h of this chunk = the 16-bit copy of the state that enters it, transposed to [K][V] through a shared-memory
        // tile, 64 rows k at a time, and TMA stores (stored from the chain's registers it was 64 two-byte stores per
        // thread and chunk on the serial path)
        if (!wait(kSbfReady, ph)) break;
        ptx::tc_fence_after_sync();
        bool fine = true;
#pragma unroll 1
        for (int kh = 0; fine && kh < 2; ++kh) {
          uint32_t x[32];  // lanes (columns v) 32 q .. + 15 | + 16 .., 32-bit columns of two k: the layout of 8 x 8 matrices
          ptx::tmem_ld_pack8(tm + kColSbf + 32 * kh, reinterpret_cast<uint32_t(&)[16]>(x[0]));
          ptx::tmem_ld_pack8(tm + (16u << 16) + kColSbf + 32 * kh, reinterpret_cast<uint32_t(&)[16]>(x[16]));
          ptx::tmem_wait_ld();
          if (kh == 1) {
            ptx::tc_fence_before_sync();
            warp_arrive(&bars[kHRead], lane);
          }
          // the tile is free once the store of its previous half has read it
          if (i + kh > 0) {
            if (warp == 16 && lane == 0) {
              ptx::tma_store_wait_read();
              ptx::mbar_arrive(&bars[kHFree]);
            }
            __syncwarp();
            if (!(fine = wait(kHFree, (2 * i + kh - 1) & 1))) break;
          }
          const uint32_t tile = ptx::smem_u32(smem + kOffH) + ((warp & 3) >> 1) * 8192;
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const int c16 = (warp & 1) * 4 + half * 2 + ((lane >> 3) & 1);
#pragma unroll
            for (int e = 0; e < 8; e += 2) {  // rows k 8 e .. 8 e + 15
              const uint32_t(&y)[4] = reinterpret_cast<const uint32_t(&)[4]>(x[16 * half + 2 * e]);
              ptx::stmatrix_x4_trans(tile + ptx::sw128_offset(8 * (e + (lane >> 4)) + (lane & 7), c16), y);
            }
          }
          ptx::fence_proxy_async_smem();
          warp_arrive(&bars[kHReady], lane);
          if (warp == 16) {
            if (!(fine = wait(kHReady, (2 * i + kh) & 1))) break;
            if (lane == 0 && i >= lead) {
              ptx::tma_store_4d(&tm_h, smem + kOffH, 0, 0,
                                static_cast<int>(((chunk_base + first_chunk + i) * p.num_v_heads + hv) * kHeadDim + 64 * kh), 0);
              ptx::tma_store_commit();
            }
            __syncwarp();
          }
        }
        if (!fine) break;
      }
    }
    if (kAux && warp == 16 && lane == 0) ptx::tma_store_wait_all();
  } else if (warp >= 12) {
    // =========================================================== output: O^T = s gamma .* Dq + D4 of chunk j (MMA4 is issued
    // behind MMA3, as soon as Pg is there), transposed through a shared-memory tile and written with one TMA store
    // (row-masked stores for a ragged tail)
    const int tl = tid - 384;
    const uint32_t tm = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    // kNorm: the gate row of a token
    auto z_row = [&](int t) { return static_cast<const T*>(p.norm_gate) + (static_cast<int64_t>(t) * p.num_v_heads + hv) * kHeadDim; };
#pragma unroll 1
    for (int j = 0; (!kStateOnly || (kAux && p.v_new != nullptr)) && j < nproc; ++j) {
      const int t0 = seq_start + (first_chunk + j) * kChunk;
      const int valid = j < lead ? 0 : min(kChunk, seq_end - t0);  // nothing of a warm-up chunk is stored
      // two output tiles: the store of chunk j - 2 must have read this one.  kAux: one, and one for v_new: both stores of
      // chunk j - 1 must have read theirs
      uint8_t* so = smem + kOTiles + (kAux ? 0 : (j & 1) * 16384);
      if (j > (kAux ? 0 : 1)) {
        if (tl == 0) {
          if (kAux) ptx::tma_store_wait_read();
          else ptx::tma_store_wait_read_but1();
          ptx::mbar_arrive(&bars[kOFree]);
        }
        if (!wait(kOFree, (kAux ? j - 1 : j) & 1)) break;
      }
      if (kAux && p.v_new != nullptr) {
        // v_new = Vd: from the 16-bit copy in D2 (columns 16.. and 48.., two tokens each) through its own tile
        if (!wait(kVdStored, j & 1)) break;
        ptx::tc_fence_after_sync();
        const uint32_t tile = ptx::smem_u32(smem + kOffVn) + ((warp & 3) >> 1) * 8192;
        uint32_t x[2][2][8];
#pragma unroll
        for (int half = 0; half < 2; ++half)
#pragma unroll
          for (int th = 0; th < 2; ++th)
            ptx::tmem_ld_pack4(tm + (static_cast<uint32_t>(16 * half) << 16) + kColD2 + 16 + 32 * th, x[half][th]);
        ptx::tmem_wait_ld();
        ptx::tc_fence_before_sync();
        warp_arrive(&bars[kVnRead], lane);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int c16 = (warp & 1) * 4 + half * 2 + ((lane >> 3) & 1);
#pragma unroll
          for (int e = 0; e < 8; e += 2) {  // tokens 8 e .. 8 e + 15
            const uint32_t(&y)[4] = reinterpret_cast<const uint32_t(&)[4]>(x[half][e >> 2][2 * (e & 3)]);
            ptx::stmatrix_x4_trans(tile + ptx::sw128_offset(8 * (e + (lane >> 4)) + (lane & 7), c16), y);
          }
        }
        ptx::fence_proxy_async_smem();
        warp_arrive(&bars[kVnReady], lane);
        if (warp == 12 || (valid > 0 && valid < kChunk)) {
          if (!wait(kVnReady, j & 1)) break;
        }
        if (valid == kChunk) {
          if (tl == 0) {
            ptx::tma_store_4d(&tm_vn, smem + kOffVn, 0, hv, t0, 0);
            ptx::tma_store_commit();
          }
          __syncwarp();
        } else {
#pragma unroll 1
          for (int row = tl >> 4; row < valid; row += 8)
            *reinterpret_cast<uint4*>(static_cast<T*>(p.v_new) + (static_cast<int64_t>(t0 + row) * p.num_v_heads + hv) * kHeadDim +
                                      (tl & 15) * 8) =
                *reinterpret_cast<const uint4*>(smem + kOffVn + (tl & 8) * 1024 + ptx::sw128_offset(row, tl & 7));
        }
      }
      if (kStateOnly) continue;
      if (!wait(kD4Done, j & 1)) break;
      ptx::tc_fence_after_sync();
      if (warp == 12) trace(2, j, 6);
      // 16 lanes (columns v) x 64 tokens at a time in the fragment layout of 8 x 8 matrices, which stmatrix writes
      // transposed: 8 conflict-free stores per warp instead of 64 two-byte ones per thread
      // (all of s gamma first: nothing moves across the asm blocks below, and a load in front of each store would
      // expose its latency every time)
      float2 sg[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) sg[e] = *reinterpret_cast<const float2*>(&gates_of(j)->sgamma[2 * (lane & 3) + 8 * e]);
#pragma unroll 1
      for (int h16 = 0; h16 < 32; h16 += 16) {
        uint32_t r[32], q[32];
        const uint32_t lane16 = static_cast<uint32_t>(h16) << 16;
        ptx::tmem_ld_frag8(tm + lane16 + kColDq + (j & 1) * 64, q);
        ptx::tmem_ld_frag8(tm + lane16 + kColD4, r);
        ptx::tmem_wait_ld();
        const int c16 = (warp & 3) * 4 + h16 / 8 + ((lane >> 3) & 1);  // 16-byte piece of a token row
        const uint32_t half = ptx::smem_u32(so) + (c16 >> 3) * 8192;
#pragma unroll
        for (int e = 0; e < 8; e += 2) {  // tokens 8 e .. 8 e + 15
          uint32_t m[4];
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            const int y = 4 * (e + (x >> 1)) + 2 * (x & 1);
            const float2 g = sg[e + (x >> 1)];
            m[x] = pack2<T>(fmaf(g.x, __uint_as_float(q[y]), __uint_as_float(r[y])),
                            fmaf(g.y, __uint_as_float(q[y + 1]), __uint_as_float(r[y + 1])));
          }
          ptx::stmatrix_x4_trans(half + ptx::sw128_offset(8 * (e + (lane >> 4)) + (lane & 7), c16 & 7), m);
        }
      }
      ptx::tc_fence_before_sync();
      warp_arrive(&bars[kORead], lane);  // Dq and D4 may be overwritten
      if (warp == 12) trace(2, j, 12);
      ptx::fence_proxy_async_smem();
      // kNorm: the Pg warps have to be through with the previous tile first, so that they never fall two phases behind
      if (kNorm && j > 0 && !wait(kONormed, (j - 1) & 1)) break;
      warp_arrive(&bars[kOReady], lane);
      if (kNorm) {
        // gated RMS norm of the finished tile, in place, half of its rows (the Pg warps take the others); the gate rows two
        // chunks ahead go to L2
        const int row2 = tl >> 1;
        if (t0 + 2 * kChunk + row2 < seq_end) ptx::prefetch_l2(z_row(t0 + 2 * kChunk + row2) + (tl & 1) * 64);
        if (!norm_rows<T>(ptx::smem_u32(so), z_row(t0), p.num_v_heads * kHeadDim, p.norm_weight, p.norm_eps, valid, 0,
                          bar0 + 8u * kOReady, j & 1))
          break;
        ptx::fence_proxy_async_smem();
        warp_arrive(&bars[kONormed], lane);
      }
      if (valid == kChunk || valid == 0) {
        // Only the issuing warp waits for the tile to be complete, in a warm-up chunk too: the wait is also what keeps it
        // from arriving on kOFree twice while another output warp has still to look at the first arrival.
        if (warp == 12) {
          if (!wait(kTileDone, j & 1)) break;
          if (lane == 0 && valid > 0) {
            ptx::tma_store_4d(&tm_o, so, 0, hv, t0, 0);
            ptx::tma_store_commit();
          }
          __syncwarp();
        }
      } else {
        if (!wait(kTileDone, j & 1)) break;
        // ragged tail (always the last chunk of a sequence): row-masked 16-byte stores, 16 threads per row
        T* ob = static_cast<T*>(p.o);
#pragma unroll 1
        for (int row = tl >> 4; row < valid; row += 8) {
          const uint4 x = *reinterpret_cast<const uint4*>(so + (tl & 8) * 1024 + ptx::sw128_offset(row, tl & 7));
          *reinterpret_cast<uint4*>(ob + (static_cast<int64_t>(t0 + row) * p.num_v_heads + hv) * kHeadDim + (tl & 15) * 8) = x;
        }
      }
    }
    if ((!kStateOnly || kAux) && tl == 0) ptx::tma_store_wait_all();
  } else if (warp >= 10) {
    // =========================================================== Ab = A diag(beta), in place in the stage's A tile
    // (B operand of MMAu).  A is lower triangular: row r ends in 16-byte piece r / 8, what lies behind is zero (or
    // belongs to tokens past the end, whose rows nothing reads).  Six pieces per lane: warp 11 rows 32..63 pieces
    // 2..7, warp 10 the first two of those rows and the four of rows 0..31.
#pragma unroll 1
    for (int j = 0; !kWIn && !zero_v && j < nproc; ++j) {
      const int sj = j & 1;
      if (!wait(kGate0 + (j & 3), (j >> 2) & 1)) break;
      if (!wait(kVaFull0 + sj, (j >> 1) & 1)) break;
      const float* beta = gates_of(j)->beta;
      uint8_t* at = stage_ptr(sj) + kStageA;
#pragma unroll 3
      for (int x = 0; x < 6; ++x) {
        const bool low = warp == 10 && x < 4;
        const int c16 = (warp == 11) ? x + 2 : (low ? x : x - 4);
        uint4* ptr = reinterpret_cast<uint4*>(at + ptx::sw128_offset(low ? lane : 32 + lane, c16));
        uint4 raw = *ptr;
        const float4 b0 = *reinterpret_cast<const float4*>(&beta[c16 * 8]);
        const float4 b1 = *reinterpret_cast<const float4*>(&beta[c16 * 8 + 4]);
        const T* e = reinterpret_cast<const T*>(&raw);
        raw = make_uint4(pack2<T>(Cvt<T>::to_f32(e[0]) * b0.x, Cvt<T>::to_f32(e[1]) * b0.y),
                         pack2<T>(Cvt<T>::to_f32(e[2]) * b0.z, Cvt<T>::to_f32(e[3]) * b0.w),
                         pack2<T>(Cvt<T>::to_f32(e[4]) * b1.x, Cvt<T>::to_f32(e[5]) * b1.y),
                         pack2<T>(Cvt<T>::to_f32(e[6]) * b1.z, Cvt<T>::to_f32(e[7]) * b1.w));
        *ptr = raw;
      }
      ptx::fence_proxy_async_smem();
      // one barrier per stage: these warps run one chunk ahead, and a waiter must never fall two phases behind
      // (MMAu's commit releases the tile)
      warp_arrive(&bars[kAbReady0 + sj], lane);
    }
  } else {
    // =========================================================== chain warpgroups
    const int wg = warp >> 2;              // 0: tokens 0..31 of Vd, state columns 0..63; 1: the others
    const int v = tid & 127;               // TMEM lane = state column
    const uint32_t tm = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const int col_half = wg * 64;          // this warpgroup converts state columns [col_half, col_half + 64)
    bool alive = true;
    // states are fp32 or bf16 (state pools of the recurrent op); the slot of a sequence comes from h0_map /
    // seq_map, so that a serving loop can prefill straight from and into its pool
    constexpr bool st16 = kState16;
    const int64_t fs_off = (static_cast<int64_t>(out_row) * p.num_v_heads + hv) * kHeadDim * kHeadDim;
    const bool fs16 = st16 && !pass_b;  // (transition matrices are always fp32)
    float* fs_out = (final_state != nullptr && out_row >= 0 && !fs16) ? static_cast<float*>(final_state) + fs_off : nullptr;
    __nv_bfloat16* fs_out16 =
        (final_state != nullptr && out_row >= 0 && fs16) ? static_cast<__nv_bfloat16*>(final_state) + fs_off : nullptr;
    const int h0_row = p.h0_map != nullptr ? p.h0_map[seq] : seq;
    const bool h0_16 = st16 && !p.h0_kv;
    const bool h0_vk = p.transpose_state && !p.h0_kv;  // rows of h0 are [V][K]
    // [V][K] states move in 16-byte pieces where the caller's tensor starts on 16 bytes, one by one where it does not
    const bool h0_vec = (reinterpret_cast<uintptr_t>(p.h0) & 15u) == 0, fs_vec = (reinterpret_cast<uintptr_t>(final_state) & 15u) == 0;
    const int64_t h0_off = (static_cast<int64_t>(h0_row) * p.num_v_heads + hv) * kHeadDim * kHeadDim;
    const bool has_h0 = !init_identity && p.h0 != nullptr && h0_row >= 0 && lead == 0;
    const float* h0p = (has_h0 && !h0_16) ? static_cast<const float*>(p.h0) + h0_off : nullptr;
    const __nv_bfloat16* h0p16 = (has_h0 && h0_16) ? static_cast<const __nv_bfloat16*>(p.h0) + h0_off : nullptr;
    // 16 values k0 .. k0 + 15 of state column v: [V][K] rows in 16-byte pieces, [K][V] one coalesced store per k
    auto store_final16 = [&](int k0, const uint32_t (&x)[16]) {
      if (!kState16 || fs_out != nullptr) {
        if (p.transpose_state && fs_vec) {
          float4* dst = reinterpret_cast<float4*>(fs_out + v * kHeadDim + k0);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            dst[j] = make_float4(__uint_as_float(x[4 * j]), __uint_as_float(x[4 * j + 1]), __uint_as_float(x[4 * j + 2]),
                                 __uint_as_float(x[4 * j + 3]));
        } else if (p.transpose_state) {
#pragma unroll
          for (int j = 0; j < 16; ++j) fs_out[v * kHeadDim + k0 + j] = __uint_as_float(x[j]);
        } else {
          float* dst = fs_out + k0 * kHeadDim + v;
#pragma unroll
          for (int j = 0; j < 16; ++j) dst[j * kHeadDim] = __uint_as_float(x[j]);
        }
      } else if (fs_out16 != nullptr) {
        if (p.transpose_state && fs_vec) {
          uint4* dst = reinterpret_cast<uint4*>(fs_out16 + v * kHeadDim + k0);
#pragma unroll
          for (int j = 0; j < 2; ++j)
            dst[j] = make_uint4(pack2<__nv_bfloat16>(__uint_as_float(x[8 * j]), __uint_as_float(x[8 * j + 1])),
                                pack2<__nv_bfloat16>(__uint_as_float(x[8 * j + 2]), __uint_as_float(x[8 * j + 3])),
                                pack2<__nv_bfloat16>(__uint_as_float(x[8 * j + 4]), __uint_as_float(x[8 * j + 5])),
                                pack2<__nv_bfloat16>(__uint_as_float(x[8 * j + 6]), __uint_as_float(x[8 * j + 7])));
        } else if (p.transpose_state) {
#pragma unroll
          for (int j = 0; j < 16; ++j) fs_out16[v * kHeadDim + k0 + j] = __float2bfloat16_rn(__uint_as_float(x[j]));
        } else {
          __nv_bfloat16* dst = fs_out16 + k0 * kHeadDim + v;
#pragma unroll
          for (int j = 0; j < 16; ++j) dst[j * kHeadDim] = __float2bfloat16_rn(__uint_as_float(x[j]));
        }
      }
    };
    const bool write_final = fs_out != nullptr || (kState16 && fs_out16 != nullptr);

    // ---- initial state: S = exp(gL_0) * S_init (fp32) and its 16-bit copy.  This thread's 64 values are requested
    // before anything is waited for: their latency then overlaps the arrival of the first stage instead of
    // following it (with context-parallel segments of a dozen chunks a CTA's start-up is a tenth of its life).
    {
      float x[64];
      if (h0p != nullptr && !h0_vk) {  // [K][V]: consecutive lanes read consecutive floats of row k
        const float* src = h0p + col_half * kHeadDim + v;
#pragma unroll
        for (int j = 0; j < 64; ++j) x[j] = src[j * kHeadDim];
      } else if (h0p != nullptr && !h0_vec) {
        const float* src = h0p + v * kHeadDim + col_half;
#pragma unroll
        for (int j = 0; j < 64; ++j) x[j] = src[j];
      } else if (h0p != nullptr) {  // [V][K]: 16-byte pieces of row v
        const float4* src = reinterpret_cast<const float4*>(h0p + v * kHeadDim + col_half);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float4 f = src[j];
          x[4 * j] = f.x; x[4 * j + 1] = f.y; x[4 * j + 2] = f.z; x[4 * j + 3] = f.w;
        }
      } else if (kState16 && h0p16 != nullptr && !h0_vk) {
        const __nv_bfloat16* src = h0p16 + col_half * kHeadDim + v;
#pragma unroll
        for (int j = 0; j < 64; ++j) x[j] = __bfloat162float(src[j * kHeadDim]);
      } else if (kState16 && h0p16 != nullptr && !h0_vec) {
        const __nv_bfloat16* src = h0p16 + v * kHeadDim + col_half;
#pragma unroll
        for (int j = 0; j < 64; ++j) x[j] = __bfloat162float(src[j]);
      } else if (kState16 && h0p16 != nullptr) {
        const uint4* src = reinterpret_cast<const uint4*>(h0p16 + v * kHeadDim + col_half);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint4 raw = src[j];
          const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&raw);
#pragma unroll
          for (int y = 0; y < 8; ++y) x[8 * j + y] = __bfloat162float(e[y]);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 64; ++j) x[j] = (init_identity && col_half + j == v) ? 1.f : 0.f;
      }
      float egl0 = 1.f;
      if (nproc > 0) {
        alive = wait(kGate0, 0);
        egl0 = gates_of(0)->egl;
      }
#pragma unroll
      for (int kb = 0; kb < 64; kb += 16) {
        uint32_t sf[16], sb[8];
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          sf[j] = __float_as_uint(x[kb + j] * egl0);
          sf[j + 1] = __float_as_uint(x[kb + j + 1] * egl0);
          sb[j >> 1] = pack2<T>(x[kb + j], x[kb + j + 1]);
        }
        ptx::tmem_st16(tm + kColS + col_half + kb, sf);
        ptx::tmem_st8(tm + kColSbf + (col_half + kb) / 2, sb);
        if (nproc == 0 && write_final) {  // (an empty sequence: egl0 is 1, sf holds the initial state itself)
          store_final16(col_half + kb, sf);
        }
      }
      ptx::tmem_wait_st();
      ptx::tc_fence_before_sync();
      warp_arrive(&bars[kSbfReady], lane);
      warp_arrive(&bars[kSScaled], lane);
    }

#pragma unroll 1
    for (int i = 0; alive && i < nproc; ++i) {
      const int ph = i & 1;
      const int chunk = first_chunk + i;
      const int t0 = seq_start + chunk * kChunk;
      const Gates* gs = gates_of(i);
      // (the gates of chunk i are visible: convert (b) of the previous iteration waited for this ring slot)

      // ---------------- V' = rho .* Vd of this warpgroup's 32 tokens back into tensor memory (the first 16 of their own
      // 32 columns of D2; MMA3 waits for it), then Vd itself for MMA4 (and v_new).
      const int c0 = wg * 32;
      if (!(alive = wait(kD2Done, ph))) break;
      ptx::tc_fence_after_sync();
      if (warp == 0) trace(1, i, 2);
      {
        uint32_t d[32], vp[16];
        ptx::tmem_ld32(tm + kColD2 + c0, d);
        ptx::tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const float4 r4 = *reinterpret_cast<const float4*>(&gs->rho[c0 + j]);
          vp[j >> 1] = pack2<T>(mul2(f2(d[j], d[j + 1]), f2(r4.x, r4.y)));
          vp[(j >> 1) + 1] = pack2<T>(mul2(f2(d[j + 2], d[j + 3]), f2(r4.z, r4.w)));
        }
        ptx::tmem_st16(tm + kColD2 + c0, vp);
        ptx::tmem_wait_st();
        ptx::tc_fence_before_sync();
        warp_arrive(&bars[kVdReady], lane);
        if (warp == 0) trace(1, i, 3);
        // off the critical path: Vd itself, 16 bit, into the other 16 columns of its half (A operand of MMA4, source of
        // v_new).  Only where one of them waits for it: MMAu of the next chunk, which overwrites D2, is held back by them.
        if (!kStateOnly || (kAux && p.v_new != nullptr)) {
          uint32_t vd[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) vd[j] = pack2<T>(__uint_as_float(d[2 * j]), __uint_as_float(d[2 * j + 1]));
          ptx::tmem_st16(tm + kColD2 + c0 + 16, vd);
          ptx::tmem_wait_st();
          ptx::tc_fence_before_sync();
          warp_arrive(&bars[kVdStored], lane);
        }
      }

      // ---------------- state convert after MMA3 (this warpgroup's 64 columns)
      if (!(alive = wait(kSDone, ph))) break;
      ptx::tc_fence_after_sync();
      if (warp == 0) trace(1, i, 4);
      const bool last = (i + 1 == nproc);
      if (last) {
        if (write_final) {
#pragma unroll 1
          for (int kb = 0; kb < 64; kb += 16) {
            uint32_t sf[16];
            ptx::tmem_ld16(tm + kColS + col_half + kb, sf);
            ptx::tmem_wait_ld();
            store_final16(col_half + kb, sf);
          }
        }
      } else {
        // (kAux: h of this chunk has been read out of the 16-bit copy)
        if (kAux && p.h != nullptr && !(alive = wait(kHRead, ph))) break;
        // (a) critical: 16-bit copy of the new state -> MMA2 of the next chunk may start
        uint32_t sf[64];
        ptx::tmem_ld32(tm + kColS + col_half, reinterpret_cast<uint32_t(&)[32]>(sf[0]));
        ptx::tmem_ld32(tm + kColS + col_half + 32, reinterpret_cast<uint32_t(&)[32]>(sf[32]));
        ptx::tmem_wait_ld();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t sb[16];
#pragma unroll
          for (int j = 0; j < 32; j += 2)
            sb[j >> 1] = pack2<T>(__uint_as_float(sf[32 * h + j]), __uint_as_float(sf[32 * h + j + 1]));
          ptx::tmem_st16(tm + kColSbf + col_half / 2 + 16 * h, sb);
        }
        ptx::tmem_wait_st();
        ptx::tc_fence_before_sync();
        warp_arrive(&bars[kSbfReady], lane);
        if (warp == 0) trace(1, i, 5);
        // (b) off the critical path: decay of the fp32 state for the next chunk (needed by MMA3 only).  In pairs: half the
        // instructions (the output epilogue gained nothing from them, or lost: 540 k packed tokens of 8 / 8 heads 972 -> 978 us)
        if (!(alive = wait(kGate0 + ((i + 1) & 3), ((i + 1) >> 2) & 1))) break;
        const float egl_next = gates_of(i + 1)->egl;
#pragma unroll
        for (int j = 0; j < 64; j += 2) {
          const float2 y = unpack(mul2(f2(sf[j], sf[j + 1]), f2(egl_next, egl_next)));
          sf[j] = __float_as_uint(y.x);
          sf[j + 1] = __float_as_uint(y.y);
        }
        ptx::tmem_st32(tm + kColS + col_half, reinterpret_cast<const uint32_t(&)[32]>(sf[0]));
        ptx::tmem_st32(tm + kColS + col_half + 32, reinterpret_cast<const uint32_t(&)[32]>(sf[32]));
        ptx::tmem_wait_st();
        ptx::tc_fence_before_sync();
        warp_arrive(&bars[kSScaled], lane);
      }
    }
  }

  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 8) ptx::tmem_dealloc(tmem, 512);
  if (cta_trace && tid == 0) p.trace[cta_slot + 1] = static_cast<long long>(ptx::global_timer_ns());
}

}  // namespace

int launch_chunk_fwd(const FwdParams& p, const void* q, const void* k, const void* v, const void* A,
                     const void* w, bool w_in_scan, int64_t total_tokens, bool is_bf16, bool state_only, cudaStream_t stream) {
  CUtensorMap tm_q, tm_k, tm_v, tm_a, tm_w, tm_o, tm_vn, tm_h;
  int rc;
  const bool aux = p.h != nullptr || p.v_new != nullptr;
  if ((rc = make_tmap_halves(&tm_k, k, total_tokens, p.num_k_heads, 64, is_bf16)) != QLA_OK) return rc;
  if ((rc = make_tmap_halves(&tm_q, state_only ? k : q, total_tokens, p.num_k_heads, 64, is_bf16)) != QLA_OK) return rc;
  if ((rc = make_tmap_halves(&tm_v, v, total_tokens, p.num_v_heads, 64, is_bf16)) != QLA_OK) return rc;
  if ((rc = make_tmap_3d(&tm_a, A, total_tokens, p.num_v_heads, 64, 64, 64, true, is_bf16)) != QLA_OK) return rc;
  rc = w_in_scan ? make_tmap_3d(&tm_w, w, total_tokens, p.num_v_heads, 64, 64, 64, true, is_bf16)
                 : make_tmap_halves(&tm_w, w, total_tokens, p.num_v_heads, 64, is_bf16);
  if (rc != QLA_OK) return rc;
  if ((rc = make_tmap_halves(&tm_o, state_only ? v : p.o, total_tokens, p.num_v_heads, 64, is_bf16)) != QLA_OK) return rc;
  tm_vn = tm_h = tm_o;
  if (p.v_new != nullptr && (rc = make_tmap_halves(&tm_vn, p.v_new, total_tokens, p.num_v_heads, 64, is_bf16)) != QLA_OK) return rc;
  // h as rows [chunks * Hv * 128][128] (the number of chunks is only known to be at most this)
  const uint64_t h_rows = (static_cast<uint64_t>(total_tokens) / kChunk + p.num_seqs) * p.num_v_heads * kHeadDim;
  if (p.h != nullptr && (rc = make_tmap_halves(&tm_h, p.h, h_rows, 1, 64, is_bf16)) != QLA_OK) return rc;
  const unsigned grid = static_cast<unsigned>(p.num_seqs) * p.num_v_heads * (p.dual ? 2 : 1);
#define QLA_LAUNCH_FWD(BYTES, ...)                                                                                             \
  do {                                                                                                                         \
    const int rc_ = ensure_dynamic_smem<chunk_fwd_kernel<__VA_ARGS__>>(BYTES);                                                 \
    if (rc_ != QLA_OK) return rc_;                                                                                             \
    QLA_CHECK_CUDA(launch_dependent(chunk_fwd_kernel<__VA_ARGS__>, dim3(grid), dim3(kThreads), BYTES, stream, tm_q, tm_k, tm_v, \
                                    tm_a, tm_w, tm_o, tm_vn, tm_h, p));                                                        \
  } while (0)
#define QLA_DISPATCH_FWD(T)                                                                                   \
  do {                                                                                                        \
    if (w_in_scan && p.state_dtype == QLA_DT_BF16) QLA_LAUNCH_FWD(kSmemBytesWIn, T, false, false, false, false, true, true); \
    else if (w_in_scan && p.norm_gate != nullptr) QLA_LAUNCH_FWD(kSmemBytesWIn, T, false, false, false, true, false, true);  \
    else if (w_in_scan && state_only) QLA_LAUNCH_FWD(kSmemBytesWIn, T, true, false, false, false, false, true);    \
    else if (w_in_scan && traced) QLA_LAUNCH_FWD(kSmemBytesWIn, T, false, false, true, false, false, true);   \
    else if (w_in_scan) QLA_LAUNCH_FWD(kSmemBytesWIn, T, false, false, false, false, false, true);                 \
    else if (p.state_dtype == QLA_DT_BF16) QLA_LAUNCH_FWD(kSmemBytes, T, false, false, false, false, true);   \
    else if (p.norm_gate != nullptr) QLA_LAUNCH_FWD(kSmemBytes, T, false, false, false, true);                \
    else if (traced) QLA_LAUNCH_FWD(kSmemBytes, T, false, false, true);                                       \
    else if (state_only && aux) QLA_LAUNCH_FWD(kSmemBytesAux, T, true, true, false);                          \
    else if (state_only) QLA_LAUNCH_FWD(kSmemBytes, T, true, false, false);                                   \
    else if (aux) QLA_LAUNCH_FWD(kSmemBytesAux, T, false, true, false);                                       \
    else QLA_LAUNCH_FWD(kSmemBytes, T, false, false, false);                                                  \
  } while (0)
  // the traced variant (plain full forward only) is a separate instantiation so that normal launches
  // carry no tracing code
  const bool traced = p.trace != nullptr && !state_only && !aux;
  if (is_bf16) QLA_DISPATCH_FWD(__nv_bfloat16);
  else QLA_DISPATCH_FWD(__half);
#undef QLA_DISPATCH_FWD
#undef QLA_LAUNCH_FWD
  QLA_CHECK_CUDA(cudaGetLastError());
  return QLA_OK;
}

void launch_info_chunk_fwd_kernel(bool aux, bool w_in_scan, int* block_threads, size_t* dynamic_smem_bytes) {
  *block_threads = kThreads;
  *dynamic_smem_bytes = aux ? kSmemBytesAux : w_in_scan ? kSmemBytesWIn : kSmemBytes;
}

}  // namespace qla
