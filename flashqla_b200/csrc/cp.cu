// Intra-card context parallelism for the chunked forward: a long sequence is cut into segments that
// run as independent CTAs; each non-final segment first produces the state it hands to its successor.
// Reference: flash_qla/ops/gated_delta_rule/chunk/cp_context.py:117-176 (orchestration),
// chunk/hopper/cp_fwd.py:7-63 (warm-up lengths) and :102-250 (chaining of the initial states).
//
//   plan  : per (segment, head) walk the chunk-end gates backwards from the segment end until the
//           accumulated log decay drops below `threshold`; that many trailing chunks, started from a
//           zero state, reproduce the segment-end state to exp(threshold).  If the whole segment does
//           not decay that far the (segment, head) is a "fallback": all chunks are run and the exact
//           K x K transition matrix M of the segment is needed as well.
//   chain : for fallback entries  h0[seg + 1] += M[seg] * h0[seg], in segment order.
#include "chunk_params.cuh"

namespace qla {
namespace {

// Warm-up length of a segment, found by one warp: lanes take 32 consecutive chunk-end gates at a time, so that a
// segment costs one memory latency per 32 chunks (one thread that walked them paid it per chunk: 38 us of a
// 36-segment plan with weak gates).  Returns the number of chunks; *reached says whether the decay passed the threshold.
__device__ __forceinline__ int warm_chunks(const QlaCpPlanArgs& a, int start, int end, int h, bool* reached) {
  const int lane = threadIdx.x & 31;
  const int nchunks = (end - start + kChunk - 1) / kChunk;
  float carry = 0.f;
  for (int i0 = 0; i0 < nchunks; i0 += 32) {
    const int i = i0 + lane;
    float acc = 0.f;
    if (i < nchunks) {
      const int c = a.reverse ? i : nchunks - 1 - i;  // backward: the decay accumulates from the segment's start
      const int last = min(end, start + (c + 1) * kChunk) - 1;
      acc = a.g_cumsum[static_cast<int64_t>(last) * a.num_v_heads + h];
    }
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const float n = __shfl_up_sync(0xffffffffu, acc, off);
      if (lane >= off) acc += n;
    }
    acc += carry;
    const unsigned below = __ballot_sync(0xffffffffu, i < nchunks && acc < a.threshold);
    if (below != 0) {
      *reached = true;
      return i0 + __ffs(below);
    }
    carry = __shfl_sync(0xffffffffu, acc, 31);
  }
  *reached = false;
  return nchunks;
}

constexpr int kPlanThreads = 512;

// A state of the caller's (fp32 or bf16, [K][V] or [V][K]) as fp32 [K][V]; no row: zero.  All kPlanThreads threads.
__device__ __forceinline__ void copy_state(const QlaCpPlanArgs& a, float* dst, int row, int h) {
  constexpr int kElems = kHeadDim * kHeadDim;
  if (row < 0) {
    for (int i = threadIdx.x * 4; i < kElems; i += kPlanThreads * 4)
      *reinterpret_cast<float4*>(dst + i) = make_float4(0.f, 0.f, 0.f, 0.f);
    return;
  }
  const int64_t off = (static_cast<int64_t>(row) * a.num_v_heads + h) * kElems;
  const float* s32 = static_cast<const float*>(a.h0) + off;
  const __nv_bfloat16* s16 = static_cast<const __nv_bfloat16*>(a.h0) + off;
  const bool b16 = a.h0_dtype == QLA_DT_BF16;
  if (!a.h0_transposed) {
#pragma unroll 4
    for (int i = threadIdx.x; i < kElems; i += kPlanThreads) dst[i] = b16 ? __bfloat162float(s16[i]) : s32[i];
    return;
  }
  // transposed through shared memory, 64 source rows at a time: both sides coalesced
  __shared__ float tile[64][kHeadDim + 1];
  for (int v0 = 0; v0 < kHeadDim; v0 += 64) {
    __syncthreads();
#pragma unroll 4
    for (int i = threadIdx.x; i < 64 * kHeadDim; i += kPlanThreads)
      tile[i >> 7][i & 127] = b16 ? __bfloat162float(s16[v0 * kHeadDim + i]) : s32[v0 * kHeadDim + i];
    __syncthreads();
#pragma unroll 4
    for (int i = threadIdx.x; i < 64 * kHeadDim; i += kPlanThreads)
      dst[(i >> 6) * kHeadDim + v0 + (i & 63)] = tile[i & 63][i >> 6];
  }
}

// One CTA per (segment, head): warp 0 finds the warm-up length; all threads write the segment's start state.
__global__ void __launch_bounds__(kPlanThreads) cp_plan_kernel(const QlaCpPlanArgs a) {
  grid_dep_wait();    // earlier kernels of the stream have completed (see launch_dependent)
  grid_dep_launch();
  const int seg = blockIdx.x, h = blockIdx.y;
  const int num_heads = a.num_v_heads;
  if (threadIdx.x < 32) {
    const int start = a.cu_seqlens[seg], end = a.cu_seqlens[seg + 1];
    int warm = 0, ml = 0;
    if (a.seg_next[seg] >= 0 && end > start) {
      bool reached;
      warm = warm_chunks(a, start, end, h, &reached);
      if (!reached) ml = warm;
    }
    if (threadIdx.x == 0) {
      a.warm_limit[seg * num_heads + h] = warm;
      a.m_limit[seg * num_heads + h] = ml;
    }
  }
  if (a.cp_h0 == nullptr) return;
  const int raw = a.seg_start_of[seg];
  int row = -1;
  if (raw >= 0 && a.h0 != nullptr) row = a.h0_map != nullptr ? a.h0_map[raw] : raw;
  copy_state(a, a.cp_h0 + (static_cast<int64_t>(seg) * num_heads + h) * kHeadDim * kHeadDim, row, h);
}

// The plan with the warm-up folded into the main scan (forward, or reverse for the backward scan): one CTA per
// (original sequence, head), a warp per segment.  A (sequence, head) in which every segment decays below the threshold needs no state-only pass:
// the main scan's CTA of segment s simply starts lead[s] = warm(s - 1) chunks early, from a zero state.  If some
// segment never decays that far the limits are those of cp_plan_kernel (state-only pass, transition matrices,
// chain) and lead is 0.  Only the row of cp_h0 that starts the sequence is written here.
__global__ void __launch_bounds__(kPlanThreads) cp_plan_lead_kernel(const QlaCpPlanArgs a) {
  grid_dep_wait();
  grid_dep_launch();
  const int r = blockIdx.x, h = blockIdx.y;
  const int num_heads = a.num_v_heads;
  const int s0 = a.raw_first_seg[r], s1 = a.raw_first_seg[r + 1];
  int any = 0;
  for (int seg = s0 + static_cast<int>(threadIdx.x >> 5); seg < s1; seg += kPlanThreads / 32) {
    const int start = a.cu_seqlens[seg], end = a.cu_seqlens[seg + 1];
    int warm = 0, ml = 0;
    if (a.seg_next[seg] >= 0 && end > start) {
      bool reached;
      warm = warm_chunks(a, start, end, h, &reached);
      if (!reached) ml = warm;
    }
    if ((threadIdx.x & 31) == 0) {
      a.warm_limit[seg * num_heads + h] = warm;
      a.m_limit[seg * num_heads + h] = ml;
    }
    any |= ml;
  }
  any = __syncthreads_or(any);  // (also orders the limits written above before the reads below)
  // the neighbour whose warm-up this segment's scan runs itself: the segment before it (forward), behind it (backward)
  for (int seg = s0 + threadIdx.x; seg < s1; seg += kPlanThreads) {
    const int nb = a.reverse ? seg + 1 : seg - 1;
    a.lead[seg * num_heads + h] = (!any && nb >= s0 && nb < s1) ? a.warm_limit[nb * num_heads + h] : 0;
  }
  __syncthreads();
  if (!any)
    for (int seg = s0 + threadIdx.x; seg < s1; seg += kPlanThreads) a.warm_limit[seg * num_heads + h] = 0;
  // start state of the sequence (backward: the gradient of its final state, into the last segment's row): the
  // caller's (any dtype / layout, through h0_map) or zero
  int row = -1;
  if (a.h0 != nullptr) row = a.h0_map != nullptr ? a.h0_map[r] : r;
  copy_state(a, a.cp_h0 + (static_cast<int64_t>(a.reverse ? s1 - 1 : s0) * num_heads + h) * kHeadDim * kHeadDim, row, h);
}

// The chain  h[next] += M[seg] h[seg]  over the segments of one sequence and head, in order.  A link is a dependent
// 128 x 128 by 128 x 8 product: the columns are split over CTAs (8 each), warp w of a CTA has rows 16 w .. 16 w + 15.  The
// product runs on mma.sync with both operands split into two TF32 values (hi hi + hi lo + lo hi: 2^-22 of a product, beside
// fp32 sums of 128 terms).  A warp's rows of M come straight from global memory (L2) as fragments, those of the next
// link while this one is multiplied; the carried columns pass through shared memory, split by the thread that
// formed them, in two buffers: one barrier per link.  What bounds it: 64 KB of M per link and CTA, L2 to SM (40 bytes per ns
// and SM).  36 links of 4 heads take 59 us; with fp32 products from shared memory and seven barriers per link they took 96.
constexpr int kChainCols = 8;
constexpr int kChainStride = 144;  // floats from column to column of the carried state: conflict-free float4 fragments
constexpr int kChainThreads = 256;
constexpr int kChainFlags = 256;

// x = hi + lo, both TF32 (Veltkamp's splitting; lo loses what lies below 2^-22 of x)
__device__ __forceinline__ void split_tf32(float x, float& hi, float& lo) {
  const float c = __fmul_rn(x, 8193.f);
  hi = __fsub_rn(c, __fsub_rn(c, x));
  lo = __uint_as_float(__float_as_uint(__fsub_rn(x, hi)) & 0xffffe000u);
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const float (&a)[4], float b0, float b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(__float_as_uint(a[0])), "r"(__float_as_uint(a[1])), "r"(__float_as_uint(a[2])), "r"(__float_as_uint(a[3])),
        "r"(__float_as_uint(b0)), "r"(__float_as_uint(b1)));
}

__global__ void __launch_bounds__(kChainThreads, 1) cp_chain_kernel(float* __restrict__ h0, const float* __restrict__ M,
                                                                    const int32_t* __restrict__ m_limit,
                                                                    const int32_t* __restrict__ raw_first_seg, int num_heads,
                                                                    int reverse) {
  grid_dep_wait();
  grid_dep_launch();
  const int c0 = blockIdx.x * kChainCols, h = blockIdx.y, r = blockIdx.z, tid = threadIdx.x;
  const int s0 = raw_first_seg[r], links = raw_first_seg[r + 1] - s0 - 1;
  __shared__ __align__(16) float s_h[2][2][kChainCols * kChainStride];  // [buffer][hi | lo][column][row]
  __shared__ int flags[kChainFlags];
  // link i leads from segment seg_of(i) to seg_of(i + 1)
  auto seg_of = [&](int i) { return reverse ? s0 + links - i : s0 + i; };
  const int warp = tid >> 5, g = (tid & 31) >> 2, c = tid & 3;
  // this thread's values of a state: rows row and row + 8, columns c0 + 2 c, + 1 (fragment of the product's accumulator)
  const int row = 16 * warp + g;
  auto state_of = [&](int i) {
    return h0 + (static_cast<int64_t>(seg_of(i)) * num_heads + h) * kHeadDim * kHeadDim + row * kHeadDim + c0 + 2 * c;
  };
  auto load_state = [&](int i, float (&x)[4]) {
    const float* s = state_of(i);
    const float2 lo = *reinterpret_cast<const float2*>(s), hi = *reinterpret_cast<const float2*>(s + 8 * kHeadDim);
    x[0] = lo.x; x[1] = lo.y; x[2] = hi.x; x[3] = hi.y;
  };
  auto carry = [&](int buf, const float (&x)[4]) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float hi, lo;
      split_tf32(x[e], hi, lo);
      const int at = (2 * c + (e & 1)) * kChainStride + row + 8 * (e >> 1);
      s_h[buf][0][at] = hi;
      s_h[buf][1][at] = lo;
    }
  };
  // Rows row and row + 8 of M, columns 16 t + 4 c .. + 3: values 0, 1 are slots c, c + 4 of k-step 2 t, values 2, 3 of 2 t + 1.
  float4 raw[8][2];
  auto load_m = [&](int i) {
    const float* m = M + ((static_cast<int64_t>(seg_of(i)) * num_heads + h) * kHeadDim + row) * kHeadDim + 4 * c;
#pragma unroll
    for (int t = 0; t < 8; ++t)
#pragma unroll
      for (int x = 0; x < 2; ++x) raw[t][x] = *reinterpret_cast<const float4*>(m + 8 * x * kHeadDim + 16 * t);
  };
  int buf = 0;
  for (int b0 = 0; b0 < links; b0 += kChainFlags) {
    const int nb = min(kChainFlags, links - b0);
    int mine = 0;
    __syncthreads();
    for (int i = tid; i < nb; i += kChainThreads) mine |= (flags[i] = m_limit[seg_of(b0 + i) * num_heads + h]);
    // the usual case (every segment decays below the threshold) has nothing to chain
    if (__syncthreads_or(mine) == 0) continue;
    bool have_h = false;
    float add[4] = {0.f, 0.f, 0.f, 0.f};  // the next state as it is: what the product is added to
    if (flags[0] != 0) {
      load_m(b0);
      load_state(b0 + 1, add);
    }
    for (int i = 0; i < nb; ++i) {
      const bool next = i + 1 < nb && flags[i + 1] != 0;
      if (flags[i] == 0) {  // (uniform)
        have_h = false;
        if (next) {
          load_m(b0 + i + 1);
          load_state(b0 + i + 2, add);
        }
        continue;
      }
      if (!have_h) {
        float x[4];
        load_state(b0 + i, x);
        carry(buf, x);
      }
      have_h = true;
      float mh[16][4], ml[16][4];
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const float a[8] = {raw[t][0].x, raw[t][1].x, raw[t][0].y, raw[t][1].y, raw[t][0].z, raw[t][1].z, raw[t][0].w, raw[t][1].w};
#pragma unroll
        for (int e = 0; e < 8; ++e) split_tf32(a[e], mh[2 * t + (e >> 2)][e & 3], ml[2 * t + (e >> 2)][e & 3]);
      }
      float out[4] = {add[0], add[1], add[2], add[3]};
      if (next) {
        load_m(b0 + i + 1);
        load_state(b0 + i + 2, add);
      }
      __syncthreads();  // the carried columns are complete
      float acc[2][3][4] = {};
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const float4 xh = *reinterpret_cast<const float4*>(&s_h[buf][0][g * kChainStride + 16 * t + 4 * c]);
        const float4 xl = *reinterpret_cast<const float4*>(&s_h[buf][1][g * kChainStride + 16 * t + 4 * c]);
        mma_tf32(acc[0][0], ml[2 * t], xh.x, xh.y);
        mma_tf32(acc[0][1], mh[2 * t], xl.x, xl.y);
        mma_tf32(acc[0][2], mh[2 * t], xh.x, xh.y);
        mma_tf32(acc[1][0], ml[2 * t + 1], xh.z, xh.w);
        mma_tf32(acc[1][1], mh[2 * t + 1], xl.z, xl.w);
        mma_tf32(acc[1][2], mh[2 * t + 1], xh.z, xh.w);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e)
        out[e] += ((acc[0][0][e] + acc[1][0][e]) + (acc[0][1][e] + acc[1][1][e])) + (acc[0][2][e] + acc[1][2][e]);
      buf ^= 1;
      carry(buf, out);
      float* dst = state_of(b0 + i + 1);
      *reinterpret_cast<float2*>(dst) = make_float2(out[0], out[1]);
      *reinterpret_cast<float2*>(dst + 8 * kHeadDim) = make_float2(out[2], out[3]);
    }
    // (a link behind this batch reads the state written last, each value by the thread that wrote it)
  }
}

}  // namespace
}  // namespace qla

extern "C" QLA_API int qla_cp_plan(const QlaCpPlanArgs* a, void* stream) {
  using namespace qla;
  QLA_CHECK_ARG(a != nullptr && a->g_cumsum && a->cu_seqlens && a->seg_next && a->warm_limit && a->m_limit,
                "NULL pointer in QlaCpPlanArgs");
  QLA_CHECK_ARG(a->num_segments > 0 && a->num_v_heads > 0 && a->num_v_heads <= 65535, "bad sizes");
  QLA_CHECK_ARG(a->cp_h0 == nullptr || a->seg_start_of != nullptr, "cp_h0 needs seg_start_of");
  QLA_CHECK_SUPPORTED(a->h0 == nullptr || a->h0_dtype == QLA_DT_F32 || a->h0_dtype == QLA_DT_BF16,
                      "initial states must be fp32 or bf16");
  if (a->lead != nullptr) {
    QLA_CHECK_ARG(a->cp_h0 != nullptr && a->raw_first_seg != nullptr && a->num_raw_seqs > 0,
                  "lead needs cp_h0, raw_first_seg and num_raw_seqs");
    dim3 grid_lead(a->num_raw_seqs, a->num_v_heads);
    QLA_CHECK_CUDA(launch_dependent(cp_plan_lead_kernel, grid_lead, dim3(kPlanThreads), 0, static_cast<cudaStream_t>(stream), *a));
    return QLA_OK;
  }
  dim3 grid(a->num_segments, a->num_v_heads);
  QLA_CHECK_CUDA(launch_dependent(cp_plan_kernel, grid, dim3(kPlanThreads), 0, static_cast<cudaStream_t>(stream), *a));
  return QLA_OK;
}

extern "C" QLA_API int qla_cp_chain(const QlaCpChainArgs* a, void* stream) {
  using namespace qla;
  QLA_CHECK_ARG(a != nullptr && a->h0 && a->M && a->m_limit && a->raw_first_seg, "NULL pointer in QlaCpChainArgs");
  QLA_CHECK_ARG(a->num_raw_seqs > 0 && a->num_v_heads > 0, "bad sizes");
  dim3 grid(kHeadDim / kChainCols, a->num_v_heads, a->num_raw_seqs);
  QLA_CHECK_CUDA(launch_dependent(cp_chain_kernel, grid, dim3(kChainThreads), 0, static_cast<cudaStream_t>(stream), a->h0, a->M,
                                  a->m_limit, a->raw_first_seg, a->num_v_heads, a->reverse));
  return QLA_OK;
}
