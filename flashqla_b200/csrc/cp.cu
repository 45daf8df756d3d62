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
#include "warp_pieces.cuh"

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
// 128 x 128 by 128 x 8 product: the columns are split over CTAs (8 each), the matrices of the next links are already on
// their way into shared memory while one is multiplied (they are read once per CTA, from L2), and the carried columns
// stay in shared memory.  32 segments of one sequence: 36 us; with 32-column slabs, rows read from global memory in
// front of every product, the same chain took 950 us.
constexpr int kChainCols = 8;
constexpr int kChainStride = kHeadDim + 4;  // floats per row of M: 16-byte rows, conflict-free float4 reads
constexpr int kChainThreads = 256;
constexpr int kChainFlags = 256;
constexpr size_t kChainSmem = (2 * kHeadDim * kChainStride + 3 * kHeadDim * kChainCols) * sizeof(float);

__global__ void __launch_bounds__(kChainThreads) cp_chain_kernel(float* __restrict__ h0, const float* __restrict__ M,
                                                                 const int32_t* __restrict__ m_limit,
                                                                 const int32_t* __restrict__ raw_first_seg, int num_heads,
                                                                 int reverse) {
  grid_dep_wait();
  grid_dep_launch();
  const int c0 = blockIdx.x * kChainCols, h = blockIdx.y, r = blockIdx.z, tid = threadIdx.x;
  const int s0 = raw_first_seg[r], links = raw_first_seg[r + 1] - s0 - 1;
  extern __shared__ __align__(16) float chain_smem[];
  float* sM[2] = {chain_smem, chain_smem + kHeadDim * kChainStride};
  float* sH = chain_smem + 2 * kHeadDim * kChainStride;  // the carried columns [128][8]
  float* sP = sH + kHeadDim * kChainCols;                // partial sums [2][128][8]
  __shared__ int flags[kChainFlags];
  // link i leads from segment seg_of(i) to seg_of(i + 1)
  auto seg_of = [&](int i) { return reverse ? s0 + links - i : s0 + i; };
  auto state_of = [&](int i) { return h0 + (static_cast<int64_t>(seg_of(i)) * num_heads + h) * kHeadDim * kHeadDim + c0; };
  auto load_m = [&](int i, int buf) {
    const float* m = M + (static_cast<int64_t>(seg_of(i)) * num_heads + h) * kHeadDim * kHeadDim;
    for (int e = tid; e < kHeadDim * 32; e += kChainThreads)
      mm::cp_async16(sM[buf] + (e >> 5) * kChainStride + (e & 31) * 4, m + e * 4, true);
  };
  // thread: rows row, row + 32, row + 64, row + 96, columns cq .. cq + 3, a quarter of the inner dimension
  const int row = tid & 31, cq = ((tid >> 5) & 1) * 4, jq = tid >> 6;
  for (int b0 = 0; b0 < links; b0 += kChainFlags) {
    const int nb = min(kChainFlags, links - b0);
    int mine = 0;
    __syncthreads();
    for (int i = tid; i < nb; i += kChainThreads) mine |= (flags[i] = m_limit[seg_of(b0 + i) * num_heads + h]);
    // the usual case (every segment decays below the threshold) has nothing to chain
    if (__syncthreads_or(mine) == 0) continue;
    int buf = 0;
    bool have_h = false;
    if (flags[0] != 0) load_m(b0, 0);
    mm::cp_async_commit();
    for (int i = 0; i < nb; ++i, buf ^= 1) {
      if (i + 1 < nb && flags[i + 1] != 0) load_m(b0 + i + 1, buf ^ 1);
      mm::cp_async_commit();
      if (flags[i] == 0) {  // (uniform)
        have_h = false;
        continue;
      }
      const int e4 = tid * 4, er = e4 / kChainCols, ec = e4 & (kChainCols - 1);  // this thread's 4 of the 1024 values
      float4 add = *reinterpret_cast<const float4*>(state_of(b0 + i + 1) + er * kHeadDim + ec);
      if (!have_h) *reinterpret_cast<float4*>(sH + e4) = *reinterpret_cast<const float4*>(state_of(b0 + i) + er * kHeadDim + ec);
      have_h = true;
      mm::cp_async_wait<1>();
      __syncthreads();
      float acc[4][4] = {};
#pragma unroll 2
      for (int j = jq * 32; j < jq * 32 + 32; j += 4) {
        float4 m[4], x[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          m[q] = *reinterpret_cast<const float4*>(sM[buf] + (row + 32 * q) * kChainStride + j);
          x[q] = *reinterpret_cast<const float4*>(sH + (j + q) * kChainCols + cq);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float mv[4] = {m[q].x, m[q].y, m[q].z, m[q].w};
#pragma unroll
          for (int y = 0; y < 4; ++y) {
            acc[q][0] = fmaf(mv[y], x[y].x, acc[q][0]);
            acc[q][1] = fmaf(mv[y], x[y].y, acc[q][1]);
            acc[q][2] = fmaf(mv[y], x[y].z, acc[q][2]);
            acc[q][3] = fmaf(mv[y], x[y].w, acc[q][3]);
          }
        }
      }
      // the four quarters of the inner dimension: 2, 3 hand over to 0, 1, then 1 to 0 (fixed order)
#pragma unroll
      for (int half = 2; half > 0; half >>= 1) {
        __syncthreads();
        if (jq >= half && jq < 2 * half) {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            *reinterpret_cast<float4*>(sP + ((jq - half) * kHeadDim + row + 32 * q) * kChainCols + cq) =
                make_float4(acc[q][0], acc[q][1], acc[q][2], acc[q][3]);
        }
        __syncthreads();
        if (jq < half) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float4 p = *reinterpret_cast<const float4*>(sP + (jq * kHeadDim + row + 32 * q) * kChainCols + cq);
            acc[q][0] += p.x; acc[q][1] += p.y; acc[q][2] += p.z; acc[q][3] += p.w;
          }
        }
      }
      if (jq == 0) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
          *reinterpret_cast<float4*>(sP + (kHeadDim + row + 32 * q) * kChainCols + cq) =
              make_float4(acc[q][0], acc[q][1], acc[q][2], acc[q][3]);
      }
      __syncthreads();
      const float4 p = *reinterpret_cast<const float4*>(sP + kHeadDim * kChainCols + e4);
      add.x += p.x; add.y += p.y; add.z += p.z; add.w += p.w;
      *reinterpret_cast<float4*>(sH + e4) = add;
      *reinterpret_cast<float4*>(state_of(b0 + i + 1) + er * kHeadDim + ec) = add;
    }
    mm::cp_async_wait<0>();
    __threadfence_block();  // a link behind this batch reads the state written last (by the same thread)
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
  { const int rc = ensure_dynamic_smem<cp_chain_kernel>(kChainSmem); if (rc != QLA_OK) return rc; }
  QLA_CHECK_CUDA(launch_dependent(cp_chain_kernel, grid, dim3(kChainThreads), kChainSmem, static_cast<cudaStream_t>(stream), a->h0, a->M,
                                  a->m_limit, a->raw_first_seg, a->num_v_heads, a->reverse));
  return QLA_OK;
}
