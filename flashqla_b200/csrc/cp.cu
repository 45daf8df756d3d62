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

// A state of the caller's (fp32 or bf16, [K][V] or [V][K]) as fp32 [K][V]; no row: zero.  All kPlanThreads threads of kCopyParts CTAs
// (blockIdx.z - 1), a quarter each, beside the one that plans.
constexpr int kCopyParts = 4;
__device__ __forceinline__ void copy_state(const QlaCpPlanArgs& a, float* dst, int row, int h) {
  constexpr int kElems = kHeadDim * kHeadDim / kCopyParts;  // 32 rows of either
  const int first = static_cast<int>(blockIdx.z - 1) * kElems;
  if (row < 0) {
    for (int i = threadIdx.x * 4; i < kElems; i += kPlanThreads * 4)
      *reinterpret_cast<float4*>(dst + first + i) = make_float4(0.f, 0.f, 0.f, 0.f);
    return;
  }
  const int64_t off = (static_cast<int64_t>(row) * a.num_v_heads + h) * kHeadDim * kHeadDim + first;
  const float* s32 = static_cast<const float*>(a.h0) + off;
  const __nv_bfloat16* s16 = static_cast<const __nv_bfloat16*>(a.h0) + off;
  const bool b16 = a.h0_dtype == QLA_DT_BF16;
  if (!a.h0_transposed) {
#pragma unroll
    for (int i = threadIdx.x; i < kElems; i += kPlanThreads) dst[first + i] = b16 ? __bfloat162float(s16[i]) : s32[i];
    return;
  }
  // transposed through shared memory, 32 source rows: both sides coalesced
  __shared__ float tile[32][kHeadDim + 1];
#pragma unroll
  for (int i = threadIdx.x; i < kElems; i += kPlanThreads) tile[i >> 7][i & 127] = b16 ? __bfloat162float(s16[i]) : s32[i];
  __syncthreads();
#pragma unroll
  for (int i = threadIdx.x; i < kElems; i += kPlanThreads) dst[(i >> 5) * kHeadDim + (first >> 7) + (i & 31)] = tile[i & 31][i >> 5];
}

// 1 + kCopyParts CTAs per (segment, head): a warp of the first finds the warm-up length; the others write the segment's start state.
__global__ void __launch_bounds__(kPlanThreads) cp_plan_kernel(const QlaCpPlanArgs a) {
  grid_dep_wait();    // earlier kernels of the stream have completed (see launch_dependent)
  grid_dep_launch();
  const int seg = blockIdx.x, h = blockIdx.y;
  const int num_heads = a.num_v_heads;
  if (blockIdx.z != 0) {
    const int raw = a.seg_start_of[seg];
    int row = -1;
    if (raw >= 0 && a.h0 != nullptr) row = a.h0_map != nullptr ? a.h0_map[raw] : raw;
    copy_state(a, a.cp_h0 + (static_cast<int64_t>(seg) * num_heads + h) * kHeadDim * kHeadDim, row, h);
    return;
  }
  if (threadIdx.x >= 32) return;
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

// The plan with the warm-up folded into the main scan (forward, or reverse for the backward scan): 1 + kCopyParts CTAs per
// (original sequence, head), a warp of the first per segment.  A (sequence, head) in which every segment decays below the threshold needs
// no state-only pass: the main scan's CTA of segment s simply starts lead[s] = warm(s - 1) chunks early, from a zero state.  If some
// segment never decays that far the limits are those of cp_plan_kernel (state-only pass, transition matrices,
// chain) and lead is 0.  Only the row of cp_h0 that starts the sequence is written here.
__global__ void __launch_bounds__(kPlanThreads) cp_plan_lead_kernel(const QlaCpPlanArgs a) {
  grid_dep_wait();
  grid_dep_launch();
  const int r = blockIdx.x, h = blockIdx.y;
  const int num_heads = a.num_v_heads;
  const int s0 = a.raw_first_seg[r], s1 = a.raw_first_seg[r + 1];
  if (blockIdx.z != 0) {
    // start state of the sequence (backward: the gradient of its final state, into the last segment's row): the
    // caller's (any dtype / layout, through h0_map) or zero
    int row = -1;
    if (a.h0 != nullptr) row = a.h0_map != nullptr ? a.h0_map[r] : r;
    copy_state(a, a.cp_h0 + (static_cast<int64_t>(a.reverse ? s1 - 1 : s0) * num_heads + h) * kHeadDim * kHeadDim, row, h);
    return;
  }
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
}

// The chain  h[next] += M[seg] h[seg]  over the segments of one sequence and head, in order.  A link is a dependent
// 128 x 128 by 128 x 8 product in fp32: the columns are split over CTAs (8 each), warp w of a CTA has rows 16 w .. 16 w + 15, and a
// lane every fourth row and 16 of the inner index of each: 4 x 8 sums, two columns per instruction, which the eight lanes
// of a row then add up in a tree.  M comes by bulk copies into three stages, two links ahead; the carried columns pass through shared
// memory in two buffers: one barrier per link.  What bounds it: reads of shared memory, 48 of 16 bytes per thread and link.  36 links of
// 1 / 4 / 8 heads take 53 / 54 / 54 us (59 / 60 / 61 with every thread's part of M straight from L2; 59 with split TF32 factors on
// mma.sync, whose error against 64 bits was 2 to 7 times that of fp32; 53 / 84 / 165 with the rows split over clusters of four CTAs).
constexpr int kChainCols = 8;
constexpr int kChainGroup = 4 * kChainCols + 4;  // floats from four rows of the carried columns to the next four: conflict-free float4
constexpr int kChainThreads = 256;
constexpr int kChainFlags = 256;
constexpr int kChainStages = 3;
constexpr uint32_t kChainTile = kHeadDim * kHeadDim * 4;
constexpr size_t kChainSmem = kChainStages * kChainTile;

// A warp's wait for the matrix in `stage`, the same verdict for all of it.  Given up, the status word says so (192 + stage as the
// barrier); the thread that requests the copies then waits for those still on their way, `ahead` links from this one on, or for
// another while: shared memory stays allocated until they have landed.
static __device__ __noinline__ bool chain_wait(uint64_t* full, int stage, uint32_t uses, int* status, int ahead, const int* flags) {
  if (__all_sync(__activemask(), ptx::mbar_wait_polling(&full[stage], (uses >> stage) & 1, status, kStatusBarrierTimeout | ((192 + stage) << 8),
                                                        ptx::kWaitLimitNs)))
    return true;
  for (int x = 0; x < ahead; ++x) {
    const int s = (stage + x) % kChainStages;
    if (flags[x] != 0) ptx::mbar_wait_nocall(ptx::smem_u32(&full[s]), (uses >> s) & 1, true);
  }
  return false;
}

__global__ void __launch_bounds__(kChainThreads, 1) cp_chain_kernel(float* __restrict__ h0, const float* __restrict__ M,
                                                                    const int32_t* __restrict__ m_limit,
                                                                    const int32_t* __restrict__ raw_first_seg, int num_heads,
                                                                    int reverse, int* status) {
  grid_dep_wait();
  grid_dep_launch();
  const int c0 = blockIdx.x * kChainCols, h = blockIdx.y, r = blockIdx.z, tid = threadIdx.x;
  const int s0 = raw_first_seg[r], links = raw_first_seg[r + 1] - s0 - 1;
  __shared__ __align__(16) float s_h[2][kHeadDim / 4 * kChainGroup];  // [buffer][row / 4][row % 4][column]
  __shared__ int flags[kChainFlags];
  extern __shared__ __align__(128) uint8_t s_m[];  // M of links i, i + 1, i + 2 by turns
  __shared__ uint64_t full[kChainStages];
  uint32_t uses = 0;     // of a stage: bit x, the parity of its next phase
  bool ready = false;    // the barriers are initialised
  bool gave_up = false;  // a wait of this warp has
  // link i leads from segment seg_of(i) to seg_of(i + 1)
  auto seg_of = [&](int i) { return reverse ? s0 + links - i : s0 + i; };
  // rows 16 warp + rg + 4 i (i = 0..3), inner indices 32 t + 4 sl .. + 3 (t = 0..3)
  const int warp = tid >> 5, rg = (tid >> 3) & 3, sl = tid & 7;
  // after the sums this thread has row `row`, columns col .. col + 3
  const int row = 16 * warp + rg + 4 * (sl >> 1), col = 4 * (sl & 1);
  auto state_of = [&](int i) {
    return reinterpret_cast<float4*>(h0 + ((static_cast<int64_t>(seg_of(i)) * num_heads + h) * kHeadDim + row) * kHeadDim + c0 + col);
  };
  auto carry = [&](int buf, float4 x) {
    *reinterpret_cast<float4*>(&s_h[buf][(row >> 2) * kChainGroup + (row & 3) * kChainCols + col]) = x;
  };
  auto request = [&](int i) {  // thread 0: M of link i (number i % kChainFlags of its batch)
    const int stage = i % kChainFlags % kChainStages;
    ptx::mbar_expect_tx(&full[stage], kChainTile);
    ptx::bulk_load(s_m + stage * kChainTile, M + (static_cast<int64_t>(seg_of(i)) * num_heads + h) * kHeadDim * kHeadDim, kChainTile, &full[stage]);
  };
  // this thread's four values of the product of the matrix in `stage` and the carried columns in `buf`
  auto product = [&](int stage, int buf) {
    F2 acc[4][4] = {};  // [i][pair of columns]
    const float* part = reinterpret_cast<const float*>(s_m + stage * kChainTile) + (16 * warp + rg) * kHeadDim + 4 * sl;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      float4 m[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) m[i] = *reinterpret_cast<const float4*>(part + 4 * i * kHeadDim + 32 * t);
      const float* x = &s_h[buf][(8 * t + sl) * kChainGroup];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const ulonglong2 lo = *reinterpret_cast<const ulonglong2*>(x + e * kChainCols), hi = *reinterpret_cast<const ulonglong2*>(x + e * kChainCols + 4);
        const F2 xs[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float mv = e == 0 ? m[i].x : e == 1 ? m[i].y : e == 2 ? m[i].z : m[i].w;
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[i][c] = fma2(f2(mv, mv), xs[c], acc[i][c]);
        }
      }
    }
    // the eight lanes of a row: a lane passes on the half it does not keep, three times
    auto add = [&](float2 keep, float2 send, int lanes) {
      return make_float2(keep.x + __shfl_xor_sync(0xffffffffu, send.x, lanes), keep.y + __shfl_xor_sync(0xffffffffu, send.y, lanes));
    };
    const bool b2 = sl & 4, b1 = sl & 2, b0 = sl & 1;
    float2 y[2][4], z[4], out[2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) y[i][c] = add(unpack(b2 ? acc[2 + i][c] : acc[i][c]), unpack(b2 ? acc[i][c] : acc[2 + i][c]), 4);
#pragma unroll
    for (int c = 0; c < 4; ++c) z[c] = add(b1 ? y[1][c] : y[0][c], b1 ? y[0][c] : y[1][c], 2);
#pragma unroll
    for (int c = 0; c < 2; ++c) out[c] = add(b0 ? z[2 + c] : z[c], b0 ? z[c] : z[2 + c], 1);
    return make_float4(out[0].x, out[0].y, out[1].x, out[1].y);
  };
  int buf = 0;
  for (int b0 = 0; b0 < links; b0 += kChainFlags) {
    const int nb = min(kChainFlags, links - b0);
    int mine = 0;
    if (b0 != 0 && __syncthreads_or(gave_up)) return;
    for (int i = tid; i < nb; i += kChainThreads) mine |= (flags[i] = m_limit[seg_of(b0 + i) * num_heads + h]);
    // the usual case (every segment decays below the threshold) has nothing to chain
    if (__syncthreads_or(mine) == 0) continue;
    bool have_h = false;
    float4 add = make_float4(0.f, 0.f, 0.f, 0.f);  // the next state as it is: what the product is added to
    if (flags[0] != 0) add = *state_of(b0 + 1);
    if (tid == 0) {
      if (!ready) {
        for (int x = 0; x < kChainStages; ++x) ptx::mbar_init(&full[x], 1);
        ptx::fence_mbar_init();
      }
      for (int x = 0; x < kChainStages - 1 && x < nb; ++x)
        if (flags[x] != 0) request(b0 + x);
    }
    ready = true;
    for (int i = 0; i < nb; ++i) {
      const bool next = i + 1 < nb && flags[i + 1] != 0, work = flags[i] != 0;  // (uniform)
      if (work && !have_h) carry(buf, *state_of(b0 + i));
      have_h = work;
      float4 out = add;
      if (next) add = *state_of(b0 + i + 2);
      __syncthreads();  // the carried columns are complete, and the matrix of the link before has been read
      if (tid == 0 && i + kChainStages - 1 < nb && flags[i + kChainStages - 1] != 0) request(b0 + i + kChainStages - 1);
      if (!work) continue;
      const int stage = i % kChainStages;
      if (!ptx::mbar_try_wait(&full[stage], (uses >> stage) & 1) &&
          !chain_wait(full, stage, uses, status, tid == 0 ? min(kChainStages, nb - i) : 0, flags + i)) {
        for (gave_up = true; ++i < nb;) __syncthreads();  // (the other warps' barriers)
        break;
      }
      uses ^= 1u << stage;
      const float4 x = product(stage, buf);
      out.x += x.x; out.y += x.y; out.z += x.z; out.w += x.w;
      buf ^= 1;
      carry(buf, out);
      *state_of(b0 + i + 1) = out;
    }
    // (a link behind this batch reads the state written last, each value by the thread that wrote it)
  }
}

}  // namespace

void launch_info_cp_chain_kernel(int* block_threads, size_t* dynamic_smem_bytes) {
  *block_threads = kChainThreads;
  *dynamic_smem_bytes = kChainSmem;
}
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
    dim3 grid_lead(a->num_raw_seqs, a->num_v_heads, 1 + kCopyParts);
    QLA_CHECK_CUDA(launch_dependent(cp_plan_lead_kernel, grid_lead, dim3(kPlanThreads), 0, static_cast<cudaStream_t>(stream), *a));
    return QLA_OK;
  }
  dim3 grid(a->num_segments, a->num_v_heads, a->cp_h0 != nullptr ? 1 + kCopyParts : 1);
  QLA_CHECK_CUDA(launch_dependent(cp_plan_kernel, grid, dim3(kPlanThreads), 0, static_cast<cudaStream_t>(stream), *a));
  return QLA_OK;
}

extern "C" QLA_API int qla_cp_chain(const QlaCpChainArgs* a, void* stream) {
  using namespace qla;
  QLA_CHECK_ARG(a != nullptr && a->h0 && a->M && a->m_limit && a->raw_first_seg, "NULL pointer in QlaCpChainArgs");
  QLA_CHECK_ARG(a->num_raw_seqs > 0 && a->num_v_heads > 0, "bad sizes");
  dim3 grid(kHeadDim / kChainCols, a->num_v_heads, a->num_raw_seqs);
  const int rc = ensure_dynamic_smem<cp_chain_kernel>(kChainSmem);
  if (rc != QLA_OK) return rc;
  QLA_CHECK_CUDA(launch_dependent(cp_chain_kernel, grid, dim3(kChainThreads), kChainSmem, static_cast<cudaStream_t>(stream), a->h0, a->M,
                                  a->m_limit, a->raw_first_seg, a->num_v_heads, a->reverse, a->has_status != 0 ? a->status : nullptr));
  return QLA_OK;
}
