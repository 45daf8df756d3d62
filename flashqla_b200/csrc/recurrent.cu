// Recurrent gated-delta-rule step(s): decode (1 token), spec-decode verify (T draft tokens with a
// cached state per step), tree verify (a step may restart from the cached state of its parent)
// and ragged sequences (cu_seqlens).  Three kernels, the same bits, cover what the reference spreads over 29
// generated kernels (flash_qla/ops/gated_delta_rule/recurrent_fused.py:290-6249): recurrent_kernel takes every call,
// recurrent_step_kernel one step, recurrent_chain_kernel several (takes_step, takes_chain say which of those).  The per-token
// math follows the canonical body at :346-487 and the reload rule of the warp kernels at
// :5803-5836 (a parent equal to the previous step is not reloaded).
//
// The op is HBM-bound (several steps per state: bound by instruction issue unless fp32 states are cached): every (sequence, v-head)
// streams a 64 KiB fp32 state in and out.
// Mapping: the state of one head is [V=128 rows][K=128 floats]; a row is 512 B.  Eight lanes share
// a row, each lane owning four float4 (columns j*32 + sub*4 .. +3, j = 0..3), so one warp
// instruction moves four whole rows = 2 KiB, fully coalesced, 128-bit per lane.  A thread keeps R
// rows in registers for the whole call (R*16 floats); the K-reductions (S.k and S.q) are three
// xor-shuffles over the eight lanes of a row.  A CTA of 128 threads covers 16*R rows.
#include "common.cuh"
#include "warp_pieces.cuh"

namespace qla {
namespace {

__device__ __forceinline__ float sum2(F2 x) {
  const float2 v = unpack(x);
  return v.x + v.y;
}

// Four consecutive values: raw 16-bit or fp32 memory -> two pairs and back.
template <typename T>
__device__ __forceinline__ void unpack4(uint2 raw, F2 (&out)[2]);
template <>
__device__ __forceinline__ void unpack4<__nv_bfloat16>(uint2 raw, F2 (&out)[2]) {
  const float2 a = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&raw.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&raw.y));
  out[0] = f2(a.x, a.y); out[1] = f2(b.x, b.y);
}
template <>
__device__ __forceinline__ void unpack4<__half>(uint2 raw, F2 (&out)[2]) {
  const float2 a = __half22float2(*reinterpret_cast<__half2*>(&raw.x));
  const float2 b = __half22float2(*reinterpret_cast<__half2*>(&raw.y));
  out[0] = f2(a.x, a.y); out[1] = f2(b.x, b.y);
}
__device__ __forceinline__ void store4(float* p, const F2 (&x)[2]) {
  *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(x[0], x[1]);
}
__device__ __forceinline__ void store4(__nv_bfloat16* p, const F2 (&x)[2]) {
  const float2 a = unpack(x[0]), b = unpack(x[1]);
  __nv_bfloat162 lo = __floats2bfloat162_rn(a.x, a.y), hi = __floats2bfloat162_rn(b.x, b.y);
  uint2 raw;
  raw.x = *reinterpret_cast<uint32_t*>(&lo);
  raw.y = *reinterpret_cast<uint32_t*>(&hi);
  *reinterpret_cast<uint2*>(p) = raw;
}

__device__ __forceinline__ float group8_sum(float x) {
  x += __shfl_xor_sync(0xffffffffu, x, 1);
  x += __shfl_xor_sync(0xffffffffu, x, 2);
  x += __shfl_xor_sync(0xffffffffu, x, 4);
  return x;
}

constexpr int kRecStages = 2;  // state tiles staged per CTA: the current one and the next

// One 16-byte (fp32 pool) or 8-byte (16-bit pool) piece of a state row: the four values a lane owns.
template <typename StateT>
struct StatePiece;
template <>
struct StatePiece<float> {
  using Raw = ulonglong2;
  static __device__ __forceinline__ void copy_async(Raw* dst, const float* src) { mm::cp_async16(dst, src, true); }
  static __device__ __forceinline__ void unpack(const Raw& x, F2 (&out)[2]) { out[0] = x.x; out[1] = x.y; }
};
template <>
struct StatePiece<__nv_bfloat16> {
  using Raw = uint2;
  static __device__ __forceinline__ void copy_async(Raw* dst, const __nv_bfloat16* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(mm::smem_addr(dst)), "l"(src) : "memory");
  }
  static __device__ __forceinline__ void unpack(const Raw& x, F2 (&out)[2]) { unpack4<__nv_bfloat16>(x, out); }
};

// kTree: a step may restart from the cached state of an earlier one (parents given).  That state is requested one step
// ahead, before the arithmetic of the step in between, into registers of its own.
// kOne: one token per sequence; nothing of the loop over steps is left.
template <typename T, typename InterT, typename StateT, int R, bool kTree, bool kOne>
__device__ __forceinline__ void recurrent_items(const QlaRecurrentArgs& p, const uint32_t total_items) {
  constexpr int D = kHeadDim;
  constexpr int BV = 16 * R;
  constexpr int kTiles = D / BV;
  // [kRecStages][R * 4 pieces][128 threads] float4: every thread stages exactly the 16-byte pieces it owns, so
  // no barrier is needed between the copy and its use
  using Piece = StatePiece<StateT>;
  extern __shared__ __align__(16) uint8_t s_stage_raw[];
  typename Piece::Raw* s_stage = reinterpret_cast<typename Piece::Raw*>(s_stage_raw);
  grid_dep_wait();    // earlier kernels of the stream have completed (see launch_dependent)
  grid_dep_launch();  // the next one may be scheduled; it waits the same way
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane & 7, grp = lane >> 3;
  const int col0 = sub * 4;  // first owned column of j = 0; j-th is col0 + 32 j

  // A slot outside the pool is never touched: the sequence runs from a zero state without write-back, and
  // the status word says that an index was bad.
  auto bad_index = [&]() {
    if (p.status != nullptr && threadIdx.x == 0) atomicCAS(p.status, 0, kStatusBadIndex);
  };
  // Work item -> (sequence, v-head, row tile) and the sequence's pool slot, looked up once, when the item's tile is
  // requested (32-bit arithmetic: 64-bit divisions are long sequences of instructions).
  struct Item {
    int n, h, tile;
    int64_t slot;
  };
  auto locate = [&](uint32_t item) {
    Item x;
    x.tile = static_cast<int>(item % kTiles);
    const uint32_t nh = item / kTiles;
    x.n = static_cast<int>(nh / static_cast<uint32_t>(p.num_v_heads));
    x.h = static_cast<int>(nh) - x.n * p.num_v_heads;
    x.slot = p.state_indices ? p.state_indices[x.n] : x.n;
    if (x.slot >= p.state_slots) {
      bad_index();
      x.slot = -1;
    }
    return x;
  };
  // The state tile of an item is requested one item ahead (cp.async, L2 only): the copy of the next tile is
  // in flight while this one is computed and written back, which keeps reads queued at the memory the whole
  // time instead of only at the start of every CTA.
  auto prefetch = [&](const Item& x, int stage) {
    if (x.slot < 0) return;
    const int row0 = x.tile * BV + warp * 4 + grp;
    const StateT* sp = static_cast<const StateT*>(p.state) + ((x.slot * p.num_v_heads + x.h) * D + row0) * D + col0;
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        Piece::copy_async(&s_stage[(stage * R * 4 + r * 4 + j) * 128 + threadIdx.x], sp + (r * 16) * D + j * 32);
  };

  const T* qb = static_cast<const T*>(p.q);
  const T* kb = static_cast<const T*>(p.k);
  const T* vb = static_cast<const T*>(p.v);
  T* ob = static_cast<T*>(p.o);
  InterT* ib = static_cast<InterT*>(p.inter);
  const bool l2norm = (p.flags & QLA_REC_QK_L2NORM) != 0;

  Item next = locate(blockIdx.x);  // (the grid is at most total_items)
  prefetch(next, 0);
  mm::cp_async_commit();
  int it = 0;
  for (uint32_t item = blockIdx.x; item < total_items; item += gridDim.x, ++it) {
  const Item cur = next;
  if (item + gridDim.x < total_items) {
    next = locate(item + gridDim.x);
    prefetch(next, (it + 1) % kRecStages);
    // Its q, k, v and gate rows to L2, one line per thread, the first 16 steps: with several steps per state the kernel is
    // bound by latency and issue, and each item began by waiting for these rows (256 sequences x 4 steps: 485 -> 463 us).
    // With one step per state HBM is the bound, the rows come in the shadow of the state, and the extra requests cost
    // 8 us of 168, so decode does without.
    const int step = static_cast<int>(threadIdx.x / 8u), what = static_cast<int>(threadIdx.x & 7u);
    if (!kOne && p.tokens_per_seq > 1 && step < p.tokens_per_seq) {
      const int64_t t = static_cast<int64_t>(next.n) * p.tokens_per_seq + step;
      const int64_t qk = (t * p.num_k_heads + next.h / (p.num_v_heads / p.num_k_heads)) * D + (what & 1) * 64;
      const int64_t vg = t * p.num_v_heads + next.h;
      const int e = p.a_dtype == QLA_DT_F32 ? 4 : 2;
      const void* line = what < 2 ? static_cast<const void*>(qb + qk)
                         : what < 4 ? static_cast<const void*>(kb + qk)
                         : what == 4 ? static_cast<const void*>(vb + vg * D + next.tile * BV)
                         : what == 5 ? static_cast<const void*>(static_cast<const uint8_t*>(p.a) + vg * e)
                                     : static_cast<const void*>(static_cast<const uint8_t*>(p.b) + vg * e);
      asm volatile("prefetch.global.L2 [%0];" ::"l"(line) : "memory");
    }
  }
  mm::cp_async_commit();
  mm::cp_async_wait<kRecStages - 1>();  // all but the newest group: this item's tile has landed

  const int tile = cur.tile, h = cur.h, n = cur.n;
  const int64_t sidx = cur.slot;
  const int hk = h / (p.num_v_heads / p.num_k_heads);

  int t0, len;
  if (kOne) {
    t0 = n;
    len = 1;
  } else if (p.tokens_per_seq > 0) {
    t0 = n * p.tokens_per_seq;
    len = p.tokens_per_seq;
  } else {
    t0 = p.cu_seqlens[n];
    len = p.cu_seqlens[n + 1] - t0;
    // boundaries that leave the token range would read q / k / v and write o out of bounds
    if (t0 < 0 || len < 0 || t0 > p.total_tokens || len > p.total_tokens - t0) {
      bad_index();
      t0 = max(0, min(t0, p.total_tokens));
      len = max(0, min(len, p.total_tokens - t0));
    }
  }
  int64_t cidx = -1;
  if (p.inter != nullptr) {
    cidx = p.inter_indices ? p.inter_indices[n] : n;
    if (cidx >= p.inter_slots) {
      bad_index();
      cidx = -1;
    }
  }

  const int row0 = tile * BV + warp * 4 + grp;  // row of r = 0; r-th row is row0 + 16 r

  F2 S[R][4][2];
  if (sidx >= 0) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        Piece::unpack(s_stage[((it % kRecStages) * R * 4 + r * 4 + j) * 128 + threadIdx.x], S[r][j]);
      }
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        S[r][j][0] = S[r][j][1] = 0;
  }

  // Decay and beta of 32 steps at a time, lane = step: the activations (exponentials, a logarithm, a division) are worth
  // more instructions than the rest of a step, and every lane of the CTA needs the same two numbers.
  float decay_l = 0.f, beta_l = 0.f;
  auto fetch_gates = [&](int first) {
    const int step = first + lane;
    if (step >= len) return;
    const int64_t i = static_cast<int64_t>(t0 + step) * p.num_v_heads + h;
    float g = load_scalar(p.a, p.a_dtype, i);
    const float b_raw = load_scalar(p.b, p.a_dtype, i);
    if (!(p.flags & QLA_REC_A_IS_LOG_DECAY)) {
      const float x = g + load_scalar(p.dt_bias, p.dt_bias_dtype, h);
      const float bx = p.softplus_beta * x;
      const float sp = (bx <= p.softplus_threshold) ? log1pf(expf(bx)) / p.softplus_beta : x;
      g = -expf(load_scalar(p.A_log, p.a_log_dtype, h)) * sp;
    }
    decay_l = expf(g);
    beta_l = (p.flags & QLA_REC_B_IS_BETA) ? b_raw : 1.f / (1.f + expf(-b_raw));
  };

  // Inputs of a step (q, k row pieces, v) are requested one step ahead, so that with several draft
  // tokens their global-memory latency overlaps the previous step's arithmetic instead of heading every step.
  uint2 q_raw[4], k_raw[4];
  T v_raw[R];
  auto fetch_inputs = [&](int64_t t) {
    const T* qp = qb + (t * p.num_k_heads + hk) * D + col0;
    const T* kp = kb + (t * p.num_k_heads + hk) * D + col0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      q_raw[j] = *reinterpret_cast<const uint2*>(qp + j * 32);
      k_raw[j] = *reinterpret_cast<const uint2*>(kp + j * 32);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) v_raw[r] = vb[(t * p.num_v_heads + h) * D + row0 + 16 * r];
  };
  if (len > 0) {
    fetch_inputs(t0);
    fetch_gates(0);  // (requested together with the first step's rows)
  }

  // kTree: parent of a step (step - 1 where the table says nothing usable), and the cached state of the next step's parent
  using InterPiece = StatePiece<InterT>;
  typename InterPiece::Raw saved[kTree ? R : 1][4];
  bool restart = false;  // the next step starts from `saved`
  int par_next = 0;      // parent of the step after
  auto parent_of = [&](int step) {
    if (step >= len) return step - 1;
    if (step >= p.parents_steps) {  // the parents table is narrower than this sequence
      bad_index();
      return step - 1;
    }
    return p.parents[static_cast<int64_t>(n) * p.parents_stride + step];
  };
  const bool tree = kTree && cidx >= 0;
  if (tree) par_next = parent_of(1);

  for (int step = 0; kOne ? step < 1 : step < len; ++step) {
    const int64_t t = t0 + step;

    if (kTree && restart) {
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j) InterPiece::unpack(saved[r][j], S[r][j]);
    }
    if (tree && step + 1 < len) {
      const int par = par_next;
      par_next = parent_of(step + 2);
      // a parent equal to the step itself needs no reload; a step behind it has not been written in this call either way
      restart = par != step && par >= 0 && par < p.inter_steps;
      if (par != step && !restart) bad_index();
      if (restart) {
        const InterT* src = ib + (((cidx * p.inter_steps + par) * p.num_v_heads + h) * D + row0) * D + col0;
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int j = 0; j < 4; ++j)
            saved[r][j] = *reinterpret_cast<const typename InterPiece::Raw*>(src + (r * 16) * D + j * 32);
      }
    }

    F2 qv[4][2], kv[4][2];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      unpack4<T>(q_raw[j], qv[j]);
      unpack4<T>(k_raw[j], kv[j]);
    }
    float vrow[R];
#pragma unroll
    for (int r = 0; r < R; ++r) vrow[r] = Cvt<T>::to_f32(v_raw[r]);
    if (!kOne && step + 1 < len) fetch_inputs(t + 1);

    // q and k stay as loaded: the factors scale / |q| and 1 / |k| are folded into the scalars that use them.  With the
    // state S before the step (decayed: e^g S) the output is q . (e^g S + delta k) = e^g (q . S) + delta (q . k): both
    // products with S are formed in one pass and reduced together, before the update.
    F2 qk2 = mul2(qv[0][0], kv[0][0]);
    F2 qq2 = 0, kk2 = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (j + i > 0) qk2 = fma2(qv[j][i], kv[j][i], qk2);
        if (l2norm) {
          qq2 = fma2(qv[j][i], qv[j][i], qq2);
          kk2 = fma2(kv[j][i], kv[j][i], kk2);
        }
      }
    const float qk = group8_sum(sum2(qk2));
    float qs = p.scale, ks = 1.f;
    if (l2norm) {
      qs *= rsqrtf(group8_sum(sum2(qq2)) + 1e-6f);
      ks = rsqrtf(group8_sum(sum2(kk2)) + 1e-6f);
    }

    if (!kOne && step > 0 && (step & 31) == 0) fetch_gates(step);
    const float decay = __shfl_sync(0xffffffffu, decay_l, step & 31), beta = __shfl_sync(0xffffffffu, beta_l, step & 31);

    float dot[R], out[R];  // k . S, q . S
#pragma unroll
    for (int r = 0; r < R; ++r) {
      F2 ak[2] = {0, 0}, aq[2] = {0, 0};
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          ak[i] = fma2(S[r][j][i], kv[j][i], ak[i]);
          aq[i] = fma2(S[r][j][i], qv[j][i], aq[i]);
        }
      dot[r] = sum2(ak[0]) + sum2(ak[1]);
      out[r] = sum2(aq[0]) + sum2(aq[1]);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      dot[r] = group8_sum(dot[r]);
      out[r] = group8_sum(out[r]);
    }
    const F2 decay2 = f2(decay, decay);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float delta = (vrow[r] - decay * dot[r] * ks) * beta * ks;  // times k / |k|: one factor here
      const F2 delta2 = f2(delta, delta);
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) S[r][j][i] = fma2(kv[j][i], delta2, mul2(S[r][j][i], decay2));
      out[r] = fmaf(delta, qk, decay * out[r]) * qs;
    }
    if (sub == 0) {
#pragma unroll
      for (int r = 0; r < R; ++r)
        ob[(t * p.num_v_heads + h) * D + row0 + 16 * r] = Cvt<T>::from_f32(out[r]);
    }

    if (cidx >= 0 && (kOne || step < p.inter_steps)) {
      InterT* dst = ib + (((cidx * p.inter_steps + step) * p.num_v_heads + h) * D + row0) * D + col0;
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j) store4(dst + (r * 16) * D + j * 32, S[r][j]);
    }
  }

  if (!(p.flags & QLA_REC_DISABLE_STATE_UPDATE) && sidx >= 0) {
    StateT* sp = static_cast<StateT*>(p.state) + ((sidx * p.num_v_heads + h) * D + row0) * D + col0;
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j) store4(sp + (r * 16) * D + j * 32, S[r][j]);
  }
  }  // items
}

template <typename T, typename InterT, typename StateT, int R, bool kTree>
__global__ void __launch_bounds__(128) recurrent_kernel(const __grid_constant__ QlaRecurrentArgs p, const uint32_t total_items) {
  recurrent_items<T, InterT, StateT, R, kTree, false>(p, total_items);
}
template <typename T, typename InterT, typename StateT, int R>
__global__ void __launch_bounds__(128, R == 2 ? 5 : 7) recurrent_step_kernel(const __grid_constant__ QlaRecurrentArgs p, const uint32_t total_items) {
  recurrent_items<T, InterT, StateT, R, false, true>(p, total_items);
}

constexpr int kBlockSteps = 4;  // draft tokens prepared at a time, one per warp

// What a block of steps needs beside the state, fp32: q and k as loaded, v of the tile's rows, and per step the scalars (ks = 1 / |k|,
// qs = scale / |q|).
template <int R>
struct alignas(16) StepInputs {
  float q[kBlockSteps][kHeadDim], k[kBlockSteps][kHeadDim], v[kBlockSteps][16 * R];
  struct alignas(16) Scalars {
    float decay, beta, ks, qs, qk, pad[3];
  } s[kBlockSteps];
};

// Several steps per sequence, all sequences of one length, no tree.  q, k, v and gates of a block of steps are unpacked, multiplied and
// activated once per CTA and read from shared memory by its rows; in recurrent_kernel every warp does that for itself, which is most
// of its instructions.
template <typename T, typename InterT, typename StateT, int R>
__global__ void __launch_bounds__(128, R == 2 ? 5 : 8) recurrent_chain_kernel(const QlaRecurrentArgs p, const uint32_t total_items) {
  constexpr int D = kHeadDim;
  constexpr int BV = 16 * R;
  constexpr int kTiles = D / BV;
  // [kRecStages][R * 4 pieces][128 threads] float4: every thread stages exactly the 16-byte pieces it owns, so
  // no barrier is needed between the copy and its use
  using Piece = StatePiece<StateT>;
  extern __shared__ __align__(16) uint8_t s_stage_raw[];
  typename Piece::Raw* s_stage = reinterpret_cast<typename Piece::Raw*>(s_stage_raw);
  __shared__ StepInputs<R> s_inputs[2];
  grid_dep_wait();    // earlier kernels of the stream have completed (see launch_dependent)
  grid_dep_launch();  // the next one may be scheduled; it waits the same way
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int sub = lane & 7, grp = lane >> 3;
  const int col0 = sub * 4;  // first owned column of j = 0; j-th is col0 + 32 j
  const int len = p.tokens_per_seq;

  // A slot outside the pool is never touched: the sequence runs from a zero state without write-back, and
  // the status word says that an index was bad.
  auto bad_index = [&]() {
    if (p.status != nullptr && threadIdx.x == 0) atomicCAS(p.status, 0, kStatusBadIndex);
  };
  // Work item -> (sequence, v-head, row tile) and the sequence's pool slot, looked up once, when the item's tile is
  // requested (32-bit arithmetic: 64-bit divisions are long sequences of instructions).
  struct Item {
    int n, h, tile, t0;
    int64_t slot;
  };
  auto locate = [&](uint32_t item) {
    Item x;
    x.tile = static_cast<int>(item % kTiles);
    const uint32_t nh = item / kTiles;
    x.n = static_cast<int>(nh / static_cast<uint32_t>(p.num_v_heads));
    x.h = static_cast<int>(nh) - x.n * p.num_v_heads;
    x.slot = p.state_indices ? p.state_indices[x.n] : x.n;
    if (x.slot >= p.state_slots) {
      bad_index();
      x.slot = -1;
    }
    x.t0 = x.n * len;
    return x;
  };
  // The state tile of an item is requested one item ahead (cp.async, L2 only): the copy of the next tile is
  // in flight while this one is computed and written back, which keeps reads queued at the memory the whole
  // time instead of only at the start of every CTA.
  auto prefetch = [&](const Item& x, int stage) {
    if (x.slot < 0) return;
    const int row0 = x.tile * BV + warp * 4 + grp;
    const StateT* sp = static_cast<const StateT*>(p.state) + ((x.slot * p.num_v_heads + x.h) * D + row0) * D + col0;
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        Piece::copy_async(&s_stage[(stage * R * 4 + r * 4 + j) * 128 + threadIdx.x], sp + (r * 16) * D + j * 32);
  };

  const T* qb = static_cast<const T*>(p.q);
  const T* kb = static_cast<const T*>(p.k);
  const T* vb = static_cast<const T*>(p.v);
  T* ob = static_cast<T*>(p.o);
  InterT* ib = static_cast<InterT*>(p.inter);
  const bool l2norm = (p.flags & QLA_REC_QK_L2NORM) != 0;

  // Rows and gates of a block of steps: warp w requests step first + w while the block in front is computed, and writes what the
  // CTA needs of it to shared memory behind that block, once for all rows of the tile.
  uint2 q_raw, k_raw;
  T v_raw;
  float a_raw, b_raw, a_log, dt_bias;
  auto request = [&](const Item& x, int first) {
    const int step = first + warp;
    if (step >= len) return;
    const int64_t t = x.t0 + step, th = t * p.num_v_heads + x.h;
    const int64_t qk = (t * p.num_k_heads + x.h / (p.num_v_heads / p.num_k_heads)) * D + lane * 4;
    q_raw = *reinterpret_cast<const uint2*>(qb + qk);
    k_raw = *reinterpret_cast<const uint2*>(kb + qk);
    if (BV == 32 || lane < BV) v_raw = vb[th * D + x.tile * BV + lane];
    a_raw = load_scalar(p.a, p.a_dtype, th);
    b_raw = load_scalar(p.b, p.a_dtype, th);
    if (!(p.flags & QLA_REC_A_IS_LOG_DECAY)) {
      a_log = load_scalar(p.A_log, p.a_log_dtype, x.h);
      dt_bias = load_scalar(p.dt_bias, p.dt_bias_dtype, x.h);
    }
  };
  auto prepare = [&](const Item& x, int first, StepInputs<R>& in) {
    if (first + warp >= len) return;
    F2 q[2], k[2];
    unpack4<T>(q_raw, q);
    unpack4<T>(k_raw, k);
    store4(&in.q[warp][lane * 4], q);
    store4(&in.k[warp][lane * 4], k);
    if (BV == 32 || lane < BV) in.v[warp][lane] = Cvt<T>::to_f32(v_raw);
    // (sums in the order of recurrent_kernel: a state cached in 16 bits is the rounded value of one cached in fp32)
    __syncwarp();
    F2 qk2 = 0, qq2 = 0, kk2 = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const ulonglong2 kp = *reinterpret_cast<const ulonglong2*>(&in.k[warp][col0 + 32 * j]);
      const ulonglong2 qp = *reinterpret_cast<const ulonglong2*>(&in.q[warp][col0 + 32 * j]);
      qk2 = j == 0 ? mul2(qp.x, kp.x) : fma2(qp.x, kp.x, qk2);
      qk2 = fma2(qp.y, kp.y, qk2);
      if (l2norm) {
        qq2 = fma2(qp.y, qp.y, fma2(qp.x, qp.x, qq2));
        kk2 = fma2(kp.y, kp.y, fma2(kp.x, kp.x, kk2));
      }
    }
    const float qk = group8_sum(sum2(qk2));
    float qs = p.scale, ks = 1.f;
    if (l2norm) {
      qs *= rsqrtf(group8_sum(sum2(qq2)) + 1e-6f);
      ks = rsqrtf(group8_sum(sum2(kk2)) + 1e-6f);
    }
    float g = a_raw;
    if (!(p.flags & QLA_REC_A_IS_LOG_DECAY)) {
      const float y = g + dt_bias, by = p.softplus_beta * y;
      g = -expf(a_log) * (by <= p.softplus_threshold ? log1pf(expf(by)) / p.softplus_beta : y);
    }
    const float decay = expf(g), beta = (p.flags & QLA_REC_B_IS_BETA) ? b_raw : 1.f / (1.f + expf(-b_raw));
    if (lane == 0) {
      *reinterpret_cast<float4*>(&in.s[warp].decay) = make_float4(decay, beta, ks, qs);
      in.s[warp].qk = qk;
    }
  };

  Item next = locate(blockIdx.x);  // (the grid is at most total_items)
  prefetch(next, 0);
  mm::cp_async_commit();
  request(next, 0);
  prepare(next, 0, s_inputs[0]);
  __syncthreads();
  int it = 0, buf = 0;
  for (uint32_t item = blockIdx.x; item < total_items; item += gridDim.x, ++it) {
  const Item cur = next;
  const bool more = item + gridDim.x < total_items;
  if (more) {
    next = locate(item + gridDim.x);
    prefetch(next, (it + 1) % kRecStages);
  }
  mm::cp_async_commit();
  mm::cp_async_wait<kRecStages - 1>();  // all but the newest group: this item's tile has landed

  const int tile = cur.tile, h = cur.h, n = cur.n;
  const int64_t sidx = cur.slot;
  int64_t cidx = -1;
  if (p.inter != nullptr) {
    cidx = p.inter_indices ? p.inter_indices[n] : n;
    if (cidx >= p.inter_slots) {
      bad_index();
      cidx = -1;
    }
  }

  const int row0 = tile * BV + warp * 4 + grp;  // row of r = 0; r-th row is row0 + 16 r

  F2 S[R][4][2];
  if (sidx >= 0) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        Piece::unpack(s_stage[((it % kRecStages) * R * 4 + r * 4 + j) * 128 + threadIdx.x], S[r][j]);
      }
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        S[r][j][0] = S[r][j][1] = 0;
  }

  T* orow = ob + (static_cast<int64_t>(cur.t0) * p.num_v_heads + h) * D + row0;
  InterT* irow = ib + ((cidx * p.inter_steps * p.num_v_heads + h) * D + row0) * D + col0;  // (cidx < 0: not used)

  for (int first = 0; first < len; first += kBlockSteps, buf ^= 1) {
  // the block behind this one: of this item or the next one's first
  const bool ends = first + kBlockSteps >= len;
  if (!ends) request(cur, first + kBlockSteps);
  else if (more) request(next, 0);
  const StepInputs<R>& in = s_inputs[buf];
#pragma unroll 1
  for (int i = 0, count = min(kBlockSteps, len - first); i < count; ++i) {
    const int step = first + i;
    // With the state S before the step (decayed: e^g S) the output is q . (e^g S + delta k) = e^g (q . S) + delta (q . k): both
    // products with S are formed in one pass and reduced together, before the update.
    F2 kv[4][2];
    F2 ak[R][2], aq[R][2];  // k . S, q . S
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const ulonglong2 k2 = *reinterpret_cast<const ulonglong2*>(&in.k[i][col0 + 32 * j]);
      const ulonglong2 q2 = *reinterpret_cast<const ulonglong2*>(&in.q[i][col0 + 32 * j]);
      kv[j][0] = k2.x;
      kv[j][1] = k2.y;
      const F2 qv[2] = {q2.x, q2.y};
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          ak[r][e] = j == 0 ? mul2(S[r][j][e], kv[j][e]) : fma2(S[r][j][e], kv[j][e], ak[r][e]);
          aq[r][e] = j == 0 ? mul2(S[r][j][e], qv[e]) : fma2(S[r][j][e], qv[e], aq[r][e]);
        }
    }
    const float4 sc = *reinterpret_cast<const float4*>(&in.s[i].decay);
    const float decay = sc.x, beta = sc.y, ks = sc.z, qs = sc.w, qk = in.s[i].qk;
    float dot[R], out[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      dot[r] = sum2(ak[r][0]) + sum2(ak[r][1]);
      out[r] = sum2(aq[r][0]) + sum2(aq[r][1]);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      dot[r] = group8_sum(dot[r]);
      out[r] = group8_sum(out[r]);
    }
    const F2 decay2 = f2(decay, decay);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float delta = fmaf(-(decay * dot[r]), ks, in.v[i][warp * 4 + grp + 16 * r]) * beta * ks;  // times k / |k|: one factor here
      const F2 delta2 = f2(delta, delta);
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) S[r][j][e] = fma2(kv[j][e], delta2, mul2(S[r][j][e], decay2));
      out[r] = fmaf(delta, qk, decay * out[r]) * qs;
    }
    if (sub == 0) {
#pragma unroll
      for (int r = 0; r < R; ++r) orow[16 * r] = Cvt<T>::from_f32(out[r]);
    }
    orow += p.num_v_heads * D;

    if (cidx >= 0 && step < p.inter_steps) {
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j) store4(irow + (r * 16) * D + j * 32, S[r][j]);
      irow += static_cast<int64_t>(p.num_v_heads) * D * D;
    }
  }
  if (!ends) prepare(cur, first + kBlockSteps, s_inputs[buf ^ 1]);
  else if (more) prepare(next, 0, s_inputs[buf ^ 1]);
  __syncthreads();  // (the other buffer is complete; this one has been read)
  }  // blocks of steps

  if (!(p.flags & QLA_REC_DISABLE_STATE_UPDATE) && sidx >= 0) {
    StateT* sp = static_cast<StateT*>(p.state) + ((sidx * p.num_v_heads + h) * D + row0) * D + col0;
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j) store4(sp + (r * 16) * D + j * 32, S[r][j]);
  }
  }  // items
}

// Resident CTAs of `Fn` on the current device (SMs x CTAs per SM), looked up once per device; its shared-memory limit is raised then.
template <auto Fn>
int resident_ctas(size_t smem, int* out) {
  static int cached[64] = {};
  int dev = 0;
  QLA_CHECK_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && cached[dev] > 0) {
    *out = cached[dev];
    return QLA_OK;
  }
  const int rc = ensure_dynamic_smem<Fn>(smem);
  if (rc != QLA_OK) return rc;
  int sms = 0, per_sm = 0;
  QLA_CHECK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  QLA_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, Fn, 128, smem));
  *out = sms * (per_sm > 0 ? per_sm : 1);
  if (dev >= 0 && dev < 64) cached[dev] = *out;
  return QLA_OK;
}

constexpr int kSms = 148;
enum Form { kPlain, kTree, kChain, kStep };  // recurrent_kernel without and with parents, recurrent_chain_kernel, recurrent_step_kernel
template <typename T, typename InterT, typename StateT, int R, Form kForm>
constexpr auto kernel_of() {
  if constexpr (kForm == kChain) return &recurrent_chain_kernel<T, InterT, StateT, R>;
  else if constexpr (kForm == kStep) return &recurrent_step_kernel<T, InterT, StateT, R>;
  else return &recurrent_kernel<T, InterT, StateT, R, kForm == kTree>;
}
template <typename T, typename InterT, typename StateT, int R, Form kForm>
int resident_tiles(int* out) {
  constexpr size_t smem = kRecStages * R * 4 * 128 * sizeof(typename StatePiece<StateT>::Raw);
  return resident_ctas<kernel_of<T, InterT, StateT, R, kForm>()>(smem, out);
}

template <typename T, typename InterT, typename StateT, int R, Form kForm>
int launch_recurrent_rows(const QlaRecurrentArgs& a, cudaStream_t stream) {
  const int64_t items = static_cast<int64_t>(a.num_seqs) * a.num_v_heads * (kHeadDim / (16 * R));
  QLA_CHECK_SUPPORTED(items < (int64_t(1) << 31), "too many (sequence, head) pairs");
  constexpr size_t smem = kRecStages * R * 4 * 128 * sizeof(typename StatePiece<StateT>::Raw);
  int resident = 0;
  const int rc = resident_tiles<T, InterT, StateT, R, kForm>(&resident);
  if (rc != QLA_OK) return rc;
  // one CTA per item while they all fit at once; otherwise as many CTAs as are resident, each walking the
  // items with stride gridDim.x
  const unsigned grid = static_cast<unsigned>(items < resident ? items : resident);
  QLA_CHECK_CUDA(launch_dependent(kernel_of<T, InterT, StateT, R, kForm>(), dim3(grid), dim3(128), smem, stream, a,
                                  static_cast<uint32_t>(items)));
  QLA_CHECK_CUDA(cudaGetLastError());
  return QLA_OK;
}

template <typename T, typename InterT, typename StateT, Form kForm>
int launch_recurrent_form(const QlaRecurrentArgs& a, int rows, cudaStream_t stream) {
  // (recurrent_kernel; the height of the other two comes with the call.)
  // Tiles of 16 rows while they are all resident at once, which spreads a small batch over the most SMs; a second round of
  // them costs the latency of every step again.  With the line at four tiles of 32 rows per SM: 96 heads of 7 tree steps 17.5 us, now
  // 13.2; 112 heads of 4 steps 11.4 -> 9.7; 144 heads of one step 7.0 -> 5.3, with a bf16 pool 6.8 -> 4.8.  (Just above the line it is
  // rough: 80 heads of 8 steps with fp32 scratch 14.3 with 16 rows, 14.7 with 32; of 4 steps 9.7 and 9.2; 92 of 8 15.5 and 14.8.)
  if (rows == 0) {
    const int64_t tiles = static_cast<int64_t>(a.num_seqs) * a.num_v_heads * (kHeadDim / 16);
    int resident = 2 * kSms;  // (at least: the smallest calls, which are host-bound, do not look it up)
    if (tiles > resident) {
      const int rc = resident_tiles<T, InterT, StateT, 1, kForm>(&resident);
      if (rc != QLA_OK) return rc;
    }
    rows = tiles <= resident ? 16 : 32;
    // A tree's tiles of 32 rows with fp32 scratch are resident three per SM, not four: a second round of them that is more than a
    // quarter full takes longer than two rounds of 16 rows.  128 / 136 / 144 / 147 heads of 8 steps, us: 16 rows 22.5 / 23.3 / 23.3 /
    // 23.9, 32 rows 21.3 / 23.5 / 24.9 / 26.0; of 3 steps 11.4 / 11.4 / 11.4 / 11.5 and 11.3 / 11.6 / 12.3 / 12.5.
    if constexpr (kForm == kTree && std::is_same<InterT, float>::value) {
      int resident32 = 0;
      if (rows == 32 && tiles <= 2 * static_cast<int64_t>(resident)) {
        const int rc = resident_tiles<T, InterT, StateT, 2, kForm>(&resident32);
        if (rc != QLA_OK) return rc;
        if (4 * (tiles / 2) > 5 * static_cast<int64_t>(resident32)) rows = 16;
      }
    }
  }
  return rows == 16 ? launch_recurrent_rows<T, InterT, StateT, 1, kForm>(a, stream)
                    : launch_recurrent_rows<T, InterT, StateT, 2, kForm>(a, stream);
}
// Several steps, of which every state is cached in 16 bits or none is: instructions are most of the time, and recurrent_chain_kernel has
// fewer of them (us, recurrent_kernel / recurrent_chain_kernel, 32 heads: 256 sequences of 4 steps 370 / 333, of 8 629 / 579, without a cache
// 330 / 273 and 558 / 464).  But five tiles of 32 rows are resident per SM, not four, and what a tile costs beside its steps (rows and
// gates of a block of four steps through shared memory) is paid for each tile and block.  So the rounds decide; us, recurrent_kernel / recurrent_chain_kernel,
// bf16 cache, states from HBM:
// - to two and a half tiles of 32 rows per SM the chain kernel, with 16 rows while every SM has one such tile: 16 heads of 4 steps 4.95 / 4.53, 74 heads
//   8.40 / 7.47, 80 heads of 8 14.5 / 13.2.  But above four steps its second block comes late where the steps are all there is (4 heads of 6
//   5.4 / 6.1, without a cache of 64 29 / 36), and a second block of one or two steps costs as much as one of four (64 heads of 6 9.5 / 9.7).
// - to one round of the general kernel that one (96 heads of 4 10.0 / 10.2, 132 of 8 15.7 / 17.1; eight tiles of 16 rows per SM 18.2), to one of the chain
//   kernel (185 heads) the chain kernel (160 heads of 4 13.4 / 11.3, of 8 19.9 / 17.7).
// - beyond, the general kernel where its last round is nearly full (288 heads of 4 18.0 / 19.3, 592 of 8 50.7 / 51.9) or, above four steps, has just begun (300 of
//   8 30.1 / 30.5, 448 of 8 40.6 / 42.3), and with a second block of one or two steps unless the chain kernel has a round less (256 of 5
//   20.1 / 21.7, 512 of 5 35.7 / 33.8).  With more and more rounds that matters less than the instructions.
// The lines are rough: around them the two differ by up to 4 %.
template <typename T, typename InterT, typename StateT>
int takes_chain(const QlaRecurrentArgs& a, int64_t tiles, bool* chain, int* rows) {
  const int steps = a.tokens_per_seq;
  const bool cached = a.inter != nullptr, late = cached && steps > 4, stub = cached && (steps == 5 || steps == 6);
  if (2 * tiles <= 5 * kSms) {
    *chain = steps <= 4 || tiles > (stub ? 2 : 1) * kSms;
    if (*rows == 0) *rows = (*chain ? 2 : 1) * tiles <= kSms ? 16 : 32;
    return QLA_OK;
  }
  if (*rows == 0) *rows = 32;
  int general = 0, own = 0;
  int rc = resident_tiles<T, InterT, StateT, 2, kPlain>(&general);
  if (rc == QLA_OK) rc = resident_tiles<T, InterT, StateT, 2, kChain>(&own);
  if (rc != QLA_OK) return rc;
  const int64_t rounds = (tiles + general - 1) / general, fill = 20 * (tiles - (rounds - 1) * general);  // (20ths of a round)
  const bool fewer = (tiles + own - 1) / own < rounds;
  if (rounds == 1 || tiles <= own) *chain = rounds > 1;
  else if (stub && rounds > 4) *chain = rounds > (steps == 5 ? 10 : 7);
  else if (rounds > (late || steps == 2 ? 4 : 2)) *chain = true;
  else
    *chain = (fewer || !stub) && fill >= (!late ? 0 : rounds == 3 ? 3 : 5) * general &&
             fill <= (steps == 3 || steps == 4 ? 17 : late && !fewer ? 14 : 15) * general;
  return QLA_OK;
}
// One step: the kernel without the loop, of which five tiles of 32 rows are resident per SM, not four, and seven of 16 (us, recurrent_kernel /
// recurrent_step_kernel, states from HBM, 32 heads: bf16 pools 16 sequences 11.9 / 10.1, 64 37.6 / 30.4, 128 71.0 / 57.0; fp32 pools
// 4 6.1 / 5.8, 12 12.2 / 10.7, 24 20.0 / 18.0, 32 24.5 / 23.5, 48 34.8 / 35.0, 64 44.7 / 47.3, 256 163.6 / 187: from about 1200 fp32 heads on HBM is the
// bound, and the memory does better with fewer tiles in flight).  fp32 pools, states from HBM and in L2:
// - to seven tiles of 16 rows per SM this one (120 heads 6.70 / 6.57, 5.01 / 4.61), with 32 rows where three and a half of 16 per SM are passed and two
//   and a half of 32 are not (72 heads, 16 and 32 rows 5.80 / 5.25, 4.49 / 4.04; 96 heads 6.23 / 6.53, 4.50 / 5.01); to one round of the general kernel
//   that one (140 heads 7.00 / 7.00, 5.06 / 5.23);
// - beyond this one (160 heads 8.70 / 7.17, 6.54 / 5.29), except where more than two thirds of the general kernel's second round are full (296 heads 11.1 /
//   11.1, 8.14 / 8.48).
// bf16 pools the same beyond one round of the general kernel (160 heads 7.55 / 5.76, 6.09 / 4.61; 240 8.70 / 8.19, 7.17 / 6.83; 280 8.92 / 8.62, 7.22 / 7.28;
// 296 9.13 / 9.00, 7.28 / 7.34; 300 10.8 / 8.9, 8.54 / 7.34; 512 15.3 / 12.7, 12.7 / 10.4); to there the general one (120 heads 5.16 / 5.21, 4.44 / 4.61).
template <typename T, typename InterT, typename StateT>
int takes_step(const QlaRecurrentArgs& a, int64_t tiles, bool* step, int* rows) {
  constexpr bool kState16 = std::is_same<StateT, __nv_bfloat16>::value;
  *step = kState16 ? tiles > 2 * kSms : tiles <= 4 * 1024;
  if (!*step) return QLA_OK;
  if (tiles <= 2 * kSms) {
    if (*rows == 0) *rows = 4 * tiles > 7 * kSms ? 32 : 16;
    return QLA_OK;
  }
  int general = 0, low = 0;
  int rc = resident_tiles<T, InterT, StateT, 2, kPlain>(&general);
  if (rc == QLA_OK) rc = resident_tiles<T, InterT, StateT, 1, kStep>(&low);
  if (rc != QLA_OK) return rc;
  if (tiles <= general) *step = !kState16 && 2 * tiles <= low;
  else *step = 3 * tiles <= 5 * general || tiles > 2 * general;
  if (*rows == 0 && *step) *rows = 2 * tiles > low || 2 * tiles <= 5 * kSms ? 32 : 16;
  return QLA_OK;
}
template <typename T, typename InterT, typename StateT>
int launch_recurrent_state(const QlaRecurrentArgs& a, int rows, cudaStream_t stream) {
  const int64_t tiles = static_cast<int64_t>(a.num_seqs) * a.num_v_heads * (kHeadDim / 32);
  if (a.tokens_per_seq == 1) {
    bool step = false;
    const int rc = takes_step<T, InterT, StateT>(a, tiles, &step, &rows);
    if (rc != QLA_OK) return rc;
    if (step) return launch_recurrent_form<T, InterT, StateT, kStep>(a, rows, stream);
  }
  if (a.parents != nullptr) return launch_recurrent_form<T, InterT, StateT, kTree>(a, rows, stream);
  // (with fp32 states in the cache HBM is the bound: 256 sequences of 4 steps 480 / 481 us, 16 of 8 50.1 / 51.7)
  if (a.tokens_per_seq > 1 && (a.inter == nullptr || a.inter_dtype == QLA_DT_BF16)) {
    bool chain = false;
    const int rc = takes_chain<T, InterT, StateT>(a, tiles, &chain, &rows);
    if (rc != QLA_OK) return rc;
    if (chain) return launch_recurrent_form<T, InterT, StateT, kChain>(a, rows, stream);
  }
  return launch_recurrent_form<T, InterT, StateT, kPlain>(a, rows, stream);
}
template <typename T, typename InterT>
int launch_recurrent(const QlaRecurrentArgs& a, int rows, cudaStream_t stream) {
  return a.state_dtype == QLA_DT_BF16 ? launch_recurrent_state<T, InterT, __nv_bfloat16>(a, rows, stream)
                                      : launch_recurrent_state<T, InterT, float>(a, rows, stream);
}

}  // namespace
}  // namespace qla

namespace qla {
namespace {
// One CTA per (sequence, v-head): 128 x 128 values = 64 KiB of fp32 state, 128-bit accesses.
template <typename InterT>
__global__ void __launch_bounds__(256) state_commit_kernel(const QlaStateCommitArgs a) {
  const int n = blockIdx.x, hv = blockIdx.y;
  const int acc = a.accepted[n];
  if (acc <= 0) return;
  const int64_t sslot = a.state_indices ? a.state_indices[n] : n;
  const int64_t islot = a.inter_indices ? a.inter_indices[n] : n;
  if (acc > a.inter_steps || sslot < 0 || sslot >= a.state_slots || islot < 0 || islot >= a.inter_slots) {
    if (a.status != nullptr && threadIdx.x == 0) atomicCAS(a.status, 0, kStatusBadIndex);
    return;
  }
  constexpr int kElems = kHeadDim * kHeadDim;
  const InterT* src = static_cast<const InterT*>(a.inter) +
                      ((islot * a.inter_steps + (acc - 1)) * a.num_v_heads + hv) * static_cast<int64_t>(kElems);
  const int64_t dst_off = (sslot * a.num_v_heads + hv) * static_cast<int64_t>(kElems);
  float* dst = static_cast<float*>(a.state) + dst_off;
  __nv_bfloat16* dst16 = static_cast<__nv_bfloat16*>(a.state) + dst_off;
  for (int i = threadIdx.x * 8; i < kElems; i += 256 * 8) {
    float x[8];
    if (sizeof(InterT) == 4) {
      const float4 lo = *reinterpret_cast<const float4*>(src + i), hi = *reinterpret_cast<const float4*>(src + i + 4);
      x[0] = lo.x; x[1] = lo.y; x[2] = lo.z; x[3] = lo.w; x[4] = hi.x; x[5] = hi.y; x[6] = hi.z; x[7] = hi.w;
    } else {
      const uint4 raw = *reinterpret_cast<const uint4*>(src + i);
      const InterT* e = reinterpret_cast<const InterT*>(&raw);
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] = Cvt<InterT>::to_f32(e[j]);
    }
    if (a.state_dtype == QLA_DT_BF16) {
      const F2 lo[2] = {f2(x[0], x[1]), f2(x[2], x[3])}, hi[2] = {f2(x[4], x[5]), f2(x[6], x[7])};
      store4(dst16 + i, lo);
      store4(dst16 + i + 4, hi);
    } else {
      *reinterpret_cast<float4*>(dst + i) = make_float4(x[0], x[1], x[2], x[3]);
      *reinterpret_cast<float4*>(dst + i + 4) = make_float4(x[4], x[5], x[6], x[7]);
    }
  }
}
}  // namespace
}  // namespace qla

namespace qla {
// (32-row tiles of an fp32 pool: the largest variant; 16-row tiles and bf16 pools use a half / a quarter)
void launch_info_recurrent_kernel(int* block_threads, size_t* dynamic_smem_bytes) {
  *block_threads = 128;
  *dynamic_smem_bytes = kRecStages * 2 * 4 * 128 * sizeof(float4);
}
}  // namespace qla

namespace qla {
namespace {
bool starts_on(const void* p, unsigned bytes) { return (reinterpret_cast<uintptr_t>(p) & (bytes - 1)) == 0; }
constexpr const char* kAlignment = "q and k must start on 8 bytes, states and cached states on 16 (bf16 in the update: 8)";
}  // namespace
}  // namespace qla

extern "C" QLA_API int qla_state_commit(const QlaStateCommitArgs* args, void* stream) {
  using namespace qla;
  QLA_CHECK_ARG(args != nullptr, "args is NULL");
  const QlaStateCommitArgs& a = *args;
  QLA_CHECK_ARG(a.num_seqs >= 0 && a.num_v_heads > 0, "bad sizes");
  if (a.num_seqs == 0) return QLA_OK;
  QLA_CHECK_ARG(a.inter && a.accepted && a.state, "NULL tensor pointer");
  QLA_CHECK_ARG(a.inter_slots > 0 && a.inter_steps > 0 && a.state_slots > 0, "extents must be positive");
  QLA_CHECK_SUPPORTED(a.inter_dtype == QLA_DT_F32 || a.inter_dtype == QLA_DT_BF16,
                      "intermediate_states_buffer must be fp32 or bf16");
  QLA_CHECK_SUPPORTED(a.state_dtype == QLA_DT_F32 || a.state_dtype == QLA_DT_BF16, "the state pool must be fp32 or bf16");
  QLA_CHECK_ARG(starts_on(a.inter, 16) && starts_on(a.state, a.state_dtype == QLA_DT_BF16 ? 8 : 16), kAlignment);
  dim3 grid(a.num_seqs, a.num_v_heads);
  if (a.inter_dtype == QLA_DT_F32) state_commit_kernel<float><<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(a);
  else state_commit_kernel<__nv_bfloat16><<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(a);
  QLA_CHECK_CUDA(cudaGetLastError());
  return QLA_OK;
}

extern "C" QLA_API int qla_recurrent_update(const QlaRecurrentArgs* args, void* stream) {
  using namespace qla;
  QLA_CHECK_ARG(args != nullptr, "args is NULL");
  const QlaRecurrentArgs& a = *args;
  QLA_CHECK_ARG(a.num_seqs >= 0 && a.total_tokens >= 0, "negative sizes");
  if (a.num_seqs == 0 || a.total_tokens == 0) return QLA_OK;
  QLA_CHECK_ARG(a.num_k_heads > 0 && a.num_v_heads > 0 && a.num_v_heads % a.num_k_heads == 0,
                "num_value_heads must be divisible by num_key_heads");
  QLA_CHECK_ARG(a.q && a.k && a.v && a.a && a.b && a.o && a.state, "NULL tensor pointer");
  QLA_CHECK_ARG((a.flags & QLA_REC_A_IS_LOG_DECAY) || (a.A_log && a.dt_bias),
                "A_log and dt_bias are required unless a_is_log_decay");
  QLA_CHECK_ARG(a.tokens_per_seq > 0 || a.cu_seqlens != nullptr,
                "either tokens_per_seq > 0 or cu_seqlens must be given");
  QLA_CHECK_ARG(a.tokens_per_seq == 0 ||
                    static_cast<int64_t>(a.tokens_per_seq) * a.num_seqs == a.total_tokens,
                "total_tokens must equal num_seqs * tokens_per_seq");
  QLA_CHECK_SUPPORTED(a.qkv_dtype == QLA_DT_BF16 || a.qkv_dtype == QLA_DT_F16,
                      "q, k, v must be bf16 or fp16");
  QLA_CHECK_ARG(a.state_slots > 0, "state_slots must be positive");
  QLA_CHECK_SUPPORTED(a.state_dtype == QLA_DT_F32 || a.state_dtype == QLA_DT_BF16,
                      "initial_state_source must be fp32 or bf16");
  // (the pieces in which the kernel moves them)
  QLA_CHECK_ARG(starts_on(a.q, 8) && starts_on(a.k, 8) && starts_on(a.state, a.state_dtype == QLA_DT_BF16 ? 8 : 16) &&
                    starts_on(a.inter, a.inter_dtype == QLA_DT_BF16 ? 8 : 16), kAlignment);
  QLA_CHECK_ARG(a.parents == nullptr || a.parents_steps > 0, "parents_steps (second extent of parents) must be positive");
  QLA_CHECK_ARG(a.parents == nullptr || a.tokens_per_seq <= a.parents_steps,
                "retrieve_parent_token has fewer columns than tokens per sequence");
  if (a.inter != nullptr) {
    QLA_CHECK_ARG(a.inter_slots > 0 && a.inter_steps > 0, "inter extents must be positive");
    QLA_CHECK_SUPPORTED(a.inter_dtype == QLA_DT_F32 || a.inter_dtype == QLA_DT_BF16,
                        "intermediate_states_buffer must be fp32 or bf16");
  }
  QLA_CHECK_ARG(a.parents == nullptr || a.inter != nullptr,
                "retrieve_parent_token needs intermediate_states_buffer");
  QLA_CHECK_ARG(a.rows_per_cta == 0 || a.rows_per_cta == 16 || a.rows_per_cta == 32,
                "rows_per_cta must be 0, 16 or 32");
  const int rows = a.rows_per_cta;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool inter_bf16 = a.inter != nullptr && a.inter_dtype == QLA_DT_BF16;
  if (a.qkv_dtype == QLA_DT_BF16) {
    return inter_bf16 ? launch_recurrent<__nv_bfloat16, __nv_bfloat16>(a, rows, s)
                      : launch_recurrent<__nv_bfloat16, float>(a, rows, s);
  }
  return inter_bf16 ? launch_recurrent<__half, __nv_bfloat16>(a, rows, s)
                    : launch_recurrent<__half, float>(a, rows, s);
}
