// The layer's prologue maps (q / k L2 norm, gate activation, beta sigmoid) around the backward of a forward that applied
// them inside its kernels.  Reference: separate differentiable passes in front of the op (l2norm,
// flash_qla/utils/math.py:14-21 via chunk/__init__.py:332-334; gate formulas recurrent_fused.py:346-487).
//
// All of it is bound by HBM: rows are read and written once, 16 bytes per lane.  As torch operations these maps were
// some forty launches and 15 passes over fp32 copies of q, k, dq, dk: 1.5 ms of a 2.4 ms step at 12 800 tokens with
// 16 / 32 heads, against 0.16 ms here.
#include "common.cuh"

namespace qla {
namespace {

constexpr int kRowThreads = 16;  // a row of 128 16-bit values: 16 bytes per lane
constexpr int kBlock = 256;

__device__ __forceinline__ float row_sum(float x) {
#pragma unroll
  for (int off = 1; off < kRowThreads; off <<= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
  return x;
}
template <typename T>
__device__ __forceinline__ void unpack8(const uint4& raw, float (&x)[8]) {
  const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
  for (int j = 0; j < 8; ++j) x[j] = Cvt<T>::to_f32(e[j]);
}
template <typename T>
__device__ __forceinline__ uint4 pack8(const float (&x)[8]) {
  uint4 raw;
  T* e = reinterpret_cast<T*>(&raw);
#pragma unroll
  for (int j = 0; j < 8; ++j) e[j] = Cvt<T>::from_f32(x[j]);
  return raw;
}

// kBackward = false: qn, kn = x r with r = (sum x^2 + eps)^-1/2, rounded to 16 bits.
// kBackward = true: with x_hat = x r (rounded, the value the backward worked with),
//   dx = r (dx_hat - x_hat (x_hat . dx_hat)), in place over dq / dk.
template <typename T, bool kBackward>
__global__ void __launch_bounds__(kBlock) norm_rows_kernel(const QlaLayerBwdArgs a) {
  grid_dep_wait();
  grid_dep_launch();
  const int lane = threadIdx.x & (kRowThreads - 1);
  const int64_t stride = static_cast<int64_t>(gridDim.x) * (kBlock / kRowThreads);
  // whole warps stay in the loop (the shuffles of row_sum need both half warps): the bound is that of the warp's
  // first row, a row past the end repeats the last one and is not stored
  for (int64_t first = static_cast<int64_t>(blockIdx.x) * (kBlock / kRowThreads) + (threadIdx.x >> 5) * 2; first < 2 * a.rows;
       first += stride) {
    const int64_t mine = first + ((threadIdx.x >> 4) & 1);
    const bool store = mine < 2 * a.rows;
    const int64_t at = store ? mine : 2 * a.rows - 1;
    const bool is_k = at >= a.rows;
    const int64_t off = (is_k ? at - a.rows : at) * 16 + lane;  // in 16-byte pieces
    float x[8];
    unpack8<T>(static_cast<const uint4*>(is_k ? a.k : a.q)[off], x);
    uint4* io = static_cast<uint4*>(kBackward ? (is_k ? a.dk : a.dq) : (is_k ? a.kn : a.qn));
    float d[8];
    if (kBackward) unpack8<T>(io[off], d);
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) ss = fmaf(x[j], x[j], ss);
    const float r = rsqrtf(row_sum(ss) + a.eps);
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] *= r;
    if (kBackward) {
      float dot = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        x[j] = Cvt<T>::to_f32(Cvt<T>::from_f32(x[j]));
        dot = fmaf(x[j], d[j], dot);
      }
      dot = row_sum(dot);
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] = r * (d[j] - x[j] * dot);
    }
    if (store) io[off] = pack8<T>(x);
  }
}

__device__ __forceinline__ void store_scalar(void* p, int dtype, int64_t i, float x) {
  if (dtype == QLA_DT_F32) static_cast<float*>(p)[i] = x;
  else if (dtype == QLA_DT_BF16) static_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(x);
  else static_cast<__half*>(p)[i] = __float2half_rn(x);
}

constexpr int kGateTokens = 64;  // tokens of a block: sums over tokens are formed per block, then over blocks in order

// Gate and beta of kGateTokens tokens, all heads: a warp walks heads (coalesced) for its share of the tokens.
__global__ void __launch_bounds__(kBlock) gate_bwd_kernel(const QlaLayerBwdArgs a) {
  grid_dep_wait();
  grid_dep_launch();
  __shared__ float part[kBlock / 32][32][2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t t0 = static_cast<int64_t>(blockIdx.x) * kGateTokens;
  float* out = static_cast<float*>(a.workspace) + static_cast<int64_t>(blockIdx.x) * 2 * a.num_v_heads;
  for (int h0 = 0; h0 < a.num_v_heads; h0 += 32) {
    const int h = h0 + lane;
    const bool ok = h < a.num_v_heads;
    float coef = 0.f, bias = 0.f, sum_a = 0.f, sum_d = 0.f;
    if (ok && a.da != nullptr) {
      coef = -expf(a.A_log[h]);
      bias = a.dt_bias[h];
    }
    for (int t = warp; t < kGateTokens; t += kBlock / 32) {
      const int64_t tok = t0 + t;
      if (tok >= a.tokens || !ok) continue;
      const int64_t i = tok * a.num_v_heads + h;
      if (a.da != nullptr) {
        // g = coef softplus(x), softplus with beta 1 and threshold 20 (the forward's)
        const float x = load_scalar(a.a, a.gate_dtype, i) + bias, dg = a.dg[i];
        const float sp = x <= 20.f ? log1pf(expf(x)) : x;
        const float da = dg * coef * (x <= 20.f ? 1.f / (1.f + expf(-x)) : 1.f);
        store_scalar(a.da, a.gate_dtype, i, da);
        sum_a = fmaf(dg, coef * sp, sum_a);
        sum_d += da;
      }
      if (a.db_raw != nullptr) {
        const float b = a.beta[i];
        store_scalar(a.db_raw, a.beta_dtype, i, a.db[i] * b * (1.f - b));
      }
    }
    if (a.da == nullptr) continue;
    part[warp][lane][0] = sum_a;
    part[warp][lane][1] = sum_d;
    __syncthreads();
    if (warp < 2 && ok) {
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < kBlock / 32; ++w) s += part[w][lane][warp];
      out[warp * a.num_v_heads + h] = s;
    }
    __syncthreads();
  }
}

// dsums[0 | 1][h] = sum over the blocks of gate_bwd_kernel; one block per 8 values, 32 threads each.
__global__ void __launch_bounds__(kBlock) gate_sums_kernel(const float* partial, int blocks, int num_heads, float* dsums) {
  grid_dep_wait();
  grid_dep_launch();
  const int lane = threadIdx.x & 31, v = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5);
  if (v >= 2 * num_heads) return;
  float s = 0.f;
  for (int b = lane; b < blocks; b += 32) s += partial[static_cast<int64_t>(b) * 2 * num_heads + v];
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if (lane == 0) dsums[v] = s;
}

int gate_blocks(const QlaLayerBwdArgs& a) { return static_cast<int>((a.tokens + kGateTokens - 1) / kGateTokens); }

template <typename T>
int launch_rows(const QlaLayerBwdArgs& a, cudaStream_t stream) {
  const int64_t blocks = (2 * a.rows + kBlock / kRowThreads - 1) / (kBlock / kRowThreads);
  // eight resident blocks per SM fill the memory pipeline; more rows than that are walked
  const dim3 grid(static_cast<unsigned>(blocks < 148 * 8 ? blocks : 148 * 8));
  if (a.qn != nullptr) QLA_CHECK_CUDA(launch_dependent(norm_rows_kernel<T, false>, grid, dim3(kBlock), 0, stream, a));
  if (a.dq != nullptr) QLA_CHECK_CUDA(launch_dependent(norm_rows_kernel<T, true>, grid, dim3(kBlock), 0, stream, a));
  return QLA_OK;
}

}  // namespace
}  // namespace qla

extern "C" QLA_API size_t qla_layer_bwd_workspace_bytes(const QlaLayerBwdArgs* a) {
  if (a == nullptr || a->da == nullptr || a->tokens <= 0) return 0;
  return static_cast<size_t>(qla::gate_blocks(*a)) * 2 * a->num_v_heads * sizeof(float);
}

extern "C" QLA_API int qla_layer_bwd(const QlaLayerBwdArgs* args, void* stream_) {
  using namespace qla;
  QLA_CHECK_ARG(args != nullptr, "args is NULL");
  const QlaLayerBwdArgs& a = *args;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  QLA_CHECK_ARG(a.rows >= 0 && a.tokens >= 0, "negative sizes");
  if (a.rows > 0) {
    QLA_CHECK_SUPPORTED(a.qkv_dtype == QLA_DT_BF16 || a.qkv_dtype == QLA_DT_F16, "q, k must be bf16 or fp16");
    QLA_CHECK_ARG(a.q && a.k && (!a.qn == !a.kn) && (!a.dq == !a.dk), "NULL row tensor");
    const int rc = a.qkv_dtype == QLA_DT_BF16 ? launch_rows<__nv_bfloat16>(a, stream) : launch_rows<__half>(a, stream);
    if (rc != QLA_OK) return rc;
  }
  if (a.tokens == 0 && a.dsums != nullptr && a.num_v_heads > 0)  // the sums over no tokens
    QLA_CHECK_CUDA(cudaMemsetAsync(a.dsums, 0, 2 * sizeof(float) * a.num_v_heads, stream));
  if (a.tokens == 0 || (a.da == nullptr && a.db_raw == nullptr)) return QLA_OK;
  QLA_CHECK_ARG(a.num_v_heads > 0, "num_v_heads must be positive");
  QLA_CHECK_ARG(a.da == nullptr || (a.a && a.A_log && a.dt_bias && a.dg && a.dsums && a.workspace), "NULL gate tensor");
  QLA_CHECK_ARG(a.db_raw == nullptr || (a.beta && a.db), "NULL beta tensor");
  QLA_CHECK_CUDA(launch_dependent(gate_bwd_kernel, dim3(gate_blocks(a)), dim3(kBlock), 0, stream, a));
  if (a.da != nullptr)
    QLA_CHECK_CUDA(launch_dependent(gate_sums_kernel, dim3((2 * a.num_v_heads + kBlock / 32 - 1) / (kBlock / 32)), dim3(kBlock), 0,
                                    stream, static_cast<const float*>(a.workspace), gate_blocks(a), a.num_v_heads, a.dsums));
  return QLA_OK;
}
