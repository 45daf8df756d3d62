// Host side of TMA: tensor-map encoding through the driver entry point obtained from the runtime.
#include "ptx_sm100.cuh"

namespace qla {

EncodeTiledFn get_encode_tiled() {
  static EncodeTiledFn fn = []() -> EncodeTiledFn {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

namespace {
int encode(CUtensorMap* out, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides,
           const cuuint32_t* box, bool swizzle128, bool is_bf16) {
  EncodeTiledFn enc = get_encode_tiled();
  if (enc == nullptr) {
    set_last_error("cuTensorMapEncodeTiled is not available from the driver");
    return QLA_ERR_CUDA;
  }
  if ((reinterpret_cast<uintptr_t>(base) & 15u) != 0) {
    set_last_error("tensor base address must be 16-byte aligned for TMA");
    return QLA_ERR_INVALID_ARG;
  }
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  auto make = [&]() {
    return enc(out, is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, rank, const_cast<void*>(base),
               dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               swizzle128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  CUresult r = make();
  if (r == CUDA_ERROR_INVALID_CONTEXT) {
    // A thread that has not used the runtime yet (autograd's, when its allocations came from the cache) has no current
    // context, and this is a driver call: selecting the device it is on brings the primary context about.
    int dev = 0;
    QLA_CHECK_CUDA(cudaGetDevice(&dev));
    QLA_CHECK_CUDA(cudaSetDevice(dev));
    r = make();
  }
  if (r != CUDA_SUCCESS) {
    set_last_error("cuTensorMapEncodeTiled failed with CUresult %d (extents %llu x %llu x %llu)", static_cast<int>(r),
                   static_cast<unsigned long long>(dims[0]), static_cast<unsigned long long>(dims[1]),
                   static_cast<unsigned long long>(dims[2]));
    return QLA_ERR_CUDA;
  }
  return QLA_OK;
}
}  // namespace

int make_tmap_3d(CUtensorMap* out, const void* base, uint64_t tokens, uint64_t heads, uint64_t width,
                 uint32_t box_rows, uint32_t box_width, bool swizzle128, bool is_bf16) {
  const cuuint64_t dims[3] = {width, heads, tokens};
  const cuuint64_t strides[2] = {width * 2, heads * width * 2};
  const cuuint32_t box[3] = {box_width, 1, box_rows};
  return encode(out, base, 3, dims, strides, box, swizzle128, is_bf16);
}

int make_tmap_halves(CUtensorMap* out, const void* base, uint64_t tokens, uint64_t heads, uint32_t box_rows, bool is_bf16) {
  const cuuint64_t dims[4] = {64, heads, tokens, 2};
  const cuuint64_t strides[3] = {256, heads * 256, 128};
  const cuuint32_t box[4] = {64, 1, box_rows, 2};
  return encode(out, base, 4, dims, strides, box, true, is_bf16);
}

}  // namespace qla
