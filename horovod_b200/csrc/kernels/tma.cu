// Tensor maps for tma.cuh.
#include "tma.cuh"

namespace hvd {
namespace kern {

namespace {

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                              const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                              const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn Encode() {
  static const EncodeFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      p = nullptr;
    }
    return reinterpret_cast<EncodeFn>(p);
  }();
  return fn;
}

}  // namespace

bool TmaAvailable() { return Encode() != nullptr; }

bool MakeMap(CUtensorMap* map, const void* p, bool bf16, int64_t channels, int64_t rows1,
             int64_t rows2, int64_t pitch1, int64_t pitch2, int box1, int box2) {
  if (Encode() == nullptr) return false;
  const cuuint64_t sizes[3] = {static_cast<cuuint64_t>(channels), static_cast<cuuint64_t>(rows1),
                               static_cast<cuuint64_t>(rows2)};
  const cuuint64_t pitches[2] = {static_cast<cuuint64_t>(pitch1) * 2,
                                 static_cast<cuuint64_t>(pitch2) * 2};
  const cuuint32_t box[3] = {64, static_cast<cuuint32_t>(box1), static_cast<cuuint32_t>(box2)};
  const cuuint32_t steps[3] = {1, 1, 1};
  return Encode()(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                  3, const_cast<void*>(p), sizes, pitches, box, steps,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace kern
}  // namespace hvd
