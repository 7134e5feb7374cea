// Host side of the TMA support: cuTensorMapEncodeTiled is looked up through the runtime
// (cudaGetDriverEntryPoint), so the library does not link against libcuda.
#include <mutex>

#include "fmb_tma.cuh"

namespace fmb {

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

int make_tmap_3d(CUtensorMap* map, const void* base, int dtype, uint64_t d, uint64_t heads, uint64_t rows,
                 uint64_t head_stride_bytes, uint64_t row_stride_bytes, uint32_t box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(FMB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  const cuuint64_t gdim[3] = {d, heads, rows > 0 ? rows : 1};
  const cuuint64_t gstride[2] = {head_stride_bytes, row_stride_bytes};
  const cuuint32_t box[3] = {64, 1, box_rows};
  const cuuint32_t estride[3] = {1, 1, 1};
  const CUresult r = fn(map, dtype == FMB_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3,
                        const_cast<void*>(base), gdim, gstride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return fail(FMB_ERR_CUDA, "cuTensorMapEncodeTiled failed (code %d): d %llu heads %llu rows %llu strides %llu, %llu", (int)r,
                (unsigned long long)d, (unsigned long long)heads, (unsigned long long)rows,
                (unsigned long long)head_stride_bytes, (unsigned long long)row_stride_bytes);
  return FMB_OK;
}

}  // namespace fmb
