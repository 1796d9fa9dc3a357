// cimx_strip_f32.cu — strip and column kernels (cimx_strip.cuh) for float32
// input.
#include "cimx_strip.cuh"

namespace cimx {

int launch_strip_f32(const SlabArgs& a, int tout, cudaStream_t st) {
  return tout == DT_F32 ? strip::launch_strip_td<float, float>(a, st) : CIMX_FUSED_DECLINED;
}

int launch_columns_f32(const PassDesc& d, const float* w, int K, int anchor, bool skip,
                       const void* in, int tout, void* out, cudaStream_t st) {
  return tout == DT_F32
             ? strip::launch_columns_td<float, float>(d, w, K, anchor, skip, in, out, st)
             : CIMX_FUSED_DECLINED;
}

}  // namespace cimx
