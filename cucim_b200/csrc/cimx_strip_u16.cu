// cimx_strip_u16.cu — strip and column kernels (cimx_strip.cuh) for uint16_t
// input.
#include "cimx_strip.cuh"

namespace cimx {

int launch_strip_u16(const SlabArgs& a, int tout, cudaStream_t st) {
  if (tout == DT_F32) return strip::launch_strip_td<uint16_t, float>(a, st);
  if (tout == DT_U16) return strip::launch_strip_td<uint16_t, uint16_t>(a, st);
  return CIMX_FUSED_DECLINED;
}

int launch_columns_u16(const PassDesc& d, const float* w, int K, int anchor, bool skip,
                       const void* in, int tout, void* out, cudaStream_t st) {
  using strip::launch_columns_td;
  if (tout == DT_F32) return launch_columns_td<uint16_t, float>(d, w, K, anchor, skip, in, out, st);
  if (tout == DT_U16) return launch_columns_td<uint16_t, uint16_t>(d, w, K, anchor, skip, in, out, st);
  return CIMX_FUSED_DECLINED;
}

}  // namespace cimx
