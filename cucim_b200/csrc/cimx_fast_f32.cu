// cimx_fast_f32.cu — instantiations of the volume kernel (cimx_vol.cuh) for
// float input. Split by input dtype so the kernels compile in parallel.
#include "cimx_vol.cuh"

namespace cimx {

int launch_vol_f32(const VolArgs& v, int tout, cudaStream_t st) {
  if (tout == DT_F32) return vol::launch_vol_td<float, float>(v, st);
  return CIMX_FUSED_DECLINED;
}

}  // namespace cimx
