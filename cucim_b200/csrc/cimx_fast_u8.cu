// cimx_fast_u8.cu — instantiations of the volume kernel (cimx_vol.cuh) for
// uint8_t input. Split by input dtype so the kernels compile in parallel.
#include "cimx_vol.cuh"

namespace cimx {

int launch_vol_u8(const VolArgs& v, int tout, cudaStream_t st) {
  if (tout == DT_F32) return vol::launch_vol_td<uint8_t, float>(v, st);
  if (tout == DT_U8) return vol::launch_vol_td<uint8_t, uint8_t>(v, st);
  if (tout == DT_U16) return vol::launch_vol_td<uint8_t, uint16_t>(v, st);
  return CIMX_FUSED_DECLINED;
}

}  // namespace cimx
