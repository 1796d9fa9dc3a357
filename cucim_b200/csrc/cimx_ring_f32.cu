// cimx_ring_f32.cu — long float32 passes along a strided axis
// (cimx_ring.cuh).
#include "cimx_ring.cuh"

namespace cimx {

int launch_ring_f32(const PassDesc& d, const float* w, int K, int anchor, bool skip,
                    const void* in, void* out, cudaStream_t st) {
  using namespace ring;
  if (skip_kind(w, K, skip) == 2) {
    if (K <= 65) return launch_ring_k<65, 65, true>(d, w, K, anchor, skip, in, out, st);
    return launch_ring_k<129, 129, true>(d, w, K, anchor, skip, in, out, st);
  }
  switch ((K + 6) / 8 * 8 + 1) {
#define CIMX_KT(K_) \
  case K_: return launch_ring_k<K_, 8, false>(d, w, K, anchor, skip, in, out, st);
    CIMX_KT(25) CIMX_KT(33) CIMX_KT(41) CIMX_KT(49) CIMX_KT(57) CIMX_KT(65) CIMX_KT(73)
    CIMX_KT(81) CIMX_KT(89) CIMX_KT(97) CIMX_KT(105) CIMX_KT(113) CIMX_KT(121) CIMX_KT(129)
#undef CIMX_KT
    default: return CIMX_FUSED_DECLINED;
  }
}

}  // namespace cimx
