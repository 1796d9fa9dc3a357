// cimx_fused.h — entry into the fast kernels of the plain path (cimx_vol.cuh
// and cimx_strip.cuh, instantiated per input dtype in
// cimx_{fast,strip}_{f32,u16,u8}.cu)
// and the dispatcher that decides whether a pass list can use them
// (cimx_fused.cu).
#pragma once

#include "cimx_internal.h"

namespace cimx {

// Returned by try_fused when no fast kernel covers the pass list; the caller
// then runs the passes one launch at a time.
constexpr int CIMX_FUSED_DECLINED = 1;

constexpr int kSlabMaxK = 65;   // longest pass the strip and column kernels take
constexpr int kLongMaxK = 129;  // the same for a float32 pass of its own: as far as
                                // k_ring and k_strip are instantiated

// One pass of the strip and volume kernels (float32 weights, already trimmed).
struct SlabPass {
  int K, anchor, mode;
  double cval;
  int cval_as_input, dt, skip, pad;
  float w[kLongMaxK];
};

struct SlabArgs {
  const void* in;
  void* out;
  long long B, Y, X;
  int has_y, has_x;  // has_y 0: py is the identity (one tap of 1)
  int add;             // float32 results are added to what `out` holds
  SlabPass py, px;
};

// The three passes of a 3-D filter (z, y, x over the last three axes), for
// the single-launch volume kernel (cimx_vol.cuh).
struct VolArgs {
  const void* in;
  void* out;
  long long B, Z, Y, X;
  int zchunk;  // slices per CTA; 0: chosen from the grid size
  SlabPass pz, py, px;
};

// Tap-count bounds of the strip kernels' instantiations (cimx_strip.cuh): steps
// of four for float32 (every gaussian length is odd, the most common are
// bounds themselves), of eight for the integer types.
constexpr int kt_step(size_t elem) { return elem == 4 ? 4 : 8; }
constexpr int kt_bound(size_t elem, int K) {
  return K <= 5 ? 5 : K <= 9 ? 9 : 9 + (K - 9 + kt_step(elem) - 1) / kt_step(elem) * kt_step(elem);
}

// What the skip rule leaves out of a pass: 0 nothing, 1 only the centre tap
// (an odd Gaussian derivative), 2 others.
inline int skip_kind(const float* w, int K, bool skip) {
  if (!skip) return 0;
  for (int k = 0; k < K; ++k)
    if (w[k] == 0.f && k != K / 2) return 2;
  return (K & 1) ? 1 : 2;
}

// Runs the whole pass list `ds` (already resolved against the input shape)
// in fast launches when they cover it. Returns CIMX_OK, a negative error, or
// CIMX_FUSED_DECLINED (nothing was launched). `add` (float32): out += the
// result, rounded like a pass of its own; declined unless the last launch is a
// strip launch. `no_scratch`: there is no scratch memory, so that kernels without
// any are taken where others would be faster.
int try_fused(const CimxArray* in, const CimxArray* out, PassDesc* ds, int npasses,
              int lib_flags, cudaStream_t stream, bool add = false, bool no_scratch = false);

// the magnitude of a 2-D image's two 3-tap gradient chains (cimx_edges.cu)
int try_grad2d(const CimxArray* in, const CimxArray* out, const CimxPass* passes, int naxes,
               int passes_per_axis, cudaStream_t st);

// the last two axes of a float64 array in one launch (cimx_strip_f64.cu)
int try_strip_f64(const PassDesc& dy, const PassDesc& dx, const void* in, void* out,
                  cudaStream_t st, bool no_scratch);

// elementwise copy with conversion (used when a filter has no passes)
int launch_copy_cast(const void* in, int tin, void* out, int tout, int64_t n,
                     cudaStream_t stream);

// Whether a float32 pass along a strided axis takes the ring kernel
// (cimx_ring.cuh) rather than k_columns: axis 0 of 8192^2 / of 256^3, us, ring
// against k_columns: 21 taps 104 / 39 against 115 / 37, 25 taps 108 / 38 against
// 124 / 42, 41 taps 126 / 39 against 160 / 50, 65 taps 181 / 56 against 213 / 73.
// A step is 64 rows: shorter axes leave its warps idle.
inline bool ring_takes(int64_t L, int K) { return K > kSlabMaxK || (K >= 22 && L >= 48); }
// Whether a pass beyond kSlabMaxK taps takes it at all, or the generic kernel. Not
// where half of its 64 columns are idle and a tile of the generic kernel is exactly
// as wide (524 x 1000 x 32, 97 / 129 taps: 146 / 181 us against 123 / 148; 508 x
// 1000 x 33 206 / 250 against 217 / 265), nor along two samples on unaligned rows,
// whose folding every 4-byte copy repeats (167772 x 2 x 50, 66 / 97 / 129 taps:
// 3.8 / 5.6 / 8.5 ms against 4.2 / 5.3 / 6.6).
inline bool ring_long(int64_t L, int64_t inner, int K) {
  return !(inner == 32 && L >= 64) && !(L == 2 && inner % 4 != 0 && K > 81);
}
int launch_ring_f32(const PassDesc& d, const float* w, int K, int anchor, bool skip,
                    const void* in, void* out, cudaStream_t st);

// single-launch 3-D filter, by input dtype; equal K in {3, 5} on every axis
int launch_vol_f32(const VolArgs& v, int tout, cudaStream_t st);
int launch_vol_u16(const VolArgs& v, int tout, cudaStream_t st);
int launch_vol_u8(const VolArgs& v, int tout, cudaStream_t st);

// the last two axes (or the last alone) in one launch, and one pass along a
// strided axis, by input dtype; up to kSlabMaxK taps
int launch_strip_f32(const SlabArgs& a, int tout, cudaStream_t st);
int launch_columns_f32(const PassDesc& d, const float* w, int K, int anchor, bool skip,
                       const void* in, int tout, void* out, cudaStream_t st);
int launch_strip_u16(const SlabArgs& a, int tout, cudaStream_t st);
int launch_columns_u16(const PassDesc& d, const float* w, int K, int anchor, bool skip,
                       const void* in, int tout, void* out, cudaStream_t st);
int launch_strip_u8(const SlabArgs& a, int tout, cudaStream_t st);
int launch_columns_u8(const PassDesc& d, const float* w, int K, int anchor, bool skip,
                      const void* in, int tout, void* out, cudaStream_t st);

}  // namespace cimx
