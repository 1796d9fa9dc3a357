// cimx_edges.cu — two parts of the skimage edge filters.
//
// 1. The gradient magnitude of a 2-D image from two chains of 3-tap passes
// (sobel, scharr, prewitt: filters/edges.py:148-241), in one launch: a thread
// takes one column and kGradRows rows, the three columns' rows in registers,
// and computes the values that the separate passes would store.
//
// 2. The `mask=` argument
// (python/cucim/src/cucim/skimage/filters/edges.py:75-85,
// _mask_filter_result): the mask is eroded with the full-connectivity
// footprint (every element of the 3 x ... x 3 neighbourhood,
// generate_binary_structure(ndim, ndim)) with border_value 0, and the
// filter result is multiplied by the eroded mask in place. One thread per
// output element reads the 3^ndim neighbourhood of the mask directly (the
// erosion is never stored).
#include <algorithm>
#include <vector>

#include "cimx_common.cuh"
#include "cimx_fused.h"
#include "cimx_internal.h"

namespace cimx {
namespace {

// Bound: the launch and HBM for large images. 1023 x 1537 uint8: 1 launch
// instead of conversion, two separable filters, two square-and-add launches and
// the root: 91.8 -> 12.3 us a call.
constexpr int kGradRows = 8;

struct GradArgs {
  const void* in;
  float* out;
  int H, W, mode;
  float scale;       // img_as_float of integers: the product with 1 / max
  float edge[2][3];  // axis 0, axis 1
  float smooth[2][3];  // along the other axis
  unsigned on[2][2];   // taps that take part: [axis][edge, smooth]
};

template <class T>
__global__ void __launch_bounds__(256) k_grad2d(const GradArgs a) {
  const int x = blockIdx.x * 32 + (threadIdx.x & 31);
  const int y0 = (blockIdx.y * 8 + (threadIdx.x >> 5)) * kGradRows;
  if (x >= a.W || y0 >= a.H) return;
  const T* in = static_cast<const T*>(a.in);
  int col[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) col[k] = map_coord32(x - 1 + k, a.W, a.mode);
  auto chain = [](float u, float v, float w, const float(&t)[3], unsigned on) {
    float acc = 0.f;
    if (on & 1u) acc = fmaf(u, t[0], acc);
    if (on & 2u) acc = fmaf(v, t[1], acc);
    if (on & 4u) acc = fmaf(w, t[2], acc);
    return acc;
  };
  float s[3][3], e1[3];  // rows y - 1 .. y + 1: values, and edges along the row
  bool out_row[3];
  auto load = [&](int i, int y) {
    const int row = map_coord32(y, a.H, a.mode);
    out_row[i] = row < 0;
    const T* p = in + static_cast<long long>(max(row, 0)) * a.W;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      float v = static_cast<float>(__ldg(p + max(col[k], 0)));
      if (sizeof(T) < 4) v = __fmul_rn(v, a.scale);
      s[i][k] = row < 0 || col[k] < 0 ? 0.f : v;  // constant mode: the fill value 0
    }
    e1[i] = row < 0 ? 0.f : chain(s[i][0], s[i][1], s[i][2], a.edge[1], a.on[1][0]);
  };
  load(0, y0 - 1);
  load(1, y0);
  float* out = a.out + static_cast<long long>(y0) * a.W + x;
#pragma unroll
  for (int j = 0; j < kGradRows; ++j) {
    if (y0 + j >= a.H) break;
    const int r0 = j % 3, r1 = (j + 1) % 3, r2 = (j + 2) % 3;
    load(r2, y0 + j + 1);
    float e0[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
      e0[k] = col[k] < 0 ? 0.f : chain(s[r0][k], s[r1][k], s[r2][k], a.edge[0], a.on[0][0]);
    const float d0 = chain(e0[0], e0[1], e0[2], a.smooth[0], a.on[0][1]);
    const float d1 = chain(e1[r0], e1[r1], e1[r2], a.smooth[1], a.on[1][1]);
    out[static_cast<long long>(j) * a.W] =
        sqrtf(__fadd_rn(__fmul_rn(d0, d0), __fmul_rn(d1, d1)));
  }
}

struct MaskShape {
  int ndim;
  int64_t shape[CIMX_MAX_NDIM];
};

inline unsigned grid_for(int64_t n, int threads = 256) {
  const int64_t b = (n + threads - 1) / threads;
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>(b, 148LL * 32));
}

// binary_erosion's truth value of one mask element (nonzero; NaN is nonzero)
__device__ __forceinline__ bool mask_true(const void* m, int t, int64_t i) {
  switch (t) {
    case 'H': case 'h': return static_cast<const uint16_t*>(m)[i] != 0;
    case 'e': return (static_cast<const uint16_t*>(m)[i] & 0x7fffu) != 0;
    case 'I': case 'i': return static_cast<const uint32_t*>(m)[i] != 0;
    case 'f': return static_cast<const float*>(m)[i] != 0.0f;
    case 'd': return static_cast<const double*>(m)[i] != 0.0;
    case 'L': case 'Q': case 'l': case 'q': return static_cast<const uint64_t*>(m)[i] != 0;
    default: return static_cast<const uint8_t*>(m)[i] != 0;  // '?', 'B', 'b'
  }
}

template <class F>
__global__ void k_mask_erode_mul(F* __restrict__ res, const void* __restrict__ mask, int tm,
                                 MaskShape s, int64_t n) {
  int nb = 1;
  for (int d = 0; d < s.ndim; ++d) nb *= 3;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t c[CIMX_MAX_NDIM];
    int64_t r = i;
    for (int d = s.ndim - 1; d >= 0; --d) {
      c[d] = r % s.shape[d];
      r /= s.shape[d];
    }
    bool keep = true;
    for (int o = 0; o < nb && keep; ++o) {
      int code = o;
      int64_t j = 0;
      for (int d = 0; d < s.ndim; ++d) {
        const int64_t x = c[d] + (code % 3) - 1;
        code /= 3;
        if (x < 0 || x >= s.shape[d]) {  // border_value=0
          keep = false;
          break;
        }
        j = j * s.shape[d] + x;
      }
      if (keep) keep = mask_true(mask, tm, j);
    }
    res[i] = res[i] * (keep ? F(1) : F(0));  // result *= mask
  }
}

}  // namespace

// The magnitude of a 2-D image's two gradient chains in one launch: per axis an
// edge pass along it and a smoothing pass along the other one, 3 centred taps
// each, one boundary mode, fill value 0. `out` has been checked (shape of `in`,
// C-contiguous).
int try_grad2d(const CimxArray* in, const CimxArray* out, const CimxPass* passes, int naxes,
               int passes_per_axis, cudaStream_t st) {
  if (in->ndim != 2 || naxes != 2 || passes_per_axis != 2 || out->dtype != DT_F32)
    return CIMX_FUSED_DECLINED;
  const int t = in->dtype;
  if (t != DT_F32 && t != DT_U8 && t != DT_U16) return CIMX_FUSED_DECLINED;
  const int64_t H = in->shape[0], W = in->shape[1], es = dtype_size(t);
  // contiguous, not overlapping (the general path reports those)
  if (H < 1 || W < 1 || H >= (1 << 30) || W >= (1 << 30)) return CIMX_FUSED_DECLINED;
  if ((W > 1 && in->strides[1] != es) || (H > 1 && in->strides[0] != W * es))
    return CIMX_FUSED_DECLINED;
  const char *i0 = static_cast<const char*>(in->data), *o0 = static_cast<const char*>(out->data);
  if (!i0 || !o0 || (i0 < o0 + H * W * 4 && o0 < i0 + H * W * es)) return CIMX_FUSED_DECLINED;
  GradArgs a{};
  std::vector<double> taps;
  for (int ax = 0; ax < 2; ++ax)
    for (int p = 0; p < 2; ++p) {
      PassDesc d{};
      const CimxPass& q = passes[2 * ax + p];
      if (q.ntaps != 3 || (q.flags & CIMX_F_COMPLEX_TAPS)) return CIMX_FUSED_DECLINED;
      if (make_pass(in, q, taps, d) != CIMX_OK) return CIMX_FUSED_DECLINED;
      if (d.axis != (p == 0 ? ax : 1 - ax) || d.anchor != 1 || d.w64 || d.cval != 0.0)
        return CIMX_FUSED_DECLINED;
      if (ax + p == 0) a.mode = d.mode;
      if (d.mode != a.mode) return CIMX_FUSED_DECLINED;
      for (int k = 0; k < 3; ++k) {
        const float w = static_cast<float>(d.taps[k]);
        (p == 0 ? a.edge : a.smooth)[ax][k] = w;
        if (!(d.skip_zero && w == 0.f)) a.on[ax][p] |= 1u << k;
      }
    }
  a.in = in->data;
  a.out = static_cast<float*>(out->data);
  a.H = static_cast<int>(H);
  a.W = static_cast<int>(W);
  a.scale = t == DT_U8 ? static_cast<float>(1.0 / 255.0) : static_cast<float>(1.0 / 65535.0);
  const int64_t gy = (H + 8 * kGradRows - 1) / (8 * kGradRows);
  if (gy > 65535) return CIMX_FUSED_DECLINED;
  const dim3 grid((unsigned)((W + 31) / 32), (unsigned)gy);
  if (t == DT_F32) k_grad2d<float><<<grid, 256, 0, st>>>(a);
  else if (t == DT_U8) k_grad2d<uint8_t><<<grid, 256, 0, st>>>(a);
  else k_grad2d<uint16_t><<<grid, 256, 0, st>>>(a);
  return cuda_fail(cudaGetLastError(), "gradient magnitude launch");
}

}  // namespace cimx

using namespace cimx;

extern "C" int cimx_edge_magnitude(const CimxArray* in, const CimxArray* out,
                                   const CimxPass* passes, int naxes, int passes_per_axis,
                                   void* stream) {
  if (!in || !out || !passes || naxes < 1 || passes_per_axis < 0)
    return fail(CIMX_E_INVALID, "bad edge-magnitude arguments");
  if (in->dtype == out->dtype)
    return cimx_gradient_magnitude(in, out, passes, naxes, passes_per_axis, stream);
  if (out->dtype != DT_F32 && out->dtype != DT_F64)
    return fail(CIMX_E_DTYPE, "edge magnitude output must be float32 or float64");
  int rc;
  if ((rc = check_array(in, "input")) || (rc = check_array(out, "output")) ||
      (rc = check_same_shape(in, out)))
    return rc;
  int64_t n = 1;
  for (int d = 0; d < in->ndim; ++d) n *= in->shape[d];
  if (n == 0) return CIMX_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  rc = try_grad2d(in, out, passes, naxes, passes_per_axis, st);
  if (rc != CIMX_FUSED_DECLINED) return rc;
  // the image as floats, then the general path
  const size_t bytes = (size_t)n * dtype_size(out->dtype);
  CimxArray img = *out;
  img.data = scratch_alloc(bytes, st);
  if (!img.data) return fail(CIMX_E_NOMEM, "scratch allocation for the float image failed");
  rc = cimx_convert(in, &img, 1, stream);
  if (rc == CIMX_OK) rc = cimx_gradient_magnitude(&img, out, passes, naxes, passes_per_axis, stream);
  scratch_free(img.data, bytes, st);
  return rc;
}

extern "C" int cimx_mask_erode_multiply(const CimxArray* result, const CimxArray* mask,
                                        void* stream) {
  if (!result || !mask) return fail(CIMX_E_INVALID, "NULL argument");
  if (result->dtype != DT_F32 && result->dtype != DT_F64)
    return fail(CIMX_E_DTYPE, "the filter result must be float32 or float64");
  if (mask->dtype != '?' && dtype_size(mask->dtype) == 0)
    return fail(CIMX_E_DTYPE, "unsupported mask dtype");
  if (mask->ndim != result->ndim || result->ndim < 1 || result->ndim > CIMX_MAX_NDIM)
    return fail(CIMX_E_INVALID, "mask shape must equal the image shape");
  MaskShape s{};
  s.ndim = result->ndim;
  int64_t n = 1;
  for (int d = 0; d < s.ndim; ++d) {
    if (mask->shape[d] != result->shape[d])
      return fail(CIMX_E_INVALID, "mask shape must equal the image shape");
    s.shape[d] = result->shape[d];
    n *= s.shape[d];
  }
  // both C-contiguous
  const int msize = mask->dtype == '?' ? 1 : dtype_size(mask->dtype);
  int64_t er = dtype_size(result->dtype), em = msize;
  for (int d = s.ndim - 1; d >= 0; --d) {
    if (s.shape[d] != 1 && (result->strides[d] != er || mask->strides[d] != em))
      return fail(CIMX_E_LAYOUT, "result and mask must be C-contiguous");
    er *= s.shape[d];
    em *= s.shape[d];
  }
  if (n == 0) return CIMX_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (result->dtype == DT_F32)
    k_mask_erode_mul<float><<<grid_for(n), 256, 0, st>>>(static_cast<float*>(result->data),
                                                         mask->data, mask->dtype, s, n);
  else
    k_mask_erode_mul<double><<<grid_for(n), 256, 0, st>>>(static_cast<double*>(result->data),
                                                          mask->data, mask->dtype, s, n);
  return cuda_fail(cudaGetLastError(), "mask launch");
}
