// cimx_strip.cuh — the passes along the last two axes (y, x) of a (B, Y, X)
// view in one launch, as a strip walk.
//
// A CTA owns a strip of 2 NT staged columns (output columns plus the x halo)
// and a chunk of rows. Every thread holds one column pair and walks down the
// rows, kG output rows at a time:
//   * the input rows that the group's y chains read are a window in the
//     thread's registers (f32x2 pairs): each input row is loaded once per
//     chunk, straight from global memory, and no shared memory, barrier or
//     halo row is spent on the y pass. A tap is one operand of kG FMAs;
//   * the kG results, rounded through the output dtype, go to shared memory
//     as row pairs; after one barrier (the buffer is doubled) every thread
//     runs the x chains of 8 consecutive columns of one row pair from a
//     register window;
//   * the next group's rows are loaded before the x pass and used after it.
// Boundary modes: rows are mapped when they are loaded, columns once per
// thread; constant mode substitutes the fill values where the separate passes
// would read them.
//
// Bound: the FP32 pipe (Ky + Kx FMAs per output; fma.rn.f32x2 issues one
// instruction per two FMAs, which leaves half the issue slots for the rest),
// HBM for short taps. What is left is instruction overhead (about as many
// other instructions as FMA pairs at 17 taps: the window's shift, the row-pair
// packing, addresses) at 14 warps per SM.
//
// Measured on a B200 against the TMA tile kernel this replaces (32 x 128
// tiles, y and x passes out of shared memory), us: 128 x 1024^2 float32, 3 /
// 5 / 9 / 17 taps on both axes 187 / 187 / 238 / 286 against 287 / 384 / 323 /
// 413 (the first two: row-streaming kernel); 16 x 2048^2, 33 taps 241 against
// 335; one 2048^2 image, 33 taps 23.7 against 33.0; 256 x 512^2 uint16, 17
// taps 176 (to float32) and 189 (to uint16) against 278 and 314, and 255 x 511
// x 509, whose rows the tile kernel could not load, 214 against 813. An x pass
// alone, 256^3 float32, 17 / 57 taps: 33 / 53 against 65 / 156; 8192^2, 129 taps
// 293 us (82 % of the FMA rate) against 699 on k_rows (taps in shared memory).
//
// Also measured, against the kernel as it then was at 128 x 1024^2, 17 taps: one
// column per thread with scalar FMAs, which doubles the warps, 1.24 times as long
// (twice the shared reads per FMA); taps in shared memory 1.16 times; a transposed
// FIR (chains in registers instead of inputs) spilled at every tap count.
#pragma once

#include <algorithm>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "cimx_common.cuh"
#include "cimx_fast.cuh"
#include "cimx_fused.h"

namespace cimx {
namespace strip {

using fast::f2;
using fast::fma2;
using fast::hi2;
using fast::lo2;
using fast::pack2;

constexpr int kG = 8;   // rows per group
constexpr int kP = 8;   // x outputs per thread
constexpr int kRP = kG / 2;

// two neighbouring elements of T, as loaded
template <class T> struct Raw;
template <> struct Raw<float> { using type = f2; };
template <> struct Raw<uint16_t> { using type = uint32_t; };
template <> struct Raw<uint8_t> { using type = uint32_t; };

// VEC: p is aligned to a pair; else the elements p[0] and p[d1]
template <class T, bool VEC>
__device__ __forceinline__ typename Raw<T>::type load_pair(const T* p, int d1) {
  if constexpr (sizeof(T) == 4) {
    if constexpr (VEC) return __ldg(reinterpret_cast<const f2*>(p));
    else return pack2(__ldg(p), __ldg(p + d1));
  } else if constexpr (sizeof(T) == 2) {
    if constexpr (VEC) return __ldg(reinterpret_cast<const uint32_t*>(p));
    else return static_cast<uint32_t>(__ldg(p)) | (static_cast<uint32_t>(__ldg(p + d1)) << 16);
  } else {
    if constexpr (VEC) {
      const uint32_t v = __ldg(reinterpret_cast<const unsigned short*>(p));
      return (v & 0xFFu) | ((v & 0xFF00u) << 8);
    } else {
      return static_cast<uint32_t>(__ldg(p)) | (static_cast<uint32_t>(__ldg(p + d1)) << 16);
    }
  }
}

template <class T>
__device__ __forceinline__ f2 widen(typename Raw<T>::type r) {
  if constexpr (sizeof(T) == 4) return r;
  else
    return pack2(fast::exact_float(static_cast<uint16_t>(r & 0xFFFFu)),
                 fast::exact_float(static_cast<uint16_t>(r >> 16)));
}

// map_coord by repeated folding: the same index without a division, whose
// inlined code costs these kernels registers. An overhang takes one turn per
// axis length: of a row, fewer than the taps; of a column, up to the staged
// columns of the CTA (rows of 2, 64 turns: slabs of 64 x 2, 9 taps, 1.9 ms for
// 2^24 float32, on the generic kernels 14).
__device__ __forceinline__ int fold(int i, int n, int mode) {
  if (static_cast<unsigned>(i) < static_cast<unsigned>(n)) return i;
  if (mode == CIMX_MODE_CONSTANT) return -1;
  if (mode == CIMX_MODE_NEAREST) return i < 0 ? 0 : n - 1;
  if (n == 1) return 0;
  const int low = mode == CIMX_MODE_REFLECT ? -1 : 0;
  do {
    if (mode == CIMX_MODE_GRID_WRAP) i += i < 0 ? n : -n;
    else i = i < 0 ? low - i : 2 * (n - 1) - low - i;
  } while (static_cast<unsigned>(i) >= static_cast<unsigned>(n));
  return i;
}

// kN consecutive rows r .. of a line of n rows, `stride` elements apart,
// mapped where they lie outside. Returns a bit per row that constant mode
// replaces by the fill value.
template <class T, int kN>
__device__ __forceinline__ uint32_t load_rows(typename Raw<T>::type (&v)[kN], const T* p, int d1,
                                              bool vec, int r, int n, long long stride, int mode) {
  uint32_t fill = 0;
  if (r >= 0 && r + kN <= n) {
    const T* q = p + r * stride;
    if (vec) {
#pragma unroll
      for (int g = 0; g < kN; ++g) v[g] = load_pair<T, true>(q + g * stride, d1);
    } else {
#pragma unroll
      for (int g = 0; g < kN; ++g) v[g] = load_pair<T, false>(q + g * stride, d1);
    }
  } else {
#pragma unroll
    for (int g = 0; g < kN; ++g) {
      int m = fold(r + g, n, mode);
      if (m < 0) {
        m = 0;
        fill |= 1u << g;
      }
      v[g] = load_pair<T, false>(p + m * stride, d1);
    }
  }
  return fill;
}

constexpr int act_words(int KT) { return (KT + 31) / 32; }

// Tests of the taps of one chain: KT slots, K of them in use. GEN false: K lies
// in (KT - NP, KT] and only the centre tap may be left out (slot `centre`, the
// zero of an odd Gaussian derivative). GEN true: a bit per slot. Taps sit in
// the first K slots (LAST false) or in the last K.
template <int KT, int NP, bool GEN, bool LAST>
__device__ __forceinline__ bool tap_on(int k, int K, int centre,
                                       const uint32_t (&act)[act_words(KT)]) {
  if constexpr (GEN) {
    return (act[k >> 5] >> (k & 31)) & 1u;
  } else {
    const int j = LAST ? KT - 1 - k : k;
    bool on = true;
    if (j > KT - NP) on = j < K;
    if (2 * j + 1 > KT - NP && 2 * j + 1 <= KT) on = on && k != centre;
    return on;
  }
}

// W: float, or f2 for (w, w)
template <int KT, class W>
struct SlotTaps {
  int K, centre;        // centre: slot of a centre tap that is left out, or -1
  uint32_t act[act_words(KT)];
  W w[KT];
};

// cast<D>() of a chain result. `trunc`: every result of the launch is known
// (trunc_bounded) to lie in [0, max(D) + 1), where the cast is truncation
// toward zero: adding 2^23 rounded toward zero leaves the integer in the low
// mantissa bits, without the conversion unit.
template <class D>
__device__ __forceinline__ D narrow(float v, int trunc) {
  if constexpr (sizeof(D) < 4)
    if (trunc) return static_cast<D>(__float_as_uint(__fadd_rz(v, 8388608.0f)));
  return fast::narrow_cast<D>(v);
}
// the same as the float that the next pass reads
template <class D>
__device__ __forceinline__ float narrow_to_float(float v, int trunc) {
  if constexpr (sizeof(D) < 4)
    if (trunc) return __fsub_rn(__fadd_rz(v, 8388608.0f), 8388608.0f);
  return fast::narrow_float<D>(v);
}

// byte offset of staged column c (even) within a row pair of the buffer: 8
// bytes per column and 16 spare bytes every 8 columns, so that the 16-byte
// window reads of 8 lanes at a stride of 8 columns hit distinct banks
__host__ __device__ constexpr int mid_off(int c) { return c * 8 + (c >> 3) * 16; }
// Row pairs are 2 nt columns long and have room for the window of the last 8
// columns, whose slots beyond the taps in use are read and not used.
template <int KX> __host__ __device__ constexpr int mid_row_bytes(int nt) {
  return mid_off(2 * nt + KX + 15);
}
template <int KX> constexpr int smem_bytes(int nt) { return 2 * kRP * mid_row_bytes<KX>(nt); }

// kP consecutive outputs: vec 2 = one store of all of them (32 bytes for
// float32, a whole sector), 1 = two halves, 0 = one by one up to `left`.
template <class D>
__device__ __forceinline__ void store_row(D* p, const float (&v)[kP], int left, int vec, int trunc) {
  if (vec == 2) {
    if (left <= 0) return;
    if constexpr (sizeof(D) == 4) {
      asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]),
                   "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                   : "memory");
    } else {
      uint32_t w[2 * sizeof(D)];
      constexpr int kPer = 4 / sizeof(D);
#pragma unroll
      for (int i = 0; i < static_cast<int>(2 * sizeof(D)); ++i) {
        w[i] = 0;
#pragma unroll
        for (int e = 0; e < kPer; ++e)
          w[i] |= static_cast<uint32_t>(narrow<D>(v[i * kPer + e], trunc)) << (8 * sizeof(D) * e);
      }
      if constexpr (sizeof(D) == 2) *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
      else *reinterpret_cast<uint2*>(p) = make_uint2(w[0], w[1]);
    }
  } else if (vec == 1) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (4 * h < left) {
        typename fast::Vec4<D>::type q;
        q.x = narrow<D>(v[4 * h], trunc);
        q.y = narrow<D>(v[4 * h + 1], trunc);
        q.z = narrow<D>(v[4 * h + 2], trunc);
        q.w = narrow<D>(v[4 * h + 3], trunc);
        reinterpret_cast<typename fast::Vec4<D>::type*>(p)[h] = q;
      }
  } else {
#pragma unroll
    for (int e = 0; e < kP; ++e)
      if (e < left) p[e] = narrow<D>(v[e], trunc);
  }
}

// v = old + v, old the outputs that store_row() is about to replace
__device__ __forceinline__ void add_row(float (&v)[kP], const float* p, int left, int vec) {
  if (vec > 0) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (4 * h < left) {
        const float4 q = reinterpret_cast<const float4*>(p)[h];
        v[4 * h] = __fadd_rn(q.x, v[4 * h]);
        v[4 * h + 1] = __fadd_rn(q.y, v[4 * h + 1]);
        v[4 * h + 2] = __fadd_rn(q.z, v[4 * h + 2]);
        v[4 * h + 3] = __fadd_rn(q.w, v[4 * h + 3]);
      }
  } else {
#pragma unroll
    for (int e = 0; e < kP; ++e)
      if (e < left) v[e] = __fadd_rn(p[e], v[e]);
  }
}

// ---------------------------------------------------------------- strip

// KY = 1: no y pass (rows are staged as they are, the x pass alone).
// CTAs per SM asked of the compiler: the row window takes 2 (KY + 7) registers
// per thread, and a spill waits for the loads in flight (float32, 9 taps at
// three CTAs: 96 bytes spilled, 128 x 1024^2 in 474 us against 238 at two).
constexpr int kStripThreads = 256;
constexpr int kLongThreads = 224;  // beyond kSlabMaxK taps: shared memory
constexpr int kShortThreads = 128;
constexpr int kShortTaps = 5;
template <class T> constexpr int strip_ctas(int KY) { return KY <= (sizeof(T) == 4 ? 5 : 9) ? 3 : 2; }

template <int KY, int KX>
struct StripArgs {
  const void* in;
  void* out;
  long long B;
  int Y, X;
  int tiles_x, xw;     // tiles per row, output columns per tile (a multiple of 16)
  int chunk;           // output rows per CTA (a multiple of kG)
  int ay, ax, my, mx;
  int vec_in;          // aligned pair loads
  int vec_out;         // store_row()
  double cval_y, cval_x;
  int cin_y, cin_x, dt_y, dt_x;
  int trunc;           // truncating narrowing casts (narrow())
  int add;             // float32: out += the result instead of out = it
  SlotTaps<KY, f2> y;  // in the last slots
  SlotTaps<KX, f2> x;  // in the first slots
};

template <int KY, int KX>
struct ShortArgs : StripArgs<KY, KX> {
  int group;                   // rows per group, whole slabs
  short src[kG * kShortTaps];  // row of the group that [row][y tap slot] reads, -1: fill
};
template <int KY, int KX, bool SHORT>
using StripKernelArgs = std::conditional_t<SHORT, ShortArgs<KY, KX>, StripArgs<KY, KX>>;

//
// SHORT: slabs of up to kG rows and up to kShortTaps taps. A group of kG rows
// that ends with the slab would be mostly waste, so the rows of all slabs form
// one (1, B Y, X) slab and a group takes whole slabs of it: each row is loaded
// once, and as the row that a tap reads depends on the slab's rows and the mode
// (a.src), a thread's column passes through shared memory of its own, which
// other threads do not touch. 2^24 elements, 3 taps, slabs of 1 / 2 / 4 / 8 rows
// of 1024, float32: 43 / 43 / 43 / 43 us against 294 / 154 / 84 / 49 with a group
// per slab, uint8 43 / 43 / 43 / 43 against 332 / 173 / 92 / 53; rows of 64: 68 /
// 68 / 67 / 66 against 437 / 249 / 147 / 82; 10 rows and more 58 / 57.
template <class T, class D, int KY, int KX, int NP, bool GEN, bool SHORT>
__global__ void __launch_bounds__(SHORT ? kShortThreads : kStripThreads,
                                  SHORT ? 6 : strip_ctas<T>(KY))
    k_strip(const __grid_constant__ StripKernelArgs<KY, KX, SHORT> a) {
  extern __shared__ __align__(16) unsigned char sm_strip[];
  const int t = threadIdx.x, NT = blockDim.x;
  const int tile = blockIdx.x % a.tiles_x, ch = blockIdx.x / a.tiles_x;
  const int x0 = tile * a.xw;
  const int r0 = ch * a.chunk;
  const int n = min(a.chunk, a.Y - r0);  // output rows
  const float cy = fill_value<float>(a.cval_y, a.cin_y, a.dt_y);
  const float cx = fill_value<float>(a.cval_x, a.cin_x, a.dt_x);

  // this thread's staged columns and where they read
  const int gx = x0 - a.ax + 2 * t;
  const int m0 = fold(gx, a.X, a.mx), m1 = fold(gx + 1, a.X, a.mx);
  const bool f0 = m0 < 0, f1 = m1 < 0;  // x fill value
  const bool anyfill = __any_sync(0xffffffffu, f0 || f1);
  const int c0 = f0 ? 0 : m0;
  const int d1 = (f1 ? 0 : m1) - c0;
  const bool vec = __all_sync(0xffffffffu, a.vec_in && d1 == 1 && (c0 & 1) == 0);

  // this thread's x work: row pair rp, columns x0 + 8 cg ..
  const int xg = a.xw / kP;  // even
  const int rp = t / xg, cg = t - rp * xg;
  const bool xwork = rp < kRP;
  const bool xwarp = (t & ~31) < kRP * xg;  // any lane of the warp has x work
  const int rs = mid_row_bytes<KX>(NT);
  const unsigned char* win0 = sm_strip + (xwork ? rp : 0) * rs + cg * mid_off(kP);
  unsigned char* put0 = sm_strip + mid_off(2 * t);
  const int xo = x0 + cg * kP;
  int group = kG;
  if constexpr (SHORT) group = a.group;
  f2* const own = reinterpret_cast<f2*>(sm_strip + 2 * kRP * rs) + t;  // SHORT: [row * NT]

  for (long long b = blockIdx.y; b < a.B; b += gridDim.y) {
    const T* in = static_cast<const T*>(a.in) + b * a.Y * a.X + c0;
    D* out = static_cast<D*>(a.out) + b * a.Y * a.X + static_cast<long long>(r0 + 2 * rp) * a.X;

    // window slot i of the group at output row g0 is input row
    // r0 + g0 - ay - (KY - ky) + i; slots below KY - ky are not read
    f2 win[KY + kG - 1];
    typename Raw<T>::type next[kG];
    int r = SHORT ? r0 - (KY - 1) : r0 - a.ay - (KY - a.y.K);
#pragma unroll
    for (int i = 0; !SHORT && i < KY - 1; i += kG) {
      const uint32_t fill = load_rows<T>(next, in, d1, vec, r + i, a.Y, a.X, a.my);
#pragma unroll
      for (int g = 0; g < kG && i + g < KY - 1; ++g)
        win[i + g] = (fill >> g) & 1u ? pack2(cy, cy) : widen<T>(next[g]);
    }
    r += KY - 1;  // row of next[0]
    uint32_t fill = load_rows<T>(next, in, d1, vec, r, a.Y, a.X, SHORT ? CIMX_MODE_NEAREST : a.my);

    int par = 0;
    for (int g0 = 0; g0 < n; g0 += group, par ^= 1) {
#pragma unroll
      for (int g = 0; g < kG; ++g) win[KY - 1 + g] = widen<T>(next[g]);
      if (fill) {
#pragma unroll
        for (int g = 0; g < kG; ++g)
          if ((fill >> g) & 1u) win[KY - 1 + g] = pack2(cy, cy);
      }
      r += group;
      if constexpr (SHORT) {
#pragma unroll
        for (int g = 0; g < kG; ++g) own[g * NT] = win[KY - 1 + g];
      }
      {
        f2 acc[kG];
        if constexpr (SHORT) {
#pragma unroll
          for (int g = 0; g < kG; ++g) acc[g] = 0ull;
#pragma unroll
          for (int k = 0; k < KY; ++k)
            if (tap_on<KY, NP, GEN, true>(k, a.y.K, a.y.centre, a.y.act)) {
#pragma unroll
              for (int g = 0; g < kG; ++g) {
                const int i = a.src[g * KY + k];
                acc[g] = fma2(i < 0 ? pack2(cy, cy) : own[i * NT], a.y.w[k], acc[g]);
              }
            }
        } else if constexpr (KY == 1) {
#pragma unroll
          for (int g = 0; g < kG; ++g) acc[g] = win[g];
        } else {
#pragma unroll
          for (int g = 0; g < kG; ++g) acc[g] = 0ull;
#pragma unroll
          for (int k = 0; k < KY; ++k)
            if (tap_on<KY, NP, GEN, true>(k, a.y.K, a.y.centre, a.y.act)) {
#pragma unroll
              for (int g = 0; g < kG; ++g) acc[g] = fma2(win[g + k], a.y.w[k], acc[g]);
            }
        }
        if (KY > 1 && sizeof(D) < 4) {
#pragma unroll
          for (int g = 0; g < kG; ++g)
            acc[g] = pack2(narrow_to_float<D>(lo2(acc[g]), a.trunc),
                           narrow_to_float<D>(hi2(acc[g]), a.trunc));
        }
        if (anyfill) {
#pragma unroll
          for (int g = 0; g < kG; ++g)
            acc[g] = pack2(f0 ? cx : lo2(acc[g]), f1 ? cx : hi2(acc[g]));
        }
        unsigned char* put = put0 + par * kRP * rs;
#pragma unroll
        for (int q = 0; q < kRP; ++q)
          *reinterpret_cast<float4*>(put + q * rs) =
              make_float4(lo2(acc[2 * q]), lo2(acc[2 * q + 1]), hi2(acc[2 * q]), hi2(acc[2 * q + 1]));
      }
#pragma unroll
      for (int i = 0; !SHORT && i < KY - 1; ++i) win[i] = win[i + kG];
      if (g0 + group < n)
        fill = load_rows<T>(next, in, d1, vec, r, a.Y, a.X, SHORT ? CIMX_MODE_NEAREST : a.my);
      __syncthreads();
      if (xwarp) {
        const unsigned char* src = win0 + par * kRP * rs;
        f2 acc[kP];
#pragma unroll
        for (int p = 0; p < kP; ++p) acc[p] = 0ull;
        f2 w[KX + kP + 1];
#pragma unroll
        for (int e = 0; e < kP; e += 2) {
          const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(src + mid_off(e));
          w[e] = v.x;
          w[e + 1] = v.y;
        }
#pragma unroll
        for (int k = 0; k < KX; ++k) {
          if ((k & 1) == 0) {  // the elements that taps k and k + 1 add
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(src + mid_off(k + kP));
            w[k + kP] = v.x;
            w[k + kP + 1] = v.y;
          }
          if (tap_on<KX, NP, GEN, false>(k, a.x.K, a.x.centre, a.x.act)) {
#pragma unroll
            for (int p = 0; p < kP; ++p) acc[p] = fma2(w[k + p], a.x.w[k], acc[p]);
          }
        }
        D* orow = out + static_cast<long long>(g0) * a.X + xo;
#pragma unroll
        for (int h = 0; h < 2; ++h, orow += a.X) {
          if (!(xwork && g0 + 2 * rp + h < n && (!SHORT || 2 * rp + h < group))) continue;
          float v[kP];
#pragma unroll
          for (int p = 0; p < kP; ++p) v[p] = h ? hi2(acc[p]) : lo2(acc[p]);
          if constexpr (sizeof(D) == 4)
            if (a.add) add_row(v, orow, a.X - xo, a.vec_out);
          store_row<D>(orow, v, a.X - xo, a.vec_out, a.trunc);
        }
      }
    }
    __syncthreads();  // the buffers are reused by the next slab
  }
}

// ---------------------------------------------------------------- columns
//
// One pass along a strided axis of the view (outer, L, inner): a thread holds
// one column and walks down a chunk of the axis with its window in registers,
// kG outputs at a time. No shared memory and no barrier; the next group's rows
// are in flight while a group is computed. One column and scalar FMAs rather
// than a pair: half the registers, so twice the warps (256^3 float32, axis 0,
// 25 / 33 taps: 36 / 42 us against 44 / 44).
//
// Bound: HBM up to about 17 taps (256^3 float32, axis 0, 17 taps: 29 us = 4.6
// TB/s), instruction issue beyond (57 taps: 68 us, 57 % of the FMA pipe).
// Before: 3 / 9 / 17 taps on a streaming kernel with a cp.async ring 38 / 42 /
// 70 us; 25 / 33 / 57 taps on the column-pair kernel 70 / 76 / 95 us; 512 x
// 1024^2 uint16, 9 taps, axis 0, to float32 / uint16 754 / 792 against 673 /
// 572 us.

constexpr int kColThreads = 128;
constexpr int col_ctas(int KT) { return KT <= 17 ? 8 : KT <= 33 ? 6 : KT <= 49 ? 5 : 4; }

template <int KT, int V>
struct ColArgs {
  const void* in;
  void* out;
  long long inner, columns;  // columns: outer * inner / V
  int L, chunk, anchor, mode;
  double cval;
  int cin, dt;
  int trunc;
  SlotTaps<KT, std::conditional_t<V == 2, f2, float>> y;  // in the last slots
};

// V: adjacent columns per thread, 2 for up to 5 taps of 8- and 16-bit values to
// float32 on aligned pairs, where loads of a byte or two per lane hold the SM's
// load path (256 x 1024^2 uint8 / uint16, 3 taps along axis 0: 250 / 273 us, with
// one column 316 / 333).
template <class T, class D, int KT, int NP, bool GEN, int G, int V>
__global__ void __launch_bounds__(kColThreads, col_ctas(KT))
    k_columns(const __grid_constant__ ColArgs<KT, V> a) {
  static_assert(V == 1 || sizeof(D) == 4, "pairs are stored as floats");
  using Row = std::conditional_t<V == 2, typename Raw<T>::type, T>;
  using W = std::conditional_t<V == 2, f2, float>;
  const long long column = static_cast<long long>(blockIdx.x) * kColThreads + threadIdx.x;
  if (column >= a.columns) return;  // no barrier in this kernel
  const long long o = column / (a.inner / V), i = (column - o * (a.inner / V)) * V;
  const int l0 = blockIdx.y * a.chunk;
  const int n = min(a.chunk, a.L - l0);
  const float cv = fill_value<float>(a.cval, a.cin, a.dt);
  const bool fills = a.mode == CIMX_MODE_CONSTANT;
  const T* in = static_cast<const T*>(a.in) + o * a.L * a.inner + i;
  D* out = static_cast<D*>(a.out) + (o * a.L + l0) * a.inner + i;
  // kN rows r .. into v, mapped where they lie outside the axis
  auto row = [](const T* p) {
    if constexpr (V == 2) return load_pair<T, true>(p, 1);
    else return __ldg(p);
  };
  auto load = [&](auto& v, int r) {
    constexpr int kN = sizeof(v) / sizeof(Row);
    if (r >= 0 && r + kN <= a.L) {
      const T* q = in + r * a.inner;
#pragma unroll
      for (int g = 0; g < kN; ++g) v[g] = row(q + g * a.inner);
    } else {
#pragma unroll
      for (int g = 0; g < kN; ++g) v[g] = row(in + max(fold(r + g, a.L, a.mode), 0) * a.inner);
    }
  };
  // the value of a loaded row: the fill value outside in constant mode
  auto value = [&](Row v, int r) {
    const bool outside = fills && static_cast<unsigned>(r) >= static_cast<unsigned>(a.L);
    if constexpr (V == 2) {
      return outside ? pack2(cv, cv) : widen<T>(v);
    } else {
      const float x = fast::exact_float(v);
      return outside ? cv : x;
    }
  };
  auto store = [&](D* p, W v) {
    if constexpr (V == 2) *reinterpret_cast<f2*>(p) = v;
    else *p = narrow<D>(v, a.trunc);
  };
  W win[KT + G - 1];
  Row next[G];
  int r = l0 - a.anchor - (KT - a.y.K);
  {
    Row first[KT - 1];
    load(first, r);
#pragma unroll
    for (int j = 0; j < KT - 1; ++j) win[j] = value(first[j], r + j);
  }
  r += KT - 1;
  load(next, r);
  for (int g0 = 0; g0 < n; g0 += G) {
#pragma unroll
    for (int g = 0; g < G; ++g) win[KT - 1 + g] = value(next[g], r + g);
    r += G;
    if (g0 + G < n) load(next, r);
    W acc[G];
#pragma unroll
    for (int g = 0; g < G; ++g) acc[g] = 0;
#pragma unroll
    for (int k = 0; k < KT; ++k)
      if (tap_on<KT, NP, GEN, true>(k, a.y.K, a.y.centre, a.y.act)) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
          if constexpr (V == 2) acc[g] = fma2(win[g + k], a.y.w[k], acc[g]);
          else acc[g] = fmaf(win[g + k], a.y.w[k], acc[g]);
        }
      }
#pragma unroll
    for (int j = 0; j < KT - 1; ++j) win[j] = win[j + G];
    if (g0 + G <= n) {
#pragma unroll
      for (int g = 0; g < G; ++g) store(out + g * a.inner, acc[g]);
    } else {
#pragma unroll
      for (int g = 0; g < G; ++g)
        if (g0 + g < n) store(out + g * a.inner, acc[g]);
    }
    out += G * a.inner;
  }
}

inline f2 two_lanes(float w) {
  uint32_t b;
  std::memcpy(&b, &w, 4);
  return (static_cast<f2>(b) << 32) | b;
}

inline bool aligned(const void* p, size_t m) { return reinterpret_cast<uintptr_t>(p) % m == 0; }

// The taps of one pass in the first or the last of KT slots.
inline void set_tap(f2& t, float w) { t = two_lanes(w); }
inline void set_tap(float& t, float w) { t = w; }
template <int KT, class W>
void put_taps(SlotTaps<KT, W>& t, const float* w, int K, bool skip, bool last) {
  const int lead = last ? KT - K : 0;
  t.K = K;
  t.centre = skip ? lead + K / 2 : -1;
  for (int k = 0; k < K; ++k) {
    const int i = lead + k;
    set_tap(t.w[i], w[k]);
    if (!(skip && w[k] == 0.f)) t.act[i >> 5] |= 1u << (i & 31);
  }
}

// Rows per CTA, a multiple of G: whole waves of CTAs against the rows that
// each further chunk loads again. `cols` CTAs lie side by side, `slots` are
// resident at once, a row costs `per_row` and the start of a chunk `lead`.
inline int choose_chunk(long long rows, double cols, double slots, int G, double per_row,
                        double lead) {
  double best = 0;
  long long chunk = G;
  auto consider = [&](long long c) {
    const double w = cols * ((rows + c - 1) / c) / slots;
    const double waves = w <= 4 ? std::max(1.0, std::ceil(w)) : w + 0.5;
    const double cost = waves * (c * per_row + lead);
    if (best == 0 || cost < best * 0.999) {
      best = cost;
      chunk = c;
    }
  };
  for (int nch = 1; nch <= 64; ++nch) {
    const long long c = ((rows + nch - 1) / nch + G - 1) / G * G;
    consider(c);
    if (c <= G) return static_cast<int>(chunk);
  }
  for (long long c = rows / 64 / G * G; c >= G; c -= std::max<long long>(1, (c / 8 + G - 1) / G) * G)
    consider(c);
  return static_cast<int>(chunk);
}

// Whether one pass of integer results stays in [0, max(D) + 1): non-negative
// taps and fill values, and the largest input times the sum of the taps below
// it. `bound`: the largest input, then the largest result (truncated by the
// store). A float32 FMA chain of K non-negative terms exceeds the exact sum by
// at most K 2^-24 of it, below 4e-6 for 65 taps.
template <class T> constexpr double type_bound() { return sizeof(T) == 2 ? 65535.0 : 255.0; }
template <class T, class D>
int trunc_bounded(const float* w, int K, int mode, double cval, double& bound) {
  if constexpr (sizeof(T) == 4 || sizeof(D) == 4) return 0;
  const double dmax = type_bound<D>();
  if (mode == CIMX_MODE_CONSTANT && !(cval >= 0.0 && cval <= bound)) return 0;
  double sum = 0;
  for (int k = 0; k < K; ++k) {
    if (!(w[k] >= 0.f)) return 0;
    sum += w[k];
  }
  bound *= sum * (1.0 + 4e-6);
  return bound < dmax + 1.0;
}

static_assert(smem_bytes<kLongMaxK>(kLongThreads) <= 48 * 1024 &&
                  smem_bytes<kSlabMaxK>(kStripThreads) <= 48 * 1024,
              "no opt-in shared memory");

// choose_chunk, `most` rows at most, for a grid whose y extent, up to 65535, counts
// the chunks
inline int choose_chunk_y(long long rows, double cols, double slots, int G, double per_row,
                          double lead, int most) {
  const long long least = ((rows + 65534) / 65535 + G - 1) / G * G;
  return std::max(std::min(choose_chunk(rows, cols, slots, G, per_row, lead), most),
                  static_cast<int>(least));
}

template <class T, class D, int KY, int KX, int NP, bool GEN, bool SHORT = false>
int launch_strip_k(const SlabArgs& s, cudaStream_t st) {
  static_assert(!SHORT || KY == kShortTaps, "table size");
  StripKernelArgs<KY, KX, SHORT> a{};
  a.in = s.in;
  a.out = s.out;
  a.B = SHORT ? 1 : s.B;
  a.Y = static_cast<int>(SHORT ? s.B * s.Y : s.Y);
  a.X = static_cast<int>(s.X);
  a.ay = s.py.anchor;
  a.ax = s.px.anchor;
  a.my = s.py.mode;
  a.mx = s.px.mode;
  a.cval_y = s.py.cval;
  a.cval_x = s.px.cval;
  a.cin_y = s.py.cval_as_input;
  a.cin_x = s.px.cval_as_input;
  a.dt_y = s.py.dt;
  a.dt_x = s.px.dt;
  a.add = s.add;
  put_taps(a.y, s.py.w, s.py.K, s.py.skip, true);
  put_taps(a.x, s.px.w, s.px.K, s.px.skip, false);
  double bound = type_bound<T>();
  a.trunc = (KY == 1 || trunc_bounded<T, D>(s.py.w, s.py.K, s.py.mode, s.py.cval, bound)) &&
            trunc_bounded<T, D>(s.px.w, s.px.K, s.px.mode, s.px.cval, bound);
  a.vec_in = a.X % 2 == 0 && aligned(a.in, 2 * sizeof(T));
  a.vec_out = a.X % 8 == 0 && aligned(a.out, 8 * sizeof(D))   ? 2
              : a.X % 4 == 0 && aligned(a.out, 4 * sizeof(D)) ? 1
                                                                : 0;

  int group = kG;
  if constexpr (SHORT) {
    const int L = static_cast<int>(s.Y), lead = KY - s.py.K;
    a.group = group = kG / L * L;
    for (int g = 0; g < group; ++g)
      for (int k = 0; k < s.py.K; ++k) {
        const int m = map_coord32(g % L - s.py.anchor + k, L, s.py.mode);
        a.src[g * KY + lead + k] = static_cast<short>(m < 0 ? -1 : g / L * L + m);
      }
  }
  constexpr int kMost = SHORT ? kShortThreads : KX > kSlabMaxK ? kLongThreads : kStripThreads;
  auto smem = [](int nt) { return smem_bytes<KX>(nt) + (SHORT ? kG * nt * (int)sizeof(f2) : 0); };

  auto* kern = k_strip<T, D, KY, KX, NP, GEN, SHORT>;
  static int occ[kStripThreads / 32 + 1] = {};  // resident CTAs per SM, by warps
  static std::once_flag once;
  std::call_once(once, [&] {
    for (int nt = 64; nt <= kMost; nt += 32) {
      int v = 0;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, kern, nt, smem(nt)) != cudaSuccess || v < 1)
        v = 1;
      occ[nt / 32] = v;
    }
  });
  // the last shape's geometry, so that repeated calls skip the search
  struct Shape {
    long long B, Y, X;
    int ky, kx, group, nt, xw, tiles_x, chunk;
  };
  thread_local Shape last{};
  if (last.B != a.B || last.Y != a.Y || last.X != a.X || last.ky != a.y.K || last.kx != a.x.K ||
      last.group != group) {
    // CTA width: the staged columns of all tiles together as few as possible
    int nt = 0;
    long long tiles = 0, best = 0;
    for (int w = 64; w <= kMost; w += 32) {
      int xw = (2 * w - (a.x.K - 1)) / 16 * 16;
      // long filters: four warps of x work, one per scheduler, of the six or
      // seven that stage (8192^2, 129 taps: 414 us with five)
      if (KX > kSlabMaxK) xw = std::min(xw, 256);
      if (xw < 16) continue;
      const long long tl = (a.X + xw - 1) / xw;
      long long cost = tl * w;
      const int res = occ[w / 32] * w;  // fewer than 8 warps cannot fill the pipe
      if (res < 256) cost = cost * 256 / res;
      if (nt == 0 || cost < best) {
        nt = w;
        tiles = tl;
        best = cost;
      }
    }
    const int xw = static_cast<int>(((a.X + tiles - 1) / tiles + 15) / 16 * 16);
    const int tiles_x = static_cast<int>((a.X + xw - 1) / xw);
    const int chunk = choose_chunk(a.Y, (double)tiles_x * a.B, 148.0 * occ[nt / 32], group,
                                   a.y.K + a.x.K + 6, 4.0 * a.y.K + 150);
    last = Shape{a.B, a.Y, a.X, a.y.K, a.x.K, group, nt, xw, tiles_x, chunk};
  }
  const int nt = last.nt;
  a.xw = last.xw;
  a.tiles_x = last.tiles_x;
  a.chunk = last.chunk;
  const long long gx = (a.Y + a.chunk - 1LL) / a.chunk * a.tiles_x;
  if (gx > 0x7fffffffLL) return CIMX_FUSED_DECLINED;
  const dim3 grid((unsigned)gx, (unsigned)std::min<long long>(a.B, 65535));
  kern<<<grid, nt, smem(nt), st>>>(a);
  return cuda_fail(cudaGetLastError(), "strip launch");
}

// Rows per chunk of up to 9 taps where there are many waves of them: HBM bound, and
// the CTAs at work should read and write close together (100000 x 50 x 50, 3 taps,
// chunks of 64 / 96 / 256 / 1560 rows: float32 339 / 349 / 360 / 396 us, uint8 230 /
// 223 / 221 / 264; 256 x 1024^2 float32 360 / 356 / 364, uint16 277 / 272 / 269). Few
// waves: whole ones (4 x 1000 x 4096, 9 taps, 31 us against 36).
template <class D> constexpr int close_chunk() { return sizeof(D) == 4 ? 96 : 256; }

template <class T, class D, int KT, int NP, bool GEN, int V = 1>
int launch_columns_k(const PassDesc& d, const float* w, int K, int anchor, bool skip,
                     const void* in, void* out, cudaStream_t st) {
  constexpr int G = kG;
  ColArgs<KT, V> a{};
  a.in = in;
  a.out = out;
  a.inner = d.inner;
  a.columns = d.outer * d.inner / V;
  a.L = static_cast<int>(d.L);
  a.anchor = anchor;
  a.mode = d.mode;
  a.cval = d.cval;
  a.cin = d.cval_as_input ? 1 : 0;
  a.dt = fast::dt_code<T>();
  double bound = type_bound<T>();
  a.trunc = trunc_bounded<T, D>(w, K, d.mode, d.cval, bound);
  put_taps(a.y, w, K, skip, true);
  auto* kern = k_columns<T, D, KT, NP, GEN, G, V>;
  static int occ = 0;
  static std::once_flag once;
  std::call_once(once, [&] {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kColThreads, 0) != cudaSuccess ||
        occ < 1)
      occ = 1;
  });
  const long long gx = (a.columns + kColThreads - 1) / kColThreads;
  struct Shape {  // the last shape's chunk, so that repeated calls skip the search
    long long gx, L;
    int K, chunk;
  };
  thread_local Shape last{};
  if (last.gx != gx || last.L != d.L || last.K != K) {
    constexpr int kClose = close_chunk<D>();
    const bool close = K <= 9 && gx * ((d.L + kClose - 1) / kClose) >= 8LL * 148 * occ;
    last = Shape{gx, d.L, K,
                 choose_chunk_y(d.L, (double)gx, 148.0 * occ, G, K + 4, 3.0 * K + 80,
                                close ? kClose : 1 << 30)};
  }
  a.chunk = last.chunk;
  if (gx > 0x7fffffffLL) return CIMX_FUSED_DECLINED;
  const dim3 grid((unsigned)gx, (unsigned)((d.L + a.chunk - 1) / a.chunk));
  kern<<<grid, kColThreads, 0, st>>>(a);
  return cuda_fail(cudaGetLastError(), "column pass launch");
}

// The x pass alone (KY = 1, an identity y pass) or both passes, which
// strip_fuses() (cimx_fused.cu) sends here up to 33 taps.
template <class T, class D>
int launch_strip_td(const SlabArgs& s, cudaStream_t st) {
  const int K = std::max(s.py.K, s.px.K), k0 = std::min(s.py.K, s.px.K);
  const int kt = kt_bound(sizeof(T), K);
  const bool masked = skip_kind(s.py.w, s.py.K, s.py.skip) == 2 ||
                      skip_kind(s.px.w, s.px.K, s.px.skip) == 2;
  if (!s.has_y) {
    if constexpr (sizeof(T) == 4) {
      if (masked && K > kSlabMaxK) return launch_strip_k<T, D, 1, kLongMaxK, kLongMaxK, true>(s, st);
    }
    if (masked) return launch_strip_k<T, D, 1, 65, 65, true>(s, st);
    if constexpr (sizeof(T) == 4) {
      if (K > kSlabMaxK) {
        switch ((kt + 7 - 1) / 8 * 8 + 1) {
#define CIMX_KT(K_) case K_: return launch_strip_k<T, D, 1, K_, 8, false>(s, st);
          CIMX_KT(73) CIMX_KT(81) CIMX_KT(89) CIMX_KT(97) CIMX_KT(105) CIMX_KT(113) CIMX_KT(121)
          CIMX_KT(129)
#undef CIMX_KT
          default: return CIMX_FUSED_DECLINED;
        }
      }
    }
    switch (kt) {
      case 5: case 9: return launch_strip_k<T, D, 1, 9, 9, false>(s, st);
#define CIMX_KT(K_) case K_: return launch_strip_k<T, D, 1, K_, 8, false>(s, st);
      case 13: CIMX_KT(17) case 21: CIMX_KT(25) case 29: CIMX_KT(33) case 37: CIMX_KT(41)
      case 45: CIMX_KT(49) case 53: CIMX_KT(57) case 61: CIMX_KT(65)
#undef CIMX_KT
      default: return CIMX_FUSED_DECLINED;
    }
  }
  if (masked || kt_bound(sizeof(T), k0) != kt) {
    if (K <= 9) return launch_strip_k<T, D, 9, 9, 9, true>(s, st);
    if (K <= 17) return launch_strip_k<T, D, 17, 17, 17, true>(s, st);
    return launch_strip_k<T, D, 65, 65, 65, true>(s, st);  // only without scratch memory
  }
  constexpr int kStep = kt_step(sizeof(T));
  switch (kt) {
    case 5:
      // from 9 rows on, a group would be a part of a slab
      if (s.Y <= kG && s.B * s.Y < (1LL << 30))
        return launch_strip_k<T, D, 5, 5, 5, false, true>(s, st);
      return launch_strip_k<T, D, 5, 5, 5, false>(s, st);
    case 9: return launch_strip_k<T, D, 9, 9, 4, false>(s, st);
#define CIMX_KT(K_) case K_: return launch_strip_k<T, D, K_, K_, kStep, false>(s, st);
    CIMX_KT(17) CIMX_KT(25) CIMX_KT(33)
    default: break;
  }
  if constexpr (kStep == 4) {
    switch (kt) {
      CIMX_KT(13) CIMX_KT(21) CIMX_KT(29)
      default: break;
    }
  }
#undef CIMX_KT
  return launch_strip_k<T, D, 65, 65, 65, true>(s, st);  // only without scratch memory
}

template <class T, class D>
int launch_columns_td(const PassDesc& d, const float* w, int K, int anchor, bool skip,
                      const void* in, void* out, cudaStream_t st) {
  if (skip_kind(w, K, skip) == 2) {
    if (K <= 17) return launch_columns_k<T, D, 17, 17, true>(d, w, K, anchor, skip, in, out, st);
    if (K <= 33) return launch_columns_k<T, D, 33, 33, true>(d, w, K, anchor, skip, in, out, st);
    return launch_columns_k<T, D, 65, 65, true>(d, w, K, anchor, skip, in, out, st);
  }
  switch (kt_bound(sizeof(T), K)) {
    case 5:
      if constexpr (sizeof(T) < 4 && sizeof(D) == 4)
        if (d.inner % 2 == 0 && aligned(in, 2 * sizeof(T)) && aligned(out, 2 * sizeof(D)))
          return launch_columns_k<T, D, 5, 5, false, 2>(d, w, K, anchor, skip, in, out, st);
      return launch_columns_k<T, D, 5, 5, false>(d, w, K, anchor, skip, in, out, st);
    case 9: return launch_columns_k<T, D, 9, 4, false>(d, w, K, anchor, skip, in, out, st);
#define CIMX_KT(K_) \
  case K_: return launch_columns_k<T, D, K_, 8, false>(d, w, K, anchor, skip, in, out, st);
    case 13: CIMX_KT(17) case 21: CIMX_KT(25) case 29: CIMX_KT(33) case 37: CIMX_KT(41)
    case 45: CIMX_KT(49) case 53: CIMX_KT(57) case 61: CIMX_KT(65)
#undef CIMX_KT
    default: return CIMX_FUSED_DECLINED;
  }
}

}  // namespace strip
}  // namespace cimx
