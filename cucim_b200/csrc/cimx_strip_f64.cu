// cimx_strip_f64.cu — the passes along the last two axes of a float64 array in
// one launch: the strip walk of cimx_strip.cuh with one column per thread.
//
// A CTA owns 256 staged columns (output columns plus the x halo) and a chunk of
// rows, 8 at a time: the rows that the y chains read are a window in registers,
// each loaded once per chunk; the 8 results go to shared memory (two buffers, one
// barrier per group); then every thread runs the x chains of 8 columns of one
// row, and the warp's 8 x 32 results pass through shared memory once more so
// that its stores cover 256 consecutive bytes at any alignment.
//
// Bound: HBM up to about 17 taps, the float64 pipe (half the float32 rate)
// beyond (a row loads its halo again once per 240 columns). 2003 x 3001, 17 taps:
// 34.8 us a call against 86.1 in two launches of the generic kernels, whose taps
// and inputs all come from shared memory.
#include <cmath>

#include "cimx_strip.cuh"

namespace cimx {
namespace strip64 {

using strip::fold;
using strip::SlotTaps;
using strip::tap_on;

constexpr int kThreads = 256;
constexpr int kG = 8;   // rows per group
constexpr int kP = 8;   // x outputs per thread
constexpr int kMaxK = 49;  // instantiated up to here: 182 registers, two more per tap
constexpr int ctas(int KT) { return KT <= 25 ? 2 : 1; }

// bytes per staged row, 16 modulo 128: the rows of 8 lanes hit distinct banks
constexpr int row_bytes(int KT) { return (kThreads + KT + kP + 15) / 16 * 128 + 16; }
constexpr int kOutPitch = 4 * kP + 2;  // doubles per row of a warp's results
constexpr int smem_bytes(int KT) {
  return 2 * kG * row_bytes(KT) + kThreads / 32 * kG * kOutPitch * (int)sizeof(double);
}

template <int KT>
struct Args {
  const double* in;
  double* out;
  long long B;
  int Y, X, tiles, xw, chunk;  // xw: output columns per CTA
  int ay, ax, my, mx;
  double cy, cx;
  SlotTaps<KT, double> y;  // in the last slots
  SlotTaps<KT, double> x;  // in the first slots
};

template <int KT, int NP>
__global__ void __launch_bounds__(kThreads, ctas(KT)) k_strip64(const __grid_constant__ Args<KT> a) {
  extern __shared__ __align__(16) unsigned char sm_strip64[];
  constexpr int RB = row_bytes(KT);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int x0 = blockIdx.x % a.tiles * a.xw, r0 = blockIdx.x / a.tiles * a.chunk;
  const int n = min(a.chunk, a.Y - r0);
  const int m = fold(x0 - a.ax + t, a.X, a.mx);
  const bool fill_x = m < 0;
  const bool staged = t < a.xw + KT - 1;
  // x work: row rp of the group, columns x0 + cg ..
  const int rp = lane & 7, cg = (4 * warp + (lane >> 3)) * kP;
  const int wide = min(a.xw, a.X - x0);
  const bool xwork = 32 * warp < wide;  // any column of the warp
  double* const back =
      reinterpret_cast<double*>(sm_strip64 + 2 * kG * RB) + warp * kG * kOutPitch;

  for (long long b = blockIdx.y; b < a.B; b += gridDim.y) {
    const double* in = a.in + b * a.Y * a.X + max(m, 0);
    double* out = a.out + (b * a.Y + r0) * a.X + x0 + 32 * warp + lane;
    uint32_t fill = 0;  // rows of `next` outside, in constant mode
    double win[KT + kG - 1], next[kG];
    auto load = [&](int r) {
      fill = 0;
      if (r >= 0 && r + kG <= a.Y) {
        const double* q = in + static_cast<long long>(r) * a.X;
#pragma unroll
        for (int g = 0; g < kG; ++g) next[g] = __ldg(q + static_cast<long long>(g) * a.X);
      } else {
#pragma unroll
        for (int g = 0; g < kG; ++g) {
          const int row = fold(r + g, a.Y, a.my);
          if (row < 0) fill |= 1u << g;
          next[g] = __ldg(in + static_cast<long long>(max(row, 0)) * a.X);
        }
      }
    };
    int r = r0 - a.ay - (KT - a.y.K);
#pragma unroll
    for (int i = 0; i < KT - 1; i += kG) {
      load(r + i);
#pragma unroll
      for (int g = 0; g < kG && i + g < KT - 1; ++g)
        win[i + g] = (fill >> g) & 1u ? a.cy : next[g];
    }
    r += KT - 1;
    load(r);
    int par = 0;
    for (int g0 = 0; g0 < n; g0 += kG, par ^= 1) {
#pragma unroll
      for (int g = 0; g < kG; ++g) win[KT - 1 + g] = (fill >> g) & 1u ? a.cy : next[g];
      r += kG;
      unsigned char* const buf = sm_strip64 + par * kG * RB;
      {
        double acc[kG];
#pragma unroll
        for (int g = 0; g < kG; ++g) acc[g] = 0.0;
#pragma unroll
        for (int k = 0; k < KT; ++k)
          if (tap_on<KT, NP, false, true>(k, a.y.K, a.y.centre, a.y.act)) {
#pragma unroll
            for (int g = 0; g < kG; ++g) acc[g] = fma(win[g + k], a.y.w[k], acc[g]);
          }
        if (staged) {
#pragma unroll
          for (int g = 0; g < kG; ++g)
            *reinterpret_cast<double*>(buf + g * RB + 8 * t) = fill_x ? a.cx : acc[g];
        }
      }
#pragma unroll
      for (int i = 0; i < KT - 1; ++i) win[i] = win[i + kG];
      if (g0 + kG < n) load(r);
      __syncthreads();
      if (xwork) {
        const unsigned char* src = buf + rp * RB + cg * 8;
        double acc[kP], w[KT + kP + 1];
        auto two = [&](int e) {
          const double2 v = *reinterpret_cast<const double2*>(src + e * 8);
          w[e] = v.x;
          w[e + 1] = v.y;
        };
#pragma unroll
        for (int p = 0; p < kP; ++p) acc[p] = 0.0;
#pragma unroll
        for (int e = 0; e < kP; e += 2) two(e);
#pragma unroll
        for (int k = 0; k < KT; ++k) {
          if ((k & 1) == 0) two(k + kP);
          if (tap_on<KT, NP, false, false>(k, a.x.K, a.x.centre, a.x.act)) {
#pragma unroll
            for (int p = 0; p < kP; ++p) acc[p] = fma(w[k + p], a.x.w[k], acc[p]);
          }
        }
        double2* put = reinterpret_cast<double2*>(back + rp * kOutPitch + (lane >> 3) * kP);
#pragma unroll
        for (int p = 0; p < kP; p += 2) put[p / 2] = make_double2(acc[p], acc[p + 1]);
        __syncwarp();
        if (32 * warp + lane < wide) {
#pragma unroll
          for (int g = 0; g < kG; ++g)
            if (g0 + g < n) out[static_cast<long long>(g0 + g) * a.X] = back[g * kOutPitch + lane];
        }
        __syncwarp();
      }
    }
    __syncthreads();  // the buffers are reused by the next slab
  }
}

template <int KT, int NP>
int launch_k(Args<KT>& a, const PassDesc& dy, const PassDesc& dx, cudaStream_t st) {
  auto taps = [](SlotTaps<KT, double>& s, const PassDesc& d, int lead) {
    s.K = d.K;
    s.centre = -1;
    for (int k = 0; k < d.K; ++k) s.w[lead + k] = d.taps[k];
  };
  taps(a.y, dy, KT - dy.K);
  taps(a.x, dx, 0);
  auto* kern = k_strip64<KT, NP>;
  constexpr int smem = smem_bytes(KT);
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  static int occ = 0;
  std::call_once(once, [&] {
    attr = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kThreads, smem) != cudaSuccess ||
        occ < 1)
      occ = 1;
  });
  if (attr != cudaSuccess) return cuda_fail(attr, "float64 strip shared memory attribute");
  const int most = (kThreads - (KT - 1)) / kP * kP;
  a.tiles = (a.X + most - 1) / most;
  a.xw = ((a.X + a.tiles - 1) / a.tiles + kP - 1) / kP * kP;
  a.chunk = strip::choose_chunk(a.Y, (double)a.tiles * a.B, 148.0 * occ, kG, 2.0 * a.y.K + 8,
                                4.0 * a.y.K + 100);
  const long long gx = (long long)((a.Y + a.chunk - 1) / a.chunk) * a.tiles;
  if (gx > 0x7fffffffLL) return CIMX_FUSED_DECLINED;
  kern<<<dim3((unsigned)gx, (unsigned)std::min<long long>(a.B, 65535)), kThreads, smem, st>>>(a);
  return cuda_fail(cudaGetLastError(), "float64 strip launch");
}

template <int KT, int NP>
int launch(const PassDesc& dy, const PassDesc& dx, const void* in, void* out, cudaStream_t st) {
  auto fill = [](const PassDesc& d) { return d.cval; };  // float64: as input or as weight
  Args<KT> a{};
  a.in = static_cast<const double*>(in);
  a.out = static_cast<double*>(out);
  a.B = dy.outer;
  a.Y = static_cast<int>(dy.L);
  a.X = static_cast<int>(dx.L);
  a.ay = dy.anchor;
  a.ax = dx.anchor;
  a.my = dy.mode;
  a.mx = dx.mode;
  a.cy = fill(dy);
  a.cx = fill(dx);
  return launch_k<KT, NP>(a, dy, dx, st);
}

}  // namespace strip64

namespace strip64 {

// Whether the strip beats the two launches of the generic kernels. Up to 25 taps
// always, beyond, one CTA per SM, by the two costs in us of 2^24 elements at 33
// taps (longer filters scale both alike): the strip's staged columns and rows (a
// slab's window, its last group) against the generic tiles' rows and columns.
// Measured, strip against generic: slabs of 8 x 256 (two CTAs side by side) 745 /
// 884, 20 x 256 505 / 443, 64 x 256 288 / 241, 512 x 256 265 / 243, 64 x 280 296 /
// 313, 64 x 450 (three) 275 / 256, 512 x 450 222 / 253, 20 x 64 976 / 728, 512 x 64
// 441 / 525, 64 x 1000 213 / 241. Small arrays: the launch saved counts.
inline bool pays(int KT, double B, double Y, double X) {
  if (KT < 33 || B * Y * X < (1 << 19)) return true;
  const double most = (kThreads - (KT - 1)) / kP * kP;
  const double staged = kThreads * std::ceil(X / most) / X;
  const double strip = 40 + (95 * kG * std::ceil(Y / kG) + 2240) / Y * staged;
  const double generic = 45 + 94 * 64 * std::ceil(Y / 64) / Y + 92 * 256 * std::ceil(X / 256) / X;
  return strip < generic;
}

}  // namespace strip64

// The passes dy, dx along the last two axes of a float64 array with float64
// taps. Declined: unequal tap bounds, zero taps that are left out, few rows, and
// (but for no_scratch: the generic kernels take a scratch array) what pays()
// leaves to the generic kernels.
int try_strip_f64(const PassDesc& dy, const PassDesc& dx, const void* in, void* out,
                  cudaStream_t st, bool no_scratch) {
  using namespace strip64;
  const int K = std::max(dy.K, dx.K);
  if (!dy.w64 || !dx.w64 || K > kMaxK || dy.L < kG || dx.L < 32) return CIMX_FUSED_DECLINED;
  if (dy.L >= (1LL << 30) || dx.L >= (1LL << 30)) return CIMX_FUSED_DECLINED;
  auto bound = [](int k) { return k <= 9 ? 9 : (k + 6) / 8 * 8 + 1; };
  if (bound(dy.K) != bound(dx.K)) return CIMX_FUSED_DECLINED;
  if (!no_scratch && !pays(bound(K), dy.outer, dy.L, dx.L)) return CIMX_FUSED_DECLINED;
  for (const PassDesc* d : {&dy, &dx}) {
    if (d->anchor < 0 || d->anchor >= d->K) return CIMX_FUSED_DECLINED;
    for (int k = 0; k < d->K && d->skip_zero; ++k)
      if (d->taps[k] == 0.0) return CIMX_FUSED_DECLINED;
  }
  switch (bound(K)) {
    case 9: return launch<9, 9>(dy, dx, in, out, st);
#define CIMX_KT(K_) case K_: return launch<K_, 8>(dy, dx, in, out, st);
    CIMX_KT(17) CIMX_KT(25) CIMX_KT(33) CIMX_KT(41) CIMX_KT(49)
#undef CIMX_KT
    default: return CIMX_FUSED_DECLINED;
  }
}

}  // namespace cimx
