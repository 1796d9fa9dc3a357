// cimx_ring.cuh — one float32 pass along a strided axis with a long filter.
//
// A CTA walks down 64 columns, 64 rows at a time, a column pair per lane and 8
// rows per warp. The rows sit in a ring in shared memory: those of the current
// step and the next 64, which cp.async brings in meanwhile; one barrier per
// step. Ring slots come in multiples of 8, so that a block of 8 rows never
// wraps. The chains are unrolled with their taps in the constant bank, the
// inputs streaming through the registers in blocks of 8: 8 shared loads per 64
// two-lane FMAs and nothing else. (k_columns, cimx_strip.cuh, keeps the whole
// window in registers: no shared memory, but scalar FMAs, one move per tap and
// group, and from 50 taps on too few warps.)
//
// Bound: the FP32 pipe, K FMAs per output. 8192^2 along axis 0, 57 / 129 taps:
// 165 / 314 us (70 / 77 % of the FMA rate) against 197 us (k_columns) / 545 us
// (shared-memory tiles, taps read from shared memory); 256^3, 57 taps 52 against
// 68 us. Also measured: a run-time tap count, taps in shared memory: 394 us at
// 129 taps (16 outputs per thread 409).
#pragma once

#include "cimx_strip.cuh"

namespace cimx {
namespace ring {

using fast::f2;
using fast::fma2;
using fast::hi2;
using fast::lo2;

constexpr int kThreads = 256;
constexpr int kCols = 64;
constexpr int kRows = 64;  // per step: 8 per warp
constexpr int step_rows(int KT) { return (KT - 1 + 7) / 8 * 8 + kRows; }
constexpr int ring_rows(int KT) { return step_rows(KT) + kRows; }
constexpr int smem_bytes(int KT) { return ring_rows(KT) * kCols * (int)sizeof(float); }

template <int KT>
struct RingArgs {
  const float* in;
  float* out;
  long long inner;
  int L, chunk, tiles;  // chunk: output rows per CTA, tiles: CTAs side by side
  int anchor, mode, vec;  // vec: 16-byte loads and 8-byte stores are aligned
  double cval;
  int cin;
  strip::SlotTaps<KT, f2> y;  // in the first slots
};

template <int KT, int NP, bool GEN>
__global__ void __launch_bounds__(kThreads, 3) k_ring(const __grid_constant__ RingArgs<KT> a) {
  extern __shared__ __align__(16) float sm_ring[];
  constexpr int S = step_rows(KT), R = ring_rows(KT);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long o = blockIdx.x / a.tiles;
  const long long i0 = static_cast<long long>(blockIdx.x % a.tiles) * kCols;
  const int l0 = blockIdx.y * a.chunk;
  const int n = min(a.chunk, a.L - l0);
  const float cv = fill_value<float>(a.cval, a.cin, DT_F32);
  const float* const in = a.in + o * a.L * a.inner + i0;
  const int width = static_cast<int>(min(static_cast<long long>(kCols), a.inner - i0));

  // staged rows j0 .. j0 + rows - 1 (row l0 - anchor + j of the axis) to slots
  // s0 ..
  auto stage = [&](int j0, int rows, int s0) {
    if (a.vec) {
      const int c = (tid & 15) * 4;
      for (int j = tid >> 4; j < rows; j += kThreads / 16) {
        const int m = strip::fold(l0 - a.anchor + j0 + j, a.L, a.mode);
        float* dst = sm_ring + (s0 + j) * kCols + c;
        if (c < width) {
          if (m >= 0) fast::cp_async16(dst, in + m * a.inner + c);
          else *reinterpret_cast<float4*>(dst) = make_float4(cv, cv, cv, cv);
        }
      }
    } else {
      const int c = tid & 63;
      for (int j = tid >> 6; j < rows; j += kThreads / 64) {
        const int m = strip::fold(l0 - a.anchor + j0 + j, a.L, a.mode);
        float* dst = sm_ring + (s0 + j) * kCols + c;
        if (c < width) {
          if (m >= 0) fast::cp_async4(dst, in + m * a.inner + c);
          else *dst = cv;
        }
      }
    }
    fast::cp_commit();
  };

  stage(0, min(S, KT - 1 + n), 0);  // rows beyond feed nothing that is stored
  fast::cp_wait<0>();
  __syncthreads();
  const int c = 2 * lane;
  float* out = a.out + (o * a.L + l0) * a.inner + i0 + c;
  int base = 0;  // slot of the step's first row
  for (int g0 = 0; g0 < n; g0 += kRows) {
    if (g0 + kRows < n) {
      // into the slots that this step does not read: those of the step before
      const int next = base + S >= R ? base + S - R : base + S;
      const int first = min(kRows, R - next);
      stage(S + g0, first, next);
      if (first < kRows) stage(S + g0 + first, kRows - first, 0);
    }
    const int left = n - g0 - 8 * warp;  // rows of this warp that are stored
    if (left > 0 && c < width) {
      int slot = base + 8 * warp;
      if (slot >= R) slot -= R;
      constexpr int kBlocks = (KT + 7 + 7) / 8;
      f2 win[8 * kBlocks], acc[8];
      auto load = [&](int b) {
        const float* at = sm_ring + slot * kCols + c;
#pragma unroll
        for (int j = 0; j < 8; ++j) win[8 * b + j] = *reinterpret_cast<const f2*>(at + j * kCols);
        slot += 8;
        if (slot >= R) slot -= R;
      };
      load(0);
#pragma unroll
      for (int p = 0; p < 8; ++p) acc[p] = 0ull;
#pragma unroll
      for (int k = 0; k < KT; ++k) {
        if (k % 8 == 0 && k / 8 + 1 < kBlocks) load(k / 8 + 1);
        if (strip::tap_on<KT, NP, GEN, false>(k, a.y.K, a.y.centre, a.y.act)) {
#pragma unroll
          for (int p = 0; p < 8; ++p) acc[p] = fma2(win[k + p], a.y.w[k], acc[p]);
        }
      }
      float* q = out + (g0 + 8 * warp) * a.inner;
      if (a.vec && left >= 8) {
#pragma unroll
        for (int p = 0; p < 8; ++p) *reinterpret_cast<f2*>(q + p * a.inner) = acc[p];
      } else {
#pragma unroll
        for (int p = 0; p < 8; ++p)
          if (p < left) {
            q[p * a.inner] = lo2(acc[p]);
            if (c + 1 < width) q[p * a.inner + 1] = hi2(acc[p]);
          }
      }
    }
    fast::cp_wait<0>();
    __syncthreads();
    base += kRows;
    if (base >= R) base -= R;
  }
}

template <int KT, int NP, bool GEN>
int launch_ring_k(const PassDesc& d, const float* w, int K, int anchor, bool skip, const void* in,
                  void* out, cudaStream_t st) {
  RingArgs<KT> a{};
  a.in = static_cast<const float*>(in);
  a.out = static_cast<float*>(out);
  a.inner = d.inner;
  a.L = static_cast<int>(d.L);
  a.anchor = anchor;
  a.mode = d.mode;
  a.vec = d.inner % 4 == 0 && strip::aligned(in, 16) && strip::aligned(out, 8);
  a.cval = d.cval;
  a.cin = d.cval_as_input ? 1 : 0;
  strip::put_taps(a.y, w, K, skip, false);
  auto* kern = k_ring<KT, NP, GEN>;
  constexpr int smem = smem_bytes(KT);
  static_assert(smem <= 75 * 1024, "three CTAs per SM");
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  std::call_once(once, [&] {
    attr = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  });
  if (attr != cudaSuccess) return cuda_fail(attr, "ring pass shared memory attribute");
  a.tiles = static_cast<int>((d.inner + kCols - 1) / kCols);
  const long long gx = a.tiles * d.outer;
  // a row costs K and its load and store, the start of a chunk its rows' loads
  a.chunk = strip::choose_chunk_y(d.L, (double)gx, 148.0 * 3, kRows, K + 8, 4.0 * K + 1000,
                                  1 << 30);
  if (gx > 0x7fffffffLL) return CIMX_FUSED_DECLINED;
  kern<<<dim3((unsigned)gx, (unsigned)((d.L + a.chunk - 1) / a.chunk)), kThreads, smem, st>>>(a);
  return cuda_fail(cudaGetLastError(), "ring pass launch");
}

}  // namespace ring
}  // namespace cimx
