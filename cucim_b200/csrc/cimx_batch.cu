// cimx_batch.cu — many uneven tiles in one launch: for every
// uint8 RGB tile, rgb2gray, then a gaussian (its own sigma, mode 'nearest'),
// then the sobel gradient magnitude (mode 'reflect'), float32 out — the
// pipeline of skimage.color.rgb2gray -> skimage.filters.gaussian ->
// skimage.filters.sobel (color/colorconv.py:1038-1095,
// _shared/filters.py:21-166, filters/edges.py:148-306), computed with exactly
// the arithmetic of the per-tile path of this library:
//   gray  = (float)(0.0721 b + (0.2125 r + 0.7154 g)) in float64 fused multiply-adds,
//           r = (float)u8 * (float)(1/255) widened to float64;
//   T     = gaussian along y of gray (float32 FMA chain, taps ascending, from +0),
//   S     = gaussian along x of T, both with 'nearest' borders;
//   d0    = smooth along x of (edge along y of S), d1 = smooth along y of (edge along x of S),
//           edge taps [-a, 0, a] (a = 1/sqrt(2) in float32), smooth [1/4, 1/2, 1/4],
//           'reflect' borders, float32 intermediates;
//   out   = sqrt(d0*d0 + d1*d1), each product and the sum rounded to float32.
//
// Work: a tile is cut into strips of up to C - 2 - 2r output columns and chunks
// of rows; a CTA of C threads walks down a strip, 16 rows at a time, on C staged
// columns:
//   * gray rows live in a ring in shared memory, the K - 1 + 16 rows that a
//     group's y chains read: every pixel is converted once per strip (1.1 to
//     1.35 times in all, for the halo columns) and its words are loaded while
//     the previous group is filtered;
//   * y chains: a thread takes a column pair and 8 rows, the rows streaming
//     through a register window in blocks of 8 (ring slots in multiples of 8:
//     a block never wraps), one f32x2 FMA per tap and pair;
//   * x chains: a thread takes a row pair and 8 columns of the result;
//   * edges and magnitude: a thread takes one column and 4 rows, so that a
//     warp's stores cover consecutive floats at any alignment.
// Two barriers per 16 rows. C = 256: two CTAs per SM up to 65 taps (113 KB each,
// set by the batch's largest radius). C = 128 up to 17 taps, where the halo of
// narrow strips is short: four CTAs per SM, whose barriers and loads overlap, and
// 64 x 64 tiles leave half as many columns idle (4000 of them, 5 / 17 taps, 225 /
// 253 us against 362 / 407 with C = 256; 1000 of 128 x 128 227 / 247 against 205 /
// 228; the mean over 1 to 4000 tiles of 32 to 4096 a side 0.87).
//
// Chunks have 14 to 510 rows (batch_groups): few tiles are cut into short ones,
// or they would leave the chip idle (one tile of 1024^2 is 10 strips of 510 rows),
// many tiles into long ones, which convert fewer halo rows. The tile table gives
// every tile a range of block indexes; its items are spread evenly over that
// range (find_item), so that consecutive CTAs take about one item each whatever
// the tile sizes. 16 tiles of 256^2, 17 taps: 21 us, against 574 with 510-row
// chunks whose indexes lay at the start of each range, a CTA's a grid apart.
//
// Bound: instruction issue, shared between the FMAs (about K (1 + 256 /
// (254 - 2r)) per pixel) and the conversion and edge arithmetic (about 100
// instructions per pixel), at 16 warps per SM with barriers (51 % of the issue
// slots used). 1024 tiles of 64-1024 a side, sigmas 0.5-8: 2.97 ms (3.16 with
// the indexes a grid apart); 64 x 64 blocks with a halo on all sides, whose gray
// region is 2.3 times the output at 33 taps and 4.1 at 65, 6.99.
// The launch reads only device memory that the caller prepared, so it can
// be captured in a CUDA graph and replayed.
#include <algorithm>
#include <cmath>
#include <mutex>

#include "cimx_common.cuh"
#include "cimx_fast.cuh"
#include "cimx_internal.h"

namespace cimx {
namespace {

constexpr int kBT = 64;          // side of the blocks that the tile table counts
constexpr int kBCols = 256;      // staged columns of a strip and threads of its CTA
constexpr int kBNarrow = 128;    // the same for short filters
constexpr int kBG = 16;          // rows per group
constexpr int kBSRows = kBG + 2;      // smoothed rows kept for the edge passes
constexpr int kBMaxTaps = 129;   // radius <= 64
constexpr int kBNarrowTaps = 17;
static_assert(sizeof(CimxBatchTile) == 56, "CimxBatchTile layout is part of the ABI");

struct BatchArgs {
  const CimxBatchTile* tiles;
  int ntiles;
  long long nblocks;
  const float* taps;
  int max_r;
  int rows;  // most output rows per chunk
  int places;  // per block index
  int per;   // places per CTA, at most one per warp
  float edge[3], smooth[3];
};

__device__ __forceinline__ int nearest_idx(int i, int n) { return i < 0 ? 0 : (i >= n ? n - 1 : i); }

// gray = (float)(0.0721 b + (0.2125 r + 0.7154 g)) in float64 fused
// multiply-adds, in the order in which the per-tile rgb2gray kernel contracts
// them, of three bytes. A channel is (double)((float)u * (float)(1 / 255)):
// with c = (float)(1 / 255), 2^23 + u is a float and 2^23 c is one too, so one
// FMA, (2^23 + u) c - 2^23 c, gives u c rounded once; the float is widened by
// rebiasing its exponent (the conversion unit is a sixteenth of the FMA rate, a
// table's random reads conflict on the banks). That makes 2^-127 of a zero,
// which vanishes beside any other channel; black pixels are put right at the
// end.
__device__ __forceinline__ float luma(uint32_t r, uint32_t g, uint32_t b) {
  auto chan = [](uint32_t u) {
    constexpr float c = static_cast<float>(1.0 / 255.0);
    const uint32_t f = __float_as_uint(fmaf(__uint_as_float(0x4B000000u | u), c, -8388608.0f * c));
    return __hiloint2double(static_cast<int>((f >> 3) + ((1023u - 127u) << 20)),
                            static_cast<int>(f << 29));
  };
  const float v = __double2float_rn(
      __fma_rn(0.0721, chan(b), __fma_rn(0.2125, chan(r), __dmul_rn(0.7154, chan(g)))));
  return (r | g | b) ? v : 0.f;
}

using fast::f2;
using fast::fma2;
using fast::hi2;
using fast::lo2;
using fast::pack2;

// Shared memory of one CTA, in this order: taps as (w, w) pairs; the gray ring,
// a multiple of 8 rows that covers the K - 1 + kBG rows of one group's chains;
// T, the group's y results as row pairs, 16 spare bytes per row pair so that 8
// row pairs hit distinct banks; S, kBSRows smoothed rows as a ring of row pairs.
// The x chains read up to 16 columns past a row pair: values that no stored
// output uses, the last of them in S.
constexpr int kTapBytes = (kBMaxTaps + 1) * 8;
__host__ __device__ constexpr int t_pitch(int C) { return C * 8 + 16; }
__host__ __device__ constexpr int t_bytes(int C) { return kBG / 2 * t_pitch(C); }
__host__ __device__ constexpr int ring_rows(int K) { return (K - 1 + 7) / 8 * 8 + kBG; }
__host__ __device__ constexpr int s_pitch(int C, int K) { return (C - (K - 1) + 7) / 8 * 8 + 4; }
// for K taps and fewer: S is widest for the shortest filter with K's ring, and
// the next longer ring adds 8 KB against 8 columns of S
__host__ __device__ constexpr int batch_smem(int C, int K) {
  const int widest = C + 8 - (K - 1 + 7) / 8 * 8 + 4;
  return kTapBytes + ring_rows(K) * C * 4 + t_bytes(C) + kBSRows * widest * 4;
}
static_assert(batch_smem(kBCols, 65) <= 113 * 1024 - 256, "two CTAs per SM up to 65 taps");
static_assert(batch_smem(kBCols, kBMaxTaps) <= 223 * 1024, "longest filter");
static_assert(batch_smem(kBNarrow, kBNarrowTaps) <= 48 * 1024, "four CTAs per SM, no opt-in");
static_assert(kBCols - (kBMaxTaps - 1) - 2 >= kBT && kBNarrow - (kBNarrowTaps - 1) - 2 >= kBT,
              "a tile has no more strips than columns of blocks");

// acc[p] = the chain over taps k = 0 .. K-1 of x(p + k) * w[k] for 8
// consecutive outputs of two lines, taps ascending from +0. `load8(b, v)` gives
// the inputs 8 b .. 8 b + 7, called with b = 0, 1, .. in turn, up to 7 inputs
// past the last one used.
template <class Load8>
__device__ __forceinline__ void chain8(f2 (&acc)[8], const f2* w, int K, Load8 load8) {
  f2 lo[8], hi[8];
#pragma unroll
  for (int p = 0; p < 8; ++p) acc[p] = 0ull;
  auto block = [&](const f2(&u)[8], const f2(&v)[8], const f2* wk) {
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      const ulonglong2 w2 = *reinterpret_cast<const ulonglong2*>(wk + j);
#pragma unroll
      for (int p = 0; p < 8; ++p) acc[p] = fma2(p + j < 8 ? u[p + j] : v[p + j - 8], w2.x, acc[p]);
#pragma unroll
      for (int p = 0; p < 8; ++p)
        acc[p] = fma2(p + j + 1 < 8 ? u[p + j + 1] : v[p + j - 7], w2.y, acc[p]);
    }
  };
  load8(lo);
  int k = 0;
  for (; k + 16 <= K; k += 16) {
    load8(hi);
    block(lo, hi, w + k);
    load8(lo);
    block(hi, lo, w + k + 8);
  }
  if (k + 8 <= K) {
    load8(hi);
    block(lo, hi, w + k);
    k += 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) lo[j] = hi[j];
  }
  if (k < K) {  // 1 to 7 taps more
    load8(hi);
#pragma unroll
    for (int j = 0; j < 7; ++j)
      if (k + j < K) {
        const f2 wj = w[k + j];
#pragma unroll
        for (int p = 0; p < 8; ++p) acc[p] = fma2(p + j < 8 ? lo[p + j] : hi[p + j - 8], wj, acc[p]);
      }
  }
}

// one strip of one chunk of a tile
struct BatchItem {
  int tile, x0, xw, y0, rows;  // tile < 0: nothing to do
};

// The item of a place. Every block index has a.places of them; a tile's items are
// spread over its places, the others have none.
template <int C>
__device__ __forceinline__ BatchItem find_item(const BatchArgs& a, long long place, int lane) {
  const long long g = place / a.places;
  // the last tile whose first block <= g, found by a warp: each round probes 32
  // evenly spaced tiles of (lo, hi] and keeps the span between the last probe
  // <= g and the next one (three rounds for 4096 tiles)
  int lo = 0, hi = a.ntiles - 1;
  while (hi > lo) {
    const int step = (hi - lo + 31) / 32;
    const int cand = lo + 1 + lane * step;
    const bool le = cand <= hi && a.tiles[cand].first_block <= g;
    const int nle = __popc(__ballot_sync(0xffffffffu, le));
    if (nle == 0) {
      hi = lo;
    } else {
      lo += 1 + (nle - 1) * step;
      hi = min(hi, lo + step - 1);
    }
  }
  BatchItem it{-1, 0, 0, 0, 0};
  const CimxBatchTile& t = a.tiles[lo];
  const int K = t.ntaps, H = t.height, W = t.width;
  const long long j = place - t.first_block * a.places;
  // a block index outside the tile (inconsistent table) is skipped
  if (j < 0 || K < 1 || K / 2 > a.max_r || H < 1 || W < 1) return it;
  const int r = K / 2;
  const int wmax = C - 2 - 2 * r;
  const long long np = (W + kBT - 1LL) / kBT * ((H + kBT - 1LL) / kBT) * a.places;
  if (j >= np) return it;
  const int nx = (W + wmax - 1) / wmax;
  int ny = static_cast<int>(min((H + a.rows - 1LL) / a.rows, np / nx));
  const int xw = (W + nx - 1) / nx;
  const int rows = ((H + ny - 1) / ny + 2 + kBG - 1) / kBG * kBG - 2;
  ny = (H + rows - 1) / rows;
  // item k has place k np / (nx ny)
  const long long ni = static_cast<long long>(nx) * ny;
  const long long k = (j * ni + np - 1) / np;
  if (k >= ni || k * np / ni != j) return it;
  it.x0 = static_cast<int>(k % nx) * xw;
  it.y0 = static_cast<int>(k / nx) * rows;
  it.xw = min(xw, W - it.x0);
  it.rows = min(rows, H - it.y0);
  if (it.xw > 0 && it.rows > 0) it.tile = lo;
  return it;
}

// MID: the edge taps have a middle one
template <int C, bool MID>
__global__ void __launch_bounds__(C, 512 / C) k_batch_gray_gauss_sobel(const BatchArgs a) {
  extern __shared__ __align__(16) unsigned char sm_batch[];
  __shared__ BatchItem s_item[C / 32];
  constexpr int kTPitch = t_pitch(C);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (warp < a.per) {  // one place per warp
    const long long place = static_cast<long long>(blockIdx.x) * a.per + warp;
    BatchItem it{-1, 0, 0, 0, 0};
    if (place < a.nblocks * a.places) it = find_item<C>(a, place, lane);
    if (lane == 0) s_item[warp] = it;
  }
  __syncthreads();
  f2* const taps = reinterpret_cast<f2*>(sm_batch);
  float* const ring = reinterpret_cast<float*>(sm_batch + kTapBytes);

  for (int n = 0; n < a.per; ++n) {
    const BatchItem it = s_item[n];
    if (it.tile < 0) continue;  // the same for every thread
    const CimxBatchTile& t = a.tiles[it.tile];
    const int H = t.height, W = t.width, K = t.ntaps, r = K / 2;
    // row pitches: a tile may be a region of a larger slide (0 = packed)
    const long long in_pitch = t.rgb_pitch > 0 ? t.rgb_pitch : 3LL * W;
    const long long out_pitch = t.out_pitch > 0 ? t.out_pitch : W;
    const uint8_t* const rgb = t.rgb;
    float* const out = t.out;
    const int R = ring_rows(K), SP = s_pitch(C, K);
    unsigned char* const T = reinterpret_cast<unsigned char*>(ring + R * C);
    f2* const S = reinterpret_cast<f2*>(T + t_bytes(C));
    // the smoothed row s of the walk is row ys + s of the tile, and the
    // smoothed column c is column x0 - 1 + c; gray row j is row ys - r + j,
    // gray column c is column x0 - 1 - r + c (both 'nearest')
    const int ys = it.y0 - 1;
    const int ns = it.xw + 2;           // smoothed columns
    const int need = ns + 2 * r;        // staged columns in use
    const int groups = (it.rows + 2 + kBG - 1) / kBG;

    for (int k = tid; k < K; k += C) {
      const float w = a.taps[t.taps_offset + k];
      taps[k] = pack2(w, w);
    }

    // gray: 4 consecutive pixels of every fourth row. Inside the tile's row
    // their 12 bytes come from three or four aligned words (each holds at least
    // one of the bytes, so it lies in the tile's allocation); at its ends byte
    // by byte.
    const int gc = tid % (C / 4) * 4, grow = tid / (C / 4);
    const int xs = it.x0 - 1 - r + gc;
    const bool gon = gc < need;
    const bool words = xs >= 0 && xs + 3 < W;
    uint32_t wv[4][4];
    unsigned shv[4];
    auto gray_load = [&](int j0) {
      if (!gon) return;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int y = min(max(ys - r + j0 + grow + 4 * u, 0), H - 1);
        const uint8_t* row = rgb + y * in_pitch;
        if (words) {
          const uintptr_t pa = reinterpret_cast<uintptr_t>(row + 3LL * xs);
          const uint32_t* wp = reinterpret_cast<const uint32_t*>(pa & ~static_cast<uintptr_t>(3));
          shv[u] = static_cast<unsigned>(pa & 3) * 8u;
          wv[u][0] = __ldg(wp);
          wv[u][1] = __ldg(wp + 1);
          wv[u][2] = __ldg(wp + 2);
          wv[u][3] = 0u;
          if (shv[u]) wv[u][3] = __ldg(wp + 3);
        } else {
          shv[u] = 0;
          wv[u][0] = wv[u][1] = wv[u][2] = wv[u][3] = 0u;
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            const uint8_t* px = row + 3LL * nearest_idx(xs + p, W);
#pragma unroll
            for (int c = 0; c < 3; ++c)
              wv[u][(3 * p + c) / 4] |= static_cast<uint32_t>(__ldg(px + c)) << ((3 * p + c) % 4 * 8);
          }
        }
      }
    };
    auto gray_store = [&](int slot) {  // ring slot of the first of the kBG rows (a multiple of 8)
      if (!gon) return;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t v0 = __funnelshift_r(wv[u][0], wv[u][1], shv[u]);
        const uint32_t v1 = __funnelshift_r(wv[u][1], wv[u][2], shv[u]);
        const uint32_t v2 = __funnelshift_r(wv[u][2], wv[u][3], shv[u]);
        int q = slot + grow + 4 * u;
        if (q >= R) q -= R;
        *reinterpret_cast<float4*>(ring + q * C + gc) = make_float4(
            luma(v0 & 255u, (v0 >> 8) & 255u, (v0 >> 16) & 255u),
            luma(v0 >> 24, v1 & 255u, (v1 >> 8) & 255u),
            luma((v1 >> 16) & 255u, v1 >> 24, v2 & 255u),
            luma((v2 >> 8) & 255u, (v2 >> 16) & 255u, v2 >> 24));
      }
    };

    // the first group's rows: R = K - 1 + kBG rounded up, a multiple of 8; the
    // last fill may wrap on to the ring's start when R is not a multiple of
    // kBG, so it fills only what is left
    for (int j = 0; j + kBG <= R; j += kBG) {
      gray_load(j);
      gray_store(j);
    }
    if (R % kBG) {  // 8 rows left, filled together with the 8 before them
      gray_load(R - kBG);
      gray_store(R - kBG);
    }
    __syncthreads();

    int base = 0;           // ring slot of the group's first gray row
    for (int g = 0; g < groups; ++g) {
      const bool more = g + 1 < groups;
      // the kBG rows after the ring's last one
      if (more) gray_load(R + g * kBG);
      {
        // y chains: column pair p, rows 8 q .. 8 q + 7 of the group
        const int p = tid % (C / 2), q = tid / (C / 2);
        if (2 * p < need) {
          int slot = base + 8 * q;
          if (slot >= R) slot -= R;
          const float* col = ring + 2 * p;
          f2 acc[8];
          chain8(acc, taps, K, [&](f2(&v)[8]) {
            const float* at = col + slot * C;
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = *reinterpret_cast<const f2*>(at + j * C);
            slot += 8;
            if (slot == R) slot = 0;
          });
          unsigned char* put = T + 4 * q * kTPitch + 16 * p;
#pragma unroll
          for (int i = 0; i < 4; ++i)
            *reinterpret_cast<float4*>(put + i * kTPitch) = make_float4(
                lo2(acc[2 * i]), lo2(acc[2 * i + 1]), hi2(acc[2 * i]), hi2(acc[2 * i + 1]));
        }
      }
      __syncthreads();
      if (more) gray_store(base);
      base += kBG;
      if (base >= R) base -= R;
      {
        // x chains: row pair rp, smoothed columns c0 .. c0 + 7
        const int rp = tid & 7, c0 = (tid >> 3) * 8;
        if (c0 < ns) {
          const unsigned char* at = T + rp * kTPitch + c0 * 8;
          f2 acc[8];
          chain8(acc, taps, K, [&](f2(&v)[8]) {
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
              const ulonglong2 e = *reinterpret_cast<const ulonglong2*>(at + j * 8);
              v[j] = e.x;
              v[j + 1] = e.y;
            }
            at += 64;
          });
          // 'reflect' around the tile: the first row (here), column and the last
          // column once more; the last row where the edges read it
          if (g == 0 && rp == 0 && ys < 0) {
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[e] = pack2(hi2(acc[e]), hi2(acc[e]));
          }
          const int x = it.x0 - 1 + c0;
          f2* row = S + ((g * (kBG / 2) + rp) % (kBSRows / 2)) * SP + c0;
          if (x >= 0 && x + 7 < W - 1) {
#pragma unroll
            for (int e = 0; e < 8; e += 2)
              *reinterpret_cast<ulonglong2*>(row + e) = make_ulonglong2(acc[e], acc[e + 1]);
          } else {
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (x + e >= 0 && x + e < W && c0 + e < ns) {
                row[e] = acc[e];
                if (x + e == 0) row[e - 1] = acc[e];
                if (x + e == W - 1) row[e + 1] = acc[e];
              }
          }
        }
      }
      __syncthreads();
      {
        // edges (E0 along y, E1 along x), smoothing and magnitude of output
        // rows s = 16 g - 1 + 4 rq + i of the walk, from the row pairs s - 1 ..
        // s + 4. Each value is the same chain as a separate pass over stored E0
        // and E1 would compute, two rows at a time.
        const int rq = warp & 3;
        const int s0 = g * kBG - 1 + 4 * rq;
        const f2* pair[3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
          pair[i] = S + (max(g * (kBG / 2) - 1 + 2 * rq + i, 0) % (kBSRows / 2)) * SP;
        const int below = H - (ys + s0 - 1);  // index of the row below the last one
        const bool bottom = below < 6;
        auto edge2 = [&](f2 u, f2 v, f2 w) {
          f2 e = fma2(u, pack2(a.edge[0], a.edge[0]), 0ull);
          if (MID) e = fma2(v, pack2(a.edge[1], a.edge[1]), e);
          return fma2(w, pack2(a.edge[2], a.edge[2]), e);
        };
        auto smooth2 = [&](f2 u, f2 v, f2 w) {
          return fma2(w, pack2(a.smooth[2], a.smooth[2]),
                      fma2(v, pack2(a.smooth[1], a.smooth[1]),
                           fma2(u, pack2(a.smooth[0], a.smooth[0]), 0ull)));
        };
        for (int c = (warp >> 2) * 32 + lane; c < it.xw; c += C / 4) {
          f2 v[3][3], e1[3];
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int k = 0; k < 3; ++k) v[i][k] = pair[i][c + k];
          if (bottom) {
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
              for (int k = 0; k < 3; ++k) {
                if (i > 0 && below == 2 * i) v[i][k] = pack2(hi2(v[i - 1][k]), hi2(v[i][k]));
                if (below == 2 * i + 1) v[i][k] = pack2(lo2(v[i][k]), lo2(v[i][k]));
              }
          }
#pragma unroll
          for (int i = 0; i < 3; ++i) e1[i] = edge2(v[i][0], v[i][1], v[i][2]);
          float* o = out + (ys + s0) * out_pitch + it.x0 + c;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            f2 e0[3];
#pragma unroll
            for (int k = 0; k < 3; ++k)
              e0[k] = edge2(v[i][k], pack2(hi2(v[i][k]), lo2(v[i + 1][k])), v[i + 1][k]);
            const f2 d0 = smooth2(e0[0], e0[1], e0[2]);
            const f2 d1 = smooth2(e1[i], pack2(hi2(e1[i]), lo2(e1[i + 1])), e1[i + 1]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const float p = h ? hi2(d0) : lo2(d0), q = h ? hi2(d1) : lo2(d1);
              const int s = s0 + 2 * i + h;
              if (s >= 1 && s <= it.rows)
                o[(2 * i + h) * out_pitch] = sqrtf(__fadd_rn(__fmul_rn(p, p), __fmul_rn(q, q)));
            }
          }
        }
      }
    }
    __syncthreads();  // the next item's ring may lie over this one's S
  }
}

// Row groups per chunk, from the batch's mean tile (its table is on the device):
// whole waves of CTAs against the rows that every chunk converts and filters
// again. The weights are microseconds of a lone CTA (one tile of 200 x 200, 5 to
// 129 taps: 5 to 17 for an empty chunk, 4.2 to 7.5 a group); two on an SM take
// 1.4 times as long.
int batch_groups(long long nblocks, int ntiles, int C, int K) {
  const double slots = 148.0 * (C == kBNarrow ? 4 : K <= 65 ? 2 : 1);
  const int side = std::max(
      kBT, static_cast<int>(kBT * std::sqrt(static_cast<double>(nblocks) / ntiles)));
  const int nx = (side + C - 2 - K) / (C - 1 - K);
  int groups = 0;
  double best = 0;
  for (int g : {1, 2, 3, 6, 16, 32}) {
    const int ny = (side + kBG * g - 3) / (kBG * g - 2);
    const int used = ((side + ny - 1) / ny + 2 + kBG - 1) / kBG;
    const double item = 14 + 0.05 * K + used * (4.1 + 0.026 * K);
    const double waves = static_cast<double>(ntiles) * nx * ny / slots;
    const double cost = item * std::max(1.0, 0.8 * (waves + 0.8));
    if (groups == 0 || cost < best) {
      best = cost;
      groups = g;
    }
  }
  return groups;
}

}  // namespace
}  // namespace cimx

using namespace cimx;

extern "C" int cimx_batch_gray_gauss_sobel(const CimxBatchTile* tiles, int ntiles,
                                           long long nblocks, const float* taps, int max_taps,
                                           const float* edge_taps, const float* smooth_taps,
                                           void* stream) {
  if (ntiles < 0 || nblocks < 0) return fail(CIMX_E_INVALID, "batch: negative counts");
  if (ntiles == 0 || nblocks == 0) return CIMX_OK;
  if (!tiles || !taps || !edge_taps || !smooth_taps)
    return fail(CIMX_E_INVALID, "batch: NULL argument");
  if (max_taps < 1 || max_taps > kBMaxTaps || max_taps % 2 == 0)
    return fail(CIMX_E_INVALID, "batch: max_taps must be odd and at most 129");
  BatchArgs a{};
  a.tiles = tiles;
  a.ntiles = ntiles;
  a.nblocks = nblocks;
  a.taps = taps;
  a.max_r = max_taps / 2;
  for (int k = 0; k < 3; ++k) {
    a.edge[k] = edge_taps[k];
    a.smooth[k] = smooth_taps[k];
  }
  const bool narrow = max_taps <= kBNarrowTaps;
  const int C = narrow ? kBNarrow : kBCols;
  const size_t smem = batch_smem(C, max_taps);
  constexpr int kDynLimit = 223 * 1024;
  using Kernel = void (*)(const BatchArgs);
  static constexpr Kernel kKernels[2][2] = {
      {k_batch_gray_gauss_sobel<kBCols, false>, k_batch_gray_gauss_sobel<kBCols, true>},
      {k_batch_gray_gauss_sobel<kBNarrow, false>, k_batch_gray_gauss_sobel<kBNarrow, true>}};
  const Kernel kern = kKernels[narrow][edge_taps[1] != 0.f];
  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  std::call_once(once, [] {
    for (auto* k : kKernels[0]) {
      const cudaError_t e =
          cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kDynLimit);
      if (e != cudaSuccess) attr_err = e;
    }
  });
  if (attr_err != cudaSuccess) return cuda_fail(attr_err, "batch: shared memory attribute");
  const int groups = batch_groups(nblocks, ntiles, C, max_taps);
  a.rows = kBG * groups - 2;
  a.places = std::max(1, 8 / groups);
  // about one item per CTA; a place without one costs its lookup, of which few
  // matter
  const int wmax = C - 2 - 2 * a.max_r;
  a.per = static_cast<int>(std::max(
      1LL, std::min({nblocks * a.places / 1024, C / 32LL,
                     (long long)wmax * a.rows / (kBT * kBT * a.places)})));
  const long long grid = (nblocks * a.places + a.per - 1) / a.per;
  if (grid > 0x7fffffffLL) return fail(CIMX_E_INVALID, "batch: too many blocks");
  kern<<<(unsigned)grid, C, smem, static_cast<cudaStream_t>(stream)>>>(a);
  return cuda_fail(cudaGetLastError(), "batch launch");
}
