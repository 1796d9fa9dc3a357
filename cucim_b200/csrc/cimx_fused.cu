// cimx_fused.cu — decides whether a pass list runs on the fast kernels
// (cimx_strip.cuh, cimx_vol.cuh) and schedules them: a 3-D filter with short
// taps on all three axes is one launch of the volume kernel (k_vol);
// otherwise passes along leading axes are one launch each (k_columns; the
// generic kernel for what it does not cover), the passes along the last two
// axes run fused in one strip launch (k_strip) or, where their taps are long
// or unequal, as a column launch and a strip launch. Intermediates follow
// cuCIM's _run_1d_filters ping-pong: every pass writes the output dtype, the
// last launch writes the caller's output, one scratch buffer takes the others.
#include <algorithm>
#include <cstring>

#include "cimx_common.cuh"
#include "cimx_fused.h"

namespace cimx {
namespace {

// (T, D) pairs with fast kernels; all of them use float32 weights.
bool fast_pair(int t, int d) {
  switch (t) {
    case DT_F32: return d == DT_F32;
    case DT_U16: return d == DT_F32 || d == DT_U16;
    case DT_U8: return d == DT_F32 || d == DT_U8 || d == DT_U16;
    default: return false;
  }
}

struct Trimmed {
  int K = 0, anchor = 0;
  bool interior_zero = false;
  float w[kLongMaxK];
};

// Taps rounded to float32; with the elementwise-kernel rule, zero taps at
// both ends are dropped (exact: they never enter the chain).
bool trim(const PassDesc& d, int max_k, Trimmed& t) {
  if (d.w64) return false;
  int lo = 0, hi = d.K;
  auto w = [&](int k) { return static_cast<float>(d.taps[k]); };
  if (d.skip_zero) {
    while (lo < hi && w(lo) == 0.f) ++lo;
    while (hi > lo && w(hi - 1) == 0.f) --hi;
  }
  t.K = hi - lo;
  if (t.K < 1 || t.K > max_k) return false;
  t.anchor = d.anchor - lo;
  t.interior_zero = false;
  for (int k = lo; k < hi; ++k) {
    t.w[k - lo] = w(k);
    if (d.skip_zero && w(k) == 0.f) t.interior_zero = true;
  }
  return true;
}

bool aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

int launch_strip(const SlabArgs& a, int tin, int tout, cudaStream_t st) {
  if (a.B == 0) return CIMX_OK;
  switch (tin) {
    case DT_F32: return launch_strip_f32(a, tout, st);
    case DT_U16: return launch_strip_u16(a, tout, st);
    case DT_U8: return launch_strip_u8(a, tout, st);
    default: return CIMX_FUSED_DECLINED;
  }
}

int launch_columns(const PassDesc& d, const Trimmed& t, int tin, const void* in, int tout,
                   void* out, cudaStream_t st) {
  if (d.outer * d.L * d.inner == 0) return CIMX_OK;
  const bool skip = d.skip_zero && t.interior_zero;
  if (tin == DT_F32 && tout == DT_F32 && ring_takes(d.L, t.K))
    return launch_ring_f32(d, t.w, t.K, t.anchor, skip, in, out, st);
  switch (tin) {
    case DT_F32: return launch_columns_f32(d, t.w, t.K, t.anchor, skip, in, tout, out, st);
    case DT_U16: return launch_columns_u16(d, t.w, t.K, t.anchor, skip, in, tout, out, st);
    case DT_U8: return launch_columns_u8(d, t.w, t.K, t.anchor, skip, in, tout, out, st);
    default: return CIMX_FUSED_DECLINED;
  }
}

// Extents the column and strip kernels take: narrower inner extents than 32
// leave most of a warp's sectors unused, the strip works on 8 rows at a time,
// and both index with 32 bits along an axis.
constexpr int kColumnsMinInner = 32;
constexpr int kStripMinRows = 4;
constexpr int64_t kMaxExtent = 1LL << 30;

// Whether the y and x passes share one strip launch. Fused, a value is read
// and written once; apart, each pass has all registers and the y pass no x
// halo. Measured on 256^3 float32, (y, x) fused against apart: 9 / 9 taps 42
// against 58 us, 17 / 17 51 against 62, 33 / 33 71 against 83, 57 / 57 130
// against 120; unequal counts (tested tap by tap when fused): 9 / 17 52
// against 65, 33 / 17 96 against 78.
bool strip_fuses(size_t elem, const PassDesc& dy, const Trimmed& y, const PassDesc& dx,
                 const Trimmed& x) {
  const int K = std::max(y.K, x.K);
  if (K <= 17) return true;
  if (K > 33 || kt_bound(elem, y.K) != kt_bound(elem, x.K)) return false;
  return skip_kind(y.w, y.K, dy.skip_zero && y.interior_zero) < 2 &&
         skip_kind(x.w, x.K, dx.skip_zero && x.interior_zero) < 2;
}

void fill_slab_pass(SlabPass& s, const PassDesc& d, const Trimmed& t, int pass_in) {
  s.K = t.K;
  s.anchor = t.anchor;
  s.mode = d.mode;
  s.cval = d.cval;
  s.cval_as_input = d.cval_as_input ? 1 : 0;
  s.dt = pass_in;
  s.skip = (d.skip_zero && t.interior_zero) ? 1 : 0;
  s.pad = 0;
  std::fill(std::begin(s.w), std::end(s.w), 0.f);
  std::copy(t.w, t.w + t.K, s.w);
}

int launch_vol(const VolArgs& v, int tin, int tout, cudaStream_t st) {
  switch (tin) {
    case DT_F32: return launch_vol_f32(v, tout, st);
    case DT_U16: return launch_vol_u16(v, tout, st);
    case DT_U8: return launch_vol_u8(v, tout, st);
    default: return CIMX_FUSED_DECLINED;
  }
}

// z, y and x passes over the last three axes with the same short taps: one
// launch of the volume kernel, no intermediate volume. Against a column and a strip
// launch (CIMX_L_NO_VOLUME), us: 256 x 1024^2, 3 taps float32 506 / 733, uint16 to
// float32 484 / 647, uint16 540 / 660, uint8 530 / 612; 203 x 1021 x 1016 uint16 418
// / 541. With 5 taps it keeps the float32 volumes (671 / 733) but for 512^3 (411 /
// 381) and loses the integer ones (uint16 707 / 654, uint8 717 / 637, uint16 to
// float32 684 / 644), like 3 taps with a zero centre to integers (uint16 768 / 675):
// left to the autotuner, which tries both.
int try_vol(const CimxArray* in, const CimxArray* out, const PassDesc* ds, int zchunk,
            cudaStream_t st) {
  const int nd = in->ndim;
  const int D = out->dtype;
  if (!fast_pair(in->dtype, D)) return CIMX_FUSED_DECLINED;
  Trimmed t[3];
  for (int i = 0; i < 3; ++i)
    if (!trim(ds[i], 5, t[i])) return CIMX_FUSED_DECLINED;
  const int K = t[0].K;
  if ((K != 3 && K != 5) || t[1].K != K || t[2].K != K) return CIMX_FUSED_DECLINED;
  // the x chain takes its halo from the neighbouring lanes: centred taps,
  // and no wrap-around (whose halo lies at the far end of the row)
  if (t[2].anchor != K / 2 || ds[2].mode == CIMX_MODE_GRID_WRAP) return CIMX_FUSED_DECLINED;
  const long long X = in->shape[nd - 1], Y = in->shape[nd - 2], Z = in->shape[nd - 3];
  long long B = 1;
  for (int k = 0; k < nd - 3; ++k) B *= in->shape[k];
  if (X % 4 != 0 || X < 8 || Y < 1 || Z < 1 || B < 1) return CIMX_FUSED_DECLINED;
  if (Y * X >= (1LL << 31) || Z >= (1LL << 31)) return CIMX_FUSED_DECLINED;
  if (!aligned(in->data, 4 * dtype_size(in->dtype)) || !aligned(out->data, 4 * dtype_size(D)))
    return CIMX_FUSED_DECLINED;
  VolArgs v{};
  v.in = in->data;
  v.out = out->data;
  v.B = B;
  v.Z = Z;
  v.Y = Y;
  v.X = X;
  v.zchunk = zchunk;
  fill_slab_pass(v.pz, ds[0], t[0], in->dtype);
  fill_slab_pass(v.py, ds[1], t[1], D);
  fill_slab_pass(v.px, ds[2], t[2], D);
  return launch_vol(v, in->dtype, D, st);
}

}  // namespace

int try_fused(const CimxArray* in, const CimxArray* out, PassDesc* ds, int npasses,
              int lib_flags, cudaStream_t st, bool add, bool no_scratch) {
  const int nd = in->ndim;
  const int D = out->dtype;
  if (npasses < 1 || npasses > CIMX_MAX_NDIM || nd < 1) return CIMX_FUSED_DECLINED;
  if (add && D != DT_F32) return CIMX_FUSED_DECLINED;
  if (npasses == 2 && nd >= 2 && ds[0].axis == nd - 2 && ds[1].axis == nd - 1 &&
      in->dtype == DT_F64 && D == DT_F64)
    return try_strip_f64(ds[0], ds[1], in->data, out->data, st, no_scratch);
  // passes in strictly ascending axis order, float32 weights
  int prev_axis = -1;
  for (int i = 0; i < npasses; ++i) {
    if (ds[i].axis <= prev_axis || ds[i].w64) return CIMX_FUSED_DECLINED;
    prev_axis = ds[i].axis;
  }

  if (!add && nd >= 3 && npasses == 3 && ds[0].axis == nd - 3 && ds[1].axis == nd - 2 &&
      ds[2].axis == nd - 1 && !(lib_flags & CIMX_L_NO_VOLUME)) {
    static const int kChunks[4] = {0, 32, 64, 128};
    const int rc = try_vol(in, out, ds, kChunks[(lib_flags >> CIMX_L_ZCHUNK_SHIFT) & 3], st);
    if (rc != CIMX_FUSED_DECLINED) return rc;
  }

  // The launches, in order: one per leading axis (in columns, or generic),
  // then one or two for the last two axes.
  enum Kind { kColumns, kGeneric, kStrip };
  struct Step {
    Kind kind;
    int y, x;  // the passes it takes; kStrip: y is -1 for a lone x pass
  };
  Step steps[CIMX_MAX_NDIM];
  Trimmed tr[CIMX_MAX_NDIM];
  int nl = 0;  // launches
  int64_t n = 1, longest = 0;
  for (int k = 0; k < nd; ++k) {
    n *= in->shape[k];
    longest = std::max<int64_t>(longest, in->shape[k]);
  }
  if (longest >= kMaxExtent) return CIMX_FUSED_DECLINED;
  auto plan = [&](bool fuse_all) {
    bool fast = false;  // any launch that the generic kernels would not make
    nl = 0;
    for (int i = 0; i < npasses; ++i) {
      const int tin = i == 0 ? in->dtype : D;
      Step s{kGeneric, i, -1};
      const bool f32 = tin == DT_F32 && D == DT_F32;
      if (nd >= 2 && fast_pair(tin, D) && trim(ds[i], f32 ? kLongMaxK : kSlabMaxK, tr[i])) {
        if (ds[i].axis == nd - 1) {
          if (n / std::max<int64_t>(1, in->shape[nd - 1]) >= kStripMinRows) s = {kStrip, -1, i};
        } else if (ds[i].axis == nd - 2 && i + 1 < npasses && tr[i].K <= kSlabMaxK &&
                   trim(ds[i + 1], kSlabMaxK, tr[i + 1]) &&
                   (fuse_all || strip_fuses(dtype_size(tin), ds[i], tr[i], ds[i + 1], tr[i + 1]))) {
          s = {kStrip, i, i + 1};
          ++i;
        } else if (ds[i].inner >= kColumnsMinInner &&
                   (tr[i].K <= kSlabMaxK || ring_long(ds[i].L, ds[i].inner, tr[i].K)) &&
                   (ds[i].axis == nd - 2 || !(lib_flags & CIMX_L_NO_STREAM))) {
          s.kind = kColumns;
        }
      }
      fast |= s.kind != kGeneric;
      steps[nl++] = s;
    }
    return fast;
  };
  if (!plan(false)) return CIMX_FUSED_DECLINED;
  if (add && steps[nl - 1].kind != kStrip) return CIMX_FUSED_DECLINED;

  // ping-pong schedule: the last launch writes `out`. With `add`, `out` holds
  // the sum so far, which no other launch may touch: a second scratch buffer
  // takes its turns.
  const size_t tbytes = (size_t)n * dtype_size(D);
  void *temp = nullptr, *temp2 = nullptr;
  if (nl >= 2) {
    temp = scratch_alloc(tbytes, st);
    // without scratch memory, both tail passes in one launch whatever their taps
    if (!temp && (!plan(true) || nl >= 2))
      return fail(CIMX_E_NOMEM, "scratch allocation for the ping-pong buffer failed");
  }
  if (add && nl >= 3) {
    temp2 = scratch_alloc(tbytes, st);
    if (!temp2) {
      scratch_free(temp, tbytes, st);
      return CIMX_FUSED_DECLINED;
    }
  }
  int rc = CIMX_OK;
  const void* src = in->data;
  int tsrc = in->dtype;
  for (int j = 0; j < nl && rc == CIMX_OK; ++j) {
    const Step& s = steps[j];
    void* const other = add ? temp2 : out->data;  // the buffer that takes turns with temp
    void* dst = j == nl - 1 ? out->data : (nl - 1 - j) % 2 ? temp : other;
    switch (s.kind) {
      case kColumns: rc = launch_columns(ds[s.y], tr[s.y], tsrc, src, D, dst, st); break;
      case kGeneric: {
        PassDesc d = ds[s.y];
        d.in = src;
        d.out = dst;
        d.tin = tsrc;
        d.tout = D;
        rc = launch_generic_pass(d, st);
        break;
      }
      default: {
        SlabArgs a{};
        a.in = src;
        a.out = dst;
        a.X = in->shape[nd - 1];
        a.Y = in->shape[nd - 2];
        a.B = (a.X * a.Y == 0) ? 0 : n / (a.X * a.Y);
        int pass_in = tsrc;
        if (s.y >= 0) {
          fill_slab_pass(a.py, ds[s.y], tr[s.y], pass_in);
          a.has_y = 1;
          pass_in = D;
        } else {
          // the x pass alone: all rows of the array as one slab, staged by an
          // identity y pass
          if (a.B * a.Y < kMaxExtent) {
            a.Y *= a.B;
            a.B = 1;
          }
          a.py.K = 1;
          a.py.mode = CIMX_MODE_NEAREST;  // no halo: K = 1, anchor 0
          a.py.dt = pass_in;
          a.py.w[0] = 1.f;
        }
        a.has_x = 1;
        a.add = add && j == nl - 1;
        fill_slab_pass(a.px, ds[s.x], tr[s.x], pass_in);
        rc = launch_strip(a, tsrc, D, st);
      }
    }
    src = dst;
    tsrc = D;
  }
  scratch_free(temp2, tbytes, st);
  scratch_free(temp, tbytes, st);
  // every check that can decline ran before the first launch
  return rc == CIMX_FUSED_DECLINED ? fail(CIMX_E_INVALID, "fast kernel missing") : rc;
}

}  // namespace cimx
