// What the bulk-copy-fed dp4a kernels share (wv_gemv_tma.cu: one activation row, wv_gemv_rows.cu: a few): the block shape, the
// way a lane finds and loads its chunk's fragment in a tile, and the bytes per row of each plane.
#pragma once
#include "wv_gemv_common.cuh"
#include "wv_tma_common.cuh"

#ifndef TMA_CONSUMER_WARPS
#define TMA_CONSUMER_WARPS 16
#endif
#define TMA_THREADS ((TMA_CONSUMER_WARPS + 1) * 32)
#define TMA_MAX_STAGES 8
#ifndef TMA_MAX_ROW_GROUPS
#define TMA_MAX_ROW_GROUPS 8
#endif

// Per-lane shared-memory addresses (32-bit) of this lane's chunk in row 0 of its row group,
// relative to a stage base; a row further down adds the plane's row bytes.
struct LaneOff { unsigned lo, hi, p0, p1, km; };

// G: a geometry with off[5] (plane sections of a stage) and rb[5] (bytes per row of each plane)
template <int F, typename G>
__device__ __forceinline__ LaneOff lane_offsets(const G& g, int row0, int c, int group) {
  constexpr WvFmtInfo fi = wv_fmt_info(F);
  LaneOff o;
  o.lo = g.off[0] + row0 * g.rb[0] + c * fi.bits_lo * 4;
  o.hi = g.off[1] + row0 * g.rb[1] + c * fi.bits_hi * 4;
  unsigned pi;
  if constexpr (fi.kind == WK_KQUANT) pi = (c >> 3) * 8;
  else if constexpr (fi.kind == WK_BINARY || fi.kind == WK_AFFINE) pi = ((c * 32) / group) * 4;
  else if constexpr (fi.pgroup == 16) pi = c * 8;
  else pi = c * 4;
  o.p0 = g.off[2] + row0 * g.rb[2] + pi;
  o.p1 = g.off[3] + row0 * g.rb[3] + pi;
  o.km = g.off[4] + row0 * g.rb[4] + c * (fi.has_min ? 4 : 2);
  return o;
}

// Weight fragment at addresses a.* (already advanced to the wanted row and stage).
template <int F>
__device__ __forceinline__ void load_frag_smem(FragT<F>& f, const LaneOff& a) {
  constexpr WvFmtInfo fi = wv_fmt_info(F);
  constexpr int BL = fi.bits_lo, BH = fi.bits_hi;
  if constexpr (BL == 1) f.lo[0] = lds32(a.lo);
  else if constexpr (BL == 2) { const uint2 v = lds64(a.lo); f.lo[0] = v.x; f.lo[1] = v.y; }
  else if constexpr (BL == 4) { const uint4 v = lds128(a.lo); f.lo[0] = v.x; f.lo[1] = v.y; f.lo[2] = v.z; f.lo[3] = v.w; }
  else {
    // a.lo is the chunk's 32 bytes, or their upper half for the lanes that read the halves in the
    // opposite order (see the kernel): the other half is always at a.lo ^ 16
    const uint4 v = lds128(a.lo), u = lds128(a.lo ^ 16u);
    f.lo[0] = v.x; f.lo[1] = v.y; f.lo[2] = v.z; f.lo[3] = v.w; f.lo[4] = u.x; f.lo[5] = u.y; f.lo[6] = u.z; f.lo[7] = u.w;
  }
  if constexpr (BH == 1) f.hi[0] = lds32(a.hi);
  if constexpr (BH == 2) { const uint2 v = lds64(a.hi); f.hi[0] = v.x; f.hi[1] = v.y; }
  if constexpr (fi.kind == WK_KQUANT) {
    const uint2 dd = lds64(a.p0);
    f.pr[0] = dd.x; f.pr[1] = dd.y;
    if constexpr (fi.has_min) f.pr[2] = lds32(a.km); else f.pr[2] = lds16(a.km);
  } else if constexpr (fi.kind == WK_CLASSIC || fi.kind == WK_AFFINE) {
    f.pr[0] = lds32(a.p0);
    if constexpr (fi.has_min) f.pr[1] = lds32(a.p1);
  } else if constexpr (fi.pgroup == 16) {
    const uint2 v = lds64(a.p0);
    f.pr[0] = v.x; f.pr[1] = v.y;
  } else {
    f.pr[0] = lds32(a.p0);
  }
}

static unsigned align128(unsigned v) { return (v + 127u) & ~127u; }

// Bytes per row of each plane in the device layout; false when a plane's rows are not
// 16-byte multiples (then consecutive rows cannot be fetched by bulk copies).
static bool plane_row_bytes(const WvDevBlob& b, unsigned rb[5]) {
  const WvFmtInfo fi = wv_fmt_info(b.format);
  const unsigned cpr = (unsigned)(b.cols >> 5);
  rb[0] = cpr * fi.bits_lo * 4; rb[1] = cpr * fi.bits_hi * 4; rb[2] = rb[3] = rb[4] = 0;
  switch (fi.kind) {
  case WK_CLASSIC: rb[2] = cpr * 4; rb[3] = fi.has_min ? cpr * 4 : 0; break;
  case WK_KQUANT: if (cpr % 8) return false; rb[2] = cpr; rb[4] = cpr * (fi.has_min ? 4 : 2); break;
  case WK_IQ: case WK_TERNARY: rb[2] = cpr * (fi.pgroup == 16 ? 8 : 4); break;
  case WK_BINARY: if ((b.cols % b.group) || (b.group % 32)) return false; rb[2] = (unsigned)(b.cols / b.group) * 4; break;
  case WK_AFFINE: if ((b.cols % b.group) || (b.group % 32)) return false; rb[2] = rb[3] = (unsigned)(b.cols / b.group) * 4; break;
  default: return false;
  }
  for (int i = 0; i < 5; i++) if (rb[i] % 16) return false;
  return true;
}
