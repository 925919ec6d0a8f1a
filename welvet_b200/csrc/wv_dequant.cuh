// One dequantised weight, bit for bit: restates the reference's Unpack formulas (quant/q4_0.go:47-79, q4_1.go:51-76,
// q5_0.go:47-68, q5_1.go:48-70, q8_0.go:46-66, kquant.go:178-188, iq.go:169-180, ternary.go:53-62,
// binary.go:49-84, affine_g64.go:121-175, core/floatconv.go:21-46) with one explicitly rounded float32 operation per Go
// operation. Used where weights go one at a time: unpack, decoded rows, the weight-by-weight GEMV.
#pragma once
#include "wv_common.cuh"

static __constant__ float c_iq4nl[16] = WV_IQ4NL_GRID;

__device__ __forceinline__ float f16_bits_to_f32(unsigned h) {  // core/floatconv.go:21-36
  unsigned sign = (h & 0x8000u) << 16, expo = (h >> 10) & 0x1fu, mant = h & 0x3ffu;
  if (expo == 0) {
    if (mant == 0) return __uint_as_float(sign);
    float d = __fmul_rn((float)mant, 5.9604644775390625e-08f);  // mant / 1024 / 16384, exact
    return __uint_as_float(sign | __float_as_uint(d));
  }
  if (expo == 31) return __uint_as_float(sign | 0x7f800000u | (mant << 13));
  return __uint_as_float(sign | ((expo - 15 + 127) << 23) | (mant << 13));
}

__device__ __forceinline__ float wv_dequant(const WvDevBlob& b, const WvFmtInfo fi, long long i) {
  if (fi.kind == WK_NONE) {
    if (b.dtype == WV_DT_F32) return __uint_as_float(b.lo[i]);
    unsigned h = reinterpret_cast<const uint16_t*>(b.lo)[i];
    return b.dtype == WV_DT_F16 ? f16_bits_to_f32(h) : __uint_as_float(h << 16);
  }
  unsigned u = wv_dev_code(b, fi.bits_lo, fi.bits_hi, i);
  switch (fi.kind) {
  case WK_CLASSIC: {
    float scale = b.p0[i >> 5];
    if (fi.has_min) return __fadd_rn(b.p1[i >> 5], __fmul_rn((float)u, scale));
    return __fmul_rn((float)((int)u - fi.mid), scale);
  }
  case WK_KQUANT: {
    float2 dd = reinterpret_cast<const float2*>(b.p0)[i >> 8];
    int g = (int)((i & 255) >> 4);
    long long ch = i >> 5;
    unsigned su, mu = 0;
    if (fi.has_min) { unsigned km = b.km[ch]; su = (km >> (8 * (g & 1))) & 0xffu; mu = (km >> (16 + 8 * (g & 1))) & 0xffu; }
    else { unsigned km = reinterpret_cast<const uint16_t*>(b.km)[ch]; su = (km >> (8 * (g & 1))) & 0xffu; }
    float sc = __fdiv_rn(__fmul_rn(dd.x, (float)su), 255.0f);
    if (sc == 0.0f) sc = __fdiv_rn(dd.x, 255.0f);
    if (fi.has_min) {
      float mn = __fdiv_rn(__fmul_rn(dd.y, (float)(int)(signed char)mu), 127.0f);
      return __fadd_rn(mn, __fmul_rn((float)u, sc));
    }
    return __fmul_rn(sc, (float)((int)u - fi.mid));
  }
  case WK_IQ: {
    float scale = b.p0[i / fi.pgroup];
    if (fi.table) return __fmul_rn(scale, c_iq4nl[u & 15]);
    if (fi.sign) return (u & 1) ? scale : -scale;
    return __fmul_rn(scale, __fsub_rn((float)u, (float)fi.mid + 0.5f));
  }
  case WK_TERNARY: {
    float scale = b.p0[i >> 4];
    return u == 0 ? -scale : (u == 2 ? scale : 0.0f);
  }
  case WK_BINARY: {
    float scale = b.p0[i / b.group];
    return (u & 1) ? scale : -scale;
  }
  case WK_AFFINE: {
    long long g = i / b.group;
    return __fadd_rn(__fmul_rn(b.p0[g], (float)u), b.p1[g]);
  }
  }
  return 0.0f;
}
