// Batched Dense MatVec (batch >= 2 activation rows against one packed matrix) on the fifth-generation tensor
// cores: Y[batch][rows] = X[batch][cols] * W^T with W streamed and dequantised once, whatever the batch.
//
// The reference runs dense.Forward row by row over the batch (layers/dense/simd.go:557-614 per row,
// gemv_parallel.go:12-391); its WebGPU shaders do the same per dispatch. Here the batch is the N dimension of a
// tcgen05.mma: a CTA owns 128 rows of W (the MMA's M) and a range of the columns (split-K). A pipeline stage is a
// 32-column slice. The 512 producer threads form four groups of 128 (a thread per row); each group owns a run of
// consecutive columns and the groups' slices go through the pipeline in turn, so that a thread reads its row 128 bits to
// 64 bytes at a time although every slice is one chunk wide (the order in which slices are summed is free as long as X
// takes the same one). A thread dequantises a 32-weight chunk to TF32 values and stores them to tensor memory, where a row is
// a lane and a value a column (the MMA's A operand); one thread copies the matching slice of X (rounded to TF32 by a kernel in
// front) to shared memory, one elected thread issues four tcgen05.mma (M 128, N = batch padded to 16, K 8) per slice into a
// TMEM accumulator, and tcgen05.commit hands the stage back. At the end all producer warps read the accumulator with
// tcgen05.ld; the splits of a row tile are one thread-block cluster, which adds its accumulators up in split order through
// distributed shared memory.
//
// Bound: the latency and the instructions of the producers (0.7 to 1 us for the four groups' slices of a round), at 256 rows the
// tensor pipe as well. With W's slices in tensor memory instead of shared memory a chunk takes two stores instead of eight and no
// proxy fence, and shared memory holds X alone: the rest is L1, where the second half of every 128-byte line of W waits for the
// next unit (forcing the whole carve-out on the same code: Q8_0, 33 rows, 4096 x 4096 13.8 -> 17.2 us). us per launch, slices of
// W in shared memory and sums of one row of W at a time / in tensor memory, four rows at a time / and with the early start described
// at tcg_round_x_kernel, as now: Q8_0 4096 x 4096, 33 rows 16.7 / 13.7 / 12.4; Q8_0 14336 x 4096, 8 rows 39.1 / 30.4 / 27.3; Q4_K
// 4096 x 4096, 128 rows 18.7 / 16.0 / 15.1 and 256 rows 24.7 / 22.1 / 21.4; Q4_K 14336 x 4096, 256 rows 55.6 / 47.9 / 46.0.
//
// Arithmetic: X is rounded to TF32 (round to nearest, 11 significant bits) with its low bits cleared, a weight by adding half a
// unit of the eleventh bit to it, the rest being the tensor core's truncation, which reads an operand's upper 19 bits only;
// products are exact in the FP32 accumulator. Each term
// is off by at most 2^-11 + 2^-11 + 2^-22 of |w x|, i.e. |y - y_ref| <= 9.8e-4 * sum |w x| before accumulation
// rounding. TF32 keeps FP32's exponent range, so no operand needs scaling.
//
// Every wait is bounded: a wait that runs out records a code in the mapped error word, raises the CTA's abort flag,
// and all roles fall through to the common exit. There the copies of X and the MMAs still in flight are waited for (bounded
// again) before the TMEM columns and the shared memory are given back.
#include "wv_gemv_common.cuh"
#include "wv_tma_common.cuh"
#include "wv_dev_hooks.h"
#include <cuda.h>
#include <cudaTypedefs.h>
#include <atomic>
#include <mutex>
#include <vector>

#define TCG_PRODUCERS 512
#define TCG_THREADS (TCG_PRODUCERS + 64)     // + the MMA warp and the warp whose first lane issues the X copies
#define TCG_M 128
#define TCG_GROUPS (TCG_PRODUCERS / TCG_M)
#define TCG_MAX_STAGES (2 * TCG_GROUPS)
#define TCG_MAX_SPLIT 16    // cluster size (beyond 8 the kernel has to ask for it)

// ------------------------------------------------------------------ weight loads
template <int N> __device__ __forceinline__ void tcg_words(unsigned (&d)[N], const void* p) {
  if constexpr (N == 1) d[0] = __ldg(reinterpret_cast<const unsigned*>(p));
  else if constexpr (N == 2) { const uint2 v = __ldg(reinterpret_cast<const uint2*>(p)); d[0] = v.x; d[1] = v.y; }
  else if constexpr (N == 4) { const uint4 v = __ldg(reinterpret_cast<const uint4*>(p)); d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w; }
  else {
    static_assert(N % 8 == 0, "whole 256-bit loads");
#pragma unroll
    for (int i = 0; i < N; i += 8)
      asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                   : "=r"(d[i]), "=r"(d[i + 1]), "=r"(d[i + 2]), "=r"(d[i + 3]), "=r"(d[i + 4]), "=r"(d[i + 5]), "=r"(d[i + 6]), "=r"(d[i + 7])
                   : "l"(reinterpret_cast<const char*>(p) + 4 * i));
  }
}
// A thread's unit of loading: U consecutive chunks of its row, 64 bytes of the lo plane at most. The 32 lanes of a warp are 32
// rows, so every load touches 32 different lines and the L1 tag stage is what limits them: few wide loads, not many narrow ones
// (chunk by chunk the tag stage was busy for 17 of the 39 thousand cycles of a 4096 x 4096 Q8_0 launch).
template <int F> struct TcgUnit { static constexpr int U = wv_fmt_info(F).bits_lo == 8 ? 2 : 4; };

// VEC: the row's first chunk and the unit's are multiples of U chunks, so that every plane is read with one or two aligned
// vector loads; otherwise chunk by chunk. cnt: chunks of the unit that exist (VEC reads all U: rows are whole units).
template <int F, bool VEC>
__device__ __forceinline__ void tcg_load(FragT<F> (&f)[TcgUnit<F>::U], const WvDevBlob& b, long long ch, int cnt) {
  constexpr WvFmtInfo fi = wv_fmt_info(F);
  constexpr int U = TcgUnit<F>::U, BL = fi.bits_lo, BH = fi.bits_hi;
  if constexpr (!VEC) {
#pragma unroll
    for (int u = 0; u < U; u++) if (u < cnt) load_frag<F>(f[u], b, ch + u);
  } else {
    unsigned lo[U * BL];
    tcg_words(lo, b.lo + ch * BL);
#pragma unroll
    for (int i = 0; i < U * BL; i++) f[i / BL].lo[i % BL] = lo[i];
    if constexpr (BH > 0) {
      unsigned hi[U * BH];
      tcg_words(hi, b.hi + ch * BH);
#pragma unroll
      for (int i = 0; i < U * BH; i++) f[i / BH].hi[i % BH] = hi[i];
    }
    if constexpr (fi.kind == WK_KQUANT) {          // a unit lies inside one super-block of eight chunks
      const float2 dd = __ldg(reinterpret_cast<const float2*>(b.p0) + (ch >> 3));
      unsigned km[U];
      if constexpr (fi.has_min) tcg_words(km, b.km + ch);
      else {
        unsigned k2[U / 2];
        tcg_words(k2, reinterpret_cast<const unsigned short*>(b.km) + ch);
#pragma unroll
        for (int u = 0; u < U; u++) km[u] = (k2[u / 2] >> (16 * (u & 1))) & 0xffffu;
      }
#pragma unroll
      for (int u = 0; u < U; u++) { f[u].pr[0] = __float_as_uint(dd.x); f[u].pr[1] = __float_as_uint(dd.y); f[u].pr[2] = km[u]; }
    } else if constexpr (fi.kind == WK_BINARY || fi.kind == WK_AFFINE) {
      // Whole chunks per group. Every load is 32 lines, so a group's parameters are loaded once for the chunks of it that are in the
      // unit, and groups of one chunk like those of the other formats: a load per chunk made these formats slower at few rows of W
      // than they had been (six rows, 1024 x 14336, groups of 64: 22.3 us once, 23.9 with a load per chunk, 21.2 now).
      const unsigned cpg = (unsigned)b.group >> 5;
      if (cpg == 1) {
        unsigned p0[U], p1[U];
        tcg_words(p0, b.p0 + ch);
        if constexpr (fi.has_min) tcg_words(p1, b.p1 + ch);
#pragma unroll
        for (int u = 0; u < U; u++) {
          f[u].pr[0] = p0[u];
          if constexpr (fi.has_min) f[u].pr[1] = p1[u];
        }
        return;
      }
      unsigned gi = (unsigned)ch / cpg, in = (unsigned)ch - gi * cpg;      // `in` is the same for every row: a row is whole groups
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (u == 0 || in == 0) {
          f[u].pr[0] = __float_as_uint(__ldg(b.p0 + gi));
          if constexpr (fi.has_min) f[u].pr[1] = __float_as_uint(__ldg(b.p1 + gi));
        } else {
          f[u].pr[0] = f[u > 0 ? u - 1 : 0].pr[0];
          if constexpr (fi.has_min) f[u].pr[1] = f[u > 0 ? u - 1 : 0].pr[1];
        }
        if (++in == cpg) { in = 0; gi++; }
      }
    } else {
      constexpr int NG = fi.pgroup == 16 ? 2 : 1;
      unsigned p0[U * NG];
      tcg_words(p0, b.p0 + ch * NG);
#pragma unroll
      for (int i = 0; i < U * NG; i++) f[i / NG].pr[i % NG] = p0[i];
      if constexpr (fi.has_min) {
        unsigned p1[U];
        tcg_words(p1, b.p1 + ch);
#pragma unroll
        for (int u = 0; u < U; u++) f[u].pr[1] = p1[u];
      }
    }
  }
}

// ------------------------------------------------------------------ dequantisation of a chunk (32 weights)
__device__ __forceinline__ float tcg_tf32(float v) {
  unsigned o;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(o) : "f"(v));
  return __uint_as_float(o);
}
// Round to nearest, ties away from zero, as cvt.rna.tf32 does (which costs several instructions here): half a unit of the
// eleventh bit is added to the magnitude; the tensor core reads a TF32 operand's upper 19 bits and ignores the rest
// (clearing them first changes no bit of any output). `half` is
// zero for chunks whose scales or mins are not finite, so that a NaN's mantissa cannot run over (a finite value may round
// up to infinity, as it does with cvt.rna). The products with the scale bytes count, not the stored parameters: a finite d can
// give an infinite scale, and that times a code of zero is a NaN.
__device__ __forceinline__ float tcg_round(float v, unsigned half) { return __uint_as_float(__float_as_uint(v) + half); }
__device__ __forceinline__ bool tcg_finite(unsigned bits) { return (bits & 0x7f800000u) != 0x7f800000u; }

// The unpack kernel's arithmetic with the parameters hoisted. The two places where the reference divides (k-quant scale
// / 255, min / 127) multiply by the reciprocal here: the difference is one unit in the 24th bit, against the rounding
// to 11 bits that follows. piece(p, v): the weights 4 p .. 4 p + 3.
template <int F, typename P>
__device__ __forceinline__ void tcg_convert(const FragT<F>& f, const float* tbl, P piece) {
  constexpr WvFmtInfo fi = wv_fmt_info(F);
  constexpr int BL = fi.bits_lo, BH = fi.bits_hi, SPW = 8 / BL;
  constexpr unsigned MASK = 0x01010101u * ((1u << BL) - 1u);
  constexpr unsigned MASKH = BH ? (0x01010101u * ((1u << BH) - 1u)) << BL : 0u;
  float sc[2], mn[2] = {0.f, 0.f};
  bool fin = true;
  if constexpr (fi.kind == WK_KQUANT) {
    const float d = __uint_as_float(f.pr[0]);
#pragma unroll
    for (int h = 0; h < 2; h++) {
      // scale bytes of zero were stored as 1 at upload: both stand for d / 255 (quant/kquant.go:180-182)
      sc[h] = d * (float)(unsigned char)(f.pr[2] >> (8 * h)) * (1.0f / 255.0f);
      if constexpr (fi.has_min) mn[h] = __uint_as_float(f.pr[1]) * (float)(signed char)(f.pr[2] >> (16 + 8 * h)) * (1.0f / 127.0f);
    }
  } else {
    sc[0] = sc[1] = __uint_as_float(f.pr[0]);
    if constexpr (fi.pgroup == 16) sc[1] = __uint_as_float(f.pr[1]);
    if constexpr (fi.has_min) mn[0] = mn[1] = __uint_as_float(f.pr[1]);
  }
#pragma unroll
  for (int h = 0; h < 2; h++) fin = fin && tcg_finite(__float_as_uint(sc[h])) && (!fi.has_min || tcg_finite(__float_as_uint(mn[h])));
  const unsigned half = fin ? 0x1000u : 0u;
  if constexpr (fi.sign) {                           // +- scale: rounded once, the code is its sign
    const unsigned r = __float_as_uint(tcg_round(sc[0], half));
#pragma unroll
    for (int p = 0; p < 8; p++) {
      float v[4];
#pragma unroll
      for (int q = 0; q < 4; q++) v[q] = __uint_as_float(r ^ ((~f.lo[0] << (31 - (4 * p + q))) & 0x80000000u));
      piece(p, v);
    }
    return;
  }
  // code -> float without an integer conversion: the code lands in the mantissa of 2^23, and subtracting 2^23 + mid
  // leaves (code - mid) exactly. Groups of SPW words' worth of codes complete SPW pieces of four consecutive weights each.
  constexpr float magic = 8388608.0f + (float)fi.mid;
  float w[4 * SPW];
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int s = k % SPW;
    unsigned bytes = (f.lo[k / SPW] >> (BL * s)) & MASK;      // the codes of group k, one per byte
    if constexpr (BH > 0) {
      const int hw = (k * BH) >> 3, sh = (k * BH) & 7;
      unsigned hv = f.hi[hw];
      hv = sh >= BL ? (hv >> (sh - BL)) : (hv << (BL - sh));
      bytes |= hv & MASKH;
    }
    const int h = k >> 2;                                    // groups 0-3 are the first 16 weights
    float v[4];
#pragma unroll
    for (int m = 0; m < 4; m++) {
      if constexpr (fi.table) v[m] = sc[h] * tbl[(bytes >> (8 * m)) & 0xffu];
      else v[m] = __uint_as_float(__byte_perm(bytes, 0x4B000000u, 0x7650 + m));
    }
    if constexpr (!fi.table) {
#pragma unroll
      for (int m = 0; m < 4; m += 2) {
        float2 q = __fadd2_rn(make_float2(v[m], v[m + 1]), make_float2(-magic, -magic));
        if constexpr (fi.half_mid) q = __fadd2_rn(q, make_float2(-0.5f, -0.5f));
        if constexpr (fi.has_min) q = __ffma2_rn(q, make_float2(sc[h], sc[h]), make_float2(mn[h], mn[h]));
        else if constexpr (fi.kind == WK_TERNARY) {           // zero whatever the scale
          q.x = q.x == 0.f ? 0.f : q.x * sc[h];
          q.y = q.y == 0.f ? 0.f : q.y * sc[h];
        } else q = __fmul2_rn(q, make_float2(sc[h], sc[h]));
        v[m] = q.x; v[m + 1] = q.y;
      }
    }
#pragma unroll
    for (int m = 0; m < 4; m++) w[m * SPW + s] = tcg_round(v[m], half);
    if (s == SPW - 1) {
      const int j0 = (k / SPW) * 4 * SPW;                     // first weight of these SPW groups
#pragma unroll
      for (int p = 0; p < SPW; p++) {
        const float o[4] = {w[4 * p], w[4 * p + 1], w[4 * p + 2], w[4 * p + 3]};
        piece(j0 / 4 + p, o);
      }
    }
  }
}

// ------------------------------------------------------------------ tcgen05 plumbing
__device__ __forceinline__ void tcg_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tcg_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Shared-memory operand descriptor: K-major, 128-byte swizzle, rows 128 bytes apart, 8-row groups 1024 bytes apart.
__device__ __forceinline__ unsigned long long tcg_desc(unsigned saddr) {
  return (unsigned long long)((saddr & 0x3FFFFu) >> 4) | (1ull << 16) | ((unsigned long long)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// A in tensor memory (lane = row, a column per TF32 value), B in shared memory.
__device__ __forceinline__ void tcg_mma_tf32(unsigned tmem_d, unsigned tmem_a, unsigned long long db, unsigned idesc, unsigned accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tcg_st16(unsigned taddr, const float (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]), "f"(v[10]),
        "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15]) : "memory");
}
__device__ __forceinline__ void tcg_commit(unsigned bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tcg_ld16(unsigned taddr, float (&v)[16]) {
  unsigned r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

struct TcgGeom {
  int row_begin, row_end;     // rows of the blob this launch covers
  int cpr;                    // chunks (32 columns) per row
  int batch, npad;            // activation rows, and that padded to a multiple of 16 (the MMA's N)
  int ksplit, cps;            // column splits (= cluster size) and chunks per split
  int rounds;                 // rounds of TCG_GROUPS stages in the ring: 2, or 1 where the activations leave no room
  unsigned b_bytes;           // a stage in shared memory: a slice of X, npad x 128 bytes
  int y_stride;               // floats between consecutive activation rows' outputs
#ifdef WV_DEV_HOOKS
  int stall;                  // > 0: the first producer warp stops short of this slice, so that a wait runs out
  unsigned spin;              // limit of the waits
#endif
};
#ifdef WV_DEV_HOOKS
#define TCG_SPIN g.spin
#else
#define TCG_SPIN TMA_SPIN_LIMIT
#endif

// Tensor memory: all 512 columns, the accumulator in the first 256, then a stage's slice of A in 32 columns each.
#define TCG_TMEM 512
#define TCG_TMEM_A 256
static_assert(TCG_TMEM_A + 32 * TCG_MAX_STAGES <= TCG_TMEM, "stages of A");

__device__ __forceinline__ bool elect_one() {
  unsigned p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ float4 ld_cluster4(unsigned saddr, int rank) {
  unsigned a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}

// The column order of a CTA: its nk chunks are units of U; group q owns the chunks first .. first + n, the first groups one
// unit more where they do not divide. Round i takes one chunk of every group that has an i-th one: those are always the
// first active(i) groups.
struct TcgOrder {
  int first[TCG_GROUPS], n[TCG_GROUPS];      // in chunks
  __device__ __forceinline__ TcgOrder(int nk, int U) {
    const int nu = (nk + U - 1) / U, base = nu / TCG_GROUPS, rem = nu % TCG_GROUPS;
#pragma unroll
    for (int q = 0; q < TCG_GROUPS; q++) {
      first[q] = (base * q + min(q, rem)) * U;
      n[q] = max(0, min((base + (q < rem ? 1 : 0)) * U, nk - first[q]));
    }
  }
  __device__ __forceinline__ int active(int i) const {
    int a = 0;
#pragma unroll
    for (int q = 0; q < TCG_GROUPS; q++) a += i < n[q] ? 1 : 0;
    return a;
  }
};

// The sums of the activation rows that CTA sp of the cluster stores, over the splits' accumulators in split order: four rows of W a
// thread, the loads from all CTAs in flight together. It is bound by their latency (some 0.5 us a turn of the loop): one row of
// W at a time, 256 rows took 7.2 of the 27 us of a 4096 x 4096 launch in Q4_K. One loop for up to eight splits and one for more.
template <int N>
__device__ __forceinline__ void tcg_add_splits(const TcgGeom& g, unsigned acc_s, float* __restrict__ y, int sp, int m0) {
  for (int e = threadIdx.x; ; e += TCG_THREADS) {
    const int m = (e / (TCG_M / 4)) * g.ksplit + sp, row_l = (e & (TCG_M / 4 - 1)) * 4;
    if (m >= g.batch) break;
    float4 v[N];
#pragma unroll
    for (int u = 0; u < N; u++) if (u < g.ksplit) v[u] = ld_cluster4(acc_s + 4u * (unsigned)(m * TCG_M + row_l), u);
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int u = 0; u < N; u++) if (u < g.ksplit) { sum.x += v[u].x; sum.y += v[u].y; sum.z += v[u].z; sum.w += v[u].w; }
    float* o = y + (size_t)m * g.y_stride + m0 + row_l;
    const int left = g.row_end - m0 - row_l;
    if (left >= 4 && (reinterpret_cast<uintptr_t>(o) & 15) == 0) *reinterpret_cast<float4*>(o) = sum;
    else {
      if (left > 0) o[0] = sum.x;
      if (left > 1) o[1] = sum.y;
      if (left > 2) o[2] = sum.z;
      if (left > 3) o[3] = sum.w;
    }
  }
}

// grid (row tiles, splits), cluster (1, splits)
template <int F, bool VEC>
__global__ void __launch_bounds__(TCG_THREADS, 1)
gemm_tcgen05_kernel(const WvDevBlob b, const __grid_constant__ CUtensorMap xmap, float* __restrict__ y, const TcgGeom g, int* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char tcg_smem[];
  __shared__ __align__(8) unsigned long long s_bar[2 * TCG_MAX_STAGES + 1];
  __shared__ unsigned s_tmem;
  __shared__ int s_abort;
  __shared__ int s_made[TCG_PRODUCERS / 32];      // slices each producer warp has arrived for
  __shared__ float s_tbl[16];          // IQ4_NL's grid
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);     // one value per warp, and the compiler knows it
  const int mt = blockIdx.x, sp = blockIdx.y;
  const int m0 = g.row_begin + mt * TCG_M;
  const int kc0 = sp * g.cps, kc1 = min(g.cpr, kc0 + g.cps);
  constexpr int U = TcgUnit<F>::U;
  const int nst = max(0, kc1 - kc0);             // slices = pipeline stages to work through
  const TcgOrder order(nst, U);
  // the dynamic segment is declared 1024-byte aligned; round up all the same (the swizzle pattern is relative to 1024 bytes)
  const unsigned sbase = (smem_u32(tcg_smem) + 1023u) & ~1023u;
  // The ring: round i's slice of group q is stage (i mod rounds) * 4 + q, in its (i / rounds)-th use
  auto full_bar = [&](int s) { return smem_u32(&s_bar[s]); };
  auto empty_bar = [&](int s) { return smem_u32(&s_bar[TCG_MAX_STAGES + s]); };
  const unsigned done_bar = smem_u32(&s_bar[2 * TCG_MAX_STAGES]);
  const int rsh = g.rounds - 1;                  // log2(rounds)
  auto stage_of = [&](int i, int q) { return (i & rsh) * TCG_GROUPS + q; };

  if (tid == 0) {
    s_abort = 0;
    for (int s = 0; s < TCG_MAX_STAGES; s++) { mbar_init(full_bar(s), TCG_M / 32 + 1); mbar_init(empty_bar(s), 1); }
    mbar_init(done_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (wv_fmt_info(F).table && tid < 16) s_tbl[tid] = c_grid4nl[tid];
  if (warp == TCG_PRODUCERS / 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "n"(TCG_TMEM) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcg_fence_before();
  __syncthreads();
  tcg_fence_after();
  const unsigned tmem = __shfl_sync(0xffffffffu, *(volatile unsigned*)&s_tmem, 0);
  // The weights do not depend on the preceding kernel: the producers start at once, up to a full ring. Only then do they, and from
  // the start the warps that copy X and issue the MMAs, wait for it (X was rounded by the kernel right before this one).
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  int copied_i = 0, copied_q = 0;                // copying warp: the round it reached, and the groups it served in that round

  if (warp < TCG_PRODUCERS / 32) {
    // ------------------------------------------------------------ producers
    const int grp = warp / (TCG_M / 32);                         // owns a run of the CTA's columns
    const int row_l = tid & (TCG_M - 1);
    const int row = min(m0 + row_l, g.row_end - 1);              // rows past the end repeat the last one and are not stored
    const int mine = order.n[0] * (grp == 0) + order.n[1] * (grp == 1) + order.n[2] * (grp == 2) + order.n[3] * (grp == 3);
    const long long ch0 = (long long)row * g.cpr + kc0 + order.first[0] * (grp == 0) + order.first[1] * (grp == 1) + order.first[2] * (grp == 2) + order.first[3] * (grp == 3);
    const unsigned a_t = tmem + ((unsigned)((warp & 3) * 32) << 16) + TCG_TMEM_A;      // this warp's rows of the A slices
    // one unit ahead: its loads travel while the current unit is converted
    FragT<F> nxt[U];
    if (mine > 0) tcg_load<F, VEC>(nxt, b, ch0, mine);
    bool dead = false;
    int made = 0;
    for (int i0 = 0; i0 < mine && !dead; i0 += U) {
      FragT<F> cur[U];
#pragma unroll
      for (int u = 0; u < U; u++) cur[u] = nxt[u];
      if (i0 + U < mine) tcg_load<F, VEC>(nxt, b, ch0 + i0 + U, mine - i0 - U);
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int i = i0 + u;
        if (i >= mine || dead) break;
        // From here on a stage is free only after X has come; however long the kernels before take, that is not a time-out.
        if (i == g.rounds) asm volatile("griddepcontrol.wait;" ::: "memory");
#ifdef WV_DEV_HOOKS
        if (g.stall > 0 && warp == 0 && i + 1 >= g.stall) { dead = true; break; }
#endif
        bool bad = *(volatile int*)&s_abort != 0;
        const int s = stage_of(i, grp), use = i >> rsh;
        if (!bad && use > 0 && !mbar_wait(empty_bar(s), (use - 1) & 1, TCG_SPIN)) { atomicCAS_system(err, 0, 500 + s); *(volatile int*)&s_abort = 1; bad = true; }
        if (__any_sync(0xffffffffu, bad)) { dead = true; break; }     // the whole warp leaves together (the stores below are warp-wide)
        tcg_fence_after();                    // the MMAs that read this stage before have been waited for
        float a[16];
        tcg_convert<F>(cur[u], s_tbl, [&](int p, const float (&v)[4]) {      // pieces come in rising order
#pragma unroll
          for (int e = 0; e < 4; e++) a[4 * (p & 3) + e] = v[e];
          if ((p & 3) == 3) tcg_st16(a_t + (unsigned)(s * 32 + (p >> 2) * 16), a);
        });
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tcg_fence_before();
        __syncwarp();                                 // every lane's stores come before the one arrival
        if (lane == 0) mbar_arrive(full_bar(s));      // one arrival per warp
        made = i + 1;
      }
    }
    if (lane == 0) s_made[warp] = made;
    asm volatile("griddepcontrol.wait;" ::: "memory");
  } else if (warp == TCG_PRODUCERS / 32 + 1) {
    // ------------------------------------------------------------ X copies: a stage's slice of the rounded activations arrives
    // by a tensor-map copy with the 128-byte swizzle, i.e. already in the operand layout; rows past the batch are zero-filled
    // by the copy engine. Here and in the MMA warp the whole warp runs the loop and one elected lane issues: the operands
    // of these instructions live in uniform registers, and from a loop that only lane 0 ran, which the compiler cannot know to be
    // uniform, every stage cost some 450 cycles of issue: 64 us instead of 36 for 16 rows at 14336 x 4096 in Q4_K, whatever
    // else the kernel did.
    const bool leader = elect_one();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    bool run = true;
    for (int i = 0; i < order.n[0] && run; i++) {
      const int use = i >> rsh, na = order.active(i);
      copied_i = i; copied_q = 0;
#pragma unroll
      for (int q = 0; q < TCG_GROUPS; q++) {
        if (q >= na || !run) break;
        const int s = stage_of(i, q);
        if (use > 0 && __any_sync(0xffffffffu, !mbar_wait(empty_bar(s), (use - 1) & 1, TCG_SPIN))) { atomicCAS_system(err, 0, 530 + s); *(volatile int*)&s_abort = 1; run = false; break; }
        if (leader) {
          mbar_expect_tx(full_bar(s), g.b_bytes);
          tma_load_2d(sbase + (unsigned)s * g.b_bytes, &xmap, (kc0 + order.first[q] + i) * 32, 0, full_bar(s));
        }
        __syncwarp();
        copied_q = q + 1;
      }
    }
  } else {
    // ------------------------------------------------------------ MMA issuer
    const bool leader = elect_one();
    const unsigned idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((unsigned)(g.npad >> 3) << 17) | ((unsigned)(TCG_M >> 4) << 24);
    bool run = true;
    asm volatile("griddepcontrol.wait;" ::: "memory");           // X comes after it
    for (int i = 0; i < order.n[0] && run; i++) {
      const int na = order.active(i);
#pragma unroll
      for (int q = 0; q < TCG_GROUPS; q++) {
        if (q >= na || !run) break;
        const int s = stage_of(i, q);
        if (__any_sync(0xffffffffu, !mbar_wait(full_bar(s), (i >> rsh) & 1, TCG_SPIN))) { atomicCAS_system(err, 0, 510 + s); *(volatile int*)&s_abort = 1; run = false; break; }
        tcg_fence_after();
        if (leader) {
          const unsigned long long db = tcg_desc(sbase + (unsigned)s * g.b_bytes);
#pragma unroll
          for (int k = 0; k < 4; k++)   // 8 TF32 values = 8 columns of A, 32 bytes further along K inside X's swizzled row
            tcg_mma_tf32(tmem, tmem + (unsigned)(TCG_TMEM_A + 32 * s + 8 * k), db + (unsigned long long)(2 * k), idesc, (i > 0 || q > 0 || k > 0) ? 1u : 0u);
          tcg_commit(empty_bar(s));        // arrives when these MMAs have read the stage
        }
        __syncwarp();
      }
    }
    if (leader) tcg_commit(done_bar);      // arrives when every MMA issued above has finished
    __syncwarp();
  }

  // ---------------------------------------------------------------- epilogue: warp w reads TMEM lanes 32 (w % 4) .. + 31 (the
  // quarter a warp may access), 16 columns out of every 64. A split's accumulator waits in the ring's memory, which nothing
  // uses any more once every MMA has finished (each stage that was filled has been read by one).
  float* acc = reinterpret_cast<float*>(tcg_smem + (sbase - smem_u32(tcg_smem)));    // [batch][128]
  if (warp < TCG_PRODUCERS / 32) {
    bool ok = !*(volatile int*)&s_abort;
    if (ok && !mbar_wait(done_bar, 0, TCG_SPIN)) { atomicCAS_system(err, 0, 520); *(volatile int*)&s_abort = 1; ok = false; }
    ok = __all_sync(0xffffffffu, ok);     // tcgen05.ld is warp-wide
    tcg_fence_after();
    const int row_l = (warp & 3) * 32 + lane;
    const bool row_ok = m0 + row_l < g.row_end;
    for (int c0 = (warp >> 2) * 16; c0 < g.npad && ok; c0 += 64) {
      float v[16];
      if (nst > 0) tcg_ld16(tmem + ((unsigned)((warp & 3) * 32) << 16) + (unsigned)c0, v);
      else {
#pragma unroll
        for (int j = 0; j < 16; j++) v[j] = 0.f;
      }
      if (g.ksplit > 1) {                          // rows past the batch as well: the ring has npad * 512 bytes and more
#pragma unroll
        for (int j = 0; j < 16; j++) acc[(c0 + j) * TCG_M + row_l] = v[j];
      } else if (row_ok) {
        float* o = y + (size_t)c0 * g.y_stride + m0 + row_l;
        const int left = g.batch - c0;
        if (left >= 16) {                          // whole: no test per row
#pragma unroll
          for (int j = 0; j < 16; j++) o[(size_t)j * g.y_stride] = v[j];
        } else {
#pragma unroll
          for (int j = 0; j < 16; j++) if (j < left) o[(size_t)j * g.y_stride] = v[j];
        }
      }
    }
  }
  tcg_fence_before();
  __syncthreads();
  if (*(volatile int*)&s_abort) {      // the same for every thread: nobody raises it after the barrier
    if (warp == TCG_PRODUCERS / 32) mbar_wait(done_bar, 0, TCG_SPIN);        // the MMAs issued before the abort
    if (warp == TCG_PRODUCERS / 32 + 1) {
      // A stage's barrier completes when its copy has landed and its group's four warps have arrived: the arrivals that will
      // never come are made up for here, then the last uses of every stage are waited for (the earlier ones have been read).
#pragma unroll
      for (int q = 0; q < TCG_GROUPS; q++) {
        const int issued = min(order.n[q], copied_i + (q < copied_q ? 1 : 0));
        for (int i = max(0, issued - g.rounds); i < issued; i++) {
          const int s = stage_of(i, q);
          if (lane < TCG_M / 32 && s_made[q * (TCG_M / 32) + lane] <= i) mbar_arrive(full_bar(s));
          __syncwarp();
          mbar_wait(full_bar(s), (i >> rsh) & 1, TCG_SPIN);
        }
      }
    }
    __syncthreads();
  }
  if (warp == TCG_PRODUCERS / 32) {
    tcg_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TCG_TMEM) : "memory");
  }
  if (g.ksplit == 1) return;
  // ---------------------------------------------------------------- the cluster adds its accumulators up in split order: CTA sp
  // stores every ksplit-th activation row's 128 sums. Every thread of every CTA reaches both barriers on all paths.
  __syncwarp();
  cluster_arrive();
  cluster_wait();
  const unsigned acc_s = smem_u32(acc);
  if (g.ksplit <= 8) tcg_add_splits<8>(g, acc_s, y, sp, m0);
  else tcg_add_splits<TCG_MAX_SPLIT>(g, acc_s, y, sp, m0);
  __syncwarp();
  cluster_arrive();      // the other CTAs may still be reading this one's sums
  cluster_wait();
}

// X rounded to TF32 (round to nearest), element for element. The kernel behind it may start as soon as this one has (it waits for
// this one's end before it reads X): its set-up and its first slices of W then run beside the preceding kernel's end and this one.
// us per launch, started after this kernel's own wait / before it: Q8_0 4096 x 4096, 33 rows 13.7 / 12.4; Q5_1 1024 x 1024, 64 rows
// 8.1 / 7.3; Q8_0 14336 x 4096, 8 rows 30.4 / 27.3; at 256 rows the copy itself counts (22.1 / 21.8, with more blocks 21.4).
__global__ void __launch_bounds__(256) tcg_round_x_kernel(const float4* __restrict__ x, float4* __restrict__ xr, size_t n4) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (size_t)gridDim.x * blockDim.x) {
    const float4 v = x[i];
    xr[i] = make_float4(tcg_tf32(v.x), tcg_tf32(v.y), tcg_tf32(v.z), tcg_tf32(v.w));
  }
}

// ------------------------------------------------------------------ host side
#ifdef WV_DEV_HOOKS
static int g_tcg_stall = 0;
static unsigned g_tcg_spin = TMA_SPIN_LIMIT;
extern "C" void wv_set_tcg_stall(int slice, int spin) { g_tcg_stall = slice; g_tcg_spin = spin > 0 ? (unsigned)spin : TMA_SPIN_LIMIT; }
#endif
static PFN_cuTensorMapEncodeTiled_v12000 tcg_encode_fn() {
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = []() -> PFN_cuTensorMapEncodeTiled_v12000 {     // once, whichever thread is first
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    cudaGetLastError();
    return nullptr;
  }();
  return fn;
}

// Buffers for the rounded activations. A call's buffer may not be written by another call before its GEMM has read it, and a
// captured call's may not be freed or used by anything else while a graph holds it:
//   * a stream has a buffer of its own, which grows with what it is asked for (set-up time); calls on one stream are ordered,
//     and its lock is held over both launches, so that two threads on one stream do not interleave them;
//   * there are TCG_STREAM_BUFS of those; further streams allocate and free in stream order, call by call;
//   * a stream that is being captured gets a buffer for this capture. The graph keeps it (a user object), graphs instantiated
//     from it too, and it comes back for later captures when the last of them is gone.
#define TCG_STREAM_BUFS 16
struct TcgBuf { float* p; size_t floats; unsigned long long stream, capture; TcgBuf* next; };
struct TcgStreamBuf { std::mutex mu; unsigned long long stream = 0; float* p = nullptr; size_t floats = 0; };
struct TcgBufs {
  std::mutex mu;                                   // everything below but `returned`
  TcgStreamBuf streams[TCG_STREAM_BUFS];
  int nstreams = 0;
  std::vector<TcgBuf*> captured, idle;             // held by a graph or by a capture in progress; free for the next capture
  std::atomic<TcgBuf*> returned{nullptr};          // given back by graphs that went away: a lock-free list, as the driver calls back
  void collect() {                                 // under mu
    for (TcgBuf* b = returned.exchange(nullptr); b;) {
      TcgBuf* next = b->next;
      for (size_t i = 0; i < captured.size(); i++) if (captured[i] == b) { captured[i] = captured.back(); captured.pop_back(); break; }
      idle.push_back(b);
      b = next;
    }
  }
};
static TcgBufs& tcg_bufs() { static TcgBufs* b = new TcgBufs; return *b; }     // outlives every graph
static void CUDART_CB tcg_give_back(void* q) {
  TcgBuf* b = static_cast<TcgBuf*>(q);
  std::atomic<TcgBuf*>& head = tcg_bufs().returned;
  b->next = head.load();
  while (!head.compare_exchange_weak(b->next, b)) {}
}
// Allocation is legal for this thread whatever another one (or this one) is capturing.
struct TcgRelaxed {
  cudaStreamCaptureMode m = cudaStreamCaptureModeRelaxed;
  TcgRelaxed() { cudaThreadExchangeStreamCaptureMode(&m); }
  ~TcgRelaxed() { cudaThreadExchangeStreamCaptureMode(&m); }
};
struct TcgLease { float* p = nullptr; bool free_after = false; std::unique_lock<std::mutex> lock; };

static int tcg_lease(TcgLease& out, size_t floats, cudaStream_t st) {
  auto fail = [&]() { cudaGetLastError(); wv_set_error("batched matvec: %zu bytes for the rounded activations unavailable", floats * 4); return WV_ENOMEM; };
  TcgBufs& bufs = tcg_bufs();
  unsigned long long id = 0, cap = 0;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  cudaGraph_t graph = nullptr;
  if (cudaStreamGetCaptureInfo(st, &status, &cap, &graph) != cudaSuccess) { cudaGetLastError(); status = cudaStreamCaptureStatusNone; }
  // a stream's number (a handle may be reused); it may not be asked for in a capture, whose own number tells handles apart
  if (status != cudaStreamCaptureStatusNone || cudaStreamGetId(st, &id) != cudaSuccess) { cudaGetLastError(); id = reinterpret_cast<uintptr_t>(st); }
  if (status == cudaStreamCaptureStatusActive) {
    std::lock_guard<std::mutex> lk(bufs.mu);
    bufs.collect();
    for (TcgBuf* b : bufs.captured) if (b->capture == cap && b->stream == id && b->floats >= floats) { out.p = b->p; return WV_OK; }
    TcgBuf* b = nullptr;
    for (size_t i = 0; i < bufs.idle.size() && !b; i++) if (bufs.idle[i]->floats >= floats) { b = bufs.idle[i]; bufs.idle[i] = bufs.idle.back(); bufs.idle.pop_back(); }
    TcgRelaxed relaxed;
    if (!b) {        // those that are too small stay for now: freeing waits for the device, which a capture forbids
      float* p = nullptr;
      if (cudaMalloc(&p, floats * 4) != cudaSuccess) return fail();
      b = new TcgBuf{p, floats, 0, 0, nullptr};
    }
    b->stream = id; b->capture = cap;
    cudaUserObject_t obj = nullptr;
    if (cudaUserObjectCreate(&obj, b, tcg_give_back, 1, cudaUserObjectNoDestructorSync) != cudaSuccess) { bufs.idle.push_back(b); return fail(); }
    bufs.captured.push_back(b);
    // if the graph does not take it, the buffer goes back through the release
    if (cudaGraphRetainUserObject(graph, obj, 1, cudaGraphUserObjectMove) != cudaSuccess) { cudaUserObjectRelease(obj, 1); return fail(); }
    out.p = b->p;
    return WV_OK;
  }
  TcgStreamBuf* sb = nullptr;
  {
    std::lock_guard<std::mutex> lk(bufs.mu);
    for (int i = 0; i < bufs.nstreams && !sb; i++) if (bufs.streams[i].stream == id) sb = &bufs.streams[i];
    if (!sb && bufs.nstreams < TCG_STREAM_BUFS) { sb = &bufs.streams[bufs.nstreams++]; sb->stream = id; }
  }
  if (!sb) {
    if (cudaMallocAsync(&out.p, floats * 4, st) != cudaSuccess) return fail();
    out.free_after = true;
    return WV_OK;
  }
  out.lock = std::unique_lock<std::mutex>(sb->mu);
  if (sb->floats < floats) {
    TcgRelaxed relaxed;
    cudaStreamSynchronize(st);            // nothing else has ever used this buffer
    if (sb->p) cudaFree(sb->p);
    sb->p = nullptr; sb->floats = 0;
    {
      std::lock_guard<std::mutex> lk(bufs.mu);      // set-up time: what captures left behind goes as well
      bufs.collect();
      for (TcgBuf* q : bufs.idle) { cudaFree(q->p); delete q; }
      bufs.idle.clear();
    }
    if (cudaMalloc(&sb->p, floats * 4) != cudaSuccess) return fail();
    sb->floats = floats;
  }
  out.p = sb->p;
  return WV_OK;
}

int wv_sm_count();

// Column splits for `mtiles` row tiles of `cpr` chunks: the splits of a tile are one cluster, and how many clusters of each
// size run at once is a property of the chip (a cluster lives inside one GPC). The estimate counts waves of clusters,
// each costing its slices plus some 24 slices' worth of start-up and epilogue; equal costs go to the smaller split.
static int tcg_cps(int cpr, int ks, int unit) { return ((cpr + ks - 1) / ks + unit - 1) / unit * unit; }    // chunks per split, whole units
template <typename K>
static int tcg_splits(K kern, int dev, int mtiles, int cpr, int unit) {
  static int active[64][TCG_MAX_SPLIT + 1] = {};       // resident clusters of each size, per device (0: not asked yet)
  if (dev < 0 || dev >= 64) return 1;
  int best = 1;
  long long cost = -1;
  for (int ks = 1; ks <= TCG_MAX_SPLIT && (ks == 1 || cpr / ks >= 8); ks++) {      // at least 8 chunks (256 columns) per split
    const int cps = tcg_cps(cpr, ks, unit);
    if ((cpr + cps - 1) / cps != ks) continue;          // every split of a cluster has columns
    if (!active[dev][ks]) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(1, ks); cfg.blockDim = dim3(TCG_THREADS); cfg.dynamicSmemBytes = 200 * 1024;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = 1; at[0].val.clusterDim.y = ks; at[0].val.clusterDim.z = 1;
      cfg.attrs = at; cfg.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) { cudaGetLastError(); n = -1; }
      active[dev][ks] = n;
    }
    const int n = ks == 1 ? wv_sm_count() : active[dev][ks];
    if (n < 1) continue;
    const long long c = (long long)((mtiles + n - 1) / n) * (cps + 24);
    if (cost < 0 || c < cost) { cost = c; best = ks; }
  }
  return best;
}

template <int F, bool VEC>
static int launch_tcg(const WvDevBlob& b, const float* dx, float* dy, int batch, int rb, int re, cudaStream_t st) {
  auto kern = gemm_tcgen05_kernel<F, VEC>;
  auto enc = tcg_encode_fn();
  if (!enc) return 1;
  static unsigned attr_mask = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  if (!(attr_mask & (1u << (dev & 31)))) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 210 * 1024) != cudaSuccess) { wv_set_error("batched matvec: cannot raise the shared-memory limit"); return WV_ECUDA; }
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) { wv_set_error("batched matvec: cannot allow clusters of 16"); return WV_ECUDA; }
    attr_mask |= 1u << (dev & 31);
  }
  TcgGeom g{};
  g.row_begin = rb; g.row_end = re;
  g.cpr = b.cols >> 5;
  g.batch = batch;
  g.npad = (batch + 15) & ~15;
  g.y_stride = b.rows;
  const int rows = re - rb;
  const int mtiles = (rows + TCG_M - 1) / TCG_M;
  const int unit = VEC ? TcgUnit<F>::U : 1;
  const int ks = tcg_splits(kern, dev, mtiles, g.cpr, unit);
  g.cps = tcg_cps(g.cpr, ks, unit);
  g.ksplit = ks;
  g.b_bytes = (unsigned)g.npad * 128u;
  g.rounds = TCG_MAX_STAGES * g.b_bytes <= 200u * 1024u ? 2 : 1;      // two up to 192 rows
#ifdef WV_DEV_HOOKS
  g.stall = g_tcg_stall; g.spin = g_tcg_spin;
#endif
  const size_t smem = (size_t)g.rounds * TCG_GROUPS * g.b_bytes + 1024;
  // X rounded to TF32 once, by a small kernel in front (each of the row tiles would otherwise round it again), into a
  // buffer of the library; the main kernel fetches it through a tensor map encoded per call.
  TcgLease lease;
  if (const int rc = tcg_lease(lease, (size_t)batch * b.cols, st)) return rc;
  float* xr = lease.p;
  struct FreeAfter { TcgLease& l; cudaStream_t st; ~FreeAfter() { if (l.free_after) cudaFreeAsync(l.p, st); } } free_after{lease, st};
  CUtensorMap xmap;
  {
    cuuint64_t dims[2] = {(cuuint64_t)b.cols, (cuuint64_t)batch};
    cuuint64_t strides[1] = {(cuuint64_t)b.cols * 4};
    cuuint32_t box[2] = {32, (cuuint32_t)g.npad};
    cuuint32_t estr[2] = {1, 1};
    if (enc(&xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, xr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) return 1;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(mtiles, g.ksplit); cfg.blockDim = dim3(TCG_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = 1; at[1].val.clusterDim.y = (unsigned)g.ksplit; at[1].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = g.ksplit > 1 ? 2 : 1;
  int* err = wv_tma_err_ptr();
  {
    const size_t n4 = (size_t)batch * b.cols / 4;
    cudaLaunchConfig_t rc_ = {};
    int blocks = (int)((n4 + 255) / 256);
    // Two blocks fit beside a CTA of the kernel before. Up to three turns of those they are all resident early; beyond, the copy is
    // what counts (100 rows of 6400 columns 16.0 us a call with 296 blocks, 16.2 with all; 256 of 4096 21.8 and 21.6).
    const int beside = 2 * wv_sm_count(), all = 8 * wv_sm_count();
    if (blocks > 3 * beside) { if (blocks > all) blocks = all; }
    else if (blocks > beside) blocks = beside;
    rc_.gridDim = dim3(blocks); rc_.blockDim = dim3(256); rc_.stream = st;
    rc_.attrs = at; rc_.numAttrs = 1;
    if (cudaLaunchKernelEx(&rc_, tcg_round_x_kernel, reinterpret_cast<const float4*>(dx), reinterpret_cast<float4*>(xr), n4) != cudaSuccess) {
      wv_set_error("batched matvec (rounding) launch: %s", cudaGetErrorString(cudaGetLastError())); return WV_ECUDA;
    }
  }
  if (cudaLaunchKernelEx(&cfg, kern, b, xmap, dy, g, err) != cudaSuccess) { wv_set_error("batched matvec launch: %s", cudaGetErrorString(cudaGetLastError())); return WV_ECUDA; }
  return WV_OK;
}

// Batched y[m][rows] = x[m][cols] W^T for 2 <= batch <= 256 activation rows. Returns 1 for what this kernel does not
// take (FormatNone, rows that do not start on chunk boundaries, unaligned x), so that the caller runs the rows one by one.
int wv_launch_gemm_tcgen05(const WvDevBlob& b, const float* dx, float* dy, int batch, int row_begin, int row_end, cudaStream_t st) {
  if (batch < 2 || batch > 256 || !b.fast || b.format == WV_NONE || (b.cols & 31) || row_end <= row_begin) return 1;
  if ((reinterpret_cast<uintptr_t>(dx) & 15) || !wv_tma_err_ptr()) return 1;
  switch (b.format) {
#define WV_F(f) case f: return (b.cols >> 5) % TcgUnit<f>::U ? launch_tcg<f, false>(b, dx, dy, batch, row_begin, row_end, st) : launch_tcg<f, true>(b, dx, dy, batch, row_begin, row_end, st);
  WV_F(WV_Q8_0) WV_F(WV_Q4_0) WV_F(WV_Q4_1) WV_F(WV_Q5_0) WV_F(WV_Q5_1)
  WV_F(WV_Q2_K) WV_F(WV_Q3_K) WV_F(WV_Q4_K) WV_F(WV_Q5_K) WV_F(WV_Q6_K)
  WV_F(WV_IQ1_S) WV_F(WV_IQ2_XXS) WV_F(WV_IQ2_XS) WV_F(WV_IQ3_XXS) WV_F(WV_IQ3_S) WV_F(WV_IQ4_NL) WV_F(WV_IQ4_XS)
  WV_F(WV_TERNARY) WV_F(WV_BINARY) WV_F(WV_AFFINE)
#undef WV_F
  }
  return 1;
}
