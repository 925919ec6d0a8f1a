// GEMV for matrices whose rows do not start on a chunk (or vector) boundary: cols % 32 != 0 for the packed formats,
// cols % 8 != 0 for FormatNone. Exact dequantised weights, float32 products and sums.
//
// A packed plane is a flat stream, so row r covers the chunks start/32 .. (start + cols - 1)/32 with start = r * cols, and
// its first and last chunk may belong to two rows. A lane takes whole chunks with the vector loads of the aligned kernels
// (chunk boundaries are aligned whatever the row length) and meets them with x shifted by start % 32. x sits in shared
// memory with 32 zeros in front of it and behind it, which is what the neighbours' weights in a shared chunk are
// multiplied with, and with one word of padding every 32, so that lanes 32 floats apart hit 32 different banks wherever
// the row starts. A row whose sum comes out infinite or NaN is summed again over its own weights, one by one: zero times a
// neighbour's infinity is no zero, and codes summed before they are scaled overflow for activations whose products with the
// weights do not.
//
// Bound: launch and memory latency for one activation row (a 2730 x 1022 matrix is 1 - 3 MB), instructions from some eight rows
// on (33 rows of Q4_0 at 9001 x 100: 78 % of the issue slots). A weight of a lane's
// chunk costs some 14 instructions there, all included; the weight-by-weight kernel this replaces spent some 60 (64-bit index arithmetic, bit extraction from global memory
// and, for the k-quants, two divisions). Measured back to back on a stream, Q8_0, Q4_0, Q4_K and IQ3_S at 2730 x 1022
// and 1022 x 2730: 271 us before for the eight launches, 41.6 us now (3.7 to 6.1 us a launch, of which about 4 us is the
// host's own cost of a call).
#include "wv_dequant.cuh"
#include "wv_gemv_common.cuh"
#include "wv_tma_common.cuh"

#define RAG_THREADS 256
#define RAG_MAX_COLS 49152    // x in shared memory: 33/32 * 4 bytes per column, 203 KB; wider rows read x from global memory

// Slot of logical position i (column + 32) in the padded shared copy of x.
__device__ __forceinline__ int rag_slot(int i) { return i + (i >> 5); }

// x of one batch row into its padded slots, zeros around it.
__device__ __forceinline__ void rag_stage_x(float* xs, const float* __restrict__ xb, int cols) {
  for (int i = threadIdx.x; i < cols; i += RAG_THREADS) xs[rag_slot(i + 32)] = xb[i];
  if (threadIdx.x < 32) xs[threadIdx.x] = 0.f;
  else if (threadIdx.x < 96) xs[rag_slot(cols + threadIdx.x)] = 0.f;    // positions cols + 32 .. cols + 95
}

// Dot of one chunk with the 32 activations xv(j).
template <int F, typename X>
__device__ __forceinline__ float rag_chunk(const FragT<F>& f, X xv, const float* tbl) {
  constexpr WvFmtInfo fi = wv_fmt_info(F);
  constexpr int BL = fi.bits_lo, BH = fi.bits_hi, SPW = 8 / BL;
  constexpr unsigned MASK = 0x01010101u * ((1u << BL) - 1u);
  constexpr unsigned MASKH = BH ? (0x01010101u * ((1u << BH) - 1u)) << BL : 0u;
  float sc[2], mn[2] = {0.f, 0.f};
  if constexpr (fi.kind == WK_KQUANT) {
    const float d = __uint_as_float(f.pr[0]);
    sc[0] = __fdiv_rn(__fmul_rn(d, (float)(unsigned char)(f.pr[2])), 255.0f);
    sc[1] = __fdiv_rn(__fmul_rn(d, (float)(unsigned char)(f.pr[2] >> 8)), 255.0f);
    if (sc[0] == 0.f) sc[0] = __fdiv_rn(d, 255.0f);
    if (sc[1] == 0.f) sc[1] = __fdiv_rn(d, 255.0f);
    if constexpr (fi.has_min) {
      const float dm = __uint_as_float(f.pr[1]);
      mn[0] = __fdiv_rn(__fmul_rn(dm, (float)(signed char)(f.pr[2] >> 16)), 127.0f);
      mn[1] = __fdiv_rn(__fmul_rn(dm, (float)(signed char)(f.pr[2] >> 24)), 127.0f);
    }
  } else {
    sc[0] = sc[1] = __uint_as_float(f.pr[0]);
    if constexpr (fi.pgroup == 16) sc[1] = __uint_as_float(f.pr[1]);
    if constexpr (fi.has_min) mn[0] = mn[1] = __uint_as_float(f.pr[1]);
  }
  const float magic = 8388608.0f + (float)fi.mid;   // code under the exponent of 2^23, minus this: (code - mid) exactly
  float acc[4] = {0.f, 0.f, 0.f, 0.f}, tot = 0.f;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int w = k / SPW, s = k % SPW, h = (BL == 1 || k < 4) ? 0 : 1;
    unsigned bytes = (f.lo[w] >> (BL * s)) & MASK;
    if constexpr (BH > 0) {
      const int hw = (k * BH) >> 3, sh = (k * BH) & 7;
      unsigned hv = f.hi[hw];
      hv = sh >= BL ? (hv >> (sh - BL)) : (hv << (BL - sh));
      bytes |= hv & MASKH;
    }
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const float xj = xv(WvLane<BL>::j_of(k, m));
      float q;
      if constexpr (fi.table) q = tbl[((bytes >> (8 * m)) & 0xffu) * 32];
      else q = __uint_as_float(__byte_perm(bytes, 0x4B000000u, 0x7650 + m)) - magic;
      if constexpr (fi.half_mid) q -= 0.5f;
      if constexpr (fi.sign) q = q + q - 1.0f;
      if constexpr (fi.has_min) acc[m] = fmaf(fmaf(q, sc[h], mn[h]), xj, acc[m]);
      else acc[m] = fmaf(q, xj, acc[m]);
    }
    if constexpr (!fi.has_min) {
      if (k == 3 || k == 7) {     // the scale of each half once
        tot = fmaf((acc[0] + acc[1]) + (acc[2] + acc[3]), sc[h], tot);
        acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
      }
    }
  }
  if constexpr (fi.has_min) tot = (acc[0] + acc[1]) + (acc[2] + acc[3]);
  return tot;
}

// The products of every step-th weight of a row, from `first` on.
template <int F>
__device__ __forceinline__ float rag_row_own(const WvDevBlob& b, const float* __restrict__ xb, int row, int first, int step) {
  constexpr WvFmtInfo fi = wv_fmt_info(F);
  float acc = 0.f;
  for (int c = first; c < b.cols; c += step) acc = fmaf(wv_dequant(b, fi, (long long)row * b.cols + c), __ldg(xb + c), acc);
  return acc;
}

// XS: x in shared memory (otherwise read from global memory, with the zeros around it by comparison). LPR: lanes per row; a
// warp works on 32 / LPR rows.
template <int F, bool XS, int LPR>
__global__ void __launch_bounds__(RAG_THREADS, 4) gemv_ragged_chunk_kernel(const WvDevBlob b, const float* __restrict__ x, float* __restrict__ y,
                                                                        int row_begin, int row_end) {
  constexpr WvFmtInfo fi = wv_fmt_info(F);
  constexpr int RPW = 32 / LPR;
  extern __shared__ float rag_xs[];
  __shared__ float s_tbl[fi.table ? 512 : 1];
  const int lane = threadIdx.x & 31, sl = lane % LPR, gw = (int)((blockIdx.x * RAG_THREADS + threadIdx.x) >> 5), nw = (int)(gridDim.x * RAG_THREADS) >> 5;
  const float* xb = x + (size_t)blockIdx.y * b.cols;
  float* yb = y + (size_t)blockIdx.y * b.rows;
  const int first = row_begin + gw * RPW;                 // the warp's first rows
  int row = first + lane / LPR;
  long long start = (long long)row * b.cols;
  FragT<F> cur;
  // the first chunk's weights do not depend on the preceding kernel
  if (row < row_end && sl < (int)(((start & 31) + b.cols + 31) >> 5)) load_frag<F>(cur, b, (start >> 5) + sl);
  if constexpr (fi.table) for (int i = threadIdx.x; i < 512; i += RAG_THREADS) s_tbl[i] = c_grid4nl[i >> 5];
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if constexpr (XS) rag_stage_x(rag_xs, xb, b.cols);
  __syncthreads();
  bool odd = false;
  for (int r0 = first; r0 < row_end; r0 += nw * RPW) {    // the same for the whole warp
    row = r0 + lane / LPR;
    start = (long long)row * b.cols;
    const int s = (int)(start & 31), nch = row < row_end ? (s + b.cols + 31) >> 5 : 0;
    const long long ch0 = start >> 5;
    if (r0 != first && sl < nch) load_frag<F>(cur, b, ch0 + sl);
    float acc = 0.f;
    for (int c = sl; c < nch; c += LPR) {
      FragT<F> nxt = cur;
      if (c + LPR < nch) load_frag<F>(nxt, b, ch0 + c + LPR);
      const int i0 = 32 + c * 32 - s;      // padded position of the chunk's first weight; columns i0 - 32 ...
      if constexpr (XS) {
        const float* p0 = rag_xs + rag_slot(i0);
        const int thr = s ? s : 32;         // from here on the next 32-float group: one word of padding further
        acc += rag_chunk<F>(cur, [&](int j) { return (j < thr ? p0 : p0 + 1)[j]; }, s_tbl + lane);
      } else {
        acc += rag_chunk<F>(cur, [&](int j) { const int col = i0 - 32 + j; return (col >= 0 && col < b.cols) ? __ldg(xb + col) : 0.f; },
                            s_tbl + lane);
      }
      cur = nxt;
    }
#pragma unroll
    for (int o = LPR / 2; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (sl == 0 && row < row_end) yb[row] = acc;
    odd = odd || !(fabsf(acc) <= 3.402823466e38f);          // a row past the end has a sum of zero
  }
  // Behind the loop, which so keeps its registers: the rows whose sum was not finite, read back.
  if (!__any_sync(0xffffffffu, odd)) return;
  __syncwarp();
  for (int r0 = first; r0 < row_end; r0 += nw * RPW) {
    row = r0 + lane / LPR;
    const bool redo = row < row_end && !(fabsf(yb[row]) <= 3.402823466e38f);
    float acc = redo ? rag_row_own<F>(b, xb, row, sl, LPR) : 0.f;
#pragma unroll
    for (int o = LPR / 2; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (redo && sl == 0) yb[row] = acc;
  }
}

// FormatNone: a lane takes aligned 16-byte vectors of the flat element array; elements outside the row are skipped
// (they are the neighbours' and may be anything). Vectors inside the row, all but the first and the last, need no test.
template <int DT, bool XS, int LPR>
__global__ void __launch_bounds__(RAG_THREADS) gemv_ragged_plain_kernel(const WvDevBlob b, const float* __restrict__ x, float* __restrict__ y,
                                                                        int row_begin, int row_end) {
  constexpr int EPV = DT == WV_DT_F32 ? 4 : 8, RPW = 32 / LPR;
  extern __shared__ float rag_xs[];
  const int lane = threadIdx.x & 31, sl = lane % LPR, gw = (int)((blockIdx.x * RAG_THREADS + threadIdx.x) >> 5), nw = (int)(gridDim.x * RAG_THREADS) >> 5;
  const float* xb = x + (size_t)blockIdx.y * b.cols;
  float* yb = y + (size_t)blockIdx.y * b.rows;
  const uint4* wp = reinterpret_cast<const uint4*>(b.lo);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if constexpr (XS) rag_stage_x(rag_xs, xb, b.cols);
  __syncthreads();
  for (int r0 = row_begin + gw * RPW; r0 < row_end; r0 += nw * RPW) {
    const int row = r0 + lane / LPR;
    const long long start = (long long)row * b.cols;
    const int s = (int)(start % EPV), nv = row < row_end ? (s + b.cols + EPV - 1) / EPV : 0;
    const uint4* rp = wp + start / EPV;
    float sum[4] = {0.f, 0.f, 0.f, 0.f};      // short chains of additions
    for (int v0 = sl; v0 < nv; v0 += 4 * LPR) {
      uint4 q[4];
#pragma unroll
      for (int u = 0; u < 4; u++) q[u] = v0 + LPR * u < nv ? __ldg(rp + v0 + LPR * u) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int u = 0; u < 4; u++) {
        if (XS && v0 + LPR * u >= nv) break;      // (from global memory the loads of x are better off without it)
        const int c0 = (v0 + LPR * u) * EPV - s;
        const unsigned ws[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
        auto weight = [&](int e) {
          if constexpr (DT == WV_DT_F32) return __uint_as_float(ws[e]);
          else {
            const unsigned hw = (e & 1) ? ws[e >> 1] >> 16 : ws[e >> 1] & 0xffffu;
            if constexpr (DT == WV_DT_BF16) return __uint_as_float(hw << 16);
            else return __half2float(__ushort_as_half((unsigned short)hw));
          }
        };
        if (XS && c0 >= 0 && c0 + EPV <= b.cols) {
          const float* p0 = rag_xs + rag_slot(c0 + 32);
          const int thr = 32 - (c0 & 31);     // from here on the next 32-float group: one word of padding further
#pragma unroll
          for (int e = 0; e < EPV; e++) sum[u] = fmaf(weight(e), (e < thr ? p0 : p0 + 1)[e], sum[u]);
        } else {
#pragma unroll
          for (int e = 0; e < EPV; e++) {
            const int col = c0 + e;
            if (col >= 0 && col < b.cols) sum[u] = fmaf(weight(e), XS ? rag_xs[rag_slot(col + 32)] : __ldg(xb + col), sum[u]);
          }
        }
      }
    }
    float acc = (sum[0] + sum[1]) + (sum[2] + sum[3]);
#pragma unroll
    for (int o = LPR / 2; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (sl == 0 && row < row_end) yb[row] = acc;
  }
}

// ------------------------------------------------------------------ host side
template <typename K>
static int rag_go(K kern, bool xs, int lpr, const WvDevBlob& b, const float* dx, float* dy, int batch, int rb, int re, cudaStream_t st, unsigned& attr_mask) {
  const size_t smem = xs ? ((size_t)b.cols + 96 + (b.cols + 96) / 32 + 1) * 4 : 0;
  int dev = 0;
  cudaGetDevice(&dev);
  // Whatever the size: the limit without the attribute is 48 KB for static and dynamic memory together, and IQ4_NL's
  // table makes 2 KB of the static kind.
  if (xs && !(attr_mask & (1u << (dev & 31)))) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024) != cudaSuccess) { wv_set_error("gemv (ragged): cannot raise the shared-memory limit"); return WV_ECUDA; }
    attr_mask |= 1u << (dev & 31);
  }
  // `lpr` lanes per row until the SMs hold no more CTAs side by side; then rows in turn, so that x is staged at most that often
  int per_sm = smem ? (int)((220 * 1024) / smem) : 8;
  per_sm = per_sm < 1 ? 1 : (per_sm > 8 ? 8 : per_sm);
  const int rpc = RAG_THREADS / lpr;
  int grid = (re - rb + rpc - 1) / rpc;
  if (grid > per_sm * wv_sm_count()) grid = per_sm * wv_sm_count();
  const cudaError_t e = launch_pdl(kern, dim3(grid, batch), dim3(RAG_THREADS), smem, st, b, dx, dy, rb, re);
  if (e != cudaSuccess) { wv_set_error("gemv (ragged) launch: %s", cudaGetErrorString(e)); return WV_ECUDA; }
  return WV_OK;
}
// Lanes per row. A row has `units` chunks or vectors at most: lanes beyond that idle (27 of 32 at 100 columns), and the last of a
// row's steps fills its lanes only in part (33 chunks take two steps of 32 lanes or five of eight). So as few lanes as leave
// 16 warps for every SM: with fewer warps the latency of a row's steps shows. A warp per row, whatever the shape, took 149 us
// for 33 rows of Q8_0 at 9001 x 46 and 60 us for 33 of bf16 at 2730 x 1022; the weight-by-weight kernel takes 70 and 49, this
// 34 and 45.
static int rag_lanes(int units, int rows, int batch) {
  int lpr = units <= 8 ? 8 : (units <= 16 ? 16 : 32);
  while (lpr > 8 && units <= 6 * lpr && (long long)rows * batch * (lpr / 2) / 32 >= 16 * wv_sm_count()) lpr /= 2;
  return lpr;
}
template <int F>
static int rag_format(const WvDevBlob& b, const float* dx, float* dy, int batch, int rb, int re, cudaStream_t st) {
  static unsigned attr[4] = {0, 0, 0, 0};
  if (b.cols > RAG_MAX_COLS) return rag_go(gemv_ragged_chunk_kernel<F, false, 32>, false, 32, b, dx, dy, batch, rb, re, st, attr[3]);
  switch (rag_lanes((b.cols + 62) >> 5, re - rb, batch)) {
  case 8: return rag_go(gemv_ragged_chunk_kernel<F, true, 8>, true, 8, b, dx, dy, batch, rb, re, st, attr[0]);
  case 16: return rag_go(gemv_ragged_chunk_kernel<F, true, 16>, true, 16, b, dx, dy, batch, rb, re, st, attr[1]);
  }
  return rag_go(gemv_ragged_chunk_kernel<F, true, 32>, true, 32, b, dx, dy, batch, rb, re, st, attr[2]);
}
template <int DT>
static int rag_plain(const WvDevBlob& b, const float* dx, float* dy, int batch, int rb, int re, cudaStream_t st) {
  static unsigned attr[4] = {0, 0, 0, 0};
  constexpr int EPV = DT == WV_DT_F32 ? 4 : 8;
  if (b.cols > RAG_MAX_COLS) return rag_go(gemv_ragged_plain_kernel<DT, false, 32>, false, 32, b, dx, dy, batch, rb, re, st, attr[3]);
  switch (rag_lanes((b.cols + 2 * EPV - 2) / EPV, re - rb, batch)) {
  case 8: return rag_go(gemv_ragged_plain_kernel<DT, true, 8>, true, 8, b, dx, dy, batch, rb, re, st, attr[0]);
  case 16: return rag_go(gemv_ragged_plain_kernel<DT, true, 16>, true, 16, b, dx, dy, batch, rb, re, st, attr[1]);
  }
  return rag_go(gemv_ragged_plain_kernel<DT, true, 32>, true, 32, b, dx, dy, batch, rb, re, st, attr[2]);
}
int wv_launch_gemv_flat(const WvDevBlob& b, const float* dx, float* dy, int batch, int row_begin, int row_end, cudaStream_t st);   // wv_layout.cu

int wv_launch_gemv_ragged(const WvDevBlob& b, const float* dx, float* dy, int batch, int row_begin, int row_end, cudaStream_t st) {
  if (row_end <= row_begin || batch <= 0) return WV_OK;
  if (batch > 32768) {      // the batch is the grid's second dimension
    const int rc = wv_launch_gemv_ragged(b, dx, dy, 32768, row_begin, row_end, st);
    return rc ? rc : wv_launch_gemv_ragged(b, dx + (size_t)32768 * b.cols, dy + (size_t)32768 * b.rows, batch - 32768, row_begin, row_end, st);
  }
  switch (b.format) {
#define WV_F(f) case f: return rag_format<f>(b, dx, dy, batch, row_begin, row_end, st);
  WV_F(WV_Q8_0) WV_F(WV_Q4_0) WV_F(WV_Q4_1) WV_F(WV_Q5_0) WV_F(WV_Q5_1)
  WV_F(WV_Q2_K) WV_F(WV_Q3_K) WV_F(WV_Q4_K) WV_F(WV_Q5_K) WV_F(WV_Q6_K)
  WV_F(WV_IQ1_S) WV_F(WV_IQ2_XXS) WV_F(WV_IQ2_XS) WV_F(WV_IQ3_XXS) WV_F(WV_IQ3_S) WV_F(WV_IQ4_NL) WV_F(WV_IQ4_XS)
  WV_F(WV_TERNARY)
#undef WV_F
  case WV_BINARY: if (b.group == 32) return rag_format<WV_BINARY>(b, dx, dy, batch, row_begin, row_end, st); break;
  case WV_NONE:
    if (b.dtype == WV_DT_F32) return rag_plain<WV_DT_F32>(b, dx, dy, batch, row_begin, row_end, st);
    if (b.dtype == WV_DT_F16) return rag_plain<WV_DT_F16>(b, dx, dy, batch, row_begin, row_end, st);
    return rag_plain<WV_DT_BF16>(b, dx, dy, batch, row_begin, row_end, st);
  }
  // affine groups that are no multiple of a chunk (8, 16, 24 ... weights): several parameter pairs per chunk, weight by weight
  return wv_launch_gemv_flat(b, dx, dy, batch, row_begin, row_end, st);
}
