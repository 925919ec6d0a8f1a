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
// Bound: launch and memory latency (a 2730 x 1022 matrix is 1 - 3 MB). A weight costs about 7 instructions; the
// weight-by-weight kernel this replaces spent some 60 (64-bit index arithmetic, bit extraction from global memory
// and, for the k-quants, two divisions). Measured back to back on a stream, Q8_0, Q4_0, Q4_K and IQ3_S at 2730 x 1022
// and 1022 x 2730: 271 us before for the eight launches, 43 us now (5.4 us a launch, of which about 4 us is the
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

// XS: x in shared memory (otherwise read from global memory, with the zeros around it by comparison).
template <int F, bool XS>
__global__ void __launch_bounds__(RAG_THREADS) gemv_ragged_chunk_kernel(const WvDevBlob b, const float* __restrict__ x, float* __restrict__ y,
                                                                        int row_begin, int row_end) {
  constexpr WvFmtInfo fi = wv_fmt_info(F);
  extern __shared__ float rag_xs[];
  __shared__ float s_tbl[fi.table ? 512 : 1];
  const int lane = threadIdx.x & 31, gw = (int)((blockIdx.x * RAG_THREADS + threadIdx.x) >> 5), nw = (int)(gridDim.x * RAG_THREADS) >> 5;
  const float* xb = x + (size_t)blockIdx.y * b.cols;
  float* yb = y + (size_t)blockIdx.y * b.rows;
  int row = row_begin + gw;
  long long start = (long long)row * b.cols;
  FragT<F> cur;
  // the first chunk's weights do not depend on the preceding kernel
  if (row < row_end && lane < (int)(((start & 31) + b.cols + 31) >> 5)) load_frag<F>(cur, b, (start >> 5) + lane);
  if constexpr (fi.table) for (int i = threadIdx.x; i < 512; i += RAG_THREADS) s_tbl[i] = c_grid4nl[i >> 5];
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if constexpr (XS) rag_stage_x(rag_xs, xb, b.cols);
  __syncthreads();
  bool odd = false;
  for (; row < row_end; row += nw) {
    start = (long long)row * b.cols;
    const int s = (int)(start & 31), nch = (s + b.cols + 31) >> 5;
    const long long ch0 = start >> 5;
    if (row != row_begin + gw && lane < nch) load_frag<F>(cur, b, ch0 + lane);
    float acc = 0.f;
    for (int c = lane; c < nch; c += 32) {
      FragT<F> nxt = cur;
      if (c + 32 < nch) load_frag<F>(nxt, b, ch0 + c + 32);
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
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) yb[row] = acc;
    odd = odd || !(fabsf(acc) <= 3.402823466e38f);
  }
  // Behind the loop, which so keeps its registers: the rows whose sum was not finite, read back.
  if (!odd) return;
  __syncwarp();
  for (row = row_begin + gw; row < row_end; row += nw) {
    if (fabsf(yb[row]) <= 3.402823466e38f) continue;
    float acc = rag_row_own<F>(b, xb, row, lane, 32);
#pragma unroll
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) yb[row] = acc;
  }
}

// FormatNone: a lane takes aligned 16-byte vectors of the flat element array; elements outside the row are skipped
// (they are the neighbours' and may be anything).
template <int DT, bool XS>
__global__ void __launch_bounds__(RAG_THREADS) gemv_ragged_plain_kernel(const WvDevBlob b, const float* __restrict__ x, float* __restrict__ y,
                                                                        int row_begin, int row_end) {
  constexpr int EPV = DT == WV_DT_F32 ? 4 : 8;
  extern __shared__ float rag_xs[];
  const int lane = threadIdx.x & 31, gw = (int)((blockIdx.x * RAG_THREADS + threadIdx.x) >> 5), nw = (int)(gridDim.x * RAG_THREADS) >> 5;
  const float* xb = x + (size_t)blockIdx.y * b.cols;
  float* yb = y + (size_t)blockIdx.y * b.rows;
  const uint4* wp = reinterpret_cast<const uint4*>(b.lo);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if constexpr (XS) rag_stage_x(rag_xs, xb, b.cols);
  __syncthreads();
  for (int row = row_begin + gw; row < row_end; row += nw) {
    const long long start = (long long)row * b.cols;
    const int s = (int)(start % EPV), nv = (s + b.cols + EPV - 1) / EPV;
    const uint4* rp = wp + start / EPV;
    float acc = 0.f;
    for (int v0 = lane; v0 < nv; v0 += 128) {
      uint4 q[4];
#pragma unroll
      for (int u = 0; u < 4; u++) q[u] = v0 + 32 * u < nv ? __ldg(rp + v0 + 32 * u) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int c0 = (v0 + 32 * u) * EPV - s;
        const unsigned ws[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
#pragma unroll
        for (int e = 0; e < EPV; e++) {
          float w;
          if constexpr (DT == WV_DT_F32) w = __uint_as_float(ws[e]);
          else {
            const unsigned hw = (e & 1) ? ws[e >> 1] >> 16 : ws[e >> 1] & 0xffffu;
            if constexpr (DT == WV_DT_BF16) w = __uint_as_float(hw << 16);
            else w = __half2float(__ushort_as_half((unsigned short)hw));
          }
          const int col = c0 + e;
          if (col >= 0 && col < b.cols) acc = fmaf(w, XS ? rag_xs[rag_slot(col + 32)] : __ldg(xb + col), acc);
        }
      }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) yb[row] = acc;
  }
}

// ------------------------------------------------------------------ host side
template <typename K>
static int rag_go(K kern, bool xs, const WvDevBlob& b, const float* dx, float* dy, int batch, int rb, int re, cudaStream_t st, unsigned& attr_mask) {
  const size_t smem = xs ? ((size_t)b.cols + 96 + (b.cols + 96) / 32 + 1) * 4 : 0;
  int dev = 0;
  cudaGetDevice(&dev);
  // Whatever the size: the limit without the attribute is 48 KB for static and dynamic memory together, and IQ4_NL's
  // table makes 2 KB of the static kind.
  if (xs && !(attr_mask & (1u << (dev & 31)))) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024) != cudaSuccess) { wv_set_error("gemv (ragged): cannot raise the shared-memory limit"); return WV_ECUDA; }
    attr_mask |= 1u << (dev & 31);
  }
  // a warp per row until the SMs hold no more CTAs side by side; then rows in turn, so that x is staged at most that often
  int per_sm = smem ? (int)((220 * 1024) / smem) : 8;
  per_sm = per_sm < 1 ? 1 : (per_sm > 8 ? 8 : per_sm);
  int grid = (re - rb + RAG_THREADS / 32 - 1) / (RAG_THREADS / 32);
  if (grid > per_sm * wv_sm_count()) grid = per_sm * wv_sm_count();
  const cudaError_t e = launch_pdl(kern, dim3(grid, batch), dim3(RAG_THREADS), smem, st, b, dx, dy, rb, re);
  if (e != cudaSuccess) { wv_set_error("gemv (ragged) launch: %s", cudaGetErrorString(e)); return WV_ECUDA; }
  return WV_OK;
}
template <int F>
static int rag_format(const WvDevBlob& b, const float* dx, float* dy, int batch, int rb, int re, cudaStream_t st) {
  static unsigned attr[2] = {0, 0};
  if (b.cols <= RAG_MAX_COLS) return rag_go(gemv_ragged_chunk_kernel<F, true>, true, b, dx, dy, batch, rb, re, st, attr[0]);
  return rag_go(gemv_ragged_chunk_kernel<F, false>, false, b, dx, dy, batch, rb, re, st, attr[1]);
}
template <int DT>
static int rag_plain(const WvDevBlob& b, const float* dx, float* dy, int batch, int rb, int re, cudaStream_t st) {
  static unsigned attr[2] = {0, 0};
  if (b.cols <= RAG_MAX_COLS) return rag_go(gemv_ragged_plain_kernel<DT, true>, true, b, dx, dy, batch, rb, re, st, attr[0]);
  return rag_go(gemv_ragged_plain_kernel<DT, false>, false, b, dx, dy, batch, rb, re, st, attr[1]);
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
