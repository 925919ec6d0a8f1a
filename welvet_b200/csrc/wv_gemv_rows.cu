// GEMV over a few activation rows (2 .. 5 of a batch): y[m] = W x[m] with W streamed and unpacked once for up to four rows.
// The arithmetic is that of the one-row kernels (exact integer dots over block-fixed-point activations, float32 scales);
// the layout of the work is gemv_tma_kernel's: a CTA per SM owns a band of rows that a producer thread streams through a
// shared-memory ring, a consumer lane owns one 32-column chunk.
//
// The one-row kernel keeps its chunk's activation record in registers (24 words); four of them do not fit beside the weight
// fragments. Here the records of all rows sit in shared memory ([row][word][chunk], 16 bytes per lane: no bank conflicts)
// and a tile's ROWS_RT fragments are unpacked once and met with one row's record after the other.
//
// Bound: launch overhead at the sizes that stay in L2 (a 4096 x 4096 matrix in Q4_K streams in 1.7 us, and a launch costs
// 4 us of start-up whatever it moves, which row-by-row launches pay per row); HBM for larger matrices.
// Four rows against Q4_K: 10.7 us at 4096 x 4096 (18.8 row by row), 22.3 at 14336 x 4096 (34.8), 16.1 at 4096 x 6144 (23.1),
// 5.6 at 1024 x 1024 (12.6); two rows at 4096 x 4096: 7.2 (9.8). A further row costs 1.6 us at 4096 x 4096: its dp2a.
#include "wv_gemv_tma.cuh"

int wv_act_width();   // wv_gemv_tma.cu: development switch (3 = always take 24-bit records)

struct RowsGeom {
  int cpr, nwc, nrg, tr, nstage;    // as in TmaGeom
  unsigned stage_bytes, off[5], rb[5];
  int rows_base, rows_rem;          // CTA b owns rows_base (+1 if b < rows_rem) consecutive rows
  int m_base, m_rem;                // grid row q takes m_base (+1 if q < m_rem) activation rows
  int wide;                         // development switch: 24-bit records whatever x looks like
  unsigned rec_off, red_off, bar_off;
};
#define ROWS_NB 4                        // activation rows a CTA takes at most
#define ROWS_RT 4                        // weight rows per row group and tile
#define ROWS_REC 9u                 // uint4 per chunk and activation row: 24 words, scale and sums, six start values (24-bit record)

// The total of every row of a tile over the warp, for four row sums per lane: the lane whose index is the row's slot
// (4 t + row) mod 32 gets it in `keep`.
__device__ __forceinline__ void keep_rows(const float (&v)[4], int t, int lane, float& keep) {
  const bool b4 = lane & 16, b3 = lane & 8;
  float a0 = b4 ? v[2] : v[0], a1 = b4 ? v[3] : v[1];
  a0 += __shfl_xor_sync(0xffffffffu, b4 ? v[0] : v[2], 16);
  a1 += __shfl_xor_sync(0xffffffffu, b4 ? v[1] : v[3], 16);
  float tot = b3 ? a1 : a0;
  tot += __shfl_xor_sync(0xffffffffu, b3 ? a0 : a1, 8);
#pragma unroll
  for (int o = 4; o; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
  tot = __shfl_sync(0xffffffffu, tot, (lane & 3) * 8);      // row (lane & 3) lives in lanes [8 (lane & 3), + 8)
  if ((lane >> 2) == (t & 7)) keep = tot;
}

__device__ __forceinline__ uint4 f4u(const float4 v) { return make_uint4(__float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z), __float_as_uint(v.w)); }
__device__ __forceinline__ float4 u4f(const uint4 v) { return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w)); }

// A chunk-row with everything taken out of it that does not depend on the activations: the codes one per byte, and the
// scales and offsets as floats. Its share of an output row is sf * (S0 val0 + S1 val1) + M0 SX0 + M1 SX1, where val and SX are
// a half's sums of (code - mid) X and of x (halves taken together for the formats with one parameter group per chunk).
template <int F> struct RowsPrep {
  static constexpr WvFmtInfo fi = wv_fmt_info(F);
  static constexpr int NH = QCfg<F>::NH;
  static constexpr bool OFFSET = fi.has_min || fi.sign || fi.half_mid;
  unsigned by[8];
  float S[NH], M[OFFSET ? NH : 1];
};
template <int F>
__device__ __forceinline__ void rows_prepare(RowsPrep<F>& p, const FragT<F>& f) {
  constexpr WvFmtInfo fi = wv_fmt_info(F);
  constexpr int BL = fi.bits_lo, BH = fi.bits_hi, SPW = 8 / BL, NH = QCfg<F>::NH;
  constexpr unsigned MASK = 0x01010101u * ((1u << BL) - 1u);
  constexpr unsigned MASKH = BH ? (0x01010101u * ((1u << BH) - 1u)) << BL : 0u;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    unsigned bytes = (f.lo[k / SPW] >> (BL * (k % SPW))) & MASK;
    if constexpr (BH > 0) {
      const int hw = (k * BH) >> 3, hs = (k * BH) & 7;
      unsigned hv = f.hi[hw];
      hv = hs >= BL ? (hv >> (hs - BL)) : (hv << (BL - hs));
      bytes |= hv & MASKH;
    }
    p.by[k] = bytes;
  }
  if constexpr (fi.kind == WK_KQUANT) {       // scale bytes were remapped 0 -> 1 at upload (quant/kquant.go:180-182)
    const float d = __uint_as_float(f.pr[0]) * (1.0f / 255.0f);
    p.S[0] = d * (float)(unsigned char)(f.pr[2]); p.S[1] = d * (float)(unsigned char)(f.pr[2] >> 8);
    if constexpr (fi.has_min) {
      const float dm = __uint_as_float(f.pr[1]) * (1.0f / 127.0f);
      p.M[0] = dm * (float)(signed char)(f.pr[2] >> 16); p.M[1] = dm * (float)(signed char)(f.pr[2] >> 24);
    }
  } else {
#pragma unroll
    for (int h = 0; h < NH; h++) {
      p.S[h] = __uint_as_float(f.pr[h]);
      if constexpr (fi.half_mid) p.M[h] = -((float)fi.mid + 0.5f) * p.S[h];
    }
    if constexpr (fi.has_min) p.M[0] = __uint_as_float(f.pr[1]);
    if constexpr (fi.sign) { p.M[0] = -p.S[0]; p.S[0] = p.S[0] + p.S[0]; }
  }
}

// The ROWS_RT chunk-rows' shares for one activation row, whose record r holds L times 8 words, then {sf, sums}, then start values:
// three byte limbs (L = 3), or 16-bit activations two to a word, whose sums need one accumulator (L = 2).
template <int F, int L>
__device__ __forceinline__ void rows_dot(const RowsPrep<F> (&p)[ROWS_RT], const uint4* r, int XS, float (&v)[ROWS_RT]) {
  constexpr WvFmtInfo fi = wv_fmt_info(F);
  constexpr bool HALVES = QCfg<F>::HALVES;
  constexpr int NH = QCfg<F>::NH;
  constexpr int NA = L == 3 ? 3 : 1;
  int I[ROWS_RT][NA][NH];
  if constexpr (QCfg<F>::INT_MID) {           // -mid * sum of the limb, per half
    const uint4 i0 = r[(2 * L + 1) * XS];
    int iv[6] = {(int)i0.x, (int)i0.y, (int)i0.z, (int)i0.w, 0, 0};
    if constexpr (L == 3) { const uint4 i1 = r[(2 * L + 2) * XS]; iv[4] = (int)i1.x; iv[5] = (int)i1.y; }
#pragma unroll
    for (int rr = 0; rr < ROWS_RT; rr++)
#pragma unroll
      for (int l = 0; l < NA; l++)
#pragma unroll
        for (int h = 0; h < NH; h++) I[rr][l][h] = iv[l * 2 + h];
  } else {
#pragma unroll
    for (int rr = 0; rr < ROWS_RT; rr++)
#pragma unroll
      for (int l = 0; l < NA; l++)
#pragma unroll
        for (int h = 0; h < NH; h++) I[rr][l][h] = 0;
  }
#pragma unroll
  for (int l = 0; l < L; l++)
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const uint4 u = r[(2 * l + q) * XS];
      const unsigned xw[4] = {u.x, u.y, u.z, u.w};
      const int h = HALVES ? q : 0;
#pragma unroll
      for (int k = 0; k < 4; k++)
#pragma unroll
        for (int rr = 0; rr < ROWS_RT; rr++)
          if constexpr (L == 2) I[rr][0][h] = l == 0 ? dp2a_lo(xw[k], p[rr].by[4 * q + k], I[rr][0][h]) : dp2a_hi(xw[k], p[rr].by[4 * q + k], I[rr][0][h]);
          else I[rr][l][h] = l == L - 1 ? dp4a_us(p[rr].by[4 * q + k], xw[k], I[rr][l][h]) : dp4a_uu(p[rr].by[4 * q + k], xw[k], I[rr][l][h]);
    }
  const float4 mt = u4f(r[2 * L * XS]);       // {sf, sf SX, sf SX(first 16), sf SX(second 16)}
#pragma unroll
  for (int rr = 0; rr < ROWS_RT; rr++) {
    float t = 0.f;
#pragma unroll
    for (int h = 0; h < NH; h++) {
      float val;
      // 16-bit activations, and three limbs with codes of at most four bits, stay below 2^31
      if constexpr (L == 2) val = (float)I[rr][0][h];
      else if constexpr (fi.bits_lo + fi.bits_hi <= 4) val = (float)(I[rr][0][h] + (I[rr][1][h] << 8) + (I[rr][2][h] << 16));
      else val = fmaf(65536.0f, (float)I[rr][2][h], (float)(I[rr][0][h] + (I[rr][1][h] << 8)));
      t = fmaf(p[rr].S[h], val, t);
    }
    float e = 0.f;
    if constexpr (RowsPrep<F>::OFFSET) {
      if constexpr (HALVES) e = fmaf(p[rr].M[1], mt.w, p[rr].M[0] * mt.z);
      else e = p[rr].M[0] * mt.y;
    }
    v[rr] = fmaf(mt.x, t, e);
  }
}

template <int F>
__global__ void __launch_bounds__(TMA_THREADS, 1)
gemv_rows_kernel(const WvDevBlob b, const float* __restrict__ x, float* __restrict__ y, int row_begin, const RowsGeom g, int* __restrict__ err) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ int s_abort;
  __shared__ unsigned s_xissued;                                     // consumer warps that have issued their first loads of x
  __shared__ unsigned char s_wide[ROWS_NB][TMA_CONSUMER_WARPS];           // 24-bit records for this row and 1024 columns
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int bid = blockIdx.x;
  const int band = g.rows_base + (bid < g.rows_rem ? 1 : 0);
  const int c_lo = row_begin + bid * g.rows_base + min(bid, g.rows_rem);
  const int ntiles = (band + g.tr - 1) / g.tr;
  const int mb = (int)blockIdx.y * g.m_base + min((int)blockIdx.y, g.m_rem);       // first activation row
  const int nb = g.m_base + ((int)blockIdx.y < g.m_rem ? 1 : 0);
  const unsigned sbase = smem_u32(smem), bar0 = smem_u32(smem + g.bar_off);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (g.nstage + s); };
  const int nactive = g.nrg * g.nwc;

  if (tid == 0) {
    s_abort = 0;
    s_xissued = 0;
    for (int s = 0; s < g.nstage; s++) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), nactive); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  if (warp == TMA_CONSUMER_WARPS) {
    // ------------------------------------------------------------ producer (one thread)
    if (lane == 0) {
      const void* src[5] = {b.lo, b.hi, b.p0, b.p1, b.km};
      int s = 0, issued = 0;
      unsigned par = 1;
      for (int t = 0; t < ntiles; t++) {
        // after the first tile, hold further copies until the loads of x are on their way: they must not queue behind a
        // full ring of weight requests
        if (t == 1) for (unsigned i = 0; i < TMA_SPIN_LIMIT; i++) if (*(volatile unsigned*)&s_xissued >= (unsigned)nactive) break;
        if (t >= g.nstage) {
          if (*(volatile int*)&s_abort) break;
          if (t == g.nstage) asm volatile("griddepcontrol.wait;" ::: "memory");      // the consumers do: no time-out however long it takes
          if (!mbar_wait(empty_bar(s), par)) { atomicCAS_system(err, 0, 600 + s); *(volatile int*)&s_abort = 1; break; }
        }
        const int r0 = t * g.tr, nr = min(g.tr, band - r0);
        unsigned bytes = 0;
#pragma unroll
        for (int i = 0; i < 5; i++) bytes += g.rb[i] * nr;
        mbar_expect_tx(full_bar(s), bytes);
#pragma unroll
        for (int i = 0; i < 5; i++)
          if (g.rb[i]) bulk_g2s(sbase + (unsigned)s * g.stage_bytes + g.off[i], (const unsigned char*)src[i] + (size_t)(c_lo + r0) * g.rb[i], g.rb[i] * nr, full_bar(s));
        issued++;
        if (++s == g.nstage) { s = 0; par ^= 1u; }
      }
      // every copy issued must have landed before the CTA gives its shared memory back
      for (int t = max(0, issued - g.nstage); t < issued; t++)
        if (!mbar_wait(full_bar(t % g.nstage), (t / g.nstage) & 1)) { atomicCAS_system(err, 0, 620 + t % g.nstage); break; }
    }
    return;
  }

  // -------------------------------------------------------------- consumers
  const int wc = warp % g.nwc, rg = warp / g.nwc;
  if (rg >= g.nrg) return;
  const int c = wc * 32 + lane, XS = g.nwc * 32;
  const bool live = c < g.cpr;
  uint4* rec = reinterpret_cast<uint4*>(smem + g.rec_off);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  // Activation records, once per launch: the row groups of a column warp share the rows out among them. A lane loads its
  // chunk of x straight into registers; lanes past the last chunk write zero records and contribute exactly 0.
  bool first = true;
  for (int m = rg; m < nb; m += g.nrg) {
    const float* xc = x + (size_t)(mb + m) * b.cols + (size_t)(live ? c : 0) * 32;
    float xv[32];
    if ((reinterpret_cast<uintptr_t>(x) & 15) == 0) {      // rows are 128-byte multiples
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(xc) + q);
        xv[4 * q] = v.x; xv[4 * q + 1] = v.y; xv[4 * q + 2] = v.z; xv[4 * q + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; j++) xv[j] = __ldg(xc + j);
    }
    if (first && lane == 0) asm volatile("red.relaxed.cta.shared::cta.add.u32 [%0], 1;" ::"r"(smem_u32(&s_xissued)) : "memory");
    first = false;
    if (!live) {
#pragma unroll
      for (int j = 0; j < 32; j++) xv[j] = 0.f;
    }
    uint4* r = rec + (size_t)m * ROWS_REC * XS + c;
    // 16-bit or 24-bit records for these 1024 columns, by the rule of gemv_tma_kernel
    float am[4] = {0.f, 0.f, 0.f, 0.f}, as[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 32; j++) { const float a = fabsf(xv[j]); am[j & 3] = fmaxf(am[j & 3], a); as[j & 3] += a; }
    const float amax = fmaxf(fmaxf(am[0], am[1]), fmaxf(am[2], am[3]));
    float ta = amax, ts = (as[0] + as[1]) + (as[2] + as[3]);
#pragma unroll
    for (int o = 16; o; o >>= 1) { ta += __shfl_xor_sync(0xffffffffu, ta, o); ts += __shfl_xor_sync(0xffffffffu, ts, o); }
    // NaN compares false and an infinity fails the second test (ta and ts are both infinite then): non-finite input takes 24 bits
    const bool wide = !(ta <= 0.25f * ts && ts <= 3.4e38f) || g.wide;
    if (lane == 0) s_wide[m][wc] = wide;
    if (wide) {
      XQRegs q;
      quantize_chunk<F>(q, xv);
#pragma unroll
      for (int l = 0; l < 3; l++) {
        r[(2 * l) * XS] = make_uint4(q.xw[8 * l], q.xw[8 * l + 1], q.xw[8 * l + 2], q.xw[8 * l + 3]);
        r[(2 * l + 1) * XS] = make_uint4(q.xw[8 * l + 4], q.xw[8 * l + 5], q.xw[8 * l + 6], q.xw[8 * l + 7]);
      }
      r[6 * XS] = f4u(q.mt);
      r[7 * XS] = make_uint4((unsigned)q.iv[0], (unsigned)q.iv[1], (unsigned)q.iv[2], (unsigned)q.iv[3]);
      r[8 * XS] = make_uint4((unsigned)q.iv[4], (unsigned)q.iv[5], 0u, 0u);
    } else {
      XQRegs2 q;
      quantize_chunk2<F>(q, xv, amax);
#pragma unroll
      for (int l = 0; l < 2; l++) {
        r[(2 * l) * XS] = make_uint4(q.xw[8 * l], q.xw[8 * l + 1], q.xw[8 * l + 2], q.xw[8 * l + 3]);
        r[(2 * l + 1) * XS] = make_uint4(q.xw[8 * l + 4], q.xw[8 * l + 5], q.xw[8 * l + 6], q.xw[8 * l + 7]);
      }
      r[4 * XS] = f4u(q.mt);
      r[5 * XS] = make_uint4((unsigned)q.iv[0], (unsigned)q.iv[1], 0u, 0u);
    }
  }
  // row groups without an activation row of their own load none
  if (first && lane == 0) asm volatile("red.relaxed.cta.shared::cta.add.u32 [%0], 1;" ::"r"(smem_u32(&s_xissued)) : "memory");
  asm volatile("bar.sync 14, %0;" ::"r"(nactive * 32) : "memory");

  // -------------------------------------------------------------- main loop
  float* red = reinterpret_cast<float*>(smem + g.red_off);           // [2][nrg][nwc][ROWS_NB][32]
  LaneOff lo0 = lane_offsets<F>(g, rg * ROWS_RT, live ? c : g.cpr - 1, b.group);
  const uint4* myrec = rec + c;
  float keep[ROWS_NB];
#pragma unroll
  for (int m = 0; m < ROWS_NB; m++) keep[m] = 0.f;
  int fs = 0, par = 0;
  unsigned fpar = 0;
  bool dead = false;
  auto flush = [&](int slot0) {
    float* base = red + (size_t)(par * g.nrg + rg) * g.nwc * ROWS_NB * 32;
#pragma unroll
    for (int m = 0; m < ROWS_NB; m++) { base[(wc * ROWS_NB + m) * 32 + lane] = keep[m]; keep[m] = 0.f; }
    asm volatile("bar.sync %0, %1;" ::"r"(rg + 1), "r"(g.nwc * 32) : "memory");
    const int n = slot0 + lane, ri = (n / ROWS_RT) * g.tr + rg * ROWS_RT + (n % ROWS_RT);       // row of the band this lane's slot stands for
    for (int m = wc; m < nb; m += g.nwc) {
      float sum = 0.f;
      for (int q = 0; q < g.nwc; q++) sum += base[(q * ROWS_NB + m) * 32 + lane];
      if (n < ntiles * ROWS_RT && ri < band) y[(size_t)(mb + m) * b.rows + c_lo + ri] = sum;
    }
    par ^= 1;      // the other half next: this one may still be read while the warps run ahead to the next flush
  };
  for (int t = 0; t < ntiles; t++) {
    if (!dead && *(volatile int*)&s_abort) dead = true;
    if (!dead && !mbar_wait(full_bar(fs), fpar)) { atomicCAS_system(err, 0, 610 + fs); *(volatile int*)&s_abort = 1; dead = true; }
    FragT<F> fr[ROWS_RT];
    LaneOff a = lo0;
    const unsigned st = sbase + (unsigned)fs * g.stage_bytes;
    a.lo += st; a.hi += st; a.p0 += st; a.p1 += st; a.km += st;
#pragma unroll
    for (int rr = 0; rr < ROWS_RT; rr++) {
      load_frag_smem<F>(fr[rr], a);          // rows past the band read stale ring data and are never stored
      a.lo += g.rb[0]; a.hi += g.rb[1]; a.p0 += g.rb[2]; a.p1 += g.rb[3]; a.km += g.rb[4];
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(empty_bar(fs));
    if (++fs == g.nstage) { fs = 0; fpar ^= 1u; }
    RowsPrep<F> prep[ROWS_RT];
#pragma unroll
    for (int rr = 0; rr < ROWS_RT; rr++) rows_prepare<F>(prep[rr], fr[rr]);
#pragma unroll
    for (int m = 0; m < ROWS_NB; m++) {
      if (m < nb) {
        const uint4* r = myrec + (size_t)m * ROWS_REC * XS;
        float v[ROWS_RT];
        if (s_wide[m][wc]) rows_dot<F, 3>(prep, r, XS, v);
        else rows_dot<F, 2>(prep, r, XS, v);
        keep_rows(v, t, lane, keep[m]);
      }
    }
    if (((t * ROWS_RT + ROWS_RT - 1) & 31) == 31) flush(t * ROWS_RT + ROWS_RT - 32);
  }
  if ((ntiles * ROWS_RT) & 31) flush((ntiles * ROWS_RT) & ~31);
}

// ------------------------------------------------------------------ host side
template <int F>
static int launch_rows(const WvDevBlob& b, const float* dx, float* dy, int batch, int rb_, int re, cudaStream_t st) {
  RowsGeom g{};
  if (!plane_row_bytes(b, g.rb)) return 1;
  g.cpr = b.cols >> 5;
  g.nwc = (g.cpr + 31) / 32;
  if (g.nwc > TMA_CONSUMER_WARPS) return 1;
  // So few rows of W that row by row the CTAs of all activation rows run side by side, or nearly: that takes 3.6 - 4.4 us as long
  // as there is an SM for each and 6.9 - 7.9 us up to two for each, while this kernel spreads the rows of W alone over the chip
  // and takes 2.4 - 3.2 us and some 1.5 us for each of a CTA's activation rows (Q4_K, four rows: 24 x 4096 4.1 against 8.2 us,
  // 64 x 6144 7.5 against 9.1; three rows, 64 x 4096: 7.6 against 6.9; two rows, 128 x 9216: 7.5 against 6.9).
  const int ny = (batch + ROWS_NB - 1) / ROWS_NB, nb = (batch + ny - 1) / ny;
  const long long side = (long long)(re - rb_) * batch, sms = wv_sm_count();
  if (side <= sms || (side <= 2 * sms && nb >= 3 && nb * g.nwc >= 16)) return 1;
  g.nrg = TMA_CONSUMER_WARPS / g.nwc;
  // One row group (more than eight column warps) leaves up to seven warps idle: two activation rows are faster one by one in the
  // formats that unpack cheaply (no hi plane; 4096 x 9216: IQ1_S 14.2 against 14.7 us, Ternary 14.3 against 15.2; IQ3_S, with one,
  // 17.4 against 16.5), three are not (Ternary 21.2 against 19.6), nor are two rows of a matrix of few rows (128 x 9216, Ternary: 7.1
  // against 6.9) or of one that is streamed from HBM and would go to the tensor-core kernel (40960 x 9216, Ternary: 199 against 101).
  if (g.nrg == 1 && batch == 2 && wv_fmt_info(F).bits_hi == 0 && re - rb_ >= 8 * sms && !wv_beyond_l2(b)) return 1;
  if (g.nrg > TMA_MAX_ROW_GROUPS) g.nrg = TMA_MAX_ROW_GROUPS;
  g.tr = g.nrg * ROWS_RT;
  g.wide = wv_act_width() == 3;
  unsigned off = 0;
  for (int i = 0; i < 5; i++) { g.off[i] = off; off = align128(off + g.rb[i] * g.tr); }
  g.stage_bytes = off;
  const unsigned rec = (unsigned)ROWS_NB * ROWS_REC * g.nwc * 32 * 16, red = align128(2u * g.nrg * g.nwc * ROWS_NB * 32 * 4);
  const unsigned fixed = rec + red + 2 * TMA_MAX_STAGES * 8;
  const unsigned avail = 225u * 1024u;  // 227 KB per CTA minus static shared memory and slack
  if (fixed + 2 * g.stage_bytes > avail) return 1;
  int ns = (int)((avail - fixed) / g.stage_bytes);
  if (ns > TMA_MAX_STAGES) ns = TMA_MAX_STAGES;
  g.nstage = ns;
  g.rec_off = g.stage_bytes * ns;
  g.red_off = g.rec_off + rec;
  g.bar_off = g.red_off + red;
  const size_t smem = g.bar_off + 2 * TMA_MAX_STAGES * 8;
  int grid = wv_sm_count();
  if (grid > re - rb_) grid = re - rb_;
  g.rows_base = (re - rb_) / grid;
  g.rows_rem = (re - rb_) % grid;
  g.m_base = batch / ny;
  g.m_rem = batch % ny;
  auto kern = gemv_rows_kernel<F>;
  static unsigned attr_mask = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  if (!(attr_mask & (1u << (dev & 31)))) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024) != cudaSuccess) { wv_set_error("gemv (rows): cannot raise the shared-memory limit"); return WV_ECUDA; }
    attr_mask |= 1u << (dev & 31);
  }
  const cudaError_t e = launch_pdl(kern, dim3(grid, ny), dim3(TMA_THREADS), smem, st, b, dx, dy, rb_, g, wv_tma_err_ptr());
  if (e != cudaSuccess) { wv_set_error("gemv (rows) launch: %s", cudaGetErrorString(e)); return WV_ECUDA; }
  return WV_OK;
}

// Returns 1 for what this kernel does not take: FormatNone, IQ4_NL (float table arithmetic), planes whose rows are no 16-byte
// multiples, few rows of W (launch_rows), the formats and widths below, and rows so wide that four rows' records leave the ring
// no room for two tiles: beyond 6144 columns in Q5_1 and Q6_K, 6656 in Q5_K, 7168 in the other 4-bit formats and IQ3_S, 7680 in Q3_K,
// 8192 in Q2_K, 9216 to 11264 in the other 1- and 2-bit formats. A tile halves beyond 8192 columns (one row group instead of two),
// so that all but Q5_1 and Q6_K are taken again from there to 8704 - 9216 (Q2_K 10240).
int wv_launch_gemv_rows(const WvDevBlob& b, const float* dx, float* dy, int batch, int row_begin, int row_end, cudaStream_t st) {
  if (batch < 2 || !b.fast || b.format == WV_NONE || row_end <= row_begin || !wv_tma_err_ptr()) return 1;
  // What runs as 24-bit records on the tensor pipe row by row (gemv_mma_kernel: Q8_0, and the formats with one parameter
  // group per chunk up to 4096 columns) stays there whatever the shape, since 16-bit records would be less precise. 24-bit ones would
  // make this kernel the slower one where it was tried (Q8_0 at 4096 x 4096, four rows: 17.9 against 13.6 us).
  const WvFmtInfo fi = wv_fmt_info(b.format);
  if (b.format == WV_Q8_0 || (b.cols <= 4096 && b.format != WV_IQ3_XXS && fi.kind != WK_KQUANT && fi.pgroup != 16)) return 1;
  switch (b.format) {
#define WV_F(f) case f: return launch_rows<f>(b, dx, dy, batch, row_begin, row_end, st);
  WV_F(WV_Q4_0) WV_F(WV_Q4_1) WV_F(WV_Q5_0) WV_F(WV_Q5_1)
  WV_F(WV_Q2_K) WV_F(WV_Q3_K) WV_F(WV_Q4_K) WV_F(WV_Q5_K) WV_F(WV_Q6_K)
  WV_F(WV_IQ1_S) WV_F(WV_IQ2_XXS) WV_F(WV_IQ2_XS) WV_F(WV_IQ3_XXS) WV_F(WV_IQ3_S) WV_F(WV_IQ4_XS)
  WV_F(WV_TERNARY) WV_F(WV_BINARY) WV_F(WV_AFFINE)
#undef WV_F
  }
  return 1;
}
