// The FP64 FFT pass (same Stockham pass as fft_pass.cuh) computed in 64-bit
// fixed point with a shared exponent per sub-transform.
//
// What bounds it: FP64 arithmetic runs at 1.73 operations per clock and SM on
// this GPU, so the pass on the FP64 pipe kept that pipe 75-78 % busy at 681 /
// 843 us for the two radix-2^11 passes of two 2^22-point rows.  The same
// butterflies on the integer pipes (fix64.cuh) take 127 / 157 us, bound by the
// multiply pipe and by its latency at 16 resident warps (43 % of the issue
// slots).
//
// A thread holds 16 points (128 registers).  With 8 points, 64 registers and
// twice the resident warps the passes took 137 / 168 us: one more stage costs
// more instructions than the warps give back.  The first stage takes its
// doubles from global memory, the sub-transform's largest exponent is found (one
// shared-memory maximum per row), and every value becomes a 62-bit integer
// relative to it.  Before each radix-16 stage the row's actual largest value
// gives the number of spare leading bits ("lift"), so an impulse or a tone keeps
// as many bits as noise does; the stage's twiddle factors carry 1/16, its worst
// growth, which keeps |value| below 2^62.5 throughout.  Outputs are rounded to
// double once.  Against an extended-precision transform (relative L2, noise) one pass is
// 5e-17 off and two passes of 2^16, 2^20 and 2^22 points 6.8e-17, in FP64 arithmetic
// 2.8e-16, 3.1e-16 and 3.4e-16.
//
// Small samples beside large ones: a double keeps its 53 bits wherever it lies, a
// fixed-point value those above 2^-58 .. 2^-62 of the row's largest.  Where samples share
// one scale that is no loss (FP64 additions round at 2^-53 of the larger value), but
// where large samples cancel exactly it is, ones and 1e-20-sized samples in turn for
// instance.  So each thread adds up how many binades beyond FX_NEAR its 16 samples lie below
// the row's largest; above FX_FAR in any thread the CTA takes fx_fallback.  A
// single sample may lie 2^-36 below, four 2^-21, sixteen 2^-17 on average (41 bits and
// more are kept).  The chance halves with every unit: on normally distributed samples
// (real or complex) it is below 1e-10 a thread; two tones that beat slowly in a row
// hold many small samples in a thread (FX_NEAR 8, FX_FAR 28 sent 2 or 3 CTAs of a
// noiseless n = 2^24, k = 4000 run to the other form, 350 -> 390 us).  The check costs 2.5 % of the
// passes (the two of two 2^22-point rows 285 -> 293 us).
//
// Sub-transforms whose largest sample lies outside 2^-800 .. 2^970 (2^+-250 in a
// pass that writes |X|^2; infinities, NaN and subnormals among them) are
// transformed in FP64 by fx_fallback, as every pass was; the filter design asks for
// that form throughout (PassArgs::direct), whose results are the same bits as the former
// FP64 pass's (two 2^22-point rows: 1.61 ms, that pass 1.69).
#pragma once
#include "fft_pass.cuh"
#include "fix64.cuh"

namespace gsfft {

namespace {

// shared-memory index of element i: conflict-free for 16-byte accesses at the
// strides of the stages (i and E i for eight consecutive i); additive over
// disjoint bit fields, so constant parts become immediate offsets
__host__ __device__ constexpr int padx(int i) { return i + (i >> 3) + (i >> 6); }
// row pitch: rows 8/G elements apart (mod 8) when a warp interleaves G rows
template <int LOGR> __host__ __device__ constexpr int fx_pitch() {
  return ((padx(1 << LOGR) + 7) & ~7) + imax(1, 8 / g_of<double>(LOGR));
}
template <int LOGR> __host__ __device__ constexpr int fx_smem() {
  return imax(g_of<double>(LOGR) * fx_pitch<LOGR>() * 16, data_smem_of<double>(LOGR));
}
// threads per CTA, 16 points each, and the resident CTAs per SM that the register
// budget is sized for (128 registers a thread)
template <int LOGR> __host__ __device__ constexpr int fx_nt() { return (1 << LOGR) * g_of<double>(LOGR) / 16; }
template <int LOGR> __host__ __device__ constexpr int fx_minb() { return imax(1, 512 / fx_nt<LOGR>()); }
// log2 of the first stage's radix (the others are radix 16)
template <int LOGR> __host__ __device__ constexpr int fx_loge0() { return LOGR % 4 == 0 ? 4 : LOGR % 4; }
constexpr int FX_MAXST = 3;  // radix-16 stages after the first, at most

// exponent fields of the largest sample that the fixed-point form takes: every
// non-zero output (at least 2^-960) and every |X|^2 is then a normal double
constexpr int FX_NEAR = 16, FX_FAR = 20;  // binades
constexpr int FX_EXP_MIN = 223, FX_EXP_MAX = 1993, FX_EXP_MIN_SQ = 1023 - 250, FX_EXP_MAX_SQ = 1023 + 250;

__device__ __forceinline__ long long fx_lift(long long v, unsigned m) {
  return (long long)((unsigned long long)v * m);
}

// bits that bound a value: the highest set bit p of the OR over values gives
// |value| < 2^(p + 32)
__device__ __forceinline__ unsigned fx_bits(unsigned m, fx::C64 v) {
  const unsigned a = (unsigned)fx::top(v.x), b = (unsigned)fx::top(v.y);
  return m | (a ^ (a + a)) | (b ^ (b + b));
}
// spare leading bits of a row: |value| 2^lift stays below 2^62
__device__ __forceinline__ int fx_spare(unsigned m) { return min(max(__clz((int)m) - 1, 0), 30); }

// v 2^s (s within +-960) rounded to double
__device__ __forceinline__ double fx_double(long long v, int s) {
  const double d = __ll2double_rn(v);
  const int h = __double2hiint(d);
  return __hiloint2double(h ? h + (s << 20) : 0, __double2loint(d));
}

// |X|^2 2^(2s): squares of the operands shifted to 62 bits, one rounding
__device__ __forceinline__ double fx_square(fx::C64 X, int s) {
  const unsigned long long m =
      (unsigned long long)(X.x ^ (X.x >> 63)) | (unsigned long long)(X.y ^ (X.y >> 63));
  const int n = max(__clzll((long long)m) - 2, 0);
  const long long x = (long long)((unsigned long long)X.x << n), y = (long long)((unsigned long long)X.y << n);
  const int xh = fx::limb_hi(x), xl = fx::limb_lo(x), yh = fx::limb_hi(y), yl = fx::limb_lo(y);
  const long long t = fx::madw(yh, yl, fx::madw(xh, xl, 1LL << 30)) >> 31;
  const long long q = fx::madw(yh, yh, fx::madw(xh, xh, t));
  return fx_double(q, 64 - 2 * n + 2 * s);
}

// Reduces m over the lanes of a warp that share a row, then into dst[row]:
// rows fastest over lanes (gfast: row = lane % G) or TPF consecutive threads a
// row.
template <int G, int TPF, bool MAX>
__device__ __forceinline__ void fx_row_reduce(unsigned m, bool gfast, unsigned *dst, int g) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    if (gfast ? o >= G : o < TPF) {
      const unsigned y = __shfl_xor_sync(0xffffffffu, m, o);
      m = MAX ? max(m, y) : (m | y);
    }
  }
  const bool leader = gfast ? lane < G : (lane & (imin(TPF, 32) - 1)) == 0;
  if (leader) {
    if (MAX) atomicMax(&dst[g], m);
    else atomicOr(&dst[g], m);
  }
}

// address of point m of a first pass's input: in order, or in pairs of rows of 2^lognc
// columns (FftIo::in_lognc)
__device__ __forceinline__ long long row_pairs(long long m, int lognc) {
  if (lognc < 0) return m;
  const long long row = m >> lognc, c = m & ((1LL << lognc) - 1);
  return ((row & ~1LL) << lognc) + 2 * c + (row & 1);
}

// The pass in FP64, for sub-transforms with values outside the fixed-point
// range: load with inter-pass twiddles, runtime-stride stages, store.
template <int LOGR>
__device__ __noinline__ void fx_fallback(const PassArgs &a, double2 *sm) {
  constexpr int R = 1 << LOGR, G = g_of<double>(LOGR), NT = fx_nt<LOGR>(), RP = rowpitch<double>(LOGR);
  constexpr int ITER = R * G / NT;
  const double2 *in = reinterpret_cast<const double2 *>(a.in), *gx = reinterpret_cast<const double2 *>(a.gx);
  const double2 *thi = reinterpret_cast<const double2 *>(a.tw_hi), *tlo = reinterpret_cast<const double2 *>(a.tw_lo);
  const int logS = a.logN - LOGR, logNs = a.logNs;
  const long long Smask = (1LL << logS) - 1, Nsmask = (1LL << logNs) - 1, u0 = (long long)blockIdx.x * G;
  const bool gf_in = (1LL << logS) >= G, gf_out = (1LL << logNs) >= G;
  __syncthreads();
#pragma unroll 1
  for (int q = 0; q < ITER; q++) {
    const int lt = threadIdx.x + q * NT;
    const int g = gf_in ? lt % G : lt / R, r = gf_in ? lt / G : lt % R;
    const long long u = u0 + g, b = u >> logS, j = u & Smask,
                    m = a.tile_in ? (j & ~1LL) * R + 2 * r + (j & 1) : row_pairs(j + ((long long)r << logS), a.lognc);
    double2 v = make_double2(0.0, 0.0);
    if (u < a.total) v = gx ? gx[a.goffs[b] + m * a.gstride] : in[b * a.bstride + m];
    if (a.inverse) v.y = -v.y;
    if (logNs > 0) {
      const long long mm = (j & Nsmask) * r;
      v = cmul(v, cmul(thi[mm >> a.tw_h], tlo[mm & ((1 << a.tw_h) - 1)]));
    }
    sm[g * RP + padded(r)] = v;
  }
  __syncthreads();
  rt_cta_fft<double2, LOGR, G, NT>(sm, reinterpret_cast<const double2 *>(a.twR));
  // The thread's largest sample of row rb goes out once, and once per warp where its
  // rows are the same: an atomic per sample made these passes up to 3.4 times
  // the former FP64 pass (n = 2^24, W = 2^23 plan of a signal scaled by 2^-300: 11.7 ms).
  unsigned long long *const rm = a.samples ? reinterpret_cast<unsigned long long *>(a.row_max) : nullptr;
  double tmax = 0.0;
  long long rb = -1;
#pragma unroll 1
  for (int q = 0; q < ITER; q++) {
    const int lt = threadIdx.x + q * NT;
    const int g = gf_out ? lt % G : lt / R, k = gf_out ? lt / G : lt % R;
    const long long u = u0 + g, b = u >> logS, j = u & Smask;
    if (u >= a.total) continue;
    const long long d =
        b * a.bstride + (a.tile_out ? ((long long)(k & ~1) << logS) + 2 * j + (k & 1)
                                    : ((j >> logNs) << (logNs + LOGR)) + (j & Nsmask) + ((long long)k << logNs));
    double2 v = sm[g * RP + padded(k)];
    if (a.inverse) v.y = -v.y;
    if (a.write_complex) reinterpret_cast<double2 *>(a.out)[d] = v;
    if (a.samples) {
      const double sv = sq_sum(v);
      reinterpret_cast<double *>(a.samples)[d] = sv;
      if (rm) {
        if (b != rb) {
          if (rb >= 0) atomicMax(rm + rb, key_bits(tmax));
          rb = b;
          tmax = 0.0;
        }
        tmax = sv > tmax ? sv : tmax;
      }
    }
  }
  if (rm) {
    const long long b0 = __shfl_sync(0xffffffffu, rb, 0);
    if (__all_sync(0xffffffffu, rb == b0 && rb >= 0)) row_max_update(rm, b0, tmax);
    else if (rb >= 0) atomicMax(rm + rb, key_bits(tmax));
  }
}

// entries of the stage tables before the radix-16 stage after Ns = 2^LOGNS
template <int LOGR> __host__ __device__ constexpr int fx_stage_offset(int logns) {
  int off = 0;
  for (int l = fx_loge0<LOGR>(); l < logns; l += 4) off += 16 << l;
  return off;
}

// One radix-16 butterfly of the stage after Ns = 2^LOGNS: lift, twiddles (rows
// [e][k] of the stage's table, which carry 1/16), DFT.
template <int LOGR, int LOGNS>
__device__ __forceinline__ void fx_radix16(fx::C64 (&v)[16], const longlong2 *rp, const fx::Tw *__restrict__ tw,
                                          int k, unsigned lift, int one) {
  constexpr int NB = (1 << LOGR) / 16;
#pragma unroll
  for (int e = 0; e < 16; e++) {
    const longlong2 z = rp[padx(e * NB)];
    v[e] = fx::C64{fx_lift(z.x, lift), fx_lift(z.y, lift)};
  }
  const fx::Tw *tk = tw + fx_stage_offset<LOGR>(LOGNS) + k;
  v[0] = fx::div16(v[0]);
#pragma unroll
  for (int e = 1; e < 16; e++) v[e] = fx::cmul(v[e], __ldg(tk + (e << LOGNS)), one);
  fx::dft<16>(v, one);
}

// Middle stages, in place in shared memory.
template <int LOGR, int LOGNS, int ST>
__device__ __forceinline__ void fx_mid_stages(longlong2 *sm, const fx::Tw *__restrict__ tw, unsigned (*bits)[16], int one) {
  if constexpr (LOGNS + 4 < LOGR) {
    constexpr int G = g_of<double>(LOGR), TPF = fx_nt<LOGR>() / G;
    const int g = threadIdx.x / TPF, t = threadIdx.x % TPF;
    const int hi = t >> LOGNS, k = t & ((1 << LOGNS) - 1);
    longlong2 *s = sm + g * fx_pitch<LOGR>();
    fx::C64 v[16];
    fx_radix16<LOGR, LOGNS>(v, s + padx(t), tw, k, 1u << fx_spare(bits[ST - 1][g]), one);
    unsigned m = 0;
#pragma unroll
    for (int e = 0; e < 16; e++) m = fx_bits(m, v[e]);
    fx_row_reduce<G, TPF, false>(m, false, bits[ST], g);
    __syncthreads();
    longlong2 *wp = s + padx(hi << (LOGNS + 4)) + padx(k);
#pragma unroll
    for (int e = 0; e < 16; e++) {
      const fx::C64 z = v[fx::dft_at<16>(e)];
      wp[padx(e << LOGNS)] = make_longlong2(z.x, z.y);
    }
    __syncthreads();
    fx_mid_stages<LOGR, LOGNS + 4, ST + 1>(sm, tw, bits, one);
  }
}

template <int LOGR>
__global__ void __launch_bounds__(fx_nt<LOGR>(), fx_minb<LOGR>())
fft_fx_kernel(const __grid_constant__ PassArgs a) {
  pdl_enter();
  constexpr int R = 1 << LOGR, G = g_of<double>(LOGR), NT = fx_nt<LOGR>(), TPF = NT / G;
  constexpr int LOGE0 = fx_loge0<LOGR>(), E0 = 1 << LOGE0;
  constexpr int NB0 = R / E0, Q0 = 16 / E0, NST = (LOGR - LOGE0) / 4;  // NST radix-16 stages after the first
  static_assert(R * G == 16 * NT && G <= 16 && NT >= 16 * FX_MAXST && NST >= 1 && NST <= FX_MAXST, "16 points per thread");
  // |input| < 2^P makes the first stage's outputs stay below 2^62.5; the
  // inter-pass twiddles (scaled by 2^62) take two bits off
  constexpr int P = 62 - LOGE0, PIN = imin(P + 2, 62);
  extern __shared__ __align__(16) unsigned char smraw[];
  if (a.direct) {
    fx_fallback<LOGR>(a, reinterpret_cast<double2 *>(smraw));
    return;
  }
  __shared__ unsigned emax[G], bits[FX_MAXST][16];
  longlong2 *sm = reinterpret_cast<longlong2 *>(smraw);
  const int tid = threadIdx.x;
  const int logS = a.logN - LOGR, logNs = a.logNs;
  const long long Smask = (1LL << logS) - 1, Nsmask = (1LL << logNs) - 1, u0 = (long long)blockIdx.x * G;
  if (tid < G) emax[tid] = 0u;
  if (tid < 16 * FX_MAXST) bits[tid / 16][tid % 16] = 0u;

  unsigned far = 0;  // binades that this thread's samples lie far below their row's largest
  int s_in;  // the exponent of the fixed-point values after the first stage, per row
  {
    // adjacent lanes take adjacent sub-transforms (whole 32-byte sectors) when
    // a row holds at least G of them, else consecutive points of one
    const bool gf = (1LL << logS) >= G;
    const int g = gf ? tid % G : tid / TPF, t0 = gf ? tid / G : tid % TPF;
    const long long u = u0 + g, b = u >> logS, j = u & Smask;
    const bool live = u < a.total;
    // point t0 + r of the thread's sub-transform: src[r step] (row pairs: r steps over
    // whole pairs, so only the first address differs)
    const double2 *src;
    long long step = 1LL << logS;
    const long long m0 = j + ((long long)t0 << logS);
    if (a.gx) {
      src = reinterpret_cast<const double2 *>(a.gx) + (live ? a.goffs[b] + m0 * a.gstride : 0);
      step *= a.gstride;
    } else {
      src = reinterpret_cast<const double2 *>(a.in) + b * a.bstride +
            (a.tile_in ? (j & ~1LL) * R + 2 * t0 + (j & 1) : row_pairs(m0, a.lognc));
      if (a.tile_in) step = 2;
    }
    double2 d[16];
#pragma unroll
    for (int q = 0; q < Q0; q++)
#pragma unroll
      for (int e = 0; e < E0; e++)
        d[q * E0 + e] = live ? src[(q * TPF + e * NB0) * step] : make_double2(0.0, 0.0);
    unsigned mx = 0;
#pragma unroll
    for (int i = 0; i < 16; i++) {
      mx = max(mx, (unsigned)__double2hiint(d[i].x) & 0x7fffffffu);
      mx = max(mx, (unsigned)__double2hiint(d[i].y) & 0x7fffffffu);
    }
    __syncthreads();
    fx_row_reduce<G, TPF, true>(mx, gf, emax, g);
    __syncthreads();
    // every warp sees the same rows' maxima: the same decision in all of them
    const int lane = tid & 31, el = (int)(emax[lane % G] >> 20);
    const bool ll = u0 + lane % G < a.total;
    const int emin = a.samples ? FX_EXP_MIN_SQ : FX_EXP_MIN, emax_ok = a.samples ? FX_EXP_MAX_SQ : FX_EXP_MAX;
    bool out_of_range = __any_sync(0xffffffffu, ll && el != 0 && (el < emin || el > emax_ok));
    if (!out_of_range && __any_sync(0xffffffffu, ll && el == 0)) {
      // a row of zeros is transformed as zeros; subnormals take the FP64 form
      int any = 0;
      if (emax[g] >> 20 == 0)
#pragma unroll
        for (int i = 0; i < 16; i++)
          any |= (__double2hiint(d[i].x) | __double2hiint(d[i].y)) << 1 | __double2loint(d[i].x) |
                 __double2loint(d[i].y);
      out_of_range = __syncthreads_or(any) != 0;
    }
    if (out_of_range) {
      fx_fallback<LOGR>(a, reinterpret_cast<double2 *>(smraw));
      return;
    }
    const int em = emax[g] >> 20 ? (int)(emax[g] >> 20) : 1023;
    const bool pre = logNs > 0;
    const int c = em + 62 - (pre ? PIN : P);
    const unsigned near = (unsigned)(em - FX_NEAR - 1);
    fx::C64 v[16];
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const int ex = fx::exponent(d[i].x), ey = fx::exponent(d[i].y);
      // binades below `near`; a zero's exponent field wraps and counts none
      far += near - min((unsigned)max(ex, ey) - 1u, near);
      v[i].x = fx::from_double(d[i].x, ex, c);
      v[i].y = fx::from_double(d[i].y, ey, c);
      if (a.inverse) v[i].y = -v[i].y;
    }
    if (pre) {
      // W^(jm r), r = t0 + q TPF + e NB0: three two-level table products, then
      // running products at 60 bits
      const longlong2 *thi = reinterpret_cast<const longlong2 *>(a.fx_hi);
      const fx::Tw *tlo = reinterpret_cast<const fx::Tw *>(a.fx_lo);
      const long long jm = j & Nsmask;
      const int hmask = (1 << a.tw_h) - 1;
      auto look = [&](long long mm) {
        const longlong2 h = __ldg(thi + (mm >> a.tw_h));
        return fx::tw_mul(fx::C64{h.x, h.y}, __ldg(tlo + (mm & hmask)), a.one);
      };
      fx::C64 wq = look(jm * t0);
      const fx::Tw se = fx::limbs(look(jm * NB0));
      fx::Tw sq = se;
      if constexpr (Q0 > 1) sq = fx::limbs(look(jm * TPF));
#pragma unroll
      for (int q = 0; q < Q0; q++) {
        fx::C64 w = wq;
#pragma unroll
        for (int e = 0; e < E0; e++) {
          v[q * E0 + e] = fx::cmul(v[q * E0 + e], fx::limbs(w), a.one);
          if (e + 1 < E0) w = fx::tw_mul(w, se, a.one);
        }
        if (q + 1 < Q0) wq = fx::tw_mul(wq, sq, a.one);
      }
    }
    unsigned m = 0;
    longlong2 *s = sm + g * fx_pitch<LOGR>();
#pragma unroll
    for (int q = 0; q < Q0; q++) {
      fx::dft<E0>(v + q * E0, a.one);
#pragma unroll
      for (int e = 0; e < E0; e++) m = fx_bits(m, v[q * E0 + e]);
      longlong2 *wp = s + padx((t0 + q * TPF) << LOGE0);
#pragma unroll
      for (int e = 0; e < E0; e++) {
        const fx::C64 z = v[q * E0 + fx::dft_at<E0>(e)];
        wp[padx(e)] = make_longlong2(z.x, z.y);
      }
    }
    fx_row_reduce<G, TPF, false>(m, gf, bits[0], g);
    s_in = -1022 - (pre ? PIN - 2 : P) + 4 * NST;
  }
  if (__syncthreads_or(far > (unsigned)FX_FAR)) {
    fx_fallback<LOGR>(a, reinterpret_cast<double2 *>(smraw));
    return;
  }
  const fx::Tw *tw = reinterpret_cast<const fx::Tw *>(a.fx_tw);
  fx_mid_stages<LOGR, LOGE0, 1>(sm, tw, bits, a.one);

  // last stage: outputs t + e R/16 straight to global memory, adjacent lanes on
  // adjacent sub-transforms when Ns >= G, else on consecutive outputs
  const bool gf = a.tile_out || (1LL << logNs) >= G;
  const int g = gf ? tid % G : tid / TPF, t = gf ? tid / G : tid % TPF;
  const long long u = u0 + g, b = u >> logS, j = u & Smask;
  const bool live = u < a.total;
  const int em = emax[g] >> 20 ? (int)(emax[g] >> 20) : 1023;
  int s = s_in + em;
#pragma unroll
  for (int i = 0; i < NST; i++) s -= fx_spare(bits[i][g]);
  fx::C64 v[16];
  fx_radix16<LOGR, LOGR - 4>(v, sm + g * fx_pitch<LOGR>() + padx(t), tw, t, 1u << fx_spare(bits[NST - 1][g]),
                               a.one);
  const long long d0 = b * a.bstride + (a.tile_out ? ((long long)(t & ~1) << logS) + 2 * j + (t & 1)
                                                   : ((j >> logNs) << (logNs + LOGR)) + (j & Nsmask) + ((long long)t << logNs));
  const long long ds = (long long)(R / 16) << (a.tile_out ? logS : logNs);
  double tmax = 0.0;
  if (live) {
    double2 *out = reinterpret_cast<double2 *>(a.out) + d0;
    double *smp = reinterpret_cast<double *>(a.samples) + d0;
#pragma unroll
    for (int e = 0; e < 16; e++) {
      fx::C64 X = v[fx::dft_at<16>(e)];
      if (a.write_complex) {
        if (a.inverse) X.y = -X.y;
        out[e * ds] = make_double2(fx_double(X.x, s), fx_double(X.y, s));
      }
      if (a.samples) {
        const double sv = fx_square(X, s);
        smp[e * ds] = sv;
        tmax = sv > tmax ? sv : tmax;
      }
    }
  }
  if (a.samples && a.row_max) {
    const long long bb = __shfl_sync(0xffffffffu, b, 0);
    if (__all_sync(0xffffffffu, live && b == bb)) row_max_update(a.row_max, bb, tmax);
    else if (live) atomicMax(reinterpret_cast<unsigned long long *>(a.row_max) + b, key_bits(tmax));
  }
}

template <int LOGR>
int launch_fx(const PassArgs &a, long long total_sub, cudaStream_t st) {
  constexpr int G = g_of<double>(LOGR), SM = fx_smem<LOGR>();
  static PerContext<int> attr;  // per instantiation and CUDA context
  GS_CHECK(attr.ensure_at_least(SM, [](int v) {
    if (cudaFuncSetAttribute(fft_fx_kernel<LOGR>, cudaFuncAttributeMaxDynamicSharedMemorySize, v) == cudaSuccess)
      return (int)GSFFT_OK;
    set_last_error("fft_fx_kernel: %d bytes of shared memory refused: %s", v,
                   cudaGetErrorString(cudaGetLastError()));
    return (int)GSFFT_ERR_CUDA;
  }));
  const long long grid = (total_sub + G - 1) / G;
  if (grid > 0x7fffffffLL) return GSFFT_ERR_UNSUPPORTED;
  GS_CUDA(launch_pdl(fft_fx_kernel<LOGR>, dim3((unsigned)grid), dim3(fx_nt<LOGR>()), SM, st, a));
  GS_LAUNCHED();
  return GSFFT_OK;
}

}  // namespace

}  // namespace gsfft
