// Power-of-two complex FFT plans and execution (the pass kernel is in
// fft_pass.cuh).
#include "fft_pass.cuh"
#include "fix64.cuh"

#include <algorithm>

namespace gsfft {

namespace {

// The tables of a plan, all built by one launch.
enum TableKind { TAB_F32, TAB_F64, TAB_FX_STAGES, TAB_FX_HI, TAB_FX_LO };
struct TableJob {
  void *dst;
  int kind, count, block;  // block: first block of the job
  int lg;                  // angles in units of 2 pi / 2^lg
  int shift;               // entry m has angle m << shift (F32, F64, FX_HI, FX_LO)
  int logr;                // FX_STAGES: log2 of the pass's radix
};
constexpr int MAX_JOBS = 3 * 6;
struct TableJobs {
  TableJob j[MAX_JOBS];
  int n, blocks;
};

// F32, F64: exp(-2 pi i (m << shift) / 2^lg), the angle reduced exactly in
// integers.  FP64 passes' fixed-point twiddles: FX_STAGES the radix-16 stages' rows
// [e][k] = exp(-2 pi i e k / (16 Ns)) scaled by 2^60; FX_HI, FX_LO two-level
// tables scaled by 2^62.
__global__ void tables_kernel(TableJobs jobs) {
  int q = jobs.n - 1;
  while (q > 0 && (int)blockIdx.x < jobs.j[q].block) q--;
  const TableJob &t = jobs.j[q];
  const int i = ((int)blockIdx.x - t.block) * 256 + (int)threadIdx.x;
  if (i >= t.count) return;
  if (t.kind == TAB_F32 || t.kind == TAB_F64) {
    const long long N = 1LL << t.lg, num = ((long long)i << t.shift) & (N - 1);
    double s, c;
    sincospi(2.0 * (double)num / (double)N, &s, &c);
    if (t.kind == TAB_F32) reinterpret_cast<float2 *>(t.dst)[i] = make_float2((float)c, (float)(-s));
    else reinterpret_cast<double2 *>(t.dst)[i] = make_double2(c, -s);
  } else if (t.kind == TAB_FX_STAGES) {
    int logns = t.logr % 4 == 0 ? 4 : t.logr % 4, at = i;
    while (at >= (16 << logns)) {
      at -= 16 << logns;
      logns += 4;
    }
    const unsigned e = (unsigned)at >> logns, k = (unsigned)at & ((1u << logns) - 1u);
    const fx::C64 w = fx::unit_root((unsigned long long)e * k, logns + 4);
    reinterpret_cast<fx::Tw *>(t.dst)[i] = fx::limbs(fx::C64{(w.x + 2) >> 2, (w.y + 2) >> 2});
  } else {
    const fx::C64 w = fx::unit_root((unsigned long long)i << t.shift, t.lg);
    if (t.kind == TAB_FX_HI) reinterpret_cast<longlong2 *>(t.dst)[i] = make_longlong2(w.x, w.y);
    else reinterpret_cast<fx::Tw *>(t.dst)[i] = fx::limbs(w);
  }
}

int fx_stage_entries(int logr) {
  int n = 0;
  for (int l = logr % 4 == 0 ? 4 : logr % 4; l < logr; l += 4) n += 16 << l;
  return n;
}

int dispatch_pass(bool dbl, int logr, const PassArgs &a, long long total_sub, cudaStream_t st) {
  if (dbl) return logr <= 10 ? fft_pass_f64_lo(logr, a, total_sub, st) : fft_pass_f64_hi(logr, a, total_sub, st);
  return logr <= 10 ? fft_pass_f32_lo(logr, a, total_sub, st) : fft_pass_f32_hi(logr, a, total_sub, st);
}

}  // namespace

int fft_plan_shape(FftPlan &p, long long n, FftKind kind, int first_logr, bool spread) {
  p = FftPlan();
  if (n < 256 || (n & (n - 1)) != 0) return GSFFT_ERR_UNSUPPORTED;
  int L = 0;
  while ((1LL << L) < n) L++;
  const bool dbl = kind == FFT_FP64 || kind == FFT_FP64_DIRECT;
  const int one_pass_max = dbl ? 13 : 14;
  int r[3] = {0, 0, 0}, npass = 0;
  if (kind == FFT_FP32_TC) {
    // the second pass is a CUDA-core pass of radix 2^(L-12)
    if (L - 12 < 5 || L - 12 > 14) return GSFFT_ERR_UNSUPPORTED;
    npass = 2;
    r[0] = 12;
    r[1] = L - 12;
    p.tc[0] = true;
  } else if (kind == FFT_FP32_TC64) {
    if (L < 13 || L > 20) return GSFFT_ERR_UNSUPPORTED;
    npass = 2;
    r[0] = L - 6;
    r[1] = 6;
    p.tc[1] = true;
  } else if (L <= one_pass_max) {
    if (first_logr > 0) return GSFFT_ERR_PARAM;  // one pass: no first radix to choose
    npass = 1;
    r[0] = L;
    // one row of 2^13 is 19 us of arithmetic for one SM: few rows go in two passes of
    // 2048 points a CTA (n = 2^20 step, 2 + 5 rows of 2^13: 117 -> 113 us)
    if (spread && kind == FFT_FP64 && L >= 12) {
      npass = 2;
      r[0] = L - 6;
      r[1] = 6;
    }
  } else if (L <= 24) {
    npass = 2;
    r[0] = (L + 1) / 2;
    if (first_logr > 0) {
      if (first_logr < 7 || first_logr > one_pass_max || L - first_logr < 7 ||
          L - first_logr > one_pass_max)
        return GSFFT_ERR_PARAM;
      r[0] = first_logr;
    }
    r[1] = L - r[0];
  } else if (L <= 36) {
    if (first_logr > 0) return GSFFT_ERR_PARAM;
    npass = 3;
    r[0] = (L + 2) / 3;
    r[1] = (L - r[0] + 1) / 2;
    r[2] = L - r[0] - r[1];
  } else {
    return GSFFT_ERR_UNSUPPORTED;
  }
  if (dbl || kind == FFT_FP32)
    for (int i = 0; i < npass; i++)
      if (r[i] < (spread ? 6 : 7) || r[i] > one_pass_max) return GSFFT_ERR_UNSUPPORTED;
  p.n = n;
  p.L = L;
  p.precision = dbl ? GSFFT_FP64 : GSFFT_MIXED;
  p.direct = kind == FFT_FP64_DIRECT;
  p.npass = npass;
  int lg = 0;
  for (int i = 0; i < npass; i++) {
    p.logR[i] = r[i];
    lg += r[i];
    p.tw_h[i] = (lg + 1) / 2;
  }
  return GSFFT_OK;
}

void fft_plan_request(FftPlan &p, int max_batch, Arena &mem) {
  const bool dbl = p.precision == GSFFT_FP64;
  const size_t es = dbl ? sizeof(double2) : sizeof(float2);
  int lg = 0;
  for (int i = 0; i < p.npass; i++) {
    lg += p.logR[i];
    const size_t nlo = (size_t)1 << p.tw_h[i], nhi = (size_t)1 << (lg - p.tw_h[i]);
    mem.add(&p.tw_lo[i], es * nlo);
    mem.add(&p.tw_hi[i], es * nhi);
    mem.add(&p.tw_R[i], es << p.logR[i]);
    if (dbl && !p.direct) {
      mem.add(&p.fx_tw[i], sizeof(fx::Tw) * fx_stage_entries(p.logR[i]));
      mem.add(&p.fx_hi[i], sizeof(longlong2) * nhi);
      mem.add(&p.fx_lo[i], sizeof(fx::Tw) * nlo);
    }
  }
  if (p.tc[0]) mem.add(&p.tc_F, tc_F_bytes());
  if (p.tc[1]) mem.add(&p.tc_F, tc_F_smem_bytes());
  if (p.npass > 1) {
    p.scratch_elems = p.n * max_batch * (p.npass == 3 ? 2 : 1);
    mem.add(&p.scratch, es * p.scratch_elems);
  }
}

int fft_plan_fill(const FftPlan &p, cudaStream_t st) {
  const bool dbl = p.precision == GSFFT_FP64;
  TableJobs jobs;
  jobs.n = jobs.blocks = 0;
  auto add = [&](void *dst, int kind, int count, int lg, int shift, int logr) {
    jobs.j[jobs.n++] = TableJob{dst, kind, count, jobs.blocks, lg, shift, logr};
    jobs.blocks += (count + 255) / 256;
  };
  int lg = 0;
  for (int i = 0; i < p.npass; i++) {
    lg += p.logR[i];
    const int h = p.tw_h[i], nlo = 1 << h, nhi = 1 << (lg - h), kind = dbl ? TAB_F64 : TAB_F32;
    add(p.tw_lo[i], kind, nlo, lg, 0, 0);
    add(p.tw_hi[i], kind, nhi, lg, h, 0);
    add(p.tw_R[i], kind, 1 << p.logR[i], p.logR[i], 0, 0);
    if (dbl && !p.direct) {
      add(p.fx_tw[i], TAB_FX_STAGES, fx_stage_entries(p.logR[i]), 0, 0, p.logR[i]);
      add(p.fx_hi[i], TAB_FX_HI, nhi, lg, h, 0);
      add(p.fx_lo[i], TAB_FX_LO, nlo, lg, 0, 0);
    }
  }
  tables_kernel<<<jobs.blocks, 256, 0, st>>>(jobs);
  GS_LAUNCHED();
  if (p.tc[0]) GS_CHECK(tc_build_F(p.tc_F, st));
  if (p.tc[1]) GS_CHECK(tc_build_F_smem(p.tc_F, st));
  return GSFFT_OK;
}

int fft_plan_init(FftPlan &p, long long n, FftKind kind, int max_batch, cudaStream_t st) {
  fft_plan_free(p);
  GS_CHECK(fft_plan_shape(p, n, kind));
  Arena mem;
  fft_plan_request(p, max_batch, mem);
  void *block = nullptr;
  int s = mem.commit(&block, st);
  p.mem = block;
  if (s == GSFFT_OK) s = fft_plan_fill(p, st);
  if (s != GSFFT_OK) fft_plan_free(p);
  return s;
}

void fft_plan_free(FftPlan &p) {
  if (p.mem) cudaFree(p.mem);
  p = FftPlan();
}

// fused_first_stage (radix 2^11, 2^12): its steps of 128 and 256 in r are whole
// blocks of rows from 128 rows on, and with no more rows than the radix a block's
// rows are all read by the one CTA.  FP64 (radix 2^10 .. 2^12, pairs of rows): steps of
// R/16 and 256, from 32 rows on.
bool fft_reads_row_blocks(const FftPlan &p, int lognc) {
  if (p.npass < 2 || p.tc[0]) return false;
  const int lr = p.logR[0], lognb = p.L - lognc;
  if (p.precision == GSFFT_FP64) return lr >= 10 && lr <= 12 && p.L - lr >= 1 && lognb >= 5 && lognb <= lr;
  return (lr == 11 || lr == 12) && p.L - lr >= 2 && lognb >= 7 && lognb <= lr;
}

// FP32, two passes, the first with fused loads and stores (radix 2^11, 2^12), the second
// one that takes four sub-transforms at a time (2^10 .. 2^12): between them the
// array is kept tile by tile, point r of sub-transform j of the second pass at
// (j & ~3) R + 4 r + (j & 3).  The second pass reads whole lines in order, not a
// sector every N/R points (its loads were a third of its time: L1 lines, not DRAM),
// and the first writes lines, not half ones.  Second pass of two rows of 2^24:
// 221 -> 185 us.
// FP64 (pairs of sub-transforms, radices 2^10 .. 2^12): the same with 2 for 4; two rows
// of 2^22 in gsfft_fft 467 -> 446 us, the n = 2^27 step 885 -> 871.
static bool fft_tiled(const FftPlan &p) {
  if (p.npass != 2 || p.tc[0] || p.tc[1]) return false;
  return p.logR[0] >= (p.precision == GSFFT_FP64 ? 10 : 11) && p.logR[0] <= 12 && p.logR[1] >= 10 && p.logR[1] <= 12;
}

int fft_exec(const FftPlan &p, const void *in, void *out, int batch, int sign,
             const FftIo &io, cudaStream_t st) {
  if (p.npass == 0) return GSFFT_ERR_STATE;
  const bool dbl = p.precision == GSFFT_FP64;
  const size_t es = dbl ? 16 : 8;
  if (p.npass > 1 && (long long)batch * p.n * (p.npass == 3 ? 2 : 1) > p.scratch_elems)
    return GSFFT_ERR_PARAM;
  if (io.gather_x && batch > 8) return GSFFT_ERR_PARAM;
  if (io.in_lognc >= 0 && (io.sum_rows > 1 || io.gather_x || !fft_reads_row_blocks(p, io.in_lognc)))
    return GSFFT_ERR_UNSUPPORTED;
  if (dbl && io.sum_rows > 1) return GSFFT_ERR_UNSUPPORTED;  // FP32 passes only
  const bool tiled = fft_tiled(p) && !io.gather_x && io.sum_rows <= 1;
  const void *src = in;
  char *scr = (char *)p.scratch;
  long long Ns = 1;
  for (int i = 0; i < p.npass; i++) {
    const bool last = i == p.npass - 1;
    void *dst;
    if (last) dst = out;
    else dst = scr + (size_t)(i == 1 ? 1 : 0) * es * p.n * batch;
    PassArgs a;
    a.in = src;
    a.out = dst;
    a.N = p.n;
    a.logN = p.L;
    {
      int l = 0;
      while ((1LL << l) < Ns) l++;
      a.logNs = l;
    }
    a.bstride = p.n;
    a.batch = batch;
    a.Ns = (int)Ns;
    a.inverse = sign > 0;
    a.tw_hi = p.tw_hi[i];
    a.tw_lo = p.tw_lo[i];
    a.tw_h = p.tw_h[i];
    a.twR = p.tw_R[i];
    a.fx_tw = p.fx_tw[i];
    a.fx_hi = p.fx_hi[i];
    a.fx_lo = p.fx_lo[i];
    a.one = 1;
    a.direct = p.direct ? 1 : 0;
    a.gx = (i == 0) ? io.gather_x : nullptr;
    for (int q = 0; q < 8; q++) a.goffs[q] = io.gather_offsets[q];
    a.gstride = io.gather_stride;
    a.samples = last ? io.samples : nullptr;
    a.row_max = last ? io.row_max : nullptr;
    a.lognc = i == 0 ? io.in_lognc : -1;
    a.tile_out = tiled && i == 0;
    a.tile_in = tiled && i == 1;
    a.nsum = (i == 0) ? io.sum_rows : 1;
    a.sstride = io.sum_stride;
    a.write_complex = last ? (io.write_complex ? 1 : 0) : 1;
    const long long total_sub = (p.n >> p.logR[i]) * batch;
    a.total = total_sub;
    int s;
    if (p.tc[i]) {
      if (dbl || a.gx || (p.logR[i] != 12 && p.logR[i] != 6)) return GSFFT_ERR_UNSUPPORTED;
      TcPassArgs t;
      t.in = a.in;
      t.out = a.out;
      t.logN = a.logN;
      t.logNs = a.logNs;
      t.bstride = a.bstride;
      t.total = total_sub;
      t.inverse = a.inverse;
      t.tw_hi = a.tw_hi;
      t.tw_lo = a.tw_lo;
      t.tw_h = a.tw_h;
      t.F = p.tc_F;
      t.tw_R = p.tw_R[i];
      t.samples = a.samples;
      t.row_max = a.row_max;
      t.write_complex = a.write_complex;
      t.err = io.err;
      t.nsum = a.nsum;
      t.sstride = a.sstride;
      s = p.logR[i] == 6 ? launch_tc64_last_pass(t, st) : launch_tc4096_pass(t, st);
    } else {
      s = dispatch_pass(dbl, p.logR[i], a, total_sub, st);
    }
    if (s != GSFFT_OK) return s;
    src = dst;
    Ns <<= p.logR[i];
  }
  return GSFFT_OK;
}

}  // namespace gsfft
