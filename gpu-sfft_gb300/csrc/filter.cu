// A2: flat-window filter design on the GPU, FP64 throughout.
//
// Reference: make_multiple_t (cuExperiment.cu:277-448) with kernels K1-K4
// (:537-601) and cuShift (:507-522).  The reference runs two n-long loops on
// the host over managed memory (boxcar sum :389-396, phase ramp :410-420);
// both are sequential recurrences.  Here:
//   1. win[i] = T_{w-1}(t0 cos(pi i / w)) * tol, NaN -> 0      (K1, :538-552)
//   2. DFT_w(win) by Bluestein over power-of-two FFTs (w is odd)  (:305-308)
//   3. rotate by w/2, drop the imaginary part, place the halves around
//      index 0 of g[n] (one kernel instead of cuShift + K2 + two memcpys)
//   4. G = FFT_n(g)                                                (:362-365)
//   5. boxcar: ff[(i + b_f/2) mod n] = sum_{j=i}^{i+b_f-1} G[j mod n]; each
//      CTA computes the sum at the start of its 4096-output tile directly and
//      the rest as that sum plus a block prefix scan of G[j+b_f] - G[j]
//   6. ff /= max|ff| (K3), ff *= exp(-2 pi i ((w/2) i mod n) / n), the angle
//      reduced exactly in integers (no recurrence)
//   7. filter_time = IFFT_n(ff)[0:w] / n                           (:425-443, K4)
//
// What bounds the kernels here is FP64 arithmetic (1.73 operations per clock and
// SM), so roots of unity come from 64-bit fixed point (fix64.cuh) and the boxcar
// keeps its running sums to nine operations an output.  At n = 2^22: ramp and
// normalisation 448 -> 76 us, boxcar 236 -> 114 us, chirps 40 + 32 -> 14 + 16 us.
#include "engine.cuh"
#include "fix64.cuh"

namespace gsfft {

namespace {

constexpr int FT = 256;

__device__ double cheb(double m, double x) {  // cuExperiment.cu:593-601
  if (fabs(x) <= 1) return cos(m * acos(x));
  return cosh(m * acosh(x));
}

__global__ void cheb_window_kernel(double2 *win, int w, double t0, double tol) {
  const int i = blockIdx.x * FT + threadIdx.x;
  if (i >= w) return;
  const double v = cheb((double)(w - 1), t0 * cos(M_PI * i / (w))) * tol;
  win[i] = make_double2(isnan(v) ? 0.0 : v, 0.0);
}

// a root of unity scaled by 2^62 as doubles
__device__ __forceinline__ double2 root_double(fx::C64 w) {
  return make_double2(__ll2double_rn(w.x) * 0x1p-62, __ll2double_rn(w.y) * 0x1p-62);
}

// 2^128 / (2N), for chirps of N points
struct ChirpStep {
  unsigned long long hi, lo;
};
// chirp c[m] = exp(-pi i m^2 / N): the angle m^2 / (2N) of a turn as a 64-bit
// fraction, m^2 (2^128 / 2N) 2^-64 modulo 2^64 (m < 2^30)
__device__ __forceinline__ double2 chirp(long long m, ChirpStep k) {
  const unsigned long long m2 = (unsigned long long)m * (unsigned long long)m;
  long long c, s;
  fx::sincos62(m2 * k.hi + __umul64hi(m2, k.lo), &c, &s);
  return root_double(fx::C64{c, -s});
}

__global__ void bluestein_prep_kernel(const double2 *__restrict__ x, long long N, long long M,
                                      ChirpStep k, double2 *a, double2 *b) {
  const long long m = (long long)blockIdx.x * FT + threadIdx.x;
  if (m >= M) return;
  double2 av = make_double2(0.0, 0.0), bv = make_double2(0.0, 0.0);
  if (m < N) {
    const double2 c = chirp(m, k);
    av = cmul(x[m], c);
    bv = make_double2(c.x, -c.y);
  } else if (M - m < N) {
    const double2 c = chirp(M - m, k);
    bv = make_double2(c.x, -c.y);
  }
  a[m] = av;
  b[m] = bv;
}

__global__ void pointwise_mul_kernel(double2 *a, const double2 *__restrict__ b, long long M) {
  const long long m = (long long)blockIdx.x * FT + threadIdx.x;
  if (m < M) a[m] = cmul(a[m], b[m]);
}

__global__ void bluestein_post_kernel(const double2 *__restrict__ conv, long long N, long long M,
                                      ChirpStep k, double2 *X) {
  const long long i = (long long)blockIdx.x * FT + threadIdx.x;
  if (i >= N) return;
  double2 v = conv[i];
  v.x /= (double)M;  // M is a power of two
  v.y /= (double)M;
  X[i] = cmul(v, chirp(i, k));
}

// g[j] = Re X[j] (j < h), g[n-h+j] = Re X[j+h+1] (j < h), else 0; h = w/2
__global__ void place_kernel(const double2 *__restrict__ X, int w, int n, double2 *g) {
  const long long i = (long long)blockIdx.x * FT + threadIdx.x;
  if (i >= n) return;
  const int h = w / 2;
  double v = 0.0;
  if (i < h) v = X[i].x;
  else if (i >= n - h) v = X[i - (n - h) + h + 1].x;
  g[i] = make_double2(v, 0.0);
}

constexpr int BOX_PER = 16;              // outputs per thread, held in registers
constexpr int BOX_TILE = FT * BOX_PER;

// Block-wide exclusive scan of one double2 per thread (sums in a fixed order).
__device__ __forceinline__ double2 box_excl_scan(double2 v, double2 *ws) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double2 x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double yx = __shfl_up_sync(0xffffffffu, x.x, o), yy = __shfl_up_sync(0xffffffffu, x.y, o);
    if (lane >= o) {
      x.x += yx;
      x.y += yy;
    }
  }
  if (lane == 31) ws[wid] = x;
  // the lanes' exclusive prefixes: the inclusive ones, one lane up
  double2 e;
  e.x = __shfl_up_sync(0xffffffffu, x.x, 1);
  e.y = __shfl_up_sync(0xffffffffu, x.y, 1);
  if (lane == 0) e = make_double2(0.0, 0.0);
  __syncthreads();
  for (int i = 0; i < wid; i++) {
    e.x += ws[i].x;
    e.y += ws[i].y;
  }
  return e;
}

// max2: bit pattern of the largest |ff|^2
__global__ void __launch_bounds__(FT)
boxcar_kernel(const double2 *__restrict__ G, int n, int b_f, double2 *ff,
              unsigned long long *max2) {
  __shared__ double2 red[FT];
  __shared__ double2 ws[FT / 32];
  __shared__ unsigned long long bmax;
  const long long i0 = (long long)blockIdx.x * BOX_TILE;
  const unsigned long long nm = (unsigned long long)n - 1ull;
  if (threadIdx.x == 0) bmax = 0ull;
  // window sum at i0, by a block reduction in fixed order
  double2 s = make_double2(0.0, 0.0);
  for (int j = threadIdx.x; j < b_f; j += FT) {
    const double2 v = G[(i0 + j) & nm];
    s.x += v.x;
    s.y += v.y;
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = FT / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      red[threadIdx.x].x += red[threadIdx.x + o].x;
      red[threadIdx.x].y += red[threadIdx.x + o].y;
    }
    __syncthreads();
  }
  const double2 base = red[0];
  // running sums of the differences over this thread's outputs
  const long long t0 = i0 + (long long)threadIdx.x * BOX_PER;
  double2 p[BOX_PER], d = make_double2(0.0, 0.0);
#pragma unroll
  for (int q = 0; q < BOX_PER; q++) {
    const double2 in = G[(t0 + q + b_f) & nm], out = G[(t0 + q) & nm];
    p[q] = d;
    d.x += in.x - out.x;
    d.y += in.y - out.y;
  }
  double2 off = box_excl_scan(d, ws);
  off.x += base.x;
  off.y += base.y;
  const int shift = b_f / 2;
  unsigned long long mx = 0ull;
#pragma unroll
  for (int q = 0; q < BOX_PER; q++) {
    const long long i = t0 + q;
    const double2 v = make_double2(off.x + p[q].x, off.y + p[q].y);
    if (i < n) {
      ff[(i + shift) & nm] = v;
      const unsigned long long m = (unsigned long long)__double_as_longlong(fma(v.x, v.x, v.y * v.y));
      mx = m > mx ? m : mx;
    }
  }
  atomicMax(&bmax, mx);
  __syncthreads();
  if (threadIdx.x == 0) atomicMax(max2, bmax);
}

// ff[i] *= exp(-2 pi i (h i mod n) / n) / max|ff|.  The factor is formed in fixed
// point -- root of unity from the FFT plan's two-level table, times the reciprocal
// as a 62-bit integer -- and rounded once.
constexpr int RAMP_PER = 8;  // elements per thread (one reciprocal for all)
__global__ void normalize_ramp_kernel(double2 *ff, int n, int h, const unsigned long long *max2,
                                      const longlong2 *__restrict__ thi, const fx::Tw *__restrict__ tlo, int tw_h,
                                      int one) {
  __shared__ long long s_inv;
  __shared__ int s_exp;
  if (threadIdx.x == 0) {
    const double mx = sqrt(__longlong_as_double((long long)*max2));
    const double r = 1.0 / mx, rl = fma(-r, mx, 1.0) * r;  // 1 / mx = r + rl
    int e;
    frexp(r, &e);  // r = f 2^e, f in [1/2, 1)
    s_inv = __double2ll_rn(ldexp(r, 62 - e)) + __double2ll_rn(ldexp(rl, 62 - e));
    s_exp = e;
  }
  __syncthreads();
  const long long inv = s_inv;  // (1 / mx) 2^(62 - e)
  const int ih = fx::limb_hi(inv), il = fx::limb_lo(inv);
  const double scale = ldexp(1.0, s_exp - 60);
#pragma unroll 2
  for (int q = 0; q < RAMP_PER; q++) {
    const long long i = ((long long)blockIdx.x * RAMP_PER + q) * FT + threadIdx.x;
    if (i >= n) return;
    const long long m = ((long long)h * i) & (long long)(n - 1);
    const longlong2 wh = __ldg(thi + (m >> tw_h));
    const fx::C64 w = fx::tw_mul(fx::C64{wh.x, wh.y}, __ldg(tlo + (m & ((1 << tw_h) - 1))), one);
    const double2 f = make_double2(__ll2double_rn(fx::mul_limbs(w.x, ih, il, one)) * scale,
                                   __ll2double_rn(fx::mul_limbs(w.y, ih, il, one)) * scale);
    ff[i] = cmul(ff[i], f);
  }
}

__global__ void extract_taps_kernel(const double2 *__restrict__ g, int w, int n, double2 *ft) {
  const int i = blockIdx.x * FT + threadIdx.x;
  if (i >= w) return;
  const double2 v = g[i];
  ft[i] = make_double2(v.x / n, v.y / n);
}

unsigned grid_of(long long count) { return (unsigned)((count + FT - 1) / FT); }

}  // namespace

int design_filter(const gsfft_params &p, double2 *d_ft, double2 *d_ff, cudaStream_t st) {
  const int n = p.n, w = p.w;
  if (w < 3 || w > n || (w & 1) == 0 || p.b_f < 1 || p.b_f > n) return GSFFT_ERR_PARAM;
  long long M = 256;
  while (M < 2LL * w - 1) M <<= 1;
  ChirpStep chirp_step;
  {
    const unsigned __int128 turn = (unsigned __int128)1 << 64, D = 2ull * (unsigned)w;
    chirp_step.hi = (unsigned long long)(turn / D);
    chirp_step.lo = (unsigned long long)((turn % D << 64) / D);
  }
  FftPlan fm, fn;
  double2 *win = nullptr, *a = nullptr, *b = nullptr, *g = nullptr, *ffb = nullptr;
  unsigned long long *mx = nullptr;  // bits of max |ff|^2
  int s = GSFFT_OK;
  auto ck = [&](cudaError_t e) {
    if (e != cudaSuccess && s == GSFFT_OK) {
      set_last_error("design_filter: %s", cudaGetErrorString(e));
      s = GSFFT_ERR_CUDA;
    }
  };
  Arena mem;
  void *block = nullptr;
  mem.add(&win, sizeof(double2) * w);
  mem.add(&a, sizeof(double2) * M);
  mem.add(&b, sizeof(double2) * M);
  mem.add(&g, sizeof(double2) * (size_t)n);
  mem.add(&mx, sizeof(unsigned long long), true);
  if (!d_ff) mem.add(&ffb, sizeof(double2) * (size_t)n);
  s = fft_plan_shape(fm, M, FFT_FP64);
  if (s == GSFFT_OK) s = fft_plan_shape(fn, n, FFT_FP64);
  if (s == GSFFT_OK) {
    fft_plan_request(fm, 1, mem);
    fft_plan_request(fn, 1, mem);
    s = mem.commit(&block, st);
  }
  double2 *ff = d_ff ? d_ff : ffb;
  if (s == GSFFT_OK) s = fft_plan_fill(fm, st);
  if (s == GSFFT_OK) s = fft_plan_fill(fn, st);
  FftIo io;
  if (s == GSFFT_OK) {
    cheb_window_kernel<<<grid_of(w), FT, 0, st>>>(win, w, p.t0, p.tolerance);
    ck(cudaGetLastError());
    bluestein_prep_kernel<<<grid_of(M), FT, 0, st>>>(win, w, M, chirp_step, a, b);
    ck(cudaGetLastError());
  }
  if (s == GSFFT_OK) s = fft_exec(fm, a, a, 1, -1, io, st);
  if (s == GSFFT_OK) s = fft_exec(fm, b, b, 1, -1, io, st);
  if (s == GSFFT_OK) {
    pointwise_mul_kernel<<<grid_of(M), FT, 0, st>>>(a, b, M);
    ck(cudaGetLastError());
  }
  if (s == GSFFT_OK) s = fft_exec(fm, a, a, 1, +1, io, st);
  if (s == GSFFT_OK) {
    bluestein_post_kernel<<<grid_of(w), FT, 0, st>>>(a, w, M, chirp_step, win);
    ck(cudaGetLastError());
    place_kernel<<<grid_of(n), FT, 0, st>>>(win, w, n, g);
    ck(cudaGetLastError());
  }
  if (s == GSFFT_OK) s = fft_exec(fn, g, g, 1, -1, io, st);
  if (s == GSFFT_OK) {
    boxcar_kernel<<<(unsigned)((n + BOX_TILE - 1) / BOX_TILE), FT, 0, st>>>(g, n, p.b_f, ff, mx);
    ck(cudaGetLastError());
    const int last = fn.npass - 1;  // the pass whose table reaches n points
    normalize_ramp_kernel<<<grid_of((n + RAMP_PER - 1) / RAMP_PER), FT, 0, st>>>(
        ff, n, w / 2, mx, (const longlong2 *)fn.fx_hi[last], (const fx::Tw *)fn.fx_lo[last], fn.tw_h[last], 1);
    ck(cudaGetLastError());
  }
  if (s == GSFFT_OK) s = fft_exec(fn, ff, g, 1, +1, io, st);
  if (s == GSFFT_OK) {
    extract_taps_kernel<<<grid_of(w), FT, 0, st>>>(g, w, n, d_ft);
    ck(cudaGetLastError());
    ck(cudaStreamSynchronize(st));
  }
  if (block) cudaFree(block);
  return s;
}

}  // namespace gsfft
