// Internal declarations shared by the engine's translation units.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include <mutex>
#include <utility>
#include <vector>

#include "gsfft.h"

namespace gsfft {

// ---------------------------------------------------------------- per-context set-up
// The calling thread's current CUDA context: its device ordinal and the
// driver's context id, which is unique for the life of the process (a context
// made after cudaDeviceReset gets a new one).
struct CtxKey {
  int dev = -1;
  unsigned long long id = 0;
  bool operator==(const CtxKey &o) const { return dev == o.dev && id == o.id; }
};
int current_ctx_key(CtxKey *out);

// One value per CUDA context, computed on first use in that context under a
// lock.  Function attributes, occupancy figures and symbol addresses belong
// to a context, so caching them process-wide would skip the set-up on a
// second device, or after a device reset.
template <typename T>
class PerContext {
 public:
  template <typename F>
  T get(F &&compute) {
    CtxKey k;
    if (current_ctx_key(&k) != 0) return compute();
    std::lock_guard<std::mutex> lock(mu_);
    for (int i = 0; i < n_; i++)
      if (keys_[i] == k) return vals_[i];
    const T v = compute();
    if (n_ < kSlots) {
      keys_[n_] = k;
      vals_[n_] = v;
      n_++;
    }
    return v;
  }
  // Calls set(want) unless this context already recorded a value >= want;
  // records want when set returns 0.  For grow-only attributes such as the
  // dynamic shared memory limit of a kernel.
  template <typename F>
  int ensure_at_least(T want, F &&set) {
    CtxKey k;
    if (current_ctx_key(&k) != 0) return set(want);
    std::lock_guard<std::mutex> lock(mu_);
    int i = 0;
    for (; i < n_; i++)
      if (keys_[i] == k) break;
    if (i < n_ && !(vals_[i] < want)) return 0;
    const int rc = set(want);
    if (rc == 0) {
      if (i < n_) {
        vals_[i] = want;
      } else if (n_ < kSlots) {
        keys_[n_] = k;
        vals_[n_] = want;
        n_++;
      }
    }
    return rc;
  }
  // Calls f the first time in this context (not at all when the table is full).
  template <typename F>
  void once(F &&f) {
    CtxKey k;
    if (current_ctx_key(&k) != 0) return;
    std::lock_guard<std::mutex> lock(mu_);
    for (int i = 0; i < n_; i++)
      if (keys_[i] == k) return;
    if (n_ == kSlots) return;
    keys_[n_++] = k;
    f();
  }

 private:
  static constexpr int kSlots = 64;
  std::mutex mu_;
  CtxKey keys_[kSlots];
  T vals_[kSlots] = {};
  int n_ = 0;
};

// ---------------------------------------------------------------- errors
void set_last_error(const char *fmt, ...);

#define GS_CUDA(call)                                                        \
  do {                                                                       \
    cudaError_t e_ = (call);                                                 \
    if (e_ != cudaSuccess) {                                                 \
      ::gsfft::set_last_error("%s:%d %s: %s", __FILE__, __LINE__, #call,     \
                              cudaGetErrorString(e_));                       \
      return GSFFT_ERR_CUDA;                                                 \
    }                                                                        \
  } while (0)

#define GS_CHECK(call)                        \
  do {                                        \
    int s_ = (call);                          \
    if (s_ != GSFFT_OK) return s_;            \
  } while (0)

// Every kernel launch goes through this: checks the launch and counts it.
extern thread_local int g_launch_counter;
#define GS_LAUNCHED()                                                         \
  do {                                                                        \
    ++::gsfft::g_launch_counter;                                              \
    cudaError_t e_ = cudaGetLastError();                                      \
    if (e_ != cudaSuccess) {                                                  \
      ::gsfft::set_last_error("%s:%d launch: %s", __FILE__, __LINE__,         \
                              cudaGetErrorString(e_));                        \
      return GSFFT_ERR_CUDA;                                                  \
    }                                                                         \
  } while (0)

// ---------------------------------------------------------------- memory
// Buffers of one object in one device allocation.  A cudaMalloc or cudaFree costs
// about 10 us of host time, and a plan has some forty buffers: outer_loop, which
// makes a plan per call, spent 0.8 of its 1.25 ms on them at n = 2^20.  add()
// notes a buffer, commit() allocates the block and sets the pointers; the buffers
// added with zero = true lie together and are cleared with one memset on st.
//
// The first commit in a context also takes 512 bytes that stay: allocations below 2 MB
// share 2 MB blocks, and one that finds no block in use maps a new one (31 us, and 27 us
// to unmap it when it is freed) where it takes 2 us from a block that is there.  A plan's many
// small buffers kept such blocks in use; with one large one per plan, the calls
// that allocate their own scratch beside a living plan had gone from 45 to 120 us
// (gsfft_fft of 2^8 floats), 42 to 120 (gsfft_cutoff of 1000), 33 to 163 (gsfft_stage_estimate).
class Arena {
 public:
  template <typename T>
  void add(T **p, size_t bytes, bool zero = false) {
    (zero ? zeroed_ : plain_).emplace_back(reinterpret_cast<void **>(p), bytes);
  }
  int commit(void **block, cudaStream_t st) {
    size_t plain = 0, all = 0;
    for (const auto &w : plain_) plain += round_up(w.second);
    all = plain;
    for (const auto &w : zeroed_) all += round_up(w.second);
    *block = nullptr;
    static PerContext<int> small_block;
    small_block.once([] {
      void *stays = nullptr;
      if (cudaMalloc(&stays, 512) != cudaSuccess) cudaGetLastError();  // only slower without
    });
    const cudaError_t e = cudaMalloc(block, all ? all : 16);
    if (e != cudaSuccess) {
      set_last_error("cudaMalloc(%zu): %s", all, cudaGetErrorString(e));
      *block = nullptr;
      return GSFFT_ERR_ALLOC;
    }
    char *b = static_cast<char *>(*block);
    for (const auto &v : {plain_, zeroed_})
      for (const auto &w : v) {
        *w.first = b;
        b += round_up(w.second);
      }
    if (all > plain) GS_CUDA(cudaMemsetAsync(static_cast<char *>(*block) + plain, 0, all - plain, st));
    return GSFFT_OK;
  }

 private:
  static size_t round_up(size_t v) { return (v + 511) / 512 * 512; }
  std::vector<std::pair<void **, size_t>> plain_, zeroed_;
};

// ---------------------------------------------------------------- bounded waits
// Every wait of a kernel on an mbarrier (a TMA copy's or a tensor-core
// product's completion) gives up after `limit` SM clock cycles -- by default
// 2^30, about half a second at 2 GHz, far above any real completion -- and
// returns false, so that a kernel whose producer never arrives records an
// error and returns instead of hanging the GPU.
constexpr long long kWaitLimitCycles = 1LL << 30;
__device__ __forceinline__ bool mbar_try_wait(unsigned bar_smem_addr, unsigned parity) {
  unsigned done;
  asm volatile(
      "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
      : "=r"(done)
      : "r"(bar_smem_addr), "r"(parity)
      : "memory");
  return done != 0;
}
__device__ __forceinline__ bool mbar_wait_bounded(unsigned bar_smem_addr, unsigned parity,
                                                  long long limit = kWaitLimitCycles) {
  if (mbar_try_wait(bar_smem_addr, parity)) return true;  // no clock read when it is done
  const long long t0 = clock64();
  while (true) {
    if (mbar_try_wait(bar_smem_addr, parity)) return true;
    if (clock64() - t0 > limit) return false;
  }
}
// launches the failure-detection self-check kernel (capi.cu: gsfft_check_bounded_wait)
int launch_bounded_wait_probe(long long limit, int *gave_up, cudaStream_t st);

// ---------------------------------------------------------------- launches
// Programmatic dependent launch.  The kernels of a run begin with pdl_enter():
// griddepcontrol.wait returns once the preceding grid of the stream has
// completed and its writes are visible (at once when the kernel was launched
// normally), then launch_dependents lets the next kernel be scheduled as soon
// as every block of this grid has passed its wait.  So only the launch of the
// next kernel overlaps this one; its blocks wait before touching memory, and a
// waiting grid never holds resources its predecessor still needs (all of the
// predecessor's blocks have started by then).
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Launch `kernel` as a programmatic dependent of the stream's previous kernel.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                              cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// ---------------------------------------------------------------- complex
template <typename T> struct Cx;
template <> struct Cx<double> { typedef double2 V; };
template <> struct Cx<float> { typedef float2 V; };

__host__ __device__ __forceinline__ double2 mk(double x, double y) { return make_double2(x, y); }
__host__ __device__ __forceinline__ float2 mk(float x, float y) { return make_float2(x, y); }

template <typename V> __device__ __forceinline__ V cadd(V a, V b) { V c; c.x = a.x + b.x; c.y = a.y + b.y; return c; }
template <typename V> __device__ __forceinline__ V csub(V a, V b) { V c; c.x = a.x - b.x; c.y = a.y - b.y; return c; }
template <typename V> __device__ __forceinline__ V cconj(V a) { a.y = -a.y; return a; }
// (a.x b.x - a.y b.y, a.x b.y + a.y b.x), two fused operations per component.
template <typename V> __device__ __forceinline__ V cmul(V a, V b) {
  V c;
  c.x = fma(a.x, b.x, -(a.y * b.y));
  c.y = fma(a.x, b.y, a.y * b.x);
  return c;
}

// Keys whose unsigned order equals the order of non-negative floats.
template <typename T> struct KeyOf;
template <> struct KeyOf<double> { typedef unsigned long long K; };
template <> struct KeyOf<float> { typedef unsigned int K; };

// ---------------------------------------------------------------- FFT
struct FftPlan {
  long long n = 0;         // transform size (power of two)
  int L = 0;               // log2 n
  int precision = 0;       // GSFFT_FP64 / GSFFT_MIXED (float)
  int npass = 0;
  int logR[3] = {0, 0, 0}; // radix of each pass (log2)
  // per pass: twiddle tables for exp(-2 pi i m / Np) with Np = prod radices
  // up to and including the pass, split as hi[m >> h] * lo[m & (2^h - 1)].
  void *tw_hi[3] = {nullptr, nullptr, nullptr};
  void *tw_lo[3] = {nullptr, nullptr, nullptr};
  int tw_h[3] = {0, 0, 0};
  void *tw_R[3] = {nullptr, nullptr, nullptr};  // exp(-2 pi i m / R) for the pass radix
  bool direct = false;     // FFT_FP64_DIRECT
  // FP64, not direct: fixed-point twiddles of the pass (fft_pass_fx.cuh)
  void *fx_tw[3] = {nullptr, nullptr, nullptr};
  void *fx_hi[3] = {nullptr, nullptr, nullptr};
  void *fx_lo[3] = {nullptr, nullptr, nullptr};
  bool tc[3] = {false, false, false};  // pass runs on the tensor cores (radix 4096 or 64, FP32)
  void *tc_F = nullptr;                // DFT_64 operand of the tensor-core pass (its layout
                                       // follows the pass: tc_build_F / tc_build_F_smem)
  void *scratch = nullptr; // one transform-sized buffer per batch entry (multi-pass)
  long long scratch_elems = 0;
  void *mem = nullptr;     // the allocation of a plan of its own (fft_plan_init)
};

// One tensor-core pass of an FP32 FFT (tc_dft.cu): the radix-4096 first
// pass or the radix-64 last pass.
struct TcPassArgs {
  const void *in;       // float2
  void *out;            // float2
  int logN, logNs;
  long long bstride, total;  // row stride; sub-transforms over the batch
  int inverse;
  const void *tw_hi, *tw_lo;
  int tw_h;
  const void *F;        // three bf16 parts of the DFT_64 real form (tc_build_F)
  const void *tw_R;     // exp(-2 pi i m / 4096) for the radix-4096 form
  void *samples;        // float |X|^2 or null
  void *row_max;        // u32 bit pattern per row, with samples
  int write_complex;
  int *err;             // set when a completion wait timed out (may be null)
  int nsum = 1;         // radix-4096 form: add nsum partial inputs sstride apart
  long long sstride = 0;
};
size_t tc_F_bytes();
int tc_build_F(void *F, cudaStream_t st);
// radix 64 as the last pass (one DFT_64 product per 128 sub-transforms)
size_t tc_F_smem_bytes();
int tc_build_F_smem(void *F, cudaStream_t st);
int launch_tc64_last_pass(const TcPassArgs &a, cudaStream_t st);
// radix 4096 = 64 x 64 in one pass (four-step, both DFT_64 stages on the tensor cores)
int launch_tc4096_pass(const TcPassArgs &a, cudaStream_t st);

// Optional fused prologue/epilogue of an FFT execution.
struct FftIo {
  // gather loader (first pass): element m of batch b is x[offs[b] + m * stride]
  const void *gather_x = nullptr;
  long long gather_offsets[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // one per batch entry (batch <= 8)
  long long gather_stride = 0;
  // first-pass loader alternative: element = sum over s < sum_rows of
  // in[s * sum_stride + index], added in s order (no caller asks for it; without
  // its code in the pass kernel nvcc orders the radix 2^11 and 2^12 passes worse: n =
  // 2^27, k = 43000 step 838 -> 859 us, k = 16000 384 -> 390)
  int sum_rows = 1;
  long long sum_stride = 0;
  // first-pass loader alternative (fft_reads_row_blocks): the input is a matrix of
  // 2^in_lognc columns in blocks of four rows, point t = row 2^in_lognc + column at
  // (row & ~3) 2^in_lognc + 4 column + (row & 3); FP64 the same with pairs of rows;
  // -1 = in order
  int in_lognc = -1;
  // epilogue: |X|^2 (same precision) written to samples[b * n + k]
  void *samples = nullptr;
  // optional: per-row maximum of the samples (bit pattern, u64 for double /
  // u32 for float) accumulated with atomicMax; the caller zeroes it first
  void *row_max = nullptr;
  bool write_complex = true;
  // tensor-core passes: set when a completion wait timed out (may be null)
  int *err = nullptr;
};

// Kinds of plan: FP64 on the integer pipes or (_DIRECT) in FP64 arithmetic throughout;
// FP32 on the CUDA cores; FP32 with a radix-4096
// tensor-core pass, then a CUDA-core pass of radix n / 4096 (n = 2^(17..26)); FP32
// with a CUDA-core radix-2^(L-6) first pass, then a tensor-core radix-64 last pass
// (13 <= L <= 20).  GSFFT_ERR_UNSUPPORTED for other sizes.
enum FftKind { FFT_FP64, FFT_FP64_DIRECT, FFT_FP32, FFT_FP32_TC, FFT_FP32_TC64 };
// A plan in three steps, so that its tables and scratch (max_batch transforms) can
// share an allocation: its passes (first_logr: log2 of the first pass's radix for
// two-pass sizes of the kinds without tensor cores, 0: ceil(L/2); spread: FP64 transforms of 2^12 and
// 2^13 in two passes on several CTAs a row, for few rows), its buffers, the tables.
int fft_plan_shape(FftPlan &p, long long n, FftKind kind, int first_logr = 0, bool spread = false);
void fft_plan_request(FftPlan &p, int max_batch, Arena &mem);
int fft_plan_fill(const FftPlan &p, cudaStream_t st);
// The three steps with an allocation of its own; tables are built on st, the
// stream that the plan is then used on (or synchronised with).
int fft_plan_init(FftPlan &p, long long n, FftKind kind, int max_batch, cudaStream_t st);
void fft_plan_free(FftPlan &p);
// whether the plan's first pass reads FftIo::in_lognc input in whole sectors
bool fft_reads_row_blocks(const FftPlan &p, int lognc);
// in: batch entries at in + b*n; out: out + b*n.  sign -1 forward, +1 inverse.
int fft_exec(const FftPlan &p, const void *in, void *out, int batch, int sign,
             const FftIo &io, cudaStream_t st);

// ---------------------------------------------------------------- select
// Top-`num` of each row by key (ties at the threshold: lowest index first),
// indices written ascending.  keys: double or float samples (bit patterns of
// non-negative values).  size either fixed (size_dev == nullptr) or read from
// *size_dev (rows then have capacity `size`, only the first *size_dev used;
// batch must be 1).  When the live size <= num, all live indices are taken.
struct SelectScratch {
  void *hist = nullptr;        // batch * 2048 uint32
  void *state = nullptr;       // batch * SelState
  void *tiles = nullptr;       // batch * max_tiles * 4 uint32
  void *coop_hist = nullptr;   // single-launch form: 6 passes x 8 rows x 2048 bins, zero between calls
  int max_batch = 0, max_tiles = 0;
  bool single_launch = true;   // cluster / cooperative form allowed (else multi-launch)
};
// Byte sizes of the SelectScratch regions for max_batch rows of at most
// max_size samples (what select_scratch_request asks for); state and coop_hist
// must hold zeros when a selection starts.
struct SelectScratchBytes {
  size_t hist, state, tiles, coop_hist;
  int max_tiles;
};
SelectScratchBytes select_scratch_bytes(int max_batch, long long max_size);
void select_scratch_request(SelectScratch &s, int max_batch, long long max_size, Arena &mem);
// row_max (optional, per row, bit pattern of the largest sample) with
// floor_rel > 0: samples below floor_rel * max are taken as exact zeros, so
// rounding-level samples tie and resolve by ascending index.
int select_top(const void *keys, int key_bytes, long long size, const int *size_dev,
               int num, int batch, long long row_stride, int *out, long long out_stride,
               int *count_out, SelectScratch &s, cudaStream_t st,
               const void *row_max = nullptr, double floor_rel = 0.0);

}  // namespace gsfft
