// Instantiations of the FP64 FFT pass: radix 2^11 .. 2^13.
#include "fft_pass_fx.cuh"

namespace gsfft {

int fft_pass_f64_hi(int logr, const PassArgs &a, long long total_sub, cudaStream_t st) {
  switch (logr) {
    case 11: return launch_fx<11>(a, total_sub, st);
    case 12: return launch_fx<12>(a, total_sub, st);
    case 13: return launch_fx<13>(a, total_sub, st);
    default: return GSFFT_ERR_UNSUPPORTED;
  }
}

}  // namespace gsfft
