// Instantiations of the FP64 FFT pass: radix 2^6 .. 2^10.
#include "fft_pass_fx.cuh"

namespace gsfft {

int fft_pass_f64_lo(int logr, const PassArgs &a, long long total_sub, cudaStream_t st) {
  switch (logr) {
    case 6: return launch_fx<6>(a, total_sub, st);
    case 7: return launch_fx<7>(a, total_sub, st);
    case 8: return launch_fx<8>(a, total_sub, st);
    case 9: return launch_fx<9>(a, total_sub, st);
    case 10: return launch_fx<10>(a, total_sub, st);
    default: return GSFFT_ERR_UNSUPPORTED;
  }
}

}  // namespace gsfft
