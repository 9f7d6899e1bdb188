// Transform kernels for lengths 144..384 (see lmc_fft_impl.cuh;
// the radices are those of FFT_RADIX; FP32 butterflies take FFT_RADIX_F32).
#define LMC_FFT_NS fft_b
#include "lmc_fft_impl.cuh"
#define LMC_FFT_SIZES(X) X(144, 12, 12, 1) X(192, 12, 16, 1) X(288, 6, 6, 8) X(384, 6, 8, 8)
LMC_FFT_TU_BODY(b)
