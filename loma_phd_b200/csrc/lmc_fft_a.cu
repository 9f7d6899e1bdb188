// Transform kernels for lengths 3 (the z length of 2-D runs) and 24..96 (see lmc_fft_impl.cuh;
// the radices are those of FFT_RADIX; FP32 butterflies take FFT_RADIX_F32).
#define LMC_FFT_NS fft_a
#include "lmc_fft_impl.cuh"
#define LMC_FFT_SIZES(X) X(3, 3, 1, 1) X(24, 6, 4, 1) X(36, 6, 6, 1) X(48, 6, 8, 1) X(72, 12, 6, 1) X(96, 12, 8, 1)
LMC_FFT_TU_BODY(a)
