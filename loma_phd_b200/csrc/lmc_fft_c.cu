// Transform kernels for lengths 576..1536 (see lmc_fft_impl.cuh;
// the radices are those of FFT_RADIX; FP32 butterflies take FFT_RADIX_F32).
#define LMC_FFT_NS fft_c
#include "lmc_fft_impl.cuh"
#define LMC_FFT_SIZES(X) X(576, 6, 8, 12) X(768, 12, 8, 8) X(1152, 12, 8, 12) X(1536, 12, 8, 16)
LMC_FFT_TU_BODY(c)
