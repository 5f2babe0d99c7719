// k_fft_m.cu -- register FFTs (k_fft.cuh) of the lengths 8 ... 162 = 2^a 3^b that k_fft.cu
// does not have.  Against the Stockham transforms they took before (one shared-memory round
// trip per radix and run-time index arithmetic): 216x108x95 mixed, x-FFT with divergence 36 ->
// 13 us, y-FFT 13 -> 5, inverse x-FFT 26 -> 7.6.
#include "k_fft.cuh"

namespace tc {

#define TC_FFT_SIZES(X) X(8) X(12) X(18) X(36) X(54) X(72) X(108) X(144) X(162)
TC_FFT_LENGTHS(m, TC_FFT_SIZES)

}  // namespace tc
