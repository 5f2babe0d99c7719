// k_fft_l.cu -- register FFTs (k_fft.cuh) of the lengths 216 ... 972 = 2^a 3^b that k_fft.cu
// does not have.  Against the Stockham transforms they took before (one shared-memory round
// trip per radix and run-time index arithmetic): 216x108x95 mixed, x-FFT with divergence 36 ->
// 13 us, y-FFT 13 -> 5, inverse x-FFT 26 -> 7.6.
#include "k_fft.cuh"

namespace tc {

#define TC_FFT_SIZES(X) X(216) X(288) X(324) X(432) X(486) X(576) X(648) X(864) X(972)
TC_FFT_LENGTHS(l, TC_FFT_SIZES)

}  // namespace tc
