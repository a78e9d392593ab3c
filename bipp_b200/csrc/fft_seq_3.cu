// Lines with two or more odd factors: 240, 432, 672, 864, 1152, 1440, 1728, 2160, 2400, 2880, 3360
// cells.
#include "fft_kernels.cuh"

namespace bippb200 {

FftLinesKernel fft_seq_3(const int* radix, int ns, bool lineFast) {
  static const FftSeq table[] = {
    B2_FFT_SEQ(15, 16),
    B2_FFT_SEQ(9, 3, 16),
    B2_FFT_SEQ(7, 3, 8, 4),
    B2_FFT_SEQ(9, 3, 8, 4),
    B2_FFT_SEQ(9, 16, 8),
    B2_FFT_SEQ(15, 3, 8, 4),
    B2_FFT_SEQ(9, 3, 16, 4),
    B2_FFT_SEQ(15, 9, 16),
    B2_FFT_SEQ(15, 5, 8, 4),
    B2_FFT_SEQ(15, 3, 16, 4),
    B2_FFT_SEQ(15, 7, 8, 4),
  };
  return fft_find(table, radix, ns, lineFast);
}

}  // namespace bippb200
