// Lines with two or more odd factors: 144, 400, 576, 800, 1120, 1344, 1680, 2016, 2352, 2800, 3200
// cells.
#include "fft_kernels.cuh"

namespace bippb200 {

FftLinesKernel fft_seq_2(const int* radix, int ns, bool lineFast) {
  static const FftSeq table[] = {
    B2_FFT_SEQ(9, 16),
    B2_FFT_SEQ(5, 5, 16),
    B2_FFT_SEQ(9, 16, 4),
    B2_FFT_SEQ(5, 5, 8, 4),
    B2_FFT_SEQ(7, 5, 8, 4),
    B2_FFT_SEQ(7, 3, 16, 4),
    B2_FFT_SEQ(15, 7, 16),
    B2_FFT_SEQ(9, 7, 8, 4),
    B2_FFT_SEQ(7, 7, 3, 16),
    B2_FFT_SEQ(7, 5, 5, 16),
    B2_FFT_SEQ(5, 5, 16, 8),
  };
  return fft_find(table, radix, ns, lineFast);
}

}  // namespace bippb200
