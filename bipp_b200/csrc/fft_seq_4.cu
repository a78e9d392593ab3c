// Lines with two or more odd factors: 288, 480, 720, 960, 1200, 1568, 1920, 2240, 2592, 3024, 3456
// cells.
#include "fft_kernels.cuh"

namespace bippb200 {

FftLinesKernel fft_seq_4(const int* radix, int ns, bool lineFast) {
  static const FftSeq table[] = {
    B2_FFT_SEQ(9, 8, 4),
    B2_FFT_SEQ(15, 8, 4),
    B2_FFT_SEQ(15, 3, 16),
    B2_FFT_SEQ(15, 16, 4),
    B2_FFT_SEQ(15, 5, 16),
    B2_FFT_SEQ(7, 7, 8, 4),
    B2_FFT_SEQ(15, 16, 8),
    B2_FFT_SEQ(7, 5, 16, 4),
    B2_FFT_SEQ(9, 9, 8, 4),
    B2_FFT_SEQ(9, 7, 3, 16),
    B2_FFT_SEQ(9, 3, 16, 8),
  };
  return fft_find(table, radix, ns, lineFast);
}

}  // namespace bippb200
