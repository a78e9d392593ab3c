// Lines with two or more odd factors: 336, 560, 784, 1008, 1296, 1600, 2000, 2304, 2688, 3136,
// 3600 cells.
#include "fft_kernels.cuh"

namespace bippb200 {

FftLinesKernel fft_seq_5(const int* radix, int ns, bool lineFast) {
  static const FftSeq table[] = {
    B2_FFT_SEQ(7, 3, 16),
    B2_FFT_SEQ(7, 5, 16),
    B2_FFT_SEQ(7, 7, 16),
    B2_FFT_SEQ(9, 7, 16),
    B2_FFT_SEQ(9, 9, 16),
    B2_FFT_SEQ(5, 5, 16, 4),
    B2_FFT_SEQ(5, 5, 5, 16),
    B2_FFT_SEQ(9, 16, 16),
    B2_FFT_SEQ(7, 3, 16, 8),
    B2_FFT_SEQ(7, 7, 16, 4),
    B2_FFT_SEQ(15, 15, 16),
  };
  return fft_find(table, radix, ns, lineFast);
}

}  // namespace bippb200
