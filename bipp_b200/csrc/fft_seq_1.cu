// Powers of two, alone and after one odd radix.
#include "fft_kernels.cuh"

namespace bippb200 {

FftLinesKernel fft_seq_1(const int* radix, int ns, bool lineFast) {
  static const FftSeq table[] = {
    B2_FFT_SEQ(4, 4),
    B2_FFT_SEQ(8, 4),
    B2_FFT_SEQ(16, 4),
    B2_FFT_SEQ(16, 8),
    B2_FFT_SEQ(16, 16),
    B2_FFT_SEQ(16, 8, 4),
    B2_FFT_SEQ(16, 16, 4),
    B2_FFT_SEQ(3, 16),
    B2_FFT_SEQ(3, 8, 4),
    B2_FFT_SEQ(3, 16, 4),
    B2_FFT_SEQ(3, 16, 8),
    B2_FFT_SEQ(3, 16, 16),
    B2_FFT_SEQ(3, 16, 8, 4),
    B2_FFT_SEQ(3, 16, 16, 4),
    B2_FFT_SEQ(5, 16),
    B2_FFT_SEQ(5, 8, 4),
    B2_FFT_SEQ(5, 16, 4),
    B2_FFT_SEQ(5, 16, 8),
    B2_FFT_SEQ(5, 16, 16),
    B2_FFT_SEQ(5, 16, 8, 4),
    B2_FFT_SEQ(5, 16, 16, 4),
    B2_FFT_SEQ(7, 16),
    B2_FFT_SEQ(7, 8, 4),
    B2_FFT_SEQ(7, 16, 4),
    B2_FFT_SEQ(7, 16, 8),
    B2_FFT_SEQ(7, 16, 16),
    B2_FFT_SEQ(7, 16, 8, 4),
    B2_FFT_SEQ(7, 16, 16, 4),
  };
  return fft_find(table, radix, ns, lineFast);
}

}  // namespace bippb200
