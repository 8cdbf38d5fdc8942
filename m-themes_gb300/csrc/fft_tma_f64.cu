// fft_tma_f64.cu -- the FP64 tile passes (fft_tma.cuh).
#include "fft_tma.cuh"

namespace mth {
MTH_TMA_INST(double)
}  // namespace mth
