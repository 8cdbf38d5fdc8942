// fft_tma.cu -- the FP32 tile passes (fft_tma.cuh) and the host parts that
// both data types share.
#include "fft_tma.cuh"

namespace mth {

template <typename T>
cudaError_t tma_probe(int on);
extern template cudaError_t tma_probe<double>(int);
MTH_TMA_INST(float)

cudaError_t tma_set_wait_probe(int on) {
  cudaError_t e = tma_probe<float>(on);
  return e == cudaSuccess ? tma_probe<double>(on) : e;
}
void tma_destroy(TmaMaps* t) { delete t; }
bool tma_has(const TmaMaps* t, int pass) { return t && (pass == 0 ? t->z : pass == 1 ? t->s : t->g); }
int tma_tile_choice(bool fp32, int pass, int i) {
  static const int w[2][2][3] = {{{2, 4, 8}, {1, 2, 4}}, {{8, 16, 32}, {2, 4, 8}}};
  return w[fp32 ? 1 : 0][pass == 1 ? 0 : 1][i];
}
void tma_tiles(const TmaMaps* t, int* ks, int* kg) {
  *ks = t ? t->ks : 0;
  *kg = t ? t->kg : 0;
}

}  // namespace mth
