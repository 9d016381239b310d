// sdft_cols_a.cu -- column stages of the edges 12, 24, 48.
#include "sdft_kernels2.cuh"
#include "sdft_cols.cuh"

namespace sdft {
#define SDFT_COLS(N)                                                                                        \
  template void cols_launch_a<float, N>(const DevGeom &, const double *, int, int, int, void *, cudaStream_t);  \
  template void cols_launch_a<double, N>(const DevGeom &, const double *, int, int, int, void *, cudaStream_t); \
  template void cols_launch_c<float, N>(const DevGeom &, const void *, const EpiArgs &, int, cudaStream_t);     \
  template void cols_launch_c<double, N>(const DevGeom &, const void *, const EpiArgs &, int, cudaStream_t);
SDFT_COLS(12)
SDFT_COLS(24)
SDFT_COLS(48)
}  // namespace sdft
