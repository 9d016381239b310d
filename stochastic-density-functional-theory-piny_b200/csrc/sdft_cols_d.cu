// sdft_cols_d.cu -- column stages of the edges 54, 64, 81.
#include "sdft_kernels2.cuh"
#include "sdft_cols.cuh"

namespace sdft {
#define SDFT_COLS(N)                                                                                        \
  template void cols_launch_a<float, N>(const DevGeom &, const double *, int, int, int, void *, cudaStream_t);  \
  template void cols_launch_a<double, N>(const DevGeom &, const double *, int, int, int, void *, cudaStream_t); \
  template void cols_launch_c<float, N>(const DevGeom &, const void *, const EpiArgs &, int, cudaStream_t);     \
  template void cols_launch_c<double, N>(const DevGeom &, const void *, const EpiArgs &, int, cudaStream_t);
SDFT_COLS(54)
SDFT_COLS(64)
SDFT_COLS(81)
}  // namespace sdft
