// sdft_plane_b_f64.cu -- stage B instances, FP64 planes.
#include "sdft_plane_b.cuh"

namespace sdft {
template void fast_stage_b<double>(const DevGeom &, void *, const double *, int, cudaStream_t);
}  // namespace sdft
