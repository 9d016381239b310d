// sdft_plane_b_f32.cu -- stage B instances, FP32 planes.
#include "sdft_plane_b.cuh"

namespace sdft {
template void fast_stage_b<float>(const DevGeom &, void *, const float *, int, cudaStream_t);
}  // namespace sdft
