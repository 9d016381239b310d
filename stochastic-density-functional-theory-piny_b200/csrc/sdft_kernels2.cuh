// sdft_kernels2.cuh -- stage launches of the path whose line transforms have
// compile-time plans: every edge in SDFT_EDGES (12 to 128), any three of them.
// Other edges take the run-time-size kernels of sdft_kernels.cu.
#pragma once
#include "sdft_kernels.cuh"

namespace sdft {
bool fast_supported(int n1, int n2, int n3);
// column stages of edge N3 (sdft_cols.cuh, instantiated in sdft_cols_*.cu)
template <typename T, int N3>
void cols_launch_a(const DevGeom &g, const double *C, int nstate, int pair0, int npairs, void *X, cudaStream_t st);
template <typename T, int N3>
void cols_launch_c(const DevGeom &g, const void *X, const EpiArgs &e, int npairs, cudaStream_t st);
template <typename T>
void fast_stage_a(const DevGeom &g, const double *C, int nstate, int pair0, int npairs, void *X, cudaStream_t st);
template <typename T>
void fast_stage_b(const DevGeom &g, void *X, const T *Vp, int npairs, cudaStream_t st);
// stage B of any pair of edges (fast_stage_b calls it where it has no own instance)
template <typename T>
void any_stage_b(const DevGeom &g, void *X, const T *Vp, int npairs, cudaStream_t st);
template <typename T>
void fast_stage_c(const DevGeom &g, const void *X, const EpiArgs &e, int npairs, cudaStream_t st);
// Density (FP64 in every precision): the npairs pairs in X, dealt out over
// `groups` partial grids part[groups][N] in the permuted plane order (add: onto
// what earlier pairs left there); then the groups summed in order, times scale,
// into the package layout.
int fast_density_groups(const DevGeom &g, int npairs);
// the most groups that fast_density_groups returns for up to npairs_max pairs
int fast_density_max_groups(const DevGeom &g, int npairs_max);
void fast_stage_b_density(const DevGeom &g, const void *X, int npairs, int groups, bool add, double *part,
                          cudaStream_t st);
void fast_density_reduce(const DevGeom &g, const double *part, int groups, double scale, double *rho, cudaStream_t st);
// noise planes (FP64 in every precision)
void fast_stage_b_noise(const DevGeom &g, const unsigned char *neg, int nstate, int pair0, int npairs, void *X,
                        cudaStream_t st);
template <typename T>
void fast_vks_perm(const DevGeom &g, const double *v, T *Vp, cudaStream_t st);
}  // namespace sdft
