// sdft_xc.h -- the LDA exchange-correlation step on a stream (sdft_xc.cu).
#pragma once
#include <cuda_runtime.h>

namespace sdft {

constexpr int kXcBlocks = 592, kXcScratch = 3 * kXcBlocks;
// vks += V_xc(rho) over n points; sums[0..3) = sum x rho, sum c rho, sum V_xc rho;
// scratch: kXcScratch doubles
void launch_xc_lda(int kind, long long n, const double *rho, double *vks, double *scratch, double *sums,
                   cudaStream_t st);
// E_xc and sum V_xc rho from the sums, times scale = vol / n
inline void xc_energies(const double *sums, double scale, double *exc, double *muxc) {
  *exc = (0.75 * sums[0] + sums[1]) * scale;
  *muxc = sums[2] * scale;
}

}  // namespace sdft
