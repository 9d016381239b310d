// sdft_plane_b.cuh -- stage B of the plane edge pairs with an instance of their
// own (instantiated per precision in sdft_plane_b_f32.cu and _f64.cu).
//
// Same stage split as sdft_kernels.cu (A: pack + c-FFT, B: plane FFTs x V,
// C: c-FFT + unpack/epilogue; A and C are in sdft_cols.cuh) but every 1-D
// transform is the two-pass factorised FFT of sdft_fft2.cuh:
//   stage A writes the c-transformed columns in the permuted real-space
//   order r = pos_N3(ic) (X row r);
//   stage B forward-transforms b then a (natural -> permuted), multiplies by
//   V stored in the same permuted order, and transforms back a then b
//   (permuted -> natural);
//   stage C transforms X rows r back to natural kc (permuted -> natural).
// So no data movement is ever spent on undoing an FFT permutation.
#pragma once
#include <cuda_runtime.h>
#include <type_traits>
#include "sdft_kernels2.cuh"
#include "sdft_planes.cuh"

namespace sdft {

// ---------------------------------------------------------------------------
// plane stages
// ---------------------------------------------------------------------------
// NT threads per plane CTA: FP32 256 at 3 CTAs/SM, or the 128-thread instance
// that the default rule and the autotuner take for smaller planes; FP64 256
// where two planes fit an SM's shared memory, 512 (at one) above.  FP64 at
// 72 x 72, 32 pairs: 512 threads x 1 168 us, 256 x 2 117, 128 x 4 143; 24 x 24,
// 8 pairs: 7.2, 4.7 and 5.0 us; at 96 x 96 (one CTA) 512 threads lead by 7 %.
// PM (DevGeom::prune34): 1 = the sphere is narrower than 3/8 of both plane
// edges (R1 = 8 plans): the j1 = 3, 4 band of the first forward and last
// inverse passes is skipped; 2 = also at least a quarter of N1 wide, so the
// a-pass tests only the rows with j1 = 2, 5.
template <typename T, int N1, int N2> struct PlaneCfg {
  static constexpr bool two = plane_two_fit(plane_bytes<T>(N1, N2));
  static constexpr int NT = sizeof(T) == 4 || two ? 256 : 512;
  static constexpr int MINB = sizeof(T) == 4 ? 3 : (two ? 2 : 1);
};
template <typename T, int N1, int N2, int NT, int MINB, int PM>
__global__ void __launch_bounds__(NT, MINB)
kf_stage_b(DevGeom g, typename CT<T>::type *__restrict__ X, const T *__restrict__ Vp) {
  using C2 = typename CT<T>::type;
  constexpr int P2 = plane_pitch(N2);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int2 *rng = reinterpret_cast<int2 *>(smem_raw);
  C2 *pl = plane_of<C2>(smem_raw, N1);
  pdl_trigger();
  const int tid = threadIdx.x;
  const int r = blockIdx.x;
  const int ka = g.kamax;
  plane_ranges<NT>(g, rng, pl, P2, tid);
  pdl_wait();
  __syncthreads();
  C2 *Xrow = X + ((size_t)blockIdx.y * g.n3 + r) * g.ncols_pad;
  plane_scatter<NT>(g, Xrow, pl, P2, tid);
  __syncthreads();
  // b-transforms over the sphere rows, each row group padded to 16 lanes
  const int g1 = (ka + 1 + 15) & ~15, g2 = (ka + 15) & ~15;
  const Lines2P rowsp{ka + 1, g1, ka, P2, (N1 - ka) * P2};
  // only the sphere's elements are read before and written after the b-transforms
  const RowKb<N2> m{rng, g1, N1 - ka};
  dif<N2, 1, +1, (PM >= 1)>(pl, rowsp, g1 + g2, TwC<N2, C2>{}, tid, NT, m);
  plane_a_vmul<N1, PM>(pl, P2, N2, N2, Vp + (size_t)r * N1 * N2, ka, TwC<N1, C2>{}, tid, NT);
  dit<N2, 1, -1, (PM >= 1)>(pl, rowsp, g1 + g2, TwC<N2, C2>{}, tid, NT, m);
  plane_gather<NT>(g, pl, Xrow, P2, tid);
}

// ---------------------------------------------------------------------------
// dispatch
// ---------------------------------------------------------------------------
// Plane edges with instances of their own: the 24-per-cell grids of one to
// three cells per axis and 96 x 96, and the density grids' 32 and 64 and their
// pairs with 96.  Every other pair -- also an uneven cell's 96 with 24, 48 or 72 --
// takes the run-time-edge kernel (sdft_planes.cu), which pays for its row pitch
// and the registers of the largest radix: 64 x 64, 49 pairs, FP32, 58.0 us there
// and 46.8 here (the only pair timed both ways).
#define SDFT_FOR_PLANE(X)                                                     \
  do {                                                                        \
    switch (g.n1 * 1000 + g.n2) {                                             \
      case 24024: X(24, 24); break;                                           \
      case 24048: X(24, 48); break;                                           \
      case 24072: X(24, 72); break;                                           \
      case 48024: X(48, 24); break;                                           \
      case 48048: X(48, 48); break;                                           \
      case 48072: X(48, 72); break;                                           \
      case 72024: X(72, 24); break;                                           \
      case 72048: X(72, 48); break;                                           \
      case 72072: X(72, 72); break;                                           \
      case 96096: X(96, 96); break;                                           \
      case 32032: X(32, 32); break;                                           \
      case 32064: X(32, 64); break;                                           \
      case 64032: X(64, 32); break;                                           \
      case 64064: X(64, 64); break;                                           \
      case 32096: X(32, 96); break;                                           \
      case 96032: X(96, 32); break;                                           \
      case 64096: X(64, 96); break;                                           \
      case 96064: X(96, 64); break;                                           \
      default: any_stage_b<T>(g, Xs, Vp, npairs, st);                         \
    }                                                                         \
  } while (0)

template <typename T, int A, int B, int NT, int MINB, int PM>
static void launch_plane_b(const DevGeom &g, dim3 grid, void *X, const T *Vp, cudaStream_t st) {
  constexpr size_t sm = plane_bytes<T>(A, B);
  auto k = kf_stage_b<T, A, B, NT, MINB, PM>;
  static const bool attr_once = (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm), true);
  (void)attr_once;
  launch_pdl(g.early, k, grid, NT, sm, st, g, (typename CT<T>::type *)X, Vp);
}

template <typename T>
void fast_stage_b(const DevGeom &g, void *Xs, const T *Vp, int npairs, cudaStream_t st) {
  dim3 grid(g.n3, npairs);
  [[maybe_unused]] const bool small = g.plane_nt == 128;
  // the j1 = 3, 4 band skipped where both edges factor with R1 = 8 and the
  // sphere is narrower than 3/8 of them (DevGeom::prune34)
#define LBP(NT_, MB_)                                                                                     \
  do {                                                                                                    \
    if (pm == 2) launch_plane_b<T, A, B, NT_, MB_, (ok34 ? 2 : 0)>(g, grid, Xs, Vp, st);               \
    else if (pm == 1) launch_plane_b<T, A, B, NT_, MB_, (ok34 ? 1 : 0)>(g, grid, Xs, Vp, st);          \
    else launch_plane_b<T, A, B, NT_, MB_, 0>(g, grid, Xs, Vp, st);                                    \
  } while (0)
#define LB(A_, B_)                                                                                        \
  do {                                                                                                    \
    constexpr int A = A_, B = B_;                                                                         \
    using Cfg = PlaneCfg<T, A, B>;                                                                        \
    constexpr bool ok34 = Plan<A>::R1 == 8 && Plan<B>::R1 == 8;                                           \
    const int pm = ok34 ? g.prune34 : 0;                                                                  \
    if constexpr (std::is_same<T, float>::value) {                                                        \
      if (small) LBP(128, 6);                                                                             \
      else LBP(Cfg::NT, Cfg::MINB);                                                                       \
    } else {                                                                                              \
      LBP(Cfg::NT, Cfg::MINB);                                                                            \
    }                                                                                                     \
  } while (0)
  SDFT_FOR_PLANE(LB);
#undef LB
#undef LBP
}

}  // namespace sdft
