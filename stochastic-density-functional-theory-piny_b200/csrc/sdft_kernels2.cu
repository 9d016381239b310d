// sdft_kernels2.cu -- fast-path FFT stages with compile-time grid edges.
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
#include <cuda_runtime.h>
#include <cmath>
#include <type_traits>
#include "sdft_fft2.cuh"
#include "sdft_internal.h"
#include "sdft_kernels.cuh"
#include "sdft_kernels2.cuh"
#include "sdft_tw_edges.cuh"

namespace sdft {

template <typename T> __device__ __forceinline__ const typename CT<T>::type *twp(const DevGeom &g, int d);
template <> __device__ __forceinline__ const double2 *twp<double>(const DevGeom &g, int d) {
  return d == 1 ? g.tw1 : (d == 2 ? g.tw2 : g.tw3);
}
template <> __device__ __forceinline__ const float2 *twp<float>(const DevGeom &g, int d) {
  return d == 1 ? g.tw1f : (d == 2 ? g.tw2f : g.tw3f);
}

// ---------------------------------------------------------------------------
// plane stages
// ---------------------------------------------------------------------------
template <typename T> struct PlaneCfg;
template <> struct PlaneCfg<double> { static constexpr int NT = 512, MINB = 1; };
template <> struct PlaneCfg<float> { static constexpr int NT = 256, MINB = 3; };

// natural row ka -> line index helper for the rows touched by the sphere
template <int N1> struct RowsPerm {  // rows given in permuted-a order
  int kamax, ls;
  __device__ __forceinline__ int base(int l) const {
    const int ka = (l <= kamax) ? l : N1 - (2 * kamax + 1) + l;
    return pos<N1>(ka) * ls;
  }
  __device__ __forceinline__ bool valid(int) const { return true; }
};

// a-direction transform pair of one plane with the V multiply fused in:
// forward a-FFT (natural -> permuted) of the N2 columns, times V (stored in
// the permuted order, Vpl[pa*N2 + pb]), inverse a-FFT (permuted -> natural).
// The second forward pass and the first inverse pass work on the same
// R2-blocks of a column, so one register-resident unit does
// DFT -> x V -> inverse DFT without a round trip through shared memory.
// Rows with kamax < ka < N1 - kamax are zero on input (outside the sphere)
// and not needed on output: they are neither read nor written.
// PM >= 1: rows ka in the j1 = 3, 4 band (|ka| >= 3 N1/8, outside a sphere
// narrower than that) are skipped at compile time, with no activity test.
// PM == 2: the sphere is also at least N1/4 wide, so the rows with j1 = 0,
// 1, 6, 7 are always inside it and only j1 = 2, 5 are tested.
template <int N1, int PM = 0, typename C2, typename T, typename TW>
__device__ __forceinline__ void plane_a_vmul(C2 *pl, int P2, int nl, int N2, const T *__restrict__ Vpl, int kamax,
                                             const TW &tw1, int tid, int nthr) {
  constexpr int R1 = Plan<N1>::R1, R2 = Plan<N1>::R2;
  constexpr bool P34 = PM >= 1;
  static_assert(!P34 || R1 == 8, "the j1 = 3, 4 band needs R1 = 8");
  auto active_ka = [&](int ka) { return ka <= kamax || ka >= N1 - kamax; };
  // row ka = j2 + R2 j1 holds data (j1 a compile-time constant after unrolling)
  auto active_j = [&](int j1, int ka) {
    if (band34<R1>(P34, j1)) return false;
    if (PM == 2 && (j1 == 0 || j1 == 1 || j1 == 6 || j1 == 7)) return true;
    return active_ka(ka);
  };
#pragma unroll 1
  for (UnitIter it(tid, nthr, nl); it.j < R2; it.next()) {  // forward pass 1
    const int l = it.l, j2 = it.j;
    C2 *p = pl + l;
    C2 v[R1];
#pragma unroll
    for (int j1 = 0; j1 < R1; j1++) {
      const int ka = j2 + R2 * j1;
      v[j1] = active_j(j1, ka) ? p[ka * P2] : cmk<C2>(0.0, 0.0);
    }
    dftr<R1, +1>(v);
    p[j2 * P2] = v[0];
#pragma unroll
    for (int k1 = 1; k1 < R1; k1++) {
      C2 w = tw_at<C2>(tw1, j2 * k1);
      w.y = -w.y;
      p[(j2 + R2 * k1) * P2] = cmul(v[k1], w);
    }
  }
  __syncthreads();
#pragma unroll 1
  for (UnitIter it(tid, nthr, nl); it.j < R1; it.next()) {  // forward pass 2, x V, inverse pass 1
    const int l = it.l, k1 = it.j;
    C2 *p = pl + R2 * k1 * P2 + l;
    const T *vp = Vpl + (size_t)R2 * k1 * N2 + l;
    C2 v[R2];
#pragma unroll
    for (int j = 0; j < R2; j++) v[j] = p[j * P2];
    dftr<R2, +1>(v);
#pragma unroll
    for (int j = 0; j < R2; j++) v[j] = cscale(v[j], vp[(size_t)j * N2]);
    dftr<R2, -1>(v);
    p[0] = v[0];
#pragma unroll
    for (int j2 = 1; j2 < R2; j2++) p[j2 * P2] = cmul(v[j2], tw_at<C2>(tw1, j2 * k1));
  }
  __syncthreads();
#pragma unroll 1
  for (UnitIter it(tid, nthr, nl); it.j < R2; it.next()) {  // inverse pass 2
    const int l = it.l, j2 = it.j;
    C2 *p = pl + l;
    C2 v[R1];
#pragma unroll
    for (int k1 = 0; k1 < R1; k1++) v[k1] = p[(R2 * k1 + j2) * P2];
    dftr<R1, -1>(v);
#pragma unroll
    for (int j1 = 0; j1 < R1; j1++) {
      const int ka = j2 + R2 * j1;
      if (active_j(j1, ka)) p[ka * P2] = v[j1];
    }
  }
  __syncthreads();
}

// Sphere rows of a plane as b-lines (Lines2P order): line l < g1 is row l,
// line l >= g1 is row base2 + l - g1; element k of a line holds data when
// its signed kb lies in the row's column range.
template <int N2> struct RowKb {
  const int2 *rng;
  int g1, base2;
  struct In {
    int lo, hi;
    __device__ __forceinline__ bool operator()(int k) const {
      const int kb = k <= N2 / 2 ? k : k - N2;
      return kb >= lo && kb <= hi;
    }
  };
  __device__ __forceinline__ In line(int l) const {
    const int2 r = rng[l < g1 ? l : base2 + (l - g1)];
    return In{r.x, r.y};
  }
};

// NT threads per plane CTA: PlaneCfg's default, or (FP32) the 128-thread
// instance that the autotuner may pick for small planes (more resident CTAs).
// PM (DevGeom::prune34): 1 = the sphere is narrower than 3/8 of both plane
// edges (R1 = 8 plans): the j1 = 3, 4 band of the first forward and last
// inverse passes is skipped; 2 = also at least a quarter of N1 wide, so the
// a-pass tests only the rows with j1 = 2, 5.
template <typename T, int N1, int N2, int NT = PlaneCfg<T>::NT, int MINB = PlaneCfg<T>::MINB, int PM = 0>
__global__ void __launch_bounds__(NT, MINB)
kf_stage_b(DevGeom g, typename CT<T>::type *__restrict__ X, const T *__restrict__ Vp) {
  using C2 = typename CT<T>::type;
  constexpr int P2 = N2 + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // (the first N1 + N2 complex slots held twiddles before they moved to
  // constant memory; the row kb ranges use the first N1 of them)
  int2 *rng = reinterpret_cast<int2 *>(smem_raw);
  C2 *pl = reinterpret_cast<C2 *>(smem_raw) + N1 + N2;
  const int tid = threadIdx.x;
  const int r = blockIdx.x;
  const int ka = g.kamax;
  const bool contig = g.kb_contig != 0;
  if (contig) {
    for (int t = tid; t < N1; t += NT) rng[t] = g.kb_rng[t];
  } else {
    // zero the 2 kamax + 1 rows inside the sphere's a-range
    const Lines2 rows{ka + 1, P2, (N1 - ka) * P2};
    for (int i = tid; i < (2 * ka + 1) * N2; i += NT) {
      const int l = i / N2, b = i - l * N2;
      pl[rows.base(l) + b] = cmk<C2>(0.0, 0.0);
    }
  }
  __syncthreads();
  C2 *Xrow = X + ((size_t)blockIdx.y * g.n3 + r) * g.ncols_pad;
  for (int col = tid; col < g.ncols; col += NT) {
    const int ab = g.col_ab[col];
    pl[(ab >> 16) * P2 + (ab & 0xffff)] = Xrow[col];
  }
  __syncthreads();
  // b-transforms over the sphere rows, each row group padded to 16 lanes
  const int g1 = (ka + 1 + 15) & ~15, g2 = (ka + 15) & ~15;
  const Lines2P rowsp{ka + 1, g1, ka, P2, (N1 - ka) * P2};
  if (contig) {  // only the sphere's elements are read before and written after the b-transforms
    const RowKb<N2> m{rng, g1, N1 - ka};
    dif<N2, 1, +1, (PM >= 1)>(pl, rowsp, g1 + g2, TwC<N2, C2>{}, tid, NT, m);
    plane_a_vmul<N1, PM>(pl, P2, N2, N2, Vp + (size_t)r * N1 * N2, ka, TwC<N1, C2>{}, tid, NT);
    dit<N2, 1, -1, (PM >= 1)>(pl, rowsp, g1 + g2, TwC<N2, C2>{}, tid, NT, m);
  } else {
    dif<N2, 1, +1, (PM >= 1)>(pl, rowsp, g1 + g2, TwC<N2, C2>{}, tid, NT);
    plane_a_vmul<N1, PM>(pl, P2, N2, N2, Vp + (size_t)r * N1 * N2, ka, TwC<N1, C2>{}, tid, NT);
    dit<N2, 1, -1, (PM >= 1)>(pl, rowsp, g1 + g2, TwC<N2, C2>{}, tid, NT);
  }
  for (int col = tid; col < g.ncols; col += NT) {
    const int ab = g.col_ab[col];
    Xrow[col] = pl[(ab >> 16) * P2 + (ab & 0xffff)];
  }
}

template <typename T, int N1, int N2>
__global__ void __launch_bounds__(PlaneCfg<T>::NT, PlaneCfg<T>::MINB)
kf_stage_b_density(DevGeom g, const typename CT<T>::type *__restrict__ X, double *__restrict__ rho_pair,
                   int r3_1, int r3_2) {
  using C2 = typename CT<T>::type;
  constexpr int NT = PlaneCfg<T>::NT, P2 = N2 + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C2 *tw1 = reinterpret_cast<C2 *>(smem_raw);
  C2 *tw2 = tw1 + N1;
  C2 *pl = tw2 + N2;
  const int tid = threadIdx.x;
  const int r = blockIdx.x;
  const int ic = (r % r3_2) * r3_1 + r / r3_2;
  {
    const C2 *t1 = twp<T>(g, 1), *t2 = twp<T>(g, 2);
    for (int t = tid; t < N1; t += NT) tw1[t] = t1[t];
    for (int t = tid; t < N2; t += NT) tw2[t] = t2[t];
  }
  for (int i = tid; i < N1 * P2; i += NT) pl[i] = cmk<C2>(0.0, 0.0);
  __syncthreads();
  const C2 *Xrow = X + ((size_t)blockIdx.y * g.n3 + r) * g.ncols_pad;
  for (int col = tid; col < g.ncols; col += NT) {
    const int ab = g.col_ab[col];
    pl[(ab >> 16) * P2 + (ab & 0xffff)] = Xrow[col];
  }
  __syncthreads();
  const int ka = g.kamax;
  dif<N2, 1, +1>(pl, Lines2{ka + 1, P2, (N1 - ka) * P2}, 2 * ka + 1, tw2, tid, NT);
  dif<N1, P2, +1>(pl, Lines1{1}, N2, tw1, tid, NT);
  double *out = rho_pair + (size_t)blockIdx.y * g.N + (size_t)ic * N1 * N2;
  for (int e = tid; e < N1 * N2; e += NT) {
    const int ib = e / N1, ia = e - ib * N1;
    const C2 v = pl[pos<N1>(ia) * P2 + pos<N2>(ib)];
    out[e] = (double)v.x * (double)v.x + (double)v.y * (double)v.y;
  }
}

template <typename T, int N1, int N2>
__global__ void __launch_bounds__(PlaneCfg<T>::NT, PlaneCfg<T>::MINB)
kf_stage_b_noise(DevGeom g, const unsigned char *__restrict__ neg, int nstate, int pair0,
                 typename CT<T>::type *__restrict__ X, int r3_1, int r3_2) {
  using C2 = typename CT<T>::type;
  constexpr int NT = PlaneCfg<T>::NT, P2 = N2 + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C2 *tw1 = reinterpret_cast<C2 *>(smem_raw);
  C2 *tw2 = tw1 + N1;
  C2 *pl = tw2 + N2;
  const int tid = threadIdx.x;
  const int r = blockIdx.x;
  const int ic = (r % r3_2) * r3_1 + r / r3_2;
  const int p = pair0 + blockIdx.y;
  const int s1 = 2 * p, s2 = 2 * p + 1;
  const bool has2 = s2 < nstate;
  {
    const C2 *t1 = twp<T>(g, 1), *t2 = twp<T>(g, 2);
    for (int t = tid; t < N1; t += NT) tw1[t] = t1[t];
    for (int t = tid; t < N2; t += NT) tw2[t] = t2[t];
  }
  const double rv = sqrt((double)g.N);
  constexpr int E = N1 * N2;
  const unsigned char *n1p = neg + (size_t)s1 * g.N + (size_t)ic * E;
  const unsigned char *n2p = neg + (size_t)s2 * g.N + (size_t)ic * E;
  for (int e = tid; e < E; e += NT) {
    const int ib = e / N1, ia = e - ib * N1;
    const double v1 = n1p[e] ? -rv : rv;
    const double v2 = has2 ? (n2p[e] ? -rv : rv) : 0.0;
    pl[ia * P2 + ib] = cmk<C2>(v1, v2);
  }
  __syncthreads();
  const int ka = g.kamax;
  dif<N1, P2, -1>(pl, Lines1{1}, N2, tw1, tid, NT);
  dif<N2, 1, -1>(pl, RowsPerm<N1>{ka, P2}, 2 * ka + 1, tw2, tid, NT);
  C2 *Xrow = X + ((size_t)blockIdx.y * g.n3 + r) * g.ncols_pad;
  for (int col = tid; col < g.ncols; col += NT) {
    const int ab = g.col_ab[col];
    Xrow[col] = pl[pos<N1>(ab >> 16) * P2 + pos<N2>(ab & 0xffff)];
  }
}

// V_KS in the permuted plane order: Vp[r][pa][pb] = v[(ia*n2+ib)*n3+ic]
// with ia = ipos_N1(pa), ib = ipos_N2(pb), ic = ipos_N3(r).
template <typename T, int N1, int N2, int N3>
__global__ void kf_vks_perm(const double *__restrict__ v, T *__restrict__ Vp) {
  const size_t N = (size_t)N1 * N2 * N3;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x) {
    const int pb = (int)(i % N2);
    const int pa = (int)((i / N2) % N1);
    const int r = (int)(i / ((size_t)N1 * N2));
    const int ia = ipos<N1>(pa), ib = ipos<N2>(pb), ic = ipos<N3>(r);
    Vp[i] = (T)v[((size_t)ia * N2 + ib) * N3 + ic];
  }
}

// ---------------------------------------------------------------------------
// dispatch
// ---------------------------------------------------------------------------
template <int N> static constexpr int r1_of() { return Plan<N>::R1; }

template <typename T> static size_t pl_smem(int n1, int n2) {
  return sizeof(typename CT<T>::type) * (size_t)(n1 + n2 + n1 * (n2 + 1));
}

#define SDFT_FOR_N3(X)                \
  switch (g.n3) {                     \
    case 24: X(24); break;            \
    case 48: X(48); break;            \
    case 72: X(72); break;            \
    case 96: X(96); break;            \
    default: return false;            \
  }

#define SDFT_FOR_PLANE(X)                                             \
  do {                                                                \
    const int key = g.n1 * 1000 + g.n2;                               \
    switch (key) {                                                    \
      case 24024: X(24, 24); break;                                   \
      case 24048: X(24, 48); break;                                   \
      case 24072: X(24, 72); break;                                   \
      case 48024: X(48, 24); break;                                   \
      case 48048: X(48, 48); break;                                   \
      case 48072: X(48, 72); break;                                   \
      case 72024: X(72, 24); break;                                   \
      case 72048: X(72, 48); break;                                   \
      case 72072: X(72, 72); break;                                   \
      case 96096: X(96, 96); break;                                   \
      default: return false;                                          \
    }                                                                 \
  } while (0)

bool fast_supported(int n1, int n2, int n3) {
  auto ok = [](int n) { return n == 24 || n == 48 || n == 72 || n == 96; };
  if (!ok(n1) || !ok(n2) || !ok(n3)) return false;
  const int key = n1 * 1000 + n2;
  switch (key) {
    case 24024: case 24048: case 24072: case 48024: case 48048: case 48072:
    case 72024: case 72048: case 72072: case 96096: return true;
    default: return false;
  }
}

static void plan3(int n3, int &r1, int &r2) {
  switch (n3) {
    case 24: r1 = Plan<24>::R1; r2 = Plan<24>::R2; break;
    case 48: r1 = Plan<48>::R1; r2 = Plan<48>::R2; break;
    case 72: r1 = Plan<72>::R1; r2 = Plan<72>::R2; break;
    default: r1 = Plan<96>::R1; r2 = Plan<96>::R2; break;
  }
}

template <typename T>
bool fast_stage_a(const DevGeom &g, const double *C, int nstate, int pair0, int npairs, void *X, cudaStream_t st) {
#define LA(N) cols_launch_a<T, N>(g, C, nstate, pair0, npairs, X, st)
  SDFT_FOR_N3(LA);
#undef LA
  return true;
}

template <typename T>
bool fast_stage_c(const DevGeom &g, const void *X, const EpiArgs &e, int npairs, cudaStream_t st) {
#define LC(N) cols_launch_c<T, N>(g, X, e, npairs, st)
  SDFT_FOR_N3(LC);
#undef LC
  return true;
}

template <typename T, int A, int B, int NT, int MINB, int PM>
static void launch_plane_b(const DevGeom &g, dim3 grid, size_t sm, void *X, const T *Vp, cudaStream_t st) {
  auto k = kf_stage_b<T, A, B, NT, MINB, PM>;
  static const bool attr_once = (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm), true);
  (void)attr_once;
  k<<<grid, NT, sm, st>>>(g, (typename CT<T>::type *)X, Vp);
}

template <typename T>
bool fast_stage_b(const DevGeom &g, void *X, const T *Vp, int npairs, cudaStream_t st) {
  dim3 grid(g.n3, npairs);
  const size_t sm = pl_smem<T>(g.n1, g.n2);
  [[maybe_unused]] const bool small = g.plane_nt == 128;
  // the j1 = 3, 4 band skipped where both edges factor with R1 = 8 and the
  // sphere is narrower than 3/8 of them (DevGeom::prune34)
#define LBP(NT_, MB_)                                                                                     \
  do {                                                                                                    \
    if (pm == 2) launch_plane_b<T, A, B, NT_, MB_, (ok34 ? 2 : 0)>(g, grid, sm, X, Vp, st);               \
    else if (pm == 1) launch_plane_b<T, A, B, NT_, MB_, (ok34 ? 1 : 0)>(g, grid, sm, X, Vp, st);          \
    else launch_plane_b<T, A, B, NT_, MB_, 0>(g, grid, sm, X, Vp, st);                                    \
  } while (0)
#define LB(A_, B_)                                                                                        \
  do {                                                                                                    \
    constexpr int A = A_, B = B_;                                                                         \
    constexpr bool ok34 = Plan<A>::R1 == 8 && Plan<B>::R1 == 8;                                           \
    const int pm = ok34 ? g.prune34 : 0;                                                                  \
    if constexpr (std::is_same<T, float>::value) {                                                        \
      if (small) LBP(128, 6);                                                                             \
      else LBP(PlaneCfg<T>::NT, PlaneCfg<T>::MINB);                                                       \
    } else {                                                                                              \
      LBP(PlaneCfg<T>::NT, PlaneCfg<T>::MINB);                                                            \
    }                                                                                                     \
  } while (0)
  SDFT_FOR_PLANE(LB);
#undef LB
#undef LBP
  return true;
}

template <typename T>
bool fast_stage_b_density(const DevGeom &g, const void *X, int npairs, double *rho_pair, cudaStream_t st) {
  dim3 grid(g.n3, npairs);
  const size_t sm = pl_smem<T>(g.n1, g.n2);
  int r1, r2;
  plan3(g.n3, r1, r2);
#define LD(A, B)                                                                               \
  do {                                                                                         \
    auto k = kf_stage_b_density<T, A, B>;                                                      \
    static const bool attr_once = (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm), true); (void)attr_once;             \
    k<<<grid, PlaneCfg<T>::NT, sm, st>>>(g, (const typename CT<T>::type *)X, rho_pair, r1, r2); \
  } while (0)
  SDFT_FOR_PLANE(LD);
#undef LD
  return true;
}

template <typename T>
bool fast_stage_b_noise(const DevGeom &g, const unsigned char *neg, int nstate, int pair0, int npairs, void *X,
                        cudaStream_t st) {
  dim3 grid(g.n3, npairs);
  const size_t sm = pl_smem<T>(g.n1, g.n2);
  int r1, r2;
  plan3(g.n3, r1, r2);
#define LN(A, B)                                                                                        \
  do {                                                                                                  \
    auto k = kf_stage_b_noise<T, A, B>;                                                                 \
    static const bool attr_once = (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm), true); (void)attr_once;                      \
    k<<<grid, PlaneCfg<T>::NT, sm, st>>>(g, neg, nstate, pair0, (typename CT<T>::type *)X, r1, r2);   \
  } while (0)
  SDFT_FOR_PLANE(LN);
#undef LN
  return true;
}

template <typename T>
bool fast_vks_perm(const DevGeom &g, const double *v, T *Vp, cudaStream_t st) {
  const size_t N = (size_t)g.n1 * g.n2 * g.n3;
  int blocks = (int)std::min<size_t>((N + 255) / 256, 148 * 16);
#define LV3(A, B, Cc) kf_vks_perm<T, A, B, Cc><<<blocks, 256, 0, st>>>(v, Vp)
#define LV(A, B)                                            \
  do {                                                      \
    switch (g.n3) {                                         \
      case 24: LV3(A, B, 24); break;                        \
      case 48: LV3(A, B, 48); break;                        \
      case 72: LV3(A, B, 72); break;                        \
      case 96: LV3(A, B, 96); break;                        \
      default: return false;                                \
    }                                                       \
  } while (0)
  SDFT_FOR_PLANE(LV);
#undef LV
#undef LV3
  return true;
}

template bool fast_stage_a<double>(const DevGeom &, const double *, int, int, int, void *, cudaStream_t);
template bool fast_stage_a<float>(const DevGeom &, const double *, int, int, int, void *, cudaStream_t);
template bool fast_stage_c<double>(const DevGeom &, const void *, const EpiArgs &, int, cudaStream_t);
template bool fast_stage_c<float>(const DevGeom &, const void *, const EpiArgs &, int, cudaStream_t);
template bool fast_stage_b<double>(const DevGeom &, void *, const double *, int, cudaStream_t);
template bool fast_stage_b<float>(const DevGeom &, void *, const float *, int, cudaStream_t);
template bool fast_stage_b_density<double>(const DevGeom &, const void *, int, double *, cudaStream_t);
template bool fast_stage_b_density<float>(const DevGeom &, const void *, int, double *, cudaStream_t);
template bool fast_stage_b_noise<double>(const DevGeom &, const unsigned char *, int, int, int, void *, cudaStream_t);
template bool fast_stage_b_noise<float>(const DevGeom &, const unsigned char *, int, int, int, void *, cudaStream_t);
template bool fast_vks_perm<double>(const DevGeom &, const double *, double *, cudaStream_t);
template bool fast_vks_perm<float>(const DevGeom &, const double *, float *, cudaStream_t);

}  // namespace sdft
