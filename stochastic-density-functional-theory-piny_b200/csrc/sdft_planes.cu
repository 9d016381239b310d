// sdft_planes.cu -- plane kernels whose edges are chosen at run time among the
// compile-time plans (a warp-uniform switch per transform), and the stage
// dispatch of that path.
//
// A kernel per pair of edges would need 15 x 15 instances; switching inside
// the kernel costs two uniform branches per transform and the registers of
// the largest radix.  64 x 64 planes, 49 pairs, FP32, per launch: 58 us (an
// instance of their own 46.8, so the common pairs have one; the Stockham kernel
// with run-time radices 415).
#include <cuda_runtime.h>
#include <algorithm>
#include "sdft_kernels2.cuh"
#include "sdft_planes.cuh"

namespace sdft {

template <typename T, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
kf_stage_b_any(DevGeom g, typename CT<T>::type *__restrict__ X, const T *__restrict__ Vp) {
  using C2 = typename CT<T>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n1 = g.n1, n2 = g.n2, P2 = plane_pitch(n2), ka = g.kamax;
  int2 *rng = reinterpret_cast<int2 *>(smem_raw);
  C2 *pl = plane_of<C2>(smem_raw, n1);
  pdl_trigger();
  const int tid = threadIdx.x, r = blockIdx.x;
  plane_ranges<NT>(g, rng, pl, P2, tid);
  pdl_wait();
  __syncthreads();
  C2 *Xrow = X + ((size_t)blockIdx.y * g.n3 + r) * g.ncols_pad;
  plane_scatter<NT>(g, Xrow, pl, P2, tid);
  __syncthreads();
  const int g1 = (ka + 1 + 15) & ~15, g2 = (ka + 15) & ~15;
  const Lines2P rowsp{ka + 1, g1, ka, P2, (n1 - ka) * P2};
  switch (n2) {
#define SDFT_B(N)                                                                                             \
  case N:                                                                                                     \
    dif<N, 1, +1>(pl, rowsp, g1 + g2, TwC<N, C2>{}, tid, NT, RowKb<N>{rng, g1, n1 - ka});                     \
    break;
    SDFT_EDGES(SDFT_B)
#undef SDFT_B
  }
  const T *V = Vp + (size_t)r * n1 * n2;
  switch (n1) {
#define SDFT_A(N) \
  case N: plane_a_vmul<N>(pl, P2, n2, n2, V, ka, TwC<N, C2>{}, tid, NT); break;
    SDFT_EDGES(SDFT_A)
#undef SDFT_A
  }
  switch (n2) {
#define SDFT_B(N)                                                                                             \
  case N:                                                                                                     \
    dit<N, 1, -1>(pl, rowsp, g1 + g2, TwC<N, C2>{}, tid, NT, RowKb<N>{rng, g1, n1 - ka});                     \
    break;
    SDFT_EDGES(SDFT_B)
#undef SDFT_B
  }
  plane_gather<NT>(g, pl, Xrow, P2, tid);
}

// rows ka with |ka| <= kamax of a column line
template <int N1> struct ColKa {
  int kamax;
  struct In {
    int m;
    __device__ __forceinline__ bool operator()(int k) const { return k <= m || k >= N1 - m; }
  };
  __device__ __forceinline__ In line(int) const { return In{kamax}; }
};

// |psi1|^2 + |psi2|^2 of the pairs of group blockIdx.y on plane blockIdx.x,
// summed in pair order into part[group][plane][pa][pb]: each thread owns its
// points, so the sum over the group's pairs needs no other storage (the
// plane's 74 KB at 96 x 96 stay in L2).
template <int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
kf_density(DevGeom g, const double2 *__restrict__ X, int npairs, int groups, bool add, double *__restrict__ part) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n1 = g.n1, n2 = g.n2, P2 = plane_pitch(n2), ka = g.kamax;
  int2 *rng = reinterpret_cast<int2 *>(smem_raw);
  double2 *pl = plane_of<double2>(smem_raw, n1);
  const int tid = threadIdx.x, r = blockIdx.x, E = n1 * n2;
  const int p0 = (int)((long long)npairs * blockIdx.y / groups);
  const int p1 = (int)((long long)npairs * (blockIdx.y + 1) / groups);
  double *out = part + (size_t)blockIdx.y * g.N + (size_t)r * E;
  if (p0 == p1 && !add)
    for (int e = tid; e < E; e += NT) out[e] = 0.0;
  const Lines2 rows{ka + 1, P2, (n1 - ka) * P2};
  for (int p = p0; p < p1; p++) {
    plane_ranges<NT>(g, rng, pl, P2, tid);
    __syncthreads();
    plane_scatter<NT>(g, X + ((size_t)p * g.n3 + r) * g.ncols_pad, pl, P2, tid);
    __syncthreads();
    switch (n2) {
#define SDFT_B(N) \
  case N: dif<N, 1, +1>(pl, rows, 2 * ka + 1, TwC<N, double2>{}, tid, NT, RowKb<N>{rng, ka + 1, n1 - ka}); break;
      SDFT_EDGES(SDFT_B)
#undef SDFT_B
    }
    switch (n1) {
#define SDFT_A(N) \
  case N: dif<N, 0, +1>(pl, Lines1{1}, n2, TwC<N, double2>{}, tid, NT, ColKa<N>{ka}, P2); break;
      SDFT_EDGES(SDFT_A)
#undef SDFT_A
    }
    const bool first = p == p0 && !add;
    int a = tid / n2, b = tid - a * n2;
    const int da = NT / n2, db = NT - da * n2;
    for (int e = tid; e < E; e += NT) {
      const double2 v = pl[a * P2 + b];
      const double q = v.x * v.x + v.y * v.y;
      out[e] = first ? q : out[e] + q;
      a += da;
      b += db;
      if (b >= n2) { b -= n2; a++; }
    }
    __syncthreads();
  }
}

// groups summed in order, permuted plane order -> package layout (a fastest)
__global__ void kf_density_reduce(const double *__restrict__ part, int groups, int n1, int n2, int n3, PlanRt q1,
                                  PlanRt q2, PlanRt q3, double scale, double *__restrict__ rho) {
  const int N = n1 * n2 * n3;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int z = 0; z < groups; z++) s += part[(size_t)z * N + i];
    const int pb = i % n2, t = i / n2, pa = t % n1, r = t / n1;
    rho[q1.ipos(pa) + n1 * (q2.ipos(pb) + n2 * q3.ipos(r))] = s * scale;
  }
}

// sphere rows ka of a plane whose a-direction is in permuted order
struct RowsPermRt {
  int kamax, n1, ls;
  PlanRt q;
  __device__ __forceinline__ int base(int l) const { return q.pos(l <= kamax ? l : n1 - (2 * kamax + 1) + l) * ls; }
  __device__ __forceinline__ bool valid(int) const { return true; }
};

// +-sqrt(N) real fields of two orbitals -> a/b transforms to G
template <int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
kf_noise(DevGeom g, const unsigned char *__restrict__ neg, int nstate, int pair0, double2 *__restrict__ X, PlanRt q1,
         PlanRt q2, PlanRt q3) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n1 = g.n1, n2 = g.n2, P2 = plane_pitch(n2), E = n1 * n2;
  double2 *pl = plane_of<double2>(smem_raw, n1);
  const int tid = threadIdx.x, r = blockIdx.x;
  const int s1 = 2 * (pair0 + blockIdx.y);
  const bool has2 = s1 + 1 < nstate;
  const double rv = sqrt((double)g.N);
  const unsigned char *n1p = neg + (size_t)s1 * g.N + (size_t)q3.ipos(r) * E;
  const unsigned char *n2p = n1p + g.N;
  for (int e = tid; e < E; e += NT) {
    const int ib = e / n1, ia = e - ib * n1;
    pl[ia * P2 + ib] = make_double2(n1p[e] ? -rv : rv, has2 ? (n2p[e] ? -rv : rv) : 0.0);
  }
  __syncthreads();
  switch (n1) {
#define SDFT_A(N) \
  case N: dif<N, 0, -1>(pl, Lines1{1}, n2, TwC<N, double2>{}, tid, NT, AllElems{}, P2); break;
    SDFT_EDGES(SDFT_A)
#undef SDFT_A
  }
  const RowsPermRt rows{g.kamax, n1, P2, q1};
  switch (n2) {
#define SDFT_B(N) \
  case N: dif<N, 1, -1>(pl, rows, 2 * g.kamax + 1, TwC<N, double2>{}, tid, NT); break;
    SDFT_EDGES(SDFT_B)
#undef SDFT_B
  }
  double2 *Xrow = X + ((size_t)blockIdx.y * g.n3 + r) * g.ncols_pad;
  for (int col = tid; col < g.ncols; col += NT) {
    const int ab = g.col_ab[col];
    Xrow[col] = pl[q1.pos(ab >> 16) * P2 + q2.pos(ab & 0xffff)];
  }
}

// V_KS in the permuted plane order: Vp[r][pa][pb] = v[(ia*n2+ib)*n3+ic]
template <typename T>
__global__ void kf_vks_perm(const double *__restrict__ v, T *__restrict__ Vp, int n1, int n2, int n3, PlanRt q1,
                            PlanRt q2, PlanRt q3) {
  const size_t N = (size_t)n1 * n2 * n3;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x) {
    const int pb = (int)(i % n2);
    const int pa = (int)((i / n2) % n1);
    const int r = (int)(i / ((size_t)n1 * n2));
    Vp[i] = (T)v[((size_t)q1.ipos(pa) * n2 + q2.ipos(pb)) * n3 + q3.ipos(r)];
  }
}

// ---------------------------------------------------------------------------
// dispatch
// ---------------------------------------------------------------------------
bool fast_supported(int n1, int n2, int n3) { return plan_rt(n1).r1 && plan_rt(n2).r1 && plan_rt(n3).r1; }

template <typename T>
void fast_stage_a(const DevGeom &g, const double *C, int nstate, int pair0, int npairs, void *X, cudaStream_t st) {
  switch (g.n3) {
#define SDFT_C(N) \
  case N: cols_launch_a<T, N>(g, C, nstate, pair0, npairs, X, st); break;
    SDFT_EDGES(SDFT_C)
#undef SDFT_C
  }
}

template <typename T>
void fast_stage_c(const DevGeom &g, const void *X, const EpiArgs &e, int npairs, cudaStream_t st) {
  switch (g.n3) {
#define SDFT_C(N) \
  case N: cols_launch_c<T, N>(g, X, e, npairs, st); break;
    SDFT_EDGES(SDFT_C)
#undef SDFT_C
  }
}

constexpr int kMaxSmem = 227 * 1024;

template <typename T, int NT, int MINB>
static void launch_any_b(const DevGeom &g, void *X, const T *Vp, int npairs, cudaStream_t st) {
  auto k = kf_stage_b_any<T, NT, MINB>;
  static const bool attr_once = (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem), true);
  (void)attr_once;
  launch_pdl(g.early, k, dim3(g.n3, npairs), NT, plane_bytes<T>(g.n1, g.n2), st, g, (typename CT<T>::type *)X, Vp);
}

template <> void any_stage_b<float>(const DevGeom &g, void *X, const float *Vp, int npairs, cudaStream_t st) {
  if (g.plane_nt == 128) launch_any_b<float, 128, 6>(g, X, Vp, npairs, st);
  else launch_any_b<float, 256, 3>(g, X, Vp, npairs, st);
}
template <> void any_stage_b<double>(const DevGeom &g, void *X, const double *Vp, int npairs, cudaStream_t st) {
  if (plane_two_fit(plane_bytes<double>(g.n1, g.n2))) launch_any_b<double, 256, 2>(g, X, Vp, npairs, st);
  else launch_any_b<double, 512, 1>(g, X, Vp, npairs, st);
}

// Pair groups of the density: the pairs the busiest CTA slot works through, at
// 1.25 ns a plane point (96 x 96: 11.5 us a plane), against the groups' partial
// grids written and read once more by the reduction at 5 TB/s.
static int density_slots(const DevGeom &g) {
  return 148 * (plane_two_fit(plane_bytes<double>(g.n1, g.n2)) ? 2 : 1);
}
int fast_density_max_groups(const DevGeom &g, int npairs_max) {
  return std::min(npairs_max, (3 * density_slots(g) + g.n3 - 1) / g.n3);
}
int fast_density_groups(const DevGeom &g, int npairs) {
  const int slots = density_slots(g), lim = fast_density_max_groups(g, npairs);
  int best = 1;
  double best_cost = 1e300;
  for (int G = 1; G <= lim; G++) {
    const long long runs = (((long long)g.n3 * G + slots - 1) / slots) * ((npairs + G - 1) / G);
    const double cost = 1.25e-9 * g.n1 * g.n2 * (double)runs + 16.0 * g.N * (double)G / 5e12;
    if (cost < best_cost) { best_cost = cost; best = G; }
  }
  return best;
}

template <int NT, int MINB>
static void launch_density(const DevGeom &g, const void *X, int npairs, int groups, bool add, double *part,
                           cudaStream_t st) {
  auto k = kf_density<NT, MINB>;
  static const bool attr_once = (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem), true);
  (void)attr_once;
  k<<<dim3(g.n3, groups), NT, plane_bytes<double>(g.n1, g.n2), st>>>(g, (const double2 *)X, npairs, groups, add, part);
}

void fast_stage_b_density(const DevGeom &g, const void *X, int npairs, int groups, bool add, double *part,
                          cudaStream_t st) {
  if (plane_two_fit(plane_bytes<double>(g.n1, g.n2))) launch_density<256, 2>(g, X, npairs, groups, add, part, st);
  else launch_density<512, 1>(g, X, npairs, groups, add, part, st);
}

void fast_density_reduce(const DevGeom &g, const double *part, int groups, double scale, double *rho, cudaStream_t st) {
  const int blocks = std::min((g.N + 255) / 256, 148 * 16);
  kf_density_reduce<<<blocks, 256, 0, st>>>(part, groups, g.n1, g.n2, g.n3, plan_rt(g.n1), plan_rt(g.n2),
                                            plan_rt(g.n3), scale, rho);
}

template <int NT, int MINB>
static void launch_noise(const DevGeom &g, const unsigned char *neg, int nstate, int pair0, int npairs, void *X,
                         cudaStream_t st) {
  auto k = kf_noise<NT, MINB>;
  static const bool attr_once = (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem), true);
  (void)attr_once;
  k<<<dim3(g.n3, npairs), NT, plane_bytes<double>(g.n1, g.n2), st>>>(g, neg, nstate, pair0, (double2 *)X,
                                                                     plan_rt(g.n1), plan_rt(g.n2), plan_rt(g.n3));
}

void fast_stage_b_noise(const DevGeom &g, const unsigned char *neg, int nstate, int pair0, int npairs, void *X,
                        cudaStream_t st) {
  if (plane_two_fit(plane_bytes<double>(g.n1, g.n2))) launch_noise<256, 2>(g, neg, nstate, pair0, npairs, X, st);
  else launch_noise<512, 1>(g, neg, nstate, pair0, npairs, X, st);
}

template <typename T>
void fast_vks_perm(const DevGeom &g, const double *v, T *Vp, cudaStream_t st) {
  const int blocks = std::min((g.N + 255) / 256, 148 * 16);
  kf_vks_perm<T><<<blocks, 256, 0, st>>>(v, Vp, g.n1, g.n2, g.n3, plan_rt(g.n1), plan_rt(g.n2), plan_rt(g.n3));
}

template void fast_stage_a<double>(const DevGeom &, const double *, int, int, int, void *, cudaStream_t);
template void fast_stage_a<float>(const DevGeom &, const double *, int, int, int, void *, cudaStream_t);
template void fast_stage_c<double>(const DevGeom &, const void *, const EpiArgs &, int, cudaStream_t);
template void fast_stage_c<float>(const DevGeom &, const void *, const EpiArgs &, int, cudaStream_t);
template void fast_vks_perm<double>(const DevGeom &, const double *, double *, cudaStream_t);
template void fast_vks_perm<float>(const DevGeom &, const double *, float *, cudaStream_t);

}  // namespace sdft
