// sdft_planes.cuh -- pieces shared by the plane kernels (compile-time edge
// pairs in sdft_plane_b.cuh, run-time pairs in sdft_planes.cu).
#pragma once
#include "sdft_fft2.cuh"
#include "sdft_kernels.cuh"
#include "sdft_pdl.cuh"
#include "sdft_tw_edges.cuh"

namespace sdft {

// Dynamic shared memory of a plane CTA: the rows' kb ranges, then the plane
// with an odd row pitch.
__host__ __device__ constexpr int plane_pitch(int n2) { return n2 | 1; }
template <typename T> constexpr size_t plane_bytes(int n1, int n2) {
  return sizeof(typename CT<T>::type) * (size_t)((n1 + 1) / 2 * (sizeof(T) == 4 ? 2 : 1) + n1 * plane_pitch(n2));
}
template <typename C2> __device__ __forceinline__ C2 *plane_of(unsigned char *smem, int n1) {
  return reinterpret_cast<C2 *>(smem) + (n1 + 1) / 2 * (sizeof(C2) == 8 ? 2 : 1);
}
// whether two CTAs of a plane fit an SM (228 KB, 1 KB of it per CTA)
constexpr bool plane_two_fit(size_t bytes) { return 2 * (bytes + 1024) <= 228 * 1024; }

// The kb ranges of the plane's rows (kept in shared memory); when the columns
// do not fill them, the sphere rows of the plane are cleared and every
// element counts as in range.
template <int NT, typename C2>
__device__ __forceinline__ void plane_ranges(const DevGeom &g, int2 *rng, C2 *pl, int P2, int tid) {
  const bool contig = g.kb_contig != 0;
  for (int t = tid; t < g.n1; t += NT) rng[t] = contig ? g.kb_rng[t] : make_int2(-g.n2, g.n2);
  if (!contig) {
    const Lines2 rows{g.kamax + 1, P2, (g.n1 - g.kamax) * P2};
    for (int i = tid; i < (2 * g.kamax + 1) * g.n2; i += NT) {
      const int l = i / g.n2, b = i - l * g.n2;
      pl[rows.base(l) + b] = cmk<C2>(0.0, 0.0);
    }
  }
}
template <int NT, typename C2>
__device__ __forceinline__ void plane_scatter(const DevGeom &g, const C2 *Xrow, C2 *pl, int P2, int tid) {
  for (int col = tid; col < g.ncols; col += NT) {
    const int ab = g.col_ab[col];
    pl[(ab >> 16) * P2 + (ab & 0xffff)] = Xrow[col];
  }
}
template <int NT, typename C2>
__device__ __forceinline__ void plane_gather(const DevGeom &g, const C2 *pl, C2 *Xrow, int P2, int tid) {
  for (int col = tid; col < g.ncols; col += NT) {
    const int ab = g.col_ab[col];
    Xrow[col] = pl[(ab >> 16) * P2 + (ab & 0xffff)];
  }
}

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
    dftr<R1, +1, P34>(v);
    p[j2 * P2] = v[0];
#pragma unroll
    for (int k1 = 1; k1 < R1; k1++) {
      C2 w = tw1(j2 * k1);
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
    for (int j2 = 1; j2 < R2; j2++) p[j2 * P2] = cmul(v[j2], tw1(j2 * k1));
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

}  // namespace sdft
