// sdft_cols.cuh -- column stages A and C of the compile-time-edge path (the
// templates; sdft_cols_*.cu instantiate them edge by edge).
//
// A CTA owns CPB mirror pairs of sphere columns (2 CPB lines along c) of one
// orbital pair.  The lines live in one shared-memory buffer that every phase
// of stage C works on in place:
//   1. inverse c-transform, pass 1: a unit (line, k1) loads its R2 rows
//      straight from the column scratch into registers;
//   2. pass 2 (permuted -> natural kc);
//   3. the sphere's points (an item table lists them in CTA order): unpack,
//      kinetic term, KB force, recurrence, accumulation; the written pair is
//      packed back over the two elements the item read;
//   4. forward c-transform of the packed pair for the next application,
//      pass 1: elements outside the line's kc range count as zero, so nothing
//      is cleared;
//   5. pass 2, stored straight from registers to the column scratch.
// Stage A is phases 3 (packing only) to 5.
//
// Lines vary fastest over the threads, so a half-warp loads or stores 16
// consecutive columns of one row (one 128 B line in FP32), and with the odd
// line pitch consecutive lines fall in distinct banks.
#pragma once
#include <type_traits>
#include "sdft_fft2.cuh"
#include "sdft_kernels.cuh"
#include "sdft_pdl.cuh"
#include "sdft_tw_edges.cuh"

namespace sdft {

// Threads and resident CTAs of the column kernels.  Small CTAs: the phases
// are separated by barriers and each waits for its own loads, so what hides
// one CTA's wait is another CTA, not more threads of the same.  Stage C at
// 96^3, 256 pairs, FP32, per launch: 128 threads x 8 CTAs/SM (64 registers, 104
// bytes of spill loads a thread) 0.697 ms; x 7 and 6 0.743 and 0.758; 96 x 10 0.707; 64 x 16 with
// half the columns 0.709; 160 x 8 0.714; 192 x 8 0.791; 256 x 5 0.788;
// 256 x 6 (40 registers) 0.822.  The earlier form -- 256 x 6, two
// buffers, columns copied through shared memory before and after the
// transforms -- took 0.965 ms, 42.4 us at 48^3 and 64 pairs (28.7 now) and
// 65.7 us at N3 = 24 with moment dots (19.3 now).  (All before the order of the
// epilogue's loads, 682 -> 611 us, see epilogue_pair.)  Bound: 2.98 GB at 96^3,
// 4.9 TB/s, 0.75 of a copy; the waits for those loads.
// FP64: 128 x 5 46.5 us at 72^3 and 32 pairs, 256 x 3 53.3, 192 x 4 49.0.
template <typename T, int N3, int CPB> struct ColCfg {
  static constexpr int NL = 2 * CPB;
  static constexpr int NT = 128;
  static constexpr int MINB = sizeof(T) == 4 ? 8 : 5;
  static constexpr int P3 = N3 | 1;
};

enum ColKind : int { COL_STEP = 0, COL_DOTS = 1, COL_RAW = 2 };

// natural index k of an edge-N line holds data when its signed kc is in [lo, hi]
template <int N> __device__ __forceinline__ bool in_kc(int2 r, int k) {
  const int kc = k <= N / 2 ? k : k - N;
  return kc >= r.x && kc <= r.y;
}

// Forward c-transform of the CTA's lines, natural -> permuted rows stored to
// the column scratch (phases 4 and 5).
template <typename T, int N3, int CPB, typename C2 = typename CT<T>::type>
__device__ __forceinline__ void col_forward(C2 *buf, const int2 *rng, int ncl, C2 *Xo, int pitch, int tid) {
  using G = ColCfg<T, N3, CPB>;
  constexpr int R1 = Plan<N3>::R1, R2 = Plan<N3>::R2, NL = G::NL, NT = G::NT, P3 = G::P3;
  const TwC<N3, C2> tw{};
#pragma unroll 1
  for (int u = tid; u < NL * R2; u += NT) {
    const int l = u % NL, j2 = u / NL;
    if (l >= ncl) continue;
    C2 *p = buf + l * P3 + j2;
    const int2 r = rng[l];
    C2 v[R1];
#pragma unroll
    for (int j1 = 0; j1 < R1; j1++) v[j1] = in_kc<N3>(r, j2 + R2 * j1) ? p[R2 * j1] : cmk<C2>(0.0, 0.0);
    dftr<R1, +1>(v);
    p[0] = v[0];
#pragma unroll
    for (int k1 = 1; k1 < R1; k1++) {
      C2 w = tw(j2 * k1);
      w.y = -w.y;
      p[R2 * k1] = cmul(v[k1], w);
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int u = tid; u < NL * R1; u += NT) {
    const int l = u % NL, k1 = u / NL;
    if (l >= ncl) continue;
    const C2 *p = buf + l * P3 + R2 * k1;
    C2 v[R2];
#pragma unroll
    for (int j = 0; j < R2; j++) v[j] = p[j];
    dftr<R2, +1>(v);
    C2 *o = Xo + (size_t)(R2 * k1) * pitch + l;
#pragma unroll
    for (int j = 0; j < R2; j++) o[(size_t)j * pitch] = v[j];
  }
}

// One item: {G index, kd | km << 8 | line << 16 | mirror line << 24}, the
// sign bit set for G = 0.
struct ColItem {
  int gi, kd, km, lc, lm;
  bool g0;
  __device__ __forceinline__ explicit ColItem(int2 m)
      : gi(m.x), kd(m.y & 0xff), km((m.y >> 8) & 0xff), lc((m.y >> 16) & 0xff), lm((m.y >> 24) & 0x7f), g0(m.y < 0) {}
};

template <typename T, int N3, int CPB>
__global__ void __launch_bounds__(ColCfg<T, N3, CPB>::NT)
kf_stage_a(DevGeom g, const double *__restrict__ C, int nstate, int pair0, typename CT<T>::type *__restrict__ X) {
  using C2 = typename CT<T>::type;
  using G = ColCfg<T, N3, CPB>;
  constexpr int P3 = G::P3, NL = G::NL, NT = G::NT;
  __shared__ __align__(16) C2 buf[NL * P3];
  __shared__ int2 rng[NL];
  pdl_trigger();
  const int tid = threadIdx.x;
  const int col0 = NL * blockIdx.x;
  const int ncl = min(NL, g.ncols - col0);
  const int p = pair0 + blockIdx.y;
  const bool has2 = 2 * p + 1 < nstate;
  for (int i = tid; i < ncl; i += NT) rng[i] = g.kc_rng[col0 + i];
  if (!g.kc_contig) {
    for (int i = tid; i < ncl * P3; i += NT) buf[i] = cmk<C2>(0.0, 0.0);
    __syncthreads();
  }
  pdl_wait();
  const double *c1 = C + (size_t)(2 * p) * 2 * g.ngp, *c2 = c1 + 2 * (size_t)g.ngp;
  const int it1 = g.item_start[blockIdx.x + 1];
  for (int it = g.item_start[blockIdx.x] + tid; it < it1; it += NT) {
    const ColItem m(g.items[it]);
    const double a = c1[m.gi], b = m.g0 ? 0.0 : c1[g.ngp + m.gi];
    const double c = has2 ? c2[m.gi] : 0.0, d = has2 && !m.g0 ? c2[g.ngp + m.gi] : 0.0;
    if (!m.g0) buf[m.lm * P3 + m.km] = cmk<C2>(a + d, -b + c);
    buf[m.lc * P3 + m.kd] = cmk<C2>(a - d, b + c);
  }
  __syncthreads();
  col_forward<T, N3, CPB>(buf, rng, ncl, X + (size_t)blockIdx.y * N3 * g.ncols_pad + col0, g.ncols_pad, tid);
}

// Epilogue of both orbitals of a pair at G index gi: every load of both
// orbitals is issued before any store (OUT may alias PREV or C, so a load
// placed after a store could not be moved above it).  f1 / f2: the local
// forces; the written values return in (ar, ai), (br, bi).
struct Dots3 { double d0, d1, d2; };
template <int KIND>
__device__ __forceinline__ void epilogue_pair(const DevGeom &g, const EpiArgs &e, int s1, bool has2, int gi, bool g0,
                                              double f1r, double f1i, double f2r, double f2i, Dots3 &dt, double &mx1,
                                              double &mx2, double &ar, double &ai, double &br, double &bi) {
  const size_t n = g.ngp;
  const size_t o1 = (size_t)s1 * 2 * n + gi, o2 = o1 + 2 * n;
  if (KIND == COL_RAW && e.mode == EPI_NOISE) {
    ar = f1r; ai = f1i; br = f2r; bi = f2i;
  } else {
    const bool rec = KIND != COL_RAW && (e.mode == EPI_CHEBK || e.mode == EPI_MOMK);
    const bool acc1 = KIND != COL_RAW && e.ACC && e.nmu == 1 && !e.acoef0;
    const double w = g.ak2[gi];
    double c1r = e.C[o1], c1i = e.C[o1 + n], c2r = 0.0, c2i = 0.0;
    double x1r = 0.0, x1i = 0.0, x2r = 0.0, x2i = 0.0;
    double p1r = 0.0, p1i = 0.0, p2r = 0.0, p2i = 0.0;
    double q1r = 0.0, q1i = 0.0, q2r = 0.0, q2i = 0.0;
    if (has2) { c2r = e.C[o2]; c2i = e.C[o2 + n]; }
    if (rec) {
      p1r = e.PREV[o1]; p1i = e.PREV[o1 + n];
      if (has2) { p2r = e.PREV[o2]; p2i = e.PREV[o2 + n]; }
    }
    if (acc1) {
      q1r = e.ACC[o1]; q1i = e.ACC[o1 + n];
      if (has2) { q2r = e.ACC[o2]; q2i = e.ACC[o2 + n]; }
    }
    double h1r = 0.0, h1i = 0.0, h2r = 0.0, h2i = 0.0;
    if (KIND == COL_DOTS) {
      h1r = e.CHI[o1]; h1i = e.CHI[o1 + n];
      if (has2) { h2r = e.CHI[o2]; h2i = e.CHI[o2 + n]; }
    }
    // last: the FP32 values are widened inside the branch, which waits for them,
    // and no load after that wait is in flight with these (96^3, 256 pairs, this
    // block right after c: 682 us, here 611)
    if (e.FNLf) {
      x1r = e.FNLf[o1]; x1i = e.FNLf[o1 + n];
      if (has2) { x2r = e.FNLf[o2]; x2i = e.FNLf[o2 + n]; }
    } else if (e.FNL) {
      x1r = e.FNL[o1]; x1i = e.FNL[o1 + n];
      if (has2) { x2r = e.FNL[o2]; x2i = e.FNL[o2 + n]; }
    }
    const double k2 = g0 ? 0.0 : 2.0 * w;
    ar = f1r + x1r - k2 * c1r;
    br = f2r + x2r - k2 * c2r;
    ai = g0 ? 0.0 : f1i + x1i - k2 * c1i;
    bi = g0 ? 0.0 : f2i + x2i - k2 * c2i;
    if (KIND != COL_RAW) {
      const double sc = g0 ? e.s2 : e.s1;
      ar = sc * ar + e.pre * c1r;
      br = sc * br + e.pre * c2r;
      ai = g0 ? 0.0 : (e.s1 * ai + e.pre * c1i);
      bi = g0 ? 0.0 : (e.s1 * bi + e.pre * c2i);
      if (rec) {
        ar -= p1r;
        br -= p2r;
        if (!g0) { ai -= p1i; bi -= p2i; }
      }
    }
    if (KIND == COL_DOTS) {
      const double wr = g0 ? 1.0 : 2.0;
      dt.d0 += wr * h1r * ar + 2.0 * h1i * ai;
      if (has2) dt.d0 += wr * h2r * br + 2.0 * h2i * bi;
      if (e.mode == EPI_MOMK) {
        dt.d1 += wr * ar * c1r + 2.0 * ai * c1i;
        dt.d2 += wr * ar * ar + 2.0 * ai * ai;
        if (has2) {
          dt.d1 += wr * br * c2r + 2.0 * bi * c2i;
          dt.d2 += wr * br * br + 2.0 * bi * bi;
        }
      } else if (e.ndots > 1) {  // first step: <chi,chi>
        dt.d1 += wr * h1r * h1r + 2.0 * h1i * h1i;
        if (has2) dt.d1 += wr * h2r * h2r + 2.0 * h2i * h2i;
      }
    }
    if (KIND != COL_RAW && e.ACC) {
      if (acc1) {
        const double a = e.acoef[0];
        const double ap = e.acoefp ? e.acoefp[0] : 0.0;
        e.ACC[o1] = q1r + ap * c1r + a * ar;
        e.ACC[o1 + n] = q1i + ap * c1i + a * ai;
        if (has2) {
          e.ACC[o2] = q2r + ap * c2r + a * br;
          e.ACC[o2 + n] = q2i + ap * c2i + a * bi;
        }
      } else {
        for (int k = 0; k < (has2 ? 2 : 1); k++) {
          const size_t o = k ? o2 : o1;
          const double cr = k ? c2r : c1r, ci = k ? c2i : c1i, nr = k ? br : ar, ni = k ? bi : ai;
          for (int imu = 0; imu < e.nmu; imu++) {
            double *A = e.ACC + imu * e.acc_stride;
            const double a = e.acoef[imu];
            if (e.acoef0) {
              const double a0 = e.acoef0[imu];
              A[o] = a0 * cr + a * nr;
              A[o + n] = a0 * ci + a * ni;
            } else if (e.acoefp) {
              const double ap = e.acoefp[imu];
              A[o] += ap * cr + a * nr;
              A[o + n] += ap * ci + a * ni;
            } else {
              A[o] += a * nr;
              A[o + n] += a * ni;
            }
          }
        }
      }
    }
  }
  e.OUT[o1] = ar;
  e.OUT[o1 + n] = ai;
  mx1 = fmax(mx1, fmax(absmax_key_d(ar), absmax_key_d(ai)));
  if (has2) {
    e.OUT[o2] = br;
    e.OUT[o2 + n] = bi;
    mx2 = fmax(mx2, fmax(absmax_key_d(br), absmax_key_d(bi)));
  } else {
    br = bi = 0.0;  // an odd count's empty partner stays exactly zero
  }
}

// X is not __restrict__: with e.Xnext the CTA overwrites its own columns of
// the same scratch (read into shared memory in phase 1) for the next step.
template <typename T, int N3, int CPB, int KIND>
__global__ void __launch_bounds__(ColCfg<T, N3, CPB>::NT, ColCfg<T, N3, CPB>::MINB)
kf_stage_c(DevGeom g, const typename CT<T>::type *X, EpiArgs e) {
  using C2 = typename CT<T>::type;
  using G = ColCfg<T, N3, CPB>;
  constexpr int R1 = Plan<N3>::R1, R2 = Plan<N3>::R2, P3 = G::P3, NL = G::NL, NT = G::NT, NW = NT / 32;
  __shared__ __align__(16) C2 buf[NL * P3];
  __shared__ int2 rng[NL];
  __shared__ double red[KIND == COL_DOTS ? NW : 1][3], mred[NW][2];
  pdl_trigger();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int col0 = NL * blockIdx.x;
  const int ncl = min(NL, g.ncols - col0);
  const int s1 = 2 * (e.pair0 + blockIdx.y);
  const bool has2 = s1 + 1 < e.nstate;
  const size_t xoff = (size_t)blockIdx.y * N3 * g.ncols_pad + col0;
  const TwC<N3, C2> tw{};
  if (e.Xnext)
    for (int i = tid; i < ncl; i += NT) rng[i] = g.kc_rng[col0 + i];
  pdl_wait();
  {
    const C2 *Xp = X + xoff;
#pragma unroll 1
    for (int u = tid; u < NL * R1; u += NT) {  // phase 1
      const int l = u % NL, k1 = u / NL;
      if (l >= ncl) continue;
      const C2 *src = Xp + (size_t)(R2 * k1) * g.ncols_pad + l;
      C2 v[R2];
#pragma unroll
      for (int j = 0; j < R2; j++) v[j] = src[(size_t)j * g.ncols_pad];
      dftr<R2, -1>(v);
      C2 *p = buf + l * P3 + R2 * k1;
      p[0] = v[0];
#pragma unroll
      for (int j2 = 1; j2 < R2; j2++) p[j2] = cmul(v[j2], tw(j2 * k1));
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int u = tid; u < NL * R2; u += NT) {  // phase 2
    const int l = u % NL, j2 = u / NL;
    if (l >= ncl) continue;
    C2 *p = buf + l * P3 + j2;
    C2 v[R1];
#pragma unroll
    for (int k1 = 0; k1 < R1; k1++) v[k1] = p[R2 * k1];
    dftr<R1, -1>(v);
#pragma unroll
    for (int j1 = 0; j1 < R1; j1++) p[R2 * j1] = v[j1];
  }
  __syncthreads();
  Dots3 dt{0.0, 0.0, 0.0};
  double mx1 = 0.0, mx2 = 0.0;
  {
    const double sg = (KIND == COL_RAW && e.mode == EPI_NOISE) ? -0.5 : -2.0;
    const bool noise = KIND == COL_RAW && e.mode == EPI_NOISE;
    const int it1 = g.item_start[blockIdx.x + 1];
    for (int it = g.item_start[blockIdx.x] + tid; it < it1; it += NT) {  // phase 3
      const ColItem m(g.items[it]);
      C2 *pd = buf + m.lc * P3 + m.kd, *pm = buf + m.lm * P3 + m.km;
      const C2 F = *pd, Fm = *pm;
      const double tr = (double)F.x * e.invN, ti = (double)F.y * e.invN;
      const double trc = (double)Fm.x * e.invN, tic = (double)Fm.y * e.invN;
      double f1r = sg * (tr + trc), f1i = sg * (ti - tic), f2r = sg * (ti + tic), f2i = sg * (trc - tr);
      if (m.g0) {
        f1r = (noise ? -1.0 : -2.0) * tr;
        f2r = (noise ? -1.0 : -2.0) * ti;
        f1i = f2i = 0.0;
      }
      double ar, ai, br = 0.0, bi = 0.0;
      epilogue_pair<KIND>(g, e, s1, has2, m.gi, m.g0, f1r, f1i, f2r, f2i, dt, mx1, mx2, ar, ai, br, bi);
      if (e.Xnext) {  // stage A's packing of the pair (c1 + i c2) at +kc and -kc
        if (!m.g0) *pm = cmk<C2>(ar + bi, -ai + br);
        *pd = cmk<C2>(ar - bi, ai + br);
      }
    }
  }
  if (e.omax) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mx1 = fmax(mx1, __shfl_xor_sync(0xffffffffu, mx1, o));
      mx2 = fmax(mx2, __shfl_xor_sync(0xffffffffu, mx2, o));
    }
    if (lane == 0) { mred[warp][0] = mx1; mred[warp][1] = mx2; }
  }
  if (KIND == COL_DOTS) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      dt.d0 += __shfl_down_sync(0xffffffffu, dt.d0, off);
      dt.d1 += __shfl_down_sync(0xffffffffu, dt.d1, off);
      dt.d2 += __shfl_down_sync(0xffffffffu, dt.d2, off);
    }
    if (lane == 0) { red[warp][0] = dt.d0; red[warp][1] = dt.d1; red[warp][2] = dt.d2; }
  }
  __syncthreads();
  if (e.omax && tid < 2 && (tid == 0 || has2)) {
    double m = mred[0][tid];
    for (int w = 1; w < NW; w++) m = fmax(m, mred[w][tid]);
    atomicMax(e.omax + s1 + tid, (unsigned long long)__double_as_longlong(m));
  }
  if (KIND == COL_DOTS && tid < 3) {
    double a = 0.0;
    for (int w = 0; w < NW; w++) a += red[w][tid];
    e.dots[((size_t)(s1 >> 1) * g.nbatch + blockIdx.x) * 3 + tid] = a;
  }
  if (e.Xnext) col_forward<T, N3, CPB>(buf, rng, ncl, reinterpret_cast<C2 *>(e.Xnext) + xoff, g.ncols_pad, tid);
}

template <typename T, int N3, int CPB>
void cols_launch_a_n(const DevGeom &g, const double *C, int nstate, int pair0, int npairs, void *X, cudaStream_t st) {
  launch_pdl(g.early, kf_stage_a<T, N3, CPB>, dim3(g.nbatch, npairs), ColCfg<T, N3, CPB>::NT, 0, st, g, C, nstate, pair0,
             (typename CT<T>::type *)X);
}

template <typename T, int N3, int CPB>
void cols_launch_c_n(const DevGeom &g, const void *X, const EpiArgs &e, int npairs, cudaStream_t st) {
  using C2 = typename CT<T>::type;
  const dim3 grid(g.nbatch, npairs);
  constexpr int NT = ColCfg<T, N3, CPB>::NT;
  if (e.mode == EPI_HPSI || e.mode == EPI_NOISE) launch_pdl(g.early, kf_stage_c<T, N3, CPB, COL_RAW>, grid, NT, 0, st, g, (const C2 *)X, e);
  else if (e.dots) launch_pdl(g.early, kf_stage_c<T, N3, CPB, COL_DOTS>, grid, NT, 0, st, g, (const C2 *)X, e);
  else launch_pdl(g.early, kf_stage_c<T, N3, CPB, COL_STEP>, grid, NT, 0, st, g, (const C2 *)X, e);
}

// the CPB instance that the context's item table was made for
template <typename T, int N3>
void cols_launch_a(const DevGeom &g, const double *C, int nstate, int pair0, int npairs, void *X, cudaStream_t st) {
  constexpr int CPB = col_cpb(N3);
  if constexpr (CPB > kCPBSmall)
    if (g.cpb == kCPBSmall) return cols_launch_a_n<T, N3, kCPBSmall>(g, C, nstate, pair0, npairs, X, st);
  cols_launch_a_n<T, N3, CPB>(g, C, nstate, pair0, npairs, X, st);
}
template <typename T, int N3>
void cols_launch_c(const DevGeom &g, const void *X, const EpiArgs &e, int npairs, cudaStream_t st) {
  constexpr int CPB = col_cpb(N3);
  if constexpr (CPB > kCPBSmall)
    if (g.cpb == kCPBSmall) return cols_launch_c_n<T, N3, kCPBSmall>(g, X, e, npairs, st);
  cols_launch_c_n<T, N3, CPB>(g, X, e, npairs, st);
}

}  // namespace sdft
