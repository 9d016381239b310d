// sdft_fft2.cuh -- compile-time-size line FFTs for the fast path.
//
// A line of N = R1*R2 points is transformed in two passes over shared
// memory (the "four-step" factorisation N = R1 x R2 without the explicit
// transpose):
//
//   forward, natural -> permuted ("DIF" order, dif()):
//     pass 1, per (line, j2):  R1-point DFT of x[j2 + R2*j1] over j1, times
//                              w_N^(j2*k1), stored back at j2 + R2*k1
//     pass 2, per (line, k1):  R2-point DFT of the block R2*k1 + [0,R2),
//                              stored back in place
//     -> frequency k1 + R1*k2 ends up at position R2*k1 + k2.
//   reverse, permuted -> natural ("DIT" order, dit()): the two passes in
//     the opposite order with the same twiddles; either sign.
//
// Every unit reads and writes only its own positions, so a pass needs no
// barrier between its loads and stores (no butterflies held across a
// barrier, low register pressure); one __syncthreads separates the passes.
// Consumers index the permuted order directly (pos()/ipos()), so no data is
// ever moved just to undo the permutation.  The R-point DFTs run in
// registers with compile-time twiddles (sdft_twiddles.cuh).
#pragma once
#include "sdft_fft.cuh"
#include "sdft_twiddles.cuh"

namespace sdft {

// R1 x R2 of every edge with a compile-time plan
template <int N> struct Plan;
#define SDFT_PLAN(N, A, B) \
  template <> struct Plan<N> { static constexpr int R1 = A, R2 = B; };
SDFT_PLAN(12, 4, 3)
SDFT_PLAN(16, 4, 4)
SDFT_PLAN(18, 3, 6)
SDFT_PLAN(24, 4, 6)
SDFT_PLAN(27, 3, 9)
SDFT_PLAN(32, 4, 8)
SDFT_PLAN(36, 6, 6)
SDFT_PLAN(48, 8, 6)
SDFT_PLAN(54, 6, 9)
SDFT_PLAN(64, 8, 8)
SDFT_PLAN(72, 8, 9)
SDFT_PLAN(81, 9, 9)
SDFT_PLAN(96, 8, 12)
SDFT_PLAN(108, 9, 12)
SDFT_PLAN(128, 8, 16)
#undef SDFT_PLAN
// X(N) for every such edge
#define SDFT_EDGES(X) \
  X(12) X(16) X(18) X(24) X(27) X(32) X(36) X(48) X(54) X(64) X(72) X(81) X(96) X(108) X(128)

// the plan of edge n at run time (r1 = 0: no plan)
struct PlanRt {
  int r1, r2;
  // position of index k after a dif() pass pair, and the index at position p
  __host__ __device__ __forceinline__ int pos(int k) const { return r2 * (k % r1) + k / r1; }
  __host__ __device__ __forceinline__ int ipos(int p) const { return (p % r2) * r1 + p / r2; }
};
inline PlanRt plan_rt(int n) {
  switch (n) {
#define SDFT_P(N) case N: return PlanRt{Plan<N>::R1, Plan<N>::R2};
    SDFT_EDGES(SDFT_P)
#undef SDFT_P
    default: return PlanRt{0, 0};
  }
}

template <int R> __device__ __forceinline__ double twc_re(int t);
template <int R> __device__ __forceinline__ double twc_im(int t);
#define SDFT_TW(R)                                                                         \
  template <> __device__ __forceinline__ double twc_re<R>(int t) { return kTw##R##re[t]; } \
  template <> __device__ __forceinline__ double twc_im<R>(int t) { return kTw##R##im[t]; }
SDFT_TW(9)
SDFT_TW(16)
#undef SDFT_TW

// The register DFTs count instructions, not only flops: the plane stage is
// bound by issue slots.  A packed f32x2 add is one slot but two cycles of the
// FP32 pipe (measured: 37.0 T element-adds/s packed, 36.2 scalar), and an
// operand that needs its halves swapped, negated or duplicated first costs
// moves; so plain complex adds and subtracts are packed, and everything with
// a rotation or a twiddle is scalar, fused into multiply-adds where it can be.

// a + DIR i b and a - DIR i b
template <int DIR, typename C> __device__ __forceinline__ C add_i(C a, C b) {
  C r;
  if (DIR > 0) { r.x = a.x - b.y; r.y = a.y + b.x; } else { r.x = a.x + b.y; r.y = a.y - b.x; }
  return r;
}
template <int DIR, typename C> __device__ __forceinline__ C sub_i(C a, C b) { return add_i<-DIR>(a, b); }
// a + s b with s = exp(DIR 2 pi i/8) sqrt(2) b folded in: g = b (1 + DIR i)
template <int DIR, typename C> __device__ __forceinline__ C rot8(C b) { return add_i<DIR>(b, b); }
__device__ __forceinline__ double2 axpy(double s, double2 x, double2 y) { return make_double2(fma(s, x.x, y.x), fma(s, x.y, y.y)); }
__device__ __forceinline__ float2 axpy(float s, float2 x, float2 y) { return make_float2(fmaf(s, x.x, y.x), fmaf(s, x.y, y.y)); }
// w b with the compile-time twiddle w = exp(DIR 2 pi i e/R)
template <int R, int DIR, typename C> __device__ __forceinline__ C twmul(C b, int e) {
  using T = decltype(b.x);
  if (e == 0) return b;
  if (4 * e == R) return mul_i<DIR>(b);
  if (8 * e == R || 8 * e == 3 * R) {  // (+-1 + DIR i) / sqrt(2)
    const T h = (T)0.70710678118654752440084436210485;
    const C g = 8 * e == R ? rot8<DIR>(b) : mul_i<DIR>(rot8<DIR>(b));
    C r;
    r.x = g.x * h; r.y = g.y * h;
    return r;
  }
  C w;
  w.x = (T)twc_re<R>(e);
  w.y = (T)(DIR < 0 ? twc_im<R>(e) : -twc_im<R>(e));
  return cmul(b, w);
}

template <int DIR, typename C> __device__ __forceinline__ void dft3(C &v0, C &v1, C &v2) {
  using T = decltype(v0.x);
  const T hs = (T)(DIR * 0.86602540378443864676372317075294);  // sqrt(3)/2
  const C s = cadd(v1, v2), d = csub(v1, v2);
  const C m = axpy((T)-0.5, s, v0);
  v0 = cadd(v0, s);
  v1.x = m.x - hs * d.y; v1.y = m.y + hs * d.x;
  v2.x = m.x + hs * d.y; v2.y = m.y - hs * d.x;
}
template <int DIR, typename C> __device__ __forceinline__ void dft4(C &v0, C &v1, C &v2, C &v3) {
  const C a0 = cadd(v0, v2), a1 = csub(v0, v2), b0 = cadd(v1, v3), b1 = csub(v1, v3);
  v0 = cadd(a0, b0);
  v2 = csub(a0, b0);
  v1 = add_i<DIR>(a1, b1);
  v3 = sub_i<DIR>(a1, b1);
}
// 8 points; Z34: v[3] and v[4] are zero on input (never read)
template <int DIR, bool Z34, typename C> __device__ __forceinline__ void dft8(C *v) {
  using T = decltype(v[0].x);
  const T h = (T)0.70710678118654752440084436210485;
  const C s0 = Z34 ? v[0] : cadd(v[0], v[4]), d0 = Z34 ? v[0] : csub(v[0], v[4]);
  const C s1 = cadd(v[1], v[5]), d1 = csub(v[1], v[5]);
  const C s2 = cadd(v[2], v[6]), d2 = csub(v[2], v[6]);
  const C s3 = Z34 ? v[7] : cadd(v[3], v[7]);
  const C a0 = cadd(s0, s2), a1 = csub(s0, s2), b0 = cadd(s1, s3), b1 = csub(s1, s3);
  C f0, f1;  // d1 +- DIR i d3
  if (Z34) {  // d3 = -v[7]
    f0 = sub_i<DIR>(d1, v[7]);
    f1 = add_i<DIR>(d1, v[7]);
  } else {
    const C d3 = csub(v[3], v[7]);
    f0 = add_i<DIR>(d1, d3);
    f1 = sub_i<DIR>(d1, d3);
  }
  const C e0 = add_i<DIR>(d0, d2), e1 = sub_i<DIR>(d0, d2);
  const C g0 = rot8<DIR>(f0), g1 = mul_i<DIR>(rot8<DIR>(f1));
  v[0] = cadd(a0, b0);
  v[4] = csub(a0, b0);
  v[2] = add_i<DIR>(a1, b1);
  v[6] = sub_i<DIR>(a1, b1);
  v[1] = axpy(h, g0, e0);
  v[5] = axpy(-h, g0, e0);
  v[3] = axpy(h, g1, e1);
  v[7] = axpy(-h, g1, e1);
}

// In-register R-point DFT, natural order in and out, sign DIR.  6 and 12 are
// coprime products: the prime-factor maps (Good 1958) n = N2 n1 + N1 n2, k = k1
// mod N1 = k2 mod N2 leave no twiddles between the factors.
template <int R, int DIR, bool Z34 = false, typename C> __device__ __forceinline__ void dftr(C *v) {
  static_assert(!Z34 || R == 8, "zero inputs 3 and 4 exist for 8 points");
  if constexpr (R == 1) {
    return;
  } else if constexpr (R == 2) {
    const C a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if constexpr (R == 3) {
    dft3<DIR>(v[0], v[1], v[2]);
  } else if constexpr (R == 4) {
    dft4<DIR>(v[0], v[1], v[2], v[3]);
  } else if constexpr (R == 6) {
    // rows n2: n = 3 n1 + 2 n2 mod 6; the 3-point outputs k2 = k mod 3
    C a[3] = {cadd(v[0], v[3]), cadd(v[2], v[5]), cadd(v[4], v[1])};
    C b[3] = {csub(v[0], v[3]), csub(v[2], v[5]), csub(v[4], v[1])};
    dft3<DIR>(a[0], a[1], a[2]);
    dft3<DIR>(b[0], b[1], b[2]);
    v[0] = a[0]; v[4] = a[1]; v[2] = a[2];
    v[3] = b[0]; v[1] = b[1]; v[5] = b[2];
  } else if constexpr (R == 8) {
    dft8<DIR, Z34>(v);
  } else if constexpr (R == 12) {
    // n = 3 n1 + 4 n2 mod 12, n1 < 4, n2 < 3
    dft4<DIR>(v[0], v[3], v[6], v[9]);
    dft4<DIR>(v[4], v[7], v[10], v[1]);
    dft4<DIR>(v[8], v[11], v[2], v[5]);
    dft3<DIR>(v[0], v[4], v[8]);   // k1 = 0: k = 0, 4, 8 for k2 = 0, 1, 2
    dft3<DIR>(v[3], v[7], v[11]);  // k1 = 1: k = 9, 1, 5
    dft3<DIR>(v[6], v[10], v[2]);  // k1 = 2: k = 6, 10, 2
    dft3<DIR>(v[9], v[1], v[5]);   // k1 = 3: k = 3, 7, 11
    const C t9 = v[3], t1 = v[7], t5 = v[11], t3 = v[9], t7 = v[1], t11 = v[5];
    v[9] = t9; v[1] = t1; v[5] = t5;
    v[3] = t3; v[7] = t7; v[11] = t11;
  } else {
    static_assert(R == 9 || R == 16, "register DFT size");
    constexpr int A = R == 9 ? 3 : 4, B = R / A;
    C y[R];
#pragma unroll
    for (int j2 = 0; j2 < B; j2++) {
      C t[A];
#pragma unroll
      for (int j1 = 0; j1 < A; j1++) t[j1] = v[j2 + B * j1];
      dftr<A, DIR>(t);
#pragma unroll
      for (int k1 = 0; k1 < A; k1++) y[j2 + B * k1] = twmul<R, DIR>(t[k1], j2 * k1);
    }
#pragma unroll
    for (int k1 = 0; k1 < A; k1++) {
      C t[B];
#pragma unroll
      for (int j2 = 0; j2 < B; j2++) t[j2] = y[j2 + B * k1];
      dftr<B, DIR>(t);
#pragma unroll
      for (int k2 = 0; k2 < B; k2++) v[k1 + A * k2] = t[k2];
    }
  }
}

// Line addressing for the two-pass FFTs.  base(l) is the offset of line l,
// ES the element stride (0: given at run time, es_rt).
struct Lines1 {  // lines at l*ls
  int ls;
  __device__ __forceinline__ int base(int l) const { return l * ls; }
  __device__ __forceinline__ bool valid(int) const { return true; }
};
struct Lines2 {  // two contiguous groups of lines (rows 0..n1-1 and the top ones)
  int nl1, ls, off2;
  __device__ __forceinline__ int base(int l) const { return (l < nl1) ? l * ls : off2 + (l - nl1) * ls; }
  __device__ __forceinline__ bool valid(int) const { return true; }
};
// Two groups of rows (n1r rows from row 0, n2r rows from offset off2), each
// enumerated over a multiple of 16 lanes (g1, g2): every half-warp then
// touches 16 consecutive rows of one group, which with an odd row pitch
// (in complex elements) hit disjoint banks.  Padding lanes are not valid.
struct Lines2P {
  int n1r, g1, n2r, ls, off2;
  __device__ __forceinline__ int base(int l) const { return (l < g1) ? l * ls : off2 + (l - g1) * ls; }
  __device__ __forceinline__ bool valid(int l) const { return (l < g1) ? (l < n1r) : (l - g1 < n2r); }
};

// Unit (line l, index j) enumeration for the passes below: lines vary
// fastest across threads, so a warp touches 32 consecutive lines at the same
// j.  With line pitches of N+1 complex (odd) or unit pitch, consecutive lines
// fall in distinct banks (no shared-memory bank conflicts) and the twiddle
// index j is uniform across most of a warp (broadcast loads).  The stepping
// avoids a runtime division per unit.
struct UnitIter {
  int l, j, dl, dj, nl;
  __device__ __forceinline__ UnitIter(int tid, int nthr, int nlines) : nl(nlines) {
    dj = nthr / nl;
    dl = nthr - dj * nl;
    j = tid / nl;
    l = tid - j * nl;
  }
  __device__ __forceinline__ void next() {
    l += dl;
    j += dj;
    if (l >= nl) { l -= nl; j++; }
  }
};

// Elements of a line that hold data (mask.line(l)(k) for natural index k of
// line l): dif reads only those on input (the others count as zero and need
// not be stored), dit writes only those on output.  AllElems: every element.
struct AllK {
  __device__ __forceinline__ bool operator()(int) const { return true; }
};
struct AllElems {
  __device__ __forceinline__ AllK line(int) const { return AllK{}; }
};

// P34 (R1 = 8 only): the elements j2 + R2 j1 with j1 = 3, 4 -- natural
// indices 3N/8 .. 5N/8 - 1, i.e. |k| >= 3N/8 -- hold no data on input (dif)
// and are not needed on output (dit), as for a sphere narrower than 3N/8:
// they are neither read nor written, and no mask is evaluated for them.
template <int R1> __device__ __forceinline__ constexpr bool band34(bool p34, int j1) {
  return p34 && R1 == 8 && (j1 == 3 || j1 == 4);
}

// natural -> permuted.  twN(t): exp(-2 pi i t/N) (TwC, sdft_tw_edges.cuh).
template <int N, int ES, int DIR, bool P34 = false, typename C, typename LM, typename TW, typename MK = AllElems>
__device__ __forceinline__ void dif(C *buf, const LM &lm, int nl, const TW &twN, int tid, int nthr,
                                    const MK &mask = MK{}, int es_rt = ES) {
  const int es = ES ? ES : es_rt;
  constexpr int R1 = Plan<N>::R1, R2 = Plan<N>::R2;
  static_assert(!P34 || R1 == 8, "the j1 = 3, 4 band needs R1 = 8");
  if (nl > 0) {
#pragma unroll 1
    for (UnitIter it(tid, nthr, nl); it.j < R2; it.next()) {
      const int l = it.l, j2 = it.j;
      if (!lm.valid(l)) continue;
      C *p = buf + lm.base(l);
      C v[R1];
      const auto in = mask.line(l);
#pragma unroll
      for (int j1 = 0; j1 < R1; j1++) {
        const int k = j2 + R2 * j1;
        v[j1] = (!band34<R1>(P34, j1) && in(k)) ? p[k * es] : cmk<C>(0.0, 0.0);
      }
      dftr<R1, DIR, P34>(v);
      p[j2 * es] = v[0];
#pragma unroll
      for (int k1 = 1; k1 < R1; k1++) {
        C w = twN(j2 * k1);
        if (DIR > 0) w.y = -w.y;
        p[(j2 + R2 * k1) * es] = cmul(v[k1], w);
      }
    }
  }
  __syncthreads();
  if (nl > 0) {
#pragma unroll 1
    for (UnitIter it(tid, nthr, nl); it.j < R1; it.next()) {
      const int l = it.l, k1 = it.j;
      if (!lm.valid(l)) continue;
      C *p = buf + lm.base(l) + R2 * k1 * es;
      C v[R2];
#pragma unroll
      for (int j = 0; j < R2; j++) v[j] = p[j * es];
      dftr<R2, DIR>(v);
#pragma unroll
      for (int j = 0; j < R2; j++) p[j * es] = v[j];
    }
  }
  __syncthreads();
}

// permuted -> natural
template <int N, int ES, int DIR, bool P34 = false, typename C, typename LM, typename TW, typename MK = AllElems>
__device__ __forceinline__ void dit(C *buf, const LM &lm, int nl, const TW &twN, int tid, int nthr,
                                    const MK &mask = MK{}, int es_rt = ES) {
  const int es = ES ? ES : es_rt;
  constexpr int R1 = Plan<N>::R1, R2 = Plan<N>::R2;
  static_assert(!P34 || R1 == 8, "the j1 = 3, 4 band needs R1 = 8");
  if (nl > 0) {
#pragma unroll 1
    for (UnitIter it(tid, nthr, nl); it.j < R1; it.next()) {
      const int l = it.l, k1 = it.j;
      if (!lm.valid(l)) continue;
      C *p = buf + lm.base(l) + R2 * k1 * es;
      C v[R2];
#pragma unroll
      for (int j = 0; j < R2; j++) v[j] = p[j * es];
      dftr<R2, DIR>(v);
      p[0] = v[0];
#pragma unroll
      for (int j2 = 1; j2 < R2; j2++) {
        C w = twN(j2 * k1);
        if (DIR > 0) w.y = -w.y;
        p[j2 * es] = cmul(v[j2], w);
      }
    }
  }
  __syncthreads();
  if (nl > 0) {
#pragma unroll 1
    for (UnitIter it(tid, nthr, nl); it.j < R2; it.next()) {
      const int l = it.l, j2 = it.j;
      if (!lm.valid(l)) continue;
      C *p = buf + lm.base(l);
      C v[R1];
#pragma unroll
      for (int k1 = 0; k1 < R1; k1++) v[k1] = p[(R2 * k1 + j2) * es];
      dftr<R1, DIR>(v);
      const auto out = mask.line(l);
#pragma unroll
      for (int j1 = 0; j1 < R1; j1++) {
        const int k = j2 + R2 * j1;
        if (!band34<R1>(P34, j1) && out(k)) p[k * es] = v[j1];
      }
    }
  }
  __syncthreads();
}

}  // namespace sdft
