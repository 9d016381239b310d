"""Generate sdft_twiddles.cuh: exp(-2 pi i t/R), t = 0..R-1, for the in-register DFTs,
and sdft_tw_edges.cuh: the same for every compile-time FFT edge, in constant memory.

Each value is computed in 50-digit decimal arithmetic (pi by Machin's
formula, cos and sin by their Taylor series) and rounded once to the nearest
double (float(Decimal) rounds correctly), so every constant is the correctly
rounded double of the exact twiddle.

  python gen_twiddles.py > sdft_twiddles.cuh
  python gen_twiddles.py edges > sdft_tw_edges.cuh
"""
import sys
from decimal import Decimal, getcontext

getcontext().prec = 50
RADICES = (9, 16)
EDGES = (12, 16, 18, 24, 27, 32, 36, 48, 54, 64, 72, 81, 96, 108, 128)


def _atan_inv(n):
    """atan(1/n) by its Taylor series."""
    x = Decimal(1) / n
    x2 = x * x
    term, total, k = x, x, 1
    while True:
        term *= -x2
        t = term / (2 * k + 1)
        if t == 0 or abs(t) < Decimal(10) ** -60:
            break
        total += t
        k += 1
    return total


PI = 16 * _atan_inv(5) - 4 * _atan_inv(239)


def _cos_sin(x):
    c, s = Decimal(0), Decimal(0)
    term, k = Decimal(1), 0  # x^k / k!
    while abs(term) > Decimal(10) ** -60:
        r = k % 4
        if r == 0:
            c += term
        elif r == 1:
            s += term
        elif r == 2:
            c -= term
        else:
            s -= term
        k += 1
        term = term * x / k
    return c, s


def twiddles(R):
    re, im = [], []
    for t in range(R):
        c, s = _cos_sin(2 * PI * t / R)
        # the exact zeros (t/R a multiple of 1/4) come out as ~1e-50 here
        eps = Decimal(10) ** -40
        c = Decimal(0) if abs(c) < eps else c
        s = Decimal(0) if abs(s) < eps else s
        re.append(float(c) + 0.0)
        im.append(-float(s) + 0.0)
    return re, im


def main():
    print("// sdft_twiddles.cuh -- exp(-2 pi i t/R) constants of the in-register DFTs")
    print("// (generated by gen_twiddles.py; correctly rounded doubles).")
    print("#pragma once")
    print("namespace sdft {")
    for R in RADICES:
        re, im = twiddles(R)
        print(f"__device__ constexpr double kTw{R}re[{R}] = {{{', '.join(repr(v) for v in re)}}};")
        print(f"__device__ constexpr double kTw{R}im[{R}] = {{{', '.join(repr(v) for v in im)}}};")
    print("}  // namespace sdft")


def edges():
    off = {}
    vals = []
    for n in EDGES:
        off[n] = len(vals)
        vals += zip(*twiddles(n))
    print(f"""// sdft_tw_edges.cuh -- exp(-2 pi i t/N) of the compile-time FFT edges in constant
// memory: the warps of a pass read one twiddle index at a time, which the constant
// cache broadcasts without a shared-memory wavefront (generated by gen_twiddles.py;
// correctly rounded doubles, and those rounded to float).
#pragma once
#include <cuda_runtime.h>
namespace sdft {{
constexpr int kTwTotal = {len(vals)};
// offset of edge n's table, -1 without one
constexpr int tw_off(int n) {{
  switch (n) {{""")
    for n in EDGES:
        print(f"    case {n}: return {off[n]};")
    print("""    default: return -1;
  }
}""")
    print("static __constant__ double2 c_twd[kTwTotal] = {")
    print(",\n".join(f"    {{{r!r}, {i!r}}}" for r, i in vals))
    print("};")
    print("static __constant__ float2 c_twf[kTwTotal] = {")
    print(",\n".join(f"    {{(float){r!r}, (float){i!r}}}" for r, i in vals))
    print("};")
    print("""template <int N, typename C> struct TwC;
template <int N> struct TwC<N, float2> {
  static constexpr int off = tw_off(N);
  static_assert(off >= 0, "edge without a constant twiddle table");
  __device__ __forceinline__ float2 operator()(int t) const { return c_twf[off + t]; }
};
template <int N> struct TwC<N, double2> {
  static constexpr int off = tw_off(N);
  static_assert(off >= 0, "edge without a constant twiddle table");
  __device__ __forceinline__ double2 operator()(int t) const { return c_twd[off + t]; }
};
}  // namespace sdft""")


if __name__ == "__main__":
    edges() if sys.argv[1:] == ["edges"] else main()
