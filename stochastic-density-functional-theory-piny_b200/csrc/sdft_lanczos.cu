// sdft_lanczos.cu -- vector kernels of the device Lanczos bounds and of the
// filtered-orbital energies and KB atomic forces.
//
// Vectors are one orbital row of the context layout: re[0, ncoef) then
// im[0, ncoef) at offset ngp; G0 is entry ncoef - 1.  Reductions are
// deterministic: kRedBlocks fixed block partials, each a fixed-order tree,
// summed in block order by one thread.
#include <cuda_runtime.h>
#include <algorithm>
#include "sdft_kernels.cuh"
#include "sdft_lanczos.h"
#include "sdft_pdl.cuh"

namespace sdft {

namespace {

__device__ __forceinline__ void block_sum_to(double a, double *out) {
  __shared__ double sh[kRedThreads];
  sh[threadIdx.x] = a;
  __syncthreads();
  for (int s = kRedThreads / 2; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sh[0];
}

// half-sphere inner product <a|b> = 2 sum (re re + im im) - re(G0) re(G0)
__global__ void __launch_bounds__(kRedThreads) k_hdot_part(const double *__restrict__ a, const double *__restrict__ b,
                                                           int ncoef, int ngp, double *__restrict__ part) {
  double s = 0.0;
  for (int g = blockIdx.x * kRedThreads + threadIdx.x; g < ncoef; g += kRedBlocks * kRedThreads) {
    const double rr = a[g] * b[g], ii = a[ngp + g] * b[ngp + g];
    s += (g == ncoef - 1) ? rr + 2.0 * ii : 2.0 * (rr + ii);
  }
  block_sum_to(s, part + blockIdx.x);
}

__global__ void k_sum_fixed(const double *__restrict__ part, int n, double *__restrict__ out) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double s = 0.0;
    for (int i = 0; i < n; i++) s += part[i];
    *out = s;
  }
}

// Sum of n values spaced `stride` apart, the same in every block: per thread in
// order, then a fixed tree (blockDim.x = kRedThreads; every thread returns it).
__device__ __forceinline__ double block_sum_all(const double *__restrict__ v, int n, int stride) {
  __shared__ double sh[kRedThreads];
  double a = 0.0;
  for (int i = threadIdx.x; i < n; i += kRedThreads) a += v[(size_t)i * stride];
  sh[threadIdx.x] = a;
  __syncthreads();
  for (int s = kRedThreads / 2; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
    __syncthreads();
  }
  a = sh[0];
  __syncthreads();
  return a;
}

// w = h - alpha c - beta p in place in h (p null: no p term), alpha = sum of the
// stage-C dot partials (first of every three); part: block partials of |w|^2
__global__ void __launch_bounds__(kRedThreads)
k_lz_w(double *__restrict__ h, const double *__restrict__ c, const double *__restrict__ p,
       const double *__restrict__ dots, int nparts, const double *__restrict__ beta, double *__restrict__ alpha,
       int ncoef, int ngp, double *__restrict__ part) {
  pdl_trigger();
  pdl_wait();
  const double a = block_sum_all(dots, nparts, 3);
  const double b = p ? *beta : 0.0;
  if (blockIdx.x == 0 && threadIdx.x == 0) *alpha = a;
  double s = 0.0;
  for (int g = blockIdx.x * kRedThreads + threadIdx.x; g < ncoef; g += kRedBlocks * kRedThreads) {
    double re = h[g] - a * c[g], im = h[ngp + g] - a * c[ngp + g];
    if (p) {
      re -= b * p[g];
      im -= b * p[ngp + g];
    }
    h[g] = re;
    h[ngp + g] = im;
    s += (g == ncoef - 1) ? re * re + 2.0 * im * im : 2.0 * (re * re + im * im);
  }
  block_sum_to(s, part + blockIdx.x);
}

// beta = |w| from the block partials; p = c, c = w / beta; omax (nullable):
// atomicMax of max |c|, as stage C records it for the digit pass
__global__ void __launch_bounds__(kRedThreads)
k_lz_next(const double *__restrict__ w, double *__restrict__ c, double *__restrict__ p,
          const double *__restrict__ part, double *__restrict__ beta, int ncoef, int ngp, unsigned long long *omax) {
  pdl_trigger();
  pdl_wait();
  const double b = sqrt(fmax(block_sum_all(part, kRedBlocks, 1), 0.0));
  if (blockIdx.x == 0 && threadIdx.x == 0) *beta = b;
  double m = 0.0;
  for (int g = blockIdx.x * kRedThreads + threadIdx.x; g < ncoef; g += kRedBlocks * kRedThreads) {
    for (int q = 0; q < 2; q++) {
      const int i = q * ngp + g;
      const double x = w[i] / b;
      p[i] = c[i];
      c[i] = x;
      m = fmax(m, absmax_key_d(x));
    }
  }
  if (!omax) return;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(omax, (unsigned long long)__double_as_longlong(m));
}

// c /= d (normalisation of the start vector)
__global__ void k_lz_div(double *__restrict__ c, const double *__restrict__ nrm2, int ncoef, int ngp) {
  const double d = sqrt(*nrm2);
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < ncoef; g += gridDim.x * blockDim.x) {
    c[g] = c[g] / d;
    c[ngp + g] = c[ngp + g] / d;
  }
}

// sum over nstate rows and G != G0 of 2 ak2(G) (re^2 + im^2); blocks
// (row group, chunk of G): a thread's G stay the same over the group's rows, so
// ak2 is read once per thread and the rows stream (a fixed order)
__global__ void __launch_bounds__(kRedThreads) k_ekin_part(const double *__restrict__ v, int nstate, int ncoef,
                                                           int ngp, const double *__restrict__ ak2,
                                                           double *__restrict__ part) {
  double s = 0.0;
  const int r0 = (int)((long long)nstate * blockIdx.y / kEkRows);
  const int r1 = (int)((long long)nstate * (blockIdx.y + 1) / kEkRows);
  for (int g = 2 * (blockIdx.x * kRedThreads + threadIdx.x); g < ncoef - 1; g += 2 * kEkChunks * kRedThreads) {
    const double k0 = 2.0 * ak2[g], k1 = g + 1 < ncoef - 1 ? 2.0 * ak2[g + 1] : 0.0;
    const double *row = v + (size_t)r0 * 2 * ngp + g;  // (16-byte aligned: ngp is a multiple of 16)
#pragma unroll 4
    for (int st = r0; st < r1; st++, row += 2 * (size_t)ngp) {
      const double2 re = *reinterpret_cast<const double2 *>(row), im = *reinterpret_cast<const double2 *>(row + ngp);
      const double e0 = k0 * (re.x * re.x + im.x * im.x);
      s += k1 == 0.0 ? e0 : e0 + k1 * (re.y * re.y + im.y * im.y);
    }
  }
  block_sum_to(s, part + blockIdx.y * kEkChunks + blockIdx.x);
}

__global__ void __launch_bounds__(kRedThreads) k_sum_tree(const double *__restrict__ part, int n,
                                                          double *__restrict__ out) {
  const double a = block_sum_all(part, n, 1);
  if (threadIdx.x == 0) *out = a;
}

// i G_d c: the orbital whose KB projection is dZ/dR_d (get_nlmat,
// energy/cp/cp_energy_eext_nonloc.c:648-748, accumulates the same sums with
// the factor G_d and the Re/Im roles swapped)
// grid (x: coefficient blocks, y: orbital rows); no index division
__global__ void k_dcoef(const double *__restrict__ v, int ncoef, int ngp, const double *__restrict__ gk,
                        double *__restrict__ out) {
  const double *row = v + (size_t)blockIdx.y * 2 * ngp;
  double *o = out + (size_t)blockIdx.y * 2 * ngp;
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < ngp; g += gridDim.x * blockDim.x) {
    const bool in = g < ncoef - 1;
    const double k = in ? gk[g] : 0.0;
    const double re = in ? row[g] : 0.0, im = in ? row[ngp + g] : 0.0;
    o[g] = -k * im;
    o[ngp + g] = k * re;
  }
}

// one block per atom: the force component d of getnl_pot_pv_fatm ->
// sumnl_pot_pv_fatm_hess (cp_energy_eext_nonloc.c:1473-1500) over the merged
// projector rows (w carries vnorm / vol and the doubled weight of a merged
// conjugate pair, whose dZ obeys the same pairing as Z)
__global__ void __launch_bounds__(kRedThreads) k_nl_force_atoms(const double *__restrict__ Z0,
                                                                const double *__restrict__ Zd, int ldz,
                                                                const double *__restrict__ w,
                                                                const int *__restrict__ rs,
                                                                const int *__restrict__ rc, int nstate, double scale,
                                                                int d, double *__restrict__ f) {
  const int a = blockIdx.x, u0 = rs[a], nu = rc[a];
  double acc = 0.0;
  for (int i = threadIdx.x; i < nu * nstate; i += kRedThreads) {
    const int s = i / nu, u = u0 + (i - s * nu);
    acc += w[u] * Z0[(size_t)s * ldz + u] * Zd[(size_t)s * ldz + u];
  }
  __shared__ double sh[kRedThreads];
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int h = kRedThreads / 2; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h) sh[threadIdx.x] += sh[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) f[3 * a + d] = -2.0 * scale * sh[0];
}

inline int grid_for(int n) {
  int b = (n + 255) / 256;
  return b < 1 ? 1 : (b > 1024 ? 1024 : b);
}

}  // namespace

void launch_half_dot(const double *a, const double *b, int ncoef, int ngp, double *part, double *out,
                     cudaStream_t st) {
  k_hdot_part<<<kRedBlocks, kRedThreads, 0, st>>>(a, b, ncoef, ngp, part);
  k_sum_fixed<<<1, 32, 0, st>>>(part, kRedBlocks, out);
}

void launch_lz_w(double *h, const double *c, const double *p, const double *dots, int nparts, const double *beta,
                 double *alpha, int ncoef, int ngp, double *part, cudaStream_t st) {
  launch_pdl(true, k_lz_w, dim3(kRedBlocks), dim3(kRedThreads), 0, st, h, c, p, dots, nparts, beta, alpha, ncoef, ngp, part);
}

void launch_lz_next(const double *w, double *c, double *p, const double *part, double *beta, int ncoef, int ngp,
                    unsigned long long *omax, cudaStream_t st) {
  launch_pdl(true, k_lz_next, dim3(kRedBlocks), dim3(kRedThreads), 0, st, w, c, p, part, beta, ncoef, ngp, omax);
}

void launch_lz_div(double *c, const double *nrm2, int ncoef, int ngp, cudaStream_t st) {
  k_lz_div<<<grid_for(ncoef), 256, 0, st>>>(c, nrm2, ncoef, ngp);
}

void launch_ekin(const double *v, int nstate, int ncoef, int ngp, const double *ak2, double *part, double *out,
                 cudaStream_t st) {
  k_ekin_part<<<dim3(kEkChunks, kEkRows), kRedThreads, 0, st>>>(v, nstate, ncoef, ngp, ak2, part);
  k_sum_tree<<<1, kRedThreads, 0, st>>>(part, kEkChunks * kEkRows, out);
}

void launch_dcoef(const double *v, int nstate, int ncoef, int ngp, const double *gk, double *out, cudaStream_t st) {
  const int bx = std::min(8, (ngp + 255) / 256);
  for (int s0 = 0; s0 < nstate; s0 += 65535) {  // grid.y limit
    const int n = std::min(65535, nstate - s0);
    const size_t off = (size_t)s0 * 2 * ngp;
    k_dcoef<<<dim3(bx < 1 ? 1 : bx, n), 256, 0, st>>>(v + off, ncoef, ngp, gk, out + off);
  }
}

void launch_nl_force_atoms(const double *Z0, const double *Zd, int ldz, const double *w, const int *row_start,
                           const int *row_count, int natm, int nstate, double scale, int d, double *f,
                           cudaStream_t st) {
  k_nl_force_atoms<<<natm, kRedThreads, 0, st>>>(Z0, Zd, ldz, w, row_start, row_count, nstate, scale, d, f);
}

// Extreme eigenvalues of the symmetric tridiagonal matrix (diagonal a[0..n),
// off-diagonal b[0..n-1)) by Sturm-sequence bisection: count(x) = number of
// eigenvalues below x from the signs of the LDL^T pivots.
static int count_below(const double *a, const double *b, int n, double x) {
  int c = 0;
  double d = 1.0;
  for (int i = 0; i < n; i++) {
    const double off = i > 0 ? b[i - 1] * b[i - 1] : 0.0;
    d = (a[i] - x) - (i > 0 ? off / d : 0.0);
    if (d == 0.0) d = -1e-300;
    if (d < 0.0) c++;
  }
  return c;
}

void tridiag_extremes(const double *a, const double *b, int n, double *lo, double *hi) {
  double gl = a[0], gu = a[0];
  for (int i = 0; i < n; i++) {
    const double r = (i > 0 ? fabs(b[i - 1]) : 0.0) + (i < n - 1 ? fabs(b[i]) : 0.0);
    gl = fmin(gl, a[i] - r);
    gu = fmax(gu, a[i] + r);
  }
  const double pad = 1e-12 * fmax(1.0, fmax(fabs(gl), fabs(gu)));
  gl -= pad;
  gu += pad;
  for (int which = 0; which < 2; which++) {
    // smallest: largest x with count(x) == 0; largest: smallest x with count(x) == n
    double l = gl, u = gu;
    for (int it = 0; it < 200 && u - l > 0.0; it++) {
      const double m = 0.5 * (l + u);
      if (m <= l || m >= u) break;
      const int c = count_below(a, b, n, m);
      if (which == 0 ? c >= 1 : c >= n) u = m;
      else l = m;
    }
    (which == 0 ? *lo : *hi) = 0.5 * (l + u);
  }
}

}  // namespace sdft
