// pme.cu -- smooth PME for the permanent field and the dipole matvec.
//
// efld0_recip (newinduce_pme.f:1671-1917) and tmatxbrecip (:1919-2128):
// B-splines recomputed per pass from positions (bsplgen, pmestuff.f:64),
// spread with global atomics into one complex grid (d dipoles in Re, p in Im,
// as qgrid2in_2d), the convolution with the influence function qfac (three
// kernels, conv_dev.cuh, on the cubic grids they cover, else cuFFT forward, qfac,
// cuFFT backward; unnormalised, fft_mpi.f90:65,115), and a gather of the potential
// derivatives (fphi_mpole_site :453, fphi_uind_site :746).  Orthogonal boxes:
// the fractional <-> Cartesian matrices reduce to a_d = nfft_d * recip(d,d).
#include <vector>

#include <map>
#include <mutex>
#include <type_traits>

#include "conv.h"
#include "kernels.h"
#include "pme_dev.cuh"

namespace thp {

namespace {

constexpr int kBlock = 128;

__device__ __forceinline__ void grid_add_re(cufftDoubleComplex* g, size_t idx, double re) { red_add(&g[idx].x, re); }
__device__ __forceinline__ void grid_add_re(cufftComplex* g, size_t idx, float re) { red_add(&g[idx].x, re); }

// grid_mpole_site (pmestuff.f:163-278) for every site; rpole10 sorted
template <typename T>
__global__ void k_spread_mpole(int n, PmeGeom g, const double4* __restrict__ pos, const double* __restrict__ rp,
                               typename Cplx<T>::type* __restrict__ grid) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double4 p = pos[i];
  T tx[kBs][3], ty[kBs][3], tz[kBs][3];
  int gx = bspline_axis<3, T>(p.x, g.recip[0], g.n1, tx);
  int gy = bspline_axis<3, T>(p.y, g.recip[1], g.n2, ty);
  int gz = bspline_axis<3, T>(p.z, g.recip[2], g.n3, tz);
  const double* r = rp + (size_t)i * 10;
  // cmp (newinduce_pme.f:1750-1759) -> fmp via cart_to_frac (pmestuff.f:1131)
  T f[10];
  f[0] = (T)r[0];
  f[1] = (T)(g.a[0] * r[1]);
  f[2] = (T)(g.a[1] * r[2]);
  f[3] = (T)(g.a[2] * r[3]);
  f[4] = (T)(g.a[0] * g.a[0] * r[4]);
  f[5] = (T)(g.a[1] * g.a[1] * r[7]);
  f[6] = (T)(g.a[2] * g.a[2] * r[9]);
  f[7] = (T)(g.a[0] * g.a[1] * (2.0 * r[5]));
  f[8] = (T)(g.a[0] * g.a[2] * (2.0 * r[6]));
  f[9] = (T)(g.a[1] * g.a[2] * (2.0 * r[8]));
#pragma unroll
  for (int c = 0; c < kBs; ++c) {
    size_t kk = (size_t)wrapk(gz + c, g.n3);
    T v0 = tz[c][0], v1 = tz[c][1], v2 = tz[c][2];
#pragma unroll
    for (int b = 0; b < kBs; ++b) {
      size_t jj = (size_t)wrapk(gy + b, g.n2);
      T u0 = ty[b][0], u1 = ty[b][1], u2 = ty[b][2];
      T term0 = f[0] * u0 * v0 + f[2] * u1 * v0 + f[3] * u0 * v1 + f[5] * u2 * v0 + f[6] * u0 * v2 + f[9] * u1 * v1;
      T term1 = f[1] * u0 * v0 + f[7] * u1 * v0 + f[8] * u0 * v1;
      T term2 = f[4] * u0 * v0;
      size_t row = (kk * g.n2 + jj) * g.n1;
#pragma unroll
      for (int a = 0; a < kBs; ++a) {
        int ii = wrapk(gx + a, g.n1);
        grid_add_re(grid, row + ii, term0 * tx[a][0] + term1 * tx[a][1] + term2 * tx[a][2]);
      }
    }
  }
}

// The same with a warp per site, lane l < 25 on stencil line (y, z) =
// (l % 5, l / 5), for systems too small to fill the GPU with a thread per site.
template <typename T>
__global__ void __launch_bounds__(128) k_spread_mpole_small(int n, PmeGeom g, const double4* __restrict__ pos,
                                                            const double* __restrict__ rp,
                                                            typename Cplx<T>::type* __restrict__ grid) {
  __shared__ SiteWeights<T, 3> sw[4];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = blockIdx.x * 4 + warp;
  if (i >= n) return;  // the same for the whole warp
  SiteWeights<T, 3>& s = sw[warp];
  if (lane >= 29) stage_axis<T, 3>(g, pos[i], lane - 29, s);
  const double* r = rp + (size_t)i * 10;
  const T f0 = (T)r[0], f1 = (T)(g.a[0] * r[1]), f2 = (T)(g.a[1] * r[2]), f3 = (T)(g.a[2] * r[3]);
  const T f4 = (T)(g.a[0] * g.a[0] * r[4]), f5 = (T)(g.a[1] * g.a[1] * r[7]), f6 = (T)(g.a[2] * g.a[2] * r[9]);
  const T f7 = (T)(g.a[0] * g.a[1] * (2.0 * r[5])), f8 = (T)(g.a[0] * g.a[2] * (2.0 * r[6])),
          f9 = (T)(g.a[1] * g.a[2] * (2.0 * r[8]));
  __syncwarp();
  if (lane >= kBs * kBs) return;
  const int b = lane % kBs, c = lane / kBs;
  const T u0 = s.w[1][3 * b], u1 = s.w[1][3 * b + 1], u2 = s.w[1][3 * b + 2];
  const T v0 = s.w[2][3 * c], v1 = s.w[2][3 * c + 1], v2 = s.w[2][3 * c + 2];
  const T term0 = f0 * u0 * v0 + f2 * u1 * v0 + f3 * u0 * v1 + f5 * u2 * v0 + f6 * u0 * v2 + f9 * u1 * v1;
  const T term1 = f1 * u0 * v0 + f7 * u1 * v0 + f8 * u0 * v1;
  const T term2 = f4 * u0 * v0;
  const size_t row = ((size_t)wrapk(s.g0[2] + c, g.n3) * g.n2 + wrapk(s.g0[1] + b, g.n2)) * g.n1;
#pragma unroll
  for (int a = 0; a < kBs; ++a)
    grid_add_re(grid, row + wrapk(s.g0[0] + a, g.n1),
                term0 * s.w[0][3 * a] + term1 * s.w[0][3 * a + 1] + term2 * s.w[0][3 * a + 2]);
}

// grid_mpole_site for the two multipole sets of eprecip1's virial
// (epolar1.f:932-1040): the permanent moments with uinp added to the dipole
// into the real part, with uind added into the imaginary part, of one
// complex grid.  mu sorted [n][6] (uind xyz, uinp xyz).
template <typename T>
__global__ void k_spread_mpole2(int n, PmeGeom g, const double4* __restrict__ pos, const double* __restrict__ rp,
                                const double* __restrict__ mu, typename Cplx<T>::type* __restrict__ grid) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double4 p = pos[i];
  T tx[kBs][3], ty[kBs][3], tz[kBs][3];
  int gx = bspline_axis<3, T>(p.x, g.recip[0], g.n1, tx);
  int gy = bspline_axis<3, T>(p.y, g.recip[1], g.n2, ty);
  int gz = bspline_axis<3, T>(p.z, g.recip[2], g.n3, tz);
  const double* r = rp + (size_t)i * 10;
  const double* m = mu + (size_t)i * 6;
  T f[10], fb[3];
  f[0] = (T)r[0];
  f[1] = (T)(g.a[0] * (r[1] + m[3]));
  f[2] = (T)(g.a[1] * (r[2] + m[4]));
  f[3] = (T)(g.a[2] * (r[3] + m[5]));
  fb[0] = (T)(g.a[0] * (r[1] + m[0]));
  fb[1] = (T)(g.a[1] * (r[2] + m[1]));
  fb[2] = (T)(g.a[2] * (r[3] + m[2]));
  f[4] = (T)(g.a[0] * g.a[0] * r[4]);
  f[5] = (T)(g.a[1] * g.a[1] * r[7]);
  f[6] = (T)(g.a[2] * g.a[2] * r[9]);
  f[7] = (T)(g.a[0] * g.a[1] * (2.0 * r[5]));
  f[8] = (T)(g.a[0] * g.a[2] * (2.0 * r[6]));
  f[9] = (T)(g.a[1] * g.a[2] * (2.0 * r[8]));
#pragma unroll
  for (int c = 0; c < kBs; ++c) {
    size_t kk = (size_t)wrapk(gz + c, g.n3);
    T v0 = tz[c][0], v1 = tz[c][1], v2 = tz[c][2];
#pragma unroll
    for (int b = 0; b < kBs; ++b) {
      size_t jj = (size_t)wrapk(gy + b, g.n2);
      T u0 = ty[b][0], u1 = ty[b][1], u2 = ty[b][2];
      // the terms without a dipole are shared by the two sets
      T q0 = f[0] * u0 * v0 + f[5] * u2 * v0 + f[6] * u0 * v2 + f[9] * u1 * v1;
      T term0a = q0 + f[2] * u1 * v0 + f[3] * u0 * v1, term0b = q0 + fb[1] * u1 * v0 + fb[2] * u0 * v1;
      T q1 = f[7] * u1 * v0 + f[8] * u0 * v1;
      T term1a = q1 + f[1] * u0 * v0, term1b = q1 + fb[0] * u0 * v0;
      T term2 = f[4] * u0 * v0;
      size_t row = (kk * g.n2 + jj) * g.n1;
#pragma unroll
      for (int a = 0; a < kBs; ++a) {
        int ii = wrapk(gx + a, g.n1);
        grid_add(grid, row + ii, term0a * tx[a][0] + term1a * tx[a][1] + term2 * tx[a][2],
                 term0b * tx[a][0] + term1b * tx[a][1] + term2 * tx[a][2]);
      }
    }
  }
}

// Where a row of the influence function holds x frequency k, n1 = f1 f2 (conv.h;
// f1 = f2 = 1: at k, the order of cuFFT's grids).
struct XOrder {
  int f1, f2;
  __device__ __forceinline__ int slot(int k) const { return f2 * (k % f1) + k / f1; }
};

// Sum over the reciprocal lattice (all k but 0 with qfac > 0) of the PME
// virial terms h h vterm - eterm (eterm = 0.5 f qfac struc2, vterm =
// (2/h^2)(1 + pterm h^2) eterm; emrecip1 / eprecip1, epolar1.f:1041-1091)
// of the forward-transformed grid, times sign.  mode 0: struc2 = |G(k)|^2
// (one real grid); mode 1: struc2 = Re(A(k) conj B(k)) of the two real grids
// A (real part) and B (imaginary part) packed in G, separated by
// A = (G(k) + conj G(-k)) / 2, B = (G(k) - conj G(-k)) / 2i.  Each block
// writes its 6 sums (xx, xy, xz, yy, yz, zz) to part[block].
template <typename C, typename Q>
__global__ void __launch_bounds__(256) k_kspace_virial(int n1, int n2, int n3, XOrder xo, const C* __restrict__ grid,
                                                       const Q* __restrict__ qfac, double r1, double r2, double r3,
                                                       double pterm, double f, int mode, double sign,
                                                       double* __restrict__ part) {
  double v[6] = {0, 0, 0, 0, 0, 0};
  const long ng = (long)n1 * n2 * n3;
  const int nf1 = (n1 + 1) / 2, nf2 = (n2 + 1) / 2, nf3 = (n3 + 1) / 2;
  for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < ng; idx += (long)gridDim.x * blockDim.x) {
    const int k1 = (int)(idx % n1);
    const double qf = (double)qfac[idx - k1 + xo.slot(k1)];
    if (qf == 0.0) continue;
    const int k2 = (int)((idx / n1) % n2), k3 = (int)(idx / ((long)n1 * n2));
    const int m1 = k1 + 1 > nf1 ? k1 - n1 : k1, m2 = k2 + 1 > nf2 ? k2 - n2 : k2, m3 = k3 + 1 > nf3 ? k3 - n3 : k3;
    const C gk = grid[idx];
    double struc2;
    if (mode == 0) {
      struc2 = (double)gk.x * gk.x + (double)gk.y * gk.y;
    } else {
      const long mi = ((long)((n3 - k3) % n3) * n2 + (n2 - k2) % n2) * n1 + (n1 - k1) % n1;
      const C gm = grid[mi];  // conj G(-k) = (gm.x, -gm.y)
      const double ax = 0.5 * ((double)gk.x + gm.x), ay = 0.5 * ((double)gk.y - gm.y);
      const double bx = 0.5 * ((double)gk.y + gm.y), by = -0.5 * ((double)gk.x - gm.x);
      struc2 = ax * bx + ay * by;
    }
    const double h1 = r1 * m1, h2 = r2 * m2, h3 = r3 * m3;
    const double hsq = h1 * h1 + h2 * h2 + h3 * h3;
    const double eterm = 0.5 * f * qf * struc2;
    const double vterm = (2.0 / hsq) * (1.0 + pterm * hsq) * eterm;
    v[0] += h1 * h1 * vterm - eterm;
    v[1] += h1 * h2 * vterm;
    v[2] += h1 * h3 * vterm;
    v[3] += h2 * h2 * vterm - eterm;
    v[4] += h2 * h3 * vterm;
    v[5] += h3 * h3 * vterm - eterm;
  }
  block_reduce<6>(v);
  if (threadIdx.x == 0)
#pragma unroll
    for (int q = 0; q < 6; ++q) part[(size_t)blockIdx.x * 6 + q] = sign * v[q];
}

// The vector a site spreads.
template <typename V>
__device__ __forceinline__ void spread_load(int i, const V* __restrict__ vec, double (&v)[6]) {
  if constexpr (std::is_same<V, float>::value) {
    const float2* v2 = reinterpret_cast<const float2*>(vec + (size_t)i * 6);
    const float2 a0 = v2[0], a1 = v2[1], a2 = v2[2];
    v[0] = a0.x; v[1] = a0.y; v[2] = a1.x; v[3] = a1.y; v[4] = a2.x; v[5] = a2.y;
  } else {
    const double2* v2 = reinterpret_cast<const double2*>(vec + (size_t)i * 6);
    double2 a0 = v2[0], a1 = v2[1], a2 = v2[2];
    v[0] = a0.x; v[1] = a0.y; v[2] = a1.x; v[3] = a1.y; v[4] = a2.x; v[5] = a2.y;
  }
}

// grid_uind_site (pmestuff.f:280-405); d dipoles in Re, p dipoles in Im.
// One thread per site.  TA = 0: each site adds its 125 stencil points to the
// grid itself (a warp-per-site variant that made them contiguous measured
// 1.6x slower); TA = 16: the warp sums the stencils of 16 neighbouring sites
// at a time in a shared-memory tile first (spread_dip_warp), blocks of
// kSpreadThreads threads with one SpreadWarp<T> per warp in dynamic shared
// memory.
// V: the stored type of vec (FP32 for the mixed form's overlapped CG)
template <typename T, typename V = double, int TA = 0>
__global__ void __launch_bounds__(128) k_spread_dip(int n, PmeGeom g, const double4* __restrict__ pos,
                                                   const V* __restrict__ vec, const CgScalars* __restrict__ cg,
                                                   int check_stop, typename Cplx<T>::type* __restrict__ grid) {
  if (check_stop && cg->stop) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  SpreadWarp<T>* sw = nullptr;
  if constexpr (TA > 0) {
    extern __shared__ __align__(16) unsigned char spread_smem[];
    sw = reinterpret_cast<SpreadWarp<T>*>(spread_smem) + (threadIdx.x >> 5);
    for (int q = threadIdx.x & 31; q < SpreadWarp<T>::kPts; q += 32) sw->tile[q] = {T(0), T(0)};
  } else if (i >= n) {
    return;
  }
  const bool live = i < n;
  double v[6] = {0, 0, 0, 0, 0, 0};
  double4 pi = make_double4(0, 0, 0, 0);
  if (live) {
    spread_load(i, vec, v);
    pi = pos[i];
  }
  if constexpr (TA > 0)
    spread_dip_warp<T>(g, pi, v, live, grid, *sw);
  else
    spread_dip_site<T>(g, pi, v, grid);
}

// The same with a warp per site, for systems too small to fill the GPU with a
// thread per site: the lanes share the site's 25 stencil lines (648 atoms: 16.9
// -> 4.4 us FP64, 9,003 atoms 15.2 -> 11.2 us FP32).  update: first pp = zr + beta pp
// (inducepcg_pme2.f:553-559), written back.  rec (mixed form): the 32-byte
// partner records of vec the real-space rows read (wrapped FP32 position, d
// dipole, p dipole x, y; the p dipole z in mpz).
template <typename T>
__global__ void __launch_bounds__(128) k_spread_dip_small(int n, PmeGeom g, const double4* __restrict__ pos,
                                                          double* __restrict__ vec, const double* __restrict__ zr,
                                                          const CgScalars* __restrict__ cg, int check_stop, int update,
                                                          const float4* __restrict__ posf, float* __restrict__ rec,
                                                          float* __restrict__ mpz,
                                                          typename Cplx<T>::type* __restrict__ grid) {
  __shared__ SiteWeights<T> sw[4];
  if (check_stop && cg->stop) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = blockIdx.x * 4 + warp;
  if (i >= n) return;  // the same for the whole warp
  double v = 0.0;
  if (lane < 6) {
    const size_t q = (size_t)i * 6 + lane;
    v = vec[q];
    if (update) {
      v = zr[q] + cg->beta[lane < 3 ? 0 : 1] * v;
      vec[q] = v;
    }
    if (rec) {
      if (lane < 5)
        rec[(size_t)i * 8 + 3 + lane] = (float)v;
      else
        mpz[i] = (float)v;
    }
  } else if (lane < 9 && rec) {
    const float4 p = posf[i];
    rec[(size_t)i * 8 + (lane - 6)] = lane == 6 ? p.x : (lane == 7 ? p.y : p.z);
  }
  if (lane >= 29) stage_axis<T>(g, pos[i], lane - 29, sw[warp]);
  __syncwarp();
  T fd[3], fp[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    fd[d] = (T)(g.a[d] * __shfl_sync(0xffffffffu, v, d));
    fp[d] = (T)(g.a[d] * __shfl_sync(0xffffffffu, v, 3 + d));
  }
  spread_dip_lines<T>(g, sw[warp], lane, fd, fp, grid);
}

template <typename C, typename T>
__global__ void k_qfac(size_t ng, int n1, XOrder xo, const T* __restrict__ qfac, C* __restrict__ grid,
                       const CgScalars* __restrict__ cg, int check_stop) {
  if (check_stop && cg->stop) return;
  size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  size_t stride = (size_t)gridDim.x * blockDim.x;
  for (; q < ng; q += stride) {
    const int k1 = xo.f1 == 1 ? 0 : (int)(q % n1);
    T f = qfac[q - k1 + xo.slot(k1)];
    C v = grid[q];
    v.x *= f;
    v.y *= f;
    grid[q] = v;
  }
}

// fphi_mpole_site (pmestuff.f:453-600) restricted to the 10 components of
// cphi, then fphi_to_cphi_site (:1190) and the E0 assembly of
// newinduce_pme2.f:133-148: ef -= cphi(2:4); ef += term * d_perm.
template <typename T>
__global__ void k_gather_mpole(int n, PmeGeom g, const double4* __restrict__ pos,
                               const typename Cplx<T>::type* __restrict__ grid, const double* __restrict__ rp,
                               double term, double* __restrict__ cphi4, double* __restrict__ cphi10,
                               double* __restrict__ ef) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double4 p = pos[i];
  T tx[kBs][3], ty[kBs][3], tz[kBs][3];
  int gx = bspline_axis<3, T>(p.x, g.recip[0], g.n1, tx);
  int gy = bspline_axis<3, T>(p.y, g.recip[1], g.n2, ty);
  int gz = bspline_axis<3, T>(p.z, g.recip[2], g.n3, tz);
  T tuv000 = 0, tuv100 = 0, tuv010 = 0, tuv001 = 0, tuv200 = 0, tuv020 = 0, tuv002 = 0, tuv110 = 0, tuv101 = 0,
    tuv011 = 0;
#pragma unroll
  for (int c = 0; c < kBs; ++c) {
    size_t kk = (size_t)wrapk(gz + c, g.n3);
    T v0 = tz[c][0], v1 = tz[c][1], v2 = tz[c][2];
    T tu00 = 0, tu10 = 0, tu01 = 0, tu20 = 0, tu11 = 0, tu02 = 0;
#pragma unroll
    for (int b = 0; b < kBs; ++b) {
      size_t jj = (size_t)wrapk(gy + b, g.n2);
      T u0 = ty[b][0], u1 = ty[b][1], u2 = ty[b][2];
      T t0 = 0, t1 = 0, t2 = 0;
      size_t row = (kk * g.n2 + jj) * g.n1;
#pragma unroll
      for (int a = 0; a < kBs; ++a) {
        T tq = grid[row + wrapk(gx + a, g.n1)].x;
        t0 += tq * tx[a][0];
        t1 += tq * tx[a][1];
        t2 += tq * tx[a][2];
      }
      tu00 += t0 * u0;
      tu10 += t1 * u0;
      tu01 += t0 * u1;
      tu20 += t2 * u0;
      tu11 += t1 * u1;
      tu02 += t0 * u2;
    }
    tuv000 += tu00 * v0;
    tuv100 += tu10 * v0;
    tuv010 += tu01 * v0;
    tuv001 += tu00 * v1;
    tuv200 += tu20 * v0;
    tuv020 += tu02 * v0;
    tuv002 += tu00 * v2;
    tuv110 += tu11 * v0;
    tuv101 += tu10 * v1;
    tuv011 += tu01 * v1;
  }
  double c1 = g.a[0] * (double)tuv100, c2 = g.a[1] * (double)tuv010, c3 = g.a[2] * (double)tuv001;
  double* cp = cphi4 + (size_t)i * 4;
  cp[0] = (double)tuv000;
  cp[1] = c1;
  cp[2] = c2;
  cp[3] = c3;
  if (cphi10) {
    double* q = cphi10 + (size_t)i * 10;
    q[0] = (double)tuv000;
    q[1] = c1;
    q[2] = c2;
    q[3] = c3;
    q[4] = g.a[0] * g.a[0] * (double)tuv200;
    q[5] = g.a[1] * g.a[1] * (double)tuv020;
    q[6] = g.a[2] * g.a[2] * (double)tuv002;
    q[7] = g.a[0] * g.a[1] * (double)tuv110;
    q[8] = g.a[0] * g.a[2] * (double)tuv101;
    q[9] = g.a[1] * g.a[2] * (double)tuv011;
  }
  if (ef) {
    const double* r = rp + (size_t)i * 10;
    double* e = ef + (size_t)i * 6;
    double cc[3] = {c1, c2, c3};
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      e[j] = (e[j] - cc[j]) + term * r[1 + j];
      e[3 + j] = (e[3 + j] - cc[j]) + term * r[1 + j];
    }
  }
}

}  // namespace

namespace {

// fphi_uind_site (pmestuff.f:746-1045) field part, one thread per site,
// output dipfield [n][6] (tmatxbrecip, newinduce_pme.f:2094-2121).
template <typename T>
__global__ void __launch_bounds__(128) k_gather_dip(int n, PmeGeom g, const double4* __restrict__ pos,
                                                    const typename Cplx<T>::type* __restrict__ grid,
                                                    double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double o[6];
  gather_dip<T>(g, pos[i], grid, o);
  double2* d = reinterpret_cast<double2*>(out + (size_t)i * 6);
  d[0] = make_double2(o[0], o[1]);
  d[1] = make_double2(o[2], o[3]);
  d[2] = make_double2(o[4], o[5]);
}

// kewald.f:693-717 (bspline) and :747-812 (dftmod)
std::vector<double> dftmod_host(int nfft, int order) {
  std::vector<double> arr(order + 2, 0.0), bsarray(nfft + 2, 0.0), bsmod(nfft + 1, 0.0);
  double x = 0.0;
  arr[1] = 1.0 - x;
  arr[2] = x;
  for (int k = 3; k <= order; ++k) {
    double denom = 1.0 / (double)(k - 1);
    arr[k] = x * arr[k - 1] * denom;
    for (int i = 1; i <= k - 2; ++i) arr[k - i] = ((x + i) * arr[k - i - 1] + ((k - i) - x) * arr[k - i]) * denom;
    arr[1] = (1.0 - x) * arr[1] * denom;
  }
  for (int i = 2; i <= order + 1 && i <= nfft; ++i) bsarray[i] = arr[i - 1];
  double factor = 2.0 * kPi / (double)nfft;
  for (int i = 1; i <= nfft; ++i) {
    double s1 = 0.0, s2 = 0.0;
    for (int j = 1; j <= nfft; ++j) {
      double arg = factor * (double)((i - 1) * (j - 1));
      s1 += bsarray[j] * cos(arg);
      s2 += bsarray[j] * sin(arg);
    }
    bsmod[i] = s1 * s1 + s2 * s2;
  }
  double eps = 1.0e-7;
  if (bsmod[1] < eps) bsmod[1] = 0.5 * bsmod[2];
  for (int i = 2; i <= nfft - 1; ++i)
    if (bsmod[i] < eps) bsmod[i] = 0.5 * (bsmod[i - 1] + bsmod[i + 1]);
  if (bsmod[nfft] < eps) bsmod[nfft] = 0.5 * bsmod[nfft - 1];
  for (int i = 1; i <= nfft; ++i) {
    int k = i - 1;
    if (i > nfft / 2) k -= nfft;
    double zeta = 1.0;
    if (k != 0) {
      double s1 = 1.0, s2 = 1.0, fac = kPi * (double)k / (double)nfft;
      for (int j = 1; j <= 50; ++j) {
        double arg = fac / (fac + kPi * j);
        s1 += pow(arg, order);
        s2 += pow(arg, 2 * order);
      }
      for (int j = 1; j <= 50; ++j) {
        double arg = fac / (fac - kPi * j);
        s1 += pow(arg, order);
        s2 += pow(arg, 2 * order);
      }
      zeta = s2 / s1;
    }
    bsmod[i] = bsmod[i] * zeta * zeta;
  }
  return bsmod;
}

PmeGeom geom_of(const Ctx& c) {
  PmeGeom g;
  g.n1 = c.nfft[0];
  g.n2 = c.nfft[1];
  g.n3 = c.nfft[2];
  for (int d = 0; d < 3; ++d) {
    g.recip[d] = c.box.recip[d];
    g.a[d] = c.a_frac[d];
  }
  return g;
}

// Process-wide cache of cuFFT plans by device, dimensions and type: a
// context that is destroyed or re-targeted to another grid gives its plan
// back, and the next context of that shape takes it instead of planning
// again (planning allocates a work area and can take milliseconds).
struct PlanKey {
  int device, n1, n2, n3, mixed;
  bool operator==(const PlanKey& o) const {
    return device == o.device && n1 == o.n1 && n2 == o.n2 && n3 == o.n3 && mixed == o.mixed;
  }
};
std::mutex g_plan_mu;
std::vector<std::pair<PlanKey, cufftHandle>> g_plans;
constexpr size_t kMaxCachedPlans = 64;

bool take_plan(const PlanKey& k, cufftHandle* out) {
  std::lock_guard<std::mutex> g(g_plan_mu);
  for (size_t q = 0; q < g_plans.size(); ++q)
    if (g_plans[q].first == k) {
      *out = g_plans[q].second;
      g_plans.erase(g_plans.begin() + q);
      return true;
    }
  return false;
}

void give_plan(const PlanKey& k, cufftHandle plan) {
  std::lock_guard<std::mutex> g(g_plan_mu);
  if (g_plans.size() >= kMaxCachedPlans) {
    cufftDestroy(g_plans.front().second);
    g_plans.erase(g_plans.begin());
  }
  g_plans.emplace_back(k, plan);
}

PlanKey plan_key(const Ctx& c) { return PlanKey{c.device, c.plan_dims[0], c.plan_dims[1], c.plan_dims[2], c.mixed}; }

bool plan_cached(const PlanKey& k) {
  std::lock_guard<std::mutex> g(g_plan_mu);
  for (const auto& p : g_plans)
    if (p.first == k) return true;
  return false;
}

// the context's plan of its grid (cuFFT dims: slowest first; data [n3][n2][n1]),
// from the cache or new; not under capture
int make_plan(Ctx& c) {
  if (!take_plan(plan_key(c), &c.plan) &&
      cufftPlan3d(&c.plan, c.nfft[2], c.nfft[1], c.nfft[0], c.mixed ? CUFFT_C2C : CUFFT_Z2Z) != CUFFT_SUCCESS) {
    cudaGetLastError();  // the allocation cuFFT was refused: reported here, not by the next launch's check
    c.last_msg = "cufftPlan3d failed";
    return THP_E_CUDA;
  }
  c.have_plan = true;
  cufftSetStream(c.plan, c.stream);
  return THP_OK;
}

// cuFFT of the whole grid: forward in place, inverse into d_conv (d_grid
// itself without the three-kernel convolution)
int fft(Ctx& c, int dir) {
  cufftResult r;
  void* out = dir == CUFFT_FORWARD ? c.d_grid : c.d_conv;
  if (c.mixed)
    r = cufftExecC2C(c.plan, (cufftComplex*)c.d_grid, (cufftComplex*)out, dir);
  else
    r = cufftExecZ2Z(c.plan, (cufftDoubleComplex*)c.d_grid, (cufftDoubleComplex*)out, dir);
  if (r != CUFFT_SUCCESS) {
    c.last_msg = "cuFFT exec failed";
    return THP_E_CUDA;
  }
  return THP_OK;
}

// d_grid to zero: what cuFFT's transforms in place leave has to go before
// the next spread; the three-kernel convolution zeroes what it reads
int clear_grid(Ctx& c) {
  size_t csz = c.mixed ? sizeof(cufftComplex) : sizeof(cufftDoubleComplex);
  return cuda_status(cudaMemsetAsync(c.d_grid, 0, csz * c.ngrid, c.stream), &c, "zero grid");
}

// d_grid -> d_conv: forward transform, influence function, inverse
// transform.  Three kernels where the grid allows (at 120^3: 73 -> 38 us FP32,
// 98 -> 53 us FP64 against cuFFT's six launches and the product; 60^3 34 -> 15 us), else
// cuFFT.  real (three-kernel form only): one real per point in the front of
// d_grid, the result in d_pot.
int convolve(Ctx& c, int check_stop, bool real = false) {
  if (c.conv) {
    const conv::Sys s{c.d_grid, c.d_conv, c.d_qfac, c.d_cg, c.d_pot};
    const cudaError_t e = c.mixed ? launch_conv32(c.nfft[0], s, nullptr, 1, check_stop, real, c.stream)
                                  : launch_conv64(c.nfft[0], s, nullptr, 1, check_stop, real, c.stream);
    return spread_status(c, cuda_status(e, &c, "convolution"));
  }
  int st = fft(c, CUFFT_FORWARD);
  if (st) return st;
  const int blocks = 148 * 8;
  const XOrder xo{c.conv_r[0], c.conv_r[1]};
  if (c.mixed)
    k_qfac<cufftComplex, float><<<blocks, 256, 0, c.stream>>>(c.ngrid, c.nfft[0], xo, (const float*)c.d_qfac,
                                                             (cufftComplex*)c.d_grid, c.d_cg, check_stop);
  else
    k_qfac<cufftDoubleComplex, double><<<blocks, 256, 0, c.stream>>>(
        c.ngrid, c.nfft[0], xo, (const double*)c.d_qfac, (cufftDoubleComplex*)c.d_grid, c.d_cg, check_stop);
  st = cuda_status(cudaGetLastError(), &c, "qfac");
  if (st) return st;
  return fft(c, CUFFT_INVERSE);
}

// qfac(k) = exp(-pi^2 h^2 / a^2) / (pi V h^2 bsmod1 bsmod2 bsmod3), zero at
// h = 0 and where the exponent is below -50 (newinduce_pme.f:1802-1854)
template <typename T>
__global__ void k_qfac_init(int n1, int n2, int n3, const double* __restrict__ bsm, double r1, double r2, double r3,
                            double pterm, double volterm, XOrder xo, T* __restrict__ q) {
  const size_t ng = (size_t)n1 * n2 * n3;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < ng; t += (size_t)gridDim.x * blockDim.x) {
    const int k1 = (int)(t % n1), k2 = (int)((t / n1) % n2), k3 = (int)(t / ((size_t)n1 * n2));
    const int m1 = k1 < (n1 + 1) / 2 ? k1 : k1 - n1;
    const int m2 = k2 < (n2 + 1) / 2 ? k2 : k2 - n2;
    const int m3 = k3 < (n3 + 1) / 2 ? k3 : k3 - n3;
    double v = 0.0;
    if (m1 != 0 || m2 != 0 || m3 != 0) {
      const double h1 = r1 * m1, h2 = r2 * m2, h3 = r3 * m3;
      const double hsq = h1 * h1 + h2 * h2 + h3 * h3;
      const double term = -pterm * hsq;
      if (term > -50.0) v = exp(term) / (volterm * hsq * bsm[k1] * bsm[n1 + k2] * bsm[n1 + n2 + k3]);
    }
    q[t - k1 + xo.slot(k1)] = (T)v;
  }
}

}  // namespace

// the context's grid has a plan (a grid that the three-kernel convolution
// covers is made without one)
int ensure_plan(Ctx& c) { return c.have_plan ? THP_OK : make_plan(c); }

bool conv_covers(const int n[3], int mixed, int* r1, int* r2) {
  if (n[0] != n[1] || n[1] != n[2]) return false;
  return mixed ? conv_split32(n[0], r1, r2) : conv_split64(n[0], r1, r2);
}

// B-spline moduli by grid length, computed once per process (an O(K^2)
// trigonometric sum per axis; servers re-target contexts to new grids often)
static const std::vector<double>& dftmod_cached(int nfft) {
  static std::mutex mu;
  static std::map<int, std::vector<double>> cache;
  std::lock_guard<std::mutex> g(mu);
  auto it = cache.find(nfft);
  if (it == cache.end()) it = cache.emplace(nfft, dftmod_host(nfft, kBs)).first;
  return it->second;  // map nodes are stable: the reference outlives the lock
}

static void free_grids(Ctx& c) {
  cudaFree(c.d_grids);
  cudaFree(c.d_convs);
  for (void** p : {&c.d_grids, &c.d_convs, &c.d_qfac, &c.d_grid, &c.d_conv_buf, &c.d_pot}) *p = nullptr;
  c.cap_ngrid = c.cap_conv = 0;
}

// The grid arrays in one allocation, each on a 256-byte boundary.  They are kept
// while they are large enough (a re-targeted context reuses them).  Only the
// three-kernel convolution needs the second grid and the potential: a context
// made for another grid gets them, apart, when it first serves one, and nothing
// is freed (cudaFree would stall the other contexts of a server).
static int size_grids(Ctx& c) {
  const size_t esz = c.mixed ? sizeof(float) : sizeof(double);
  const size_t csz = c.mixed ? sizeof(cufftComplex) : sizeof(cufftDoubleComplex);
  struct Array {
    void** p;
    size_t bytes;
  };
  auto take = [&](void** base, std::initializer_list<Array> arrays) {
    size_t total = 0;
    for (const Array& g : arrays) total += (g.bytes + 255) / 256 * 256;
    if (cuda_status(cudaMalloc(base, total), &c, "alloc grid")) return false;
    char* at = static_cast<char*>(*base);
    for (const Array& g : arrays) {
      *g.p = at;
      at += (g.bytes + 255) / 256 * 256;
    }
    return true;
  };
  const size_t n = c.ngrid, nconv = c.conv ? n : 0;
  if (n > c.cap_ngrid) {
    const size_t mc = std::max(nconv, c.cap_conv);
    free_grids(c);
    if (!take(&c.d_grids, {{&c.d_grid, csz * n}, {&c.d_qfac, esz * n}, {&c.d_conv_buf, csz * mc}, {&c.d_pot, esz * mc}}))
      return THP_E_CUDA;
    c.cap_ngrid = n;
    c.cap_conv = mc;
  } else if (nconv > c.cap_conv) {
    cudaFree(c.d_convs);
    c.d_convs = nullptr;
    c.cap_conv = 0;
    if (!take(&c.d_convs, {{&c.d_conv_buf, csz * nconv}, {&c.d_pot, esz * nconv}})) return THP_E_CUDA;
    c.cap_conv = nconv;
  }
  return THP_OK;
}

int pme_init(Ctx& c) {
  for (int d = 0; d < 3; ++d) c.nfft[d] = c.cfg.nfft[d];
  c.ngrid = (size_t)c.nfft[0] * c.nfft[1] * c.nfft[2];
  for (int d = 0; d < 3; ++d) c.a_frac[d] = (double)c.nfft[d] * c.box.recip[d];
  // influence function (newinduce_pme.f:1802-1854)
  const std::vector<double>& m1 = dftmod_cached(c.nfft[0]);
  const std::vector<double>& m2 = dftmod_cached(c.nfft[1]);
  const std::vector<double>& m3 = dftmod_cached(c.nfft[2]);
  const size_t csz = c.mixed ? sizeof(cufftComplex) : sizeof(cufftDoubleComplex);
  c.conv_r[0] = c.conv_r[1] = 1;
  c.conv = conv_covers(c.nfft, c.mixed, &c.conv_r[0], &c.conv_r[1]) ? 1 : 0;
  const XOrder xo{c.conv_r[0], c.conv_r[1]};
  if (int st = size_grids(c)) return st;
  c.d_conv = c.conv ? c.d_conv_buf : c.d_grid;
  // influence function on the device (newinduce_pme.f:1802-1854): the
  // B-spline moduli go through the front of the grid buffer
  std::vector<double> bsm(m1.begin() + 1, m1.begin() + 1 + c.nfft[0]);
  bsm.insert(bsm.end(), m2.begin() + 1, m2.begin() + 1 + c.nfft[1]);
  bsm.insert(bsm.end(), m3.begin() + 1, m3.begin() + 1 + c.nfft[2]);
  double* d_bsm = reinterpret_cast<double*>(c.d_grid);  // ngrid complex >= n1+n2+n3 doubles
  cudaMemcpyAsync(d_bsm, bsm.data(), sizeof(double) * bsm.size(), cudaMemcpyHostToDevice, c.stream);
  const double a = c.cfg.aewald;
  const double pterm = (kPi / a) * (kPi / a);
  const double volterm = kPi * (c.cfg.box[0] * c.cfg.box[1] * c.cfg.box[2]);
  const int blocks = (int)std::min<size_t>((c.ngrid + 255) / 256, 148 * 16);
  if (c.mixed)
    k_qfac_init<float><<<blocks, 256, 0, c.stream>>>(c.nfft[0], c.nfft[1], c.nfft[2], d_bsm, c.box.recip[0],
                                                     c.box.recip[1], c.box.recip[2], pterm, volterm, xo,
                                                     (float*)c.d_qfac);
  else
    k_qfac_init<double><<<blocks, 256, 0, c.stream>>>(c.nfft[0], c.nfft[1], c.nfft[2], d_bsm, c.box.recip[0],
                                                      c.box.recip[1], c.box.recip[2], pterm, volterm, xo,
                                                      (double*)c.d_qfac);
  // the spread grid is zero from here on between convolutions
  if (c.conv) cudaMemsetAsync(c.d_grid, 0, csz * c.ngrid, c.stream);
  // no host wait: the influence function is ready, stream-ordered, for the
  // context's next solve (bsm is copied out before the call returns)
  if (cuda_status(cudaGetLastError(), &c, "qfac")) return THP_E_CUDA;
  // the plan is kept when the grid dimensions are unchanged; a grid that the
  // three-kernel convolution covers gets one when the virial is switched on
  const bool same = c.plan_dims[0] == c.nfft[0] && c.plan_dims[1] == c.nfft[1] && c.plan_dims[2] == c.nfft[2];
  if (!same) {
    if (c.have_plan) give_plan(plan_key(c), c.plan);
    c.have_plan = false;
    for (int d = 0; d < 3; ++d) c.plan_dims[d] = c.nfft[d];
  }
  if (!c.conv || c.want_virial) {
    if (int st = ensure_plan(c)) return st;
  }
  if (c.have_plan) cufftSetStream(c.plan, c.stream);
  return cuda_status(cudaGetLastError(), &c, "pme init");
}

// Plans one grid shape ahead of use (a server does this when a system is
// registered, so the first request of a new shape does not wait for it).
int plan_prefetch(int device, const int nfft[3], int mixed) {
  const PlanKey k{device, nfft[0], nfft[1], nfft[2], mixed};
  int r1, r2;
  if (conv_covers(nfft, mixed, &r1, &r2) || plan_cached(k)) return THP_OK;
  if (cudaSetDevice(device) != cudaSuccess) return THP_E_CUDA;
  cufftHandle plan;
  if (cufftPlan3d(&plan, nfft[2], nfft[1], nfft[0], mixed ? CUFFT_C2C : CUFFT_Z2Z) != CUFFT_SUCCESS)
    return THP_E_CUDA;
  give_plan(k, plan);
  return THP_OK;
}

void pme_free(Ctx& c) {
  if (c.have_plan) give_plan(plan_key(c), c.plan);
  c.have_plan = false;
  free_grids(c);
  c.d_conv = nullptr;
}

int zero_grid(Ctx& c) { return c.conv ? THP_OK : clear_grid(c); }

// Status st of a step between a spread and the end of its convolution.  After a
// failure no convolution will zero the charges, so they are cleared here: the
// next spread into a covered grid does not.
int spread_status(Ctx& c, int st) {
  if (st && c.conv) clear_grid(c);
  return st;
}

static int spread_mpole(Ctx& c, const PmeGeom& g) {
  const bool small = c.n < kLargeAtoms;
  const int nb = small ? (c.n + 3) / 4 : (c.n + kBlock - 1) / kBlock;
  cufftComplex* gf = (cufftComplex*)c.d_grid;
  cufftDoubleComplex* gd = (cufftDoubleComplex*)c.d_grid;
  if (c.mixed && small)
    k_spread_mpole_small<float><<<nb, kBlock, 0, c.stream>>>(c.n, g, c.d_pos, c.d_rpole, gf);
  else if (c.mixed)
    k_spread_mpole<float><<<nb, kBlock, 0, c.stream>>>(c.n, g, c.d_pos, c.d_rpole, gf);
  else if (small)
    k_spread_mpole_small<double><<<nb, kBlock, 0, c.stream>>>(c.n, g, c.d_pos, c.d_rpole, gd);
  else
    k_spread_mpole<double><<<nb, kBlock, 0, c.stream>>>(c.n, g, c.d_pos, c.d_rpole, gd);
  return spread_status(c, cuda_status(cudaGetLastError(), &c, "spread mpole"));
}

// Permanent-multipole PME: d_cphi (and cphi10 when non-null) and, when
// with_e0, completes d_ef = E_direct - cphi(2:4) + (4/3) a^3/sqrt(pi) d.
int launch_mpole_grid(Ctx& c) {
  PmeGeom g = geom_of(c);
  int st = zero_grid(c);
  if (st) return st;
  if ((st = spread_mpole(c, g))) return st;
  return convolve(c, 0);
}

// blocks of the k-space virial sums (each writes 6 partial sums)
int kspace_virial_blocks() { return 148 * 2; }

static int kspace_virial(Ctx& c, int mode, double sign, double* d_part) {
  const double pterm = (kPi / c.cfg.aewald) * (kPi / c.cfg.aewald);
  const PmeGeom g = geom_of(c);
  const XOrder xo{c.conv_r[0], c.conv_r[1]};
  if (c.mixed)
    k_kspace_virial<cufftComplex, float><<<kspace_virial_blocks(), 256, 0, c.stream>>>(
        g.n1, g.n2, g.n3, xo, (const cufftComplex*)c.d_grid, (const float*)c.d_qfac, g.recip[0], g.recip[1],
        g.recip[2], pterm, kElectric, mode, sign, d_part);
  else
    k_kspace_virial<cufftDoubleComplex, double><<<kspace_virial_blocks(), 256, 0, c.stream>>>(
        g.n1, g.n2, g.n3, xo, (const cufftDoubleComplex*)c.d_grid, (const double*)c.d_qfac, g.recip[0], g.recip[1],
        g.recip[2], pterm, kElectric, mode, sign, d_part);
  return cuda_status(cudaGetLastError(), &c, "k-space virial");
}

// launch_mpole_grid with, between the forward transform and qfac, the
// permanent-only scalar-sum virial (emrecip1), subtracted as eprecip1 does
// (epolar1.f:534-541): kspace_virial_blocks() rows of 6 into d_part.
int launch_mpole_grid_virial(Ctx& c, double* d_part, double sign) {
  PmeGeom g = geom_of(c);
  int st = ensure_plan(c);
  if (st) return st;
  if ((st = zero_grid(c))) return st;
  if ((st = spread_mpole(c, g))) return st;
  if ((st = fft(c, CUFFT_FORWARD))) return spread_status(c, st);
  if ((st = kspace_virial(c, 0, sign, d_part))) return spread_status(c, st);
  const int blocks = 148 * 8;
  const XOrder xo{c.conv_r[0], c.conv_r[1]};
  if (c.mixed)
    k_qfac<cufftComplex, float><<<blocks, 256, 0, c.stream>>>(c.ngrid, c.nfft[0], xo, (const float*)c.d_qfac,
                                                             (cufftComplex*)c.d_grid, c.d_cg, 0);
  else
    k_qfac<cufftDoubleComplex, double><<<blocks, 256, 0, c.stream>>>(
        c.ngrid, c.nfft[0], xo, (const double*)c.d_qfac, (cufftDoubleComplex*)c.d_grid, c.d_cg, 0);
  if ((st = cuda_status(cudaGetLastError(), &c, "qfac"))) return spread_status(c, st);
  if ((st = fft(c, CUFFT_INVERSE))) return spread_status(c, st);
  return c.conv ? clear_grid(c) : THP_OK;
}

// The (rpole + uinp) x (rpole + uind) scalar-sum virial of eprecip1
// (epolar1.f:932-1091) into kspace_virial_blocks() rows of d_part; uses
// (and leaves transformed) the context's grid.
int launch_pair_grid_virial(Ctx& c, double* d_part) {
  PmeGeom g = geom_of(c);
  int nb = (c.n + kBlock - 1) / kBlock;
  int st = ensure_plan(c);
  if (st) return st;
  if ((st = zero_grid(c))) return st;
  if (c.mixed)
    k_spread_mpole2<float><<<nb, kBlock, 0, c.stream>>>(c.n, g, c.d_pos, c.d_rpole, c.d_mu, (cufftComplex*)c.d_grid);
  else
    k_spread_mpole2<double><<<nb, kBlock, 0, c.stream>>>(c.n, g, c.d_pos, c.d_rpole, c.d_mu,
                                                         (cufftDoubleComplex*)c.d_grid);
  if ((st = cuda_status(cudaGetLastError(), &c, "spread mpole pair"))) return spread_status(c, st);
  if ((st = fft(c, CUFFT_FORWARD))) return spread_status(c, st);
  if ((st = kspace_virial(c, 1, 1.0, d_part))) return spread_status(c, st);
  return c.conv ? clear_grid(c) : THP_OK;
}

int launch_efld0_recip_ex(Ctx& c, double* cphi10, bool with_e0) {
  int st = launch_mpole_grid(c);
  if (st) return st;
  return launch_gather_mpole(c, cphi10, with_e0);
}

int launch_gather_mpole(Ctx& c, double* cphi10, bool with_e0) {
  PmeGeom g = geom_of(c);
  int nb = (c.n + kBlock - 1) / kBlock;
  double a = c.cfg.aewald;
  double term = (4.0 / 3.0) * a * a * a / kSqrtPi;
  if (c.mixed)
    k_gather_mpole<float><<<nb, kBlock, 0, c.stream>>>(c.n, g, c.d_pos, (const cufftComplex*)c.d_conv, c.d_rpole,
                                                       term, c.d_cphi, cphi10, with_e0 ? c.d_ef : nullptr);
  else
    k_gather_mpole<double><<<nb, kBlock, 0, c.stream>>>(c.n, g, c.d_pos, (const cufftDoubleComplex*)c.d_conv,
                                                        c.d_rpole, term, c.d_cphi, cphi10,
                                                        with_e0 ? c.d_ef : nullptr);
  return cuda_status(cudaGetLastError(), &c, "gather mpole");
}

int launch_efld0_recip(Ctx& c) { return launch_efld0_recip_ex(c, nullptr, true); }

// 1: the dipole spread of systems of at least THP_SPREAD_TILE_ATOMS (FP32
// grid) / THP_SPREAD_TILE_ATOMS_F64 atoms sums the stencils of 16
// neighbouring sites in a shared-memory tile per warp before adding them to
// the grid (at 288k atoms 105 -> 85 us per FP32 spread, 340 -> 200 us FP64);
// smaller systems, and 0, let every site add its own stencil (measured
// faster below those sizes: mixed solves of 4.5k-32k atoms against the tile's
// gain from 96k; FP64 solves of 4.5k-12k atoms against its gain from 32k).
#ifndef THP_SPREAD_TILE
#define THP_SPREAD_TILE 1
#endif
#ifndef THP_SPREAD_TILE_ATOMS
#define THP_SPREAD_TILE_ATOMS 50000
#endif
#ifndef THP_SPREAD_TILE_ATOMS_F64
#define THP_SPREAD_TILE_ATOMS_F64 20000
#endif

template <typename T, typename V, int TA>
static void spread_tiled(Ctx& c, const PmeGeom& g, const V* vec, int check_stop, typename Cplx<T>::type* grid) {
  constexpr size_t smem = sizeof(SpreadWarp<T>) * (kSpreadThreads / 32);
  static std::atomic<unsigned long long> limit_set{0};
  smem_limit_once(k_spread_dip<T, V, TA>, smem, limit_set);
  const int nb = (c.n + kSpreadThreads - 1) / kSpreadThreads;
  k_spread_dip<T, V, TA><<<nb, kSpreadThreads, smem, c.stream>>>(c.n, g, c.d_pos, vec, c.d_cg, check_stop, grid);
}

template <typename T, typename V>
static void spread_dipoles(Ctx& c, const PmeGeom& g, const V* vec, int check_stop, typename Cplx<T>::type* grid) {
  constexpr int kMin = std::is_same<T, float>::value ? THP_SPREAD_TILE_ATOMS : THP_SPREAD_TILE_ATOMS_F64;
  if (THP_SPREAD_TILE && c.n >= kMin) {
    spread_tiled<T, V, 16>(c, g, vec, check_stop, grid);
  } else if constexpr (std::is_same<V, double>::value) {
    if (c.n < kLargeAtoms) {
      k_spread_dip_small<T><<<(c.n + 3) / 4, 128, 0, c.stream>>>(c.n, g, c.d_pos, const_cast<double*>(vec), nullptr,
                                                                c.d_cg, check_stop, 0, nullptr, nullptr, nullptr, grid);
      return;
    }
    k_spread_dip<T, V, 0><<<(c.n + kBlock - 1) / kBlock, kBlock, 0, c.stream>>>(c.n, g, c.d_pos, vec, c.d_cg,
                                                                               check_stop, grid);
  } else {
    k_spread_dip<T, V, 0><<<(c.n + kBlock - 1) / kBlock, kBlock, 0, c.stream>>>(c.n, g, c.d_pos, vec, c.d_cg,
                                                                               check_stop, grid);
  }
}

int launch_convolve(Ctx& c, int check_stop, bool real) { return convolve(c, check_stop, real); }

// Spread of the small systems' CG vector (warp per site): update forms
// pp = zr + beta pp first; the mixed form also writes the partner records.
// The convolution is the caller's.
int launch_spread_small(Ctx& c, double* d_vec, int update) {
  const PmeGeom g = geom_of(c);
  int st = zero_grid(c);
  if (st) return st;
  const int nb = (c.n + 3) / 4;
  if (c.mixed)
    k_spread_dip_small<float><<<nb, 128, 0, c.stream>>>(c.n, g, c.d_pos, d_vec, c.d_zr, c.d_cg, update, update,
                                                        c.d_posf, c.d_rec, c.d_mpz, (cufftComplex*)c.d_grid);
  else
    k_spread_dip_small<double><<<nb, 128, 0, c.stream>>>(c.n, g, c.d_pos, d_vec, c.d_zr, c.d_cg, update, update,
                                                         nullptr, nullptr, nullptr, (cufftDoubleComplex*)c.d_grid);
  return spread_status(c, cuda_status(cudaGetLastError(), &c, "spread dip"));
}

// Dipole PME pass: spread of d_vec [n][6] and the convolution.  d_out (if
// non-null) receives the gathered field gradient [n][6] (tmatxbrecip's
// dipfield); the CG loop passes null and gathers inside its combine kernel.
int launch_pme_dipole(Ctx& c, const double* d_vec, double* d_out, int check_stop) {
  PmeGeom g = geom_of(c);
  int st = zero_grid(c);
  if (st) return st;
  if (c.mixed)
    spread_dipoles<float, double>(c, g, d_vec, check_stop, (cufftComplex*)c.d_grid);
  else
    spread_dipoles<double, double>(c, g, d_vec, check_stop, (cufftDoubleComplex*)c.d_grid);
  if ((st = cuda_status(cudaGetLastError(), &c, "spread dip"))) return spread_status(c, st);
  if ((st = convolve(c, check_stop))) return st;
  if (d_out) st = launch_gather_dip(c, d_out);
  return st;
}

// The overlapped mixed CG's spread of its FP32 search direction, then the
// convolution.
int launch_pme_dipole_f32(Ctx& c, const float* d_vec, int check_stop) {
  PmeGeom g = geom_of(c);
  int st = zero_grid(c);
  if (st) return st;
  spread_dipoles<float, float>(c, g, d_vec, check_stop, (cufftComplex*)c.d_grid);
  if ((st = cuda_status(cudaGetLastError(), &c, "spread dip"))) return spread_status(c, st);
  return convolve(c, check_stop);
}

int launch_gather_dip(Ctx& c, double* d_out) {
  PmeGeom g = geom_of(c);
  const int nb = (c.n + kBlock - 1) / kBlock;
  if (c.mixed)
    k_gather_dip<float><<<nb, kBlock, 0, c.stream>>>(c.n, g, c.d_pos, (const cufftComplex*)c.d_conv, d_out);
  else
    k_gather_dip<double><<<nb, kBlock, 0, c.stream>>>(c.n, g, c.d_pos, (const cufftDoubleComplex*)c.d_conv, d_out);
  return cuda_status(cudaGetLastError(), &c, "gather dip");
}

PmeGeom pme_geom(const Ctx& c) { return geom_of(c); }

}  // namespace thp
