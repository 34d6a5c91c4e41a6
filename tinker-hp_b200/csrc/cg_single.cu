// cg_single.cu -- the CG of a system whose d and p dipoles are the same.
//
// The d and p direct fields differ only through the scales of the special pairs
// (efld0_direct, newinduce_pme.f:1062-1136).  Where every pair has the same two
// scales -- molecules whose 1-2 and 1-3 neighbours are their whole polarization
// group, as water -- the two right-hand sides of inducepcg_pme2
// (newinduce_pme2.f:285-636) are equal, and so are the solutions, the CG scalars
// and the stop test of both.  The solve then runs once, with vectors [n][3] and
// a PME grid of one real per point, and writes its dipoles to both sets: half
// the vector and grid bytes, half the reductions of the spread, 32-byte partner
// records without a side array.
//
// The kernels are those of solver.cu with three components; per iteration:
//   n >= kLargeAtoms: pp and records; row beside tiled spread + convolution;
//                      combine; update
//   smaller:           spread (forms pp and the records, a warp per site); row
//                      beside the convolution; combine (8 lanes per atom); update
#include "cg_dev.cuh"
#include "conv.h"
#include "kernels.h"

namespace thp {

int group_blocks(int n, int block);

namespace {

using namespace cg;

template <typename V>
__device__ __forceinline__ void load3(const V* __restrict__ p, double (&v)[3]) {
#pragma unroll
  for (int q = 0; q < 3; ++q) v[q] = (double)p[q];
}
template <typename V>
__device__ __forceinline__ void store3(V* __restrict__ p, const double (&v)[3]) {
#pragma unroll
  for (int q = 0; q < 3; ++q) p[q] = (V)v[q];
}

// ---- spread of one real per grid point ------------------------------------------

__device__ __forceinline__ void red_vec(float* a, const float (&v)[2]) { red_add2(a, v[0], v[1]); }
__device__ __forceinline__ void red_vec(float* a, const float (&v)[4]) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(a), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3])
               : "memory");
}
__device__ __forceinline__ void red_vec(double* a, const double (&v)[1]) { red_add(a, v[0]); }

// a warp's tile: SpreadWarp for reals
template <typename T>
struct SpreadWarp1 {
  static constexpr int kPts = SpreadWarp<T>::kPts;
  T w[32][kSpreadRec];  // tx, ty, tz (10 each), scaled dipole
  int4 off[32];
  T tile[kPts];
};

// Adds the tile's nonzero points to the grid, G neighbouring points (starting
// on a multiple of G) per reduction, and zeroes them; the row length is a
// multiple of G.  Lines in (z, y) order as spread_tile_pass flushes them.
template <typename T, int G>
__device__ __forceinline__ void flush_tile1(const PmeGeom& g, int lane, int x0, int y0, int z0, int X, int Y, int Z,
                                            int SY, int SZ, T* __restrict__ tile, T* __restrict__ grid) {
  const int shift = -(x0 & (G - 1));            // tile column of the line's first group
  const int cols = (X - shift + G - 1) / G;     // groups per line
  const int xw = cols <= 4 ? 4 : (cols <= 8 ? 8 : (cols <= 16 ? 16 : 32));
  const int per = 32 / xw, c = lane & (xw - 1);
  const bool cin = c < cols;
  const int xa = shift + G * c;
  const size_t xi = (size_t)wrapk(x0 + (cin ? xa : 0), g.n1);
  int z = 0, y = lane / xw;
  int wz = wrapk(z0, g.n3), wy = wrapk(y0, g.n2) + y;
  if (wy >= g.n2) wy -= g.n2;
  const int ymod = Y % g.n2;
  for (int L = lane / xw; L < Y * Z; L += per) {
    while (y >= Y) {
      y -= Y;
      wy -= ymod;
      if (wy < 0) wy += g.n2;
      ++z;
      if (++wz == g.n3) wz = 0;
    }
    if (cin) {
      T* q = tile + z * SZ + y * SY + xa;
      T v[G];
      bool any = false;
#pragma unroll
      for (int u = 0; u < G; ++u) {
        const bool in = xa + u >= 0 && xa + u < X;
        v[u] = in ? q[u] : T(0);
        any |= v[u] != T(0);
      }
      if (any) {
#pragma unroll
        for (int u = 0; u < G; ++u)
          if (xa + u >= 0 && xa + u < X) q[u] = T(0);
        red_vec(grid + ((size_t)wz * g.n2 + wy) * g.n1 + xi, v);
      }
    }
    y += per;
    wy += per;
    if (wy >= g.n2) wy -= g.n2;
  }
}

// spread_tile_pass for reals: the sites in mk summed in the tile and flushed;
// false, having done nothing, when their stencils do not fit.
template <typename T>
__device__ __forceinline__ bool spread_tile_pass1(const PmeGeom& g, unsigned mk, int lane, int gx, int gy, int gz,
                                                  T* __restrict__ grid, SpreadWarp1<T>& s) {
  using T2 = typename Pair<T>::type;
  const bool mine = (mk >> lane) & 1u;
  int x0, y0, z0;
  const int lx = tile_axis(mine, gx, g.n1, x0), ly = tile_axis(mine, gy, g.n2, y0), lz = tile_axis(mine, gz, g.n3, z0);
  const int X = __reduce_max_sync(~0u, mine ? lx : INT_MIN) - x0 + kBs;
  const int Y = __reduce_max_sync(~0u, mine ? ly : INT_MIN) - y0 + kBs;
  const int Z = __reduce_max_sync(~0u, mine ? lz : INT_MIN) - z0 + kBs;
  // SY odd and SZ = 5 SY modulo the banks of one phase: the 25 lines of a
  // stencil fall on distinct banks
  constexpr int kBank = std::is_same<T, float>::value ? 31 : 15;
  const int SY = X | 1;
  const int SZ = Y * SY + ((5 * SY - Y * SY) & kBank);
  if (X > 32 || Z > SpreadWarp1<T>::kPts || Z * SZ > SpreadWarp1<T>::kPts) return false;
  if (mine) s.off[lane] = make_int4(lx - x0, ly - y0, lz - z0, 0);
  __syncwarp();
  const int dy = lane % 5, dz = lane / 5;
  const int lane_off = dz * SZ + dy * SY;
  for (unsigned mm = mk; mm; mm &= mm - 1) {
    const int a = __ffs(mm) - 1;
    if (lane < 25) {
      const T* r = s.w[a];
      const int4 o = s.off[a];
      const T2 u = *reinterpret_cast<const T2*>(r + 10 + 2 * dy);
      const T2 vz = *reinterpret_cast<const T2*>(r + 20 + 2 * dz);
      const T2 f0 = *reinterpret_cast<const T2*>(r + 30);
      const T f2 = r[32];
      T t[2 * kBs];
      tx_pairs(r, t);
      const T term0 = f0.y * u.y * vz.x + f2 * u.x * vz.y, term1 = f0.x * u.x * vz.x;
      T* q = s.tile + lane_off + o.z * SZ + o.y * SY + o.x;
#pragma unroll
      for (int k = 0; k < kBs; ++k) q[k] += term0 * t[2 * k] + term1 * t[2 * k + 1];
    }
    __syncwarp();
  }
  if constexpr (std::is_same<T, float>::value) {
    if ((g.n1 & 3) == 0)
      flush_tile1<T, 4>(g, lane, x0, y0, z0, X, Y, Z, SY, SZ, s.tile, grid);
    else  // the convolution's lengths are all even
      flush_tile1<T, 2>(g, lane, x0, y0, z0, X, Y, Z, SY, SZ, s.tile, grid);
  } else {
    flush_tile1<T, 1>(g, lane, x0, y0, z0, X, Y, Z, SY, SZ, s.tile, grid);
  }
  __syncwarp();
  return true;
}

// Systems below this many atoms give a warp 16 sites (one tile) instead of 32: a
// cold solve (FP64 / mixed) of 60,000 atoms 2073 / 1303 us (32 sites 2108 / 1314),
// 96,000 2931 / 1712 (2943 / 1730), 135,000 3764 / 2199 (3755 / 2206), 240,000
// 6313 / 3490 (6303 / 3475).
#ifndef THP_SPREAD1_HALF_ATOMS
#define THP_SPREAD1_HALF_ATOMS 100000
#endif

// grid_uind_site (pmestuff.f:280-405) of one dipole per site, tiles of 16, 8 or
// 1 sites as spread_dip_warp.  A warp takes spw consecutive sites: 32 (two tiles
// in turn), or 16 where 32 would leave the GPU a single short wave.
template <typename T, typename V>
__global__ void __launch_bounds__(kSpreadThreads) k1_spread(int n, PmeGeom g, const double4* __restrict__ pos,
                                                            const V* __restrict__ x, const CgScalars* __restrict__ cg,
                                                            int check_stop, int spw, T* __restrict__ grid) {
  extern __shared__ __align__(16) unsigned char spread1_smem[];
  if (check_stop && cg->stop) return;
  SpreadWarp1<T>& s = reinterpret_cast<SpreadWarp1<T>*>(spread1_smem)[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  for (int q = lane; q < SpreadWarp1<T>::kPts; q += 32) s.tile[q] = T(0);
  const int i = (blockIdx.x * (kSpreadThreads / 32) + (threadIdx.x >> 5)) * spw + lane;
  const bool live = lane < spw && i < n;
  int gx = 0, gy = 0, gz = 0;
  if (live) {
    double v[3];
    load3(x + (size_t)i * 3, v);
    const double4 p = pos[i];
    T tx[kBs][2], ty[kBs][2], tz[kBs][2];
    gx = bspline_axis<2, T>(p.x, g.recip[0], g.n1, tx);
    gy = bspline_axis<2, T>(p.y, g.recip[1], g.n2, ty);
    gz = bspline_axis<2, T>(p.z, g.recip[2], g.n3, tz);
    T* w = s.w[lane];
#pragma unroll
    for (int k = 0; k < kBs; ++k) {
      w[2 * k] = tx[k][0];
      w[2 * k + 1] = tx[k][1];
      w[10 + 2 * k] = ty[k][0];
      w[11 + 2 * k] = ty[k][1];
      w[20 + 2 * k] = tz[k][0];
      w[21 + 2 * k] = tz[k][1];
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) w[30 + d] = (T)(g.a[d] * v[d]);
  }
  __syncwarp();
  unsigned pending = __ballot_sync(~0u, live);
  int level = 0;
#pragma unroll 1
  while (pending) {
    const int first = __ffs(pending) - 1;
    const unsigned gm = level == 0 ? (0xffffu << (first & 16)) : (level == 1 ? (0xffu << (first & 24)) : (1u << first));
    const unsigned mk = pending & gm;
    if (spread_tile_pass1<T>(g, mk, lane, gx, gy, gz, grid, s)) {
      pending &= ~mk;
      if (!(pending & (0xffffu << (first & 16))))
        level = 0;
      else if (!(pending & (0xffu << (first & 24))))
        level = 1;
    } else {
      ++level;  // a single site always fits
    }
  }
}

// The same with a warp per site (small systems): update first forms
// pp = zr + beta pp; otherwise (the start) the positions go into the records
// too.  rec: the partner records of the real-space rows.
template <typename T>
__global__ void __launch_bounds__(128) k1_spread_small(int n, PmeGeom g, Box box, const double4* __restrict__ pos,
                                                       const float4* __restrict__ posf, double* __restrict__ x,
                                                       const double* __restrict__ zr,
                                                       const CgScalars* __restrict__ cg, int update,
                                                       T* __restrict__ rec, T* __restrict__ grid) {
  __shared__ SiteWeights<T> sw[4];
  if (update && cg->stop) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = blockIdx.x * 4 + warp;
  if (i >= n) return;  // the same for the whole warp
  SiteWeights<T>& s = sw[warp];
  double v = 0.0;
  if (lane < 3) {
    const size_t q = (size_t)i * 3 + lane;
    v = x[q];
    if (update) {
      v = zr[q] + cg->beta[0] * v;
      x[q] = v;
    }
    rec[(size_t)i * 8 + 3 + lane] = (T)v;
  } else if (lane == 3 && !update) {
    T* r = rec + (size_t)i * 8;
    if constexpr (std::is_same<T, float>::value) {
      const float4 p = posf[i];
      r[0] = p.x;
      r[1] = p.y;
      r[2] = p.z;
    } else {
      double4 p = pos[i];
      image3(box, p.x, p.y, p.z);
      r[0] = p.x;
      r[1] = p.y;
      r[2] = p.z;
    }
  }
  if (lane >= 29) stage_axis<T>(g, pos[i], lane - 29, s);
  __syncwarp();
  T f[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) f[d] = (T)(g.a[d] * __shfl_sync(0xffffffffu, v, d));
  if (lane >= kBs * kBs) return;
  const int b = lane % kBs, c = lane / kBs;
  const T u0 = s.w[1][2 * b], u1 = s.w[1][2 * b + 1], v0 = s.w[2][2 * c], v1 = s.w[2][2 * c + 1];
  const T t0 = f[1] * u1 * v0 + f[2] * u0 * v1, t1 = f[0] * u0 * v0;
  const int gx = s.g0[0];
  const size_t row = ((size_t)wrapk(s.g0[2] + c, g.n3) * g.n2 + wrapk(s.g0[1] + b, g.n2)) * g.n1;
  T e[kBs];
#pragma unroll
  for (int a = 0; a < kBs; ++a) e[a] = t0 * s.w[0][2 * a] + t1 * s.w[0][2 * a + 1];
  if constexpr (std::is_same<T, float>::value) {
    // pairs that start on an even point and do not cross the wrap
    bool done = false;
#pragma unroll
    for (int a = 0; a < kBs; ++a) {
      if (done) {
        done = false;
        continue;
      }
      const size_t gi = row + wrapk(gx + a, g.n1);
      if (a + 1 < kBs && gx + a != -1 && (gi & 1) == 0) {
        red_add2(grid + gi, e[a], e[a + 1]);
        done = true;
      } else {
        red_add(grid + gi, e[a]);
      }
    }
  } else {
#pragma unroll
    for (int a = 0; a < kBs; ++a) red_add(grid + row + wrapk(gx + a, g.n1), e[a]);
  }
}

// ---- vectors and rows --------------------------------------------------------------

// mu [n][6] -> the d dipoles [n][3]
__global__ void k1_take(int n, const double* __restrict__ mu6, double* __restrict__ mu3) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < 3 * n) mu3[t] = mu6[(size_t)(t / 3) * 6 + t % 3];
}

// pp = zr + beta pp (newinduce_pme2.f:553-559) and the partner records (large
// systems); update 0 writes the records of x with the positions.
template <typename T, typename V>
__global__ void __launch_bounds__(256) k1_rec(int n, int update, Box box, const double4* __restrict__ pos,
                                              const float4* __restrict__ posf, const V* __restrict__ zr,
                                              V* __restrict__ x, T* __restrict__ rec,
                                              const CgScalars* __restrict__ cg) {
  if (update && cg->stop) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double v[3];
  load3(x + (size_t)i * 3, v);
  T* r = rec + (size_t)i * 8;
  if (update) {
    double z[3];
    load3(zr + (size_t)i * 3, z);
    const double b = cg->beta[0];
#pragma unroll
    for (int q = 0; q < 3; ++q) v[q] = z[q] + b * v[q];
    store3(x + (size_t)i * 3, v);
  } else if constexpr (std::is_same<T, float>::value) {
    const float4 p = posf[i];
    r[0] = p.x;
    r[1] = p.y;
    r[2] = p.z;
  } else {
    double4 p = pos[i];
    image3(box, p.x, p.y, p.z);
    r[0] = p.x;
    r[1] = p.y;
    r[2] = p.z;
  }
  store3(r + 3, v);
}

// One block of pair-stream entries a round in FP64 (64 registers: 250 us at
// 288,000 atoms; two blocks 261, three 274) and four in FP32, both compiled for
// 8 blocks per SM (FP32: 120 us; at the compiler's 66 registers and 7 blocks 129).
#ifndef THP_GROW1_U64
#define THP_GROW1_U64 1
#endif
#ifndef THP_GROW1_U32
#define THP_GROW1_U32 4
#endif

// T_real x without the diagonal (tmatxb_pme, newinduce_pme.f:1392-1668); lane
// j < 3 of an atom writes component j
#ifndef THP_ROW1_MINB
#define THP_ROW1_MINB 8
#endif
template <typename T, bool NOL1, typename HV>
__global__ void __launch_bounds__(kBlock, THP_ROW1_MINB) k1_row(PairRows pr, Box box, const T* __restrict__ rec,
                                                 const CgScalars* __restrict__ cg, int check_stop, float interior,
                                                 HV* __restrict__ hreal) {
  if (check_stop && cg->stop) return;
  const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (4 * g >= pr.n) return;
  const int lane = threadIdx.x & 31;
  const int i = 4 * g + (lane >> 3), j = lane & 7;
  T acc[3];
  if constexpr (std::is_same<T, float>::value)
    group_row<float, THP_GROW1_U32, NOL1>(pr, PartnerRec1<float>{rec},
                                          Image32{(float)box.l[0], (float)box.l[1], (float)box.l[2]}, g, lane, acc,
                                          interior);
  else
    group_row<double, THP_GROW1_U64, NOL1>(pr, PartnerRec1<double>{rec}, Image64In{box}, g, lane, acc,
                                           (double)interior);
  if (j < 3 && i < pr.n) hreal[(size_t)i * 3 + j] = (HV)(j == 0 ? acc[0] : (j == 1 ? acc[1] : acc[2]));
}

// fphi_uind_site's field part (pmestuff.f:746-1045) of one real per point
template <typename T>
__device__ __forceinline__ void gather_dip1(const PmeGeom& g, double4 p, const T* __restrict__ pot, double (&out)[3]) {
  T tx[kBs][2], ty[kBs][2], tz[kBs][2];
  const int gx = bspline_axis<2, T>(p.x, g.recip[0], g.n1, tx);
  const int gy = bspline_axis<2, T>(p.y, g.recip[1], g.n2, ty);
  const int gz = bspline_axis<2, T>(p.z, g.recip[2], g.n3, tz);
  T a100 = 0, a010 = 0, a001 = 0;
#pragma unroll
  for (int c = 0; c < kBs; ++c) {
    const size_t kk = (size_t)wrapk(gz + c, g.n3);
    T a00 = 0, a10 = 0, a01 = 0;
#pragma unroll
    for (int b = 0; b < kBs; ++b) {
      const size_t row = (kk * g.n2 + wrapk(gy + b, g.n2)) * g.n1;
      T t0 = 0, t1 = 0;
#pragma unroll
      for (int a = 0; a < kBs; ++a) {
        const T q = __ldg(pot + row + wrapk(gx + a, g.n1));
        t0 += q * tx[a][0];
        t1 += q * tx[a][1];
      }
      a00 += t0 * ty[b][0];
      a10 += t1 * ty[b][0];
      a01 += t0 * ty[b][1];
    }
    a100 += a10 * tz[c][0];
    a010 += a01 * tz[c][0];
    a001 += a00 * tz[c][1];
  }
  out[0] = g.a[0] * (double)a100;
  out[1] = g.a[1] * (double)a010;
  out[2] = g.a[2] * (double)a001;
}

// h = hreal + x/alpha + dipfield(x) - term x and the reductions (cg_combine_block)
template <typename T, typename XV, typename V>
__global__ void __launch_bounds__(kBlock) k1_combine(int n, PmeGeom g, const double4* __restrict__ pos,
                                                     const T* __restrict__ pot, const XV* __restrict__ x,
                                                     const double* __restrict__ pol, const double* __restrict__ ef,
                                                     double term, int init, V* __restrict__ h, V* __restrict__ res,
                                                     V* __restrict__ zr, V* __restrict__ pp, CgScalars* cg,
                                                     double* __restrict__ partials) {
  if (cg->stop) return;
  const int i = blockIdx.x * kBlock + threadIdx.x;
  double red[1] = {0.0};
  if (i < n) {
    double dip[3], acc[3], xi[3], hv[3];
    gather_dip1<T>(g, pos[i], pot, dip);
    load3(h + (size_t)i * 3, acc);
    load3(x + (size_t)i * 3, xi);
    const double p = pol[i];
    const double ip = (p == 0.0) ? 1.0 / kTinyPol : 1.0 / p;
#pragma unroll
    for (int q = 0; q < 3; ++q) hv[q] = ((acc[q] + xi[q] * ip) + dip[q]) - term * xi[q];
    store3(h + (size_t)i * 3, hv);
    if (init) {
      double r3[3], z3[3];
      const double dg = diag_of(p);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        r3[q] = ef[(size_t)i * 6 + q] - hv[q];
        z3[q] = dg * r3[q];
      }
      store3(res + (size_t)i * 3, r3);
      store3(zr + (size_t)i * 3, z3);
      store3(pp + (size_t)i * 3, z3);
      red[0] = r3[0] * z3[0] + r3[1] * z3[1] + r3[2] * z3[2];
    } else {
      red[0] = xi[0] * hv[0] + xi[1] * hv[1] + xi[2] * hv[2];
    }
  }
  double tot[1];
  if (grid_reduce<1>(red, partials, &cg->counter[0], tot) && threadIdx.x == 0) {
    const double both[2] = {tot[0], tot[0]};
    cg_after_matvec(both, init, cg);
  }
}

// the same for small systems: 16 atoms per block, eight lanes each
// (cg_combine8_block); lane j < 3 finishes component j
template <typename T>
__global__ void __launch_bounds__(kBlock) k1_combine8(int n, PmeGeom g, const double4* __restrict__ pos,
                                                      const T* __restrict__ pot, const double* __restrict__ x,
                                                      const double* __restrict__ pol, const double* __restrict__ ef,
                                                      double term, int init, double* __restrict__ h,
                                                      double* __restrict__ res, double* __restrict__ zr,
                                                      double* __restrict__ pp, CgScalars* cg,
                                                      double* __restrict__ partials) {
  __shared__ SiteWeights<T> sw[16];
  if (cg->stop) return;
  const int a8 = threadIdx.x >> 3, j = threadIdx.x & 7;
  const int i0 = blockIdx.x * 16 + a8;
  const bool live = i0 < n;
  const int i = live ? i0 : n - 1;
  SiteWeights<T>& s = sw[a8];
  if (j < 3) stage_axis<T>(g, pos[i], j, s);
  __syncwarp();
  const int gx = s.g0[0];
  auto line = [&](int q) {
    const int b = q % kBs, c = q / kBs;
    return ((size_t)wrapk(s.g0[2] + c, g.n3) * g.n2 + wrapk(s.g0[1] + b, g.n2)) * g.n1;
  };
  // lines j, j + 8 and j + 16 whole, one point of the last line each, all loads
  // before the sums: the chain of loads is what bounds this kernel (a solve of
  // 648 atoms 519 -> 494 us against a loop over the lane's lines)
  T e[3][kBs];
#pragma unroll
  for (int l = 0; l < 3; ++l) {
    const size_t row = line(j + 8 * l);
#pragma unroll
    for (int a = 0; a < kBs; ++a) e[l][a] = __ldg(pot + row + wrapk(gx + a, g.n1));
  }
  const T last = j < kBs ? __ldg(pot + line(kBs * kBs - 1) + wrapk(gx + j, g.n1)) : T(0);
  double xi = 0.0, hi = 0.0, p = 0.0;
  if (live && j < 3) {
    xi = x[(size_t)i * 3 + j];
    hi = h[(size_t)i * 3 + j];
    p = pol[i];
  }
  T acc[3] = {0, 0, 0};
  auto add = [&](int q, T t0, T t1) {
    const int b = q % kBs, c = q / kBs;
    const T u0 = s.w[1][2 * b], u1 = s.w[1][2 * b + 1], v0 = s.w[2][2 * c], v1 = s.w[2][2 * c + 1];
    acc[0] += t1 * u0 * v0;
    acc[1] += t0 * u1 * v0;
    acc[2] += t0 * u0 * v1;
  };
#pragma unroll
  for (int l = 0; l < 3; ++l) {
    T t0 = 0, t1 = 0;
#pragma unroll
    for (int a = 0; a < kBs; ++a) {
      t0 += e[l][a] * s.w[0][2 * a];
      t1 += e[l][a] * s.w[0][2 * a + 1];
    }
    add(j + 8 * l, t0, t1);
  }
  if (j < kBs) add(kBs * kBs - 1, last * s.w[0][2 * j], last * s.w[0][2 * j + 1]);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < 3; ++q) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
  double red[1] = {0.0};
  if (live && j < 3) {
    const size_t q = (size_t)i * 3 + j;
    const double dip = (j == 0 ? g.a[0] : (j == 1 ? g.a[1] : g.a[2])) *
                       (double)(j == 0 ? acc[0] : (j == 1 ? acc[1] : acc[2]));
    const double ip = (p == 0.0) ? 1.0 / kTinyPol : 1.0 / p;
    const double hv = ((hi + xi * ip) + dip) - term * xi;
    h[q] = hv;
    if (init) {
      const double r = ef[(size_t)i * 6 + j] - hv, z = diag_of(p) * r;
      res[q] = r;
      zr[q] = z;
      pp[q] = z;
      red[0] = r * z;
    } else {
      red[0] = xi * hv;
    }
  }
  double tot[1];
  if (grid_reduce<1>(red, partials, &cg->counter[0], tot) && threadIdx.x == 0) {
    const double both[2] = {tot[0], tot[0]};
    cg_after_matvec(both, init, cg);
  }
}

// mu, residual and preconditioned residual of one step (k_cg_update)
template <typename V>
__global__ void __launch_bounds__(kBlock) k1_update(int n, const double* __restrict__ pol, const V* __restrict__ h,
                                                    const V* __restrict__ pp, double* __restrict__ mu,
                                                    V* __restrict__ res, V* __restrict__ zr, CgScalars* cg,
                                                    double* __restrict__ partials, double poleps, int politer,
                                                    LoopCond loop) {
  if (loop_entry(loop, cg)) return;
  const int i = blockIdx.x * kBlock + threadIdx.x;
  double red[1] = {0.0};
  if (i < n) {
    const double a = cg->alpha[0];
    double m3[3], r3[3], p3[3], h3[3], z3[3];
    load3(mu + (size_t)i * 3, m3);
    load3(res + (size_t)i * 3, r3);
    load3(pp + (size_t)i * 3, p3);
    load3(h + (size_t)i * 3, h3);
    const double dg = diag_of(pol[i]);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      m3[q] += a * p3[q];
      r3[q] -= a * h3[q];
      z3[q] = dg * r3[q];
      red[0] += r3[q] * z3[q];
    }
    store3(mu + (size_t)i * 3, m3);
    store3(res + (size_t)i * 3, r3);
    store3(zr + (size_t)i * 3, z3);
  }
  double tot[1];
  if (grid_reduce<1>(red, partials, &cg->counter[1], tot) && threadIdx.x == 0) {
    const double both[2] = {tot[0], tot[0]};
    cg_after_update(both, n, cg, poleps, politer);
    if (loop.max_loops && cg->stop) cudaGraphSetConditional(loop.handle, 0);
  }
}

// Epol and ene (k_epol), and both sets of dipoles [n][6]
template <typename V>
__global__ void __launch_bounds__(kBlock) k1_epol(int n, const double* __restrict__ mu3, const double* __restrict__ ef,
                                                  const V* __restrict__ res, double* __restrict__ mu6, CgScalars* cg,
                                                  double* __restrict__ partials) {
  const int i = blockIdx.x * kBlock + threadIdx.x;
  double red[3] = {0.0, 0.0, 0.0};
  if (i < n) {
    double m[3], e[6], r[3];
    load3(mu3 + (size_t)i * 3, m);
    load6(ef + (size_t)i * 6, e);
    load3(res + (size_t)i * 3, r);
    const double both[6] = {m[0], m[1], m[2], m[0], m[1], m[2]};
    store6(mu6 + (size_t)i * 6, both);
    red[0] = m[0] * e[3] + m[1] * e[4] + m[2] * e[5];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      red[1] -= 0.5 * (m[q] * (r[q] + e[q]));
      red[2] -= 0.5 * (m[q] * (r[q] + e[3 + q]));
    }
  }
  double tot[3];
  if (grid_reduce<3>(red, partials, &cg->counter[2], tot) && threadIdx.x == 0) {
    cg->epol = -0.5 * kElectric * tot[0];
    cg->ene[0] = tot[1];
    cg->ene[1] = tot[2];
  }
}

// The vectors of the form: FP32 storage for large mixed systems, else FP64,
// [n][3] in the front of the two-field buffers.
template <typename V>
struct Vecs {
  V *h, *res, *zr, *pp;
};
Vecs<float> vecs(Ctx& c, float) { return {c.d_hf, c.d_resf, c.d_zrf, c.d_ppf}; }
Vecs<double> vecs(Ctx& c, double) { return {c.d_h, c.d_res, c.d_zr, c.d_pp}; }

double self_term(const Ctx& c) {
  const double a = c.cfg.aewald;
  return (4.0 / 3.0) * a * a * a / kSqrtPi;
}

template <typename T>
T* records(Ctx& c);
template <>
float* records<float>(Ctx& c) { return c.d_rec; }
template <>
double* records<double>(Ctx& c) { return c.d_rec64; }

template <typename T, typename HV>
int launch_row(Ctx& c, int check_stop, HV* h) {
  const PairRows pr = pair_rows(c);
  const float interior = row_interior(c);
  const int rb = c.n < kRowSmallAtoms ? 32 : kBlock;
  const int nb = group_blocks(c.n, rb);
  prof_mark(c, c.stream2);
  if (c.n >= kStreamAtoms)
    k1_row<T, true, HV><<<nb, rb, 0, c.stream2>>>(pr, c.box, records<T>(c), c.d_cg, check_stop, interior, h);
  else
    k1_row<T, false, HV><<<nb, rb, 0, c.stream2>>>(pr, c.box, records<T>(c), c.d_cg, check_stop, interior, h);
  prof_mark(c, c.stream2);
  return cuda_status(cudaGetLastError(), &c, "real row");
}

// h = T x (and at the start the residual); V: the stored vectors, XV: x
template <typename T, typename XV, typename V>
int matvec_large(Ctx& c, XV* x, int init) {
  const Vecs<V> v = vecs(c, V{});
  k1_rec<T, XV><<<(c.n + 255) / 256, 256, 0, c.stream>>>(c.n, !init, c.box, c.d_pos, c.d_posf,
                                                        init ? nullptr : reinterpret_cast<XV*>(v.zr), x, records<T>(c),
                                                        c.d_cg);
  int st = cuda_status(cudaGetLastError(), &c, "pp update");
  if (st) return st;
  cudaEventRecord(c.ev_fork, c.stream);
  cudaStreamWaitEvent(c.stream2, c.ev_fork, 0);
  st = launch_row<T, V>(c, !init, v.h);
  cudaEventRecord(c.ev_join, c.stream2);
  constexpr size_t smem = sizeof(SpreadWarp1<T>) * (kSpreadThreads / 32);
  static std::atomic<unsigned long long> limit_set{0};
  smem_limit_once(k1_spread<T, XV>, smem, limit_set);
  const int spw = c.n < THP_SPREAD1_HALF_ATOMS ? 16 : 32, spb = spw * (kSpreadThreads / 32);
  k1_spread<T, XV><<<(c.n + spb - 1) / spb, kSpreadThreads, smem, c.stream>>>(c.n, pme_geom(c), c.d_pos, x, c.d_cg,
                                                                             !init, spw, (T*)c.d_grid);
  int st2 = spread_status(c, cuda_status(cudaGetLastError(), &c, "spread dip"));
  if (!st2) st2 = launch_convolve(c, !init, true);
  cudaStreamWaitEvent(c.stream, c.ev_join, 0);
  if (st || st2) return st ? st : st2;
  k1_combine<T, XV, V><<<(c.n + kBlock - 1) / kBlock, kBlock, 0, c.stream>>>(
      c.n, pme_geom(c), c.d_pos, (const T*)c.d_pot, x, c.d_pol, c.d_ef, self_term(c), init, v.h, v.res, v.zr, v.pp,
      c.d_cg, c.d_partials);
  return cuda_status(cudaGetLastError(), &c, "cg combine");
}

template <typename T>
int matvec_small(Ctx& c, double* x, int init) {
  const Vecs<double> v = vecs(c, 0.0);
  k1_spread_small<T><<<(c.n + 3) / 4, 128, 0, c.stream>>>(c.n, pme_geom(c), c.box, c.d_pos, c.d_posf, x, v.zr, c.d_cg,
                                                         !init, records<T>(c), (T*)c.d_grid);
  int st = spread_status(c, cuda_status(cudaGetLastError(), &c, "spread dip"));
  if (st) return st;
  cudaEventRecord(c.ev_fork, c.stream);
  cudaStreamWaitEvent(c.stream2, c.ev_fork, 0);
  st = launch_row<T, double>(c, !init, v.h);
  cudaEventRecord(c.ev_join, c.stream2);
  const int st2 = launch_convolve(c, !init, true);
  cudaStreamWaitEvent(c.stream, c.ev_join, 0);
  if (st || st2) return st ? st : st2;
  k1_combine8<T><<<(c.n + 15) / 16, kBlock, 0, c.stream>>>(c.n, pme_geom(c), c.d_pos, (const T*)c.d_pot, x, c.d_pol,
                                                          c.d_ef, self_term(c), init, v.h, v.res, v.zr, v.pp, c.d_cg,
                                                          c.d_partials);
  return cuda_status(cudaGetLastError(), &c, "cg combine");
}

bool float_vectors(const Ctx& c) { return c.mixed && c.n >= kLargeAtoms; }

}  // namespace

bool single_field(const Ctx& c) { return c.dp_equal && c.conv; }

int single_begin(Ctx& c) {
  double* mu = c.d_dip;  // the solve's dipoles [n][3]
  k1_take<<<(3 * c.n + 255) / 256, 256, 0, c.stream>>>(c.n, c.d_mu, mu);
  int st = cuda_status(cudaGetLastError(), &c, "cg start");
  if (st) return st;
  if (c.n < kLargeAtoms) return c.mixed ? matvec_small<float>(c, mu, 1) : matvec_small<double>(c, mu, 1);
  return c.mixed ? matvec_large<float, double, float>(c, mu, 1) : matvec_large<double, double, double>(c, mu, 1);
}

int single_iteration(Ctx& c, const LoopCond& loop) {
  const int nb = (c.n + kBlock - 1) / kBlock;
  int st;
  if (float_vectors(c)) {
    if ((st = matvec_large<float, float, float>(c, c.d_ppf, 0))) return st;
    k1_update<float><<<nb, kBlock, 0, c.stream>>>(c.n, c.d_pol, c.d_hf, c.d_ppf, c.d_dip, c.d_resf, c.d_zrf, c.d_cg,
                                                  c.d_partials, c.cfg.poleps, c.cfg.politer, loop);
    return cuda_status(cudaGetLastError(), &c, "cg update");
  }
  if (c.n >= kLargeAtoms)
    st = matvec_large<double, double, double>(c, c.d_pp, 0);
  else
    st = c.mixed ? matvec_small<float>(c, c.d_pp, 0) : matvec_small<double>(c, c.d_pp, 0);
  if (st) return st;
  k1_update<double><<<nb, kBlock, 0, c.stream>>>(c.n, c.d_pol, c.d_h, c.d_pp, c.d_dip, c.d_res, c.d_zr, c.d_cg,
                                                 c.d_partials, c.cfg.poleps, c.cfg.politer, loop);
  return cuda_status(cudaGetLastError(), &c, "cg update");
}

int single_epol(Ctx& c) {
  const int nb = (c.n + kBlock - 1) / kBlock;
  if (float_vectors(c))
    k1_epol<float><<<nb, kBlock, 0, c.stream>>>(c.n, c.d_dip, c.d_ef, c.d_resf, c.d_mu, c.d_cg, c.d_partials);
  else
    k1_epol<double><<<nb, kBlock, 0, c.stream>>>(c.n, c.d_dip, c.d_ef, c.d_res, c.d_mu, c.d_cg, c.d_partials);
  return cuda_status(cudaGetLastError(), &c, "epol");
}

}  // namespace thp
