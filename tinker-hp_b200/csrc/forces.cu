// forces.cu -- polarization energy gradient on the device (epolar1c).
//
// Restates epolar1c (epolar1.f:57-372) for a converged solve:
//   * eprecip1 (epolar1.f:397-1213): the dipole grid of uind (Re) / uinp (Im)
//     gathered to all 20 potential derivatives (fphi_uind_site), combined with
//     the permanent-multipole potential fphirec (its grid convolved again);
//   * epreal1c (epolar1.f:1215-2540, Thole branch): per pair the gradient of
//     the d- and p-scaled permanent field on uinp / uind and of the mutual
//     tensor (uscale) on uind x uinp, plus the induced field and its gradient
//     at every site for the torques;
//   * self torque (epolar1.f:190-206), and torque (torque.f:6-390) for the
//     Z-then-X and Bisector frames.
// Eight lanes own atom i over its interacting pairs (each pair is evaluated
// from both ends, the i-side terms only).  The three torques of a site are
// summed before one torque distribution.  Gradients are accumulated in 64-bit
// fixed point with 2^-34 kcal/mol/A resolution (in the FP64 form with a second
// word for the remainders, FixAcc), so the order in which threads add their
// contributions does not change the sums.
#include <type_traits>

#include "damp_dev.cuh"
#include "grad_dev.cuh"
#include "kernels.h"
#include "pme_dev.cuh"
#include "realspace_dev.cuh"

namespace thp {

namespace {

constexpr int kBlock = 128;
// fphi_uind_site (pmestuff.f:746-1045) in full and the force / torque of
// eprecip1 (epolar1.f:636-720).  fphirec: [n][20] permanent potential
// (unscaled), written by the field pass.
// VIR: each block also writes the sum of its sites' induced-dipole virial
// terms (epolar1.f:846-908) to vpart[block][6].
template <typename T, bool VIR>
__global__ void __launch_bounds__(kBlock) k_force_recip(int n, PmeGeom g, const double4* __restrict__ pos,
                                                        const typename Cplx<T>::type* __restrict__ grid,
                                                        const double* __restrict__ fphirec,
                                                        const double* __restrict__ mu, const double* __restrict__ rp,
                                                        double* __restrict__ trq_out,
                                                        FixAcc dep,
                                                        double* __restrict__ vpart) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double vs[6] = {0, 0, 0, 0, 0, 0};
  if (i < n) {
  const double4 p = pos[i];
  T tx[kBs][4], ty[kBs][4], tz[kBs][4];
  const int gx = bspline_axis<4, T>(p.x, g.recip[0], g.n1, tx);
  const int gy = bspline_axis<4, T>(p.y, g.recip[1], g.n2, ty);
  const int gz = bspline_axis<4, T>(p.z, g.recip[2], g.n3, tz);
  // T1/T2: 100,010,001,200,020,002,110,101,011 of the d / p grids; S: 20 of their sum
  T T1[9] = {0}, T2[9] = {0}, S[20] = {0};
#pragma unroll
  for (int c = 0; c < kBs; ++c) {
    const size_t kk = (size_t)wrapk(gz + c, g.n3);
    const T v0 = tz[c][0], v1 = tz[c][1], v2 = tz[c][2], v3 = tz[c][3];
    T a1[6] = {0}, a2[6] = {0}, s[10] = {0};
#pragma unroll
    for (int b = 0; b < kBs; ++b) {
      const size_t jj = (size_t)wrapk(gy + b, g.n2);
      const T u0 = ty[b][0], u1 = ty[b][1], u2 = ty[b][2], u3 = ty[b][3];
      T ta[3] = {0, 0, 0}, tb[3] = {0, 0, 0}, t3 = 0;
      const size_t row = (kk * g.n2 + jj) * g.n1;
#pragma unroll
      for (int a = 0; a < kBs; ++a) {
        const auto q = grid[row + wrapk(gx + a, g.n1)];
        ta[0] += q.x * tx[a][0];
        ta[1] += q.x * tx[a][1];
        ta[2] += q.x * tx[a][2];
        tb[0] += q.y * tx[a][0];
        tb[1] += q.y * tx[a][1];
        tb[2] += q.y * tx[a][2];
        t3 += (q.x + q.y) * tx[a][3];
      }
      a1[0] += ta[0] * u0; a1[1] += ta[1] * u0; a1[2] += ta[0] * u1;
      a1[3] += ta[2] * u0; a1[4] += ta[1] * u1; a1[5] += ta[0] * u2;
      a2[0] += tb[0] * u0; a2[1] += tb[1] * u0; a2[2] += tb[0] * u1;
      a2[3] += tb[2] * u0; a2[4] += tb[1] * u1; a2[5] += tb[0] * u2;
      const T t0 = ta[0] + tb[0], t1 = ta[1] + tb[1], t2 = ta[2] + tb[2];
      s[0] += t0 * u0; s[1] += t1 * u0; s[2] += t0 * u1; s[3] += t2 * u0; s[4] += t1 * u1;
      s[5] += t0 * u2; s[6] += t3 * u0; s[7] += t2 * u1; s[8] += t1 * u2; s[9] += t0 * u3;
    }
    T1[0] += a1[1] * v0; T1[1] += a1[2] * v0; T1[2] += a1[0] * v1; T1[3] += a1[3] * v0; T1[4] += a1[5] * v0;
    T1[5] += a1[0] * v2; T1[6] += a1[4] * v0; T1[7] += a1[1] * v1; T1[8] += a1[2] * v1;
    T2[0] += a2[1] * v0; T2[1] += a2[2] * v0; T2[2] += a2[0] * v1; T2[3] += a2[3] * v0; T2[4] += a2[5] * v0;
    T2[5] += a2[0] * v2; T2[6] += a2[4] * v0; T2[7] += a2[1] * v1; T2[8] += a2[2] * v1;
    S[0] += s[0] * v0; S[1] += s[1] * v0; S[2] += s[2] * v0; S[3] += s[0] * v1; S[4] += s[3] * v0;
    S[5] += s[5] * v0; S[6] += s[0] * v2; S[7] += s[4] * v0; S[8] += s[1] * v1; S[9] += s[2] * v1;
    S[10] += s[6] * v0; S[11] += s[9] * v0; S[12] += s[0] * v3; S[13] += s[7] * v0; S[14] += s[3] * v1;
    S[15] += s[8] * v0; S[16] += s[5] * v1; S[17] += s[1] * v2; S[18] += s[2] * v2; S[19] += s[4] * v1;
  }
  // 1-based views as in the reference (scaled by electric)
  const double f = kElectric;
  double FD[11], FP[11], FS[21], FR[21];
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    FD[q + 2] = f * (double)T1[q];
    FP[q + 2] = f * (double)T2[q];
  }
#pragma unroll
  for (int q = 0; q < 20; ++q) {
    FS[q + 1] = f * (double)S[q];
    FR[q + 1] = f * fphirec[(size_t)i * 20 + q];
  }
  const double* m = mu + (size_t)i * 6;
  const double fd[3] = {g.a[0] * m[0], g.a[1] * m[1], g.a[2] * m[2]};
  const double fp[3] = {g.a[0] * m[3], g.a[1] * m[4], g.a[2] * m[5]};
  const int d1[10] = {2, 5, 8, 9, 11, 16, 18, 14, 15, 20};
  const int d2[10] = {3, 8, 6, 10, 14, 12, 19, 16, 20, 17};
  const int d3[10] = {4, 9, 10, 7, 15, 17, 13, 20, 18, 19};
  double f1 = 0.0, f2 = 0.0, f3 = 0.0;
#pragma unroll
  for (int k = 1; k <= 3; ++k) {
    const double sdp = fd[k - 1] + fp[k - 1];
    f1 += sdp * FR[d1[k]] + fd[k - 1] * FP[d1[k]] + fp[k - 1] * FD[d1[k]];
    f2 += sdp * FR[d2[k]] + fd[k - 1] * FP[d2[k]] + fp[k - 1] * FD[d2[k]];
    f3 += sdp * FR[d3[k]] + fd[k - 1] * FP[d3[k]] + fp[k - 1] * FD[d3[k]];
  }
  // fmp of the permanent moments (cart_to_frac, orthogonal box)
  const double* r = rp + (size_t)i * 10;
  const double cm[10] = {r[0], r[1], r[2], r[3], r[4], r[7], r[9], 2.0 * r[5], 2.0 * r[6], 2.0 * r[8]};
  const double fm[10] = {cm[0], g.a[0] * cm[1], g.a[1] * cm[2], g.a[2] * cm[3], g.a[0] * g.a[0] * cm[4],
                         g.a[1] * g.a[1] * cm[5], g.a[2] * g.a[2] * cm[6], g.a[0] * g.a[1] * cm[7],
                         g.a[0] * g.a[2] * cm[8], g.a[1] * g.a[2] * cm[9]};
#pragma unroll
  for (int k = 0; k < 10; ++k) {
    f1 += fm[k] * FS[d1[k]];
    f2 += fm[k] * FS[d2[k]];
    f3 += fm[k] * FS[d3[k]];
  }
  f1 = 0.5 * (double)g.n1 * f1;
  f2 = 0.5 * (double)g.n2 * f2;
  f3 = 0.5 * (double)g.n3 * f3;
  dep.add(3 * i + 0, g.recip[0] * f1);
  dep.add(3 * i + 1, g.recip[1] * f2);
  dep.add(3 * i + 2, g.recip[2] * f3);
  // cphidprec = fphi_to_cphi(fphidprec/2), torque on the permanent moments
  double cp[10];
  cp[0] = 0.5 * FS[1];
  cp[1] = g.a[0] * 0.5 * FS[2];
  cp[2] = g.a[1] * 0.5 * FS[3];
  cp[3] = g.a[2] * 0.5 * FS[4];
  cp[4] = g.a[0] * g.a[0] * 0.5 * FS[5];
  cp[5] = g.a[1] * g.a[1] * 0.5 * FS[6];
  cp[6] = g.a[2] * g.a[2] * 0.5 * FS[7];
  cp[7] = g.a[0] * g.a[1] * 0.5 * FS[8];
  cp[8] = g.a[0] * g.a[2] * 0.5 * FS[9];
  cp[9] = g.a[1] * g.a[2] * 0.5 * FS[10];
  double* t = trq_out + (size_t)i * 3;
  t[0] = cm[3] * cp[2] - cm[2] * cp[3] + 2.0 * (cm[6] - cm[5]) * cp[9] + cm[8] * cp[7] + cm[9] * cp[5] -
         cm[7] * cp[8] - cm[9] * cp[6];
  t[1] = cm[1] * cp[3] - cm[3] * cp[1] + 2.0 * (cm[4] - cm[6]) * cp[8] + cm[7] * cp[9] + cm[8] * cp[6] -
         cm[8] * cp[4] - cm[9] * cp[7];
  t[2] = cm[2] * cp[1] - cm[1] * cp[2] + 2.0 * (cm[5] - cm[4]) * cp[7] + cm[7] * cp[4] + cm[9] * cp[8] -
         cm[7] * cp[5] - cm[8] * cp[9];
  if (VIR) {
    // induced dipole contribution to the internal virial (epolar1.f:846-908):
    // cphim, cphid, cphip = Cartesian gradients of the permanent, d and p
    // potentials; 1-based cphidprec(1:10) = cp, cmp(1:10) = cm
    const double cmx[4] = {0, g.a[0] * FR[2], g.a[1] * FR[3], g.a[2] * FR[4]};
    const double cdx[4] = {0, g.a[0] * FD[2], g.a[1] * FD[3], g.a[2] * FD[4]};
    const double cpx[4] = {0, g.a[0] * FP[2], g.a[1] * FP[3], g.a[2] * FP[4]};
    const double ui[3] = {m[0], m[1], m[2]}, up[3] = {m[3], m[4], m[5]};
    vs[0] = -cp[1] * cm[1] - 0.5 * (cmx[1] * (ui[0] + up[0]) + cdx[1] * up[0] + cpx[1] * ui[0]);
    vs[1] = -0.5 * (cp[1] * cm[2] + cp[2] * cm[1]) -
            0.25 * (cmx[1] * (ui[1] + up[1]) + cmx[2] * (ui[0] + up[0]) + cdx[1] * up[1] + cpx[1] * ui[1] +
                    cdx[2] * up[0] + cpx[2] * ui[0]);
    vs[2] = -0.5 * (cp[1] * cm[3] + cp[3] * cm[1]) -
            0.25 * (cmx[1] * (ui[2] + up[2]) + cmx[3] * (ui[0] + up[0]) + cdx[1] * up[2] + cpx[1] * ui[2] +
                    cdx[3] * up[0] + cpx[3] * ui[0]);
    vs[3] = -cp[2] * cm[2] - 0.5 * (cmx[2] * (ui[1] + up[1]) + cdx[2] * up[1] + cpx[2] * ui[1]);
    vs[4] = -0.5 * (cp[2] * cm[3] + cp[3] * cm[2]) -
            0.25 * (cmx[2] * (ui[2] + up[2]) + cmx[3] * (ui[1] + up[1]) + cdx[2] * up[2] + cpx[2] * ui[2] +
                    cdx[3] * up[1] + cpx[3] * ui[1]);
    vs[5] = -cp[3] * cm[3] - 0.5 * (cmx[3] * (ui[2] + up[2]) + cdx[3] * up[2] + cpx[3] * ui[2]);
    vs[0] += -2.0 * cm[4] * cp[4] - cm[7] * cp[7] - cm[8] * cp[8];
    vs[1] += -(cm[4] + cm[5]) * cp[7] - 0.5 * (cm[7] * (cp[5] + cp[4]) + cm[8] * cp[9] + cm[9] * cp[8]);
    vs[2] += -(cm[4] + cm[6]) * cp[8] - 0.5 * (cm[8] * (cp[4] + cp[6]) + cm[7] * cp[9] + cm[9] * cp[7]);
    vs[3] += -2.0 * cm[5] * cp[5] - cm[7] * cp[7] - cm[9] * cp[9];
    vs[4] += -(cm[5] + cm[6]) * cp[9] - 0.5 * (cm[9] * (cp[5] + cp[6]) + cm[7] * cp[8] + cm[8] * cp[7]);
    vs[5] += -2.0 * cm[6] * cp[6] - cm[8] * cp[8] - cm[9] * cp[9];
  }
  }  // i < n
  if (VIR) {
    block_reduce<6>(vs);
    if (threadIdx.x == 0)
#pragma unroll
      for (int q = 0; q < 6; ++q) vpart[(size_t)blockIdx.x * 6 + q] = vs[q];
  }
}

// fphi_mpole_site (pmestuff.f:453-600): the 20 fractional potential
// derivatives of the permanent-multipole grid, unscaled.
template <typename T>
__global__ void __launch_bounds__(kBlock) k_fphi_mpole20(int n, PmeGeom g, const double4* __restrict__ pos,
                                                         const typename Cplx<T>::type* __restrict__ grid,
                                                         double* __restrict__ fphi) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double4 p = pos[i];
  T tx[kBs][4], ty[kBs][4], tz[kBs][4];
  const int gx = bspline_axis<4, T>(p.x, g.recip[0], g.n1, tx);
  const int gy = bspline_axis<4, T>(p.y, g.recip[1], g.n2, ty);
  const int gz = bspline_axis<4, T>(p.z, g.recip[2], g.n3, tz);
  T S[20] = {0};
#pragma unroll
  for (int c = 0; c < kBs; ++c) {
    const size_t kk = (size_t)wrapk(gz + c, g.n3);
    const T v0 = tz[c][0], v1 = tz[c][1], v2 = tz[c][2], v3 = tz[c][3];
    T s[10] = {0};  // 00,10,01,20,11,02,30,21,12,03
#pragma unroll
    for (int b = 0; b < kBs; ++b) {
      const size_t jj = (size_t)wrapk(gy + b, g.n2);
      const T u0 = ty[b][0], u1 = ty[b][1], u2 = ty[b][2], u3 = ty[b][3];
      T t0 = 0, t1 = 0, t2 = 0, t3 = 0;
      const size_t row = (kk * g.n2 + jj) * g.n1;
#pragma unroll
      for (int a = 0; a < kBs; ++a) {
        const T q = grid[row + wrapk(gx + a, g.n1)].x;
        t0 += q * tx[a][0];
        t1 += q * tx[a][1];
        t2 += q * tx[a][2];
        t3 += q * tx[a][3];
      }
      s[0] += t0 * u0; s[1] += t1 * u0; s[2] += t0 * u1; s[3] += t2 * u0; s[4] += t1 * u1;
      s[5] += t0 * u2; s[6] += t3 * u0; s[7] += t2 * u1; s[8] += t1 * u2; s[9] += t0 * u3;
    }
    S[0] += s[0] * v0; S[1] += s[1] * v0; S[2] += s[2] * v0; S[3] += s[0] * v1; S[4] += s[3] * v0;
    S[5] += s[5] * v0; S[6] += s[0] * v2; S[7] += s[4] * v0; S[8] += s[1] * v1; S[9] += s[2] * v1;
    S[10] += s[6] * v0; S[11] += s[9] * v0; S[12] += s[0] * v3; S[13] += s[7] * v0; S[14] += s[3] * v1;
    S[15] += s[8] * v0; S[16] += s[5] * v1; S[17] += s[1] * v2; S[18] += s[2] * v2; S[19] += s[4] * v1;
  }
  double* f = fphi + (size_t)i * 20;
#pragma unroll
  for (int q = 0; q < 20; ++q) f[q] = (double)S[q];
}

// sorted dipoles [n][6] FP64 -> [n][8] FP32 (d xyz, p xyz, 2 pad): one
// 256-bit load per partner in the mixed pair pass
__global__ void k_mu_f32(int n, const double* __restrict__ mu, float* __restrict__ muf) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4* o = reinterpret_cast<float4*>(muf + (size_t)i * 8);
  const double* m = mu + (size_t)i * 6;
  o[0] = make_float4((float)m[0], (float)m[1], (float)m[2], (float)m[3]);
  o[1] = make_float4((float)m[4], (float)m[5], 0.f, 0.f);
}

struct EwC {
  double a, f1, f2, f3, f4;  // 2 a^2 powers / (sqrt(pi) a) of dampewald order 9
};

// The radial functions of one pair (each with electric/2 folded in):
// Ewald-damped e_l and bare rr_l of l = 3, 5, 7, 9, and the Thole factors
// l3, l5, l7 with their derivatives q_l = (dl_l/dr) / r.
template <typename T>
struct PairRadial {
  T e3, e5, e7, e9, rr3, rr5, rr7, rr9;
  T l3, l5, l7, q3, q5, q7;
};

// Interaction of the permanent moments of sites i and k with the induced
// dipoles u at i and v at k under one scale factor s (epolar1.f:1700-2170):
//   W = F3 (ck u.r - ci v.r + u.dk + v.di)
//     + F5 (2 v.Qi r - 2 u.Qk r - u.r dk.r - v.r di.r) + F7 (u.r qk - v.r qi)
// with r = x_k - x_i, F_l = e_l - (1 - s l_l) rr_l, qk = r.Qk r.  Adds dW/dr to
// frc (the F's own derivatives are -D_l r with D_l = e_{l+2} -
// (1 - s l_l) rr_{l+2} - s q_l rr_l), and the field and field gradient of v at i
// to uf and duf (:2230-2260).  The reference expands the second-derivative
// tensors of each moment; gathering the terms by F_l first gives the same
// sums in about a quarter of the operations.
template <typename T>
__device__ __forceinline__ void perm_terms(const PairRadial<T>& p, T s, const T (&r)[3], const T (&u)[3],
                                           const T (&v)[3], T ur, T vr, T ci, const T (&di)[3], const T (&Qi)[6],
                                           T ck, const T (&dk)[3], const T (&Qk)[6], const T (&qi)[3],
                                           const T (&qk)[3], T dir, T dkr, T qir, T qkr, T (&frc)[3], T (&uf)[3],
                                           T (&duf)[6]) {
  const T n3 = T(1) - s * p.l3, n5 = T(1) - s * p.l5, n7 = T(1) - s * p.l7;
  const T F3 = p.e3 - n3 * p.rr3, F5 = p.e5 - n5 * p.rr5, F7 = p.e7 - n7 * p.rr7;
  const T D3 = p.e5 - n3 * p.rr5 - s * p.q3 * p.rr3;
  const T D5 = p.e7 - n5 * p.rr7 - s * p.q5 * p.rr5;
  const T D7 = p.e9 - n7 * p.rr9 - s * p.q7 * p.rr7;
  const T A3 = ck * ur - ci * vr + (u[0] * dk[0] + u[1] * dk[1] + u[2] * dk[2]) +
               (v[0] * di[0] + v[1] * di[1] + v[2] * di[2]);
  const T A5 = T(2) * ((v[0] * qi[0] + v[1] * qi[1] + v[2] * qi[2]) - (u[0] * qk[0] + u[1] * qk[1] + u[2] * qk[2])) -
               ur * dkr - vr * dir;
  const T A7 = ur * qkr - vr * qir;
  const T rad = D3 * A3 + D5 * A5 + D7 * A7;
  const T cu = F3 * ck - F5 * dkr + F7 * qkr, cv = -F3 * ci - F5 * dir - F7 * qir;
  const T cdk = -F5 * ur, cdi = -F5 * vr, cqk = T(2) * F7 * ur, cqi = T(-2) * F7 * vr, c2 = T(2) * F5;
  // Q = xx xy xz yy yz zz
  const T Qkux = Qk[0] * u[0] + Qk[1] * u[1] + Qk[2] * u[2], Qivx = Qi[0] * v[0] + Qi[1] * v[1] + Qi[2] * v[2];
  const T Qkuy = Qk[1] * u[0] + Qk[3] * u[1] + Qk[4] * u[2], Qivy = Qi[1] * v[0] + Qi[3] * v[1] + Qi[4] * v[2];
  const T Qkuz = Qk[2] * u[0] + Qk[4] * u[1] + Qk[5] * u[2], Qivz = Qi[2] * v[0] + Qi[4] * v[1] + Qi[5] * v[2];
  frc[0] += cu * u[0] + cv * v[0] + cdk * dk[0] + cdi * di[0] + cqk * qk[0] + cqi * qi[0] + c2 * (Qivx - Qkux) -
            rad * r[0];
  frc[1] += cu * u[1] + cv * v[1] + cdk * dk[1] + cdi * di[1] + cqk * qk[1] + cqi * qi[1] + c2 * (Qivy - Qkuy) -
            rad * r[1];
  frc[2] += cu * u[2] + cv * v[2] + cdk * dk[2] + cdi * di[2] + cqk * qk[2] + cqi * qi[2] + c2 * (Qivz - Qkuz) -
            rad * r[2];
  const T w5 = F5 * vr, w7 = F7 * vr;
  uf[0] += F3 * v[0] - w5 * r[0];
  uf[1] += F3 * v[1] - w5 * r[1];
  uf[2] += F3 * v[2] - w5 * r[2];
  const T tx = c2 * v[0] - w7 * r[0], ty = c2 * v[1] - w7 * r[1], tz = c2 * v[2] - w7 * r[2];
  duf[0] += r[0] * tx;
  duf[1] += r[0] * ty + r[1] * tx;
  duf[2] += r[1] * ty;
  duf[3] += r[0] * tz + r[2] * tx;
  duf[4] += r[1] * tz + r[2] * ty;
  duf[5] += r[2] * tz;
}

// epreal1c pair terms seen from atom i over its interacting pairs, the self
// torque, and the torque distribution of the summed torque of site i.
// resident blocks of the mixed gradient pass the register budget is cut for
#ifndef THP_FORCE_MINB
#define THP_FORCE_MINB 4
#endif

// special partners of a site held in registers (a longer list is searched
// past those)
constexpr int kSpCache = 4;

// A warp takes four consecutive (cell-sorted) sites, eight lanes each; the
// partners come from the pair stream of the solve whose dipoles are
// differentiated (the pairs within ewaldcut at these positions, 32 consecutive
// entries per warp step), lane j of a site taking its slots j, j+8, ...  The
// lanes' sums are combined in a fixed shuffle tree and the first lane of the
// site finishes it.  The pass is bound by the pair arithmetic.
// VIR: each block also writes to vpart[block][12] the sum of its sites' pair
// virials (epolar1.f:2326-2342, half from each end of a pair) and the
// frame-atom virial of their real-space torques (:2460-2486) in 0..5, and
// the frame-atom virial of their reciprocal and self torques, which the
// reference does not add, in 6..11.
template <bool MIXED, bool VIR>
__global__ void __launch_bounds__(kBlock, MIXED ? THP_FORCE_MINB : 1) k_force_real(
    int n, Box box, EwC ew, const double4* __restrict__ pos,
    const typename std::conditional<MIXED, float, double>::type* __restrict__ mrec, const double* __restrict__ mu,
    const float* __restrict__ erec, const float* __restrict__ muf, const int* __restrict__ perm,
    const int* __restrict__ sp_off, const int* __restrict__ sp_ks, const double* __restrict__ sp_s,
    const int* __restrict__ npr, const int* __restrict__ pk, int cap8, const int* __restrict__ frs,
    const double* __restrict__ trq_recip, FixAcc dep, double* __restrict__ vpart) {
  using T = typename std::conditional<MIXED, float, double>::type;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int i0 = t >> 3, jl = t & 7;
  const bool live = i0 < n;
  const int i = live ? i0 : n - 1;  // a valid site for the loads of idle lanes
  double vout[12] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
  {
  const double4 pi4 = pos[i];
  // mixed form: partners from the 64-B FP32 site record (wrapped position,
  // 1/pdamp, thole, multipoles) and the FP32 dipole record, imaged in FP32
  float xi = 0.f, yi = 0.f, zi = 0.f, ipdi = 0.f;
  if constexpr (MIXED) {
    xi = erec[(size_t)i * 16 + 0];
    yi = erec[(size_t)i * 16 + 1];
    zi = erec[(size_t)i * 16 + 2];
    ipdi = erec[(size_t)i * 16 + 3];
  }
  const float bxf = (float)box.l[0], byf = (float)box.l[1], bzf = (float)box.l[2];
  const float hxf = 0.5f * bxf, hyf = 0.5f * byf, hzf = 0.5f * bzf;
  const T* ri = mrec + (size_t)i * 12;
  const T pti = ri[0], ci = ri[1];
  const T di[3] = {ri[2], ri[3], ri[4]};
  const T Qi[6] = {ri[5], ri[6], ri[7], ri[8], ri[9], ri[10]};
  const double* mi = mu + (size_t)i * 6;
  const T ud[3] = {(T)mi[0], (T)mi[1], (T)mi[2]}, up[3] = {(T)mi[3], (T)mi[4], (T)mi[5]};
  const int io = perm[i];
  const int s0 = sp_off[io], s1 = sp_off[io + 1];
  int spk[kSpCache];
#pragma unroll
  for (int q = 0; q < kSpCache; ++q) spk[q] = s0 + q < s1 ? __ldg(sp_ks + s0 + q) : -1;
  const T f = (T)(0.5 * kElectric);
  double gx = 0.0, gy = 0.0, gz = 0.0;
  T uf[3] = {0, 0, 0}, duf[6] = {0, 0, 0, 0, 0, 0};
  T vp[6] = {0, 0, 0, 0, 0, 0};  // pair virial, half of each pair's
  const int nn = live ? npr[i] : 0;
  const int* __restrict__ row = pk + pair_slot(cap8, i, jl);  // slot s: 4 (s - j) entries on
  int knext = jl < nn ? __ldg(row) : i;  // partners fetched one step ahead of their records
#pragma unroll 1
  for (int s = jl; s < nn; s += 8) {
    const int k = knext;
    if (s + 8 < nn) knext = __ldg(row + 4 * (size_t)(s + 8 - jl));
    T r[3], r2, pdk, ptk, ck, dk[3], Qk[6], vd[3], vq[3];
    if constexpr (MIXED) {
      float w[16], m[8];
      ld_rec8(erec + (size_t)k * 16, *reinterpret_cast<float(*)[8]>(&w[0]));
      ld_rec8(erec + (size_t)k * 16 + 8, *reinterpret_cast<float(*)[8]>(&w[8]));
      ld_rec8(muf + (size_t)k * 8, m);
      float x = w[0] - xi, y = w[1] - yi, z = w[2] - zi;
      r[0] = fabsf(x) > hxf ? x - copysignf(bxf, x) : x;
      r[1] = fabsf(y) > hyf ? y - copysignf(byf, y) : y;
      r[2] = fabsf(z) > hzf ? z - copysignf(bzf, z) : z;
      r2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
      pdk = w[3];
      ptk = w[4];
      ck = w[5];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        dk[q] = w[6 + q];
        vd[q] = m[q];
        vq[q] = m[3 + q];
      }
#pragma unroll
      for (int q = 0; q < 6; ++q) Qk[q] = w[9 + q];
    } else {
      const double4 pk4 = pos[k];
      r[0] = pk4.x - pi4.x;
      r[1] = pk4.y - pi4.y;
      r[2] = pk4.z - pi4.z;
      image3(box, r[0], r[1], r[2]);
      r2 = r2_exact(r[0], r[1], r[2]);
      pdk = pk4.w;
      const double2* rk = reinterpret_cast<const double2*>(mrec + (size_t)k * 12);
      const double2 a0 = __ldg(rk), a1 = __ldg(rk + 1), a2 = __ldg(rk + 2), a3 = __ldg(rk + 3), a4 = __ldg(rk + 4),
                    a5 = __ldg(rk + 5);
      ptk = a0.x;
      ck = a0.y;
      dk[0] = a1.x; dk[1] = a1.y; dk[2] = a2.x;
      Qk[0] = a2.y; Qk[1] = a3.x; Qk[2] = a3.y; Qk[3] = a4.x; Qk[4] = a4.y; Qk[5] = a5.x;
      const double2* mk = reinterpret_cast<const double2*>(mu + (size_t)k * 6);
      const double2 b0 = __ldg(mk), b1 = __ldg(mk + 1), b2 = __ldg(mk + 2);
      vd[0] = b0.x; vd[1] = b0.y; vd[2] = b1.x;
      vq[0] = b1.y; vq[1] = b2.x; vq[2] = b2.y;
    }
    T ds = 1, ps = 1, us = 1;
    int sq = -1;
#pragma unroll
    for (int q = 0; q < kSpCache; ++q)
      if (spk[q] == k) sq = s0 + q;
    if (sq < 0 && s1 - s0 > kSpCache)
      for (int q = s0 + kSpCache; q < s1; ++q)
        if (__ldg(sp_ks + q) == k) {
          sq = q;
          break;
        }
    if (sq >= 0) {
      ds = (T)sp_s[3 * sq];
      ps = (T)sp_s[3 * sq + 1];
      us = (T)sp_s[3 * sq + 2];
    }
    // dampewald(9) (damping.f:17-55) and the bare terms: one reciprocal root,
    // then products
    T rinv;
    if constexpr (MIXED)
      rinv = rsqrtf(r2);
    else
      rinv = rsqrt(r2);
    const T rr = r2 * rinv, r2inv = rinv * rinv;
    PairRadial<T> p;
    const T ra = (T)ew.a * rr;
    T ex, er;
    screen(ra, ex, er);
    const T b0 = er * rinv;
    const T b1 = (b0 + (T)ew.f1 * ex) * r2inv;
    const T b2 = (T(3) * b1 + (T)ew.f2 * ex) * r2inv;
    const T b3 = (T(5) * b2 + (T)ew.f3 * ex) * r2inv;
    const T b4 = (T(7) * b3 + (T)ew.f4 * ex) * r2inv;
    p.e3 = f * b1;
    p.e5 = f * b2;
    p.e7 = f * b3;
    p.e9 = f * b4;
    p.rr3 = f * rinv * r2inv;
    p.rr5 = T(3) * p.rr3 * r2inv;
    p.rr7 = T(5) * p.rr5 * r2inv;
    p.rr9 = T(7) * p.rr7 * r2inv;
    // Thole factors and their r-derivatives (epolar1.f:1620-1660)
    p.l3 = p.l5 = p.l7 = T(1);
    p.q3 = p.q5 = p.q7 = T(0);
    T pg = min(pti, ptk);
    if (pg == T(0)) pg = max(pti, ptk);
    const T pd = MIXED ? (T)ipdi * pdk : (T)pi4.w * pdk;  // mixed: the product of the reciprocals
    if (pd != T(0) && pg != T(0)) {
      const T tt = MIXED ? rr * pd : rr / pd;
      const T damp = pg * (tt * tt * tt);
      if (damp < T(50)) {
        const T ed = exp(-damp);
        p.l3 = T(1) - ed;
        p.l5 = T(1) - (T(1) + damp) * ed;
        p.l7 = T(1) - (T(1) + damp + T(0.6) * damp * damp) * ed;
        p.q3 = T(3) * damp * ed * r2inv;
        p.q5 = p.q3 * damp;
        p.q7 = p.q5 * (T(-0.2) + T(0.6) * damp);
      }
    }
    const T dir = di[0] * r[0] + di[1] * r[1] + di[2] * r[2], dkr = dk[0] * r[0] + dk[1] * r[1] + dk[2] * r[2];
    const T qi[3] = {Qi[0] * r[0] + Qi[1] * r[1] + Qi[2] * r[2], Qi[1] * r[0] + Qi[3] * r[1] + Qi[4] * r[2],
                     Qi[2] * r[0] + Qi[4] * r[1] + Qi[5] * r[2]};
    const T qk[3] = {Qk[0] * r[0] + Qk[1] * r[1] + Qk[2] * r[2], Qk[1] * r[0] + Qk[3] * r[1] + Qk[4] * r[2],
                     Qk[2] * r[0] + Qk[4] * r[1] + Qk[5] * r[2]};
    const T qir = qi[0] * r[0] + qi[1] * r[1] + qi[2] * r[2], qkr = qk[0] * r[0] + qk[1] * r[1] + qk[2] * r[2];
    const T uir = ud[0] * r[0] + ud[1] * r[1] + ud[2] * r[2], uirp = up[0] * r[0] + up[1] * r[1] + up[2] * r[2];
    const T ukr = vd[0] * r[0] + vd[1] * r[1] + vd[2] * r[2], ukrp = vq[0] * r[0] + vq[1] * r[1] + vq[2] * r[2];
    // mutual part (uscale): F3 (ud_i.up_k + ud_k.up_i) - F5 (products along r)
    T frc[3];
    {
      const T n3 = T(1) - us * p.l3, n5 = T(1) - us * p.l5;
      const T F5 = p.e5 - n5 * p.rr5;
      const T D3 = p.e5 - n3 * p.rr5 - us * p.q3 * p.rr3, D5 = p.e7 - n5 * p.rr7 - us * p.q5 * p.rr5;
      const T A3 = (ud[0] * vq[0] + ud[1] * vq[1] + ud[2] * vq[2]) + (vd[0] * up[0] + vd[1] * up[1] + vd[2] * up[2]);
      const T rad = D3 * A3 - D5 * (uir * ukrp + ukr * uirp);
#pragma unroll
      for (int q = 0; q < 3; ++q)
        frc[q] = -F5 * (ukrp * ud[q] + uir * vq[q] + uirp * vd[q] + ukr * up[q]) - rad * r[q];
    }
    // permanent moments with the induced dipoles: the p dipoles under dscale
    // and the d dipoles under pscale, in one go when the two scales agree
    // (every pair but the few special pairs where they differ)
    {
      const bool both = ds == ps;
      T u[3], v[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        u[q] = both ? ud[q] + up[q] : up[q];
        v[q] = both ? vd[q] + vq[q] : vq[q];
      }
      perm_terms<T>(p, ds, r, u, v, both ? uir + uirp : uirp, both ? ukr + ukrp : ukrp, ci, di, Qi, ck, dk, Qk, qi, qk,
                    dir, dkr, qir, qkr, frc, uf, duf);
      if (!both)
        perm_terms<T>(p, ps, r, ud, vd, uir, ukr, ci, di, Qi, ck, dk, Qk, qi, qk, dir, dkr, qir, qkr, frc, uf, duf);
    }
    gx -= (double)frc[0];
    gy -= (double)frc[1];
    gz -= (double)frc[2];
    if (VIR) {
      const T h = T(0.5);
      vp[0] += h * (r[0] * frc[0]);
      vp[1] += h * (T(0.5) * (r[1] * frc[0] + r[0] * frc[1]));
      vp[2] += h * (T(0.5) * (r[2] * frc[0] + r[0] * frc[2]));
      vp[3] += h * (r[1] * frc[1]);
      vp[4] += h * (T(0.5) * (r[2] * frc[1] + r[1] * frc[2]));
      vp[5] += h * (r[2] * frc[2]);
    }
  }
  {
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      gx += __shfl_xor_sync(0xffffffffu, gx, o);
      gy += __shfl_xor_sync(0xffffffffu, gy, o);
      gz += __shfl_xor_sync(0xffffffffu, gz, o);
#pragma unroll
      for (int q = 0; q < 3; ++q) uf[q] += __shfl_xor_sync(0xffffffffu, uf[q], o);
#pragma unroll
      for (int q = 0; q < 6; ++q) duf[q] += __shfl_xor_sync(0xffffffffu, duf[q], o);
      if (VIR)
#pragma unroll
        for (int q = 0; q < 6; ++q) vp[q] += __shfl_xor_sync(0xffffffffu, vp[q], o);
    }
  }
  if (live && jl == 0) {
  dep.add(3 * i + 0, gx);
  dep.add(3 * i + 1, gy);
  dep.add(3 * i + 2, gz);
  // torques: real-space induced field (epolar1.f:2427-2470) + reciprocal + self
  const double* u6 = mu + (size_t)i * 6;
  const double sterm = (4.0 / 3.0) * kElectric * ew.a * ew.a * ew.a / kSqrtPi;
  const double hx = 0.5 * (u6[0] + u6[3]), hy = 0.5 * (u6[1] + u6[4]), hz = 0.5 * (u6[2] + u6[5]);
  const double rdx = (double)ri[2], rdy = (double)ri[3], rdz = (double)ri[4];
  double tep[3];
  tep[0] = (double)(di[2] * uf[1] - di[1] * uf[2] + Qi[2] * duf[1] - Qi[1] * duf[3] +
                    T(2) * Qi[4] * (duf[2] - duf[5]) + (Qi[5] - Qi[3]) * duf[4]);
  tep[1] = (double)(di[0] * uf[2] - di[2] * uf[0] - Qi[4] * duf[1] + Qi[1] * duf[4] +
                    T(2) * Qi[2] * (duf[5] - duf[0]) + (Qi[0] - Qi[5]) * duf[3]);
  tep[2] = (double)(di[1] * uf[0] - di[0] * uf[1] + Qi[4] * duf[3] - Qi[2] * duf[4] +
                    T(2) * Qi[1] * (duf[0] - duf[2]) + (Qi[3] - Qi[0]) * duf[1]);
  const int iz = frs[3 * i], ix = frs[3 * i + 1], axt = frs[3 * i + 2];
  if (VIR) {
#pragma unroll
    for (int q = 0; q < 6; ++q) vout[q] = (double)vp[q];
    if (axt == 1 || axt == 2) {
      // the real-space torque (in the reference's virial) and the reciprocal +
      // self torque (not in it), converted apart; the gradient takes both
      const double tx[3] = {trq_recip[(size_t)i * 3 + 0] + sterm * (rdy * hz - rdz * hy),
                            trq_recip[(size_t)i * 3 + 1] + sterm * (rdz * hx - rdx * hz),
                            trq_recip[(size_t)i * 3 + 2] + sterm * (rdx * hy - rdy * hx)};
      double du[3], dv[3], dux[3], dvx[3];
      torque_frame(pos, i, iz, ix, axt, tep, du, dv);
      torque_frame(pos, i, iz, ix, axt, tx, dux, dvx);
      double vr[6] = {0, 0, 0, 0, 0, 0}, vx[6] = {0, 0, 0, 0, 0, 0};
      frame_virial(pos, i, iz, ix, du, dv, vr);
      frame_virial(pos, i, iz, ix, dux, dvx, vx);
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        vout[q] += vr[q];
        vout[6 + q] = vx[q];
      }
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        dep.add(3 * iz + j, du[j] + dux[j]);
        dep.add(3 * ix + j, dv[j] + dvx[j]);
        dep.add(3 * i + j, -(du[j] + dux[j]) - (dv[j] + dvx[j]));
      }
    }
  } else {
    tep[0] += trq_recip[(size_t)i * 3 + 0] + sterm * (rdy * hz - rdz * hy);
    tep[1] += trq_recip[(size_t)i * 3 + 1] + sterm * (rdz * hx - rdx * hz);
    tep[2] += trq_recip[(size_t)i * 3 + 2] + sterm * (rdx * hy - rdy * hx);
    if (axt == 1 || axt == 2) torque_dist(pos, i, iz, ix, axt, tep, dep);
  }
  }  // the site's first lane
  }
  if (VIR) {
    block_reduce<12>(vout);
    if (threadIdx.x == 0)
#pragma unroll
      for (int q = 0; q < 12; ++q) vpart[(size_t)blockIdx.x * 12 + q] = vout[q];
  }
}

// The virial of one gradient call from the partial sums, in a fixed order:
// nk rows of 6 (k-space sums), nr rows of 6 (reciprocal sites), ne rows of
// 12 (real space: the reference's terms, then the reciprocal and self
// torques' frame-atom terms).  out: 6 + 6 (xx xy xz yy yz zz twice).
__global__ void __launch_bounds__(256) k_virial_sum(int nk, const double* __restrict__ kpart, int nr,
                                                     const double* __restrict__ rpart, int ne,
                                                     const double* __restrict__ epart, double* __restrict__ out) {
  double v[12] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (int b = threadIdx.x; b < nk; b += blockDim.x)
#pragma unroll
    for (int q = 0; q < 6; ++q) v[q] += kpart[(size_t)b * 6 + q];
  for (int b = threadIdx.x; b < nr; b += blockDim.x)
#pragma unroll
    for (int q = 0; q < 6; ++q) v[q] += rpart[(size_t)b * 6 + q];
  for (int b = threadIdx.x; b < ne; b += blockDim.x)
#pragma unroll
    for (int q = 0; q < 12; ++q) v[q] += epart[(size_t)b * 12 + q];
  block_reduce<12>(v);
  if (threadIdx.x == 0)
#pragma unroll
    for (int q = 0; q < 12; ++q) out[q] = v[q];
}

}  // namespace

template <typename P>
static int alloc_once(Ctx& c, P** p, size_t count, const char* what) {
  if (*p) return THP_OK;
  return cuda_status(cudaMalloc((void**)p, sizeof(P) * count), &c, what);
}

// fphirec [n][20] (unscaled) of the convolved permanent-multipole grid
int launch_fphi_mpole20(Ctx& c) {
  int st = alloc_once(c, &c.d_fphirec, 20 * c.cap_n, "alloc fphirec");
  if (st) return st;
  const int nb = (c.n + kBlock - 1) / kBlock;
  PmeGeom g = pme_geom(c);
  if (c.mixed)
    k_fphi_mpole20<float><<<nb, kBlock, 0, c.stream>>>(c.n, g, c.d_pos, (const cufftComplex*)c.d_conv, c.d_fphirec);
  else
    k_fphi_mpole20<double><<<nb, kBlock, 0, c.stream>>>(c.n, g, c.d_pos, (const cufftDoubleComplex*)c.d_conv,
                                                        c.d_fphirec);
  return cuda_status(cudaGetLastError(), &c, "fphi mpole");
}

// sorted frame atoms of every site into d_frs
int launch_frames_sorted(Ctx& c) {
  int st = alloc_once(c, &c.d_frs, 3 * c.cap_n, "alloc frames");
  if (st) return st;
  const int nb = (c.n + kBlock - 1) / kBlock;
  k_frames_sorted<<<nb, kBlock, 0, c.stream>>>(c.n, c.d_perm, c.d_iperm, c.d_frames, c.d_frs);
  return cuda_status(cudaGetLastError(), &c, "frames");
}

// the fixed-point gradient sums (d_depfix) to zero, allocated on first use
int zero_gradient(Ctx& c) {
  const size_t words = c.mixed ? 3 : 6;
  int st = alloc_once(c, &c.d_depfix, words * c.cap_n, "alloc gradient");
  if (st) return st;
  return cuda_status(cudaMemsetAsync(c.d_depfix, 0, sizeof(unsigned long long) * words * c.n, c.stream), &c,
                     "zero gradient");
}

// fixed-point gradient (sorted) -> dE/dx [n][3] in original order
int launch_gradient_out(Ctx& c, double* d_out) {
  const int nb = (c.n + kBlock - 1) / kBlock;
  k_dep_out<<<nb, kBlock, 0, c.stream>>>(c.n, c.d_perm, fix_acc(c.d_depfix, c.n, c.mixed), d_out);
  return cuda_status(cudaGetLastError(), &c, "gradient out");
}

// Partial-sum rows of one gradient call's virial: 2 kspace_virial_blocks()
// rows of 6 (k-space sums), nb rows of 6 and nb rows of 12 (per-block site
// and pair terms), then 12 totals; grown on demand.
int virial_scratch(Ctx& c, int nr, int ne, double** kpart, double** rpart, double** epart) {
  const int nk = 2 * kspace_virial_blocks();
  const size_t rows = (size_t)nk * 6 + (size_t)nr * 6 + (size_t)ne * 12 + 12;
  if (c.virp_cap < rows) {
    cudaFree(c.d_virp);
    c.d_virp = nullptr;
    c.virp_cap = 0;
    int st = cuda_status(cudaMalloc((void**)&c.d_virp, sizeof(double) * rows), &c, "alloc virial");
    if (st) return st;
    c.virp_cap = rows;
  }
  *kpart = c.d_virp;
  *rpart = *kpart + (size_t)nk * 6;
  *epart = *rpart + (size_t)nr * 6;
  return THP_OK;
}

// The 12 totals of the partial sums (in a fixed order; nk k-space rows)
// copied to h_out when the stream reaches them.
int virial_total(Ctx& c, int nk, int nr, int ne, const double* kpart, const double* rpart, const double* epart,
                 double* h_out) {
  double* tot = const_cast<double*>(epart) + (size_t)ne * 12;
  k_virial_sum<<<1, 256, 0, c.stream>>>(nk, kpart, nr, rpart, ne, epart, tot);
  const int st = cuda_status(cudaGetLastError(), &c, "virial sum");
  if (!st) cudaMemcpyAsync(h_out, tot, sizeof(double) * 12, cudaMemcpyDeviceToHost, c.stream);
  return st;
}

// Gradient of the polarization energy for the converged dipoles in d_mu
// (sorted); writes dE/dx [n][3] in ORIGINAL atom order into d_out.
int launch_forces(Ctx& c, double* d_out) {
  int st;
  const int nb = (c.n + kBlock - 1) / kBlock;
  if (!c.have_axes) return THP_E_STATE;
  if ((st = alloc_once(c, &c.d_fphirec, 20 * c.cap_n, "alloc fphirec"))) return st;
  if ((st = zero_gradient(c))) return st;
  if ((st = alloc_once(c, &c.d_trq, 3 * c.cap_n, "alloc torque"))) return st;
  if ((st = alloc_once(c, &c.d_frs, 3 * c.cap_n, "alloc frames"))) return st;
  const bool vir = c.want_virial;
  const int nk = 2 * kspace_virial_blocks();
  double *kpart = nullptr, *rpart = nullptr, *epart = nullptr;
  const int nbr = (c.n + 15) / 16;  // the real-space pass: eight lanes per site, blocks of 16 sites
  if (vir && (st = virial_scratch(c, nb, nbr, &kpart, &rpart, &epart))) return st;
  const FixAcc dep = fix_acc(c.d_depfix, c.n, c.mixed);
  k_frames_sorted<<<nb, kBlock, 0, c.stream>>>(c.n, c.d_perm, c.d_iperm, c.d_frames, c.d_frs);
  PmeGeom g = pme_geom(c);
  // permanent-multipole potential, 20 derivatives per site (and the
  // permanent-only k-space virial, subtracted)
  if ((st = vir ? launch_mpole_grid_virial(c, kpart, -1.0) : launch_mpole_grid(c))) return st;
  if ((st = launch_fphi_mpole20(c))) return st;
  // dipole grid of uind (Re) / uinp (Im), convolved
  if ((st = launch_pme_dipole(c, c.d_mu, nullptr, 0))) return st;
  if (c.mixed && vir)
    k_force_recip<float, true><<<nb, kBlock, 0, c.stream>>>(c.n, g, c.d_pos, (const cufftComplex*)c.d_conv,
                                                            c.d_fphirec, c.d_mu, c.d_rpole, c.d_trq, dep, rpart);
  else if (c.mixed)
    k_force_recip<float, false><<<nb, kBlock, 0, c.stream>>>(c.n, g, c.d_pos, (const cufftComplex*)c.d_conv,
                                                             c.d_fphirec, c.d_mu, c.d_rpole, c.d_trq, dep, rpart);
  else if (vir)
    k_force_recip<double, true><<<nb, kBlock, 0, c.stream>>>(c.n, g, c.d_pos, (const cufftDoubleComplex*)c.d_conv,
                                                             c.d_fphirec, c.d_mu, c.d_rpole, c.d_trq, dep, rpart);
  else
    k_force_recip<double, false><<<nb, kBlock, 0, c.stream>>>(c.n, g, c.d_pos, (const cufftDoubleComplex*)c.d_conv,
                                                              c.d_fphirec, c.d_mu, c.d_rpole, c.d_trq, dep, rpart);
  if ((st = cuda_status(cudaGetLastError(), &c, "force recip"))) return st;
  // (rpole + uinp) x (rpole + uind) k-space virial: the grid is free again
  if (vir && (st = launch_pair_grid_virial(c, kpart + (size_t)kspace_virial_blocks() * 6))) return st;
  EwC ew;
  const double a = c.cfg.aewald;
  double aesq2 = 2.0 * a * a, afac = 1.0 / (kSqrtPi * a);
  ew.a = a;
  afac *= aesq2;
  ew.f1 = afac;
  afac *= aesq2;
  ew.f2 = afac;
  afac *= aesq2;
  ew.f3 = afac;
  afac *= aesq2;
  ew.f4 = afac;
  if (c.mixed) {
    if ((st = alloc_once(c, &c.d_muf, 8 * c.cap_n, "alloc dipoles f32"))) return st;
    k_mu_f32<<<nb, kBlock, 0, c.stream>>>(c.n, c.d_mu, c.d_muf);
    if ((st = cuda_status(cudaGetLastError(), &c, "dipoles f32"))) return st;
  }
#define THP_FORCE_ARGS                                                                                            \
  c.n, c.box, ew, c.d_pos, MREC, c.d_mu, c.d_erec, c.d_muf, c.d_perm, c.d_sp_off, c.d_sp_ks, c.d_sp_s, c.d_npr, c.d_pk, \
      c.maxpr / 8, c.d_frs, c.d_trq, dep, epart
  if (c.mixed) {
#define MREC c.d_mrecf
    if (vir)
      k_force_real<true, true><<<nbr, kBlock, 0, c.stream>>>(THP_FORCE_ARGS);
    else
      k_force_real<true, false><<<nbr, kBlock, 0, c.stream>>>(THP_FORCE_ARGS);
#undef MREC
  } else {
#define MREC c.d_mrec
    if (vir)
      k_force_real<false, true><<<nbr, kBlock, 0, c.stream>>>(THP_FORCE_ARGS);
    else
      k_force_real<false, false><<<nbr, kBlock, 0, c.stream>>>(THP_FORCE_ARGS);
#undef MREC
  }
#undef THP_FORCE_ARGS
  if ((st = cuda_status(cudaGetLastError(), &c, "force real"))) return st;
  if (vir && (st = virial_total(c, nk, nb, nbr, kpart, rpart, epart, c.h_vir))) return st;
  return launch_gradient_out(c, d_out);
}

}  // namespace thp
