// conv_dev.cuh -- the PME convolution (forward transform, influence function,
// inverse transform) of cubic grids in three kernels.
//
// fft_mpi.f90:65,115 and the qfac product of newinduce_pme.f:1802-1854, with
// both transforms unnormalised.  For a grid length N = R1 R2 every
// one-dimensional transform is two register-resident DFTs of R1 and R2 points
// with one exchange through shared memory between them (Cooley and Tukey
// 1965):
//   n = R2 n1 + n2, k = k1 + R1 k2:
//   X[k] = DFT_R2 over n2 of ( W_N^{n2 k1} DFT_R1 over n1 of x ).
// The three kernels of one convolution:
//   k_conv_xy    a block per z plane: x and y transforms of the plane in shared
//                memory; the grid it read is zeroed for the next spread;
//   k_conv_z     a block per tile of neighbouring (x, y) columns: z transform,
//                influence function and inverse z transform, the product and
//                the two R2 DFTs around it in the same registers;
//   k_conv_yx    a block per z plane: inverse y and x transforms.
// cuFFT needed six launches and a separate pass for the product, each reading
// and writing the whole grid; here the grid crosses L2 three times.
//
// The x frequencies stay in the order the in-place x transform leaves them
// (position R2 k1 + k2 holds frequency k1 + R1 k2): only the influence
// function has to know, and it is stored in that order.
// The including file defines conv_real as the grid's real type.
#pragma once

#include <utility>

#include "conv.h"
#include "pme_dev.cuh"

namespace thp {
namespace conv {

// ---- compile-time roots of unity ----------------------------------------------
constexpr double kTwoPi = 6.283185307179586476925286766559;

// cos and sin of x in [0, pi/4] by their Taylor series (to 1e-19)
constexpr double taylor_cos(double x) {
  double t = 1.0, s = 1.0;
  for (int k = 1; k < 12; ++k) {
    t = -t * x * x / ((2.0 * k - 1.0) * (2.0 * k));
    s += t;
  }
  return s;
}
constexpr double taylor_sin(double x) {
  double t = x, s = x;
  for (int k = 1; k < 12; ++k) {
    t = -t * x * x / ((2.0 * k) * (2.0 * k + 1.0));
    s += t;
  }
  return s;
}
// cos(2 pi k / n), exact at the multiples of pi/4's symmetries
constexpr double root_cos(int k, int n) {
  k %= n;
  if (k < 0) k += n;
  if (2 * k > n) k = n - k;                            // cos(-x) = cos x
  if (4 * k > n) return -root_cos(n - 2 * k, 2 * n);   // cos(pi - x): (n/2 - k) / n
  if (8 * k > n) return taylor_sin(kTwoPi * (n - 4 * k) / (4.0 * n));  // sin(pi/2 - x)
  return taylor_cos(kTwoPi * k / n);
}
constexpr double root_sin(int k, int n) { return root_cos(4 * k - n, 4 * n); }  // cos(x - pi/2)

template <int I>
struct Int {
  static constexpr int value = I;
};
template <typename F, int... I>
__device__ __forceinline__ void for_each_impl(F&& f, std::integer_sequence<int, I...>) {
  (f(Int<I>{}), ...);
}
// f(Int<0>{}), ..., f(Int<N-1>{}): a loop whose index is a constant
template <int N, typename F>
__device__ __forceinline__ void for_each(F&& f) {
  for_each_impl(f, std::make_integer_sequence<int, N>{});
}

// v * exp(-2 pi i K / N) (forward), the conjugate root when INV
template <int K, int N, bool INV, typename C>
__device__ __forceinline__ C mul_root(C v) {
  using T = decltype(v.x);
  constexpr int k = ((K % N) + N) % N;
  if constexpr (k == 0) {
    return v;
  } else if constexpr (4 * k == N) {  // -i (forward)
    return INV ? C{-v.y, v.x} : C{v.y, -v.x};
  } else if constexpr (2 * k == N) {
    return C{-v.x, -v.y};
  } else if constexpr (4 * k == 3 * N) {
    return INV ? C{v.y, -v.x} : C{-v.y, v.x};
  } else {
    constexpr T c = (T)root_cos(k, N);
    constexpr T s = (T)(INV ? root_sin(k, N) : -root_sin(k, N));
    return C{v.x * c - v.y * s, v.x * s + v.y * c};
  }
}

template <typename C>
__device__ __forceinline__ C cadd(C a, C b) {
  return C{a.x + b.x, a.y + b.y};
}
template <typename C>
__device__ __forceinline__ C csub(C a, C b) {
  return C{a.x - b.x, a.y - b.y};
}

// first factor of a composite DFT length
constexpr int dft_split(int n) { return n % 4 == 0 && n > 4 ? 4 : n % 2 == 0 && n > 2 ? 2 : n % 3 == 0 && n > 3 ? 3 : 1; }

// In-register DFT of N points, natural order in and out; kernel
// exp(-2 pi i k n / N) forward, its conjugate when INV.
template <int N, bool INV, typename C>
__device__ __forceinline__ void dft(C (&v)[N]) {
  using T = decltype(v[0].x);
  if constexpr (N == 2) {
    const C a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if constexpr (N == 3) {
    constexpr T s = (T)(INV ? root_sin(1, 3) : -root_sin(1, 3));
    const C t = cadd(v[1], v[2]), d = csub(v[1], v[2]);
    const C m = C{v[0].x - T(0.5) * t.x, v[0].y - T(0.5) * t.y};
    v[0] = cadd(v[0], t);
    v[1] = C{m.x - s * d.y, m.y + s * d.x};
    v[2] = C{m.x + s * d.y, m.y - s * d.x};
  } else if constexpr (N == 4) {
    const C a = cadd(v[0], v[2]), b = csub(v[0], v[2]), c = cadd(v[1], v[3]), d = csub(v[1], v[3]);
    v[0] = cadd(a, c);
    v[2] = csub(a, c);
    v[1] = INV ? C{b.x - d.y, b.y + d.x} : C{b.x + d.y, b.y - d.x};
    v[3] = INV ? C{b.x + d.y, b.y - d.x} : C{b.x - d.y, b.y + d.x};
  } else if constexpr (N == 5) {
    constexpr T c1 = (T)root_cos(1, 5), c2 = (T)root_cos(2, 5);
    constexpr T s1 = (T)(INV ? root_sin(1, 5) : -root_sin(1, 5)), s2 = (T)(INV ? root_sin(2, 5) : -root_sin(2, 5));
    const C a = cadd(v[1], v[4]), b = cadd(v[2], v[3]), c = csub(v[1], v[4]), d = csub(v[2], v[3]);
    const C p = C{v[0].x + c1 * a.x + c2 * b.x, v[0].y + c1 * a.y + c2 * b.y};
    const C q = C{v[0].x + c2 * a.x + c1 * b.x, v[0].y + c2 * a.y + c1 * b.y};
    const C r = C{s1 * c.x + s2 * d.x, s1 * c.y + s2 * d.y};
    const C u = C{s2 * c.x - s1 * d.x, s2 * c.y - s1 * d.y};
    v[0] = C{v[0].x + a.x + b.x, v[0].y + a.y + b.y};
    v[1] = C{p.x - r.y, p.y + r.x};
    v[4] = C{p.x + r.y, p.y - r.x};
    v[2] = C{q.x - u.y, q.y + u.x};
    v[3] = C{q.x + u.y, q.y - u.x};
  } else {
    constexpr int A = dft_split(N), B = N / A;
    static_assert(A > 1, "lengths of the factors 2, 3, 4 and 5");
    C t[A][B];
    for_each<B>([&](auto bi) {
      constexpr int b = decltype(bi)::value;
      C u[A];
#pragma unroll
      for (int a = 0; a < A; ++a) u[a] = v[a * B + b];
      dft<A, INV>(u);
      for_each<A>([&](auto ki) {
        constexpr int k = decltype(ki)::value;
        t[k][b] = mul_root<b * k, N, INV>(u[k]);
      });
    });
#pragma unroll
    for (int k = 0; k < A; ++k) {
      dft<B, INV>(t[k]);
#pragma unroll
      for (int q = 0; q < B; ++q) v[k + A * q] = t[k][q];
    }
  }
}

// ---- grid lengths -----------------------------------------------------------------
// The lengths of the reference's grid list (kewald.f:67-73) up to 160 as
// R1 x R2 with R <= 16: a thread holds one DFT in registers.
#define THP_CONV_LENGTHS(X) \
  X(16, 4, 4) X(18, 3, 6) X(20, 4, 5) X(24, 4, 6) X(30, 5, 6) X(32, 4, 8) X(36, 6, 6) X(40, 5, 8) X(48, 6, 8) \
  X(50, 5, 10) X(54, 6, 9) X(60, 6, 10) X(64, 8, 8) X(72, 8, 9) X(80, 8, 10) X(90, 9, 10) X(96, 8, 12) \
  X(100, 10, 10) X(108, 9, 12) X(120, 10, 12) X(128, 8, 16) X(144, 12, 12) X(150, 10, 15) X(160, 10, 16)

constexpr size_t kMaxSmem = 227 * 1024;

// a plane in shared memory: rows of N + 1 points, so that the threads of one
// warp, on consecutive rows in the second x stage, hit distinct banks
template <typename T, int N>
constexpr size_t plane_bytes() {
  return sizeof(typename Cplx<T>::type) * (size_t)N * (N + 1);
}

// exp(-2 pi i m / N), m < N
template <typename T, int N>
struct RootTable {
  alignas(2 * sizeof(T)) T v[2 * N];  // (cos, sin) pairs, one load each
  constexpr RootTable() : v() {
    for (int m = 0; m < N; ++m) {
      v[2 * m] = (T)root_cos(m, N);
      v[2 * m + 1] = (T)-root_sin(m, N);
    }
  }
};
template <typename T, int N>
__device__ __forceinline__ const RootTable<T, N>& roots();
#define THP_ROOTS(N, A, B)                                                    \
  static __device__ RootTable<conv_real, N> d_roots_##N;                      \
  template <>                                                                 \
  __device__ __forceinline__ const RootTable<conv_real, N>& roots<conv_real, N>() { \
    return d_roots_##N;                                                       \
  }
THP_CONV_LENGTHS(THP_ROOTS)
#undef THP_ROOTS

template <typename T, int N, bool INV, typename C>
__device__ __forceinline__ C mul_table(C v, int m) {
  const C w = __ldg(reinterpret_cast<const C*>(&roots<T, N>().v[2 * m]));
  const T c = w.x, s = INV ? -w.y : w.y;
  return C{v.x * c - v.y * s, v.x * s + v.y * c};
}

// the arrays of system y of the launch: one system (many null) or many
__device__ __forceinline__ Sys system_of(const Sys& one, const Sys* __restrict__ many) {
  Sys s = one;
  if (many) s = many[blockIdx.y];
  return s;
}

template <typename T, int N, int R>
constexpr int plane_threads() {  // a thread per DFT of the wider stage, within the register file
  const int want = (N * R + 31) / 32 * 32;
  const int most = sizeof(T) == 4 ? 768 : 512;
  return want < most ? want : most;
}

template <typename T, int N, int R1, int R2, int TH, bool REAL>
__global__ void __launch_bounds__(TH) k_conv_xy(Sys one, const Sys* __restrict__ many, int check_stop) {
  using C = typename Cplx<T>::type;
  extern __shared__ __align__(16) unsigned char conv_smem[];
  C* sm = reinterpret_cast<C*>(conv_smem);
  const Sys s = system_of(one, many);
  if (check_stop && s.cg->stop) return;
  constexpr int LD = N + 1;
  C* __restrict__ in = static_cast<C*>(s.in) + (size_t)blockIdx.x * N * N;
  T* __restrict__ rin = static_cast<T*>(s.in) + (size_t)blockIdx.x * N * N;
  C* __restrict__ out = static_cast<C*>(s.out) + (size_t)blockIdx.x * N * N;
  for (int b = threadIdx.x; b < N * R2; b += TH) {
    const int row = b / R2, n2 = b - row * R2;
    C v[R1];
    if constexpr (REAL) {
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1) v[n1] = C{rin[row * N + R2 * n1 + n2], T(0)};
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1) rin[row * N + R2 * n1 + n2] = T(0);
    } else {
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1) v[n1] = in[row * N + R2 * n1 + n2];
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1) in[row * N + R2 * n1 + n2] = C{T(0), T(0)};
    }
    dft<R1, false>(v);
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1)
      sm[row * LD + R2 * k1 + n2] = k1 ? mul_table<T, N, false>(v[k1], n2 * k1) : v[k1];
  }
  __syncthreads();
  for (int b = threadIdx.x; b < N * R1; b += TH) {
    const int k1 = b / N, row = b - k1 * N;
    C v[R2];
    C* q = sm + row * LD + R2 * k1;
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) v[n2] = q[n2];
    dft<R2, false>(v);
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) q[n2] = v[n2];
  }
  __syncthreads();
  for (int b = threadIdx.x; b < N * R2; b += TH) {
    const int n2 = b / N, col = b - n2 * N;
    C v[R1];
    C* q = sm + n2 * LD + col;
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) v[n1] = q[R2 * n1 * LD];
    dft<R1, false>(v);
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) q[R2 * k1 * LD] = k1 ? mul_table<T, N, false>(v[k1], n2 * k1) : v[k1];
  }
  __syncthreads();
  for (int b = threadIdx.x; b < N * R1; b += TH) {
    const int k1 = b / N, col = b - k1 * N;
    C v[R2];
    const C* q = sm + R2 * k1 * LD + col;
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) v[n2] = q[n2 * LD];
    dft<R2, false>(v);
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) out[(k1 + R1 * k2) * N + col] = v[k2];
  }
}

template <typename T, int N, int R1, int R2, int TH, bool REAL>
__global__ void __launch_bounds__(TH) k_conv_yx(Sys one, const Sys* __restrict__ many, int check_stop) {
  using C = typename Cplx<T>::type;
  extern __shared__ __align__(16) unsigned char conv_smem[];
  C* sm = reinterpret_cast<C*>(conv_smem);
  const Sys s = system_of(one, many);
  if (check_stop && s.cg->stop) return;
  constexpr int LD = N + 1;
  C* __restrict__ out = static_cast<C*>(s.out) + (size_t)blockIdx.x * N * N;
  T* __restrict__ pot = static_cast<T*>(s.pot) + (size_t)blockIdx.x * N * N;
  for (int b = threadIdx.x; b < N * R1; b += TH) {
    const int k1 = b / N, col = b - k1 * N;
    C v[R2];
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) v[k2] = out[(k1 + R1 * k2) * N + col];
    dft<R2, true>(v);
    C* q = sm + R2 * k1 * LD + col;
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) q[n2 * LD] = n2 ? mul_table<T, N, true>(v[n2], n2 * k1) : v[n2];
  }
  __syncthreads();
  for (int b = threadIdx.x; b < N * R2; b += TH) {
    const int n2 = b / N, col = b - n2 * N;
    C v[R1];
    C* q = sm + n2 * LD + col;
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) v[k1] = q[R2 * k1 * LD];
    dft<R1, true>(v);
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) q[R2 * n1 * LD] = v[n1];
  }
  __syncthreads();
  for (int b = threadIdx.x; b < N * R1; b += TH) {
    const int k1 = b / N, row = b - k1 * N;
    C v[R2];
    C* q = sm + row * LD + R2 * k1;
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) v[k2] = q[k2];
    dft<R2, true>(v);
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) q[n2] = n2 ? mul_table<T, N, true>(v[n2], n2 * k1) : v[n2];
  }
  __syncthreads();
  for (int b = threadIdx.x; b < N * R2; b += TH) {
    const int row = b / R2, n2 = b - row * R2;
    C v[R1];
    const C* q = sm + row * LD + n2;
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) v[k1] = q[R2 * k1];
    dft<R1, true>(v);
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) {
      if constexpr (REAL)
        pot[row * N + R2 * n1 + n2] = v[n1].x;
      else
        out[row * N + R2 * n1 + n2] = v[n1];
    }
  }
}

// columns of one z block: 128 bytes of each plane row segment
template <typename T>
constexpr int kZCols = 128 / (2 * (int)sizeof(T));

template <typename T, int N, int R1, int R2>
__global__ void __launch_bounds__(kZCols<T>*(R1 > R2 ? R1 : R2)) k_conv_z(Sys one, const Sys* __restrict__ many,
                                                                          int check_stop) {
  using C = typename Cplx<T>::type;
  constexpr int W = kZCols<T>, NN = N * N;
  __shared__ C sm[N * W];
  const Sys s = system_of(one, many);
  if (check_stop && s.cg->stop) return;
  const int c = threadIdx.x % W, t = threadIdx.x / W;
  const int col = blockIdx.x * W + c;
  const bool in = col < NN;
  C* __restrict__ g = static_cast<C*>(s.out) + (in ? col : 0);
  const T* __restrict__ qf = static_cast<const T*>(s.qfac) + (in ? col : 0);
  if (t < R2) {
    C v[R1];
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) v[n1] = g[(size_t)(R2 * n1 + t) * NN];
    dft<R1, false>(v);
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1)
      sm[(R2 * k1 + t) * W + c] = k1 ? mul_table<T, N, false>(v[k1], t * k1) : v[k1];
  }
  __syncthreads();
  if (t < R1) {
    C v[R2];
    T f[R2];
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) f[k2] = __ldg(qf + (size_t)(t + R1 * k2) * NN);
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) v[n2] = sm[(R2 * t + n2) * W + c];
    dft<R2, false>(v);
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) v[k2] = C{v[k2].x * f[k2], v[k2].y * f[k2]};
    dft<R2, true>(v);
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) sm[(R2 * t + n2) * W + c] = n2 ? mul_table<T, N, true>(v[n2], n2 * t) : v[n2];
  }
  __syncthreads();
  if (t < R2 && in) {
    C v[R1];
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) v[k1] = sm[(R2 * k1 + t) * W + c];
    dft<R1, true>(v);
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) g[(size_t)(R2 * n1 + t) * NN] = v[n1];
  }
}

// The three launches for one system (many null) or for count systems of one
// grid length.
template <typename T, int N, int R1, int R2, bool REAL>
cudaError_t launch(const Sys& one, const Sys* many, int count, int check_stop, cudaStream_t st) {
  constexpr int TH = plane_threads<T, N, (R1 > R2 ? R1 : R2)>();
  constexpr size_t smem = plane_bytes<T, N>();
  constexpr int W = kZCols<T>;
  static std::atomic<unsigned long long> set_xy{0}, set_yx{0};
  if (smem > 48 * 1024) {
    smem_limit_once(k_conv_xy<T, N, R1, R2, TH, REAL>, smem, set_xy);
    smem_limit_once(k_conv_yx<T, N, R1, R2, TH, REAL>, smem, set_yx);
  }
  k_conv_xy<T, N, R1, R2, TH, REAL><<<dim3(N, count), TH, smem, st>>>(one, many, check_stop);
  k_conv_z<T, N, R1, R2><<<dim3((N * N + W - 1) / W, count), W*(R1 > R2 ? R1 : R2), 0, st>>>(one, many, check_stop);
  k_conv_yx<T, N, R1, R2, TH, REAL><<<dim3(N, count), TH, smem, st>>>(one, many, check_stop);
  return cudaGetLastError();
}

// length N of type T: whether the three-kernel form covers it (a plane has to
// fit in one SM's shared memory), its factors, and its launch
template <typename T>
bool split_of(int n, int* r1, int* r2) {
#define THP_CASE(N, A, B)                         \
  if constexpr (plane_bytes<T, N>() <= kMaxSmem)  \
    if (n == N) {                                 \
      *r1 = A;                                    \
      *r2 = B;                                    \
      return true;                                \
    }
  THP_CONV_LENGTHS(THP_CASE)
#undef THP_CASE
  return false;
}

template <typename T>
cudaError_t launch_length(int n, const Sys& one, const Sys* many, int count, int check_stop, bool real,
                          cudaStream_t st) {
#define THP_CASE(N, A, B)                        \
  if constexpr (plane_bytes<T, N>() <= kMaxSmem) \
    if (n == N)                                  \
      return real ? launch<T, N, A, B, true>(one, many, count, check_stop, st) \
                  : launch<T, N, A, B, false>(one, many, count, check_stop, st);
  THP_CONV_LENGTHS(THP_CASE)
#undef THP_CASE
  return cudaErrorInvalidValue;
}

}  // namespace conv
}  // namespace thp
