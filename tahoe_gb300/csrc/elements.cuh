// Hex8 kinematics and material helpers shared by the element kernels.
// Internal to the library.
#pragma once

#include <cmath>

#include "tg_internal.h"

namespace tg {

namespace {

constexpr double kGauss = 0.57735026918962576451;    // 1/sqrt(3)

// node sign patterns of HexahedronT.cpp:23-25
__host__ __device__ constexpr double sr(int a) { return (((a + 1) >> 1) & 1) ? 1.0 : -1.0; }
__host__ __device__ constexpr double ss(int a) { return ((a >> 1) & 1) ? 1.0 : -1.0; }
__host__ __device__ constexpr double st(int a) { return ((a >> 2) & 1) ? 1.0 : -1.0; }

// reference-domain derivatives of N_a at Gauss point ip (ParentDomainT)
template <typename T>
__device__ __forceinline__ void ref_grad(int ip, T dN[3][8]) {
  const T r = T(kGauss) * T(sr(ip)), s = T(kGauss) * T(ss(ip)), t = T(kGauss) * T(st(ip));
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    const T fr = T(1) + r * T(sr(a)), fs = T(1) + s * T(ss(a)), ft = T(1) + t * T(st(a));
    dN[0][a] = T(0.125) * T(sr(a)) * fs * ft;
    dN[1][a] = T(0.125) * T(ss(a)) * fr * ft;
    dN[2][a] = T(0.125) * T(st(a)) * fr * fs;
  }
}

template <typename T>
__device__ __forceinline__ T det3(const T A[9]) {
  return A[0] * (A[4] * A[8] - A[5] * A[7]) - A[1] * (A[3] * A[8] - A[5] * A[6]) +
         A[2] * (A[3] * A[7] - A[4] * A[6]);
}
template <typename T>
__device__ __forceinline__ void inv3(const T A[9], T d, T B[9]) {
  const T id = T(1) / d;
  B[0] = (A[4] * A[8] - A[5] * A[7]) * id;
  B[1] = (A[2] * A[7] - A[1] * A[8]) * id;
  B[2] = (A[1] * A[5] - A[2] * A[4]) * id;
  B[3] = (A[5] * A[6] - A[3] * A[8]) * id;
  B[4] = (A[0] * A[8] - A[2] * A[6]) * id;
  B[5] = (A[2] * A[3] - A[0] * A[5]) * id;
  B[6] = (A[3] * A[7] - A[4] * A[6]) * id;
  B[7] = (A[1] * A[6] - A[0] * A[7]) * id;
  B[8] = (A[0] * A[4] - A[1] * A[3]) * id;
}

// Jacobian, det and spatial gradients g[l][a] = dN_a/dX_l at one point
// (ParentDomainT::ComputeDNa, ParentDomainT.cpp:426-470).
template <typename T>
__device__ __forceinline__ T point_gradients(const T (*Xe)[3], int ip, T g[3][8]) {
  T dN[3][8];
  ref_grad<T>(ip, dN);
  T J[9];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      T acc = T(0);
#pragma unroll
      for (int a = 0; a < 8; ++a) acc += Xe[a][i] * dN[k][a];
      J[i * 3 + k] = acc;
    }
  const T d = det3(J);
  T Ji[9];
  inv3(J, d, Ji);
#pragma unroll
  for (int l = 0; l < 3; ++l)
#pragma unroll
    for (int a = 0; a < 8; ++a)
      g[l][a] = Ji[0 * 3 + l] * dN[0][a] + Ji[1 * 3 + l] * dN[1][a] + Ji[2 * 3 + l] * dN[2][a];
  return d;
}

// The same for the current configuration x = X + u (updated Lagrangian):
// gradients dN/dx and det(dx/dxi), no coordinate array formed.
template <typename T>
__device__ __forceinline__ T point_gradients_current(const T (*Xe)[3], const T (*Ue)[3], int ip, T g[3][8]) {
  T dN[3][8];
  ref_grad<T>(ip, dN);
  T J[9];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      T acc = T(0);
#pragma unroll
      for (int a = 0; a < 8; ++a) acc += (Xe[a][i] + Ue[a][i]) * dN[k][a];
      J[i * 3 + k] = acc;
    }
  const T d = det3(J);
  T Ji[9];
  inv3(J, d, Ji);
#pragma unroll
  for (int l = 0; l < 3; ++l)
#pragma unroll
    for (int a = 0; a < 8; ++a)
      g[l][a] = Ji[0 * 3 + l] * dN[0][a] + Ji[1 * 3 + l] * dN[1][a] + Ji[2 * 3 + l] * dN[2][a];
  return d;
}

template <typename T>
__device__ __forceinline__ void deviatoric(const T a[6], T d[6]) {
  const T m = (a[0] + a[1] + a[2]) / T(3);
  d[0] = a[0] - m;
  d[1] = a[1] - m;
  d[2] = a[2] - m;
  d[3] = a[3];
  d[4] = a[4];
  d[5] = a[5];
}

// J = sqrt(det b), 1/J and J^(-2/3) = (det b)^(-1/3) of the Simo model.
// In FP64 without the library's FP64 sqrt, pow and division (GB300 issues
// FP64 at a small fraction of the FP32 rate, and pow is an FP64 log and exp):
// FP32 estimates of (det b)^(-1/2) and (det b)^(-1/3) refined by Newton's
// method on r^-2 = d (r <- r (3 - d r^2) / 2) and y^-3 = d
// (y <- y (4 - d y^3) / 3), two steps each -- the error of an estimate good
// to 2^-24 squares with every step, to FP64 rounding after two.  Outside
// the range of FP32 the library functions are used.  In FP32 the library
// functions throughout.
__device__ __forceinline__ void simo_roots(double d, double& J, double& invJ, double& sc) {
  if (d > 1e-30 && d < 1e30) {
    double r = (double)rsqrtf((float)d);
    r = r * (1.5 - 0.5 * d * r * r);
    r = r * (1.5 - 0.5 * d * r * r);
    double y = (double)rcbrtf((float)d);
    y = y * (4.0 - d * (y * y * y)) * (1.0 / 3.0);
    y = y * (4.0 - d * (y * y * y)) * (1.0 / 3.0);
    invJ = r;
    J = d * r;
    sc = y;
  } else {
    J = sqrt(d);
    invJ = 1.0 / J;
    sc = pow(J, -2.0 / 3.0);
  }
}
__device__ __forceinline__ void simo_roots(float d, float& J, float& invJ, float& sc) {
  J = sqrtf(d);
  invJ = 1.0f / J;
  sc = powf(J, -2.0f / 3.0f);
}

// the isotropic modulus matrix of E and nu (or of equal entries)
inline bool isotropic_moduli(const MatParams& m) {
  const double l = m.C[1], g = m.C[21];
  for (int i = 0; i < 6; ++i)
    for (int j = 0; j < 6; ++j) {
      const double want = i < 3 && j < 3 ? (i == j ? l + 2.0 * g : l) : (i == j ? g : 0.0);
      if (m.C[i * 6 + j] != want) return false;
    }
  return true;
}

struct J2View {
  int8_t* flags;
  int8_t* alloc;
  double* alpha;
  double* dgamma;
  double* norm;
  double* epsp;
  double* nhat;
  long long nip;
};

}  // namespace
}  // namespace tg
