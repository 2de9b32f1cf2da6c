// Element internal forces of a total-Lagrangian Simo group in FP64
// (TotalLagrangianT::FormKd, TotalLagrangianT.cpp:107, with SimoIso3D::s_ij,
// SimoIso3D.cpp:102-135).
//
// Bound by the FP64 pipe: GB300 issues one FP64 warp instruction per 64
// cycles and scheduler, so the operations are counted, and everything that is
// not FP64 arithmetic (shuffles, loads, sign changes) is free beside them.
// Per Gauss point 178 FP64 operations where the general kernel (elements.cu)
// takes about 350:
//   * The 8 lanes of an element hold its nodes and its points in the same
//     order, and the trilinear functions are products of (1 +- g)/2 per
//     direction, so the reference gradients du/dxi are lane differences and
//     two lane interpolations a component (27 operations in place of the 72
//     of sum_a u_a dN_a/dX), the map to X is 27 more, and the transposed steps
//     take the point stress back to nodal forces (27 + 30 in place of 72 and
//     the 21 additions of the reduction over the points).  The difference
//     comes first: it is nearly exact, so rigid displacements leave smaller
//     errors than the sums over nodes do.
//   * The first Piola-Kirchhoff stress directly: with C = dJ/dF = J F^-T,
//       w P = w mu J^(-2/3) F + w (kappa/2 (J - 1/J) - mu J^(-2/3) F:F/(3J)) C,
//     no b, no Cauchy stress, no inverse and no division.
//   * 1/J and J^(-1/3) from FP32 estimates by one step each of Householder's
//     method: e = 1 - J r, r (1 + e + e^2), and e = 1 - J y^3,
//     y (1 + e/3 + 2 e^2/9); estimates good to 2^-22 leave truncations below
//     2^-64.
// The geometry is 10 planes a point (the inverse Jacobian scaled by
// ((1 + g)/2)^2 / 2, and w det J), 80 bytes where dN/dX takes 200.
//
// Measured with the nodal gather on 59,400 elements (45x40x33): 355 us with the
// general kernel, 194 with this one; 504 elements 43 and 25 us.  Small meshes
// fill the chip best with small CTAs: 8 elements each.
#include "elements.cuh"

namespace tg {

namespace {

constexpr int kTlElems = 8;  // elements per CTA, 8 lanes each
// (1 - g)/(1 + g), g = 1/sqrt(3): weight of the far node over the near one
constexpr double kFar = (1.0 - kGauss) / (1.0 + kGauss);
constexpr double kScale = 0.125 * (1.0 + kGauss) * (1.0 + kGauss);

__device__ __forceinline__ double flip(double v, unsigned sign) {
  return __hiloint2double(__double2hiint(v) ^ (int)sign, __double2loint(v));
}
__device__ __forceinline__ double other(double v, int lane_xor) { return __shfl_xor_sync(0xffffffffu, v, lane_xor); }
__device__ __forceinline__ double blend(double v, int lane_xor) { return v + kFar * other(v, lane_xor); }

// r = 1/J, sc = J^(-2/3); the library functions outside the range of FP32
__device__ __forceinline__ void roots(double J, double& r, double& sc) {
  if (J > 1e-30 && J < 1e30) {
    const float Jf = (float)J;
    r = (double)__fdividef(1.0f, Jf);
    const double e = 1.0 - J * r;
    r += r * (e + e * e);
    double y = (double)rcbrtf(Jf);
    const double d = 1.0 - J * (y * y * y);
    y += y * (d * (1.0 / 3.0 + (2.0 / 9.0) * d));
    sc = y * y;
  } else {
    r = 1.0 / J;
    sc = pow(J, -2.0 / 3.0);
  }
}

__global__ void __launch_bounds__(kTlElems * 8) residual_tl_kernel(
    const int* __restrict__ conn, const int8_t* __restrict__ blk, int nel, const double4_32a* __restrict__ u,
    MatTable mt, const JacPlane* __restrict__ geo, const int* __restrict__ src, long long gstride,
    double4_32a* __restrict__ fint, int* status) {
  const int ip = threadIdx.x & 7;
  const long long e = (long long)blockIdx.x * kTlElems + (threadIdx.x >> 3);
  const bool valid = e < nel;
  double ue[3] = {0.0, 0.0, 0.0}, Ji[9], w = 0.0;
#pragma unroll
  for (int k = 0; k < 9; ++k) Ji[k] = 0.0;
  if (valid) {
    const double4_32a un = u[conn[e * 8 + ip]];
    ue[0] = un.x;
    ue[1] = un.y;
    ue[2] = un.z;
    const long long at = (src ? (long long)src[e] : e) * 8 + ip;
#pragma unroll
    for (int k = 0; k < 9; ++k) Ji[k] = geo[k * gstride + at].v;
    w = geo[9 * gstride + at].v;
  }
  // the material, read with constant indices from the parameter space
  const int bi = valid && blk ? blk[e] : 0;
  double mu = mt.m[0].mu, kappa = mt.m[0].kappa;
#pragma unroll
  for (int b = 1; b < kMaxBlocks; ++b)
    if (bi == b) {
      mu = mt.m[b].mu;
      kappa = mt.m[b].kappa;
    }
  // sign bits of this lane's corner; lanes that differ in one direction only:
  // r by 1, s by 3, t by 4
  const unsigned nr = sr(ip) < 0.0 ? 0x80000000u : 0u, ns = ss(ip) < 0.0 ? 0x80000000u : 0u,
                 nt = st(ip) < 0.0 ? 0x80000000u : 0u;
  double F[9];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const double v = ue[i];
    const double dr = blend(blend(flip(v - other(v, 1), nr), 3), 4);
    const double ds = blend(blend(flip(v - other(v, 3), ns), 1), 4);
    const double dt = blend(blend(flip(v - other(v, 4), nt), 1), 3);
#pragma unroll
    for (int l = 0; l < 3; ++l)
      F[i * 3 + l] = (i == l ? 1.0 : 0.0) + dr * Ji[l] + ds * Ji[3 + l] + dt * Ji[6 + l];
  }
  double C[9];
  C[0] = F[4] * F[8] - F[5] * F[7];
  C[1] = F[5] * F[6] - F[3] * F[8];
  C[2] = F[3] * F[7] - F[4] * F[6];
  C[3] = F[2] * F[7] - F[1] * F[8];
  C[4] = F[0] * F[8] - F[2] * F[6];
  C[5] = F[1] * F[6] - F[0] * F[7];
  C[6] = F[1] * F[5] - F[2] * F[4];
  C[7] = F[2] * F[3] - F[0] * F[5];
  C[8] = F[0] * F[4] - F[1] * F[3];
  const double J = F[0] * C[0] + F[1] * C[1] + F[2] * C[2];
  double a = 0.0, b = 0.0;
  const bool good = J > 0.0 && w > 0.0;
  if (good) {
    double r, sc;
    roots(J, r, sc);
    double tr = 0.0;
#pragma unroll
    for (int k = 0; k < 9; ++k) tr += F[k] * F[k];
    a = mu * sc;
    b = w * (0.5 * kappa * (J - r) - a * (tr * (r * (1.0 / 3.0))));
    a *= w;
  } else if (valid) {
    atomicOr(status, kStatusBadJacobian);
  }
  // w P on the reference domain; a bad point has no force
  double q[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    double P[3];
#pragma unroll
    for (int l = 0; l < 3; ++l) P[l] = a * F[i * 3 + l] + b * C[i * 3 + l];
#pragma unroll
    for (int k = 0; k < 3; ++k)
      q[i][k] = good ? P[0] * Ji[k * 3] + P[1] * Ji[k * 3 + 1] + P[2] * Ji[k * 3 + 2] : 0.0;
  }
  double f[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const double qr = blend(q[i][0], 3), qs = blend(q[i][1], 1), qt = blend(blend(q[i][2], 1), 3);
    const double rs = flip(qr + other(qr, 1), nr) + flip(qs + other(qs, 3), ns);
    f[i] = blend(rs, 4) + flip(qt + other(qt, 4), nt);
  }
  if (valid) fint[e * 8 + ip] = make_double4_32a(f[0], f[1], f[2], 0.0);
}

// The planes: inverse Jacobian (row k: dxi_k/dX), scaled, and w det J.
__global__ void jacobian_kernel(const double* __restrict__ X, int nnd, const int* __restrict__ conn, int nel,
                                JacPlane* __restrict__ geo, long long stride, long long off) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (long long)nel * 8) return;
  const long long e = k >> 3;
  double dN[3][8], J[9], Ji[9];
  ref_grad<double>((int)(k & 7), dN);
#pragma unroll
  for (int q = 0; q < 9; ++q) J[q] = 0.0;
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    const int n = conn[e * 8 + a];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double x = X[(long long)i * nnd + n];
#pragma unroll
      for (int l = 0; l < 3; ++l) J[i * 3 + l] += x * dN[l][a];
    }
  }
  const double d = det3(J);
  inv3(J, d, Ji);
#pragma unroll
  for (int q = 0; q < 9; ++q) geo[q * stride + off + k].v = kScale * Ji[q];
  geo[9 * stride + off + k].v = d;
}

}  // namespace

template <>
int launch_geometry<JacPlane>(Context* c, const double* X, int nnd, const int* conn, int nel, JacPlane* geo,
                              long long stride, long long off) {
  const long long nip = (long long)nel * 8;
  jacobian_kernel<<<(unsigned)((nip + 255) / 256), 256, 0, c->stream>>>(X, nnd, conn, nel, geo, stride, off);
  c->launches++;
  return ok(c, cudaGetLastError(), "jacobian_kernel") ? TG_OK : TG_ERR_CUDA;
}

int launch_residual_tl(Context* c, const JacPlane* geo, const int* src, long long gstride) {
  residual_tl_kernel<<<(c->nel + kTlElems - 1) / kTlElems, kTlElems * 8, 0, c->stream>>>(
      c->d_conn, c->d_block, c->nel, c->d_u, c->mats, geo, src, gstride, c->d_fint, c->d_status);
  c->launches++;
  return ok(c, cudaGetLastError(), "residual_tl_kernel") ? TG_OK : TG_ERR_CUDA;
}

}  // namespace tg
