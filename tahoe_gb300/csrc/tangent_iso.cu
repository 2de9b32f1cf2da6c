// Element tangents for moduli of the isotropic form, sm_103a.
//
// The spatial moduli of the Simo neo-Hookean, the isotropic Hookean and the J2
// material are, with n a symmetric tensor,
//   c = A I (x) I + 2 B I_sym + C (n (x) I + I (x) n)   (Simo: n = dev b-bar)
//   c = A I (x) I + 2 B I_sym + C n (x) n               (J2: n the flow direction)
// so the 3x3 block of nodes a and b at one point is, with g = grad N, m = n g,
//   K_ab = U_a (x) g_b + V_a (x) W_b + B g_b (x) g_a + (g_a . t_b) I
//   Simo: U = A g + C m, V = g, W = C m, t = B g + sigma g (geometric term)
//   J2:   U = A g, V = C m, W = m, t = B g
// (SolidElementT::FormStiffness with SimoIso3D::c_ijkl, SimoIso3D.cpp:16-53,
// 102-135, HookeanMatT.cpp:103 and J2SSC0HardeningT::ModuliCorrection,
// J2SSC0HardeningT.cpp:148-176; small strain and total Lagrangian,
// SmallStrainT.cpp:285, TotalLagrangianT.cpp:40).  30 FMA per block and point
// with 9 values per node, where the general 6x6 moduli (tangent_kernel,
// elements.cu) take 30 and a 6x3 product D B_b of 63 per node, all through
// shared memory: that kernel ran at 0.2 of the FP32 rate, waiting for operands.
//
// Split: 32 elements per CTA, lane = element.  First every thread forms two
// (element, point) records -- the map M from reference to spatial gradients,
// n, sigma and the coefficients, weighted -- into shared memory, component
// planes of 32 elements (no bank conflicts).  Then warp w owns rows w and 7 - w
// of the upper node-pair triangle, 9 blocks of each element in registers:
// per point it reads the record, forms its nodes' g, m, t by the constant
// reference gradients (the same for the whole warp) and adds to its blocks, so
// a block costs 2.5 shared-memory reads per point instead of 24.  One element
// per lane also keeps the warps free of divergence.
//
// Measured at 262,144 Simo elements: 0.338 ms (general kernel 0.488 ms; the
// 453 MB of element blocks alone take 0.067 ms to write), at 55,296 J2 elements
// 0.075 ms (0.137).  It is bound by instruction issue: half of the FP32 rate's
// issue slots at 12 warps an SM, 0.44 of the FMA pipe.
#include <algorithm>

#include "elements.cuh"

namespace tg {

namespace {

constexpr int kIsoElems = 32;    // elements per CTA: one per lane
constexpr int kIsoThreads = 128;
// record of a point: M[l][k] (spatial gradient k of reference direction l),
// n (6), S = B I + sigma (6), A, B, C; all but M and n weighted
constexpr int kRecM = 0, kRecN = 9, kRecS = 15, kRecA = 21, kRecB = 22, kRecC = 23, kRec = 24;

// dN_a/dxi_d at every point, [point][node]{r, s, t, 0}
struct IsoGrad {
  float4 v[8][8];
  constexpr IsoGrad() : v{} {
    for (int ip = 0; ip < 8; ++ip)
      for (int a = 0; a < 8; ++a) {
        const double fr = 1.0 + kGauss * sr(ip) * sr(a), fs = 1.0 + kGauss * ss(ip) * ss(a),
                     ft = 1.0 + kGauss * st(ip) * st(a);
        v[ip][a].x = (float)(0.125 * sr(a) * fs * ft);
        v[ip][a].y = (float)(0.125 * ss(a) * fr * ft);
        v[ip][a].z = (float)(0.125 * st(a) * fr * fs);
      }
  }
};
__constant__ IsoGrad kIsoGrad = IsoGrad();

// The 9 blocks of rows lo and 7 - lo over all points, one code path for every
// lo (a path per lo was 36 KB of loop bodies, and the warps waited for
// instructions).  FS: Simo; otherwise J2 (HAVEN) or Hookean.
template <bool FS, bool HAVEN>
__device__ __forceinline__ void iso_rows(const float* __restrict__ rec, float* __restrict__ Ke, int lo, int e,
                                         bool live) {
  using T = float;
  const int hi = 7 - lo, n0 = 8 - lo;  // blocks of row lo
  T K[9][9], G[9];                     // block values; the identity's coefficient
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    G[q] = T(0);
#pragma unroll
    for (int i = 0; i < 9; ++i) K[q][i] = T(0);
  }
#pragma unroll 1
  for (int ip = 0; ip < 8; ++ip, rec += kRec * kIsoElems) {
    T M[9], n[6], S[6];
    auto at = [&](int c) { return rec[c * kIsoElems]; };
#pragma unroll
    for (int i = 0; i < 9; ++i) M[i] = at(kRecM + i);
#pragma unroll
    for (int i = 0; i < 6; ++i) n[i] = HAVEN ? at(kRecN + i) : T(0);
#pragma unroll
    for (int i = 0; i < 6; ++i) S[i] = FS ? at(kRecS + i) : T(0);
    const T A = at(kRecA), B = at(kRecB), C = HAVEN ? at(kRecC) : T(0);
    auto grad = [&](int a, T g[3]) {
      const float4 d = kIsoGrad.v[ip][a];
#pragma unroll
      for (int k = 0; k < 3; ++k) g[k] = d.x * M[k] + d.y * M[3 + k] + d.z * M[6 + k];
    };
    auto sym = [](const T m[6], const T g[3], T o[3]) {
      o[0] = m[0] * g[0] + m[5] * g[1] + m[4] * g[2];
      o[1] = m[5] * g[0] + m[1] * g[1] + m[3] * g[2];
      o[2] = m[4] * g[0] + m[3] * g[1] + m[2] * g[2];
    };
    T ga[3], Ua[3], Va[3], Ba[3];
    auto row = [&](int a) {
      T m[3] = {T(0), T(0), T(0)};
      grad(a, ga);
      if (HAVEN) sym(n, ga, m);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        Ua[i] = A * ga[i] + (FS ? C * m[i] : T(0));
        Va[i] = FS ? ga[i] : C * m[i];
        Ba[i] = B * ga[i];
      }
    };
    row(lo);
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      if (q >= 5 && q == n0) row(hi);
      T gb[3], Wb[3] = {T(0), T(0), T(0)}, tb[3];
      grad(q < n0 ? lo + q : hi + q - n0, gb);
      if (HAVEN) {
        sym(n, gb, Wb);
        if (FS)
#pragma unroll
          for (int i = 0; i < 3; ++i) Wb[i] *= C;
      }
      if (FS) {
        sym(S, gb, tb);
      } else {
#pragma unroll
        for (int i = 0; i < 3; ++i) tb[i] = B * gb[i];
      }
      G[q] += ga[0] * tb[0] + ga[1] * tb[1] + ga[2] * tb[2];
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          K[q][i * 3 + j] += Ua[i] * gb[j];
          if (HAVEN) K[q][i * 3 + j] += Va[i] * Wb[j];
          K[q][i * 3 + j] += Ba[j] * gb[i];
        }
    }
  }
  if (!live) return;
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    const int a = q < n0 ? lo : hi, b = q < n0 ? lo + q : hi + q - n0;
    const int slot = a * 8 - a * (a - 1) / 2 + (b - a);
    float4* out = reinterpret_cast<float4*>(Ke + ((long long)e * kSlots + slot) * kKeBlock);
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      float4 r;
      r.x = K[q][p * 3 + 0] + (p == 0 ? G[q] : T(0));
      r.y = K[q][p * 3 + 1] + (p == 1 ? G[q] : T(0));
      r.z = K[q][p * 3 + 2] + (p == 2 ? G[q] : T(0));
      r.w = T(0);
      out[p] = r;
    }
  }
}

template <bool FS, bool HAVEN>
__global__ void __launch_bounds__(kIsoThreads, 3)
    tangent_iso_kernel(const double* __restrict__ X, int nnd, const int* __restrict__ conn,
                       const int8_t* __restrict__ blk, int nel, const double4_32a* __restrict__ u, MatTable mt,
                       J2View j2, float* __restrict__ Ke, int* status) {
  using T = float;
  constexpr int kPad = kIsoElems + 1;
  extern __shared__ __align__(16) unsigned char iso_dyn[];
  T* rec = reinterpret_cast<T*>(iso_dyn);           // [8 points][kRec][32 elements]
  T* sX = rec + 8 * kRec * kIsoElems;               // [8 nodes][3][33]
  T* sU = sX + 8 * 3 * kPad;
  const int tid = threadIdx.x, e0 = blockIdx.x * kIsoElems;
  for (int i = tid; i < kIsoElems * 8; i += kIsoThreads) {
    const int le = i >> 3, a = i & 7, e = min(e0 + le, nel - 1);
    const int n0 = conn[e * 8], n = conn[e * 8 + a];
    // local origin at node 0 keeps FP32 coordinate differences accurate
    sX[(a * 3 + 0) * kPad + le] = T(X[n] - X[n0]);
    sX[(a * 3 + 1) * kPad + le] = T(X[nnd + n] - X[nnd + n0]);
    sX[(a * 3 + 2) * kPad + le] = T(X[2 * nnd + n] - X[2 * nnd + n0]);
    if (FS) {
      const double4_32a un = u[n];
      sU[(a * 3 + 0) * kPad + le] = T(un.x);
      sU[(a * 3 + 1) * kPad + le] = T(un.y);
      sU[(a * 3 + 2) * kPad + le] = T(un.z);
    }
  }
  __syncthreads();
  for (int i = tid; i < kIsoElems * 8; i += kIsoThreads) {
    const int le = i & 31, ip = i >> 5, e = min(e0 + le, nel - 1);
    const MatParams& m = mt.m[blk ? blk[e] : 0];
    T J[9];
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        T acc = T(0);
#pragma unroll
        for (int a = 0; a < 8; ++a) acc += sX[(a * 3 + q) * kPad + le] * (k == 0 ? kIsoGrad.v[ip][a].x : k == 1 ? kIsoGrad.v[ip][a].y : kIsoGrad.v[ip][a].z);
        J[q * 3 + k] = acc;
      }
    const T detj = det3(J);
    T M[9], Ji[9];  // M[l*3 + k]: dN/dx_k = sum_l dN/dxi_l M[l][k]
    inv3(J, detj, Ji);
    T n6[6] = {T(0), T(0), T(0), T(0), T(0), T(0)}, S6[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
    T A = T(0), B = T(0), C = T(0);
    bool okm = detj > T(0);
    if (FS) {
      T F[9];
#pragma unroll
      for (int q = 0; q < 9; ++q) F[q] = (q % 4) == 0 ? T(1) : T(0);
#pragma unroll
      for (int a = 0; a < 8; ++a) {
        T g[3];
#pragma unroll
        for (int k = 0; k < 3; ++k)
          g[k] = Ji[k] * kIsoGrad.v[ip][a].x + Ji[3 + k] * kIsoGrad.v[ip][a].y + Ji[6 + k] * kIsoGrad.v[ip][a].z;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const T uq = sU[(a * 3 + q) * kPad + le];
#pragma unroll
          for (int k = 0; k < 3; ++k) F[q * 3 + k] += uq * g[k];
        }
      }
      const T Jd = det3(F);
      T b[6];
      b[0] = F[0] * F[0] + F[1] * F[1] + F[2] * F[2];
      b[1] = F[3] * F[3] + F[4] * F[4] + F[5] * F[5];
      b[2] = F[6] * F[6] + F[7] * F[7] + F[8] * F[8];
      b[3] = F[3] * F[6] + F[4] * F[7] + F[5] * F[8];
      b[4] = F[0] * F[6] + F[1] * F[7] + F[2] * F[8];
      b[5] = F[0] * F[3] + F[1] * F[4] + F[2] * F[5];
      const T detb = b[0] * (b[1] * b[2] - b[3] * b[3]) - b[5] * (b[5] * b[2] - b[3] * b[4]) +
                     b[4] * (b[5] * b[3] - b[1] * b[4]);
      okm = okm && Jd > T(0) && detb > T(0);
      T Js, invJ, sc;
      simo_roots(okm ? detb : T(1), Js, invJ, sc);
      T bb[6];
#pragma unroll
      for (int q = 0; q < 6; ++q) bb[q] = sc * b[q];
      deviatoric(bb, n6);
      const T mu = T(m.mu), kappa = T(m.kappa), w = detj * Jd;
      const T dU = T(0.5) * kappa * (Js - invJ), ddU = T(0.5) * kappa * (T(1) + invJ * invJ);
      const T muJ = mu * invJ, mubar = muJ * (bb[0] + bb[1] + bb[2]) * T(1.0 / 3.0);
      A = w * (dU + Js * ddU - T(2.0 / 3.0) * mubar);
      B = w * (mubar - dU);
      C = w * T(-2.0 / 3.0) * muJ;
#pragma unroll
      for (int q = 0; q < 6; ++q) S6[q] = w * (muJ * n6[q] + (q < 3 ? dU : T(0))) + (q < 3 ? B : T(0));
      T Fi[9];
      inv3(F, Jd, Fi);
#pragma unroll
      for (int l = 0; l < 3; ++l)
#pragma unroll
        for (int k = 0; k < 3; ++k)
          M[l * 3 + k] = Ji[l * 3 + 0] * Fi[0 * 3 + k] + Ji[l * 3 + 1] * Fi[1 * 3 + k] + Ji[l * 3 + 2] * Fi[2 * 3 + k];
    } else {
#pragma unroll
      for (int q = 0; q < 9; ++q) M[q] = Ji[q];
      const T mu = T(m.C[21]), lambda = T(m.C[1]);
      A = detj * lambda;
      B = detj * mu;
      if (HAVEN && m.kind == TG_MAT_SS_J2) {
        const long long gid = (long long)e * 8 + ip;
        if (j2.alloc[e] != 0 && j2.flags[gid] == TG_J2_PLASTIC) {
          const T th = T(2.0 * m.mu * j2.dgamma[gid] / j2.norm[gid]);
          const T tb = T(3.0 / (3.0 + m.hard_a / m.mu)) - th;
          A += detj * (T(2.0 / 3.0) * mu * th);
          B -= detj * mu * th;
          C = detj * T(-2) * mu * tb;
#pragma unroll
          for (int q = 0; q < 6; ++q) n6[q] = T(j2.nhat[q * j2.nip + gid]);
        }
      }
    }
    if (!okm) {
      if (e0 + le < nel) atomicOr(status, kStatusBadJacobian);
      A = B = C = T(0);
#pragma unroll
      for (int q = 0; q < 9; ++q) M[q] = T(0);
#pragma unroll
      for (int q = 0; q < 6; ++q) n6[q] = S6[q] = T(0);
    }
    T* o = rec + (ip * kRec) * kIsoElems + le;
#pragma unroll
    for (int q = 0; q < 9; ++q) o[(kRecM + q) * kIsoElems] = M[q];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      if (HAVEN) o[(kRecN + q) * kIsoElems] = n6[q];
      if (FS) o[(kRecS + q) * kIsoElems] = S6[q];
    }
    o[kRecA * kIsoElems] = A;
    o[kRecB * kIsoElems] = B;
    if (HAVEN) o[kRecC * kIsoElems] = C;
  }
  __syncthreads();
  const int lane = tid & 31, e = e0 + lane;
  const bool live = e < nel;
  iso_rows<FS, HAVEN>(rec + lane, Ke, tid >> 5, e, live);
}

template <bool FS, bool HAVEN>
int launch_t(Context* c, float* Ke, const J2View& j2) {
  const size_t dyn = sizeof(float) * (8 * kRec * kIsoElems + 2 * 8 * 3 * (kIsoElems + 1));
  if (!ok(c, cudaFuncSetAttribute(tangent_iso_kernel<FS, HAVEN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn),
          "smem attribute"))
    return TG_ERR_CUDA;
  tangent_iso_kernel<FS, HAVEN><<<(c->nel + kIsoElems - 1) / kIsoElems, kIsoThreads, dyn, c->stream>>>(
      c->d_X, c->nnd, c->d_conn, c->d_block, c->nel, c->d_u, c->mats, j2, Ke, c->d_status);
  c->launches++;
  return ok(c, cudaGetLastError(), "tangent_iso_kernel") ? TG_OK : TG_ERR_CUDA;
}

int launch_form(Context* c, float* Ke) {
  J2View j2;
  j2.flags = c->d_j2_flags;
  j2.alloc = c->d_j2_alloc;
  j2.alpha = c->d_j2_alpha;
  j2.dgamma = c->d_j2_dgamma;
  j2.norm = c->d_j2_norm;
  j2.epsp = c->d_j2_epsp;
  j2.nhat = c->d_j2_nhat;
  j2.nip = (long long)c->nel * 8;
  if (c->mats.formulation == TG_TOTAL_LAGRANGIAN) return launch_t<true, true>(c, Ke, j2);
  return c->has_j2 ? launch_t<false, true>(c, Ke, j2) : launch_t<false, false>(c, Ke, j2);
}

}  // namespace

// Total-Lagrangian Simo groups and small-strain groups of isotropic Hookean
// and J2 blocks without B-bar.  The others (B-bar's mean gradients, the updated
// configuration, anisotropic moduli) keep the general kernel; St.Venant groups
// and FP64: tangent_blocks.cu.
bool tangent_iso_applies(const Context* c, int precision) {
  if (precision != TG_MIXED || c->nel <= 0) return false;
  const int nb = c->have_blocks ? c->mats.nblocks : 1;
  const bool fs = c->mats.formulation == TG_TOTAL_LAGRANGIAN;
  if (!fs && (c->mats.formulation != TG_SMALL_STRAIN || c->mats.bbar)) return false;
  for (int b = 0; b < nb; ++b) {
    const MatParams& m = c->mats.m[b];
    if (fs ? m.kind != TG_MAT_FS_SIMO
           : !((m.kind == TG_MAT_SS_HOOKEAN || m.kind == TG_MAT_SS_J2) && isotropic_moduli(m)))
      return false;
  }
  return true;
}

int launch_tangent_iso(Context* c) { return launch_form(c, c->d_Ke32); }

}  // namespace tg
