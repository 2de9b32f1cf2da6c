// Element tangents by node-pair blocks from per-node vectors, sm_103a: FP64 for
// the materials of tangent_iso.cu, and St.Venant groups in both precisions.
//
// For isotropic moduli the 3x3 block of nodes a and b at a point is a sum of
// products of node vectors (SolidElementT::FormStiffness with SimoIso3D::c_ijkl,
// SimoIso3D.cpp:16-53,102-135, HookeanMatT.cpp:103, J2SSC0HardeningT::
// ModuliCorrection, J2SSC0HardeningT.cpp:148-176, FDHookeanMatT with FDKStV;
// SmallStrainT.cpp:285, TotalLagrangianT.cpp:40), with g = grad N:
//   Simo      (A g_a + C n g_a) (x) g_b + g_a (x) (C n g_b) + B g_b (x) g_a
//             + (g_a . (B g_b + sigma g_b)) I
//   Hooke, J2 A g_a (x) g_b + C (n g_a) (x) (n g_b) + B g_b (x) g_a + B (g_a . g_b) I
//   St.Venant lambda p_a (x) p_b + mu p_b (x) p_a + mu (g_a . g_b) F F^T
//             + (g_a . S g_b) I, with G = dN/dX for g and p = F G
// The general kernel (elements.cu) takes 85 operations a block and point, and
// for St.Venant pushes the moduli forward first, 5,000 a point by 64 of its 288
// threads: in FP64, at a warp instruction per 64 cycles and scheduler, that is
// the whole time.  Here a block and point takes 30 to 36.
//
// A CTA of 288 threads holds 8 elements: 64 threads form the points' records,
// all form the nodes' vectors, and a thread integrates one of the 36 upper
// blocks of an element over its 8 points.  (FP32 of the other materials:
// tangent_iso.cu, whose lanes keep nine blocks each; FP64 has no use for that,
// the shared-memory reads of a block are a tenth of its arithmetic.)
//
// Measured, general kernel / this one: FP64 2,926 St.Venant elements 604 / 129
// us, 59,400 Simo 2,812 / 1,927, 4,096 Hooke 170 / 148; FP32 2,926 St.Venant
// 53 / 16.  Bound by the FP64 pipe (in FP32 by its latency).
#include <type_traits>

#include "elements.cuh"

namespace tg {

namespace {

constexpr int kBlkElems = 8;
constexpr int kBlkThreads = kBlkElems * kSlots;
constexpr int kNodeVec = 13;   // 12 values of a node at a point, padded
constexpr int kPointRec = 33;  // 32 values of a point, padded
enum : int { kBlkSimo = 0, kBlkSmall = 1, kBlkStVenant = 2 };

// dN_a/dxi_d at every point
template <typename T>
struct BlkGrad {
  T v[8][8][3];
  constexpr BlkGrad() : v{} {
    for (int ip = 0; ip < 8; ++ip)
      for (int a = 0; a < 8; ++a) {
        const double fr = 1.0 + kGauss * sr(ip) * sr(a), fs = 1.0 + kGauss * ss(ip) * ss(a),
                     ft = 1.0 + kGauss * st(ip) * st(a);
        v[ip][a][0] = (T)(0.125 * sr(a) * fs * ft);
        v[ip][a][1] = (T)(0.125 * ss(a) * fr * ft);
        v[ip][a][2] = (T)(0.125 * st(a) * fr * fs);
      }
  }
};
__constant__ BlkGrad<float> kBlkGrad32 = BlkGrad<float>();
__constant__ BlkGrad<double> kBlkGrad64 = BlkGrad<double>();
template <typename T>
__device__ __forceinline__ const T* blk_grad(int ip, int a) {
  if constexpr (sizeof(T) == 4)
    return kBlkGrad32.v[ip][a];
  else
    return kBlkGrad64.v[ip][a];
}

template <typename T>
__device__ __forceinline__ void sym_apply(const T m[6], const T g[3], T o[3]) {
  o[0] = m[0] * g[0] + m[5] * g[1] + m[4] * g[2];
  o[1] = m[5] * g[0] + m[1] * g[1] + m[3] * g[2];
  o[2] = m[4] * g[0] + m[3] * g[1] + m[2] * g[2];
}

// Record of a point.  Map M[l][k] from reference-domain to the gradients g (9),
// then Simo: C n (6), sigma (6), A, B; small strain: n (6), A, B, C; St.Venant:
// F (9), S (6), F F^T (6), lambda, mu; all but M, F and n weighted.
template <typename T, int MODE>
__device__ __forceinline__ bool point_record(const T (*Xe)[3], const T (*Ue)[3], int ip, const MatParams& m,
                                             const J2View& j2, long long e, T* o) {
  T J[9], Ji[9];
#pragma unroll
  for (int q = 0; q < 9; ++q) J[q] = T(0);
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    const T* d = blk_grad<T>(ip, a);
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int k = 0; k < 3; ++k) J[q * 3 + k] += Xe[a][q] * d[k];
  }
  const T w0 = det3(J);
  if (!(w0 > T(0))) return false;
  inv3(J, w0, Ji);
  if (MODE == kBlkSmall) {
    const T mu = T(m.C[21]), lambda = T(m.C[1]);
    T A = w0 * lambda, B = w0 * mu, C = T(0);
#pragma unroll
    for (int q = 0; q < 9; ++q) o[q] = Ji[q];
#pragma unroll
    for (int q = 0; q < 6; ++q) o[9 + q] = T(0);
    const long long gid = e * 8 + ip;
    if (m.kind == TG_MAT_SS_J2 && j2.alloc[e] != 0 && j2.flags[gid] == TG_J2_PLASTIC) {
      const T th = T(2.0 * m.mu * j2.dgamma[gid] / j2.norm[gid]);
      const T tb = T(3.0 / (3.0 + m.hard_a / m.mu)) - th;
      A += w0 * (T(2.0 / 3.0) * mu * th);
      B -= w0 * mu * th;
      C = w0 * T(-2) * mu * tb;
#pragma unroll
      for (int q = 0; q < 6; ++q) o[9 + q] = T(j2.nhat[q * j2.nip + gid]);
    }
    o[15] = A;
    o[16] = B;
    o[17] = C;
    return true;
  }
  T R[9], F[9];
#pragma unroll
  for (int q = 0; q < 9; ++q) R[q] = T(0);
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    const T* d = blk_grad<T>(ip, a);
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int k = 0; k < 3; ++k) R[q * 3 + k] += Ue[a][q] * d[k];
  }
#pragma unroll
  for (int q = 0; q < 3; ++q)
#pragma unroll
    for (int k = 0; k < 3; ++k)
      F[q * 3 + k] = (q == k ? T(1) : T(0)) + R[q * 3] * Ji[k] + R[q * 3 + 1] * Ji[3 + k] + R[q * 3 + 2] * Ji[6 + k];
  const T Jd = det3(F);
  if (!(Jd > T(0))) return false;
  T b[6];
  b[0] = F[0] * F[0] + F[1] * F[1] + F[2] * F[2];
  b[1] = F[3] * F[3] + F[4] * F[4] + F[5] * F[5];
  b[2] = F[6] * F[6] + F[7] * F[7] + F[8] * F[8];
  b[3] = F[3] * F[6] + F[4] * F[7] + F[5] * F[8];
  b[4] = F[0] * F[6] + F[1] * F[7] + F[2] * F[8];
  b[5] = F[0] * F[3] + F[1] * F[4] + F[2] * F[5];
  if (MODE == kBlkStVenant) {
    const T lambda = T(m.C[1]), mu = T(m.C[21]);
    // S = lambda tr(E) I + 2 mu E, E = (F^T F - I)/2
    const T c0 = F[0] * F[0] + F[3] * F[3] + F[6] * F[6], c1 = F[1] * F[1] + F[4] * F[4] + F[7] * F[7],
            c2 = F[2] * F[2] + F[5] * F[5] + F[8] * F[8], c3 = F[1] * F[2] + F[4] * F[5] + F[7] * F[8],
            c4 = F[0] * F[2] + F[3] * F[5] + F[6] * F[8], c5 = F[0] * F[1] + F[3] * F[4] + F[6] * F[7];
    const T e0 = c0 - T(1), e1 = c1 - T(1), e2 = c2 - T(1), p = T(0.5) * lambda * (e0 + e1 + e2);
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      o[q] = Ji[q];
      o[9 + q] = F[q];
    }
    o[18] = w0 * (p + mu * e0);
    o[19] = w0 * (p + mu * e1);
    o[20] = w0 * (p + mu * e2);
    o[21] = w0 * mu * c3;
    o[22] = w0 * mu * c4;
    o[23] = w0 * mu * c5;
#pragma unroll
    for (int q = 0; q < 6; ++q) o[24 + q] = w0 * mu * b[q];
    o[30] = w0 * lambda;
    o[31] = w0 * mu;
    return true;
  }
  const T detb = b[0] * (b[1] * b[2] - b[3] * b[3]) - b[5] * (b[5] * b[2] - b[3] * b[4]) +
                 b[4] * (b[5] * b[3] - b[1] * b[4]);
  if (!(detb > T(0))) return false;
  T Js, invJ, sc;
  simo_roots(detb, Js, invJ, sc);
  T bb[6], n6[6];
#pragma unroll
  for (int q = 0; q < 6; ++q) bb[q] = sc * b[q];
  deviatoric(bb, n6);
  const T mu = T(m.mu), kappa = T(m.kappa), w = w0 * Jd;
  const T dU = T(0.5) * kappa * (Js - invJ), ddU = T(0.5) * kappa * (T(1) + invJ * invJ);
  const T muJ = mu * invJ, mubar = muJ * (bb[0] + bb[1] + bb[2]) * T(1.0 / 3.0), C = w * T(-2.0 / 3.0) * muJ;
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    o[9 + q] = C * n6[q];
    o[15 + q] = w * (muJ * n6[q] + (q < 3 ? dU : T(0)));
  }
  o[21] = w * (dU + Js * ddU - T(2.0 / 3.0) * mubar);
  o[22] = w * (mubar - dU);
  T Fi[9];
  inv3(F, Jd, Fi);
#pragma unroll
  for (int l = 0; l < 3; ++l)
#pragma unroll
    for (int k = 0; k < 3; ++k) o[l * 3 + k] = Ji[l * 3] * Fi[k] + Ji[l * 3 + 1] * Fi[3 + k] + Ji[l * 3 + 2] * Fi[6 + k];
  return true;
}

template <typename T, int MODE>
__global__ void __launch_bounds__(kBlkThreads, 2)
    tangent_blocks_kernel(const double* __restrict__ X, int nnd, const int* __restrict__ conn,
                          const int8_t* __restrict__ blk, int nel, const double4_32a* __restrict__ u, MatTable mt,
                          J2View j2, T* __restrict__ Ke, int* status) {
  extern __shared__ __align__(16) unsigned char blk_dyn[];
  __shared__ T sX[kBlkElems][8][3], sU[kBlkElems][8][3];
  T* rec = reinterpret_cast<T*>(blk_dyn);            // [64 points][kPointRec]
  T* vec = rec + kBlkElems * 8 * kPointRec;          // [64 points][8 nodes][kNodeVec]
  const int tid = threadIdx.x, e0 = blockIdx.x * kBlkElems;
  if (tid < kBlkElems * 8) {
    const int le = tid >> 3, a = tid & 7, e = min(e0 + le, nel - 1);
    const int n0 = conn[(long long)e * 8], n = conn[(long long)e * 8 + a];
    // local origin at node 0 keeps FP32 coordinate differences accurate
#pragma unroll
    for (int k = 0; k < 3; ++k) sX[le][a][k] = T(X[(long long)k * nnd + n] - X[(long long)k * nnd + n0]);
    const double4_32a un = u[n];
    sU[le][a][0] = T(un.x);
    sU[le][a][1] = T(un.y);
    sU[le][a][2] = T(un.z);
  }
  __syncthreads();
  if (tid < kBlkElems * 8) {
    const int le = tid >> 3, e = min(e0 + le, nel - 1);
    T* o = rec + tid * kPointRec;
    if (!point_record<T, MODE>(sX[le], sU[le], tid & 7, mt.m[blk ? blk[e] : 0], j2, e, o)) {
      if (e0 + le < nel) atomicOr(status, kStatusBadJacobian);
      for (int q = 0; q < kPointRec; ++q) o[q] = T(0);
    }
  }
  __syncthreads();
  // the nodes' vectors: g; then Simo A g + C n g, C n g, B g + sigma g; small
  // strain A g, n g, B g; St.Venant p, S g
  for (int i = tid; i < kBlkElems * 64; i += kBlkThreads) {
    const T* o = rec + (i >> 3) * kPointRec;
    const T* d = blk_grad<T>((i >> 3) & 7, i & 7);
    T* v = vec + i * kNodeVec;
    T g[3], h[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] = g[k] = d[0] * o[k] + d[1] * o[3 + k] + d[2] * o[6 + k];
    if (MODE == kBlkStVenant) {
#pragma unroll
      for (int k = 0; k < 3; ++k) v[3 + k] = o[9 + 3 * k] * g[0] + o[10 + 3 * k] * g[1] + o[11 + 3 * k] * g[2];
      sym_apply(o + 18, g, h);
#pragma unroll
      for (int k = 0; k < 3; ++k) v[6 + k] = h[k];
    } else {
      const T A = o[MODE == kBlkSimo ? 21 : 15], B = o[MODE == kBlkSimo ? 22 : 16];
      sym_apply(o + 9, g, h);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        v[3 + k] = A * g[k] + (MODE == kBlkSimo ? h[k] : T(0));
        v[6 + k] = h[k];
      }
      if (MODE == kBlkSimo) sym_apply(o + 15, g, h);
#pragma unroll
      for (int k = 0; k < 3; ++k) v[9 + k] = B * g[k] + (MODE == kBlkSimo ? h[k] : T(0));
    }
  }
  __syncthreads();
  const int le = tid / kSlots, slot = tid % kSlots;
  if (e0 + le >= nel) return;
  int a = 0, b = slot;
  while (b >= 8 - a) b -= 8 - a++;
  b += a;
  T K[9], G = T(0);
#pragma unroll
  for (int q = 0; q < 9; ++q) K[q] = T(0);
#pragma unroll 2
  for (int ip = 0; ip < 8; ++ip) {
    const T* o = rec + (le * 8 + ip) * kPointRec;
    const T* va = vec + ((le * 8 + ip) * 8 + a) * kNodeVec;
    const T* vb = vec + ((le * 8 + ip) * 8 + b) * kNodeVec;
    if (MODE == kBlkStVenant) {
      const T gg = va[0] * vb[0] + va[1] * vb[1] + va[2] * vb[2], lambda = o[30], mu = o[31];
      G += va[0] * vb[6] + va[1] * vb[7] + va[2] * vb[8];
      const T bb[9] = {o[24], o[29], o[28], o[29], o[25], o[27], o[28], o[27], o[26]};
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const T pl = lambda * va[3 + i], pm = mu * vb[3 + i];
#pragma unroll
        for (int j = 0; j < 3; ++j) K[i * 3 + j] += pl * vb[3 + j] + pm * va[3 + j] + gg * bb[i * 3 + j];
      }
    } else {
      const T B = o[MODE == kBlkSimo ? 22 : 16], C = MODE == kBlkSimo ? T(1) : o[17];
      G += va[0] * vb[9] + va[1] * vb[10] + va[2] * vb[11];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const T ua = va[3 + i], wa = MODE == kBlkSimo ? va[i] : C * va[6 + i], gb = B * vb[i];
#pragma unroll
        for (int j = 0; j < 3; ++j) K[i * 3 + j] += ua * vb[j] + wa * vb[6 + j] + gb * va[j];
      }
    }
  }
  using V4 = typename std::conditional<sizeof(T) == 4, float4, double4_32a>::type;
  V4* out = reinterpret_cast<V4*>(Ke + ((long long)(e0 + le) * kSlots + slot) * kKeBlock);
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    V4 row;
    row.x = K[p * 3 + 0] + (p == 0 ? G : T(0));
    row.y = K[p * 3 + 1] + (p == 1 ? G : T(0));
    row.z = K[p * 3 + 2] + (p == 2 ? G : T(0));
    row.w = T(0);
    out[p] = row;
  }
}

template <typename T, int MODE>
int launch_t(Context* c, T* Ke) {
  const size_t dyn = sizeof(T) * (kBlkElems * 8 * kPointRec + kBlkElems * 64 * kNodeVec);
  if (!ok(c, cudaFuncSetAttribute(tangent_blocks_kernel<T, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn),
          "smem attribute"))
    return TG_ERR_CUDA;
  J2View j2;
  j2.flags = c->d_j2_flags;
  j2.alloc = c->d_j2_alloc;
  j2.alpha = c->d_j2_alpha;
  j2.dgamma = c->d_j2_dgamma;
  j2.norm = c->d_j2_norm;
  j2.epsp = c->d_j2_epsp;
  j2.nhat = c->d_j2_nhat;
  j2.nip = (long long)c->nel * 8;
  tangent_blocks_kernel<T, MODE><<<(c->nel + kBlkElems - 1) / kBlkElems, kBlkThreads, dyn, c->stream>>>(
      c->d_X, c->nnd, c->d_conn, c->d_block, c->nel, c->d_u, c->mats, j2, Ke, c->d_status);
  c->launches++;
  return ok(c, cudaGetLastError(), "tangent_blocks_kernel") ? TG_OK : TG_ERR_CUDA;
}

// 0 to 2: the kernel's form for the group, -1: none
int block_form(const Context* c) {
  const int nb = c->have_blocks ? c->mats.nblocks : 1;
  if (c->nel <= 0) return -1;
  auto all = [&](auto pred) {
    for (int b = 0; b < nb; ++b)
      if (!pred(c->mats.m[b])) return false;
    return true;
  };
  if (c->mats.formulation == TG_TOTAL_LAGRANGIAN) {
    if (all([](const MatParams& m) { return m.kind == TG_MAT_FS_SIMO; })) return kBlkSimo;
    if (all([](const MatParams& m) { return m.kind == TG_MAT_FS_STVENANT && isotropic_moduli(m); })) return kBlkStVenant;
    return -1;
  }
  if (c->mats.formulation != TG_SMALL_STRAIN || c->mats.bbar) return -1;
  return all([](const MatParams& m) {
    return (m.kind == TG_MAT_SS_HOOKEAN || m.kind == TG_MAT_SS_J2) && isotropic_moduli(m);
  })
             ? kBlkSmall
             : -1;
}

}  // namespace

bool tangent_blocks_applies(const Context* c, int precision) {
  const int form = block_form(c);
  return form == kBlkStVenant || (form >= 0 && precision == TG_FP64);
}

int launch_tangent_blocks(Context* c, int precision) {
  if (precision == TG_MIXED) return launch_t<float, kBlkStVenant>(c, c->d_Ke32);
  switch (block_form(c)) {
    case kBlkSimo: return launch_t<double, kBlkSimo>(c, c->d_Ke64);
    case kBlkSmall: return launch_t<double, kBlkSmall>(c, c->d_Ke64);
    default: return launch_t<double, kBlkStVenant>(c, c->d_Ke64);
  }
}

}  // namespace tg
