// Per-RVE (segmented) reductions for batched FE^2 micro-solves.
//
// A batch of independent RVEs is uploaded as one disconnected mesh; RVE r owns
// nodes [node_off[r], node_off[r+1]) and elements [elem_off[r], elem_off[r+1]).
// Their ranges are reduced in shares of a fixed size, a fixed order (no atomics):
//  * segment_norms_kernel: ||R_r||^2 of the residual restricted to the RVE;
//  * segment_stress_kernel: sum over the RVE's element nodes of fint (x) X,
//    which is the integral of the first Piola stress over the RVE (the
//    element-level identity sum_a f_a (x) X_a = int P dV), i.e. V0 times the
//    volume-averaged P; at equilibrium it equals the reaction sum
//    sum_{boundary a} f_a (x) X_a of the macro-stress definition.
#include "tg_internal.h"

namespace tg {

namespace {

template <int NV>
__device__ __forceinline__ void cta_sum(double (&v)[NV]) {
  __shared__ double sh[NV][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < NV; ++k)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) sh[k][w] = v[k];
  __syncthreads();
  if (w == 0) {
    const int nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      double x = lane < nw ? sh[k][lane] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      v[k] = x;
    }
  }
  __syncthreads();
}

// The ranges of the segments cut into shares of kShare entries, one CTA per
// share: segment sg's shares are numbered from off[sg] / kShare + sg on, so
// they depend on nothing but the offsets (a segment's sum has the same shares
// in every batch).  The last share of a block number past its segment's end is
// empty.  FP64 sums run at 2 lanes per cycle and SM here: one CTA per segment
// took 0.5 ms for the stress of an RVE of side 24.
template <int kShare>
__device__ __forceinline__ bool share_of(int b, int nseg, const int* __restrict__ off, int& sg, int& e0, int& e1) {
  int lo = 0, hi = nseg;  // the last segment whose first share is at most b
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (off[mid] / kShare + mid <= b)
      lo = mid;
    else
      hi = mid;
  }
  sg = lo;
  e0 = off[lo] + (b - (off[lo] / kShare + lo)) * kShare;
  e1 = min(off[lo + 1], e0 + kShare);
  return e0 < e1;
}
inline int share_blocks(int total, int nseg, int share) { return total / share + nseg; }

// out[sg][v] = the sum of its shares' partials in order
template <int NV, int kShare>
__global__ void segment_combine_kernel(int nseg, const int* __restrict__ off, const double* __restrict__ part,
                                       double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nseg * NV) return;
  const int sg = i / NV, v = i % NV;
  const int b0 = off[sg] / kShare + sg, n = (off[sg + 1] - off[sg] + kShare - 1) / kShare;
  double a = 0.0;
  for (int b = 0; b < n; ++b) a += part[(long long)(b0 + b) * NV + v];
  out[i] = a;
}

constexpr int kNormShare = 2048;   // nodes
constexpr int kStressShare = 256;  // elements
constexpr int kMacroShare = 64;    // elements

__global__ void __launch_bounds__(256) segment_norms_kernel(int nseg, const int* __restrict__ off,
                                                            const double4_32a* __restrict__ R,
                                                            double* __restrict__ part) {
  int sg, n0, n1;
  if (!share_of<kNormShare>(blockIdx.x, nseg, off, sg, n0, n1)) return;
  double v[1] = {0.0};
  for (int n = n0 + threadIdx.x; n < n1; n += blockDim.x) {
    const double4_32a r = R[n];
    v[0] += r.x * r.x + r.y * r.y + r.z * r.z;
  }
  cta_sum<1>(v);
  if (threadIdx.x == 0) part[blockIdx.x] = v[0];
}

__global__ void __launch_bounds__(256) segment_stress_kernel(int nseg, const int* __restrict__ eoff,
                                                             const int* __restrict__ conn, const double* __restrict__ X,
                                                             int nnd, const double4_32a* __restrict__ fint,
                                                             double* __restrict__ part) {
  int sg, e0, e1;
  if (!share_of<kStressShare>(blockIdx.x, nseg, eoff, sg, e0, e1)) return;
  double v[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  const long long k1 = (long long)e1 * 8;
  for (long long k = (long long)e0 * 8 + threadIdx.x; k < k1; k += blockDim.x) {
    const int n = conn[k];
    const double4_32a f = fint[k];
    const double Xn[3] = {X[n], X[nnd + n], X[2 * nnd + n]};
#pragma unroll
    for (int J = 0; J < 3; ++J) {
      v[0 * 3 + J] += f.x * Xn[J];
      v[1 * 3 + J] += f.y * Xn[J];
      v[2 * 3 + J] += f.z * Xn[J];
    }
  }
  cta_sum<9>(v);
  if (threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < 9; ++k) part[(long long)blockIdx.x * 9 + k] = v[k];
}

// v = (e_k (x) e_L) X on prescribed dofs, zero elsewhere: the boundary
// displacement of a unit perturbation dF = e_k (x) e_L of the macro gradient.
__global__ void macro_perturb_kernel(int nnd, const uint8_t* __restrict__ mask, const double* __restrict__ X, int k,
                                     int L, double4_32a* __restrict__ v) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= nnd) return;
  const int m = mask[n];
  const double xl = X[(long long)L * nnd + n];
  v[n] = make_double4_32a((k == 0 && !(m & 1)) ? xl : 0.0, (k == 1 && !(m & 2)) ? xl : 0.0,
                          (k == 2 && !(m & 4)) ? xl : 0.0, 0.0);
}

// w = v + unscale * x (x: the PCG solution on the free dofs, zero elsewhere)
template <typename V>
__global__ void macro_combine_kernel(int nnd, const double4_32a* __restrict__ v, const V* __restrict__ x,
                                     const PcgScalars* __restrict__ sc, double4_32a* __restrict__ w) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= nnd) return;
  const double us = sc->unscale;
  const double4_32a a = v[n];
  const V b = x[n];
  w[n] = make_double4_32a(a.x + us * (double)b.x, a.y + us * (double)b.y, a.z + us * (double)b.z, 0.0);
}

__device__ __forceinline__ int upper_slot_of(int a, int b) { return a * 8 - a * (a - 1) / 2 + (b - a); }

// Column kL of every RVE's macro tangent: sum over the RVE's element nodes of
// (K_e w_e)_a (x) X_a, from the staged element matrices (36 upper node-pair
// blocks; lower blocks by symmetry).  Partials of a share of kMacroShare
// elements: a CTA per RVE and column left the chip waiting for the largest
// RVEs (48 RVEs of sides 4 to 12 in FP64: 1.50 ms, in shares 0.52).
template <typename T>
__global__ void __launch_bounds__(256) segment_macro_kernel(int nseg, const int* __restrict__ eoff,
                                                            const int* __restrict__ conn, const double* __restrict__ X,
                                                            int nnd, const T* __restrict__ Ke,
                                                            const double4_32a* __restrict__ w_all,
                                                            double* __restrict__ part) {
  // grid rows (blockIdx.y) are the columns, each with its own w
  const double4_32a* __restrict__ w = w_all + (long long)blockIdx.y * nnd;
  int sg, e0, e1;
  if (!share_of<kMacroShare>(blockIdx.x, nseg, eoff, sg, e0, e1)) return;
  {
    double v[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    const long long k1 = (long long)e1 * 8;
    for (long long k = (long long)e0 * 8 + threadIdx.x; k < k1; k += blockDim.x) {
      const long long e = k >> 3;
      const int a = (int)(k & 7);
      const int* ce = conn + e * 8;
      const T* Kb = Ke + e * kKeStride;
      double y0 = 0.0, y1 = 0.0, y2 = 0.0;
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const double4_32a wb = w[ce[b]];
        // the block or its transpose, chosen before the arithmetic: a warp
        // pays the FP64 pipe for either branch
        const bool up = a <= b;
        const T* B = Kb + (up ? upper_slot_of(a, b) : upper_slot_of(b, a)) * kKeBlock;
        const T m00 = B[0], m11 = B[5], m22 = B[10], m01 = B[up ? 1 : 4], m02 = B[up ? 2 : 8], m10 = B[up ? 4 : 1],
                m12 = B[up ? 6 : 9], m20 = B[up ? 8 : 2], m21 = B[up ? 9 : 6];
        y0 += (double)m00 * wb.x + (double)m01 * wb.y + (double)m02 * wb.z;
        y1 += (double)m10 * wb.x + (double)m11 * wb.y + (double)m12 * wb.z;
        y2 += (double)m20 * wb.x + (double)m21 * wb.y + (double)m22 * wb.z;
      }
      const int n = ce[a];
      const double Xn[3] = {X[n], X[nnd + n], X[2 * nnd + n]};
#pragma unroll
      for (int J = 0; J < 3; ++J) {
        v[0 * 3 + J] += y0 * Xn[J];
        v[1 * 3 + J] += y1 * Xn[J];
        v[2 * 3 + J] += y2 * Xn[J];
      }
    }
    cta_sum<9>(v);
    if (threadIdx.x == 0)
#pragma unroll
      for (int jJ = 0; jJ < 9; ++jJ) part[((long long)blockIdx.x * gridDim.y + blockIdx.y) * 9 + jJ] = v[jJ];
  }
}

// out[sg*81 + jJ*9 + kL0 + column]: the sum of the shares' partials in order
__global__ void segment_macro_combine_kernel(int nseg, const int* __restrict__ off, int ncols,
                                             const double* __restrict__ part, int kL0,
                                             const double* __restrict__ vol0, double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nseg * ncols * 9) return;
  const int sg = i / (ncols * 9), v = i % (ncols * 9), col = v / 9, jJ = v % 9;
  const int b0 = off[sg] / kMacroShare + sg, n = (off[sg + 1] - off[sg] + kMacroShare - 1) / kMacroShare;
  double a = 0.0;
  for (int b = 0; b < n; ++b) a += part[(long long)(b0 + b) * (ncols * 9) + v];
  out[(long long)sg * 81 + jJ * 9 + kL0 + col] = a * (vol0 ? 1.0 / vol0[sg] : 1.0);
}

}  // namespace

int launch_macro_perturb(Context* c, int k, int L, double4_32a* d_v) {
  macro_perturb_kernel<<<(c->nnd + 255) / 256, 256, 0, c->stream>>>(c->nnd, c->d_mask, c->d_X, k, L, d_v);
  c->launches++;
  return ok(c, cudaGetLastError(), "macro_perturb_kernel") ? TG_OK : TG_ERR_CUDA;
}

int launch_macro_combine(Context* c, const double4_32a* d_v, double4_32a* d_w) {
  const int grid = (c->nnd + 255) / 256;
  if (c->pcg_vec_precision == TG_MIXED)
    macro_combine_kernel<float4><<<grid, 256, 0, c->stream>>>(c->nnd, d_v, (const float4*)c->d_x, c->d_pcg, d_w);
  else
    macro_combine_kernel<double4_32a><<<grid, 256, 0, c->stream>>>(c->nnd, d_v, (const double4_32a*)c->d_x, c->d_pcg,
                                                                    d_w);
  c->launches++;
  return ok(c, cudaGetLastError(), "macro_combine_kernel") ? TG_OK : TG_ERR_CUDA;
}

int launch_segment_macro(Context* c, const double4_32a* d_w, int kL, int ncols, const double* d_vol0,
                         double* d_out) {
  const int nb = share_blocks(c->nel, c->nseg, kMacroShare);
  const dim3 grid(nb, ncols);
  double* part = nullptr;
  if (!ok(c, cudaMallocAsync((void**)&part, sizeof(double) * 9 * nb * ncols, c->stream), "alloc")) return TG_ERR_OOM;
  if (c->tangent_precision == TG_MIXED)
    segment_macro_kernel<float><<<grid, 256, 0, c->stream>>>(c->nseg, c->d_seg_elem, c->d_conn, c->d_X, c->nnd,
                                                             c->d_Ke32, d_w, part);
  else
    segment_macro_kernel<double><<<grid, 256, 0, c->stream>>>(c->nseg, c->d_seg_elem, c->d_conn, c->d_X, c->nnd,
                                                              c->d_Ke64, d_w, part);
  segment_macro_combine_kernel<<<(c->nseg * ncols * 9 + 127) / 128, 128, 0, c->stream>>>(c->nseg, c->d_seg_elem, ncols,
                                                                                        part, kL, d_vol0, d_out);
  c->launches += 2;
  const int s = ok(c, cudaGetLastError(), "segment_macro_kernel") ? TG_OK : TG_ERR_CUDA;
  cudaFreeAsync(part, c->stream);
  return s;
}

int launch_segment_norms(Context* c, int nseg, const int* d_node_off, double* d_out) {
  const int nb = share_blocks(c->nnd, nseg, kNormShare);
  double* part = nullptr;
  if (!ok(c, cudaMallocAsync((void**)&part, sizeof(double) * nb, c->stream), "alloc")) return TG_ERR_OOM;
  segment_norms_kernel<<<nb, 256, 0, c->stream>>>(nseg, d_node_off, c->d_R, part);
  segment_combine_kernel<1, kNormShare><<<(nseg + 127) / 128, 128, 0, c->stream>>>(nseg, d_node_off, part, d_out);
  c->launches += 2;
  const int s = ok(c, cudaGetLastError(), "segment_norms_kernel") ? TG_OK : TG_ERR_CUDA;
  cudaFreeAsync(part, c->stream);
  return s;
}

int launch_segment_stress(Context* c, int nseg, const int* d_elem_off, double* d_out) {
  const int nb = share_blocks(c->nel, nseg, kStressShare);
  double* part = nullptr;
  if (!ok(c, cudaMallocAsync((void**)&part, sizeof(double) * 9 * nb, c->stream), "alloc")) return TG_ERR_OOM;
  segment_stress_kernel<<<nb, 256, 0, c->stream>>>(nseg, d_elem_off, c->d_conn, c->d_X, c->nnd, c->d_fint, part);
  segment_combine_kernel<9, kStressShare>
      <<<(nseg * 9 + 127) / 128, 128, 0, c->stream>>>(nseg, d_elem_off, part, d_out);
  c->launches += 2;
  const int s = ok(c, cudaGetLastError(), "segment_stress_kernel") ? TG_OK : TG_ERR_CUDA;
  cudaFreeAsync(part, c->stream);
  return s;
}

}  // namespace tg
