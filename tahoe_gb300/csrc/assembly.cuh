// The value of a global 3x3 block gathered from its element contributions, and
// the (block-)Jacobi inverses of a diagonal block: shared by the assembly into
// the streamed storages and by the resident PCG, which assembles its rows
// straight into shared memory.  Internal to the library.
#pragma once

#include <type_traits>

#include "tg_internal.h"

namespace tg {

namespace {

__device__ __forceinline__ int upper_slot(int a, int b) { return a * 8 - a * (a - 1) / 2 + (b - a); }

// The value of global block j: its element contributions in the
// destination-sorted order, rows of prescribed dofs zeroed (columns are kept,
// so a product with a prescribed-increment vector gives the coupling
// K_fp du_p; PCG vectors are zero at prescribed dofs, so the kept columns
// never enter the solve).
template <typename T>
__device__ __forceinline__ void block_value(int j, uint8_t mI, const int* __restrict__ cptr,
                                            const int* __restrict__ contrib, const T* __restrict__ Ke, T acc[9]) {
  using V4 = typename std::conditional<sizeof(T) == 4, float4, double4_32a>::type;
#pragma unroll
  for (int k = 0; k < 9; ++k) acc[k] = T(0);
  const int c1 = cptr[j + 1];
  for (int c = cptr[j]; c < c1; ++c) {
    const int code = contrib[c];
    const int e = code >> 6, a = (code >> 3) & 7, b = code & 7;
    // the element block's three padded rows: one aligned vector load each
    const V4* src = reinterpret_cast<const V4*>(
        Ke + ((long long)e * kSlots + (a <= b ? upper_slot(a, b) : upper_slot(b, a))) * kKeBlock);
    const V4 k0 = src[0], k1 = src[1], k2 = src[2];
    const T m[9] = {k0.x, k0.y, k0.z, k1.x, k1.y, k1.z, k2.x, k2.y, k2.z};
    if (a <= b) {
#pragma unroll
      for (int k = 0; k < 9; ++k) acc[k] += m[k];
    } else {
#pragma unroll
      for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int q = 0; q < 3; ++q) acc[p * 3 + q] += m[q * 3 + p];
    }
  }
#pragma unroll
  for (int p = 0; p < 3; ++p)
    if (!((mI >> p) & 1))
#pragma unroll
      for (int q = 0; q < 3; ++q) acc[p * 3 + q] = T(0);
}

// (block-)Jacobi inverse of a diagonal block: Dg the inverse diagonal, B the
// inverse 3x3 block; inactive dofs get identity in the inverse's input and
// zero in its output.
template <typename T>
__device__ __forceinline__ void diagonal_inverses(uint8_t mI, const T acc[9], T Dg[9], T B[9]) {
  T A[9];
#pragma unroll
  for (int p = 0; p < 3; ++p)
#pragma unroll
    for (int q = 0; q < 3; ++q)
      A[p * 3 + q] = (((mI >> p) & 1) && ((mI >> q) & 1)) ? acc[p * 3 + q] : (p == q ? T(1) : T(0));
  // Jacobi: inverse diagonal; block-Jacobi: inverse of the 3x3 block
  const T d = A[0] * (A[4] * A[8] - A[5] * A[7]) - A[1] * (A[3] * A[8] - A[5] * A[6]) +
              A[2] * (A[3] * A[7] - A[4] * A[6]);
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
#pragma unroll
  for (int k = 0; k < 9; ++k) Dg[k] = T(0);
  Dg[0] = T(1) / A[0];
  Dg[4] = T(1) / A[4];
  Dg[8] = T(1) / A[8];
#pragma unroll
  for (int p = 0; p < 3; ++p)
#pragma unroll
    for (int q = 0; q < 3; ++q)
      if (!((mI >> p) & 1) || !((mI >> q) & 1)) {
        B[p * 3 + q] = T(0);
        Dg[p * 3 + q] = T(0);
      }
}

}  // namespace
}  // namespace tg
