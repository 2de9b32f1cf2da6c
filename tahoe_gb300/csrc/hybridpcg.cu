// Hybrid PCG, sm_103a: one launch per solve for a whole mesh of 20,000 nodes
// and more, FP32 form (smaller meshes and RVE batches: respcg.cu).
//
// The push-storage solve (pcg_cg.cu) streams half the matrix every iteration
// (174 MB on the 64^3 block) and passes 55 MB of transposed products through
// L2, in two kernels that start and end with the HBM idle.  Here one CTA per
// SM keeps a compact part of the mesh for the whole solve:
//   * rows are dealt along a space-filling (Morton) order of the node
//     coordinates, so a part's 1,800 rows reach 1,600 rows of other parts: the
//     search vector over own and halo rows sits in shared memory and no
//     product or partial product leaves the SM;
//   * a part's first 32 chunks of 8 rows keep their blocks in tensor memory,
//     the others are read every iteration (both triangles, 38 bytes a block),
//     68 values a lane in 17 16-byte loads whose registers are reloaded as
//     their blocks are used, 139 KB in flight an SM;
//   * 42 MB of them stay in L2 (evict_last), the rest passes (evict_first);
//   * r, w, p, s and the preconditioner stay in shared memory where they fit;
//   * the halo and the sums travel as sequence-numbered words (respcg.cu).
// The recurrences, precision and reductions are the resident solve's.
//
// Measured per iteration, the streamed solve / this one: 93,025 nodes
// (60x60x24) 23.3 / 9.8 us, 101,000 (53x47x41) 26.5 / 11.5, 207,000 (64x64x48)
// 41.5 / 28.2, 274,625 (64^3) 50.0 / 46.5, 328,509 (68^3) 63.8 / 57.6, 393,000
// (73x75x70) 75.9 / 75.7 and with block-Jacobi 77.7 / 84.4.  Up to about
// 110,000 nodes the streamed part is L2's and the exchange (4 us) and product
// bound it; above, HBM: 64^3 reads 217 MB an iteration at 5.9 TB/s, with 9 us
// of halo, sums and updates beside it.  L2 serves fewer bytes than it holds,
// lines of the other die being kept twice: keeping 0 / 20 / 30 / 45 / 60 MB
// took 50.0 / 47.8 / 46.8 / 46.6 / 48.6 us at 64^3 and 33.1 / 31.2 / 29.8 /
// 28.0 / 27.8 at 64x64x48; lines without a hint or prefetched a chunk ahead
// displace the kept ones (59.7, 54.3 us).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "respcg_device.cuh"

namespace tg {

namespace {

constexpr int kHybWarps = 16;
constexpr int kHybSteps = 7;                 // steps of a chunk: at most 28 blocks a row
constexpr int kHybVec = 17;                  // 16-byte words of a streamed lane: 8 columns, 63 values
constexpr int kHybTm = 2;                    // chunks per warp in tensor memory
constexpr int kHybMaxRows = 4096;            // rows of a part (sorted in shared memory)
constexpr int kHybCell = 512;                // nodes of a cell of the ordering
constexpr int kHybHalo = 8192;               // halo rows of a part
constexpr double kHybL2Keep = 42.0 * 1048576.0;  // streamed bytes kept in L2
// streamed bytes above which half the matrix is less work for the HBM than
// the whole beside what is kept: 315 MB (68^3) 57.6 against 63.8 us, 381 MB
// (73x75x70) even, 506 MB (78^3) 103 against 98
constexpr double kHybStreamMax = 340.0e6;

struct HybArgs {
  const int* row_start;   // k+1, multiples of 8 but the last
  const int* act_node;    // node of every row
  const int2* slot;       // [chunk][7][32] contributions {first, count}
  const uint16_t* lcol;   // [chunk][7][32] row of the part (own, then halo)
  const uint8_t* steps;   // per chunk
  const int* halo;        // [k][kHybHalo] rows
  const int* nhalo;       // k
  const int* contrib;
  const float* Ke;
  const uint8_t* mask;
  const double4_32a* rhs;
  float4* x;
  float4* stream;         // [chunk][17][32]
  float* xs;              // [chunk][32] solution
  float* state;           // p, s, preconditioner of every chunk, where shared memory has no room
  uint4* ll;              // sums' tables, then rows' words
  ResOut* out;
  PcgScalars* sc;
  int* status;
  WaitLimits waits;
  long long chunks;
  int rows, uwcap, chcap; // shared memory: window rows, chunks
  int in_smem;            // of p, s, preconditioner: how many are in shared memory
  float keep;             // share of the streamed chunks that is kept in L2
  int max_it;
  double tol;
};

__device__ __forceinline__ float4 ld_stream(const float4* p, uint64_t pol) {
  float4 v;
  asm volatile("ld.global.L1::no_allocate.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(p), "l"(pol));
  return v;
}

template <bool BLK>
__global__ void __launch_bounds__(kHybWarps * 32, 1) hybrid_kernel(HybArgs A) {
  constexpr int NM = BLK ? 3 : 1;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ ResShared<float> sh;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = lane & 3, q0 = lane & ~3;
  const int rank = blockIdx.x, k = gridDim.x;
  const int row0 = A.row_start[rank], row1 = A.row_start[rank + 1], nown = row1 - row0;
  const int ch0 = row0 / 8, nch = (nown + 7) / 8, nh = A.nhalo[rank];
  const int* halo = A.halo + (size_t)rank * kHybHalo;
  float4* uw = reinterpret_cast<float4*>(smem);
  uint4* tcol = reinterpret_cast<uint4*>(uw + A.uwcap);                // columns of the chunks in tensor memory
  float* rb = reinterpret_cast<float*>(tcol + kHybTm * kHybWarps * 32);  // [chunk][32]
  float* wb = rb + A.chcap * 32;
  float* extra = wb + A.chcap * 32;
  const long long plane = A.chunks * 32;
  auto state_at = [&](int which, int words) {
    return which < A.in_smem ? extra + which * A.chcap * 32 : A.state + which * plane + (long long)ch0 * 32 * words;
  };
  float* pb = state_at(0, 1);
  float* sb = state_at(1, 1);
  float* Mb = state_at(2, NM);  // [chunk][NM][32], last in both places
  float* xb = A.xs + (long long)ch0 * 32;
  uint4* inbox = A.ll;
  uint4* urow = A.ll + 4 * (size_t)min(k, kResCopies) * k;
  if (threadIdx.x < 32) tmem_alloc(&sh.tmem);
  if (threadIdx.x == 0) sh.abort_flag = 0;
  __syncthreads();
  const unsigned tm = sh.tmem + ((unsigned)(warp & 3) << 21) + (unsigned)(warp >> 2) * 128u;
  // --- the part's rows, assembled from the element blocks
  for (int i = warp, j = 0; i < nch; i += kHybWarps, ++j) {
    const int gch = ch0 + i, row = row0 + i * 8 + (lane >> 2);
    const bool live = row < row1;
    const uint8_t m = live ? A.mask[A.act_node[row]] : 0;
    const int T = A.steps[gch];
    float D[9];
    bool have = false;
#pragma unroll
    for (int e = 0; e < 9; ++e) D[e] = 0.f;
    unsigned g[4] = {0u, 0u, 0u, 0u};
    float* sp = reinterpret_cast<float*>(A.stream + (size_t)gch * kHybVec * 32);
#pragma unroll 1
    for (int t = 0; t < kHybSteps; ++t) {
      float acc[9];
#pragma unroll
      for (int e = 0; e < 9; ++e) acc[e] = 0.f;
      if (t < T) {
        const size_t at = ((size_t)gch * kHybSteps + t) * 32 + lane;
        const int2 sl = A.slot[at];
        const unsigned lc = A.lcol[at];
        slot_value<float>(sl, m, A.contrib, A.Ke, 0, acc);
        const unsigned w = (t & 1) ? lc << 16 : lc;
        g[0] |= (t >> 1) == 0 ? w : 0u;
        g[1] |= (t >> 1) == 1 ? w : 0u;
        g[2] |= (t >> 1) == 2 ? w : 0u;
        g[3] |= (t >> 1) == 3 ? w : 0u;
        if (sl.y > 0 && (int)lc == row - row0) {
          have = true;
#pragma unroll
          for (int e = 0; e < 9; ++e) D[e] = acc[e];
        }
      }
      __syncwarp();
      if (j < kHybTm) {
        tmem_st9(tm + (unsigned)j * 64u + 9u * (unsigned)t, acc);
      } else {
#pragma unroll
        for (int e = 0; e < 9; ++e) {
          const int wd = 4 + 9 * t + e;
          sp[((wd >> 2) * 32 + lane) * 4 + (wd & 3)] = acc[e];
        }
      }
    }
    const uint4 gc = make_uint4(g[0], g[1], g[2], g[3]);
    if (j < kHybTm) {
      tcol[(j * kHybWarps + warp) * 32 + lane] = gc;
    } else {
      reinterpret_cast<uint4*>(sp)[lane] = gc;
      sp[((kHybVec - 1) * 32 + lane) * 4 + 3] = 0.f;
    }
    const unsigned who = (__ballot_sync(0xffffffffu, have) >> q0) & 0xfu;
    const int src = q0 + (who ? __ffs((int)who) - 1 : 0);
    float Dg[9], B[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) D[e] = __shfl_sync(0xffffffffu, D[e], src);
    diagonal_inverses<float>(m, D, Dg, B);
#pragma unroll
    for (int d = 0; d < NM; ++d) {
      float v = BLK ? (c == 0 ? B[d] : c == 1 ? B[3 + d] : c == 2 ? B[6 + d] : 0.f)
                    : (c == 0 ? Dg[0] : c == 1 ? Dg[4] : c == 2 ? Dg[8] : 0.f);
      if (!who || !live) v = 0.f;
      Mb[(i * NM + d) * 32 + lane] = v;
    }
    pb[i * 32 + lane] = sb[i * 32 + lane] = xb[i * 32 + lane] = 0.f;
  }
  tmem_wait_st();
  auto precond = [&](int i, float r) {
    float z = 0.f;
#pragma unroll
    for (int d = 0; d < NM; ++d)
      z += Mb[(i * NM + d) * 32 + lane] * (BLK ? __shfl_sync(0xffffffffu, r, q0 + d) : r);
    return z;
  };
  // a row's new search vector: its place in the window, its word for the others
  auto publish = [&](int i, float u, unsigned seq) {
    const float u1 = __shfl_down_sync(0xffffffffu, u, 1), u2 = __shfl_down_sync(0xffffffffu, u, 2);
    const int row = i * 8 + (lane >> 2);
    if (c == 0 && row < nown) {
      uw[row] = make_float4(u, u1, u2, 0.f);
      RowWords<float>::store(urow + row0 + row, u, u1, u2, seq);
    }
  };
  // --- the right-hand side on a power of two near its size (as respcg.cu)
  unsigned seq = 0;
  int scale_exp = 0;
  Acc<float> a[3];
  {
    auto rhs_at = [&](int i) {
      const int row = row0 + i * 8 + (lane >> 2);
      if (row >= row1 || c == 3) return 0.0;
      const int n = A.act_node[row];
      return ((A.mask[n] >> c) & 1) ? reinterpret_cast<const double*>(A.rhs + n)[c] : 0.0;
    };
    AccMax mx[3];
    for (int i = warp; i < nch; i += kHybWarps) mx[0].v = max(mx[0].v, exponent_of(rhs_at(i)));
    ++seq;
    total3<AccMax, float, true>(mx, sh, k, rank, seq, inbox, A.waits);
    __syncthreads();
    const int e1 = (int)sh.tot[0];
    if (e1 > 0 && e1 < 0x7ff) scale_exp = max(-1000, min(1000, 1023 - e1));
    double sc = power_of_two(scale_exp);
    mx[0].v = mx[1].v = mx[2].v = 0;
    for (int i = warp; i < nch; i += kHybWarps) {
      const float r = (float)(rhs_at(i) * sc);
      mx[0].v = max(mx[0].v, exponent_of((double)(r * precond(i, r))));
    }
    __syncthreads();
    ++seq;
    total3<AccMax, float, true>(mx, sh, k, rank, seq, inbox, A.waits);
    __syncthreads();
    const int e2 = (int)sh.tot[0];
    if (e2 > 0 && e2 < 0x7ff && e1 > 0 && e1 < 0x7ff) scale_exp = max(-1000, min(1000, scale_exp - (e2 - 1023) / 2));
    sc = power_of_two(scale_exp);
    for (int i = warp; i < nch; i += kHybWarps) {
      const float r = (float)(rhs_at(i) * sc);
      rb[i * 32 + lane] = r;
      const float u = precond(i, r);
      publish(i, u, 1u);
      a[1].add_prod(r, u);
      a[2].add_prod(r, r);
    }
  }
  // Streamed chunks: every warp's loads run one chunk ahead of its product,
  // registers reloaded as their blocks are used; the last chunk's are
  // reloaded with the next iteration's first, before the reduction.
  const uint64_t pol_keep = l2_policy_evict_last(), pol_pass = l2_policy_evict_first();
  const int first = warp + kHybTm * kHybWarps;
  float v[4 * kHybVec];
  auto source = [&](int i, const float4*& p, uint64_t& pol) {
    const int j = i / kHybWarps + warp;
    p = A.stream + (size_t)(ch0 + i) * kHybVec * 32 + lane;
    pol = (int)((float)(j + 1) * A.keep) != (int)((float)j * A.keep) ? pol_keep : pol_pass;
  };
  auto load = [&](int q, const float4* p, uint64_t pol) {
    const float4 f = ld_stream(p + 32 * q, pol);
    v[4 * q] = f.x;
    v[4 * q + 1] = f.y;
    v[4 * q + 2] = f.z;
    v[4 * q + 3] = f.w;
  };
  if (first < nch) {
    const float4* p;
    uint64_t pol;
    source(first, p, pol);
#pragma unroll
    for (int q = 0; q < kHybVec; ++q) load(q, p, pol);
  } else {
#pragma unroll
    for (int q = 0; q < 4 * kHybVec; ++q) v[q] = 0.f;
  }
  int it = 0;
  for (;; ++it) {
    if (warp == 1 && lane == 0 && it > 0) scalars_next(sh);
    for (int h = threadIdx.x; h < nh; h += kHybWarps * 32) {
      const uint4* w = urow + halo[h];
      float x0, x1, x2;
      int tries = 0;
      while (!RowWords<float>::load(w, (unsigned)it + 1u, x0, x1, x2) && poll_again(sh, A.waits, tries)) {
      }
      uw[nown + h] = make_float4(x0, x1, x2, 0.f);
    }
    __syncthreads();
    // w = A u
    for (int i = warp, j = 0; i < nch; i += kHybWarps, ++j) {
      float a0 = 0.f, a1 = 0.f, a2 = 0.f;
      auto index = [](const uint4& g, int t) {
        const unsigned v = t < 2 ? g.x : t < 4 ? g.y : t < 6 ? g.z : g.w;
        return (t & 1) ? v >> 16 : v & 0xffffu;
      };
      auto fma9 = [&](auto f, const float4& uj) {
        a0 += f(0) * uj.x + f(1) * uj.y + f(2) * uj.z;
        a1 += f(3) * uj.x + f(4) * uj.y + f(5) * uj.z;
        a2 += f(6) * uj.x + f(7) * uj.y + f(8) * uj.z;
      };
      if (j < kHybTm) {
        const uint4 g = tcol[(j * kHybWarps + warp) * 32 + lane];
        const unsigned col = tm + (unsigned)j * 64u;
#pragma unroll
        for (int t = 0; t < kHybSteps; ++t) {
          unsigned b[9];
          __syncwarp();
          tmem_ld9(col + 9u * (unsigned)t, b);
          const float4 uj = uw[index(g, t)];
          tmem_wait_ld();
          fma9([&](int e) { return __uint_as_float(b[e]); }, uj);
        }
      } else {
        const float4* p;
        uint64_t pol;
        source(i + kHybWarps < nch ? i + kHybWarps : first, p, pol);
        const uint4 g = make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]),
                                   __float_as_uint(v[3]));
        load(0, p, pol);
#pragma unroll
        for (int t = 0; t < kHybSteps; ++t) {
          const float4 uj = uw[index(g, t)];
          fma9([&](int e) { return v[4 + 9 * t + e]; }, uj);
#pragma unroll
          for (int q = 9 * t / 4 + 1; q <= (t + 1 < kHybSteps ? (9 * t + 9) / 4 : kHybVec - 1); ++q) load(q, p, pol);
        }
      }
      const bool up = (c & 2) != 0;
      const float g0 = __shfl_xor_sync(0xffffffffu, up ? a0 : a2, 2);
      const float g1 = __shfl_xor_sync(0xffffffffu, a1, 2);
      const float b0 = (up ? a2 : a0) + g0;
      const float b1 = a1 + g1;
      const float e = __shfl_xor_sync(0xffffffffu, up ? b0 : ((c & 1) ? b0 : b1), 1);
      float w = up ? b0 + e : ((c & 1) ? b1 + e : b0 + e);
      if (c == 3) w = 0.f;
      wb[i * 32 + lane] = w;
      const int row = i * 8 + (lane >> 2);
      const float u = row < nown ? reinterpret_cast<const float*>(uw + row)[c] : 0.f;
      a[0].add_prod(u, w);
    }
    ++seq;
    total3<Acc<float>, float, true>(a, sh, k, rank, seq, inbox, A.waits);
    if (threadIdx.x == 0) scalars(sh, it, A.max_it, A.tol);
    __syncthreads();
    if (sh.code) break;
    const float al = sh.coef[0], be = sh.coef[1];
#pragma unroll
    for (int q = 0; q < 3; ++q) a[q] = Acc<float>();
#pragma unroll 2
    for (int i = warp; i < nch; i += kHybWarps) {
      const int at = i * 32 + lane;
      const float row_x = xb[at];
      const float uo = i * 8 + (lane >> 2) < nown ? reinterpret_cast<const float*>(uw + i * 8 + (lane >> 2))[c] : 0.f;
      const float pn = uo + be * pb[at], sn = wb[at] + be * sb[at];
      const float rn = rb[at] - al * sn;
      const float u = precond(i, rn);
      pb[at] = pn;
      sb[at] = sn;
      rb[at] = rn;
      xb[at] = row_x + al * pn;
      publish(i, u, (unsigned)it + 2u);
      a[1].add_prod(rn, u);
      a[2].add_prod(rn, rn);
    }
  }
  const double unscale = power_of_two(-scale_exp);
  for (int i = warp; i < nch; i += kHybWarps) {
    const float x0 = xb[i * 32 + lane];
    const float x1 = __shfl_down_sync(0xffffffffu, x0, 1), x2 = __shfl_down_sync(0xffffffffu, x0, 2);
    const int row = row0 + i * 8 + (lane >> 2);
    if (row < row1 && c == 0) A.x[A.act_node[row]] = make_float4(x0, x1, x2, 0.f);
  }
  if (threadIdx.x == 0) {
    if (sh.fail == 5) atomicOr(A.status, kStatusWaitTimeout);
    if (rank == 0) {
      ResOut o;
      o.rr = word_value(sh, sh.rr);
      o.rr0 = word_value(sh, sh.rr0);
      o.unscale = unscale;
      o.done = sh.code;
      o.fail = sh.fail;
      o.iters = it;
      o.pad = 0;
      *A.out = o;
      A.sc->unscale = unscale;
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) tmem_free(sh.tmem);
}

// ---- rows, parts and halos (device) -----------------------------------------

// Morton cell of a node: the box cut into 2^bits[d] cells a side, bits
// interleaved from the highest.
struct HybCells {
  double lo[3], inv[3];
  int bits[3];
};
__device__ __forceinline__ int cell_of(const HybCells& C, const double* __restrict__ X, int nnd, int n) {
  int q[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int top = (1 << C.bits[d]) - 1;
    q[d] = min(max((int)((float)((X[(size_t)d * nnd + n] - C.lo[d]) * C.inv[d])), 0), top);
  }
  int code = 0;
  for (int b = 18; b >= 0; --b)
#pragma unroll
    for (int d = 2; d >= 0; --d)
      if (b < C.bits[d]) code = (code << 1) | ((q[d] >> b) & 1);
  return code;
}
__global__ void hyb_count_kernel(int n, const uint8_t* __restrict__ mask, const double* __restrict__ X, HybCells C,
                                 int* __restrict__ count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && mask[i]) atomicAdd(count + cell_of(C, X, n, i), 1);
}
__global__ void hyb_place_kernel(int n, const uint8_t* __restrict__ mask, const double* __restrict__ X, HybCells C,
                                 const int* __restrict__ start, int* __restrict__ count, int* __restrict__ order) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || !mask[i]) return;
  const int q = cell_of(C, X, n, i);
  order[start[q] + atomicSub(count + q, 1) - 1] = i;
}
// nodes of a cell by index: the placement's order is that of its atomics.  A
// cell of more than kHybCell nodes (a strongly graded mesh) raises the flag.
__global__ void hyb_cell_sort_kernel(int cells, const int* __restrict__ start, int* __restrict__ order,
                                     int* __restrict__ flag) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= cells) return;
  const int a = start[q], b = start[q + 1];
  if (b - a > kHybCell) {
    atomicOr(flag, 1);
    return;
  }
  for (int i = a + 1; i < b; ++i) {
    const int v = order[i];
    int j = i;
    for (; j > a && order[j - 1] > v; --j) order[j] = order[j - 1];
    order[j] = v;
  }
}
// blocks of a row on active columns, plus a constant for its vector work
__global__ void hyb_weight_kernel(int rows, const int* __restrict__ order, const int* __restrict__ rowptr,
                                  const int* __restrict__ col, const uint8_t* __restrict__ mask,
                                  int* __restrict__ weight) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= rows) return;
  const int g = order[r];
  int w = 6;
  for (int j = rowptr[g]; j < rowptr[g + 1]; ++j) w += mask[col[j]] ? 1 : 0;
  weight[r] = w;
}
__global__ void hyb_split_kernel(int k, int rows, const int* __restrict__ prefix, int* __restrict__ start) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j > k) return;
  if (j == 0 || j == k) {
    start[j] = j == 0 ? 0 : rows;
    return;
  }
  const long long target = ((long long)j * prefix[rows] + k / 2) / k;
  int lo = 0, hi = rows;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (prefix[mid] < target)
      lo = mid + 1;
    else
      hi = mid;
  }
  start[j] = min((lo + 4) / 8 * 8, rows / 8 * 8);
}
// a part's rows by node index (consecutive nodes of a line next to each other,
// so the window's reads fall into different banks), and every node's row
__global__ void __launch_bounds__(1024) hyb_part_sort_kernel(const int* __restrict__ start, int* __restrict__ order,
                                                             int* __restrict__ rank) {
  __shared__ int v[kHybMaxRows];
  const int a = start[blockIdx.x], n = start[blockIdx.x + 1] - a;
  int m = 1;
  while (m < n) m <<= 1;
  for (int i = threadIdx.x; i < m; i += blockDim.x) v[i] = i < n ? order[a + i] : 0x7fffffff;
  __syncthreads();
  for (int s = 2; s <= m; s <<= 1)
    for (int d = s >> 1; d > 0; d >>= 1) {
      for (int i = threadIdx.x; i < m; i += blockDim.x) {
        const int j = i ^ d;
        if (j > i) {
          const int x = v[i], y = v[j];
          if ((x > y) == ((i & s) == 0)) {
            v[i] = y;
            v[j] = x;
          }
        }
      }
      __syncthreads();
    }
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    order[a + i] = v[i];
    rank[v[i]] = a + i;
  }
}
// one warp per chunk, four lanes per row: a row's active blocks go to its
// lanes in turn; flag[0] is raised for a row of more than 28
__global__ void __launch_bounds__(256) hyb_rows_kernel(int rows, int nch, const int* __restrict__ act_node,
                                                       const int* __restrict__ rowptr, const int* __restrict__ col,
                                                       const uint8_t* __restrict__ mask, const int* __restrict__ rank,
                                                       const int* __restrict__ cptr, int2* __restrict__ slot,
                                                       int* __restrict__ cidx, uint8_t* __restrict__ steps,
                                                       int* __restrict__ flag) {
  const int ch = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31, c = lane & 3;
  if (ch >= nch) return;
  const int row = ch * 8 + (lane >> 2);
  const bool live = row < rows;
  const int g = live ? act_node[row] : 0;
  const int b = live ? rowptr[g] : 0, e = live ? rowptr[g + 1] : 0;
  for (int t = 0; t < kHybSteps; ++t) {
    const size_t at = ((size_t)ch * kHybSteps + t) * 32 + lane;
    slot[at] = make_int2(0, 0);
    cidx[at] = min(ch * 8, rows - 1);
  }
  __syncwarp();
  int cnt = 0;
  for (int j0 = b; __any_sync(0xffffffffu, j0 < e); j0 += 4) {
    const int j = j0 + c;
    const bool on = j < e && mask[col[j]] != 0;
    const unsigned m = (__ballot_sync(0xffffffffu, on) >> (lane & ~3)) & 0xfu;
    const int q = cnt + __popc(m & ((1u << c) - 1u));
    if (on && q < 4 * kHybSteps) {
      const size_t at = ((size_t)ch * kHybSteps + (q >> 2)) * 32 + (lane & ~3) + (q & 3);
      slot[at] = make_int2(cptr[j], cptr[j + 1] - cptr[j]);
      cidx[at] = rank[col[j]];
    }
    cnt += __popc(m);
  }
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) cnt = max(cnt, __shfl_xor_sync(0xffffffffu, cnt, o));
  if (lane == 0) {
    steps[ch] = (uint8_t)min((cnt + 3) / 4, kHybSteps);
    if (cnt > 4 * kHybSteps) atomicOr(flag, 1);
  }
}
// one CTA per part: the other parts' rows its blocks reach, by row, and every
// block's place in the part's window
__global__ void __launch_bounds__(1024) hyb_halo_kernel(int rows, const int* __restrict__ start,
                                                        const int* __restrict__ cidx, int* __restrict__ halo,
                                                        int* __restrict__ nhalo, uint16_t* __restrict__ lcol) {
  extern __shared__ unsigned hyb_bits[];
  const int words = (rows + 31) / 32;
  unsigned* bits = hyb_bits;
  int* before = reinterpret_cast<int*>(hyb_bits + words);
  __shared__ int wsum[32], carry;
  const int p = blockIdx.x, r0 = start[p], r1 = start[p + 1];
  const size_t a = (size_t)(r0 / 8) * kHybSteps * 32, b = (size_t)((r1 + 7) / 8) * kHybSteps * 32;
  for (int i = threadIdx.x; i < words; i += blockDim.x) bits[i] = 0u;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (size_t i = a + threadIdx.x; i < b; i += blockDim.x) {
    const int r = cidx[i];
    if (r < r0 || r >= r1) atomicOr(&bits[r >> 5], 1u << (r & 31));
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int w0 = 0; w0 < words; w0 += blockDim.x) {
    const int w = w0 + threadIdx.x, n = w < words ? __popc(bits[w]) : 0;
    int inc = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    int pre = carry + inc - n;
    for (int q = 0; q < warp; ++q) pre += wsum[q];
    if (w < words) before[w] = pre;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = pre + n;
    __syncthreads();
  }
  if (threadIdx.x == 0) nhalo[p] = carry;
  for (int w = threadIdx.x; w < words; w += blockDim.x) {
    int at = before[w];
    for (unsigned m = bits[w]; m; m &= m - 1, ++at)
      if (at < kHybHalo) halo[(size_t)p * kHybHalo + at] = w * 32 + __ffs((int)m) - 1;
  }
  for (size_t i = a + threadIdx.x; i < b; i += blockDim.x) {
    const int r = cidx[i];
    lcol[i] = (uint16_t)(r >= r0 && r < r1 ? r - r0
                                           : (r1 - r0) + before[r >> 5] + __popc(bits[r >> 5] & ((1u << (r & 31)) - 1u)));
  }
}

int hyb_smem(int uwcap, int chcap, int arrays) {
  return uwcap * 16 + kHybTm * kHybWarps * 32 * 16 + chcap * 128 * (2 + arrays);
}

}  // namespace

// What a mesh keeps for the hybrid solve.
struct HybState {
  HybArgs A{};
  int k = 0;
  int smem[2] = {0, 0}, in_smem[2] = {0, 0};  // by preconditioner (Jacobi, block-Jacobi)
  long long ll_words = 0;
};

void hybrid_reset(Context* c) {
  delete c->hyb;
  c->hyb = nullptr;
}

// Plans the current mesh; *fits false where a row has more than 28 blocks, a
// part does not fit a CTA or memory is short.
int hybrid_plan(Context* c, bool* fits) {
  *fits = false;
  const int n = c->nnd, k = c->num_sms;
  if (c->composed || (int)c->h_coords.size() != 3 * n || n < 8 * k || n > 600000) return TG_OK;
  auto stream_bytes = [&](long long rows) {
    return (double)std::max<long long>((rows + 7) / 8 - k * kHybTm * kHybWarps, 1) * kHybVec * 512;
  };
  if (stream_bytes(c->neq / 3) > kHybStreamMax) return TG_OK;  // before the nodes are looked at
  hybrid_reset(c);
  cudaStream_t st = c->stream;
  // cells of about eight nodes, at most 2^18
  HybCells C;
  double len[3], vol = 1.0;
  for (int d = 0; d < 3; ++d) {
    const auto mm = std::minmax_element(c->h_coords.begin() + (size_t)d * n, c->h_coords.begin() + (size_t)(d + 1) * n);
    C.lo[d] = *mm.first;
    len[d] = std::max(*mm.second - *mm.first, 1e-300);
    vol *= len[d];
  }
  if (!(vol > 0.0) || !std::isfinite(vol)) return TG_OK;
  const double edge = std::cbrt(vol / std::max(1.0, n / 8.0));
  int total = 0;
  for (int d = 0; d < 3; ++d) {
    C.bits[d] = std::min(10, std::max(0, (int)std::ceil(std::log2(std::max(1.0, len[d] / edge)))));
    total += C.bits[d];
  }
  while (total > 18) {
    --*std::max_element(C.bits, C.bits + 3);
    --total;
  }
  for (int d = 0; d < 3; ++d) C.inv[d] = (double)(1 << C.bits[d]) / len[d];
  const int cells = 1 << total;
  std::vector<void*> tmp;
  auto release = [&]() {
    for (void* p : tmp) dfree(c, p);
    tmp.clear();
  };
  auto get = [&](auto** p, size_t m) {
    if (!dalloc(c, p, m)) return false;
    tmp.push_back((void*)*p);
    return true;
  };
  int *count = nullptr, *start = nullptr, *scan = nullptr, *order = nullptr, *weight = nullptr, *prefix = nullptr,
      *rank = nullptr, *part = nullptr, *flag = nullptr, *cidx = nullptr;
  if (!get(&count, cells) || !get(&start, (size_t)cells + 1) || !get(&scan, (size_t)std::max(n, cells) / 1024 + 4) ||
      !get(&rank, n) || !get(&flag, 1)) {
    release();
    return TG_OK;
  }
  int rows = 0;
  bool good = ok(c, cudaMemsetAsync(count, 0, sizeof(int) * cells, st), "cells") &&
              ok(c, cudaMemsetAsync(flag, 0, sizeof(int), st), "flag");
  if (good) hyb_count_kernel<<<(n + 255) / 256, 256, 0, st>>>(n, c->d_mask, c->d_X, C, count);
  if (good && scan_counts(c, cells, count, start, scan)) good = false;
  good = good && ok(c, cudaMemcpyAsync(&rows, start + cells, sizeof(int), cudaMemcpyDeviceToHost, st), "rows") &&
         ok(c, cudaStreamSynchronize(st), "sync");
  if (!good) {
    release();
    return TG_ERR_CUDA;
  }
  if (rows < 8 * k || (rows + k - 1) / k > kHybMaxRows - 64) {
    release();
    return TG_OK;
  }
  const int nch = (rows + 7) / 8;
  const double streamed = stream_bytes(rows);
  if (streamed > kHybStreamMax) {
    release();
    return TG_OK;
  }
  const size_t slots = (size_t)nch * kHybSteps * 32;
  HybState* H = new HybState();
  c->hyb = H;
  int2* slot = nullptr;
  uint16_t* lcol = nullptr;
  uint8_t* steps = nullptr;
  int *halo = nullptr, *nhalo = nullptr;
  std::vector<void*> kept;
  auto hold = [&](auto** p, size_t m) {
    if (!dalloc(c, p, m)) return false;
    kept.push_back((void*)*p);
    return true;
  };
  auto give_up = [&](int s) {
    release();
    for (void* p : kept) dfree(c, p);
    hybrid_reset(c);
    return s;
  };
  if (!hold(&order, rows) || !get(&weight, rows) || !get(&prefix, (size_t)rows + 1) || !hold(&part, (size_t)k + 1) ||
      !hold(&slot, slots) || !hold(&lcol, slots) || !hold(&steps, nch) || !get(&cidx, slots) ||
      !hold(&halo, (size_t)k * kHybHalo) || !hold(&nhalo, k))
    return give_up(TG_OK);
  hyb_place_kernel<<<(n + 255) / 256, 256, 0, st>>>(n, c->d_mask, c->d_X, C, start, count, order);
  hyb_cell_sort_kernel<<<(cells + 127) / 128, 128, 0, st>>>(cells, start, order, flag);
  hyb_weight_kernel<<<(rows + 255) / 256, 256, 0, st>>>(rows, order, c->d_rowptr, c->d_col, c->d_mask, weight);
  if (scan_counts(c, rows, weight, prefix, scan)) return give_up(TG_ERR_CUDA);
  hyb_split_kernel<<<(k + 256) / 256, 256, 0, st>>>(k, rows, prefix, part);
  std::vector<int> h_part(k + 1), h_halo(k);
  if (!ok(c, cudaMemcpyAsync(h_part.data(), part, sizeof(int) * (k + 1), cudaMemcpyDeviceToHost, st), "parts") ||
      !ok(c, cudaStreamSynchronize(st), "sync"))
    return give_up(TG_ERR_CUDA);
  int most = 0;
  for (int q = 0; q < k; ++q) {
    const int m = h_part[q + 1] - h_part[q];
    if (m <= 0 || m > kHybMaxRows) return give_up(TG_OK);
    most = std::max(most, m);
  }
  int optin = 0;
  cudaFuncAttributes fa;
  const size_t halo_smem = (size_t)(rows + 31) / 32 * 8;
  if (!ok(c, cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device), "attribute") ||
      !ok(c, cudaFuncGetAttributes(&fa, hyb_halo_kernel), "function attributes"))
    return give_up(TG_ERR_CUDA);
  if (halo_smem + fa.sharedSizeBytes > (size_t)optin) return give_up(TG_OK);
  if (!ok(c, cudaFuncSetAttribute(hyb_halo_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  optin - (int)fa.sharedSizeBytes),
          "smem attribute"))
    return give_up(TG_ERR_CUDA);
  hyb_part_sort_kernel<<<k, 1024, 0, st>>>(part, order, rank);
  hyb_rows_kernel<<<(nch + 7) / 8, 256, 0, st>>>(rows, nch, order, c->d_rowptr, c->d_col, c->d_mask, rank,
                                                 c->d_contrib_ptr, slot, cidx, steps, flag);
  hyb_halo_kernel<<<k, 1024, halo_smem, st>>>(rows, part, cidx, halo, nhalo, lcol);
  c->launches += 7;
  int over = 0;
  if (!ok(c, cudaGetLastError(), "hybrid plan kernels") ||
      !ok(c, cudaMemcpyAsync(h_halo.data(), nhalo, sizeof(int) * k, cudaMemcpyDeviceToHost, st), "halo") ||
      !ok(c, cudaMemcpyAsync(&over, flag, sizeof(int), cudaMemcpyDeviceToHost, st), "flag") ||
      !ok(c, cudaStreamSynchronize(st), "sync"))
    return give_up(TG_ERR_CUDA);
  int uw = 0;
  for (int q = 0; q < k; ++q) {
    if (h_halo[q] > kHybHalo) return give_up(TG_OK);
    uw = std::max(uw, h_part[q + 1] - h_part[q] + h_halo[q]);
  }
  if (over || uw > 65535) return give_up(TG_OK);
  const int chcap = (most + 7) / 8;
  for (int blk = 0; blk < 2; ++blk) {
    const void* fn = blk ? reinterpret_cast<const void*>(hybrid_kernel<true>)
                         : reinterpret_cast<const void*>(hybrid_kernel<false>);
    if (!ok(c, cudaFuncGetAttributes(&fa, fn), "function attributes") ||
        !ok(c, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes),
            "smem attribute"))
      return give_up(TG_ERR_CUDA);
    const int cap = optin - (int)fa.sharedSizeBytes;
    // p, s, then the preconditioner (one or three planes) as they fit
    int in = 0;
    for (int want = 1; want <= 3; ++want)
      if (hyb_smem(uw, chcap, want < 3 ? want : 2 + (blk ? 3 : 1)) <= cap) in = want;
    H->in_smem[blk] = in;
    H->smem[blk] = hyb_smem(uw, chcap, in < 3 ? in : 2 + (blk ? 3 : 1));
    if (H->smem[blk] > cap) return give_up(TG_OK);
  }
  float4* stream = nullptr;
  float *xs = nullptr, *state = nullptr;
  uint4* ll = nullptr;
  ResOut* out = nullptr;
  H->ll_words = 4LL * std::min(k, kResCopies) * k + rows;
  if (!hold(&stream, (size_t)nch * kHybVec * 32) || !hold(&xs, (size_t)nch * 32) || !hold(&state, (size_t)nch * 32 * 5) ||
      !hold(&ll, (size_t)H->ll_words) || !hold(&out, 1))
    return give_up(TG_OK);
  H->k = k;
  HybArgs& A = H->A;
  A.row_start = part;
  A.act_node = order;
  A.slot = slot;
  A.lcol = lcol;
  A.steps = steps;
  A.halo = halo;
  A.nhalo = nhalo;
  A.contrib = c->d_contrib;
  A.mask = c->d_mask;
  A.stream = stream;
  A.xs = xs;
  A.state = state;
  A.ll = ll;
  A.out = out;
  A.status = c->d_status;
  A.chunks = nch;
  A.rows = rows;
  A.uwcap = uw;
  A.chcap = chcap;
  A.keep = (float)std::min(1.0, kHybL2Keep / streamed);
  release();
  *fits = true;
  return TG_OK;
}

int hybrid_solve(Context* c, const double4_32a* d_rhs, double rel_tol, int max_it, int precond, int* iters,
                 double* rel_res) {
  HybState& H = *c->hyb;
  int s = pcg_vectors(c, TG_MIXED);
  if (s) return s;
  cudaStream_t st = c->stream;
  const int blk = precond == TG_PRECOND_BLOCK_JACOBI ? 1 : 0;
  HybArgs A = H.A;
  A.Ke = c->d_Ke32;
  A.waits = c->waits;
  A.rhs = d_rhs;
  A.x = (float4*)c->d_x;
  A.sc = c->d_pcg;
  A.in_smem = H.in_smem[blk];
  A.max_it = max_it;
  A.tol = rel_tol;
  if (!ok(c, cudaMemsetAsync(c->d_x, 0, sizeof(float4) * (size_t)c->nnd, st), "x") ||
      !ok(c, cudaMemsetAsync(A.out, 0, sizeof(ResOut), st), "out") ||
      !ok(c, cudaMemsetAsync(A.ll, 0, sizeof(uint4) * (size_t)H.ll_words, st), "exchange"))
    return TG_ERR_CUDA;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)H.k);
  cfg.blockDim = dim3(kHybWarps * 32);
  cfg.dynamicSmemBytes = (size_t)H.smem[blk];
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  c->launches++;
  if (!ok(c, cudaLaunchKernelEx(&cfg, blk ? hybrid_kernel<true> : hybrid_kernel<false>, A), "hybrid_kernel"))
    return TG_ERR_CUDA;
  ResOut o;
  if (!ok(c, cudaMemcpyAsync(&o, A.out, sizeof(o), cudaMemcpyDeviceToHost, st), "out") ||
      !ok(c, cudaStreamSynchronize(st), "pcg sync"))
    return TG_ERR_CUDA;
  PcgScalars h;
  std::memset(&h, 0, sizeof(h));
  h.rr = o.rr;
  h.rr0 = o.rr0;
  h.done = o.done ? o.done : 2;
  h.fail = o.done ? o.fail : 5;  // a wait ran out before the solve reported
  h.iters = o.iters;
  return pcg_finish(c, h, iters, rel_res);
}

}  // namespace tg
