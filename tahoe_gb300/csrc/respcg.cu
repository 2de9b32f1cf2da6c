// Resident PCG, sm_103a: a whole (block-)Jacobi CG solve in one launch with
// the matrix held in shared memory.
//
// A matrix that fits the chip's shared memory is read once per solve instead
// of once per iteration: every CTA assembles the rows of its part straight
// from the element blocks into shared memory and keeps them there, its rows'
// vectors live in registers, and the iterations touch nothing but shared
// memory and the words the CTAs exchange.  Two forms, one kernel body:
//
//   cluster  k <= 16 CTAs of one thread-block cluster per solve; the new
//            search vector and the partial sums go to the other CTAs as
//            asynchronous stores to distributed shared memory that count
//            bytes on the receiver's mbarrier.  A batch of RVEs is one launch
//            per cluster size with one cluster per RVE.
//   grid     k <= #SM CTAs of a cooperative launch (all resident); vector and
//            partial sums travel through L2 as 16-byte words that carry their
//            sequence number, so a reader polls the data itself and no
//            barrier, flag or fence stands between producer and consumer.
//            Larger RVEs of a batch share one launch: every CTA walks its
//            list of (solve, part) pairs in one global order.
//
// The recurrences are the single-reduction form of CG (Chronopoulos & Gear,
// J. Comput. Appl. Math. 25 (1989) 153-168) as in pcg_cg.cu and segpcg.cu:
//   w = A u; delta = u.w, gamma = r.u, r.r in one reduction;
//   beta = gamma / gamma_old, alpha = gamma / (delta - beta gamma / alpha_old);
//   p = u + beta p, s = w + beta s, x += alpha p, r -= alpha s, u = M^-1 r.
// Dot products are the compensated pairs of krylov_common.cuh in the FP32
// form, every sum in a fixed order that depends on the solve's own rows
// alone: a solve is bitwise repeatable and an RVE's does not depend on the
// batch it shares.
//
// Measured against the streamed kernels (product + vector kernel, 14 us an
// iteration on a 37x29x23 block, 20 us on a 16^3 FP64 cube; four kernels and
// 26 us on one RVE of side 8): 7.5, 10.5 and 5 us, with no host round trip
// inside a solve.  What bounds an iteration: the shared-memory reads of the
// values (FP32) or the FP64 pipe, then the latency of the two exchanges.
//
// Rows and storage: a warp holds chunks of 8 consecutive active rows, 4 lanes per row;
// lane l takes blocks l, l+4, ... of its row (sliced ELL per warp: step t of
// a warp is 9 planes of 32 values, unit stride across the lanes, no bank
// conflicts, and 32 16-bit column indices).  After the product lane c < 3 of a
// row owns component c of every vector.  The search vector is kept over the
// part's column window (a contiguous range of active rows).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "assembly.cuh"
#include "ff.cuh"
#include "krylov_common.cuh"
#include "respcg.cuh"

namespace tg {

namespace {

constexpr int kResClusterMax = 16;
constexpr int kResPollLimit = 1 << 21;  // polls of one exchange word before the solve is abandoned

// Shape of a CTA: warps, chunks of 8 rows per warp at most, and the steps of
// a warp's first chunk whose blocks stay in registers.  FP32: 16 warps at 128
// registers keep 16 chunks in registers beside the 27 that fit the shared
// memory, so a solve takes about 0.6 of the CTAs that shared memory alone
// would ask for; a chip's clusters are few when they are large (13 of 10
// CTAs, 8 of 11 or 12, 7 of 13 to 16).  FP64 runs at the rate of the FP64
// pipe (one warp instruction per 64 cycles and scheduler), not of the storage.
template <typename T>
struct ResShape;
template <>
struct ResShape<float> {
  static constexpr int warps = 16, slots = 3, reg = 7;
};
template <>
struct ResShape<double> {
  static constexpr int warps = 16, slots = 1, reg = 0;
};

using u64 = unsigned long long;

// Largest of unsigned values, with the accumulators' interface
struct AccMax {
  unsigned v = 0;
  __device__ __forceinline__ void shfl_merge(int o) { v = max(v, __shfl_xor_sync(0xffffffffu, v, o)); }
};
__device__ __forceinline__ u64 pack_word(const AccMax& a) { return a.v; }
__device__ __forceinline__ void merge_word(AccMax& a, u64 w) { a.v = max(a.v, (unsigned)w); }
__device__ __forceinline__ u64 pack_word(const Acc<float>& a) {
  return (u64)__float_as_uint(a.hi) | ((u64)__float_as_uint(a.lo) << 32);
}
__device__ __forceinline__ u64 pack_word(const Acc<double>& a) { return (u64)__double_as_longlong(a.s); }
__device__ __forceinline__ void merge_word(Acc<float>& a, u64 w) {
  a.merge(__uint_as_float((unsigned)w), __uint_as_float((unsigned)(w >> 32)));
}
__device__ __forceinline__ void merge_word(Acc<double>& a, u64 w) { a.add(__longlong_as_double((long long)w)); }

// 16-byte exchange words with a sequence number in the last four bytes
__device__ __forceinline__ void st_word(uint4* p, u64 a, u64 b) {
  asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}\n" ::"l"(p), "l"(a),
               "l"(b)
               : "memory");
}
__device__ __forceinline__ void ld_word(const uint4* p, u64& a, u64& b) {
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}\n"
               : "=l"(a), "=l"(b)
               : "l"(p)
               : "memory");
}
__device__ __forceinline__ unsigned word_seq(u64 b) { return (unsigned)(b >> 32); }
// the vector of one row: one word in FP32, two in FP64
template <typename T>
struct RowWords;
template <>
struct RowWords<float> {
  static constexpr int n = 1;
  static __device__ __forceinline__ void store(uint4* p, float x, float y, float z, unsigned seq) {
    st_word(p, (u64)__float_as_uint(x) | ((u64)__float_as_uint(y) << 32),
            (u64)__float_as_uint(z) | ((u64)seq << 32));
  }
  static __device__ __forceinline__ bool load(const uint4* p, unsigned seq, float& x, float& y, float& z) {
    u64 a, b;
    ld_word(p, a, b);
    x = __uint_as_float((unsigned)a);
    y = __uint_as_float((unsigned)(a >> 32));
    z = __uint_as_float((unsigned)b);
    return word_seq(b) == seq;
  }
};
template <>
struct RowWords<double> {
  static constexpr int n = 2;
  static __device__ __forceinline__ void store(uint4* p, double x, double y, double z, unsigned seq) {
    const u64 c = (u64)__double_as_longlong(z);
    st_word(p, (u64)__double_as_longlong(x), (c & 0xffffffffull) | ((u64)seq << 32));
    st_word(p + 1, (u64)__double_as_longlong(y), (c >> 32) | ((u64)seq << 32));
  }
  static __device__ __forceinline__ bool load(const uint4* p, unsigned seq, double& x, double& y, double& z) {
    u64 v0, v1, b0, b1;
    ld_word(p, v0, b0);
    ld_word(p + 1, v1, b1);
    x = __longlong_as_double((long long)v0);
    y = __longlong_as_double((long long)v1);
    z = __longlong_as_double((long long)((b0 & 0xffffffffull) | (b1 << 32)));
    return word_seq(b0) == seq && word_seq(b1) == seq;
  }
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ unsigned cluster_map(unsigned addr, int rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// stores to a CTA of the cluster that count towards its mbarrier's bytes
__device__ __forceinline__ void st_async(unsigned addr, unsigned bar, u64 v) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr), "l"(v),
               "r"(bar)
               : "memory");
}
__device__ __forceinline__ void st_async_row(unsigned addr, unsigned bar, float x, float y, float z) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                   addr),
               "f"(x), "f"(y), "f"(z), "f"(0.f), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void st_async_row(unsigned addr, unsigned bar, double x, double y, double z) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(addr),
               "d"(x), "d"(y), "r"(bar)
               : "memory");
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(
                   addr + 16u),
               "d"(z), "d"(0.0), "r"(bar)
               : "memory");
}
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, unsigned parity) {
  for (int i = 0; i < kWaitLimit; ++i) {
    unsigned ready;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, "
        "p;\n}\n"
        : "=r"(ready)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    if (ready) return true;
  }
  return false;
}

template <typename T>
struct ResArgs {
  const ResPlanDev* plans;
  const ResItem* items;
  const int* sched_ptr;  // grid form: CTA's first (item, part) pair
  const int2* sched;
  int k;                 // cluster form: CTAs per solve
  const T* Ke;
  const uint8_t* mask;
  const double4_32a* rhs;
  typename Vec4<T>::type* x;
  ResOut* out;
  uint4* ll;             // grid form: exchange words, zero before the launch
  PcgScalars* sc;        // receives unscale (single solve) or 1 (batch)
  int* status;
  int batch;             // the solution is unscaled in place
  int max_it;
  double tol;
};

// CTA-wide state of one solve
template <typename T>
struct ResShared {
  uint64_t bar_u;                    // cluster form: the window's rows of this iteration
  uint64_t bar_s[2];                 // cluster form: the CTAs' sums, by parity
  int4 peer[kResClusterMax];         // {first column, columns, window address, bar_u address} of every part
  u64 red[3][16 * 8];                // sums of every row quad of lanes
  u64 slot[2][kResClusterMax][3];    // the CTAs' sums by parity
  u64 tot[3];                        // totals
  T coef[2];                         // alpha, beta
  // the recurrence's scalars (thread 0): gamma and alpha of the last update,
  // convergence threshold, r.r now and at the start
  u64 rz, al, thr, rr, rr0;
  int code, fail;
  int abort_flag;
};

// Totals of three accumulators over every row of the solve, left in sh.tot:
// lanes, warps and CTAs in a fixed order.  seq numbers the reductions of a
// solve from 1.  On return warp 0 sees sh.tot.
//
// Each row's four lanes hold the terms of their component; two levels give the
// row sums, lane v of a row then stores value v, and warp v adds the rows' v
// sums: merging compensated pairs costs about nine instructions a level, so
// the levels a full warp tree would run mostly on idle lanes are replaced by
// one pass over shared memory.
template <typename A, typename T, bool GRID>
__device__ __forceinline__ void total3(A (&a)[3], ResShared<T>& sh, int k, int rank, unsigned seq, uint4* inbox) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int v = 0; v < 3; ++v) {
    a[v].shfl_merge(1);
    a[v].shfl_merge(2);
  }
  if ((lane & 3) < 3) {
    const A& m = (lane & 3) == 0 ? a[0] : (lane & 3) == 1 ? a[1] : a[2];
    sh.red[lane & 3][warp * 8 + (lane >> 2)] = pack_word(m);
  }
  __syncthreads();
  const int par = seq & 1;
  if (warp < 3) {
    A t;
    for (int j = lane; j < nw * 8; j += 32) merge_word(t, sh.red[warp][j]);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) t.shfl_merge(o);
    const u64 w = pack_word(t);
    if (k == 1) {
      if (lane == 0) sh.tot[warp] = w;
    } else if (GRID) {
      // to every CTA's inbox; each polls its own, so no line is read by more
      // than one SM (152 SMs polling the same lines queued at their L2
      // slices: 4.8 us a reduction)
      for (int q = lane; q < k; q += 32) st_word(inbox + (((size_t)q * 2 + par) * k + rank) * 3 + warp, w, (u64)seq << 32);
      A g;
      for (int i = lane; i < k; i += 32) {
        u64 x, y;
        int tries = 0;
        for (;;) {
          ld_word(inbox + (((size_t)rank * 2 + par) * k + i) * 3 + warp, x, y);
          if (word_seq(y) == seq) break;
          if (++tries >= kResPollLimit) {
            sh.abort_flag = 1;
            break;
          }
        }
        merge_word(g, x);
      }
      __syncwarp();
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) g.shfl_merge(o);
      if (lane == 0) sh.tot[warp] = pack_word(g);
    } else if (lane < k) {
      st_async(cluster_map(smem_addr(&sh.slot[par][rank][warp]), lane), cluster_map(smem_addr(&sh.bar_s[par]), lane), w);
    }
    if (k == 1 || GRID) {
      asm volatile("bar.sync 1, 96;" ::: "memory");
    } else if (warp == 0) {
      if (!mbar_wait_cluster(&sh.bar_s[par], ((seq - 1) >> 1) & 1)) sh.abort_flag = 1;
      __syncwarp();
      if (lane == 0) mbar_expect_tx(&sh.bar_s[par], 24u * (unsigned)k);  // of its next use
      // lane v * 8 + i adds the sums of CTAs i and i + 8
      A g;
      const int v = lane >> 3, i = lane & 7;
      if (v < 3) {
        if (i < k) merge_word(g, sh.slot[par][i][v]);
        if (i + 8 < k) merge_word(g, sh.slot[par][i + 8][v]);
      }
      g.shfl_merge(1);
      g.shfl_merge(2);
      g.shfl_merge(4);
      if (v < 3 && i == 0) sh.tot[v] = pack_word(g);
      __syncwarp();
    }
  }
}

// The recurrence's scalars from the totals delta = u.w, gamma = r.u, r.r
// (thread 0): convergence, breakdown, alpha and beta.  FP32 form: in
// double-float, from the same compensated pairs (an FP64 operation takes 64
// cycles here and its division 570: 2,200 cycles of every iteration), with
// alpha = gamma / (delta - gamma (gamma / (gamma_old alpha_old))) so that no
// squares leave FP32's range; alpha and beta are rounded to FP32 for the
// update in both.
__device__ __forceinline__ void scalars(ResShared<float>& sh, int it, int max_it, double tol) {
  using namespace ff;
  auto get = [](u64 w) { return fast_two_sum(__uint_as_float((unsigned)w), __uint_as_float((unsigned)(w >> 32))); };
  auto put = [](dfloat d) { return (u64)__float_as_uint(d.hi) | ((u64)__float_as_uint(d.lo) << 32); };
  const dfloat delta = get(sh.tot[0]), gamma = get(sh.tot[1]), rr = get(sh.tot[2]);
  if (it == 0) {
    sh.rr0 = put(rr);
    sh.thr = put(from_double(tol * tol * to_double(rr)));
  }
  const dfloat thr = get(sh.thr);
  sh.rr = put(rr);
  int code = 0, fail = 0;
  dfloat alpha = make(0.f, 0.f), beta = make(0.f, 0.f);
  if (sh.abort_flag) {
    code = 2;
    fail = 5;
  } else if (!isfinite(gamma.hi) || !isfinite(rr.hi)) {
    code = 2;
    fail = it == 0 ? 1 : 4;
  } else if (it == 0 ? rr.hi == 0.f : (rr.hi < thr.hi || (rr.hi == thr.hi && rr.lo <= thr.lo))) {
    code = 1;
  } else if (it >= max_it) {
    code = 3;
  } else {
    dfloat den = delta;
    if (it > 0) {
      const dfloat rz = get(sh.rz);
      beta = mul(gamma, rcp(rz));
      den = sub(delta, mul(gamma, mul(beta, rcp(get(sh.al)))));
    }
    if (!(den.hi > 0.f) || !isfinite(den.hi)) {
      code = 2;
      fail = isfinite(den.hi) ? 2 : 3;
    } else {
      alpha = mul(gamma, rcp(den));
    }
  }
  sh.rz = put(gamma);
  sh.al = put(alpha);
  sh.coef[0] = alpha.hi;
  sh.coef[1] = beta.hi;
  sh.code = code;
  sh.fail = fail;
}
__device__ __forceinline__ void scalars(ResShared<double>& sh, int it, int max_it, double tol) {
  auto get = [](u64 w) { return __longlong_as_double((long long)w); };
  auto put = [](double d) { return (u64)__double_as_longlong(d); };
  const double delta = get(sh.tot[0]), gamma = get(sh.tot[1]), rr = get(sh.tot[2]);
  if (it == 0) {
    sh.rr0 = put(rr);
    sh.thr = put(tol * tol * rr);
  }
  sh.rr = put(rr);
  int code = 0, fail = 0;
  double alpha = 0.0, beta = 0.0;
  if (sh.abort_flag) {
    code = 2;
    fail = 5;
  } else if (!isfinite(gamma) || !isfinite(rr)) {
    code = 2;
    fail = it == 0 ? 1 : 4;
  } else if (it == 0 ? rr == 0.0 : rr <= get(sh.thr)) {
    code = 1;
  } else if (it >= max_it) {
    code = 3;
  } else {
    double num = gamma, den = delta;
    if (it > 0) {
      const double rz = get(sh.rz), t = rz * get(sh.al);
      beta = gamma / rz;
      num = gamma * t;
      den = delta * t - gamma * gamma;
    }
    if (!(den > 0.0) || !isfinite(den)) {
      code = 2;
      fail = isfinite(den) ? 2 : 3;
    } else {
      alpha = num / den;
    }
  }
  sh.rz = put(gamma);
  sh.al = put(alpha);
  sh.coef[0] = alpha;
  sh.coef[1] = beta;
  sh.code = code;
  sh.fail = fail;
}
__device__ __forceinline__ double word_value(const ResShared<float>&, u64 w) {
  return (double)__uint_as_float((unsigned)w) + (double)__uint_as_float((unsigned)(w >> 32));
}
__device__ __forceinline__ double word_value(const ResShared<double>&, u64 w) { return __longlong_as_double((long long)w); }

// biased exponents
__device__ __forceinline__ unsigned exponent_of(double v) { return ((unsigned)__double2hiint(v) >> 20) & 0x7ffu; }
// 2^e, |e| <= 1000
__device__ __forceinline__ double power_of_two(int e) { return __hiloint2double((e + 1023) << 20, 0); }

// One block's value: its contributions in ascending order as in block_value,
// two element blocks in flight.
template <typename T>
__device__ __forceinline__ void slot_value(int2 sl, uint8_t mI, const int* __restrict__ contrib,
                                           const T* __restrict__ Ke, int elem_off, T acc[9]) {
  using V4 = typename std::conditional<sizeof(T) == 4, float4, double4_32a>::type;
#pragma unroll
  for (int q = 0; q < 9; ++q) acc[q] = T(0);
  auto src = [&](int code) {
    const int e = (code >> 6) + elem_off, a = (code >> 3) & 7, b = code & 7;
    return reinterpret_cast<const V4*>(Ke + ((long long)e * kSlots + (a <= b ? upper_slot(a, b) : upper_slot(b, a))) *
                                                kKeBlock);
  };
  auto add = [&](int code, const V4& k0, const V4& k1, const V4& k2) {
    const bool up = ((code >> 3) & 7) <= (code & 7);
    acc[0] += k0.x;
    acc[1] += up ? k0.y : k1.x;
    acc[2] += up ? k0.z : k2.x;
    acc[3] += up ? k1.x : k0.y;
    acc[4] += k1.y;
    acc[5] += up ? k1.z : k2.y;
    acc[6] += up ? k2.x : k0.z;
    acc[7] += up ? k2.y : k1.z;
    acc[8] += k2.z;
  };
  const int* cd = contrib + sl.x;
  for (int i = 0; i < sl.y; i += 2) {
    const int c0 = cd[i], c1 = i + 1 < sl.y ? cd[i + 1] : c0;
    const V4 *s0 = src(c0), *s1 = src(c1);
    const V4 a0 = s0[0], a1 = s0[1], a2 = s0[2], b0 = s1[0], b1 = s1[1], b2 = s1[2];
    add(c0, a0, a1, a2);
    if (i + 1 < sl.y) add(c1, b0, b1, b2);
  }
#pragma unroll
  for (int p = 0; p < 3; ++p)
    if (!((mI >> p) & 1))
#pragma unroll
      for (int q = 0; q < 3; ++q) acc[p * 3 + q] = T(0);
}

// One CTA's part of one solve.
template <typename T, bool GRID, bool BLK>
__device__ __forceinline__ void resident_solve(const ResArgs<T>& A, const ResItem& I, int item, int rank,
                                               unsigned char* smem, ResShared<T>& sh) {
  using V = typename Vec4<T>::type;
  constexpr int NS = ResShape<T>::slots, RB = ResShape<T>::reg, RA = RB > 0 ? RB : 1, NM = BLK ? 3 : 1;
  const ResPlanDev P = A.plans[I.plan];
  const int k = P.k;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5, c = lane & 3, q0 = lane & ~3;
  const int ch0 = P.part_chunk[rank], nch = P.part_chunk[rank + 1] - ch0;
  const int4 win = P.part_win[rank];
  const int row0 = ch0 * kResChunkRows, row1 = min(P.rows, (ch0 + nch) * kResChunkRows);
  // shared memory: the window [columns][4], the values that are not in
  // registers [steps][9][32], the column indices of every step [steps][32]
  V* uw = reinterpret_cast<V*>(smem);
  const int steps0 = P.chunk_step[ch0], allsteps = P.chunk_step[ch0 + nch] - steps0;
  int vstep[NS], cstep[NS], nst[NS];  // first value step, first index step, steps of this warp's chunks
  int vsteps = 0;                     // value steps in shared memory
  {
    // the first nw chunks keep RB steps in registers
    int pre = 0, mine = 0;
    for (int i = 0; i < min(nw, nch); ++i) {
      if (i == warp) mine = pre;
      pre += max(0, P.chunk_step[ch0 + i + 1] - P.chunk_step[ch0 + i] - RB);
    }
    const int first = nch > nw ? P.chunk_step[ch0 + nw] : P.chunk_step[ch0 + nch];
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      const int i = warp + q * nw;
      const bool on = i < nch;
      const int s0 = on ? P.chunk_step[ch0 + i] : 0;
      nst[q] = on ? P.chunk_step[ch0 + i + 1] - s0 : 0;
      cstep[q] = on ? s0 - steps0 : 0;
      vstep[q] = q == 0 ? mine : (on ? pre + s0 - first : 0);
    }
    vsteps = pre + (steps0 + allsteps - first);
  }
  T* vals = reinterpret_cast<T*>(uw + win.y);
  uint16_t* cols = reinterpret_cast<uint16_t*>(vals + (size_t)vsteps * 9 * 32);
  uint4* inbox = GRID ? A.ll + I.ll : nullptr;                         // partial sums
  uint4* urow = GRID ? inbox + 6 * (size_t)k * k : nullptr;            // rows' vectors
  for (int i = threadIdx.x; i < 3 * 128; i += blockDim.x) (&sh.red[0][0])[i] = 0;
  if (threadIdx.x == 0) sh.abort_flag = 0;
  if (!GRID && k > 1) {
    if (threadIdx.x < k) {
      const int4 wq = P.part_win[threadIdx.x];
      sh.peer[threadIdx.x] = make_int4(wq.x, wq.y, (int)cluster_map(smem_addr(smem), threadIdx.x),
                                       (int)cluster_map(smem_addr(&sh.bar_u), threadIdx.x));
    }
    if (threadIdx.x == 0) {
      mbar_init(&sh.bar_u, (unsigned)nw);
      mbar_init(&sh.bar_s[0], 1);
      mbar_init(&sh.bar_s[1], 1);
      fence_mbar_init();
      mbar_expect_tx(&sh.bar_s[0], 24u * (unsigned)k);
      mbar_expect_tx(&sh.bar_s[1], 24u * (unsigned)k);
    }
    __syncwarp();
    cluster_arrive();  // every CTA of the cluster has its barriers before data is sent
    cluster_wait();
  }
  // --- the rows of the part, assembled from the element blocks
  T rv[RA][9];
  T Mi[NS][NM];
  unsigned comp = 0;  // bit q: this lane's component of its row in chunk q is a free dof
  bool live[NS];
#pragma unroll
  for (int q = 0; q < NS; ++q) {
    const int row = (ch0 + warp + q * nw) * kResChunkRows + (lane >> 2);
    live[q] = nst[q] > 0 && row < P.rows;
    const uint8_t m = live[q] ? A.mask[I.node_off + P.act_node[row]] : 0;
    if (c < 3 && ((m >> c) & 1)) comp |= 1u << q;
    T D[9];
    bool have = false;
    auto block = [&](int t, T acc[9]) {
      const int i = (steps0 + cstep[q] + t) * 32 + lane;
      const int cl = P.col[i];
      slot_value<T>(P.slot[i], m, P.contrib, A.Ke, I.elem_off, acc);
      cols[(size_t)(cstep[q] + t) * 32 + lane] = (uint16_t)(cl - win.x);
      if (cl == row && P.slot[i].y > 0) {
        have = true;
#pragma unroll
        for (int e = 0; e < 9; ++e) D[e] = acc[e];
      }
    };
#pragma unroll
    for (int e = 0; e < 9; ++e) D[e] = T(0);
    if (q == 0 && RB > 0) {
#pragma unroll
      for (int t = 0; t < RB; ++t) {
        if (t < nst[0]) {
          block(t, rv[t]);
        } else {
#pragma unroll
          for (int e = 0; e < 9; ++e) rv[t][e] = T(0);
        }
      }
    }
    for (int t = q == 0 ? RB : 0; t < nst[q]; ++t) {
      T acc[9];
      block(t, acc);
      T* vp = vals + (size_t)(vstep[q] + t - (q == 0 ? RB : 0)) * 9 * 32 + lane;
#pragma unroll
      for (int e = 0; e < 9; ++e) vp[32 * e] = acc[e];
    }
    // the row's preconditioner from the lane that holds its diagonal block
    const unsigned who = (__ballot_sync(0xffffffffu, have) >> q0) & 0xfu;
    const int src = q0 + (who ? __ffs((int)who) - 1 : 0);
    T Dg[9], B[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) D[e] = __shfl_sync(0xffffffffu, D[e], src);
    diagonal_inverses<T>(m, D, Dg, B);
#pragma unroll
    for (int d = 0; d < NM; ++d) {
      if (BLK)
        Mi[q][d] = c == 0 ? B[d] : c == 1 ? B[3 + d] : c == 2 ? B[6 + d] : T(0);
      else
        Mi[q][d] = c == 0 ? Dg[0] : c == 1 ? Dg[4] : c == 2 ? Dg[8] : T(0);
      if (!who || !live[q]) Mi[q][d] = T(0);
    }
  }
  auto precond = [&](int q, T rq) {
    if (!BLK) return Mi[q][0] * rq;
    T z = T(0);
#pragma unroll
    for (int d = 0; d < NM; ++d) z += Mi[q][d] * __shfl_sync(0xffffffffu, rq, q0 + d);
    return z;
  };
  unsigned seq = 0;
  T r[NS], p[NS], s[NS], x[NS], u[NS];
  int scale_exp = 0;
  {
    // --- the right-hand side on a power of two near its size: first by its
    // largest entry, then by the largest r . M^-1 r (products of late Newton
    // residuals would leave FP32's range)
    double b[NS];
    AccMax a[3];
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      const int row = (ch0 + warp + q * nw) * kResChunkRows + (lane >> 2);
      b[q] = ((comp >> q) & 1) ? reinterpret_cast<const double*>(A.rhs + (I.node_off + P.act_node[row]))[c] : 0.0;
      a[0].v = max(a[0].v, exponent_of(b[q]));
    }
    ++seq;
    total3<AccMax, T, GRID>(a, sh, k, rank, seq, inbox);
    __syncthreads();
    const int e1 = (int)sh.tot[0];
    if (e1 > 0 && e1 < 0x7ff) scale_exp = max(-1000, min(1000, 1023 - e1));
    double sc = power_of_two(scale_exp);
    a[0].v = a[1].v = a[2].v = 0;
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      const T rq = T(b[q] * sc);
      a[0].v = max(a[0].v, exponent_of((double)(rq * precond(q, rq))));
    }
    __syncthreads();  // sh.tot and sh.red are read
    ++seq;
    total3<AccMax, T, GRID>(a, sh, k, rank, seq, inbox);
    __syncthreads();
    const int e2 = (int)sh.tot[0];
    if (e2 > 0 && e2 < 0x7ff && e1 > 0 && e1 < 0x7ff) scale_exp = max(-1000, min(1000, scale_exp - (e2 - 1023) / 2));
    sc = power_of_two(scale_exp);
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      r[q] = T(b[q] * sc);
      p[q] = s[q] = x[q] = T(0);
      u[q] = precond(q, r[q]);
    }
    __syncthreads();
  }
  // --- iterations
  int it = 0;
  for (;; ++it) {
    // the new search vector to every CTA whose window holds its rows
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      if (q * nw >= nch) break;
      const T u1 = __shfl_down_sync(0xffffffffu, u[q], 1), u2 = __shfl_down_sync(0xffffffffu, u[q], 2);
      if (live[q] && c == 0) {
        const int row = (ch0 + warp + q * nw) * kResChunkRows + (lane >> 2);
        uw[row - win.x] = mk<V, T>(u[q], u1, u2);
        if (k > 1) {
          if (GRID) {
            RowWords<T>::store(urow + (size_t)row * RowWords<T>::n, u[q], u1, u2, (unsigned)it + 1u);
          } else {
            for (int o = win.z; o <= win.w; ++o) {
              if (o == rank) continue;
              const int4 pq = sh.peer[o];
              const int at = row - pq.x;
              if (at >= 0 && at < pq.y)
                st_async_row((unsigned)pq.z + (unsigned)(at * (int)sizeof(V)), (unsigned)pq.w, u[q], u1, u2);
            }
          }
        }
      }
    }
    __syncwarp();
    if (GRID && k > 1) {
      // the other parts' rows of the window: below and above this part's
      const int below = row0 - win.x, away = win.y - (row1 - row0);
      for (int i = threadIdx.x; i < away; i += blockDim.x) {
        const int at = i < below ? i : i + (row1 - row0);
        const uint4* w = urow + (size_t)(win.x + at) * RowWords<T>::n;
        T x0, x1, x2;
        int tries = 0;
        while (!RowWords<T>::load(w, (unsigned)it + 1u, x0, x1, x2))
          if (++tries >= kResPollLimit) {
            sh.abort_flag = 1;
            break;
          }
        uw[at] = mk<V, T>(x0, x1, x2);
      }
      __syncthreads();
    } else if (!GRID && k > 1) {
      if (lane == 0) {
        if (warp == 0)
          mbar_expect_tx(&sh.bar_u, (unsigned)((win.y - (row1 - row0)) * (int)sizeof(V)));
        else
          mbar_arrive(&sh.bar_u);
      }
      if (!mbar_wait_cluster(&sh.bar_u, (unsigned)it & 1u)) sh.abort_flag = 1;
      __syncwarp();
    } else {
      __syncthreads();
    }
    // w = A u, one chunk after the other; component c of a row on its lane c
    T w[NS];
    Acc<T> a[3];
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      w[q] = T(0);
      if (q * nw >= nch) break;
      T a0 = T(0), a1 = T(0), a2 = T(0);
      const uint16_t* cp = cols + (size_t)cstep[q] * 32 + lane;
      if (q == 0 && RB > 0) {
#pragma unroll
        for (int t = 0; t < RB; ++t)
          if (t < nst[0]) {
            const V uj = uw[cp[32 * t]];
            a0 += rv[t][0] * uj.x + rv[t][1] * uj.y + rv[t][2] * uj.z;
            a1 += rv[t][3] * uj.x + rv[t][4] * uj.y + rv[t][5] * uj.z;
            a2 += rv[t][6] * uj.x + rv[t][7] * uj.y + rv[t][8] * uj.z;
          }
        cp += 32 * RB;
      }
      const T* vp = vals + (size_t)vstep[q] * 9 * 32 + lane;
#pragma unroll 4
      for (int t = q == 0 ? RB : 0; t < nst[q]; ++t, vp += 9 * 32, cp += 32) {
        const V uj = uw[*cp];
        a0 += vp[0] * uj.x + vp[32] * uj.y + vp[64] * uj.z;
        a1 += vp[96] * uj.x + vp[128] * uj.y + vp[160] * uj.z;
        a2 += vp[192] * uj.x + vp[224] * uj.y + vp[256] * uj.z;
      }
      // lanes 0, 1 of a row keep components 0 and 1, lanes 2, 3 component 2
      const bool up = (c & 2) != 0;
      const T g0 = __shfl_xor_sync(0xffffffffu, up ? a0 : a2, 2);
      const T g1 = __shfl_xor_sync(0xffffffffu, a1, 2);
      const T b0 = (up ? a2 : a0) + g0;
      const T b1 = a1 + g1;
      const T e = __shfl_xor_sync(0xffffffffu, up ? b0 : ((c & 1) ? b0 : b1), 1);
      w[q] = up ? b0 + e : ((c & 1) ? b1 + e : b0 + e);
      if ((comp >> q) & 1) {
        a[0].add_prod(u[q], w[q]);
        a[1].add_prod(r[q], u[q]);
        a[2].add_prod(r[q], r[q]);
      }
    }
    ++seq;
    total3<Acc<T>, T, GRID>(a, sh, k, rank, seq, inbox);
    if (threadIdx.x == 0) scalars(sh, it, A.max_it, A.tol);
    __syncthreads();
    if (sh.code) break;
    const T al = sh.coef[0], be = sh.coef[1];
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      if (q * nw >= nch) break;
      p[q] = u[q] + be * p[q];
      s[q] = w[q] + be * s[q];
      x[q] += al * p[q];
      r[q] -= al * s[q];
      u[q] = precond(q, r[q]);
    }
  }
  const double unscale = power_of_two(-scale_exp);
  const int code = sh.code;
#pragma unroll
  for (int q = 0; q < NS; ++q) {
    T xq = x[q];
    if (A.batch) xq = code == 2 ? T(0) : xq * T(unscale);
    const T x1 = __shfl_down_sync(0xffffffffu, xq, 1), x2 = __shfl_down_sync(0xffffffffu, xq, 2);
    const int row = (ch0 + warp + q * nw) * kResChunkRows + (lane >> 2);
    if (live[q] && c == 0) A.x[I.node_off + P.act_node[row]] = mk<V, T>(xq, x1, x2);
  }
  if (threadIdx.x == 0) {
    if (sh.fail == 5) atomicOr(A.status, kStatusWaitTimeout);
    if (rank == 0) {
      ResOut o;
      o.rr = word_value(sh, sh.rr);
      o.rr0 = word_value(sh, sh.rr0);
      o.unscale = unscale;
      o.done = code;
      o.fail = sh.fail;
      o.iters = it;
      o.pad = 0;
      A.out[item] = o;
      A.sc->unscale = A.batch ? 1.0 : unscale;
    }
  }
  if (!GRID && k > 1) {
    __syncwarp();
    cluster_arrive();  // no CTA leaves while data is on its way to it
    cluster_wait();
  } else {
    __syncthreads();
  }
}

template <typename T, bool BLK>
__global__ void __launch_bounds__(ResShape<T>::warps * 32, 1) resident_cluster_kernel(ResArgs<T> A) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ ResShared<T> sh;
  const int item = blockIdx.x / A.k, rank = blockIdx.x % A.k;
  resident_solve<T, false, BLK>(A, A.items[item], item, rank, smem, sh);
}

template <typename T, bool BLK>
__global__ void __launch_bounds__(ResShape<T>::warps * 32, 1) resident_grid_kernel(ResArgs<T> A) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ ResShared<T> sh;
  for (int e = A.sched_ptr[blockIdx.x]; e < A.sched_ptr[blockIdx.x + 1]; ++e) {
    const int2 w = A.sched[e];
    resident_solve<T, true, BLK>(A, A.items[w.x], w.x, w.y, smem, sh);
    const bool stop = sh.abort_flag != 0;
    __syncthreads();
    if (stop) return;  // a wait ran out: nothing more is awaited
  }
}

// contribution range of every slot of a plan's rows
__global__ void resident_slots_kernel(long long n, const int* __restrict__ blk, const int* __restrict__ cptr,
                                      int2* __restrict__ slot) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int j = blk[i];
  slot[i] = j < 0 ? make_int2(0, 0) : make_int2(cptr[j], cptr[j + 1] - cptr[j]);
}

// ---- planning ---------------------------------------------------------------

// Dynamic shared memory of one CTA and the largest cluster that can run with it.
template <typename T>
int limits_t(Context* c, size_t* cap, int* cluster) {
  int optin = 0;
  cudaFuncAttributes fa;
  if (!ok(c, cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device), "attribute"))
    return TG_ERR_CUDA;
  size_t smem = (size_t)optin;
  for (const void* fn : {reinterpret_cast<const void*>(resident_cluster_kernel<T, false>),
                         reinterpret_cast<const void*>(resident_cluster_kernel<T, true>),
                         reinterpret_cast<const void*>(resident_grid_kernel<T, false>),
                         reinterpret_cast<const void*>(resident_grid_kernel<T, true>)}) {
    if (!ok(c, cudaFuncGetAttributes(&fa, fn), "function attributes")) return TG_ERR_CUDA;
    smem = std::min(smem, (size_t)optin - fa.sharedSizeBytes);
    // one value for every caller: other contexts may configure and launch it
    if (!ok(c, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes),
            "smem attribute"))
      return TG_ERR_CUDA;
  }
  *cap = smem;
  *cluster = 1;
  const void* fn = reinterpret_cast<const void*>(resident_cluster_kernel<T, true>);
  if (!ok(c, cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1), "cluster attribute") ||
      !ok(c, cudaFuncSetAttribute(reinterpret_cast<const void*>(resident_cluster_kernel<T, false>),
                                  cudaFuncAttributeNonPortableClusterSizeAllowed, 1),
          "cluster attribute"))
    return TG_ERR_CUDA;
  for (int k = kResClusterMax; k > 1; k /= 2) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(k);
    cfg.blockDim = dim3(ResShape<T>::warps * 32);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = k;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess && n > 0) {
      *cluster = k;
      break;
    }
    cudaGetLastError();
  }
  return TG_OK;
}

}  // namespace

// Active rows, their blocks in sliced-ELL order (row, lane, step) and every
// chunk's columns, from the node-block CSR of nodes [n0, n1); node indices
// in the result are relative to n0, block indices to rowptr[n0]-independent
// positions of the CSR.
void resident_rows(int n0, int n1, const int* rowptr, const int* col, const uint8_t* mask, ResRows& R) {
  const int n = n1 - n0;
  std::vector<int> id(n, -1);
  R = ResRows{};
  for (int i = 0; i < n; ++i)
    if (mask[n0 + i]) {
      id[i] = (int)R.act_node.size();
      R.act_node.push_back(i);
    }
  const int rows = (int)R.act_node.size(), nch = (rows + kResChunkRows - 1) / kResChunkRows;
  R.chunk_step.assign(nch + 1, 0);
  R.chunk_lo.assign(nch, 0);
  R.chunk_hi.assign(nch, 0);
  std::vector<int> jb, jc;  // the active blocks of a chunk's rows, concatenated
  for (int ch = 0; ch < nch; ++ch) {
    const int r0 = ch * kResChunkRows, r1 = std::min(rows, r0 + kResChunkRows);
    int start[kResChunkRows + 1], most = 0, lo = r0, hi = r1;
    jb.clear();
    jc.clear();
    for (int r = r0; r < r1; ++r) {
      start[r - r0] = (int)jb.size();
      const int g = n0 + R.act_node[r];
      for (int j = rowptr[g]; j < rowptr[g + 1]; ++j) {
        const int a = id[col[j] - n0];
        if (a < 0) continue;
        jb.push_back(j);
        jc.push_back(a);
        lo = std::min(lo, a);
        hi = std::max(hi, a + 1);
      }
      start[r - r0 + 1] = (int)jb.size();
      most = std::max(most, (int)jb.size() - start[r - r0]);
    }
    const int nst = (most + 3) / 4, s0 = R.chunk_step[ch];
    R.chunk_step[ch + 1] = s0 + nst;
    R.chunk_lo[ch] = lo;
    R.chunk_hi[ch] = hi;
    R.blk.resize((size_t)(s0 + nst) * 32, -1);
    R.col.resize((size_t)(s0 + nst) * 32, r0);
    for (int r = r0; r < r1; ++r)
      for (int i = start[r - r0]; i < start[r - r0 + 1]; ++i) {
        const int q = i - start[r - r0];
        const size_t at = (size_t)(s0 + (q >> 2)) * 32 + (r - r0) * 4 + (q & 3);
        R.blk[at] = jb[i];
        R.col[at] = jc[i];
      }
  }
}

namespace {

// Bytes of one part with nw warps: the window, the values outside registers
// (the first nw chunks keep `reg` steps there), the columns of every step.
size_t part_bytes(const ResRows& R, int a, int b, int elem, int reg, int nw, int* lo, int* hi) {
  int l = R.chunk_lo[a], h = R.chunk_hi[a];
  size_t vsteps = 0;
  for (int ch = a; ch < b; ++ch) {
    l = std::min(l, R.chunk_lo[ch]);
    h = std::max(h, R.chunk_hi[ch]);
    const int n = R.chunk_step[ch + 1] - R.chunk_step[ch];
    vsteps += ch - a < nw ? std::max(0, n - reg) : n;
  }
  *lo = l;
  *hi = h;
  const size_t steps = (size_t)(R.chunk_step[b] - R.chunk_step[a]);
  return (size_t)(h - l) * 4 * elem + vsteps * 9 * 32 * elem + steps * 64;
}

// The chunks cut into k consecutive parts of near-equal steps; false if one
// exceeds a CTA.
bool split_parts(const ResRows& R, int k, int elem, size_t cap, ResPlan& P) {
  const int nch = (int)R.chunk_lo.size();
  if (k > nch) return false;
  const int warps = elem == 4 ? ResShape<float>::warps : ResShape<double>::warps;
  const int slots = elem == 4 ? ResShape<float>::slots : ResShape<double>::slots;
  const int reg = elem == 4 ? ResShape<float>::reg : ResShape<double>::reg;
  const long long total = R.chunk_step[nch];
  P.part_chunk.assign(k + 1, 0);
  P.part_chunk[k] = nch;
  for (int q = 1; q < k; ++q) {
    const long long target = (total * q + k / 2) / k;
    int ch = (int)(std::lower_bound(R.chunk_step.begin(), R.chunk_step.end(), (int)target) - R.chunk_step.begin());
    if (ch > 0 && target - R.chunk_step[ch - 1] < R.chunk_step[ch] - target) --ch;
    P.part_chunk[q] = std::min(std::max(ch, P.part_chunk[q - 1] + 1), nch - (k - q));
  }
  P.part_win.assign(k, make_int4(0, 0, 0, 0));
  P.smem = 0;
  int most = 0;
  for (int q = 0; q < k; ++q) most = std::max(most, P.part_chunk[q + 1] - P.part_chunk[q]);
  if (most > warps * slots) return false;
  // one chunk per warp while there are warps for it
  P.warps = std::min(warps, (most + 3) / 4 * 4);
  for (int q = 0; q < k; ++q) {
    const int a = P.part_chunk[q], b = P.part_chunk[q + 1];
    int lo, hi;
    const size_t bytes = part_bytes(R, a, b, elem, reg, P.warps, &lo, &hi);
    if (bytes > cap || hi - lo > 65535) return false;
    P.smem = std::max(P.smem, bytes);
    P.part_win[q] = make_int4(lo, hi - lo, q, q);
  }
  // the parts whose windows hold rows of part q
  for (int q = 0; q < k; ++q) {
    const int r0 = P.part_chunk[q] * kResChunkRows, r1 = P.part_chunk[q + 1] * kResChunkRows;
    for (int o = 0; o < k; ++o)
      if (P.part_win[o].x < r1 && P.part_win[o].x + P.part_win[o].y > r0) {
        P.part_win[q].z = std::min(P.part_win[q].z, o);
        P.part_win[q].w = std::max(P.part_win[q].w, o);
      }
  }
  P.k = k;
  return true;
}

}  // namespace

// A split of the rows over CTAs.  A solve of a batch takes the fewest CTAs
// that hold it (every SM has another RVE to solve); a solve alone spreads
// over the chip.  Up to the cluster limit the CTAs are one cluster, above it
// (grid) CTAs of a cooperative launch.
bool resident_plan(const ResRows& R, int elem, int num_sms, size_t cap, int max_cluster, bool alone, ResPlan& P) {
  const int nch = (int)R.chunk_lo.size();
  P.rows = (int)R.act_node.size();
  P.nchunks = nch;
  if (nch == 0) return false;
  const int most = elem == 4 ? ResShape<float>::warps * ResShape<float>::slots
                             : ResShape<double>::warps * ResShape<double>::slots;
  int kmin = 0;
  for (int k = (nch + most - 1) / most; k <= std::min(num_sms, nch) && !kmin; ++k)
    if (split_parts(R, k, elem, cap, P)) kmin = k;
  if (!kmin) return false;
  P.grid = kmin > max_cluster;
  if (alone) {
    // alone: a cluster while its CTAs hold few chunks each (its exchanges are
    // short), else every SM
    const int few = elem == 4 ? 24 : 4;
    P.grid = P.grid || (nch + max_cluster - 1) / max_cluster > few;
    const int k = std::max(kmin, std::min(nch, P.grid ? num_sms : max_cluster));
    if (k != kmin && !split_parts(R, k, elem, cap, P) && !split_parts(R, kmin, elem, cap, P)) return false;
  }
  return true;
}

size_t ResImage::rows_at(const ResRows& R) {
  const size_t at = data.size();
  for (const std::vector<int>* v : {&R.act_node, &R.blk, &R.col, &R.chunk_step})
    data.insert(data.end(), v->begin(), v->end());
  data.resize((data.size() + 3) / 4 * 4, 0);
  return at;
}
size_t ResImage::split_at(const ResPlan& P) {
  const size_t at = data.size();
  const int* w = reinterpret_cast<const int*>(P.part_win.data());
  data.insert(data.end(), w, w + 4 * P.part_win.size());  // 16-byte vectors first
  data.insert(data.end(), P.part_chunk.begin(), P.part_chunk.end());
  data.resize((data.size() + 3) / 4 * 4, 0);
  return at;
}
void resident_bind_rows(ResPlanDev& D, const int* base, size_t at, const ResRows& R) {
  D.act_node = base + at;
  D.blk = D.act_node + R.act_node.size();
  D.col = D.blk + R.blk.size();
  D.chunk_step = D.col + R.col.size();
}
void resident_bind_split(ResPlanDev& D, const int* base, size_t at, const ResPlan& P) {
  D.part_win = reinterpret_cast<const int4*>(base + at);
  D.part_chunk = base + at + 4 * P.part_win.size();
  D.rows = P.rows;
  D.k = P.k;
  D.nchunks = P.nchunks;
}

int resident_limits(Context* c, int precision, size_t* smem, int* cluster) {
  ResState& S = *c->res;
  const int p = precision == TG_MIXED ? 1 : 0;
  if (!S.limits_known[p]) {
    const int s = p ? limits_t<float>(c, &S.smem[p], &S.cluster[p]) : limits_t<double>(c, &S.smem[p], &S.cluster[p]);
    if (s) return s;
    S.limits_known[p] = true;
  }
  *smem = S.smem[p];
  *cluster = S.cluster[p];
  return TG_OK;
}

int resident_slots(Context* c, long long n, const int* d_blk, const int* d_cptr, int2* d_slot) {
  if (n == 0) return TG_OK;
  resident_slots_kernel<<<(unsigned)((n + 255) / 256), 256, 0, c->stream>>>(n, d_blk, d_cptr, d_slot);
  c->launches++;
  return ok(c, cudaGetLastError(), "resident_slots_kernel") ? TG_OK : TG_ERR_CUDA;
}

// The mesh's buffers went back to the pool with it.
void resident_reset(Context* c) {
  if (!c->res) return;
  ResState& S = *c->res;
  for (auto& a : S.mode)
    for (ResMode& m : a) m = ResMode{};
  S.d_items = nullptr;
  S.d_out = nullptr;
  S.items_cap = 0;
  S.d_ll = nullptr;
  S.ll_cap = 0;
  S.d_sched = nullptr;
  S.sched_cap = 0;
}

void resident_destroy(Context* c) {
  if (!c->res) return;
  for (cudaStream_t st : c->res->aux)
    if (st) cudaStreamDestroy(st);
  if (c->res->fork) cudaEventDestroy(c->res->fork);
  for (cudaEvent_t e : c->res->join)
    if (e) cudaEventDestroy(e);
  delete c->res;
  c->res = nullptr;
}

// A new partition into RVEs: the plans of the batch follow it.
void resident_drop_batch(Context* c) {
  if (!c->res) return;
  for (auto& a : c->res->mode) {
    if (a[1].d_plans) dfree(c, a[1].d_plans);
    a[1] = ResMode{};
  }
}

namespace {

// Plans the current mesh: every RVE of a batch (the template's plan for a
// composed mesh) or the whole mesh.  A mesh that does not fit leaves the mode
// at -1 and the streamed solves take it.
int plan_mode(Context* c, int precision, bool batch, ResMode& M) {
  M = ResMode{};
  M.state = -1;
  const int elem = precision == TG_MIXED ? 4 : 8;
  size_t cap = 0;
  int cluster = 1;
  int s = resident_limits(c, precision, &cap, &cluster);
  if (s) return s;
  const int nseg = batch ? c->nseg : 1;
  if (batch && c->inst_segments) {
    std::map<int, int> seen;  // template -> plan
    for (int i = 0; i < nseg; ++i) {
      const int t = c->h_inst_tpl[i];
      auto it = seen.find(t);
      if (it == seen.end()) {
        ResPlan P;
        bool fits = false;
        s = template_resident(c, t, precision, P, fits);
        if (s) return s;
        if (!fits) return TG_OK;
        it = seen.emplace(t, (int)M.plans.size()).first;
        M.plans.push_back(P);
      }
      M.plan_of.push_back(it->second);
    }
  } else {
    if (c->composed && !batch) return TG_OK;  // one solve over a composed batch: streamed
    if (ensure_host_mesh(c)) return TG_ERR_CUDA;
    // a mesh far above the chip's shared memory is not looked at row by row
    if (!batch && (double)c->nnzb * 9 * elem > 1.5 * (double)cap * c->num_sms) return TG_OK;
    std::vector<ResRows> rows(nseg);
    std::vector<uint8_t> mask(c->nnd, 0);
    for (int n = 0; n < c->nnd; ++n)
      for (int d = 0; d < 3; ++d)
        if (c->h_eqnos[(size_t)n * 3 + d] > 0) mask[n] |= (uint8_t)(1u << d);
    ResImage img;
    std::vector<size_t> at_rows(nseg), at_split(nseg);
    for (int i = 0; i < nseg; ++i) {
      const int n0 = batch ? c->h_seg_node[i] : 0, n1 = batch ? c->h_seg_node[i + 1] : c->nnd;
      resident_rows(n0, n1, c->h_rowptr.data(), c->h_col.data(), mask.data(), rows[i]);
      ResPlan P;
      if (!rows[i].act_node.empty() && !resident_plan(rows[i], elem, c->num_sms, cap, cluster, !batch, P)) return TG_OK;
      at_rows[i] = img.rows_at(rows[i]);
      at_split[i] = img.split_at(P);
      M.plans.push_back(P);
      M.plan_of.push_back(i);
    }
    int* d = nullptr;
    if (!dalloc(c, &d, img.data.size())) return TG_ERR_OOM;
    if (!ok(c, cudaMemcpyAsync(d, img.data.data(), sizeof(int) * img.data.size(), cudaMemcpyHostToDevice, c->stream),
            "resident rows") ||
        !ok(c, cudaStreamSynchronize(c->stream), "sync"))
      return TG_ERR_CUDA;
    for (int i = 0; i < nseg; ++i) {
      ResPlanDev& D = M.plans[i].dev;
      resident_bind_rows(D, d, at_rows[i], rows[i]);
      resident_bind_split(D, d, at_split[i], M.plans[i]);
      D.contrib = c->d_contrib;
      int2* slot = nullptr;
      if (!dalloc(c, &slot, std::max<size_t>(rows[i].blk.size(), 1))) return TG_ERR_OOM;
      D.slot = slot;
      s = resident_slots(c, (long long)rows[i].blk.size(), D.blk, c->d_contrib_ptr, slot);
      if (s) return s;
    }
  }
  std::vector<ResPlanDev> dev;
  for (const ResPlan& P : M.plans) dev.push_back(P.dev);
  if (!dalloc(c, &M.d_plans, std::max<size_t>(dev.size(), 1))) return TG_ERR_OOM;
  if (!ok(c, cudaMemcpyAsync(M.d_plans, dev.data(), sizeof(ResPlanDev) * dev.size(), cudaMemcpyHostToDevice, c->stream),
          "resident plans") ||
      !ok(c, cudaStreamSynchronize(c->stream), "sync"))
    return TG_ERR_CUDA;
  M.state = 1;
  return TG_OK;
}

int aux_streams(Context* c) {
  ResState& S = *c->res;
  if (S.fork) return TG_OK;
  for (cudaStream_t& st : S.aux)
    if (!ok(c, cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking), "stream")) return TG_ERR_CUDA;
  for (cudaEvent_t& e : S.join)
    if (!ok(c, cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "event")) return TG_ERR_CUDA;
  return ok(c, cudaEventCreateWithFlags(&S.fork, cudaEventDisableTiming), "event") ? TG_OK : TG_ERR_CUDA;
}

template <typename T>
int grow(Context* c, T** p, long long* cap, long long n) {
  if (n <= *cap && *p) return TG_OK;
  if (*p) dfree(c, *p);
  *p = nullptr;
  if (!dalloc(c, p, (size_t)std::max(n, 1LL))) return TG_ERR_OOM;
  *cap = n;
  return TG_OK;
}

template <typename T>
int solve_resident_t(Context* c, ResMode& M, const double4_32a* d_rhs, double rel_tol, int max_it, int precond,
                     int* iters, double* rel_res) {
  using V = typename Vec4<T>::type;
  const bool batch = c->nseg > 0 && c->seg_pcg_mode;
  const int precision = sizeof(T) == 4 ? TG_MIXED : TG_FP64;
  ResState& S = *c->res;
  int s = pcg_vectors(c, precision);
  if (s) return s;
  cudaStream_t st = c->stream;
  const int nseg = batch ? c->nseg : 1;
  std::vector<uint8_t> act(nseg, 1);
  if (batch && (int)c->seg_active.size() == nseg) act = c->seg_active;
  // launch classes: grid solves together, cluster solves by (CTAs, warps,
  // shared memory), the longest first
  struct Class {
    int k, warps;
    size_t smem;
    std::vector<int> seg;
  };
  std::map<std::vector<long long>, Class> cls;
  std::vector<int> grid_seg;
  for (int i = 0; i < nseg; ++i) {
    const ResPlan& P = M.plans[M.plan_of[i]];
    if (!act[i] || P.rows == 0) continue;
    if (P.grid) {
      grid_seg.push_back(i);
      continue;
    }
    const int w = P.warps;
    const long long b = (long long)((P.smem + 16383) / 16384);
    Class& C = cls[{-(long long)P.k, -w, -b}];
    C.k = P.k;
    C.warps = w;
    C.smem = std::max(C.smem, P.smem);
    C.seg.push_back(i);
  }
  std::vector<ResItem> items;
  auto add = [&](int i, long long ll) {
    const int p = M.plan_of[i];
    ResItem it{p, i, batch ? c->h_seg_node[i] : 0, 0, ll};
    // a template's contribution map counts its own elements; an uploaded
    // mesh's counts the mesh's
    if (batch && c->inst_segments) it.elem_off = c->h_seg_elem[i];
    items.push_back(it);
  };
  std::sort(grid_seg.begin(), grid_seg.end(), [&](int a, int b) {
    const int ka = M.plans[M.plan_of[a]].k, kb = M.plans[M.plan_of[b]].k;
    return ka != kb ? ka > kb : a < b;
  });
  long long ll = 0;
  for (int i : grid_seg) {
    const ResPlan& P = M.plans[M.plan_of[i]];
    add(i, ll);
    ll += 6LL * P.k * P.k + (long long)P.rows * RowWords<T>::n;
  }
  // grid solves in waves: a wave's solves take disjoint CTAs, first fit
  std::vector<std::vector<int2>> lists;
  std::vector<int> sched;
  int grid_warps = 0;
  size_t grid_smem = 0;
  {
    std::vector<int> used;
    std::vector<std::vector<std::pair<int, int>>> wave;  // (item, first CTA)
    for (size_t q = 0; q < grid_seg.size(); ++q) {
      const ResPlan& P = M.plans[M.plan_of[grid_seg[q]]];
      size_t w = 0;
      while (w < used.size() && used[w] + P.k > c->num_sms) ++w;
      if (w == used.size()) {
        used.push_back(0);
        wave.emplace_back();
      }
      wave[w].push_back({(int)q, used[w]});
      used[w] += P.k;
      grid_warps = std::max(grid_warps, P.warps);
      grid_smem = std::max(grid_smem, P.smem);
    }
    if (!used.empty()) lists.resize(*std::max_element(used.begin(), used.end()));
    for (const auto& w : wave)
      for (const auto& e : w)
        for (int r = 0; r < M.plans[M.plan_of[grid_seg[e.first]]].k; ++r)
          lists[e.second + r].push_back(make_int2(e.first, r));
    int at = 0;
    for (const auto& l : lists) {
      sched.push_back(at);
      at += (int)l.size();
    }
    sched.push_back(at);
    if (sched.size() & 1) sched.push_back(0);  // the pairs are 8-byte aligned
    for (const auto& l : lists)
      for (const int2& e : l) {
        sched.push_back(e.x);
        sched.push_back(e.y);
      }
  }
  const size_t n_grid = items.size();
  for (auto& e : cls)
    for (int i : e.second.seg) add(i, 0);
  const int n = (int)items.size();
  long long icap = S.items_cap, ocap = S.items_cap;
  s = grow(c, &S.d_items, &icap, n);
  if (!s) s = grow(c, &S.d_out, &ocap, n);
  if (s) return s;
  S.items_cap = (int)icap;
  if (n_grid) {
    s = grow(c, &S.d_ll, &S.ll_cap, ll);
    if (!s) s = grow(c, &S.d_sched, &S.sched_cap, (long long)sched.size());
    if (s) return s;
  }
  // rows outside every solve (prescribed nodes, RVEs not solved) stay zero
  if (!ok(c, cudaMemsetAsync(c->d_x, 0, sizeof(V) * (size_t)c->nnd, st), "x") ||
      !ok(c, cudaMemsetAsync(S.d_out, 0, sizeof(ResOut) * (size_t)std::max(n, 1), st), "out"))
    return TG_ERR_CUDA;
  if (n == 0) {
    // nothing iterates: a zero update
    const double one = 1.0;
    if (!ok(c, cudaMemcpyAsync(&c->d_pcg->unscale, &one, sizeof(one), cudaMemcpyHostToDevice, st), "unscale") ||
        !ok(c, cudaStreamSynchronize(st), "sync"))
      return TG_ERR_CUDA;
  } else if (!ok(c, cudaMemcpyAsync(S.d_items, items.data(), sizeof(ResItem) * n, cudaMemcpyHostToDevice, st), "items"))
    return TG_ERR_CUDA;
  ResArgs<T> A;
  A.plans = M.d_plans;
  A.items = S.d_items;
  A.sched_ptr = nullptr;
  A.sched = nullptr;
  A.k = 0;
  A.Ke = sizeof(T) == 4 ? (const T*)c->d_Ke32 : (const T*)c->d_Ke64;
  A.mask = c->d_mask;
  A.rhs = d_rhs;
  A.x = (V*)c->d_x;
  A.out = S.d_out;
  A.ll = S.d_ll;
  A.sc = c->d_pcg;
  A.status = c->d_status;
  A.batch = batch ? 1 : 0;
  const bool blk = precond == TG_PRECOND_BLOCK_JACOBI;
  A.max_it = max_it;
  A.tol = rel_tol;
  if (n_grid) {
    if (!ok(c, cudaMemcpyAsync(S.d_sched, sched.data(), sizeof(int) * sched.size(), cudaMemcpyHostToDevice, st),
            "schedule") ||
        !ok(c, cudaMemsetAsync(S.d_ll, 0, sizeof(uint4) * (size_t)ll, st), "exchange"))
      return TG_ERR_CUDA;
    ResArgs<T> G = A;
    G.sched_ptr = S.d_sched;
    G.sched = reinterpret_cast<const int2*>(S.d_sched + (lists.size() + 2) / 2 * 2);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)lists.size());
    cfg.blockDim = dim3(32u * (unsigned)grid_warps);
    cfg.dynamicSmemBytes = grid_smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    c->launches++;
    if (!ok(c, cudaLaunchKernelEx(&cfg, blk ? resident_grid_kernel<T, true> : resident_grid_kernel<T, false>, G),
            "resident_grid_kernel"))
      return TG_ERR_CUDA;
  }
  if (!cls.empty()) {
    // classes side by side: each is small beside the chip's tail otherwise
    const int nst = (int)std::min<size_t>(cls.size(), 4);
    if (nst > 1) {
      s = aux_streams(c);
      if (s) return s;
      if (!ok(c, cudaEventRecord(S.fork, st), "fork")) return TG_ERR_CUDA;
      for (int q = 0; q + 1 < nst; ++q)
        if (!ok(c, cudaStreamWaitEvent(S.aux[q], S.fork, 0), "fork")) return TG_ERR_CUDA;
    }
    size_t first = n_grid;
    int q = 0;
    for (const auto& e : cls) {
      const Class& C = e.second;
      ResArgs<T> B = A;
      B.items = S.d_items + first;
      B.out = S.d_out + first;
      B.k = C.k;
      first += C.seg.size();
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3((unsigned)(C.seg.size() * C.k));
      cfg.blockDim = dim3(32u * (unsigned)C.warps);
      cfg.dynamicSmemBytes = C.smem;
      cfg.stream = q % nst == 0 ? st : S.aux[q % nst - 1];
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = (unsigned)C.k;
      at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      c->launches++;
      if (!ok(c, cudaLaunchKernelEx(&cfg, blk ? resident_cluster_kernel<T, true> : resident_cluster_kernel<T, false>, B),
              "resident_cluster_kernel"))
        return TG_ERR_CUDA;
      ++q;
    }
    for (int a = 0; a + 1 < nst; ++a)
      if (!ok(c, cudaEventRecord(S.join[a], S.aux[a]), "join") || !ok(c, cudaStreamWaitEvent(st, S.join[a], 0), "join"))
        return TG_ERR_CUDA;
  }
  std::vector<ResOut> out(std::max(n, 1));
  if (n && !ok(c, cudaMemcpyAsync(out.data(), S.d_out, sizeof(ResOut) * n, cudaMemcpyDeviceToHost, st), "out"))
    return TG_ERR_CUDA;
  if (!ok(c, cudaStreamSynchronize(st), "pcg sync")) return TG_ERR_CUDA;
  for (int i = 0; i < n; ++i)
    if (out[i].done == 0) {  // a wait ran out before this solve reported
      out[i].done = 2;
      out[i].fail = 5;
    }
  if (!batch) {
    PcgScalars h;
    std::memset(&h, 0, sizeof(h));
    if (n) {
      h.rr = out[0].rr;
      h.rr0 = out[0].rr0;
      h.done = out[0].done;
      h.fail = out[0].fail;
      h.iters = out[0].iters;
    } else {
      h.done = 1;
    }
    return pcg_finish(c, h, iters, rel_res);
  }
  c->have_du = true;
  int worst_it = 0, broke = 0, limit = 0, nact = 0, timeout = 0;
  double worst_rel = 0.0;
  c->seg_status.assign(nseg, TG_OK);
  for (uint8_t a : act) nact += a ? 1 : 0;
  for (int i = 0; i < n; ++i) {
    const ResOut& o = out[i];
    worst_it = std::max(worst_it, o.iters);
    if (o.rr0 > 0.0) worst_rel = std::max(worst_rel, std::sqrt(o.rr / o.rr0));
    if (o.done == 2) {
      c->seg_status[items[i].seg] = TG_ERR_NAN;
      ++broke;
      timeout += o.fail == 5 ? 1 : 0;
    } else if (o.done != 1) {
      c->seg_status[items[i].seg] = TG_ERR_NOT_CONVERGED;
      ++limit;
    }
  }
  if (iters) *iters = worst_it;
  if (rel_res) *rel_res = worst_rel;
  if (timeout) {
    c->err = "PCG breakdown: exchange wait timed out";
    return TG_ERR_NAN;
  }
  if (broke && (!c->seg_tolerate || broke == nact)) {
    c->err = "PCG breakdown in " + std::to_string(broke) + " of " + std::to_string(nact) + " RVEs";
    return TG_ERR_NAN;
  }
  if (limit) {
    c->err = "PCG iteration limit reached in " + std::to_string(limit) + " RVEs";
    return TG_ERR_NOT_CONVERGED;
  }
  return TG_OK;
}

}  // namespace

// The default form solves resident where the mesh (every RVE of the batch)
// fits; the explicit forms of tg_pcg_form and the symmetric format keep their
// own kernels.
int resident_active(Context* c, int precision, bool* on) {
  *on = false;
  if (c->cg_push >= 0 || c->pcg_form != 1 || !c->cg_pdl || sym_active(c)) return TG_OK;
  if (precision != TG_MIXED && precision != TG_FP64) return TG_OK;
  if (!c->res) c->res = new ResState();
  const bool batch = c->nseg > 0 && c->seg_pcg_mode;
  ResMode& M = c->res->mode[precision == TG_MIXED ? 1 : 0][batch ? 1 : 0];
  if (M.state == 0) {
    const int s = plan_mode(c, precision, batch, M);
    if (s) return s;
  }
  *on = M.state > 0;
  return TG_OK;
}

int pcg_solve_resident(Context* c, const double4_32a* d_rhs, double rel_tol, int max_it, int precond, int* iters,
                       double* rel_res) {
  const int precision = c->tangent_precision;
  const bool batch = c->nseg > 0 && c->seg_pcg_mode;
  ResMode& M = c->res->mode[precision == TG_MIXED ? 1 : 0][batch ? 1 : 0];
  return precision == TG_MIXED ? solve_resident_t<float>(c, M, d_rhs, rel_tol, max_it, precond, iters, rel_res)
                               : solve_resident_t<double>(c, M, d_rhs, rel_tol, max_it, precond, iters, rel_res);
}

}  // namespace tg
