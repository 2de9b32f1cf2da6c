// Device side shared by the resident (respcg.cu) and the hybrid (hybridpcg.cu)
// PCG: exchange words, distributed shared memory, tensor memory as storage,
// reductions and the recurrence's scalars.  Internal to the library.
#pragma once

#include <type_traits>

#include "assembly.cuh"
#include "ff.cuh"
#include "krylov_common.cuh"
#include "respcg.cuh"

namespace tg {

namespace {

constexpr int kResClusterMax = 16;
constexpr int kResCopies = 16;         // tables of the CTAs' sums (grid form)

// Shape of a CTA: warps, chunks of 8 rows per warp at most, and for a warp's
// first `off` chunks the steps whose blocks stay out of shared memory.
//
// FP32: 16 warps at 128 registers.  A warp's first chunk keeps four of its
// seven steps (27 blocks a row) in registers, its second and third lie in
// tensor memory, the rest in shared memory, so a CTA holds 64 chunks where shared memory alone
// held 26: the SM's tensor memory is 256 KB that this solve's warps read
// beside the shared-memory pipe (a step costs that pipe 5 wavefronts from
// registers or tensor memory, its column indices and gathered vectors, and 14
// from shared memory).  A fifth step in registers spills more than it saves:
// solves of 3,375 to 19,683 nodes take 1 to 4% longer, of 1 to 512 RVEs of sides
// 6 to 20 0 to 13% (64 of side 20 7.79 against 8.79 ms), and four hold
// what five do of meshes of this form (fewer than 20,000 nodes) unless their
// nodes are numbered at random (11,000 nodes against 12,500).  Fewer CTAs a solve also means more solves at once: a
// chip runs 46 clusters of 3 CTAs, 28 of 5, 15 of 7 to 9, 8 of 11 or 12.
// FP64 runs at the rate of the FP64 pipe (one warp instruction per 64 cycles
// and scheduler), not of the storage.  A CTA of 16 warps keeps the first chunk
// of each warp in tensor memory and a second in shared memory where there is
// room: 29 chunks where shared memory alone held 13, so a solve of a batch
// takes half the CTAs, the 6,000 cycles of exchange and sums an iteration
// stand beside twice the product, and clusters of 6 fill the chip where
// clusters of 13 leave 61 of 152 SMs out.  (Smaller CTAs, several to an SM,
// allocate no tensor memory.)
template <typename T>
struct ResShape;
template <>
struct ResShape<float> {
  static constexpr int warps = 16, slots = 4, reg = 4, tm = 7, off = 3, state = 6;
};
template <>
struct ResShape<double> {
  static constexpr int warps = 16, slots = 2, reg = 0, tm = 7, off = 1, state = 0;
};
// steps of chunk i of a part of nw warps that stay out of shared memory
template <typename T>
__host__ __device__ constexpr int res_off_steps(int i, int nw) {
  if (sizeof(T) == 8) return nw == ResShape<T>::warps && i < ResShape<T>::off * nw ? ResShape<T>::tm : 0;
  return i < nw ? ResShape<T>::reg : i < ResShape<T>::off * nw ? ResShape<T>::tm : 0;
}
constexpr int kTmemColumns = 512;

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

// Tensor memory as plain storage: a warp reads and writes the 32 lanes of its
// quarter, one 32-bit value per thread and column.
__device__ __forceinline__ void tmem_alloc(unsigned* at) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(at)),
               "n"(kTmemColumns)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free(unsigned addr) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "n"(kTmemColumns));
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st9(unsigned a, const float* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(a),
               "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])),
               "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])),
               "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7]))
               : "memory");
  asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(a + 8u), "r"(__float_as_uint(v[8])) : "memory");
}
__device__ __forceinline__ void tmem_ld9(unsigned a, unsigned* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(a));
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(v[8]) : "r"(a + 8u));
}
__device__ __forceinline__ void tmem_ld18(unsigned a, unsigned* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(a));
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=r"(v[16]), "=r"(v[17]) : "r"(a + 16u));
}

template <typename T>
struct ResArgs {
  const ResPlanDev* plans;
  const ResItem* items;
  int k;                 // CTAs per solve
  int count;             // grid form: solves, dealt to the launch's groups of k CTAs
  const T* Ke;
  const uint8_t* mask;
  const double4_32a* rhs;
  typename Vec4<T>::type* x;
  ResOut* out;
  uint4* ll;             // grid form: exchange words, zero before the launch
  PcgScalars* sc;        // receives unscale (single solve) or 1 (batch)
  int* status;
  WaitLimits waits;
  int batch;             // the solution is unscaled in place
  int nnd;               // nodes of one right-hand side and solution
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
  u64 part[3][8];                    // grid form: sums of the polling warps
  u64 tot[3];                        // totals
  T coef[2];                         // alpha, beta
  // the recurrence's scalars: gamma and alpha of the last update (FP32: 1 /
  // (gamma alpha) and 1 / gamma), convergence threshold, r.r now and at the start
  u64 rz, al, thr, rr, rr0;
  int code, fail;
  int abort_flag;
  unsigned tmem;                     // the CTA's tensor memory
};

// After a poll of an exchange word that found it unwritten: whether to poll
// again.  A wait that ran out ends the CTA's others within 64 polls.
template <typename T>
__device__ __forceinline__ bool poll_again(ResShared<T>& sh, const WaitLimits& W, int& tries) {
  if (++tries & 63) return true;
  if (tries >= W.polls) sh.abort_flag = 1;
  return *reinterpret_cast<volatile int*>(&sh.abort_flag) == 0;
}

// Totals of three accumulators over every row of the solve, returned to
// thread 0 (and left in sh.tot): lanes, warps and CTAs in a fixed order.  seq
// numbers the reductions of a solve from 1.
//
// Each row's four lanes hold the terms of their component; two levels give the
// row sums, lane v of a row then stores value v, and warp v adds the rows' v
// sums: merging compensated pairs costs about nine instructions a level, so
// the levels a full warp tree would run mostly on idle lanes are replaced by
// one pass over shared memory.
// ROWS: lane v of a row already holds the row's value v in a[0].
template <typename A, typename T, bool GRID, bool ROWS = false>
__device__ __forceinline__ void total3(A (&a)[3], ResShared<T>& sh, int k, int rank, unsigned seq, uint4* inbox,
                                       const WaitLimits& W) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (!ROWS)
#pragma unroll
    for (int v = 0; v < 3; ++v) {
      a[v].shfl_merge(1);
      a[v].shfl_merge(2);
    }
  if ((lane & 3) < 3) {
    const A& m = ROWS || (lane & 3) == 0 ? a[0] : (lane & 3) == 1 ? a[1] : a[2];
    sh.red[lane & 3][warp * 8 + (lane >> 2)] = pack_word(m);
  }
  __syncthreads();
  const int par = seq & 1;
  if (GRID && k > 1) {
    // the sums go to kResCopies tables; a CTA polls the table of its rank
    // (one table polled by 152 SMs: 4.8 us a reduction, its lines queue at
    // their L2 slices; a table per CTA, 152^2 scattered sectors: 2.8 us)
    const int pw = min(nw, 5), copies = min(k, kResCopies);
    if (warp >= pw) return;
    const unsigned np = 32u * (unsigned)pw;
    if (warp < 3) {
      A t;
      for (int j = lane; j < nw * 8; j += 32) merge_word(t, sh.red[warp][j]);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) t.shfl_merge(o);
      if (lane == 0) sh.tot[warp] = pack_word(t);
    }
    asm volatile("bar.sync 1, %0;" ::"r"(np) : "memory");
    const u64 w0 = sh.tot[0], w1 = sh.tot[1], w2 = sh.tot[2];
    const u64 h0 = (w2 & 0xffffffffull) | ((u64)seq << 32), h1 = (w2 >> 32) | ((u64)seq << 32);
    for (int q = threadIdx.x; q < copies && rank != W.mute; q += (int)np) {
      uint4* w = inbox + (((size_t)q * 2 + par) * k + rank) * 2;
      st_word(w, w0, h0);
      st_word(w + 1, w1, h1);
    }
    const int mine = rank % copies;
    A g[3];
    for (int i = threadIdx.x; i < k; i += (int)np) {
      const uint4* w = inbox + (((size_t)mine * 2 + par) * k + i) * 2;
      u64 x0, y0, x1, y1;
      int tries = 0;
      for (;;) {
        ld_word(w, x0, y0);
        ld_word(w + 1, x1, y1);
        if ((word_seq(y0) == seq && word_seq(y1) == seq) || !poll_again(sh, W, tries)) break;
      }
      merge_word(g[0], x0);
      merge_word(g[1], x1);
      merge_word(g[2], (y0 & 0xffffffffull) | (y1 << 32));
    }
    __syncwarp();
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
#pragma unroll
      for (int v = 0; v < 3; ++v) g[v].shfl_merge(o);
    if (lane < 3) sh.part[lane][warp] = pack_word(lane == 0 ? g[0] : lane == 1 ? g[1] : g[2]);
    asm volatile("bar.sync 1, %0;" ::"r"(np) : "memory");
    if (warp == 0) {
      A t;
      const int v = lane >> 3, i = lane & 7;
      if (v < 3 && i < pw) merge_word(t, sh.part[v][i]);
      t.shfl_merge(1);
      t.shfl_merge(2);
      t.shfl_merge(4);
      if (v < 3 && i == 0) sh.tot[v] = pack_word(t);
      __syncwarp();
    }
    return;
  }
  if (warp < 3) {
    A t;
    for (int j = lane; j < nw * 8; j += 32) merge_word(t, sh.red[warp][j]);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) t.shfl_merge(o);
    const u64 w = pack_word(t);
    if (k == 1) {
      if (lane == 0) sh.tot[warp] = w;
      asm volatile("bar.sync 1, 96;" ::: "memory");
    } else {
      if (lane < k)
        st_async(cluster_map(smem_addr(&sh.slot[par][rank][warp]), lane), cluster_map(smem_addr(&sh.bar_s[par]), lane), w);
      if (warp == 0) {
        if (!mbar_wait_cluster(&sh.bar_s[par], ((seq - 1) >> 1) & 1)) sh.abort_flag = 1;
        __syncwarp();
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
        if (lane == 0) mbar_expect_tx(&sh.bar_s[par], 24u * (unsigned)k);  // of its next use
      }
    }
  }
}

// The recurrence's scalars from the totals delta = u.w, gamma = r.u, r.r
// (thread 0): convergence, breakdown, alpha and beta.  FP32 form: in
// double-float, from the same compensated pairs (an FP64 operation takes 64
// cycles here and its division 570: 2,200 cycles of every iteration), with
// alpha = gamma / (delta - gamma (gamma / (gamma_old alpha_old))) so that no
// squares leave FP32's range; alpha and beta are rounded to FP32 for the
// update in both.  Beside the FP64 scalars of the streamed solves, in 4.7
// million iterations of RVEs of sides 4 to 24 and meshes of 216 to 97,000
// nodes: alpha and beta before their rounding differ by at most 2e-6 of an FP32
// ulp, after it by nothing, and no solve ends at another iteration.  The
// reciprocals of the old values are formed off the
// critical path by scalars_next.
__device__ __forceinline__ ff::dfloat word_ff(u64 w) {
  return ff::fast_two_sum(__uint_as_float((unsigned)w), __uint_as_float((unsigned)(w >> 32)));
}
__device__ __forceinline__ u64 ff_word(ff::dfloat d) {
  return (u64)__float_as_uint(d.hi) | ((u64)__float_as_uint(d.lo) << 32);
}
__device__ __forceinline__ void scalars(ResShared<float>& sh, int it, int max_it, double tol) {
  using namespace ff;
  const dfloat delta = word_ff(sh.tot[0]), gamma = word_ff(sh.tot[1]), rr = word_ff(sh.tot[2]);
  if (it == 0) {
    sh.rr0 = ff_word(rr);
    sh.thr = ff_word(from_double(tol * tol * to_double(rr)));
  }
  const dfloat thr = word_ff(sh.thr), iz = word_ff(sh.rz), iza = word_ff(sh.al);
  dfloat alpha = make(0.f, 0.f), beta = make(0.f, 0.f), den = delta;
  if (it > 0) {
    beta = mul(gamma, iz);
    den = sub(delta, mul(gamma, mul(gamma, iza)));
  }
  int code = 0, fail = 0;
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
  } else if (!(den.hi > 0.f) || !isfinite(den.hi)) {
    code = 2;
    fail = isfinite(den.hi) ? 2 : 3;
  } else {
    alpha = mul(gamma, rcp(den));
  }
  sh.coef[0] = alpha.hi;
  sh.coef[1] = beta.hi;
  sh.code = code;
  sh.fail = fail;
  sh.rr = ff_word(rr);
  sh.tot[0] = ff_word(alpha);  // for scalars_next
}
// 1 / gamma and 1 / (gamma alpha) for the next iteration (one thread, after
// the barrier that publishes alpha and beta)
__device__ __forceinline__ void scalars_next(ResShared<float>& sh) {
  using namespace ff;
  const dfloat iz = rcp(word_ff(sh.tot[1]));
  sh.rz = ff_word(iz);
  sh.al = ff_word(mul(iz, rcp(word_ff(sh.tot[0]))));
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
__device__ __forceinline__ void scalars_next(ResShared<double>&) {}
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

}  // namespace
}  // namespace tg
