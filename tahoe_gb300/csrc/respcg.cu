// Resident PCG, sm_103a: a whole (block-)Jacobi CG solve in one launch with
// the matrix held on the SMs.
//
// A matrix that fits the chip's registers, tensor memory and shared memory is
// read once per solve instead of once per iteration: every CTA assembles the
// rows of its part straight from the element blocks and keeps them there, and
// the iterations touch nothing but them and the words the CTAs exchange
// (ResShape, respcg_device.cuh, says which chunk lies where).  Two forms, one
// kernel body:
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
//            A batch's larger RVEs are one launch per size, its groups of k
//            CTAs dealing the solves.
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
// Measured against the streamed kernels (product + vector kernel: 20 us an
// iteration on a 16^3 FP64 cube, 39 on a 28^3 one; four kernels and 26 us on
// one RVE of side 8): 9.3, 24.2 and 4.5 us, with no host round trip inside a
// solve; 4,096 RVEs 540 -> 214 ms with stress, tangent and residuals.  What
// bounds an iteration: of 12,300 cycles of an RVE of side 15 in a cluster 4,900
// are the product (shared-memory reads), 1,200 the update and the rest the
// latency of the exchanges and sums; in FP64 the FP64 pipe.  Whole FP32 meshes
// of 20,000 nodes and more: hybridpcg.cu.
//
// Rows and storage: a warp holds chunks of 8 consecutive active rows, 4 lanes per row;
// lane l takes blocks l, l+4, ... of its row (sliced ELL per warp: step t of
// a warp is 9 planes of 32 values, unit stride across the lanes, no bank
// conflicts, and 32 16-bit column indices).  After the product lane c < 3 of a
// row owns component c of every vector.  The search vector is kept over the
// part's column window (a contiguous range of active rows).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <exception>
#include <map>
#include <mutex>
#include <new>
#include <string>
#include <thread>
#include <unordered_map>
#include <vector>

#include "respcg_device.cuh"

namespace tg {

namespace {

// One CTA's part of one solve.
template <typename T, bool GRID, bool BLK, int NS>
__device__ __forceinline__ void resident_solve(const ResArgs<T>& A, const ResItem& I, int item, int rank,
                                               unsigned char* smem, ResShared<T>& sh) {
  using V = typename Vec4<T>::type;
  using Shape = ResShape<T>;
  constexpr bool F32 = sizeof(T) == 4;
  constexpr int RB = Shape::reg, OFF = Shape::off, RA = RB > 0 ? RB : 1, NM = BLK ? 3 : 1;
  const ResPlanDev P = A.plans[I.plan];
  const int k = P.k;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5, c = lane & 3, q0 = lane & ~3;
  const int ch0 = P.part_chunk[rank], nch = P.part_chunk[rank + 1] - ch0;
  const int4 win = P.part_win[rank];
  const int row0 = ch0 * kResChunkRows, row1 = min(P.rows, (ch0 + nch) * kResChunkRows);
  // shared memory: the window [columns][4]; FP32: every chunk's p, s, x and
  // preconditioner [chunks][.][32]; the values that are in neither registers
  // nor tensor memory [steps][9][32]; the columns, eight steps of a lane in
  // one 16-byte word [groups][32][8] (padded with the chunk's first row)
  V* uw = reinterpret_cast<V*>(smem);
  const int steps0 = P.chunk_step[ch0];
  // this warp's chunks: first value step and column group in shared memory,
  // steps, packed (the loop below is short of registers)
  unsigned lay[NS];
  auto vstep_of = [&](int q) { return (int)(lay[q] >> 20); };
  auto cgrp_of = [&](int q) { return (int)((lay[q] >> 8) & 0xfffu); };
  auto nst_of = [&](int q) { return (int)(lay[q] & 0xffu); };
  int vsteps = 0;  // value steps in shared memory
  {
#pragma unroll
    for (int q = 0; q < NS; ++q) lay[q] = 0u;
    int groups = 0;
    for (int i0 = 0; i0 < nch; i0 += 32) {
      const int i = i0 + lane;
      const int b = i < nch ? P.chunk_step[ch0 + i] : 0, n = i < nch ? P.chunk_step[ch0 + i + 1] - b : 0;
      const int v = max(0, n - res_off_steps<T>(i, nw)), gr = (n + 7) >> 3;
      int inc = v, ging = gr;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o), z = __shfl_up_sync(0xffffffffu, ging, o);
        if (lane >= o) {
          inc += y;
          ging += z;
        }
      }
#pragma unroll
      for (int q = 0; q < NS; ++q) {
        const int mine = warp + q * nw;  // this warp's chunk of slot q
        const int from = mine & 31;
        const int ve = __shfl_sync(0xffffffffu, vsteps + inc - v, from), ne = __shfl_sync(0xffffffffu, n, from),
                  ge = __shfl_sync(0xffffffffu, groups + ging - gr, from);
        if (mine < nch && mine >= i0 && mine < i0 + 32)
          lay[q] = ((unsigned)ve << 20) | ((unsigned)ge << 8) | (unsigned)ne;
      }
      vsteps += __shfl_sync(0xffffffffu, inc, 31);
      groups += __shfl_sync(0xffffffffu, ging, 31);
    }
  }
  T* state = reinterpret_cast<T*>(uw + win.y);  // p, s, x
  T* prec = state + (F32 ? (size_t)nch * 3 * 32 : 0);
  T* vals = prec + (F32 ? (size_t)nch * NM * 32 : 0);
  uint16_t* cols = reinterpret_cast<uint16_t*>(vals + (size_t)vsteps * 9 * 32);
  uint4* inbox = GRID ? A.ll + I.ll : nullptr;                         // partial sums
  uint4* urow = GRID ? inbox + 4 * (size_t)min(k, kResCopies) * k : nullptr;  // rows' vectors
  // columns of this warp's quarter: two chunks of 64 (FP64: one of 126)
  const unsigned tm = sh.tmem + ((unsigned)(warp & 3) << 21) + (unsigned)(warp >> 2) * 128u;
  const long long at0 = (long long)I.vec * A.nnd + I.node_off;  // of this right-hand side
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
  T Mr[NS][NM], pr[NS], sr[NS], xr[NS];  // registers in FP64; FP32 keeps them in shared memory
  unsigned comp = 0;   // bit q: this lane's component of its row in chunk q is a free dof
  unsigned live = 0;   // bit q: the row exists
  unsigned peers[NS];  // cluster form: the other parts whose windows hold the row
#pragma unroll
  for (int q = 0; q < NS; ++q) {
    const int i = warp + q * nw;
    const int row = (ch0 + i) * kResChunkRows + (lane >> 2);
    const bool lv = i < nch && row < P.rows;
    if (lv) live |= 1u << q;
    const uint8_t m = lv ? A.mask[I.node_off + P.act_node[row]] : 0;
    if (c < 3 && ((m >> c) & 1)) comp |= 1u << q;
    peers[q] = 0u;
    if (!GRID && k > 1 && lv && c == 0)
      for (int o = win.z; o <= win.w; ++o)
        if (o != rank && row >= sh.peer[o].x && row < sh.peer[o].x + sh.peer[o].y) peers[q] |= 1u << o;
    T D[9];
    bool have = false;
    const int step0 = i < nch ? P.chunk_step[ch0 + i] : 0, nst = nst_of(q), cgrp = cgrp_of(q);
    auto block = [&](int t, T acc[9]) {
      const int at = (step0 + t) * 32 + lane;
      const int cl = P.col[at];
      const int2 sl = P.slot[at];
      slot_value<T>(sl, m, P.contrib, A.Ke, I.elem_off, acc);
      cols[((size_t)(cgrp + (t >> 3)) * 32 + lane) * 8 + (t & 7)] = (uint16_t)(cl - win.x);
      if (cl == row && sl.y > 0) {
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
        if (t < nst) {
          block(t, rv[t]);
        } else {
#pragma unroll
          for (int e = 0; e < 9; ++e) rv[t][e] = T(0);
        }
      }
    }
    // the columns' padding: the chunk's first row
    for (int t = nst; t < (nst + 7) / 8 * 8; ++t)
      cols[((size_t)(cgrp + (t >> 3)) * 32 + lane) * 8 + (t & 7)] =
          (uint16_t)((ch0 + i) * kResChunkRows - win.x);
    if constexpr (F32) {
      if (q > 0 && q < OFF && nst > 0)
        for (int t = 0; t < Shape::tm; ++t) {
          T acc[9];
          if (t < nst) {
            block(t, acc);
          } else {
#pragma unroll
            for (int e = 0; e < 9; ++e) acc[e] = T(0);
          }
          __syncwarp();
          tmem_st9(tm + (unsigned)(q - 1) * 64u + 9u * (unsigned)t, acc);
        }
    }
    if constexpr (!F32) {
      if (q == 0 && nw == Shape::warps)
        for (int t = 0; t < Shape::tm; ++t) {
          T acc[9];
#pragma unroll
          for (int e = 0; e < 9; ++e) acc[e] = T(0);
          if (t < nst) block(t, acc);
          float h[18];
#pragma unroll
          for (int e = 0; e < 9; ++e) {
            h[2 * e] = __int_as_float(__double2loint(acc[e]));
            h[2 * e + 1] = __int_as_float(__double2hiint(acc[e]));
          }
          __syncwarp();
          tmem_st9(tm + 18u * (unsigned)t, h);
          tmem_st9(tm + 18u * (unsigned)t + 9u, h + 9);
        }
    }
    const int off = F32 ? (q == 0 ? RB : q < OFF ? Shape::tm : 0) : q == 0 && nw == Shape::warps ? Shape::tm : 0;
    for (int t = off; t < nst; ++t) {
      T acc[9];
      block(t, acc);
      T* vp = vals + (size_t)(vstep_of(q) + t - off) * 9 * 32 + lane;
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
      T v = BLK ? (c == 0 ? B[d] : c == 1 ? B[3 + d] : c == 2 ? B[6 + d] : T(0))
                : (c == 0 ? Dg[0] : c == 1 ? Dg[4] : c == 2 ? Dg[8] : T(0));
      if (!who || !lv) v = T(0);
      if (F32) {
        if (i < nch) prec[((size_t)i * NM + d) * 32 + lane] = v;
      } else {
        Mr[q][d] = v;
      }
    }
    if (F32) {
      if (i < nch)
#pragma unroll
        for (int v = 0; v < 3; ++v) state[((size_t)i * 3 + v) * 32 + lane] = T(0);
    } else {
      pr[q] = sr[q] = xr[q] = T(0);
    }
  }
  if (F32 || nw == Shape::warps) tmem_wait_st();
  // M^-1 r of a row's component (whole warps; zero for a warp without a chunk)
  auto precond = [&](int q, T rq) {
    const bool on = warp + q * nw < nch;
    const T* Mq = prec + (size_t)(on ? warp + q * nw : 0) * NM * 32 + lane;
    T z = T(0);
#pragma unroll
    for (int d = 0; d < NM; ++d) {
      T m;
      if constexpr (F32)
        m = on ? Mq[32 * d] : T(0);
      else
        m = Mr[q][d];
      z += m * (BLK ? __shfl_sync(0xffffffffu, rq, q0 + d) : rq);
    }
    return z;
  };
  unsigned seq = 0;
  T r[NS], u[NS];
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
      b[q] = ((comp >> q) & 1) ? reinterpret_cast<const double*>(A.rhs + (at0 + P.act_node[row]))[c] : 0.0;
      a[0].v = max(a[0].v, exponent_of(b[q]));
    }
    ++seq;
    total3<AccMax, T, GRID>(a, sh, k, rank, seq, inbox, A.waits);
    __syncthreads();
    const int e1 = (int)sh.tot[0];
    if (e1 > 0 && e1 < 0x7ff) scale_exp = max(-1000, min(1000, 1023 - e1));
    double sc = power_of_two(scale_exp);
    a[0].v = a[1].v = a[2].v = 0;
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      if (q * nw >= nch) break;
      const T rq = T(b[q] * sc);
      a[0].v = max(a[0].v, exponent_of((double)(rq * precond(q, rq))));
    }
    __syncthreads();  // sh.tot and sh.red are read
    ++seq;
    total3<AccMax, T, GRID>(a, sh, k, rank, seq, inbox, A.waits);
    __syncthreads();
    const int e2 = (int)sh.tot[0];
    if (e2 > 0 && e2 < 0x7ff && e1 > 0 && e1 < 0x7ff) scale_exp = max(-1000, min(1000, scale_exp - (e2 - 1023) / 2));
    sc = power_of_two(scale_exp);
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      r[q] = T(b[q] * sc);
      u[q] = T(0);
      if (q * nw < nch) u[q] = precond(q, r[q]);
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
      if (((live >> q) & 1) && c == 0) {
        const int row = (ch0 + warp + q * nw) * kResChunkRows + (lane >> 2);
        uw[row - win.x] = mk<V, T>(u[q], u1, u2);
        if (GRID && k > 1) RowWords<T>::store(urow + (size_t)row * RowWords<T>::n, u[q], u1, u2, (unsigned)it + 1u);
        for (unsigned to = peers[q]; to; to &= to - 1) {
          const int4 pq = sh.peer[__ffs((int)to) - 1];
          st_async_row((unsigned)pq.z + (unsigned)((row - pq.x) * (int)sizeof(V)), (unsigned)pq.w, u[q], u1, u2);
        }
      }
    }
    __syncwarp();
    if (!GRID && k > 1 && lane == 0) {
      if (warp == 0)
        mbar_expect_tx(&sh.bar_u, (unsigned)((win.y - (row1 - row0)) * (int)sizeof(V)));
      else
        mbar_arrive(&sh.bar_u);
    }
    if (warp == 1 && lane == 0 && it > 0) scalars_next(sh);
    // gamma and r.r while the vectors travel
    Acc<T> a[3];
    if (F32)
#pragma unroll
      for (int q = 0; q < NS; ++q)
        if ((comp >> q) & 1) {
          a[1].add_prod(r[q], u[q]);
          a[2].add_prod(r[q], r[q]);
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
        while (!RowWords<T>::load(w, (unsigned)it + 1u, x0, x1, x2) && poll_again(sh, A.waits, tries)) {
        }
        uw[at] = mk<V, T>(x0, x1, x2);
      }
      __syncthreads();
    } else if (!GRID && k > 1) {
      if (!mbar_wait_cluster(&sh.bar_u, (unsigned)it & 1u)) sh.abort_flag = 1;
      __syncwarp();
    } else {
      __syncthreads();
    }
    // w = A u, one chunk after the other: a lane's column indices of eight
    // steps are one load, so a batch's gathers are all in flight together
    // (indices read step by step left 5 wavefronts a step waiting on two
    // dependent loads)
    T w[NS], A0[NS], A1[NS], A2[NS];
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      A0[q] = A1[q] = A2[q] = T(0);
      if (q * nw >= nch) break;
      T a0 = T(0), a1 = T(0), a2 = T(0);
      auto fma9 = [&](T m0, T m1, T m2, T m3, T m4, T m5, T m6, T m7, T m8, const V& uj) {
        a0 += m0 * uj.x + m1 * uj.y + m2 * uj.z;
        a1 += m3 * uj.x + m4 * uj.y + m5 * uj.z;
        a2 += m6 * uj.x + m7 * uj.y + m8 * uj.z;
      };
      auto index = [](const uint4& g, int t) {
        const unsigned v = t < 2 ? g.x : t < 4 ? g.y : t < 6 ? g.z : g.w;
        return (t & 1) ? v >> 16 : v & 0xffffu;
      };
      const int nst = nst_of(q);
      const uint4* cg = reinterpret_cast<const uint4*>(cols) + cgrp_of(q) * 32 + lane;
      const T* vp = vals + vstep_of(q) * (9 * 32) + lane;
      int t0 = 0;  // steps done
      if constexpr (F32) {
        if (q < OFF) {
          t0 = q == 0 ? RB : Shape::tm;
          if (nst > 0) {
            const uint4 g = *cg;
            if (q == 0) {
              auto batch = [&](auto from, auto to) {
                constexpr int lo = decltype(from)::value, hi = decltype(to)::value;
                V uj[4];
#pragma unroll
                for (int t = lo; t < hi; ++t) uj[t - lo] = uw[index(g, t)];
#pragma unroll
                for (int t = lo; t < hi; ++t)
                  fma9(rv[t][0], rv[t][1], rv[t][2], rv[t][3], rv[t][4], rv[t][5], rv[t][6], rv[t][7], rv[t][8],
                       uj[t - lo]);
              };
              batch(std::integral_constant<int, 0>{}, std::integral_constant<int, (RB < 4 ? RB : 4)>{});
              if (RB > 4 && nst > 4) batch(std::integral_constant<int, 4>{}, std::integral_constant<int, RB>{});
            } else {
              const unsigned col = tm + (unsigned)(q - 1) * 64u;
              auto pair = [&](auto at) {
                constexpr int t = decltype(at)::value;
                constexpr bool two = t + 1 < Shape::tm;
                unsigned b[18];
                __syncwarp();
                if (two)
                  tmem_ld18(col + 9u * (unsigned)t, b);
                else
                  tmem_ld9(col + 9u * (unsigned)t, b);
                const V v0 = uw[index(g, t)];
                V v1 = v0;
                if (two) v1 = uw[index(g, t + 1)];
                tmem_wait_ld();
                auto f = [&](int e) { return __uint_as_float(b[e]); };
                fma9(f(0), f(1), f(2), f(3), f(4), f(5), f(6), f(7), f(8), v0);
                if (two) fma9(f(9), f(10), f(11), f(12), f(13), f(14), f(15), f(16), f(17), v1);
              };
              pair(std::integral_constant<int, 0>{});
              pair(std::integral_constant<int, 2>{});
              if (nst > 4) {
                pair(std::integral_constant<int, 4>{});
                pair(std::integral_constant<int, 6>{});
              }
            }
          }
        }
      }
      if constexpr (!F32) {
        if (q == 0 && nw == Shape::warps && nst > 0) {
          const uint4 g = *cg;
#pragma unroll
          for (int t = 0; t < Shape::tm; ++t)
            if (t < 4 || nst > 4) {
              unsigned b[18];
              __syncwarp();
              tmem_ld18(tm + 18u * (unsigned)t, b);
              const V uj = uw[index(g, t)];
              tmem_wait_ld();
              auto f = [&](int e) { return __hiloint2double((int)b[2 * e + 1], (int)b[2 * e]); };
              fma9(f(0), f(1), f(2), f(3), f(4), f(5), f(6), f(7), f(8), uj);
            }
          t0 = Shape::tm;
        }
      }
      for (; t0 < nst; t0 = (t0 | 7) + 1) {
        const uint4 g = cg[(t0 >> 3) * 32];
        const int e = min(nst, (t0 | 7) + 1);
#pragma unroll
        for (int t = 0; t < 8; ++t)
          if ((t0 & ~7) + t >= t0 && (t0 & ~7) + t < e) {
            const V uj = uw[index(g, t)];
            fma9(vp[0], vp[32], vp[64], vp[96], vp[128], vp[160], vp[192], vp[224], vp[256], uj);
            vp += 9 * 32;
          }
      }
      A0[q] = a0;
      A1[q] = a1;
      A2[q] = a2;
    }
    // sums over a row's lanes, component c to lane c: lanes 0, 1 keep
    // components 0 and 1, lanes 2, 3 component 2
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      w[q] = T(0);
      if (q * nw >= nch) continue;
      const bool up = (c & 2) != 0;
      const T g0 = __shfl_xor_sync(0xffffffffu, up ? A0[q] : A2[q], 2);
      const T g1 = __shfl_xor_sync(0xffffffffu, A1[q], 2);
      const T b0 = (up ? A2[q] : A0[q]) + g0;
      const T b1 = A1[q] + g1;
      const T e = __shfl_xor_sync(0xffffffffu, up ? b0 : ((c & 1) ? b0 : b1), 1);
      w[q] = up ? b0 + e : ((c & 1) ? b1 + e : b0 + e);
      if (F32) {
        if ((comp >> q) & 1) a[0].add_prod(u[q], w[q]);
      } else {
        // lane v of a row forms the row's value v from its gathered
        // components: three FP64 operations where the lanes' own terms and
        // their two merging levels took nine
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const T ud = __shfl_sync(0xffffffffu, u[q], q0 + d), rd = __shfl_sync(0xffffffffu, r[q], q0 + d),
                  wd = __shfl_sync(0xffffffffu, w[q], q0 + d);
          a[0].add_prod(c == 2 ? rd : ud, c == 0 ? wd : rd);
        }
      }
    }
    ++seq;
    total3<Acc<T>, T, GRID, !F32>(a, sh, k, rank, seq, inbox, A.waits);
    if (threadIdx.x == 0) scalars(sh, it, A.max_it, A.tol);
    __syncthreads();
    if (sh.code) break;
    const T al = sh.coef[0], be = sh.coef[1];
    if constexpr (F32) {
      // two chunks at a time, loads first: the stores of one would order the
      // next one's loads behind them
#pragma unroll
      for (int q2 = 0; q2 < NS; q2 += 2) {
        if (q2 * nw >= nch) break;
        T po[2], so[2], xo[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int i = warp + (q2 + h) * nw;
          const T* sq = state + i * (3 * 32) + lane;
          const bool on = i < nch;
          po[h] = on ? sq[0] : T(0);
          so[h] = on ? sq[32] : T(0);
          xo[h] = on ? sq[64] : T(0);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int q = q2 + h;
          po[h] = u[q] + be * po[h];
          so[h] = w[q] + be * so[h];
          xo[h] += al * po[h];
          r[q] -= al * so[h];
          u[q] = precond(q, r[q]);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int i = warp + (q2 + h) * nw;
          T* sq = state + i * (3 * 32) + lane;
          if (i < nch) {
            sq[0] = po[h];
            sq[32] = so[h];
            sq[64] = xo[h];
          }
        }
      }
    } else {
#pragma unroll
      for (int q = 0; q < NS; ++q) {
        if (q * nw >= nch) break;
        pr[q] = u[q] + be * pr[q];
        sr[q] = w[q] + be * sr[q];
        xr[q] += al * pr[q];
        r[q] -= al * sr[q];
        u[q] = precond(q, r[q]);
      }
    }
  }
  const double unscale = power_of_two(-scale_exp);
  const int code = sh.code;
#pragma unroll
  for (int q = 0; q < NS; ++q) {
    if (q * nw >= nch) break;
    const int i = warp + q * nw;
    T xq = F32 ? (i < nch ? state[((size_t)i * 3 + 2) * 32 + lane] : T(0)) : xr[q];
    if (A.batch) xq = code == 2 ? T(0) : xq * T(unscale);
    const T x1 = __shfl_down_sync(0xffffffffu, xq, 1), x2 = __shfl_down_sync(0xffffffffu, xq, 2);
    const int row = (ch0 + i) * kResChunkRows + (lane >> 2);
    if (((live >> q) & 1) && c == 0) A.x[at0 + P.act_node[row]] = mk<V, T>(xq, x1, x2);
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

// Tensor memory of a CTA with all its warps: such a CTA has the SM to itself
// (its launch asks for more than half the shared memory), so the allocation
// never waits for another.
template <typename T>
__device__ __forceinline__ bool tmem_begin(ResShared<T>& sh) {
  const bool use = blockDim.x == ResShape<T>::warps * 32;
  if (use && threadIdx.x < 32) tmem_alloc(&sh.tmem);
  __syncthreads();
  return use;
}
template <typename T>
__device__ __forceinline__ void tmem_end(ResShared<T>& sh, bool use) {
  __syncthreads();
  if (use && threadIdx.x < 32) tmem_free(sh.tmem);
}

template <typename T, bool BLK, int NS>
__global__ void __launch_bounds__(ResShape<T>::warps * 32, 1) resident_cluster_kernel(ResArgs<T> A) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ ResShared<T> sh;
  const int item = blockIdx.x / A.k, rank = blockIdx.x % A.k;
  const bool tmem = tmem_begin(sh);
  resident_solve<T, false, BLK, NS>(A, A.items[item], item, rank, smem, sh);
  tmem_end(sh, tmem);
}

template <typename T, bool BLK, int NS>
__global__ void __launch_bounds__(ResShape<T>::warps * 32, 1) resident_grid_kernel(ResArgs<T> A) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ ResShared<T> sh;
  const bool tmem = tmem_begin(sh);
  const int groups = gridDim.x / A.k, rank = blockIdx.x % A.k;
  for (int item = blockIdx.x / A.k; item < A.count; item += groups) {
    resident_solve<T, true, BLK, NS>(A, A.items[item], item, rank, smem, sh);
    const bool stop = sh.abort_flag != 0;
    __syncthreads();
    if (stop) break;  // a wait ran out: nothing more is awaited
  }
  tmem_end(sh, tmem);
}

// The kernel of a launch class.  FP64 has one for parts of at most a chunk a
// warp (NS = 1): the second chunk's code costs a single solve of 4,000 rows 7%.
template <typename T>
const void* resident_kernel(bool grid, bool blk, bool one) {
  constexpr int N = ResShape<T>::slots, L = sizeof(T) == 8 ? 1 : N;
  if (one)
    return grid ? (blk ? (const void*)resident_grid_kernel<T, true, L> : (const void*)resident_grid_kernel<T, false, L>)
                : (blk ? (const void*)resident_cluster_kernel<T, true, L>
                       : (const void*)resident_cluster_kernel<T, false, L>);
  return grid ? (blk ? (const void*)resident_grid_kernel<T, true, N> : (const void*)resident_grid_kernel<T, false, N>)
              : (blk ? (const void*)resident_cluster_kernel<T, true, N>
                     : (const void*)resident_cluster_kernel<T, false, N>);
}

// The rows of a whole mesh on the device (a mesh of 50,000 nodes took 17 ms on
// the host, as long as its load step).  rank: index of every active node.
__global__ void rows_flag_kernel(int n, const uint8_t* __restrict__ mask, int* __restrict__ flag) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) flag[i] = mask[i] ? 1 : 0;
}
__global__ void rows_node_kernel(int n, const uint8_t* __restrict__ mask, const int* __restrict__ rank,
                                 int* __restrict__ act_node) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && mask[i]) act_node[rank[i]] = i;
}
// one warp per chunk, four lanes per row: steps and column range (FILL
// false), or the blocks and columns of every step (FILL true); a row's active
// blocks go to its lanes in turn
template <bool FILL>
__global__ void __launch_bounds__(256) rows_chunk_kernel(int rows, int nch, const int* __restrict__ act_node,
                                                         const int* __restrict__ rowptr, const int* __restrict__ col,
                                                         const uint8_t* __restrict__ mask,
                                                         const int* __restrict__ rank, int* __restrict__ step,
                                                         int* __restrict__ lo, int* __restrict__ hi,
                                                         int* __restrict__ blk, int* __restrict__ cidx) {
  const int ch = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31, c = lane & 3;
  if (ch >= nch) return;
  const int r0 = ch * kResChunkRows, row = r0 + (lane >> 2);
  const bool live = row < rows;
  const int g = live ? act_node[row] : 0;
  const int b = live ? rowptr[g] : 0, e = live ? rowptr[g + 1] : 0;
  int l = r0, h = min(rows, r0 + kResChunkRows), cnt = 0;
  const int s0 = FILL ? step[ch] : 0, s1 = FILL ? step[ch + 1] : 0;
  if (FILL)
    for (int t = s0; t < s1; ++t) {
      blk[(size_t)t * 32 + lane] = -1;
      cidx[(size_t)t * 32 + lane] = r0;
    }
  __syncwarp();
  for (int j0 = b; __any_sync(0xffffffffu, j0 < e); j0 += 4) {
    const int j = j0 + c;
    const bool on = j < e && mask[col[j]] != 0;
    const unsigned m = (__ballot_sync(0xffffffffu, on) >> (lane & ~3)) & 0xfu;
    if (on) {
      const int a = rank[col[j]], q = cnt + __popc(m & ((1u << c) - 1u));
      l = min(l, a);
      h = max(h, a + 1);
      if (FILL) {
        const size_t at = (size_t)(s0 + (q >> 2)) * 32 + (lane & ~3) + (q & 3);
        blk[at] = j;
        cidx[at] = a;
      }
    }
    cnt += __popc(m);
  }
  if (!FILL) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      l = min(l, __shfl_xor_sync(0xffffffffu, l, o));
      h = max(h, __shfl_xor_sync(0xffffffffu, h, o));
      cnt = max(cnt, __shfl_xor_sync(0xffffffffu, cnt, o));
    }
    if (lane == 0) {
      step[ch] = (cnt + 3) / 4;
      lo[ch] = l;
      hi[ch] = h;
    }
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

// Dynamic shared memory of one CTA, the largest cluster that can run with it,
// and for every cluster size the largest with as many at a time on the chip.
template <typename T>
int limits_t(Context* c, ResLimits* L) {
  int optin = 0;
  cudaFuncAttributes fa;
  if (!ok(c, cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device), "attribute"))
    return TG_ERR_CUDA;
  size_t smem = (size_t)optin;
  for (int q = 0; q < 8; ++q) {
    const void* fn = resident_kernel<T>(q & 1, q & 2, q & 4);
    if (!ok(c, cudaFuncGetAttributes(&fa, fn), "function attributes")) return TG_ERR_CUDA;
    smem = std::min(smem, (size_t)optin - fa.sharedSizeBytes);
    // one value for every caller: other contexts may configure and launch it
    if (!ok(c, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes),
            "smem attribute") ||
        (!(q & 1) &&
         !ok(c, cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1), "cluster attribute")))
      return TG_ERR_CUDA;
  }
  L->smem = smem;
  L->cluster = 1;
  int many[kResClusterMax + 1] = {};
  for (int k = 1; k <= kResClusterMax; ++k) {
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
    if (cudaOccupancyMaxActiveClusters(&many[k], resident_kernel<T>(false, true, false), &cfg) == cudaSuccess &&
        many[k] > 0)
      L->cluster = (k & (k - 1)) == 0 ? k : L->cluster;
    else
      cudaGetLastError();
  }
  for (int k = 1; k <= kResClusterMax; ++k) {
    L->widest[k] = k;
    for (int j = k + 1; j <= L->cluster && many[k] > 0 && many[j] == many[k]; ++j) L->widest[k] = j;
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
  const int rows = R.rows = (int)R.act_node.size(), nch = (rows + kResChunkRows - 1) / kResChunkRows;
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

// Bytes of one part with nw warps: the window, FP32's vectors and
// preconditioner, the values outside registers and tensor memory
// (res_off_steps), the columns in groups of eight steps.
size_t part_bytes(const ResRows& R, int a, int b, int elem, int nw, int* lo, int* hi) {
  int l = R.chunk_lo[a], h = R.chunk_hi[a];
  const int state = elem == 4 ? ResShape<float>::state : ResShape<double>::state;
  size_t vsteps = 0, groups = 0;
  for (int ch = a; ch < b; ++ch) {
    l = std::min(l, R.chunk_lo[ch]);
    h = std::max(h, R.chunk_hi[ch]);
    const int n = R.chunk_step[ch + 1] - R.chunk_step[ch];
    vsteps += std::max(0, n - (elem == 4 ? res_off_steps<float>(ch - a, nw) : res_off_steps<double>(ch - a, nw)));
    groups += (n + 7) / 8;
  }
  *lo = l;
  *hi = h;
  return (size_t)(h - l) * 4 * elem + (size_t)(b - a) * state * 32 * elem + vsteps * 9 * 32 * elem + groups * 512;
}

// The chunks cut into k consecutive parts of near-equal work; false if one
// exceeds a CTA.  A CTA has a warp for each of its chunks (in fours), or all it
// can have (full).
bool split_parts(const ResRows& R, int k, int elem, size_t cap, ResPlan& P, bool full = false) {
  const int nch = (int)R.chunk_lo.size();
  if (k > nch) return false;
  const int warps = elem == 4 ? ResShape<float>::warps : ResShape<double>::warps;
  const int slots = elem == 4 ? ResShape<float>::slots : ResShape<double>::slots;
  // a chunk's work is its steps and its vector updates (about two steps')
  auto work = [&](int ch) { return (long long)R.chunk_step[ch] + 2LL * ch; };
  const long long total = work(nch);
  P.part_chunk.assign(k + 1, 0);
  P.part_chunk[k] = nch;
  for (int q = 1; q < k; ++q) {
    const long long target = (total * q + k / 2) / k;
    int lo = 0, hi = nch;  // first chunk start with at least the target before it
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (work(mid) < target)
        lo = mid + 1;
      else
        hi = mid;
    }
    int ch = lo;
    if (ch > 0 && target - work(ch - 1) < work(ch) - target) --ch;
    P.part_chunk[q] = std::min(std::max(ch, P.part_chunk[q - 1] + 1), nch - (k - q));
  }
  P.part_win.assign(k, make_int4(0, 0, 0, 0));
  P.smem = 0;
  int most = 0, longest = 0;
  for (int ch = 0; ch < nch; ++ch) longest = std::max(longest, R.chunk_step[ch + 1] - R.chunk_step[ch]);
  for (int q = 0; q < k; ++q) most = std::max(most, P.part_chunk[q + 1] - P.part_chunk[q]);
  if (most > warps * slots) return false;
  // one chunk per warp while there are warps for it
  P.warps = full ? warps : std::min(warps, (most + 3) / 4 * 4);
  P.one = elem == 8 && most <= P.warps;
  for (int q = 0; q < k; ++q) {
    const int a = P.part_chunk[q], b = P.part_chunk[q + 1];
    int lo, hi;
    const size_t bytes = part_bytes(R, a, b, elem, P.warps, &lo, &hi);
    // (the kernel packs a chunk's steps, groups and value steps in 8, 12 and 12 bits)
    if (bytes > cap || hi - lo > 65535 || longest > 255) return false;
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

constexpr int kPollRows = 8;  // rows that a thread of the grid form polls

// A split of the rows over CTAs.  A solve of a batch takes the fewest CTAs
// that hold it (every SM has another RVE to solve), in FP64 as many more as
// leave the number of clusters that run at once the same; a solve alone spreads
// over the chip.  Up to the cluster limit the CTAs are one cluster, above it
// (grid) CTAs of a cooperative launch.
bool resident_plan(const ResRows& R, int elem, int num_sms, const ResLimits& L, bool alone, ResPlan& P) {
  const size_t cap = L.smem;
  const int max_cluster = L.cluster;
  const int nch = (int)R.chunk_lo.size();
  P.rows = R.rows;
  P.nchunks = nch;
  if (nch == 0) return false;
  // a chunk whose columns alone exceed a CTA: no split holds it (shuffled node
  // numbers; trying every number of CTAs takes half a millisecond)
  for (int ch = 0; ch < nch; ++ch)
    if ((size_t)(R.chunk_hi[ch] - R.chunk_lo[ch]) * 4 * elem > cap) return false;
  const int most = elem == 4 ? ResShape<float>::warps * ResShape<float>::slots
                             : ResShape<double>::warps * ResShape<double>::slots;
  int kmin = 0;
  for (int k = (nch + most - 1) / most; k <= std::min(num_sms, nch) && !kmin; ++k)
    if (split_parts(R, k, elem, cap, P)) kmin = k;
  if (!kmin) return false;
  P.grid = kmin > max_cluster;
  if (alone) {
    // alone: a cluster while its CTAs hold few chunks each (its exchanges are
    // short), else every SM.  Cluster / grid, us an iteration, by the chunks of
    // a CTA of the cluster: FP32 16 3.6 / 5.0, 30 4.5 / 4.9, 36 4.9 / 5.2, 51
    // 5.8 / 5.1; FP64 2 6.6 / 8.4, 5 7.5 / 8.6, 7 9.0 / 8.9, 12 15.1 / 9.3.
    const int few = elem == 4 ? 40 : 6;
    P.grid = P.grid || (nch + max_cluster - 1) / max_cluster > few;
    const int k = std::max(kmin, std::min(nch, P.grid ? num_sms : max_cluster));
    if (!P.grid) {
      if (k != kmin && !split_parts(R, k, elem, cap, P) && !split_parts(R, kmin, elem, cap, P)) return false;
    } else {
      // Every thread polls its share of the other parts' rows in the window,
      // 0.26 us a row: few where the nodes are numbered along the mesh, the
      // whole mesh where they are not.  Above kPollRows a CTA has all its warps
      // whatever its chunks (and in FP64 its tensor memory).  Shuffled numbers,
      // streamed / a warp a chunk / all warps, us an iteration: FP32 4,913
      // nodes 10.4 / 13.7 / 6.7, 9,261 10.8 / 14.1 / 9.7; FP64 5,832 21.7 / 26.2
      // (the fewest CTAs that held it) / 15.5.
      ResPlan best;
      auto attempt = [&](bool full) {
        ResPlan Q = P;
        if (!split_parts(R, k, elem, cap, Q, full)) return false;
        best = Q;
        return true;
      };
      auto polls = [&]() {
        int away = 0;
        for (int q = 0; q < k; ++q)
          away = std::max(away, best.part_win[q].y - (best.part_chunk[q + 1] - best.part_chunk[q]) * kResChunkRows);
        return away / (32 * best.warps);
      };
      bool good = attempt(false);
      if (!good || polls() > kPollRows) good = attempt(true) || good;
      if (good) P = best;  // else the fewest CTAs
    }
  } else if (!P.grid && elem == 8) {
    // the chip holds 15 clusters of 7, of 8 and of 9: in FP64, where a CTA's
    // time is that of its chunks, the largest costs nothing (48 RVEs with nine
    // solves each 31.2 -> 29.9 ms); FP32's time is the exchanges' (64 RVEs
    // 6.95 -> 7.18 ms)
    const int k = std::min(nch, L.widest[kmin]);
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

int resident_limits(Context* c, int precision, ResLimits* limits) {
  ResState& S = *c->res;
  const int p = precision == TG_MIXED ? 1 : 0;
  if (!S.limits_known[p]) {
    const int s = p ? limits_t<float>(c, &S.limits[p]) : limits_t<double>(c, &S.limits[p]);
    if (s) return s;
    S.limits_known[p] = true;
  }
  *limits = S.limits[p];
  return TG_OK;
}

int resident_slots(Context* c, long long n, const int* d_blk, const int* d_cptr, int2* d_slot) {
  if (n == 0) return TG_OK;
  resident_slots_kernel<<<(unsigned)((n + 255) / 256), 256, 0, c->stream>>>(n, d_blk, d_cptr, d_slot);
  c->launches++;
  return ok(c, cudaGetLastError(), "resident_slots_kernel") ? TG_OK : TG_ERR_CUDA;
}

namespace {
// A device buffer of a mode's plans.
template <typename T>
bool hold(Context* c, ResMode& M, T** p, size_t n) {
  if (!dalloc(c, p, n)) return false;
  M.bufs.push_back((void*)*p);
  return true;
}
void drop_mode(Context* c, ResMode& M) {
  for (void* p : M.bufs) dfree(c, p);
  M = ResMode{};
}

// Rows of the whole mesh on the device; R receives what the split needs.
int rows_of_mesh(Context* c, ResMode& M, ResRows& R, ResPlanDev& D) {
  R = ResRows{};
  const int n = c->nnd;
  cudaStream_t st = c->stream;
  struct Scratch {
    Context* c;
    std::vector<void*> p;
    ~Scratch() {
      for (void* q : p) dfree(c, q);
    }
    bool get(int** q, size_t m) {
      if (!dalloc(c, q, m)) return false;
      p.push_back(*q);
      return true;
    }
  } scratch{c, {}};
  int *flag = nullptr, *rank = nullptr, *tmp = nullptr, *node = nullptr;
  if (!scratch.get(&flag, (size_t)n) || !scratch.get(&rank, (size_t)n + 1) ||
      !scratch.get(&tmp, (size_t)n / 1024 + 4))
    return TG_ERR_OOM;
  rows_flag_kernel<<<(n + 255) / 256, 256, 0, st>>>(n, c->d_mask, flag);
  int s = scan_counts(c, n, flag, rank, tmp);
  if (s) return s;
  if (!ok(c, cudaMemcpyAsync(&R.rows, rank + n, sizeof(int), cudaMemcpyDeviceToHost, st), "rows") ||
      !ok(c, cudaStreamSynchronize(st), "sync"))
    return TG_ERR_CUDA;
  const int nch = (R.rows + kResChunkRows - 1) / kResChunkRows;
  R.chunk_step.assign(nch + 1, 0);
  R.chunk_lo.assign(nch, 0);
  R.chunk_hi.assign(nch, 0);
  c->launches++;
  if (nch == 0) return TG_OK;
  int *cnt = nullptr, *step = nullptr, *lohi = nullptr;
  if (!hold(c, M, &node, (size_t)R.rows) || !scratch.get(&cnt, (size_t)nch) || !hold(c, M, &step, (size_t)nch + 1) ||
      !scratch.get(&lohi, 2 * (size_t)nch))
    return TG_ERR_OOM;
  rows_node_kernel<<<(n + 255) / 256, 256, 0, st>>>(n, c->d_mask, rank, node);
  const int grid = (nch + 7) / 8;
  rows_chunk_kernel<false><<<grid, 256, 0, st>>>(R.rows, nch, node, c->d_rowptr, c->d_col, c->d_mask, rank, cnt, lohi,
                                                 lohi + nch, nullptr, nullptr);
  s = scan_counts(c, nch, cnt, step, tmp);
  if (s) return s;
  if (!ok(c, cudaGetLastError(), "rows kernels") ||
      !ok(c, cudaMemcpyAsync(R.chunk_step.data(), step, sizeof(int) * (nch + 1), cudaMemcpyDeviceToHost, st), "rows") ||
      !ok(c, cudaMemcpyAsync(R.chunk_lo.data(), lohi, sizeof(int) * nch, cudaMemcpyDeviceToHost, st), "rows") ||
      !ok(c, cudaMemcpyAsync(R.chunk_hi.data(), lohi + nch, sizeof(int) * nch, cudaMemcpyDeviceToHost, st), "rows") ||
      !ok(c, cudaStreamSynchronize(st), "sync"))
    return TG_ERR_CUDA;
  const size_t slots = (size_t)R.chunk_step[nch] * 32;
  int *blk = nullptr, *cidx = nullptr;
  int2* slot = nullptr;
  if (!hold(c, M, &blk, slots) || !hold(c, M, &cidx, slots) || !hold(c, M, &slot, slots)) return TG_ERR_OOM;
  rows_chunk_kernel<true><<<grid, 256, 0, st>>>(R.rows, nch, node, c->d_rowptr, c->d_col, c->d_mask, rank, step, nullptr,
                                                nullptr, blk, cidx);
  c->launches += 3;
  if (!ok(c, cudaGetLastError(), "rows kernels")) return TG_ERR_CUDA;
  s = resident_slots(c, (long long)slots, blk, c->d_contrib_ptr, slot);
  if (s) return s;
  D.act_node = node;
  D.blk = blk;
  D.col = cidx;
  D.chunk_step = step;
  D.slot = slot;
  D.contrib = c->d_contrib;
  return TG_OK;
}
}  // namespace

// The mesh's buffers went back to the pool with it.
void resident_reset(Context* c) {
  hybrid_reset(c);
  if (!c->res) return;
  ResState& S = *c->res;
  for (auto& a : S.mode)
    for (ResMode& m : a) m = ResMode{};
  S.d_items = nullptr;
  S.d_out = nullptr;
  S.items_cap = 0;
  S.d_ll = nullptr;
  S.ll_cap = 0;
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
  for (auto& a : c->res->mode) drop_mode(c, a[1]);
}

namespace {

// fn(0) to fn(n - 1), many of them on a few host threads: the first solve of
// 1,024 RVEs of side 8 that are all numbered differently took 108 ms with one,
// 66 with eight.
template <typename F>
void each_plan(int n, const F& fn) {
  std::atomic<int> next{0};
  std::exception_ptr thrown;
  std::mutex mu;
  auto work = [&]() {
    try {
      for (int p; (p = next++) < n;) fn(p);
    } catch (...) {
      std::lock_guard<std::mutex> lock(mu);
      thrown = std::current_exception();
      next = n;
    }
  };
  std::vector<std::thread> threads;
  const int more = std::min({7, n / 16, (int)std::thread::hardware_concurrency() - 1});
  try {
    for (int t = 0; t < more; ++t) threads.emplace_back(work);
  } catch (...) {
    // no more threads: this one does the rest
  }
  work();
  for (std::thread& t : threads) t.join();
  if (thrown) std::rethrow_exception(thrown);
}

// Plans the current mesh: every RVE of a batch (the template's plan for a
// composed mesh) or the whole mesh; M.state 1 where it fits.
int plan_rows(Context* c, int precision, bool batch, ResMode& M) {
  const int elem = precision == TG_MIXED ? 4 : 8;
  ResLimits limits;
  int s = resident_limits(c, precision, &limits);
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
        it = seen.emplace(t, fits ? (int)M.plans.size() : -1).first;
        if (fits) M.plans.push_back(P);
      }
      M.plan_of.push_back(it->second);
    }
  } else if (!batch) {
    if (c->composed) return TG_OK;  // one solve over a composed batch: streamed
    // a mesh above the chip's chunks is not looked at row by row
    const int chunks = elem == 4 ? ResShape<float>::warps * ResShape<float>::slots
                                 : ResShape<double>::warps * ResShape<double>::slots;
    if ((long long)c->neq > 3LL * c->num_sms * chunks * kResChunkRows || c->neq == 0) return TG_OK;
    ResRows R;
    ResPlan P;
    s = rows_of_mesh(c, M, R, P.dev);
    if (s) return s;
    if (!resident_plan(R, elem, c->num_sms, limits, true, P)) return TG_OK;
    ResImage img;
    const size_t at = img.split_at(P);
    int* d = nullptr;
    if (!hold(c, M, &d, img.data.size())) return TG_ERR_OOM;
    if (!ok(c, cudaMemcpyAsync(d, img.data.data(), sizeof(int) * img.data.size(), cudaMemcpyHostToDevice, c->stream),
            "resident split") ||
        !ok(c, cudaStreamSynchronize(c->stream), "sync"))
      return TG_ERR_CUDA;
    resident_bind_split(P.dev, d, at, P);
    M.plans.push_back(P);
    M.plan_of.push_back(0);
  } else {
    // RVEs of equal structure (connectivity and free dofs, counted from their
    // own first node) have one plan: the contribution map of the first, which
    // counts the mesh's elements, serves the others at their distance from it.
    // One row image, slot array and launch for all of them: the first solve of
    // 4,096 RVEs of side 8, planned one by one, took 330 ms (the second 64);
    // so 109.
    if (ensure_host_mesh(c)) return TG_ERR_CUDA;
    std::vector<uint8_t> mask(c->nnd, 0);
    for (int n = 0; n < c->nnd; ++n)
      for (int d = 0; d < 3; ++d)
        if (c->h_eqnos[(size_t)n * 3 + d] > 0) mask[n] |= (uint8_t)(1u << d);
    std::vector<int> first;  // RVE of every plan
    std::unordered_map<unsigned long long, std::vector<int>> seen;  // hash -> plans
    for (int i = 0; i < nseg; ++i) {
      const int n0 = c->h_seg_node[i], n1 = c->h_seg_node[i + 1];
      const long long e0 = c->h_seg_elem[i], e1 = c->h_seg_elem[i + 1];
      if (n0 == n1) return TG_OK;  // an RVE without nodes: refused by the streamed solve
      auto equal = [&](int j) {
        const int m0 = c->h_seg_node[j];
        const long long f0 = c->h_seg_elem[j];
        if (c->h_seg_node[j + 1] - m0 != n1 - n0 || c->h_seg_elem[j + 1] - f0 != e1 - e0 ||
            !std::equal(mask.begin() + n0, mask.begin() + n1, mask.begin() + m0))
          return false;
        for (long long k = 0; k < (e1 - e0) * 8; ++k)
          if (c->h_conn[e0 * 8 + k] - n0 != c->h_conn[f0 * 8 + k] - m0) return false;
        return true;
      };
      unsigned long long h = (unsigned long long)(n1 - n0) * 0x9e3779b97f4a7c15ull + (unsigned long long)(e1 - e0);
      for (int n = n0; n < n1; ++n) h = (h ^ mask[n]) * 0x100000001b3ull;
      for (long long k = e0 * 8; k < e1 * 8; ++k) h = (h ^ (unsigned)(c->h_conn[k] - n0)) * 0x100000001b3ull;
      int plan = -1;
      for (int p : seen[h])
        if (plan < 0 && equal(first[p])) plan = p;
      if (plan < 0) {
        plan = (int)first.size();
        first.push_back(i);
        seen[h].push_back(plan);
      }
      M.plan_of.push_back(plan);
    }
    const int np = (int)first.size();
    std::vector<ResRows> rows(np);
    std::vector<ResPlan> plans(np);
    std::vector<uint8_t> fits(np, 1);
    each_plan(np, [&](int p) {
      const int n0 = c->h_seg_node[first[p]], n1 = c->h_seg_node[first[p] + 1];
      resident_rows(n0, n1, c->h_rowptr.data(), c->h_col.data(), mask.data(), rows[p]);
      if (!rows[p].act_node.empty() && !resident_plan(rows[p], elem, c->num_sms, limits, false, plans[p])) fits[p] = 0;
    });
    ResImage blocks, img;  // every plan's blocks, then the rest
    std::vector<size_t> at_blk(np), at_rows(np), at_split(np);
    std::vector<int> kept(np, -1);
    for (int p = 0; p < np; ++p) {
      if (!fits[p]) continue;
      kept[p] = (int)M.plans.size();
      ResPlan& P = plans[p];
      at_blk[p] = blocks.data.size();
      blocks.data.insert(blocks.data.end(), rows[p].blk.begin(), rows[p].blk.end());
      rows[p].blk.clear();
      at_rows[p] = img.rows_at(rows[p]);
      at_split[p] = img.split_at(P);
      P.elem0 = c->h_seg_elem[first[p]];
      M.plans.push_back(P);
    }
    for (int& p : M.plan_of) p = kept[p];
    int *d = nullptr, *blk = nullptr;
    int2* slot = nullptr;
    if (!hold(c, M, &d, img.data.size()) || !hold(c, M, &slot, blocks.data.size()) ||
        !hold(c, M, &blk, blocks.data.size()))
      return TG_ERR_OOM;
    if (!ok(c, cudaMemcpyAsync(d, img.data.data(), sizeof(int) * img.data.size(), cudaMemcpyHostToDevice, c->stream),
            "resident rows") ||
        !ok(c, cudaMemcpyAsync(blk, blocks.data.data(), sizeof(int) * blocks.data.size(), cudaMemcpyHostToDevice,
                               c->stream),
            "resident blocks") ||
        !ok(c, cudaStreamSynchronize(c->stream), "sync"))
      return TG_ERR_CUDA;
    s = resident_slots(c, (long long)blocks.data.size(), blk, c->d_contrib_ptr, slot);
    M.bufs.pop_back();
    dfree(c, blk);  // the slots name their contributions
    if (s) return s;
    for (int p = 0; p < np; ++p) {
      if (kept[p] < 0) continue;
      ResPlan& P = M.plans[kept[p]];
      ResPlanDev& D = P.dev;
      resident_bind_rows(D, d, at_rows[p], rows[p]);
      resident_bind_split(D, d, at_split[p], P);
      D.blk = nullptr;
      D.slot = slot + at_blk[p];
      D.contrib = c->d_contrib;
    }
  }
  for (int p : M.plan_of) M.streamed += p < 0 ? 1 : 0;
  if (M.plans.empty()) return TG_OK;
  std::vector<ResPlanDev> dev;
  for (const ResPlan& P : M.plans) dev.push_back(P.dev);
  if (!hold(c, M, &M.d_plans, std::max<size_t>(dev.size(), 1))) return TG_ERR_OOM;
  if (!ok(c, cudaMemcpyAsync(M.d_plans, dev.data(), sizeof(ResPlanDev) * dev.size(), cudaMemcpyHostToDevice, c->stream),
          "resident plans") ||
      !ok(c, cudaStreamSynchronize(c->stream), "sync"))
    return TG_ERR_CUDA;
  M.state = 1;
  return TG_OK;
}
// A mesh that does not fit the chip, or whose plans find no room in device
// memory, keeps nothing: mode -1, and the streamed solves take it.
int plan_mode(Context* c, int precision, bool batch, ResMode& M) {
  drop_mode(c, M);
  int s = TG_OK;
  try {
    s = plan_rows(c, precision, batch, M);
  } catch (const std::bad_alloc&) {
    c->err = "no host memory for the plans of the solves on the chip";
    s = TG_ERR_OOM;
  }
  if (!s && M.state == 1) return TG_OK;
  drop_mode(c, M);
  M.state = -1;
  return s == TG_ERR_OOM ? TG_OK : s;
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

// Launches of a batch's classes on streams beside the context's own.  The
// context's stream waits for them on every way out: what it frees or
// overwrites next is read by them.
struct AuxStreams {
  Context* c;
  int n = 0;  // streams that follow the context's
  int fork(int want) {
    const int s = want > 0 ? aux_streams(c) : TG_OK;
    if (s || want <= 0) return s;
    if (!ok(c, cudaEventRecord(c->res->fork, c->stream), "fork")) return TG_ERR_CUDA;
    for (; n < want; ++n)
      if (!ok(c, cudaStreamWaitEvent(c->res->aux[n], c->res->fork, 0), "fork")) return TG_ERR_CUDA;
    return TG_OK;
  }
  int join() {
    bool good = true;
    for (int a = 0; a < n; ++a)
      good = ok(c, cudaEventRecord(c->res->join[a], c->res->aux[a]), "join") &&
             ok(c, cudaStreamWaitEvent(c->stream, c->res->join[a], 0), "join") && good;
    n = 0;
    return good ? TG_OK : TG_ERR_CUDA;
  }
  ~AuxStreams() { join(); }
};

// Runs the solves of the listed RVEs (act; one for a whole mesh) for nvec
// right-hand sides, nnd nodes apart in d_rhs and x, and reports each in out.
// x is zero away from the solved rows; with keep_x they stay as they are.
template <typename T>
int run_resident(Context* c, ResMode& M, bool batch, const std::vector<uint8_t>& act, const double4_32a* d_rhs, int nvec,
                 typename Vec4<T>::type* x, double rel_tol, int max_it, int precond, std::vector<ResItem>& items,
                 std::vector<ResOut>& out, bool keep_x = false) {
  using V = typename Vec4<T>::type;
  ResState& S = *c->res;
  int s = TG_OK;
  cudaStream_t st = c->stream;
  const int nseg = (int)act.size();
  // launch classes by form, CTAs, warps and shared memory, the largest first
  struct Class {
    bool grid, one;
    int k, warps;
    size_t smem;
    std::vector<int> seg;
  };
  std::map<std::vector<long long>, Class> cls;
  for (int i = 0; i < nseg; ++i) {
    if (!act[i] || M.plan_of[i] < 0 || M.plans[M.plan_of[i]].rows == 0) continue;
    const ResPlan& P = M.plans[M.plan_of[i]];
    const long long b = (long long)((P.smem + 16383) / 16384);
    Class& C = cls[{P.grid ? 0 : 1, -(long long)P.k, -P.warps, P.one ? 1 : 0, -b}];
    C.grid = P.grid;
    C.one = P.one;
    C.k = P.k;
    C.warps = P.warps;
    C.smem = std::max(C.smem, P.smem);
    C.seg.push_back(i);
  }
  items.clear();
  long long ll = 0;  // exchange words of the grid solves
  for (auto& e : cls)
    for (int i : e.second.seg)
      for (int v = 0; v < nvec; ++v) {
        const ResPlan& P = M.plans[M.plan_of[i]];
        ResItem it{M.plan_of[i], i, batch ? c->h_seg_node[i] : 0, 0, v, 0, ll};
        // a template's contribution map counts its own elements, an uploaded
        // RVE's the mesh's from the plan's first RVE on
        if (batch) it.elem_off = c->h_seg_elem[i] - P.elem0;
        if (P.grid) ll += 4LL * std::min(P.k, kResCopies) * P.k + (long long)P.rows * RowWords<T>::n;
        items.push_back(it);
      }
  const int n = (int)items.size();
  long long icap = S.items_cap, ocap = S.items_cap;
  s = grow(c, &S.d_items, &icap, n);
  if (!s) s = grow(c, &S.d_out, &ocap, n);
  if (s) return s;
  S.items_cap = (int)icap;
  if (ll) {
    s = grow(c, &S.d_ll, &S.ll_cap, ll);
    if (s) return s;
  }
  // rows outside every solve (prescribed nodes, RVEs not solved) stay zero
  if ((!keep_x && !ok(c, cudaMemsetAsync(x, 0, sizeof(V) * (size_t)c->nnd * nvec, st), "x")) ||
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
  A.k = A.count = 0;
  A.Ke = sizeof(T) == 4 ? (const T*)c->d_Ke32 : (const T*)c->d_Ke64;
  A.mask = c->d_mask;
  A.rhs = d_rhs;
  A.x = x;
  A.nnd = c->nnd;
  A.out = S.d_out;
  A.ll = S.d_ll;
  A.sc = c->d_pcg;
  A.status = c->d_status;
  A.waits = c->waits;
  A.batch = batch ? 1 : 0;
  const bool blk = precond == TG_PRECOND_BLOCK_JACOBI;
  A.max_it = max_it;
  A.tol = rel_tol;
  if (ll && !ok(c, cudaMemsetAsync(S.d_ll, 0, sizeof(uint4) * (size_t)ll, st), "exchange")) return TG_ERR_CUDA;
  // the classes run beside each other: each is small beside the chip's tail
  // otherwise
  const int naux = (int)std::min<size_t>(std::max<size_t>(cls.size(), 1) - 1, kResAux);
  AuxStreams beside{c};
  s = beside.fork(naux);
  if (s) return s;
  size_t first = 0;
  int q = 0;
  for (auto& e : cls) {
    Class& C = e.second;
    // a CTA that allocates tensor memory: alone on its SM
    if (C.warps == ResShape<T>::warps) C.smem = std::max(C.smem, (size_t)116 << 10);
    const size_t solves = C.seg.size() * (size_t)nvec;
    ResArgs<T> B = A;
    B.items = S.d_items + first;
    B.out = S.d_out + first;
    B.k = C.k;
    B.count = (int)solves;
    first += solves;
    cudaLaunchConfig_t cfg = {};
    // a cooperative launch holds as many groups of k CTAs as the chip at once
    const size_t groups = C.grid ? std::min<size_t>(solves, std::max(1, c->num_sms / C.k)) : solves;
    cfg.gridDim = dim3((unsigned)(groups * C.k));
    cfg.blockDim = dim3(32u * (unsigned)C.warps);
    cfg.dynamicSmemBytes = C.smem;
    cfg.stream = q % (naux + 1) ? S.aux[q % (naux + 1) - 1] : st;
    cudaLaunchAttribute at[1];
    if (C.grid) {
      at[0].id = cudaLaunchAttributeCooperative;
      at[0].val.cooperative = 1;
    } else {
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = (unsigned)C.k;
      at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = 1;
    c->launches++;
    void* args[] = {&B};
    if (!ok(c, cudaLaunchKernelExC(&cfg, resident_kernel<T>(C.grid, blk, C.one), args),
            C.grid ? "resident_grid_kernel" : "resident_cluster_kernel"))
      return TG_ERR_CUDA;
    ++q;
  }
  s = beside.join();
  if (s) return s;
  out.assign(std::max(n, 1), ResOut{});
  if (n && !ok(c, cudaMemcpyAsync(out.data(), S.d_out, sizeof(ResOut) * n, cudaMemcpyDeviceToHost, st), "out"))
    return TG_ERR_CUDA;
  if (!ok(c, cudaStreamSynchronize(st), "pcg sync")) return TG_ERR_CUDA;
  out.resize(n);
  for (ResOut& o : out)
    if (o.done == 0) {  // a wait ran out before this solve reported
      o.done = 2;
      o.fail = 5;
    }
  return TG_OK;
}

template <typename T>
int solve_resident_t(Context* c, ResMode& M, const double4_32a* d_rhs, double rel_tol, int max_it, int precond,
                     int* iters, double* rel_res) {
  using V = typename Vec4<T>::type;
  const bool batch = c->nseg > 0 && c->seg_pcg_mode;
  int s = pcg_vectors(c, sizeof(T) == 4 ? TG_MIXED : TG_FP64);
  if (s) return s;
  const int nseg = batch ? c->nseg : 1;
  std::vector<uint8_t> act(nseg, 1);
  if (batch && (int)c->seg_active.size() == nseg) act = c->seg_active;
  // RVEs that do not fit: the streamed per-RVE solve first, which sets the
  // others' rows to zero; an RVE takes the same solve in every batch
  int worst_it = 0;
  double worst_rel = 0.0;
  bool streamed = false;
  if (batch && M.streamed > 0) {
    std::vector<uint8_t> sub(act);
    for (int i = 0; i < nseg; ++i) {
      if (M.plan_of[i] >= 0) sub[i] = 0;
      streamed = streamed || sub[i];
    }
    if (streamed) {
      const bool tolerate = c->seg_tolerate;
      sub.swap(c->seg_active);
      c->seg_tolerate = true;
      s = push_solve(c) ? push_prepare(c, c->tangent_precision) : ensure_full_assembly(c);
      if (!s) {
        std::memset(c->h_pcg, 0, sizeof(PcgScalars));
        s = pcg_solve_segmented(c, d_rhs, rel_tol, max_it, precond, &worst_it, &worst_rel);
        // what single RVEs came to is in seg_status
        if ((s == TG_ERR_NAN && c->h_pcg[0].fail != 5) || s == TG_ERR_NOT_CONVERGED) s = TG_OK;
      }
      sub.swap(c->seg_active);
      c->seg_tolerate = tolerate;
      if (s) return s;
    }
  }
  std::vector<ResItem> items;
  std::vector<ResOut> out;
  s = run_resident<T>(c, M, batch, act, d_rhs, 1, (V*)c->d_x, rel_tol, max_it, precond, items, out, streamed);
  if (s) return s;
  const int n = (int)items.size();
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
  int broke = 0, limit = 0, nact = 0, timeout = 0;
  if (!streamed) c->seg_status.assign(nseg, TG_OK);
  for (int i = 0; i < n; ++i) {
    const ResOut& o = out[i];
    worst_it = std::max(worst_it, o.iters);
    if (o.rr0 > 0.0) worst_rel = std::max(worst_rel, std::sqrt(o.rr / o.rr0));
    c->seg_status[items[i].seg] = o.done == 2 ? TG_ERR_NAN : o.done != 1 ? TG_ERR_NOT_CONVERGED : TG_OK;
    timeout += o.done == 2 && o.fail == 5 ? 1 : 0;
  }
  for (int i = 0; i < nseg; ++i) {
    if (!act[i]) continue;
    ++nact;
    broke += c->seg_status[i] == TG_ERR_NAN ? 1 : 0;
    limit += c->seg_status[i] == TG_ERR_NOT_CONVERGED ? 1 : 0;
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

// w = v + x, nine vectors (x: the solutions on the free dofs, zero elsewhere)
namespace {
template <typename V>
__global__ void resident_add_kernel(long long n, const double4_32a* __restrict__ v, const V* __restrict__ x,
                                    double4_32a* __restrict__ w) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double4_32a a = v[i];
  const V b = x[i];
  w[i] = make_double4_32a(a.x + (double)b.x, a.y + (double)b.y, a.z + (double)b.z, 0.0);
}

template <typename T>
int macro_resident_t(Context* c, ResMode& M, int nvec, const double4_32a* d_b, const double4_32a* d_v,
                     double4_32a* d_w, double rel_tol, int max_it, int precond, int* iters) {
  using V = typename Vec4<T>::type;
  V* x = nullptr;
  const long long nv = (long long)c->nnd * nvec;
  if (!ok(c, cudaMallocAsync((void**)&x, sizeof(V) * (size_t)nv, c->stream), "alloc")) return TG_ERR_OOM;
  std::vector<ResItem> items;
  std::vector<ResOut> out;
  int s = run_resident<T>(c, M, true, std::vector<uint8_t>(c->nseg, 1), d_b, nvec, x, rel_tol, max_it, precond, items,
                          out);
  if (!s) {
    resident_add_kernel<V><<<(unsigned)((nv + 255) / 256), 256, 0, c->stream>>>(nv, d_v, x, d_w);
    c->launches++;
    if (!ok(c, cudaGetLastError(), "resident_add_kernel")) s = TG_ERR_CUDA;
  }
  cudaFreeAsync(x, c->stream);
  if (s) return s;
  int worst = 0, limit = 0;
  static const char* why[] = {"", "non-finite initial residual", "p.Ap <= 0 (indefinite operator)", "p.Ap not finite",
                              "non-finite update", "exchange wait timed out"};
  for (const ResOut& o : out) {
    worst = std::max(worst, o.iters);
    if (o.done == 2) {
      c->err = std::string("multi-vector PCG breakdown: ") + why[o.fail >= 0 && o.fail <= 5 ? o.fail : 0];
      return TG_ERR_NAN;
    }
    limit += o.done == 3 ? 1 : 0;
  }
  if (iters) *iters = worst;
  return limit ? TG_ERR_NOT_CONVERGED : TG_OK;
}
}  // namespace

int macro_solve_resident(Context* c, int precision, int nvec, const double4_32a* d_b, const double4_32a* d_v,
                         double4_32a* d_w, double rel_tol, int max_it, int precond, int* iters) {
  ResMode& M = c->res->mode[precision == TG_MIXED ? 1 : 0][1];
  return precision == TG_MIXED
             ? macro_resident_t<float>(c, M, nvec, d_b, d_v, d_w, rel_tol, max_it, precond, iters)
             : macro_resident_t<double>(c, M, nvec, d_b, d_v, d_w, rel_tol, max_it, precond, iters);
}

// The default form solves resident where the mesh (every RVE of the batch)
// fits; the explicit forms of tg_pcg_form and the symmetric format keep their
// own kernels.
constexpr int kHybridNodes = 20000;

int resident_active(Context* c, int precision, bool* on) {
  *on = false;
  if (c->cg_push >= 0 || c->pcg_form != 1 || !c->cg_pdl || sym_active(c)) return TG_OK;
  if (precision != TG_MIXED && precision != TG_FP64) return TG_OK;
  if (!c->res) c->res = new ResState();
  const bool batch = c->nseg > 0 && c->seg_pcg_mode;
  ResMode& M = c->res->mode[precision == TG_MIXED ? 1 : 0][batch ? 1 : 0];
  if (M.state == 0) {
    // A whole mesh in FP32 above kHybridNodes: the hybrid form, whose compact
    // parts exchange a fifth of the rows that the grid form's slabs do.  Per
    // iteration, grid form / hybrid: 3,375 nodes 4.7 / 5.2 us, 9,261 5.2 / 4.4,
    // 15,625 4.8 / 5.1, 27,360 6.3 / 5.1, 38,475 7.4 / 5.7, 60,025 9.0 / 6.9.
    // The grid form keeps what the hybrid refuses.
    int s = TG_OK;
    bool fits = false;
    if (!batch && precision == TG_MIXED && c->nnd >= kHybridNodes) s = hybrid_plan(c, &fits);
    if (!s && fits)
      M.state = 2;
    else if (!s)
      s = plan_mode(c, precision, batch, M);
    if (s) return s;
  }
  *on = M.state > 0;
  return TG_OK;
}

int resident_route(Context* c, int precision, int* route) {
  bool on = false;
  const int s = resident_active(c, precision, &on);
  *route = TG_ROUTE_STREAMED;
  if (s || !on) return s;
  const ResMode& M = c->res->mode[precision == TG_MIXED ? 1 : 0][c->nseg > 0 && c->seg_pcg_mode ? 1 : 0];
  *route = M.state == 2 ? TG_ROUTE_HYBRID : M.streamed > 0 ? TG_ROUTE_SOME : TG_ROUTE_CHIP;
  return TG_OK;
}

// Whether a batch's every RVE is solved on the chip.
bool resident_whole(const Context* c, int precision) {
  return c->res->mode[precision == TG_MIXED ? 1 : 0][1].streamed == 0;
}

// The mode of the next solve of a precision, given up: a solve found no room for
// its buffers.
void resident_refuse(Context* c, int precision) {
  ResMode& M = c->res->mode[precision == TG_MIXED ? 1 : 0][c->nseg > 0 && c->seg_pcg_mode ? 1 : 0];
  drop_mode(c, M);
  M.state = -1;
}

int pcg_solve_resident(Context* c, const double4_32a* d_rhs, double rel_tol, int max_it, int precond, int* iters,
                       double* rel_res) {
  const int precision = c->tangent_precision;
  const bool batch = c->nseg > 0 && c->seg_pcg_mode;
  ResMode& M = c->res->mode[precision == TG_MIXED ? 1 : 0][batch ? 1 : 0];
  if (M.state == 2) return hybrid_solve(c, d_rhs, rel_tol, max_it, precond, iters, rel_res);
  return precision == TG_MIXED ? solve_resident_t<float>(c, M, d_rhs, rel_tol, max_it, precond, iters, rel_res)
                               : solve_resident_t<double>(c, M, d_rhs, rel_tol, max_it, precond, iters, rel_res);
}

}  // namespace tg
