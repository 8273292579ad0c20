// LU panel of at most 16 thread-block-cluster CTAs with the active columns in registers.
//
// What bounds a panel is the chain of its columns: pivot search, exchange of the pivot row,
// update, one column after the other.  panel_kernel spends 3.6-4.4 us on a column (a grid
// barrier through L2 and a handful of block barriers); here the chain per column is two warp
// reductions of the pivot key -> one named barrier of the warps that own rows (none when a CTA
// has at most 32 rows) -> st.async of the CTA's candidate key and row into every CTA of the
// cluster -> one mbarrier wait -> registers.
// The panel is factored in sub-panels of W columns.  Thread t of the first ceil(rows / 32)
// warps holds row t's W entries in registers; rows never move: a row's position in the
// partially pivoted order is a register (pos), which the interchange p <-> j updates, and the
// rows go to their final places only when the panel is written back.  So the interchanges of
// the step are also known without simulating them: row r of the panel ends at pos(r).
// After a sub-panel, the W pivot rows are exchanged through global memory (L2), every CTA solves
// U12 = L11^-1 A12 for the remaining columns and applies the rank-W update to its rows in shared
// memory.  Every element sees the operations of panel_kernel in its order: the same factors, bit
// for bit.
//
// Measured (one B200, 128 columns FP32 / 64 columns FP64, kernel alone): 120 rows 132 / 88 us,
// 400 rows 161 / 100 us, 1000 rows 175 / 106 us, 2700 rows 245 / - us.  The whole mixed
// factorisation against the cluster panel before it (the panel_kernel algorithm with its exchange
// in distributed shared memory): N = 400 1.79 -> 1.24 ms, 1743 7.2 -> 4.36 ms, 3000 13.1 -> 8.3 ms;
// FP64, N = 4000, 27.8 -> 22.9 ms.  A column takes about 0.7 us of latency (reductions, barrier,
// 330 cycles of remote store); the rank-W updates of 2700 rows another 40 us (FMA-bound on 16 SMs).
//
// Dynamic shared memory: P [NB][rpc | 1] column-major, then U12 [NB - W][W].
#pragma once
#include "common.cuh"
#include "lu.cuh"
#include "tc_common.cuh"

namespace hprmat {

constexpr int kRegPanelThreads = 384;
constexpr int kRegPanelWarps = kRegPanelThreads / 32;
constexpr int kRegPanelRows = 256;  // most rows per CTA (one thread each)
constexpr int kRegPanelFW = kRegPanelRows / 32;

// Sub-panel width: 16 columns, 8 in FP64 (the row updates of a column step run at half rate and
// a row's message is twice as long).
template <typename T, int NB> constexpr int panel_width() {
  constexpr int w = sizeof(T) == sizeof(double2) ? 8 : 16;
  return NB < w ? NB : w;
}

template <typename T, int NB>
__host__ __device__ constexpr size_t panel_reg_smem(int rpc) {
  constexpr int W = panel_width<T, NB>();
  return ((size_t)NB * (size_t)(rpc | 1) + (NB - W) * W + 2) * sizeof(T);
}

// A wait that runs out: the thread sets SW_TIMEOUT, waits for no message any more and goes through the
// remaining columns with whatever the buffers hold, so that every CTA still meets the others at the cluster's
// barriers.  Positions may then be any integers, and rows may share one.  So the thread also sets a flag in every
// CTA's shared memory, which all of them read behind the last barrier, before anything that goes by a position
// is written; a panel that gave up, or comes after one, leaves no_interchanges.  The panels of N = 3000 take
// 193.7 us in the mean with this, 193.3 without.
constexpr unsigned kPanelWaitLimit = 1u << 22;
__device__ __forceinline__ void st_cluster_u32(uint32_t dst, unsigned v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(dst), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t mapa_u32(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ __forceinline__ void panel_give_up(int* status, int site, const unsigned* s_gave_up, int G) {
  atomicExch(status + SW_TIMEOUT, site);
  for (int d = 0; d < G; ++d) st_cluster_u32(mapa_u32(tc::smem_u32(s_gave_up), (uint32_t)d), 1u);
}
// Messages to a CTA whose wait ran out may still be in flight when all have been sent (after the last
// cluster barrier), and its shared memory has to outlive them: remote stores take about a microsecond,
// this a millisecond.
__device__ __forceinline__ void drain_messages() {
  for (int i = 0; i < 1000; ++i) __nanosleep(1000);
}

// 16 bytes into a CTA of the cluster, counted by that CTA's mbarrier.
__device__ __forceinline__ void st_async16(uint32_t dst, uint4 v, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
               "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar)
               : "memory");
}

// A row of W entries as 16-byte pieces of shared memory.
template <int W>
__device__ __forceinline__ void store_row(uint4* dst, const float2* v) {
  static_assert(W % 2 == 0, "whole 16-byte pieces");
#pragma unroll
  for (int q = 0; q < W / 2; ++q)
    dst[q] = make_uint4(__float_as_uint(v[2 * q].x), __float_as_uint(v[2 * q].y), __float_as_uint(v[2 * q + 1].x),
                        __float_as_uint(v[2 * q + 1].y));
}
template <int W>
__device__ __forceinline__ void load_row(const uint4* src, float2* v) {
#pragma unroll
  for (int q = 0; q < W / 2; ++q) {
    const uint4 x = src[q];
    v[2 * q] = make_float2(__uint_as_float(x.x), __uint_as_float(x.y));
    v[2 * q + 1] = make_float2(__uint_as_float(x.z), __uint_as_float(x.w));
  }
}
template <int W>
__device__ __forceinline__ void store_row(uint4* dst, const double2* v) {
#pragma unroll
  for (int q = 0; q < W; ++q)
    dst[q] = make_uint4((unsigned)__double2loint(v[q].x), (unsigned)__double2hiint(v[q].x),
                        (unsigned)__double2loint(v[q].y), (unsigned)__double2hiint(v[q].y));
}
template <int W>
__device__ __forceinline__ void load_row(const uint4* src, double2* v) {
#pragma unroll
  for (int q = 0; q < W; ++q) {
    const uint4 x = src[q];
    v[q] = make_double2(__hiloint2double((int)x.y, (int)x.x), __hiloint2double((int)x.w, (int)x.z));
  }
}

// crecip without a branch on which part is larger (the lanes of a warp differ there): the same
// operations on (larger, smaller), so the same bits; 0 for 0.
template <typename T> __device__ __forceinline__ T pivot_recip(T a) {
  using R = typename RealOf<T>::R;
  const bool xy = fabs(a.x) >= fabs(a.y);
  const R big = xy ? a.x : a.y, small = xy ? a.y : a.x;
  const R t = small / (big == R(0) ? R(1) : big);
  const R d = fma(small, t, big);
  const R r1 = R(1) / (d == R(0) ? R(1) : d), r2 = t / (d == R(0) ? R(1) : d);
  T r;
  r.x = xy ? r1 : r2;
  r.y = xy ? -r2 : -r1;
  if (big == R(0)) r.x = r.y = R(0);
  return r;
}

// |re| + |im| as an integer that orders like it (NaN above all), and its mag_hi key.
__device__ __forceinline__ unsigned growth_key(float2 v) { return __float_as_uint(cabs1(v)); }
__device__ __forceinline__ unsigned growth_key(double2 v) { return mag_hi(cabs1(v)); }
template <typename T> __device__ __forceinline__ unsigned growth_mag_hi(unsigned k) {
  return sizeof(T) == sizeof(float2) ? mag_hi((double)__uint_as_float(k)) : k;
}

// Key (lo, hi) and reciprocal of a candidate.
__device__ __forceinline__ void store_head(uint4* dst, uint2 key, float2 inv) {
  dst[0] = make_uint4(key.x, key.y, __float_as_uint(inv.x), __float_as_uint(inv.y));
}
__device__ __forceinline__ void load_head(const uint4* src, uint2& key, float2& inv) {
  const uint4 h = src[0];
  key = make_uint2(h.x, h.y);
  inv = make_float2(__uint_as_float(h.z), __uint_as_float(h.w));
}
__device__ __forceinline__ void store_head(uint4* dst, uint2 key, double2 inv) {
  dst[0] = make_uint4(key.x, key.y, 0u, 0u);
  store_row<1>(dst + 1, &inv);
}
__device__ __forceinline__ void load_head(const uint4* src, uint2& key, double2& inv) {
  key = *reinterpret_cast<const uint2*>(src);
  load_row<1>(src + 1, &inv);
}
// The lane with the largest key, given the largest high word: the high word alone decides unless
// lanes share it.
__device__ __forceinline__ int winner_lane(uint2 key, unsigned mh) {
  unsigned bal = __ballot_sync(0xffffffffu, key.y == mh);
  if (bal & (bal - 1u)) {
    const unsigned ml = __reduce_max_sync(0xffffffffu, key.y == mh ? key.x : 0u);
    bal = __ballot_sync(0xffffffffu, key.y == mh && key.x == ml);
  }
  return __ffs(bal) - 1;
}

// v - sum_k l_k u_k for the remaining columns of the CTA's active rows, right after a sub-panel:
// columns c_begin .. ncols of P, L21 in the columns l0 .. l0 + W, U12 in Us (column c at
// Us + (c - c_begin) W).  A warp takes 32 RPT rows, RPT = 2 per thread where there are more than
// 32, so that a broadcast load of U12 feeds two rows; the warps beyond the rows' take other
// columns.  active(r): row r takes part.
template <int W, int RPT, typename T, class Active>
__device__ void panel_rank_update(T* P, int rpcp, int nrows, int l0, int c_begin, int ncols, const T* Us, int warp,
                                  int lane, Active active) {
  const int RW = (nrows + 32 * RPT - 1) / (32 * RPT);
  if (RW == 0) return;
  const int ngrp = kRegPanelWarps / RW;
  const int grp = warp / RW, rw = warp - grp * RW;
  if (grp >= ngrp) return;
  int row[RPT];
  bool on[RPT], any = false;
#pragma unroll
  for (int q = 0; q < RPT; ++q) {
    const int r = 32 * (rw + q * RW) + lane;
    on[q] = r < nrows && active(r);
    row[q] = r < nrows ? r : 0;
    any |= on[q];
  }
  if (!__any_sync(0xffffffffu, any)) return;
  T l[RPT][W];
#pragma unroll
  for (int k = 0; k < W; ++k)
#pragma unroll
    for (int q = 0; q < RPT; ++q) l[q][k] = P[(size_t)(l0 + k) * rpcp + row[q]];
  for (int c = c_begin + grp; c < ncols; c += ngrp) {
    T* pc = P + (size_t)c * rpcp;
    T acc[RPT];
#pragma unroll
    for (int q = 0; q < RPT; ++q) acc[q] = pc[row[q]];
    T u[W];
    load_row<W>(reinterpret_cast<const uint4*>(Us + (size_t)(c - c_begin) * W), u);
#pragma unroll
    for (int k = 0; k < W; ++k)
#pragma unroll
      for (int q = 0; q < RPT; ++q) cfms(acc[q], l[q][k], u[k]);
#pragma unroll
    for (int q = 0; q < RPT; ++q)
      if (on[q]) pc[row[q]] = acc[q];
  }
}

// The panel of a.ncols <= NB columns and m = N - k0 rows on a.G <= 16 CTAs of a.rpc <= 256
// rows.  a.cand_rows: NB x NB scratch for the pivot rows' exchange.
template <typename T, int NB>
__global__ void __launch_bounds__(kRegPanelThreads, 1) panel_reg_kernel(PanelArgs<T> a) {
  constexpr int NT = kRegPanelThreads;
  constexpr int W = panel_width<T, NB>();
  using R = typename RealOf<T>::R;
  using PK = PivotKey<T>;
  // a candidate's 16-byte pieces: key (and FP32's reciprocal), FP64's reciprocal, row
  constexpr int kHead = sizeof(T) == sizeof(double2) ? 2 : 1;
  constexpr int kMsg = kHead + W * (int)sizeof(T) / 16;
  constexpr int kPerSt = 32 / kMsg;                                     // destinations of one warp-wide st.async
  constexpr int kSends = (kMaxClusterCTAs + kPerSt - 1) / kPerSt;  // of the warps together
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int m = a.N - a.k0;
  const int G = a.G;
  const int b = (int)blockIdx.x;
  const int r0 = b * a.rpc;
  const int nloc = max(min(r0 + a.rpc, m) - r0, 0);
  const int rpcp = a.rpc | 1;
  T* P = reinterpret_cast<T*>(smem_raw);  // [NB][rpcp]
  T* Us = reinterpret_cast<T*>(smem_raw + (((size_t)NB * rpcp * sizeof(T) + 15) & ~(size_t)15));
  __shared__ __align__(16) uint4 slot[2][kRegPanelFW][kMsg];      // a warp's candidate
  __shared__ __align__(16) uint4 rbuf[2][kMaxClusterCTAs][kMsg];  // every CTA's candidate
  __shared__ __align__(16) T lu11[W * W];  // the sub-panel's pivot rows, row-major
  __shared__ int s_pos[kRegPanelRows];     // position of every row
  __shared__ int s_prow[W];                // this CTA's row that became pivot j of the sub-panel, or -1
  __shared__ int s_ipiv[NB];
  __shared__ unsigned s_growth, s_gave_up;
  __shared__ uint64_t bar[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ncols = a.ncols;
  const int FW = (a.rpc + 31) / 32;  // warps that own rows
  constexpr uint32_t kFull = 0xffffffffu;
  constexpr uint32_t kMsgBytes = kMsg * 16;

  const int gave_up_before = tid == 0 ? a.status[SW_TIMEOUT] : 0;
  if (tid == 0) {
    s_growth = 0u;
    tc::mbar_init(&bar[0], 1);
    tc::mbar_init(&bar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (G > 1) {
      tc::mbar_expect_tx(&bar[0], G * kMsgBytes);
      if (ncols > 1) tc::mbar_expect_tx(&bar[1], G * kMsgBytes);
    }
    if (b == 0) *a.sw.n_extra = 0;
  }
  for (int c = warp; c < ncols; c += NT / 32) {
    const T* src = a.W + (size_t)(a.k0 + r0) + (size_t)(a.k0 + c) * a.ld;
    for (int lr = lane; lr < nloc; lr += 32) cp_async_elem(P + (size_t)c * rpcp + lr, src + lr);
  }
  // this lane's part of a candidate's message: piece sp to the CTAs sd + kPerSt (warp + FW i)
  const int sd = lane / kMsg, sp = lane % kMsg;
  uint32_t rdst[kSends], rbar[kSends];
  if (G > 1) {
#pragma unroll
    for (int i = 0; i < kSends; ++i) {
      const int d = sd + kPerSt * (warp + FW * i);
      const bool to = sd < kPerSt && warp < FW && d < G;
      rdst[i] = to ? mapa_u32(tc::smem_u32(&rbuf[0][b][sp]), (uint32_t)d) : 0u;
      rbar[i] = to ? mapa_u32(tc::smem_u32(&bar[0]), (uint32_t)d) : 0u;
    }
  }
  if (tid == 0) s_gave_up = gave_up_before != 0;
  cp_async_wait_all();
  if (G > 1) {
    cluster_arrive();
    cluster_wait();
  }
  int pos = r0 + tid;     // current position of this thread's row
  bool act = tid < nloc;  // a row of the trailing matrix
  bool alive = true;      // the bounded waits have not run out
  for (int c0 = 0; c0 < ncols; c0 += W) {
    const int wc = min(W, ncols - c0);
    if (tid < W) s_prow[tid] = -1;
    __syncthreads();
    if (warp < FW) {
      const bool mine = act;  // this thread's row takes part in the sub-panel
      T v[W], u[W], l = czero<T>();
#pragma unroll
      for (int c = 0; c < W; ++c) {
        v[c] = (mine && c < wc) ? P[(size_t)(c0 + c) * rpcp + tid] : czero<T>();
        u[c] = czero<T>();
      }
      // v[0] is the current column: a step moves the entries one register down, so that one copy
      // of the code serves every column (16 unrolled ones would not stay in the instruction cache).
      // The updates of v[1 ..] by the step before, and the candidate's reciprocal, run under the
      // latency of the pivot search.
      T v0 = v[0];
      bool upd = false;
      T* pcol = P + (size_t)c0 * rpcp + tid;
      for (int j = 0; j < wc; ++j, pcol += rpcp) {
        const int jj = c0 + j;
        const int par = jj & 1;
        // the warp's candidate: largest key, i.e. largest modulus, lowest position
        const uint2 key = act ? PK::key2(v0, pos) : make_uint2(0u, 0u);
        const unsigned mh = __reduce_max_sync(kFull, key.y);
        const T inv = pivot_recip(v0);
        if (j > 0) {
          if (upd) {
#pragma unroll
            for (int c = 2; c < W; ++c) {
              T t = v[c];
              cfms(t, l, u[c]);
              v[c - 1] = t;
            }
          } else {
#pragma unroll
            for (int c = 2; c < W; ++c) v[c - 1] = v[c];
          }
          v[0] = v0;
        }
        const int wl = winner_lane(key, mh);
        uint4* sl = slot[par][warp];
        if (lane == wl) {
          store_head(sl, key, inv);
          store_row<W>(sl + kHead, v);
        }
        // the CTA's candidate
        const uint4* won = sl;
        if (FW > 1) {
          asm volatile("bar.sync 1, %0;" ::"r"(FW * 32) : "memory");
          const uint2 k = lane < FW ? *reinterpret_cast<const uint2*>(&slot[par][lane][0]) : make_uint2(0u, 0u);
          won = slot[par][winner_lane(k, __reduce_max_sync(kFull, k.y))];
        } else {
          __syncwarp();
        }
        if (G > 1) {
          // to every CTA, contiguous messages
          const uint4 piece = won[sp];
#pragma unroll
          for (int i = 0; i < kSends; ++i) {
            if (FW * i * kPerSt >= G) break;
            if (rbar[i]) st_async16(rdst[i] + par * (uint32_t)sizeof(rbuf[0]), piece, rbar[i] + par * 8u);
          }
          if (alive) {
            unsigned it = 0;
            while (!tc::mbar_try_wait(&bar[par], (uint32_t)(jj >> 1) & 1u))
              if (++it >= kPanelWaitLimit) {
                panel_give_up(a.status, 2, &s_gave_up, G);
                alive = false;
                break;
              }
          }
          const uint2 k = lane < G ? *reinterpret_cast<const uint2*>(&rbuf[par][lane][0]) : make_uint2(0u, 0u);
          won = rbuf[par][winner_lane(k, __reduce_max_sync(kFull, k.y))];
        }
        uint2 wk;
        T winv;
        load_head(won, wk, winv);
        load_row<W>(won + kHead, u);
        const int p = PK::row2(wk);
        upd = act && pos != p;
        l = v[0];
        if (upd) l = cmul(l, winv);
        v0 = v[1 < W ? 1 : 0];
        if (upd) cfms(v0, l, u[1 < W ? 1 : 0]);
        if (upd) {
          if (pos == jj) pos = p;
        } else if (act) {  // this row is the pivot: final
          act = false;
          pos = jj;
          s_prow[j] = tid;
        }
        if (mine) *pcol = l;
        s_ipiv[jj] = p;  // every thread the same value
        if (G > 1 && tid == 0 && alive && jj + 2 < ncols) tc::mbar_expect_tx(&bar[par], G * kMsgBytes);
      }
      if (tid < kRegPanelRows) s_pos[tid] = pos;
    }
    const int c1 = c0 + W;
    __syncthreads();
    if (c1 >= ncols) break;
    // the pivot rows, from the sub-panel's columns on, to every CTA
    const int rem = ncols - c1;
    if (G > 1) {
      for (int idx = tid; idx < W * NB; idx += NT) {
        const int j = idx / NB, c = idx % NB;
        const int pr = s_prow[j];
        if (pr >= 0 && c >= c0 && c < ncols) __stcg(a.cand_rows + (size_t)(c0 + j) * NB + c, P[(size_t)c * rpcp + pr]);
      }
      cluster_arrive();
      cluster_wait();
    }
    // U12 = L11^-1 A12, one column per thread, by columns of L11 (lu11: column-major)
    T x[W];
    if (tid < rem) {
      const int c = c1 + tid;
#pragma unroll
      for (int j = 0; j < W; ++j)
        x[j] = G > 1 ? __ldcg(a.cand_rows + (size_t)(c0 + j) * NB + c) : P[(size_t)c * rpcp + s_prow[j]];
    }
    for (int idx = tid; idx < W * W; idx += NT) {
      const int j = idx / W, k = idx % W;
      lu11[k * W + j] = G > 1 ? __ldcg(a.cand_rows + (size_t)(c0 + j) * NB + c0 + k) : P[(size_t)(c0 + k) * rpcp + s_prow[j]];
    }
    __syncthreads();
    if (tid < rem) {
      const int c = c1 + tid;
#pragma unroll
      for (int k = 0; k < W - 1; ++k) {
        T lk[W];
        load_row<W>(reinterpret_cast<const uint4*>(lu11 + k * W), lk);
#pragma unroll
        for (int j = k + 1; j < W; ++j) cfms(x[j], lk[j], x[k]);
      }
      store_row<W>(reinterpret_cast<uint4*>(Us + (size_t)tid * W), x);
      T* pc = P + (size_t)c * rpcp;
#pragma unroll
      for (int j = 0; j < W; ++j) {
        const int pr = s_prow[j];
        if (pr >= 0) pc[pr] = x[j];
      }
    }
    __syncthreads();
    auto active = [&](int r) { return s_pos[r] >= c1; };
    if (FW > 1)
      panel_rank_update<W, 2>(P, rpcp, nloc, c0, c1, ncols, Us, warp, lane, active);
    else
      panel_rank_update<W, 1>(P, rpcp, nloc, c0, c1, ncols, Us, warp, lane, active);
  }
  // no CTA leaves while another may still write into its shared memory (and every row of W was
  // read, before the first exchange, before any is written)
  if (G > 1) {
    cluster_arrive();
    cluster_wait();
    if (s_gave_up) {
      if (b == 0) no_interchanges(a.sw, a.ipiv, a.k0, ncols, tid, NT);
      if (!alive) drain_messages();
      return;
    }
  }
  // write back: row lr to its position
  for (int rg = 0; rg < FW; ++rg) {
    const int lr = rg * 32 + lane;
    if (lr >= nloc) break;
    T* dst = a.W + (size_t)(a.k0 + s_pos[lr]) + (size_t)a.k0 * a.ld;
    const T* src = P + lr;
#pragma unroll 8
    for (int c = warp; c < ncols; c += NT / 32) dst[(size_t)c * a.ld] = src[(size_t)c * rpcp];
  }
  // pivot rows: max |u_ij|, and a zero pivot (the first one goes to info)
  if (tid < nloc && s_pos[tid] < ncols) {
    const int ps = s_pos[tid];
    unsigned g = 0u;
#pragma unroll 4
    for (int c = ps; c < ncols; ++c) g = max(g, growth_key(P[(size_t)c * rpcp + tid]));
    atomicMax(&s_growth, growth_mag_hi<T>(g));
    const T d = P[(size_t)ps * rpcp + tid];
    if (d.x == R(0) && d.y == R(0)) {
      const int col = a.k0 + ps + 1;
      if (atomicCAS(a.status + SW_INFO, 0, col) > col) atomicMin(a.status + SW_INFO, col);
    }
  }
  if (a.lup != nullptr) {  // L21 rows into the LU planes: consecutive threads on consecutive columns
#pragma unroll 2
    for (int lr = warp; lr < nloc; lr += NT / 32) {
      const int ps = s_pos[lr];
      if (ps < ncols) continue;
      float* dst = a.lup + (size_t)(a.k0 + ps) * a.lup_ld + a.k0;
#pragma unroll
      for (int c = lane; c < NB; c += 32) {
        if (c >= ncols) break;
        const T v = P[(size_t)c * rpcp + lr];
        float hr, lrr, hi_, li;
        tf32_split((float)v.x, hr, lrr);
        tf32_split((float)v.y, hi_, li);
        dst[c] = hr;
        dst[a.lup_plane + c] = lrr;
        dst[2 * a.lup_plane + c] = hi_;
        dst[3 * a.lup_plane + c] = li;
      }
    }
  }
  // the step's row interchanges: panel row r0 + tid ended at pos
  if (tid < nloc) {
    const int src = a.k0 + r0 + tid, dst = a.k0 + s_pos[tid];
    if (dst < a.k0 + ncols) {
      a.sw.top_src[dst - a.k0] = src;
    } else if (dst != src) {
      const int e = atomicAdd(a.sw.n_extra, 1);
      a.sw.extra_dst[e] = dst;
      a.sw.extra_src[e] = src;
    }
  }
  if (b == 0 && tid < ncols) a.ipiv[a.k0 + tid] = a.k0 + s_ipiv[tid];
  __syncthreads();
  if (tid == 0 && a.growth_bits && s_growth > 0u) atomicMax(a.growth_bits, s_growth);
}

// ---------------------------------------------------------------- tall panels
// A panel whose rows exceed one cluster's shared memory, in sub-panels of kSubW = 16 columns over
// global memory (L2):
//   panel_sub_kernel   one cluster of 16 CTAs factors 16 columns of all rows, as panel_reg_kernel does
//                      (8 columns at a time in registers, RPT rows per thread); rows stay in place,
//                      their positions in pos[] carry over from sub-panel to sub-panel;
//   panel_rest_kernel  all SMs: U12 = L11^-1 A12 of the 16 pivot rows and the rank-16 update of the
//                      panel's remaining columns; U12 goes to ubuf, the pivot rows stay as they were
//                      (other CTAs read them);
//   panel_planes_kernel, panel_place_kernel  after the last sub-panel: the L21 rows into the LU
//                      planes, and the pivot and displaced rows to their final places.
// Against panel_kernel (a grid barrier per column, 3.6-4.4 us): a column costs about 0.8 us, a
// sub-panel's load, store and update 10-20 us more.  Measured, 128 columns FP32: 3100-6400 rows 500 ->
// 320 us, 25600 rows 700 -> 570 us (a kernel per 1, 2, 3, 4 rows a thread: 30, 39, 47, 58 us a
// sub-panel); the factorisation at N = 6400 28 -> 22.9 ms, 25600 357 -> 326 ms; FP64, N = 4000,
// 20.0 -> 18.7 ms.  The same factors bit for bit.
constexpr int kSubW = 16, kSubIW = 8;
constexpr int kSubThreads = 512, kSubWarps = kSubThreads / 32;

template <typename T>
struct SubArgs {
  T* W;
  long ld;
  int N, k0, ncols;      // the panel
  int c0;                // first column of the sub-panel, panel-relative
  int rpc, G;            // rows per CTA, CTAs (one cluster)
  int* pos;              // [m] position of every row of the panel (written by c0 = 0)
  int* prow;             // [NB] row that became pivot j
  T* xrows;              // [kSubW][kSubW] exchange of the first half's pivot rows
  T* ubuf;               // [NB][ldu] U rows right of their sub-panel
  int ldu;
  int* ipiv;
  int* status;
  StepSwaps sw;
  unsigned* growth_bits;
  float* lup;
  long lup_ld, lup_plane;
};

template <typename T>
__host__ __device__ constexpr size_t panel_sub_smem(int rpc) {
  return (size_t)kSubW * (size_t)(rpc | 1) * sizeof(T) + 16;
}

template <typename T, int RPT>
__global__ void __launch_bounds__(kSubThreads, 1) panel_sub_kernel(SubArgs<T> a) {
  constexpr int NT = kSubThreads, W = kSubW, IW = kSubIW;
  using PK = PivotKey<T>;
  constexpr int kHead = sizeof(T) == sizeof(double2) ? 2 : 1;
  constexpr int kMsg = kHead + IW * (int)sizeof(T) / 16;
  constexpr int kPerSt = 32 / kMsg;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int m = a.N - a.k0;
  const int G = a.G, b = (int)blockIdx.x;
  const int r0 = b * a.rpc;
  const int nloc = max(min(r0 + a.rpc, m) - r0, 0);
  const int rpcp = a.rpc | 1;
  T* P = reinterpret_cast<T*>(smem_raw);  // [W][rpcp]
  __shared__ __align__(16) uint4 slot[2][kSubWarps][kMsg];
  __shared__ __align__(16) uint4 rbuf[2][kMaxClusterCTAs][kMsg];
  __shared__ __align__(16) T lu[W * W], u12[IW * IW];
  __shared__ int s_prow[W], s_ipiv[W];
  __shared__ unsigned s_gave_up;
  __shared__ uint64_t bar[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wc = min(W, a.ncols - a.c0);
  const int FW = min(kSubWarps, (a.rpc + 31) / 32);
  constexpr uint32_t kFull = 0xffffffffu;
  constexpr uint32_t kMsgBytes = kMsg * 16;
  const int gave_up_before = tid == 0 ? a.status[SW_TIMEOUT] : 0;
  if (tid == 0) {
    tc::mbar_init(&bar[0], 1);
    tc::mbar_init(&bar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    tc::mbar_expect_tx(&bar[0], G * kMsgBytes);
    if (wc > 1) tc::mbar_expect_tx(&bar[1], G * kMsgBytes);
    if (b == 0 && a.c0 == 0) *a.sw.n_extra = 0;
  }
  if (tid < W) s_prow[tid] = -1;
  if (b == 0 && tid < wc) a.prow[a.c0 + tid] = a.c0 + tid;  // a row for panel_rest_kernel should none become the pivot
  for (int c = 0; c < wc; ++c) {
    const T* src = a.W + (size_t)(a.k0 + r0) + (size_t)(a.k0 + a.c0 + c) * a.ld;
    for (int lr = tid; lr < nloc; lr += NT) cp_async_elem(P + (size_t)c * rpcp + lr, src + lr);
  }
  int pos[RPT];
  bool act[RPT], mine[RPT];
#pragma unroll
  for (int q = 0; q < RPT; ++q) {
    const int lr = tid + q * NT;
    pos[q] = lr < nloc ? (a.c0 == 0 ? r0 + lr : a.pos[r0 + lr]) : 0;
    mine[q] = act[q] = lr < nloc && pos[q] >= a.c0;
  }
  const int sd = lane / kMsg, sp = lane % kMsg;
  constexpr int kSends = (kMaxClusterCTAs + kPerSt - 1) / kPerSt;
  uint32_t rdst[kSends], rbar[kSends];
#pragma unroll
  for (int i = 0; i < kSends; ++i) {
    const int d = sd + kPerSt * (warp + FW * i);
    const bool to = sd < kPerSt && warp < FW && d < G;
    rdst[i] = to ? mapa_u32(tc::smem_u32(&rbuf[0][b][sp]), (uint32_t)d) : 0u;
    rbar[i] = to ? mapa_u32(tc::smem_u32(&bar[0]), (uint32_t)d) : 0u;
  }
  if (tid == 0) s_gave_up = gave_up_before != 0;
  cp_async_wait_all();
  cluster_arrive();
  cluster_wait();
  __syncthreads();
  bool alive = true;
  for (int pc = 0; pc < wc; pc += IW) {
    const int wp = min(IW, wc - pc);
    if (warp < FW) {
      T v[RPT][IW], u[IW], l[RPT], v0[RPT];
      bool upd[RPT];
#pragma unroll
      for (int q = 0; q < RPT; ++q) {
#pragma unroll
        for (int c = 0; c < IW; ++c)
          v[q][c] = (act[q] && c < wp) ? P[(size_t)(pc + c) * rpcp + tid + q * NT] : czero<T>();
        l[q] = czero<T>();
        v0[q] = v[q][0];
        upd[q] = false;
      }
      bool held[RPT];  // rows that take part in this half
#pragma unroll
      for (int q = 0; q < RPT; ++q) held[q] = act[q];
#pragma unroll
      for (int c = 0; c < IW; ++c) u[c] = czero<T>();
      T* pcol = P + (size_t)pc * rpcp + tid;
      for (int j = 0; j < wp; ++j, pcol += rpcp) {
        const int jl = pc + j, jj = a.c0 + jl, par = jl & 1;
        uint2 key = make_uint2(0u, 0u);
        int bq = 0;
        T vb = v0[0];
#pragma unroll
        for (int q = 0; q < RPT; ++q) {
          const uint2 kq = act[q] ? PK::key2(v0[q], pos[q]) : make_uint2(0u, 0u);
          if (kq.y > key.y || (kq.y == key.y && kq.x > key.x)) {
            key = kq;
            bq = q;
            vb = v0[q];
          }
        }
        const unsigned mh = __reduce_max_sync(kFull, key.y);
        const T inv = pivot_recip(vb);
        if (j > 0) {
#pragma unroll
          for (int q = 0; q < RPT; ++q) {
            if (upd[q]) {
#pragma unroll
              for (int c = 2; c < IW; ++c) {
                T t = v[q][c];
                cfms(t, l[q], u[c]);
                v[q][c - 1] = t;
              }
            } else {
#pragma unroll
              for (int c = 2; c < IW; ++c) v[q][c - 1] = v[q][c];
            }
            v[q][0] = v0[q];
          }
        }
        const int wl = winner_lane(key, mh);
        uint4* sl = slot[par][warp];
        if (lane == wl) {
          store_head(sl, key, inv);
#pragma unroll
          for (int q = 0; q < RPT; ++q)
            if (bq == q) store_row<IW>(sl + kHead, v[q]);
        }
        asm volatile("bar.sync 1, %0;" ::"r"(FW * 32) : "memory");
        const uint4* won;
        {
          const uint2 k = lane < FW ? *reinterpret_cast<const uint2*>(&slot[par][lane][0]) : make_uint2(0u, 0u);
          won = slot[par][winner_lane(k, __reduce_max_sync(kFull, k.y))];
        }
        {
          const uint4 piece = won[sp];
#pragma unroll
          for (int i = 0; i < kSends; ++i) {
            if (FW * i * kPerSt >= G) break;
            if (rbar[i]) st_async16(rdst[i] + par * (uint32_t)sizeof(rbuf[0]), piece, rbar[i] + par * 8u);
          }
          if (alive) {
            unsigned it = 0;
            while (!tc::mbar_try_wait(&bar[par], (uint32_t)(jl >> 1) & 1u))
              if (++it >= kPanelWaitLimit) {
                panel_give_up(a.status, 3, &s_gave_up, G);
                alive = false;
                break;
              }
          }
          const uint2 k = lane < G ? *reinterpret_cast<const uint2*>(&rbuf[par][lane][0]) : make_uint2(0u, 0u);
          won = rbuf[par][winner_lane(k, __reduce_max_sync(kFull, k.y))];
        }
        uint2 wk;
        T winv;
        load_head(won, wk, winv);
        load_row<IW>(won + kHead, u);
        const int p = PK::row2(wk);
#pragma unroll
        for (int q = 0; q < RPT; ++q) {
          upd[q] = act[q] && pos[q] != p;
          l[q] = v[q][0];
          if (upd[q]) l[q] = cmul(l[q], winv);
          v0[q] = v[q][1];
          if (upd[q]) {
            cfms(v0[q], l[q], u[1]);
            if (pos[q] == jj) pos[q] = p;
          } else if (act[q]) {  // this row is the pivot: final
            act[q] = false;
            pos[q] = jj;
            s_prow[jl] = tid + q * NT;
          }
          if (held[q]) pcol[q * NT] = l[q];
        }
        s_ipiv[jl] = p;  // every thread the same value
        if (tid == 0 && alive && jl + 2 < wc) tc::mbar_expect_tx(&bar[par], G * kMsgBytes);
      }
    }
    __syncthreads();
    if (pc + IW >= wc) break;
    // the first half's pivot rows (L11 and the raw second half) to every CTA
    for (int idx = tid; idx < IW * W; idx += NT) {
      const int j = idx / W, c = idx % W;
      const int pr = s_prow[pc + j];
      if (pr >= 0) __stcg(a.xrows + idx, P[(size_t)c * rpcp + pr]);
    }
    cluster_arrive();
    cluster_wait();
    if (tid < IW * W) lu[tid] = __ldcg(a.xrows + tid);
    __syncthreads();
    if (tid < IW) {  // U12, one column per thread
      T x[IW];
#pragma unroll
      for (int j = 0; j < IW; ++j) x[j] = lu[j * W + IW + tid];
#pragma unroll
      for (int k = 0; k < IW - 1; ++k)
#pragma unroll
        for (int j = k + 1; j < IW; ++j) cfms(x[j], lu[j * W + k], x[k]);
#pragma unroll
      for (int j = 0; j < IW; ++j) {
        u12[j * IW + tid] = x[j];
        const int pr = s_prow[pc + j];
        if (pr >= 0) P[(size_t)(IW + tid) * rpcp + pr] = x[j];
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < RPT; ++q) {
      if (!act[q]) continue;
      T* pr = P + tid + q * NT;
      T lr[IW];
#pragma unroll
      for (int k = 0; k < IW; ++k) lr[k] = pr[(size_t)k * rpcp];
#pragma unroll
      for (int c = 0; c < IW; ++c) {
        if (IW + c >= wc) break;
        T t = pr[(size_t)(IW + c) * rpcp];
#pragma unroll
        for (int k = 0; k < IW; ++k) cfms(t, lr[k], u12[k * IW + c]);
        pr[(size_t)(IW + c) * rpcp] = t;
      }
    }
    // (a thread's own rows; the next half's loads are its own too)
  }
  cluster_arrive();
  cluster_wait();
  // (before the last sub-panel positions are only compared and prow is the one index)
  const bool last = a.c0 + W >= a.ncols, gave_up = last && s_gave_up;
  if (gave_up && b == 0) no_interchanges(a.sw, a.ipiv, a.k0, a.ncols, tid, NT);
  // the sub-panel back in place, positions, pivots
#pragma unroll
  for (int q = 0; q < RPT; ++q) {
    const int lr = tid + q * NT;
    if (lr >= nloc) continue;
    if (mine[q]) {
      T* dst = a.W + (size_t)(a.k0 + r0 + lr) + (size_t)(a.k0 + a.c0) * a.ld;
#pragma unroll
      for (int c = 0; c < W; ++c)
        if (c < wc) dst[(size_t)c * a.ld] = P[(size_t)c * rpcp + lr];
    }
    a.pos[r0 + lr] = gave_up ? r0 + lr : pos[q];
    if (last && !gave_up) {  // the step's row interchanges
      const int src = a.k0 + r0 + lr, dst = a.k0 + pos[q];
      if (pos[q] < a.ncols) {
        a.sw.top_src[pos[q]] = src;
      } else if (dst != src) {
        const int e = atomicAdd(a.sw.n_extra, 1);
        a.sw.extra_dst[e] = dst;
        a.sw.extra_src[e] = src;
      }
    }
  }
  if (tid < wc && s_prow[tid] >= 0) a.prow[a.c0 + tid] = r0 + s_prow[tid];
  if (b == 0 && tid < wc && !gave_up) a.ipiv[a.k0 + a.c0 + tid] = a.k0 + s_ipiv[tid];
  if (!alive) drain_messages();
}

// 64 rows per CTA of 256 threads: 2 x 32 rows, four column groups.
constexpr int kRestRows = 64;
template <typename T, int NB>
__global__ void __launch_bounds__(256) panel_rest_kernel(SubArgs<T> a) {
  constexpr int W = kSubW;
  __shared__ __align__(16) T lu[W * W];        // L11, column-major
  __shared__ __align__(16) T Us[(NB > W ? NB - W : 1) * W];  // U12, W consecutive values per column
  __shared__ int s_prow[W];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m = a.N - a.k0, c1 = a.c0 + W, rem = a.ncols - c1;
  const int row = blockIdx.x * kRestRows + (warp & 1) * 32 + lane;
  const bool on = row < m && a.pos[row] >= c1;
  T l[W];
  {  // this row's multipliers, in flight while U12 is formed
    const T* src = a.W + (size_t)(a.k0 + min(row, m - 1)) + (size_t)(a.k0 + a.c0) * a.ld;
#pragma unroll
    for (int k = 0; k < W; ++k) l[k] = src[(size_t)k * a.ld];
  }
  if (tid < W) s_prow[tid] = a.prow[a.c0 + tid];
  __syncthreads();
  T x[W];
  if (tid < rem) {
    const T* src = a.W + (size_t)a.k0 + (size_t)(a.k0 + c1 + tid) * a.ld;
#pragma unroll
    for (int j = 0; j < W; ++j) x[j] = src[s_prow[j]];
  }
  {
    const int j = tid % W, k = tid / W;
    lu[k * W + j] = a.W[(size_t)(a.k0 + s_prow[j]) + (size_t)(a.k0 + a.c0 + k) * a.ld];
  }
  __syncthreads();
  if (tid < rem) {
#pragma unroll
    for (int k = 0; k < W - 1; ++k) {
      T lk[W];
      load_row<W>(reinterpret_cast<const uint4*>(lu + k * W), lk);
#pragma unroll
      for (int j = k + 1; j < W; ++j) cfms(x[j], lk[j], x[k]);
    }
    store_row<W>(reinterpret_cast<uint4*>(Us + (size_t)tid * W), x);
    if (blockIdx.x == 0)
#pragma unroll
      for (int j = 0; j < W; ++j) a.ubuf[(size_t)(a.c0 + j) * a.ldu + c1 + tid] = x[j];
  }
  __syncthreads();
  if (!on) return;
  T* dst = a.W + (size_t)(a.k0 + row) + (size_t)(a.k0 + c1) * a.ld;
#pragma unroll 2
  for (int c = warp >> 1; c < rem; c += 4) {
    T v = dst[(size_t)c * a.ld];
    T u[W];
    load_row<W>(reinterpret_cast<const uint4*>(Us + (size_t)c * W), u);
#pragma unroll
    for (int k = 0; k < W; ++k) cfms(v, l[k], u[k]);
    dst[(size_t)c * a.ld] = v;
  }
}

// L21 rows (positions >= ncols) into the LU planes: 32 rows x 128 columns per CTA through shared
// memory, so that both sides are coalesced.
template <int NB>
__global__ void __launch_bounds__(256) panel_planes_kernel(SubArgs<float2> a) {
  __shared__ float2 tile[32][NB + 1];
  __shared__ int s_pos[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m = a.N - a.k0, r0 = blockIdx.x * 32;
  if (tid < 32) s_pos[tid] = r0 + tid < m ? a.pos[r0 + tid] : -1;
  const float2* src = a.W + (size_t)(a.k0 + r0 + lane) + (size_t)a.k0 * a.ld;
  if (r0 + lane < m)
#pragma unroll 8
    for (int c = warp; c < a.ncols; c += 8) tile[lane][c] = src[(size_t)c * a.ld];
  __syncthreads();
  for (int lr = warp; lr < 32; lr += 8) {
    const int ps = s_pos[lr];
    if (ps < a.ncols) continue;
    float* dst = a.lup + (size_t)(a.k0 + ps) * a.lup_ld + a.k0;
    for (int c = lane; c < a.ncols; c += 32) {
      const float2 v = tile[lr][c];
      float hr, lrr, hi_, li;
      tf32_split(v.x, hr, lrr);
      tf32_split(v.y, hi_, li);
      dst[c] = hr;
      dst[a.lup_plane + c] = lrr;
      dst[2 * a.lup_plane + c] = hi_;
      dst[3 * a.lup_plane + c] = li;
    }
  }
}

// Pivot rows (with their U columns from ubuf) and displaced rows to their final places, 8 columns
// per CTA; max |u_ij| and zero pivots.  At most NB pivot rows and as many displaced ones.
constexpr int kPlaceCols = 8;
template <typename T, int NB>
__global__ void __launch_bounds__(256) panel_place_kernel(SubArgs<T> a) {
  using R = typename RealOf<T>::R;
  __shared__ __align__(16) T tmp[kPlaceCols][2 * NB];
  __shared__ int s_src[2 * NB], s_dst[2 * NB];
  const int tid = threadIdx.x;
  const int ne = *a.sw.n_extra, cnt = a.ncols + ne;
  const int cb = blockIdx.x * kPlaceCols, nc = min(kPlaceCols, a.ncols - cb);
  for (int i = tid; i < cnt; i += 256) {
    s_src[i] = i < a.ncols ? a.sw.top_src[i] : a.sw.extra_src[i - a.ncols];
    s_dst[i] = i < a.ncols ? a.k0 + i : a.sw.extra_dst[i - a.ncols];
  }
  __syncthreads();
  unsigned g = 0u;
  for (int idx = tid; idx < cnt * nc; idx += 256) {
    const int i = idx % cnt, cc = idx / cnt, c = cb + cc;
    T v;
    if (i < a.ncols && c >= (i / kSubW + 1) * kSubW)
      v = a.ubuf[(size_t)i * a.ldu + c];
    else
      v = a.W[(size_t)s_src[i] + (size_t)(a.k0 + c) * a.ld];
    tmp[cc][i] = v;
    if (c >= i) g = max(g, growth_key(v));
    if (c == i && v.x == R(0) && v.y == R(0)) {  // zero pivot: the first one goes to info
      const int col = a.k0 + c + 1;
      if (atomicCAS(a.status + SW_INFO, 0, col) > col) atomicMin(a.status + SW_INFO, col);
    }
  }
  __syncthreads();
  for (int idx = tid; idx < cnt * nc; idx += 256) {
    const int i = idx % cnt, cc = idx / cnt;
    a.W[(size_t)s_dst[i] + (size_t)(a.k0 + cb + cc) * a.ld] = tmp[cc][i];
  }
  g = __reduce_max_sync(0xffffffffu, g);
  if ((tid & 31) == 0 && g > 0u && a.growth_bits) atomicMax(a.growth_bits, growth_mag_hi<T>(g));
}

}  // namespace hprmat
