// Blocked right-looking complex LU with partial pivoting, and the triangular solves that
// use its factors.  Templates over the complex element type T (double2 = FP64 path,
// float2 = panels/solves of the mixed path).
//
// Storage: the matrix W is column-major with leading dimension ld (complex elements).
// Block step s factors columns [k0, k0+ncols) with k0 = s*nb:
//   1. the panel: panel_reg_kernel (panel.cuh) where the rows fit in one thread-block cluster, its
//      sub-panels (panel_sub_kernel, panel_rest_kernel) where 16 columns of them do,
//      else panel_kernel -- cooperative launch, the panel rows spread over all SMs and held
//                           in shared memory; one grid barrier per column: every CTA posts
//                           its local |re|+|im| maximum (the modulus LAPACK's izamax uses)
//                           and that row, then all CTAs pick the same pivot, swap and
//                           eliminate their rows.  Writes ipiv and the step's row-interchange
//                           list.
//   2. trsm_reg_kernel   -- applies the step's row interchanges to the columns right of the
//                           panel and solves with the unit lower diagonal block:
//                           U12 = L11^-1 P A12.
//   3. trailing update   -- A22 -= L21 U12 (cgemm_update_kernel here; the mixed path uses
//                           the tcgen05 kernel of tc_gemm.cu).
// Row interchanges are applied only to columns at or right of the current panel; the
// forward solve applies each step's interchanges to the right-hand side just before that
// step's block column, which is consistent with the factors stored that way.
#pragma once
#include "common.cuh"

namespace hprmat {

constexpr int kMaxNB = 128;

// Row-interchange list of one block step (global row indices).
struct StepSwaps {
  int* top_src;    // [nbmax]  source row of final row k0+j, j < ncols
  int* extra_dst;  // [nbmax]  rows >= k0+ncols that receive a displaced row
  int* extra_src;  // [nbmax]
  int* n_extra;    // [1]
};

template <typename T>
struct PanelArgs {
  T* W;
  long ld;
  int N, k0, ncols, rpc, G;
  int* ipiv;                      // [N] global pivot rows (0-based)
  T* cand_rows;                   // [2][G][NB]
  unsigned long long* keys;       // [NB] winning pivot key per panel column (zeroed per launch)
  T* rowj;                        // [2][NB]
  int* status;                    // device status block
  StepSwaps sw;
  unsigned* growth_bits;          // running max |u_ij| (mag_hi key)
  // Optional (mixed path): the "LU planes", hi/lo TF32 splits of Re/Im of the factors,
  // row-major (row stride lup_ld floats, planes lup_plane floats apart).  The panel writes
  // its L21 rows there; they are the K-major A operand of the tensor-core updates.
  float* lup;
  long lup_ld;
  long lup_plane;
  // Optional timing trace, per column kPanelTraceW stamps: CTA 0 at column start, candidate
  // posted, barrier passed, pivot row in place, update done; then every CTA's arrival.
  long long* trace = nullptr;
};
constexpr int kPanelTraceW = 5 + 160;

// Pivot candidates are compared by PivotKey<T> (common.cuh): |re|+|im| as an integer key
// that orders over the element type's whole range (FP64 panels: magnitudes far outside the
// float range too), with the lowest row winning among equal moduli.

// The interchange list and pivots of a panel that gave up (a bounded wait ran out): no row moves, so
// that the kernels behind it in the stream find valid rows until the host reads SW_TIMEOUT.
__device__ __forceinline__ void no_interchanges(const StepSwaps& sw, int* ipiv, int k0, int ncols, int tid, int nthreads) {
  for (int j = tid; j < ncols; j += nthreads) sw.top_src[j] = ipiv[k0 + j] = k0 + j;
  if (tid == 0) *sw.n_extra = 0;
}

// End of panel_kernel: the CTA's factored rows back into W, its L21 rows into the LU planes (mixed
// path), and from CTA 0 the pivots, the growth and the step's row-interchange list.
template <typename T, int NB, int NT>
__device__ void panel_finish(const PanelArgs<T>& a, const T* P, int rpcp, int r0, int nloc, const int* s_loc_ipiv,
                             unsigned s_growth, int b, int tid) {
  const int ncols = a.ncols;
  // write the factored rows back
  for (int c = 0; c < ncols; ++c)
    for (int lr = tid; lr < nloc; lr += NT)
      a.W[(size_t)(a.k0 + r0 + lr) + (size_t)(a.k0 + c) * a.ld] = P[(size_t)c * rpcp + lr];
  // L21 rows into the LU planes (mixed path): global row k0 + g, columns k0 .. k0+ncols
  if (a.lup != nullptr) {
    const int lr0 = max(ncols - r0, 0);
    const int nl = nloc - lr0;
    for (int idx = tid; idx < nl * ncols; idx += NT) {
      int c = idx % ncols;
      int lr = lr0 + idx / ncols;
      size_t off = (size_t)(a.k0 + r0 + lr) * a.lup_ld + (size_t)(a.k0 + c);
      float hr, lrr, hi_, li;
      T v = P[(size_t)c * rpcp + lr];
      tf32_split((float)v.x, hr, lrr);
      tf32_split((float)v.y, hi_, li);
      a.lup[off] = hr;
      a.lup[a.lup_plane + off] = lrr;
      a.lup[2 * a.lup_plane + off] = hi_;
      a.lup[3 * a.lup_plane + off] = li;
    }
  }
  if (b == 0) {
    __syncthreads();
    if (tid < ncols) a.ipiv[a.k0 + tid] = a.k0 + s_loc_ipiv[tid];
    if (tid == 0 && a.growth_bits) atomicMax(a.growth_bits, s_growth);
    // Row-interchange list of this step: simulate the swaps on the touched positions.
    if (tid < 32) {
      __shared__ int pos[2 * NB], src[2 * NB];
      __shared__ int cnt;
      for (int j = tid; j < ncols; j += 32) { pos[j] = a.k0 + j; src[j] = a.k0 + j; }
      if (tid == 0) cnt = ncols;
      __syncwarp();
      for (int j = 0; j < ncols; ++j) {
        int bp = a.k0 + s_loc_ipiv[j];
        if (bp == a.k0 + j) continue;
        int slot;
        if (bp < a.k0 + ncols) {
          slot = bp - a.k0;
        } else {
          int found = -1;
          for (int base = ncols; base < cnt; base += 32) {
            int s = base + tid;
            unsigned m_ = __ballot_sync(0xffffffffu, s < cnt && pos[s] == bp);
            if (m_) { found = base + __ffs(m_) - 1; break; }
          }
          if (found < 0) {
            if (tid == 0) { pos[cnt] = bp; src[cnt] = bp; cnt = cnt + 1; }
            __syncwarp();
            found = cnt - 1;
          }
          slot = found;
        }
        if (tid == 0) { int t = src[j]; src[j] = src[slot]; src[slot] = t; }
        __syncwarp();
      }
      for (int j = tid; j < ncols; j += 32) a.sw.top_src[j] = src[j];
      if (tid == 0) {
        int ne = 0;
        for (int s = ncols; s < cnt; ++s)
          if (src[s] != pos[s]) { a.sw.extra_dst[ne] = pos[s]; a.sw.extra_src[ne] = src[s]; ++ne; }
        *a.sw.n_extra = ne;
      }
    }
  }
}

template <typename T, int NB, int NT>
__global__ void __launch_bounds__(NT, 1) panel_kernel(PanelArgs<T> a) {
  using R = typename RealOf<T>::R;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int m = a.N - a.k0;
  const int b = blockIdx.x;
  const int r0 = b * a.rpc;
  const int r1 = min(r0 + a.rpc, m);
  const int nloc = max(r1 - r0, 0);
  const int rpcp = a.rpc | 1;  // odd column stride: conflict-free row gathers
  T* P = reinterpret_cast<T*>(smem_raw);                 // [NB][rpcp] column-major
  T* urow = P + (size_t)NB * rpcp;                       // [NB]
  using PK = PivotKey<T>;
  using PM = typename PK::M;
  __shared__ PM red_v[NT / 32];
  __shared__ int red_i[NT / 32];
  __shared__ int s_piv, s_loc_ipiv[NB];
  __shared__ unsigned s_growth;
  const int tid = threadIdx.x;
  const int ncols = a.ncols;

  // load rows [r0, r1) of the panel
  for (int c = 0; c < ncols; ++c)
    for (int lr = tid; lr < nloc; lr += NT)
      P[(size_t)c * rpcp + lr] = a.W[(size_t)(a.k0 + r0 + lr) + (size_t)(a.k0 + c) * a.ld];
  if (tid == 0) s_growth = 0u;
  __syncthreads();

  // Column jc's pivot candidate: the largest |re|+|im| of the local rows >= jc (lowest row on
  // ties) into s_piv, and its key into the column's global maximum.  v_of(lr) gives the
  // current value of column jc in local row lr.
  auto candidate = [&](int jc, PM bv, int bi) {
    for (int o = 16; o > 0; o >>= 1) {
      PM ov = __shfl_down_sync(0xffffffffu, bv, o);
      int oi = __shfl_down_sync(0xffffffffu, bi, o);
      if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    if ((tid & 31) == 0) { red_v[tid >> 5] = bv; red_i[tid >> 5] = bi; }
    __syncthreads();
    if (tid < 32) {
      bv = (tid < NT / 32) ? red_v[tid] : PM(0);
      bi = (tid < NT / 32) ? red_i[tid] : 0x7fffffff;
      for (int o = 16; o > 0; o >>= 1) {
        PM ov = __shfl_down_sync(0xffffffffu, bv, o);
        int oi = __shfl_down_sync(0xffffffffu, bi, o);
        if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
      }
      if (tid == 0) {
        s_piv = bi;
        if (bi != 0x7fffffff) atomicMax(a.keys + jc, PK::key(bv, bi));
      }
    }
    __syncthreads();
  };
  // Post the candidate row of column jc and, from its owner, row jc.  Columns > jc still
  // wait for the rank-1 update of column jc - 1 (multipliers in column jc - 1, pivot row in
  // urow) when pend is set; the posted values include it.
  auto post = [&](int jc, bool pend) {
    const int pb = jc & 1;
    const int ci = s_piv;
    const bool have = ci != 0x7fffffff;
    const bool own = jc >= r0 && jc < r1;
    for (int c = tid; c < ncols; c += NT) {
      if (have) {
        T v = P[(size_t)c * rpcp + (ci - r0)];
        if (pend && c > jc) cfms(v, P[(size_t)(jc - 1) * rpcp + (ci - r0)], urow[c]);
        a.cand_rows[((size_t)pb * a.G + b) * NB + c] = v;
      }
      if (own) {
        T v = P[(size_t)c * rpcp + (jc - r0)];
        if (pend && c > jc) cfms(v, P[(size_t)(jc - 1) * rpcp + (jc - r0)], urow[c]);
        a.rowj[(size_t)pb * NB + c] = v;
      }
    }
  };
  auto arrive = [&](int jc) {
    __syncthreads();
    if (tid == 0) {
      if (a.trace) {
        const long long t = device_ns();
        long long* tr = a.trace + (size_t)jc * kPanelTraceW;
        if (b < 160) tr[5 + b] = t;
        if (b == 0) tr[1] = t;
      }
      grid_arrive(a.status + SW_BARRIER);
    }
  };

  // column 0: candidate, post, arrive
  {
    PM bv = 0;
    int bi = 0x7fffffff;
    for (int lr = max(-r0, 0) + tid; lr < nloc; lr += NT) {
      const PM v = PK::mag(P[lr]);
      if (v > bv) { bv = v; bi = r0 + lr; }
    }
    candidate(0, bv, bi);
    post(0, false);
    arrive(0);
  }
  const int warp = tid >> 5, lane = tid & 31;
  for (int j = 0; j < ncols; ++j) {
    const int buf = j & 1;
    long long* tr = a.trace ? a.trace + (size_t)j * kPanelTraceW : nullptr;
    if (tr && b == 0 && tid == 0) tr[0] = device_ns();
    // every CTA has posted its candidate of column j
    if (!grid_wait(a.status + SW_BARRIER, a.status + SW_TIMEOUT, (unsigned)a.G * (j + 1), 1)) {
      if (b == 0) no_interchanges(a.sw, a.ipiv, a.k0, ncols, tid, NT);
      return;
    }
    if (tr && b == 0 && tid == 0) tr[2] = device_ns();
    // the winning key names the pivot row; its owner CTA is row / rpc
    if (tid == 0) {
      unsigned long long key = __ldcg(a.keys + j);
      s_piv = PK::row(key);
    }
    __syncthreads();
    const int p = s_piv;
    const int win = p / a.rpc;
    unsigned g = 0u;  // pivot growth: largest |re|+|im| in the U part of the pivot row (mag_hi key)
    for (int c = tid; c < ncols; c += NT) {
      T u = __ldcg(reinterpret_cast<const T*>(a.cand_rows) + ((size_t)buf * a.G + win) * NB + c);
      urow[c] = u;
      if (p != j && p >= r0 && p < r1)
        P[(size_t)c * rpcp + (p - r0)] = __ldcg(reinterpret_cast<const T*>(a.rowj) + (size_t)buf * NB + c);
      if (p != j && j >= r0 && j < r1) P[(size_t)c * rpcp + (j - r0)] = u;
      if (c >= j) g = max(g, mag_hi((double)cabs1(u)));
    }
    if (tid < ((ncols + 31) & ~31)) {  // whole warps that may hold entries
      for (int o = 16; o > 0; o >>= 1) g = max(g, __shfl_down_sync(0xffffffffu, g, o));
      if ((tid & 31) == 0 && g > 0u) atomicMax(&s_growth, g);
    }
    if (tid == 0) s_loc_ipiv[j] = p;
    __syncthreads();
    if (tr && b == 0 && tid == 0) tr[3] = device_ns();
    // scale column j below the diagonal (multipliers; a zero pivot leaves them unscaled, as
    // xGETF2 does, and is reported in info)
    const T piv = urow[j];
    const bool zero = (piv.x == R(0) && piv.y == R(0));
    if (zero && b == 0 && tid == 0) atomicCAS(a.status + SW_INFO, 0, a.k0 + j + 1);
    const T inv = zero ? czero<T>() : crecip(piv);
    const int lo = max(j + 1 - r0, 0);
    if (j + 1 < ncols) {
      // column j + 1 first: scale, update, candidate; post it and arrive, then finish the
      // rank-1 update of columns j + 2 .. while the other CTAs arrive
      const int jn = j + 1;
      PM bv = 0;
      int bi = 0x7fffffff;
      for (int lr = lo + tid; lr < nloc; lr += NT) {
        T l = P[(size_t)j * rpcp + lr];
        if (!zero) {
          l = cmul(l, inv);
          P[(size_t)j * rpcp + lr] = l;
        }
        T v = P[(size_t)jn * rpcp + lr];
        cfms(v, l, urow[jn]);
        P[(size_t)jn * rpcp + lr] = v;
        const PM av = PK::mag(v);
        if (av > bv) { bv = av; bi = r0 + lr; }
      }
      candidate(jn, bv, bi);
      post(jn, true);
      arrive(jn);
      // rank-1 update of columns j + 2 .. ncols - 1: lanes over rows, warps over columns,
      // four independent columns per step
      constexpr int NW = NT / 32;
      for (int lr = lo + lane; lr < nloc; lr += 32) {
        const T l = P[(size_t)j * rpcp + lr];
        int c = jn + 1 + warp;
        for (; c + 3 * NW < ncols; c += 4 * NW) {
          T v[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) v[q] = P[(size_t)(c + q * NW) * rpcp + lr];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            cfms(v[q], l, urow[c + q * NW]);
            P[(size_t)(c + q * NW) * rpcp + lr] = v[q];
          }
        }
        for (; c < ncols; c += NW) {
          T v = P[(size_t)c * rpcp + lr];
          cfms(v, l, urow[c]);
          P[(size_t)c * rpcp + lr] = v;
        }
      }
      __syncthreads();
    } else {
      for (int lr = lo + tid; lr < nloc; lr += NT) {
        if (!zero) P[(size_t)j * rpcp + lr] = cmul(P[(size_t)j * rpcp + lr], inv);
      }
      __syncthreads();
    }
    if (tr && b == 0 && tid == 0) tr[4] = device_ns();
  }

  panel_finish<T, NB, NT>(a, P, rpcp, r0, nloc, s_loc_ipiv, s_growth, b, tid);
}

// -------------------------------------------------------------------------------------
// Hardware barrier of a thread-block cluster, for panels that fit in one (panel.cuh).
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

constexpr int kMaxClusterCTAs = 16;

// -------------------------------------------------------------------------------------
// Apply the step's row interchanges to columns [c_begin, c_end) of X and solve with the
// unit lower triangle L11 = W[k0:k0+ncols, k0:k0+ncols].  Optionally emit the result as the
// B-operand planes of the mixed path (per column, NB consecutive K values).
template <typename T>
struct TrsmArgs {
  const T* W;
  long ld;
  int k0, ncols;
  const int* top_src;
  const int* extra_dst;
  const int* extra_src;
  const int* n_extra;
  T* X;
  long ldx;
  int c_begin, c_end;
  float* bop;        // optional B-operand planes
  long bop_plane;
  int bop_col0;      // column of X that maps to B-operand column 0
  unsigned* growth_bits;
  float* lup;        // optional LU planes: U12 rows k0.. (row-major, see PanelArgs)
  long lup_ld;
  long lup_plane;
  int mode;          // 0: interchanges and solve; 1: interchanges only; 2: solve only (rows k0..)
};

// Interchanges and substitution with the right-hand sides in registers: LN = NB / 16 lanes share a
// column, lane g holding rows LN a + g in x[a], a < 16.  A step broadcasts x_k within the lanes of a
// column and updates the rows below; L11 is staged in shared memory once per CTA, and a group of 2 NB
// threads walks over blocks of 32 columns (no barrier between the steps).  x moves one register down
// every LN steps and its end takes the finished row, so that the code of LN steps serves several
// blocks of them and the rows are back in place after 16; the displaced rows travel through the same
// shared memory meanwhile.
// Measured, average over the steps: FP64, N = 4000 with NB = 64, against one barrier and one L2 read
// of L's column per step: 41 -> 12 us.  Mixed, NB = 128, against the inverse of L11, a row gather, a
// tensor-core product and a split of its result as four launches:
// N = 400 40 -> 22 us, N = 3000 46 -> 23, N = 6400 48 -> 27, N = 25600 66 -> 71 (0.3 % of that
// factorisation); and no inverse enters U any more.  Bound by the chain of NB broadcasts and updates,
// in the wide case by the traffic of U12's three copies.
// One group per CTA while the blocks do not fill the SMs, else two, which hide each other's latency
// (N = 25600: 78 us with one, 71 with two, 87 with two columns per thread).
constexpr int kTrsmCols = 32;
template <int NB> constexpr int trsm_threads() { return kTrsmCols * (NB / 16); }  // of a group
template <typename T, int NB> constexpr size_t trsm_smem(int groups) {
  return ((size_t)NB * (NB + 1) + (size_t)groups * kTrsmCols * (NB + 1)) * sizeof(T);
}

template <typename T, int LN, int Q>
__device__ __forceinline__ void trsm_block(T (&x)[16], const T* L, int ldl, int g) {
  // LN steps: x[q] holds row LN q + g of the rows from this block on; L at its diagonal block.  The
  // finished rows among the Q meet rows of L past the last one, that is the zeros above the diagonal
  // of the next column.
#pragma unroll
  for (int e = 0; e < LN; ++e) {
    T xk;
    xk.x = LN > 1 ? __shfl_sync(0xffffffffu, x[0].x, e, LN) : x[0].x;
    xk.y = LN > 1 ? __shfl_sync(0xffffffffu, x[0].y, e, LN) : x[0].y;
    const T* Lc = L + (size_t)e * ldl + g;
    if (g > e) cfms(x[0], Lc[0], xk);
#pragma unroll
    for (int q = 1; q < Q; ++q) cfms(x[q], Lc[LN * q], xk);
  }
}

template <typename T, int NB>
__global__ void __launch_bounds__(2 * trsm_threads<NB>()) trsm_reg_kernel(TrsmArgs<T> a) {
  using R = typename RealOf<T>::R;
  constexpr int LN = NB / 16, NT = trsm_threads<NB>(), LDA = NB + 1, CW = kTrsmCols;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* L = reinterpret_cast<T*>(smem_raw);  // column-major, strictly lower part, and one column of zeros
  const int grp = threadIdx.x / NT, tid = threadIdx.x % NT, ngrp = (int)blockDim.x / NT;
  T* A = L + (size_t)NB * (NB + 1) + (size_t)grp * CW * LDA;  // [column][row]
  auto group_sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "r"(NT) : "memory"); };
  const int ncols = a.ncols;
  const bool swap = a.mode != 2, solve = a.mode != 1;
  const int ne = swap ? *a.n_extra : 0;
  if (solve) {
    // 16-byte copies where the columns are aligned for them; zero outside the strictly lower part of
    // ncols x ncols: trsm_block also reads there, for rows that are finished or do not exist
    constexpr int V = 16 / (int)sizeof(T);
    const T* Wl = a.W + (size_t)a.k0 + (size_t)a.k0 * a.ld;
    const bool wide = a.ld % V == 0 && (reinterpret_cast<uintptr_t>(Wl) & 15) == 0;
    for (int idx = threadIdx.x; idx < NB * (NB / V) + NB / V; idx += blockDim.x) {
      const int k = idx / (NB / V), i = idx % (NB / V) * V;
      T* d = L + (size_t)k * NB + i;
      const T* src = Wl + i + (size_t)k * a.ld;
      if (k < ncols && wide && i > k && i + V <= ncols) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(d)), "l"(src)
                     : "memory");
      } else {
#pragma unroll
        for (int v = 0; v < V; ++v) {
          if (k < ncols && i + v > k && i + v < ncols)
            cp_async_elem(d + v, src + v);
          else
            d[v] = czero<T>();
        }
      }
    }
    cp_async_wait_all();
    __syncthreads();
  }
  R gmax = R(0);
  // copies: row j of every second column; the indexes stay out of the loops
  static_assert(NT == 2 * NB, "two columns per pass");
  const int j = tid % NB, c0 = tid / NB;
  const bool has = j < ncols, ext = j < ne;
  const size_t top = (size_t)(swap && has ? a.top_src[j] : a.k0 + j);
  const size_t esrc = ext ? (size_t)a.extra_src[j] : 0, edst = ext ? (size_t)a.extra_dst[j] : 0;
  for (int cb = a.c_begin + ((int)blockIdx.x * ngrp + grp) * CW; cb < a.c_end; cb += (int)gridDim.x * ngrp * CW) {
    const int ncw = min(CW, a.c_end - cb);
    T* Xc = a.X + (size_t)cb * a.ldx;
    for (int cc = c0; cc < ncw; cc += 2) {
      if (has)
        cp_async_elem(A + cc * LDA + j, Xc + top + (size_t)cc * a.ldx);
      else
        A[cc * LDA + j] = czero<T>();
    }
    cp_async_wait_all();
    group_sync();
    const int g = tid % LN, cs = tid / LN;  // this thread's row class and column
    T* col = A + min(cs, ncw - 1) * LDA + g;
    T x[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) x[q] = col[LN * q];
    group_sync();
    if (ext)
      for (int cc = c0; cc < ncw; cc += 2) cp_async_elem(A + cc * LDA + j, Xc + esrc + (size_t)cc * a.ldx);
    if (solve) {
      for (int kb = 0; kb < 16; ++kb) {
        if (LN * kb < ncols) {
          const T* Lb = L + (size_t)LN * kb * NB + LN * kb;
          switch (kb >> 2) {
            case 0: trsm_block<T, LN, 16>(x, Lb, NB, g); break;
            case 1: trsm_block<T, LN, 12>(x, Lb, NB, g); break;
            case 2: trsm_block<T, LN, 8>(x, Lb, NB, g); break;
            default: trsm_block<T, LN, 4>(x, Lb, NB, g); break;
          }
        }
        const T done = x[0];
#pragma unroll
        for (int q = 0; q + 1 < 16; ++q) x[q] = x[q + 1];
        x[15] = done;
      }
    }
    cp_async_wait_all();
    group_sync();
    if (ext)  // every row of X this block needs has been read
      for (int cc = c0; cc < ncw; cc += 2) Xc[edst + (size_t)cc * a.ldx] = A[cc * LDA + j];
    group_sync();
    if (cs < ncw) {
#pragma unroll
      for (int q = 0; q < 16; ++q) col[LN * q] = x[q];
    }
    group_sync();
    T* Xo = Xc + a.k0 + j;
    if (has) {
#pragma unroll 4
      for (int cc = c0; cc < ncw; cc += 2) {
        const T v = A[cc * LDA + j];
        Xo[(size_t)cc * a.ldx] = v;
        gmax = fmax(gmax, cabs1(v));
      }
    }
    if (a.bop != nullptr) {  // B operand of the trailing update (zero beyond ncols)
      float* b = a.bop + (size_t)(cb - a.bop_col0) * NB + j;
#pragma unroll 4
      for (int cc = c0; cc < ncw; cc += 2) {
        const T v = A[cc * LDA + j];
        float hr, lr, hi_, li;
        tf32_split((float)v.x, hr, lr);
        tf32_split((float)v.y, hi_, li);
        b[(size_t)cc * NB] = hr;
        b[(size_t)cc * NB + a.bop_plane] = lr;
        b[(size_t)cc * NB + 2 * a.bop_plane] = hi_;
        b[(size_t)cc * NB + 3 * a.bop_plane] = li;
      }
    }
    if (a.lup != nullptr) {  // row-major: consecutive threads on consecutive columns
      if (const int cc = tid % 32; cc < ncw) {
        float* d = a.lup + (size_t)a.k0 * a.lup_ld + (size_t)(cb + cc);
#pragma unroll 4
        for (int jj = tid / 32; jj < ncols; jj += NT / 32) {
          const T v = A[cc * LDA + jj];
          float hr, lr, hi_, li;
          tf32_split((float)v.x, hr, lr);
          tf32_split((float)v.y, hi_, li);
          float* e = d + (size_t)jj * a.lup_ld;
          e[0] = hr;
          e[a.lup_plane] = lr;
          e[2 * a.lup_plane] = hi_;
          e[3 * a.lup_plane] = li;
        }
      }
    }
    group_sync();
  }
  if (a.growth_bits && solve) {
    for (int o = 16; o > 0; o >>= 1) gmax = fmax(gmax, __shfl_down_sync(0xffffffffu, gmax, o));
    if ((tid & 31) == 0 && gmax > R(0)) atomicMax(a.growth_bits, mag_hi((double)gmax));
  }
}

// dst[i + j ldd] = W[src(i) + (col0 + j) ld], i < nr, j < ncol, src(i) = rows[i] (or row0 + i
// without a row list): a block of W, optionally with its rows gathered.
template <typename T>
__global__ void gather_block_kernel(const T* __restrict__ W, long ld, const int* __restrict__ rows, int row0, int nr,
                                    int col0, int ncol, T* __restrict__ dst, long ldd) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nr) return;
  const int src = rows ? rows[i] : row0 + i;
  for (int j = blockIdx.y; j < ncol; j += gridDim.y) dst[(size_t)i + (size_t)j * ldd] = W[(size_t)src + (size_t)(col0 + j) * ld];
}

// The rows of a step's interchange list that move below the panel: dst[(extra_dst[e] - row0) +
// j ldd] = W[extra_src[e] + (col0 + j) ld], e < *n_extra, j < ncol.
template <typename T>
__global__ void patch_rows_kernel(const T* __restrict__ W, long ld, const int* __restrict__ extra_dst,
                                  const int* __restrict__ extra_src, const int* __restrict__ n_extra, int row0,
                                  int col0, int ncol, T* __restrict__ dst, long ldd) {
  const int ne = *n_extra;
  for (int idx = threadIdx.x; idx < ne * ncol; idx += blockDim.x) {
    const int e = idx % ne, j = idx / ne;
    dst[(size_t)(extra_dst[e] - row0) + (size_t)j * ldd] = W[(size_t)extra_src[e] + (size_t)(col0 + j) * ld];
  }
}

// Solve with the upper triangle U11 = W[k0:k0+ncols, k0:k0+ncols] (non-unit diagonal) for
// rows k0..k0+ncols of columns [c_begin, c_end) of X.
template <typename T, int NB, int CW, int NT>
__global__ void __launch_bounds__(NT) trsm_upper_kernel(const T* __restrict__ W, long ld, int k0,
                                                        int ncols, T* X, long ldx, int c_begin,
                                                        int c_end) {
  constexpr int NBP = NB + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* A = reinterpret_cast<T*>(smem_raw);  // [CW][NBP]
  T* rd = A + CW * NBP;                   // [NB]
  const int tid = threadIdx.x;
  const int cb = c_begin + blockIdx.x * CW;
  const int ncw = min(CW, c_end - cb);
  if (ncw <= 0) return;
  for (int j = tid; j < ncols; j += NT) {
    T d = W[(size_t)(k0 + j) + (size_t)(k0 + j) * ld];
    rd[j] = (d.x == 0 && d.y == 0) ? czero<T>() : crecip(d);
  }
  for (int idx = tid; idx < ncw * ncols; idx += NT) {
    int j = idx % ncols, cc = idx / ncols;
    A[cc * NBP + j] = X[(size_t)(k0 + j) + (size_t)(cb + cc) * ldx];
  }
  for (int j = ncols - 1; j >= 0; --j) {
    __syncthreads();
    for (int cc = tid; cc < ncw; cc += NT) A[cc * NBP + j] = cmul(A[cc * NBP + j], rd[j]);
    __syncthreads();
    if (j == 0) break;
    const T* Ucol = W + (size_t)(k0 + j) * ld + k0;
    for (int idx = tid; idx < j * ncw; idx += NT) {
      int i = idx % j, cc = idx / j;
      T v = A[cc * NBP + i];
      cfms(v, Ucol[i], A[cc * NBP + j]);
      A[cc * NBP + i] = v;
    }
  }
  __syncthreads();
  for (int idx = tid; idx < ncw * ncols; idx += NT) {
    int j = idx % ncols, cc = idx / ncols;
    X[(size_t)(k0 + j) + (size_t)(cb + cc) * ldx] = A[cc * NBP + j];
  }
}

// -------------------------------------------------------------------------------------
// C[M x N] -= A[M x K] * B[K x N], all column-major complex (SIMT, FMA units).  Used for
// the FP64 LU's trailing update, the block updates of the triangular solves and the dense
// FP64 residual.  64 x 64 output tile per 256-thread CTA, 4 x 4 outputs per thread,
// K staged through shared memory 16 at a time.
template <typename T>
__global__ void __launch_bounds__(256) cgemm_update_kernel(int M, int N, int K, const T* __restrict__ A,
                                                           long lda, const T* __restrict__ B, long ldb,
                                                           T* C, long ldc) {
  constexpr int BM = 64, BN = 64, BK = 16;
  __shared__ T As[BK][BM];
  __shared__ T Bs[BK][BN + 1];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  T acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = czero<T>();
  for (int kb = 0; kb < K; kb += BK) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      int e = tid + 256 * q;
      int r = e & 63, k = e >> 6;
      int gm = m0 + r, gk = kb + k;
      As[k][r] = (gm < M && gk < K) ? A[(size_t)gm + (size_t)gk * lda] : czero<T>();
      int kk = e & 15, cc = e >> 4;
      int gn = n0 + cc, gk2 = kb + kk;
      Bs[kk][cc] = (gn < N && gk2 < K) ? B[(size_t)gk2 + (size_t)gn * ldb] : czero<T>();
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      T av[4], bv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = As[k][tx + 16 * i];
#pragma unroll
      for (int j = 0; j < 4; ++j) bv[j] = Bs[k][ty + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) cfma(acc[i][j], av[i], bv[j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    int gm = m0 + tx + 16 * i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int gn = n0 + ty + 16 * j;
      if (gn >= N) continue;
      T* p = C + (size_t)gm + (size_t)gn * ldc;
      T v = *p;
      v.x -= acc[i][j].x;
      v.y -= acc[i][j].y;
      *p = v;
    }
  }
}

// C[M x N] -= A[M x K] * B[K x N] for few columns (N <= 8, K <= 128): the block updates of
// triangular solves with one or a few right-hand sides, where the 64 x 64 tiles of
// cgemm_update_kernel would compute mostly empty columns.  One thread per row of A (coalesced
// column reads), B staged in shared memory.
template <typename T>
__global__ void __launch_bounds__(256) cgemv_update_kernel(int M, int N, int K, const T* __restrict__ A, long lda,
                                                           const T* __restrict__ B, long ldb, T* C, long ldc) {
  constexpr int kMaxN = 8, kMaxK = 128;
  __shared__ T Bs[kMaxN][kMaxK];
  for (int e = threadIdx.x; e < K * N; e += blockDim.x) {
    const int k = e % K, n = e / K;
    Bs[n][k] = B[(size_t)k + (size_t)n * ldb];
  }
  __syncthreads();
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= M) return;
  T acc[kMaxN];
#pragma unroll
  for (int n = 0; n < kMaxN; ++n) acc[n] = czero<T>();
  for (int k = 0; k < K; ++k) {
    const T a = A[(size_t)m + (size_t)k * lda];
#pragma unroll
    for (int n = 0; n < kMaxN; ++n)
      if (n < N) cfma(acc[n], a, Bs[n][k]);
  }
#pragma unroll
  for (int n = 0; n < kMaxN; ++n) {
    if (n < N) {
      T* p = C + (size_t)m + (size_t)n * ldc;
      T v = *p;
      v.x -= acc[n].x;
      v.y -= acc[n].y;
      *p = v;
    }
  }
}

// -------------------------------------------------------------------------------------
// Inverse of one NB x NB triangle, 16 columns of it per CTA, by blocks of 16: X = T^-1 E_jb from
//   X_ib = D_ib^-1 (E_ib - sum_k T_{ib,k} X_k),  ib = jb, jb + 1, .. (lower) or jb, jb - 1, .. (upper),
// D_ib the diagonal blocks, whose inverses every CTA forms for itself, one column per thread.  The
// CTAs of a triangle are independent, so a chain of 7 block steps of one SM each replaces the
// column sweep over the whole triangle on one SM (128 columns with two block barriers each).
// Tm: the triangle (column-major, ld; order nc, identity beyond it), of which the strict lower part
// with a unit diagonal or the upper part is read.  The result (rows of all blocks, 16 columns) is left in X [NB][kTiLd], row-major, zero outside the
// triangle.  256 threads.
constexpr int kTiB = 16;
constexpr int kTiLd = kTiB + 2;  // even: 16-byte pieces stay aligned
template <typename T, int NB>
__host__ __device__ constexpr size_t tri_block_smem() {  // T blocks, diagonal inverses, X, one block of sums
  return ((size_t)(NB / kTiB) * (NB / kTiB + 1) / 2 * kTiB * kTiB + (size_t)NB * kTiB + (size_t)NB * kTiLd +
          (size_t)kTiB * kTiLd) * sizeof(T);
}
template <typename T, int NB>
__device__ T* tri_block_inverse(unsigned char* smem, bool upper, int jb, const T* __restrict__ Tm, long ld, int nc) {
  constexpr int B = kTiB, nb = NB / B;
  T* blk = reinterpret_cast<T*>(smem);              // blocks (ib, kb) of T, column-major B x B
  T* dinv = blk + (size_t)nb * (nb + 1) / 2 * B * B;  // [nb][B][B] column-major
  T* X = dinv + (size_t)NB * B;                     // [NB][kTiLd]
  T* rhs = X + (size_t)NB * kTiLd;                  // [B][kTiLd]: (k, c)
  const int tid = threadIdx.x;
  // the blocks of this chain: ib from jb to the triangle's end, kb between jb and ib
  const int nchain = upper ? jb + 1 : nb - jb;
  auto row_block = [&](int s) { return upper ? jb - s : jb + s; };
  auto slot = [&](int si, int sk) { return blk + (size_t)(si * (si + 1) / 2 + sk) * B * B; };
  // all copies in flight at once; thread (i, j) of every block
  {
    const int bi = tid % B, bj = tid / B;
    for (int si = 0; si < nchain; ++si)
      for (int sk = 0; sk <= si; ++sk) {
        const int i = row_block(si) * B + bi, j = row_block(sk) * B + bj;
        T* dst = slot(si, sk) + tid;
        if (i < nc && j < nc) {
          cp_async_elem(dst, Tm + (size_t)i + (size_t)j * ld);
        } else {
          T v = czero<T>();
          if (i == j) v.x = 1;
          *dst = v;
        }
      }
  }
  for (int t = tid; t < NB * kTiLd; t += 256) X[t] = czero<T>();
  cp_async_wait_all();
  __syncthreads();
  // inverses of the diagonal blocks: thread (s, c) solves D_s x = e_c in registers
  if (tid < nchain * B) {
    const int s = tid / B, c = tid % B;
    const T* D = slot(s, s);
    T x[B];
#pragma unroll
    for (int i = 0; i < B; ++i) {
      x[i] = czero<T>();
      if (i == c) x[i].x = 1;
    }
    if (!upper) {
#pragma unroll
      for (int k = 0; k < B; ++k)
#pragma unroll
        for (int i = k + 1; i < B; ++i) cfms(x[i], D[k * B + i], x[k]);
    } else {
#pragma unroll
      for (int k = B - 1; k >= 0; --k) {
        const T d = D[k * B + k];
        x[k] = cmul(x[k], (d.x == 0 && d.y == 0) ? czero<T>() : crecip(d));
#pragma unroll
        for (int i = 0; i < k; ++i) cfms(x[i], D[k * B + i], x[k]);
      }
    }
#pragma unroll
    for (int i = 0; i < B; ++i) dinv[(size_t)s * B * B + c * B + i] = x[i];
  }
  __syncthreads();
  // thread (i, c) forms entry (i, c) of every block of the chain
  const int i = tid % B, c = tid / B;
  X[(size_t)(row_block(0) * B + i) * kTiLd + c] = dinv[c * B + i];
  __syncthreads();
  for (int s = 1; s < nchain; ++s) {
    T acc[2] = {czero<T>(), czero<T>()};
    for (int k = 0; k < s; ++k) {
      const T* L = slot(s, k);
      const T* xk = X + (size_t)row_block(k) * B * kTiLd + c;
#pragma unroll
      for (int e = 0; e < B; ++e) cfms(acc[e & 1], L[e * B + i], xk[e * kTiLd]);
    }
    rhs[i * kTiLd + c] = cadd(acc[0], acc[1]);
    __syncthreads();
    const T* D = dinv + (size_t)s * B * B + i;
    T o[2] = {czero<T>(), czero<T>()};
#pragma unroll
    for (int e = 0; e < B; ++e) cfma(o[e & 1], D[e * B], rhs[e * kTiLd + c]);
    X[(size_t)(row_block(s) * B + i) * kTiLd + c] = cadd(o[0], o[1]);
    __syncthreads();
  }
  return X;
}

// Explicit inverses of the diagonal blocks, used by the triangular solves with many
// right-hand sides (each block solve becomes a small dense product instead of a chain of
// nb dependent steps).  Grid (steps, 2, NB / 16): blockIdx.y = 0: unit lower L11, 1: upper U11;
// blockIdx.z: 16 columns of the inverse.  Output per step: inv[(2*s + y) * NB * NB], column-major
// NB x NB, zero outside the triangle, explicit unit diagonal for L11^-1, identity beyond the order
// of the last block.  Measured (NB = 128): 4 steps 203 -> 19 us, 24 steps 218 -> 30 us; against a
// column sweep over each triangle on one SM.
template <typename T, int NB>
__global__ void __launch_bounds__(256) tri_inverse_kernel(const T* __restrict__ W, long ld, int N, T* inv) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int s = blockIdx.x, jb = blockIdx.z;
  const bool upper = blockIdx.y == 1;
  const int k0 = s * NB;
  const int nc = min(NB, N - k0);
  const T* X = tri_block_inverse<T, NB>(smem_raw, upper, jb, W + (size_t)k0 + (size_t)k0 * ld, ld, nc);
  T* out = inv + ((size_t)2 * s + (upper ? 1 : 0)) * NB * NB + (size_t)jb * kTiB * NB;
  for (int idx = threadIdx.x; idx < NB * kTiB; idx += 256) out[idx] = X[(size_t)(idx % NB) * kTiLd + idx / NB];
}

// One diagonal block of a triangular solve with many right-hand sides:
//   X[k0:k0+ncols, col] = Tinv * (P X)[k0:k0+ncols, col]
// where P is the step's row-interchange list (forward solve; pass top_src = nullptr for
// the backward solve).  Each CTA stages the NB x NB inverse in shared memory with wide
// independent loads, then handles CW right-hand sides: thread (i, cc) forms row i of
// column cc.  With rop != nullptr the result is also written as B-operand planes of the
// tensor-core update (per right-hand side NB consecutive values, zero padded; planes
// rop_plane apart).  Dynamic shared memory: NB*NB + 2*CW*NB elements of T.
template <typename T, int NB, int CW>
__global__ void __launch_bounds__(NB * CW) diag_apply_kernel(const T* __restrict__ Tinv, int ncols, int k0,
                                                             const int* top_src, const int* extra_dst,
                                                             const int* extra_src, const int* n_extra,
                                                             T* X, long ldx, int nrhs, float* rop, long rop_plane) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* ts = reinterpret_cast<T*>(smem_raw);  // [NB * NB] column-major
  T* bv = ts + NB * NB;                     // [CW][NB]
  T* ev = bv + CW * NB;                     // [CW][NB]
  constexpr int NT = NB * CW;
  const int tid = threadIdx.x;
  const int i = tid % NB, cc = tid / NB;
  const int col = blockIdx.x * CW + cc;
  const bool active = col < nrhs;
  T* x = X + (size_t)(active ? col : 0) * ldx;
  const int ne = top_src ? *n_extra : 0;
  // stage the inverse: 16-byte loads, all independent
  {
    const float4* src = reinterpret_cast<const float4*>(Tinv);
    float4* dst = reinterpret_cast<float4*>(ts);
    constexpr int n16 = NB * NB * (int)sizeof(T) / 16;
#pragma unroll 8
    for (int q = tid; q < n16; q += NT) dst[q] = __ldg(src + q);
  }
  if (active && i < ncols) bv[cc * NB + i] = x[top_src ? top_src[i] : k0 + i];
  if (active && i < ne) ev[cc * NB + i] = x[extra_src[i]];
  __syncthreads();
  if (active && i < ne) x[extra_dst[i]] = ev[cc * NB + i];
  T acc0 = czero<T>(), acc1 = czero<T>();
  if (active && i < ncols) {
    const T* b = bv + cc * NB;
    int j = 0;
#pragma unroll 4
    for (; j + 1 < ncols; j += 2) {
      cfma(acc0, ts[i + j * NB], b[j]);
      cfma(acc1, ts[i + (j + 1) * NB], b[j + 1]);
    }
    if (j < ncols) cfma(acc0, ts[i + j * NB], b[j]);
    acc0 = cadd(acc0, acc1);
    x[k0 + i] = acc0;
  }
  if (active && rop != nullptr) {
    float hr, lr, hi_, li;
    tf32_split((float)acc0.x, hr, lr);
    tf32_split((float)acc0.y, hi_, li);
    size_t off = (size_t)col * NB + i;
    rop[off] = hr;
    rop[rop_plane + off] = lr;
    rop[2 * rop_plane + off] = hi_;
    rop[3 * rop_plane + off] = li;
  }
}

}  // namespace hprmat
