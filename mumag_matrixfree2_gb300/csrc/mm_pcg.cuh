// The whole demag PCG (start, iterations with their V-cycles, stopping test) as one launch.
//
// As separate kernels an iteration is a chain of 7-13 dependent launches, and below ~1M rows their
// ramps, tails and dependent loads cost more than their bytes or FP64 operations: on GB300 the 10
// kernels of the 80 nm cube (357,911 rows) take 3.8-19 us each (128 us together, bytes worth 30 us),
// the 7 of a 1,331-row mesh 4.9 us each.  Here one block per SM stays resident, and the steps of an
// iteration are phases separated by a barrier (1.24 us for 152 blocks; 0.3 us as one cluster).
//
// Every row is summed in the order of the separate kernels and every reduction keeps their partials
// and their trees, so both forms give the same bits, for any number of blocks here.
//
// The steps of an iteration are a table that one loop runs, with one copy of each kind's code: with the
// phases inlined in turn the kernel was 147 KB, every phase of every iteration missed the instruction
// cache, and a phase of the 1,331-row mesh took 4 us.
//
// What bounds a phase now: below ~100k rows its barrier, the scalar that one thread forms (3 us, beside the first
// loads) and a chain of three dependent loads; above, loads in flight (24 warps of 80 registers) against L2 and HBM
// latency, with the FP64 pipe 41 % busy and HBM 28 % (357,911 rows), 53 and 47 % (1,601,613 rows).  Deeper prefetching was slower: operators streamed to shared memory by a
// copying warp, prefetched to L2 one unit ahead, or shares dealt out in turn instead of contiguous.
#pragma once

#include "mm_kernels.cuh"

namespace mmk {

constexpr int PT = 768;          // threads per block: one block per SM at 80 registers a thread
constexpr int PW = PT / 32;      // its warps
constexpr int PLEV = 10;         // levels a launch can hold (deeper hierarchies use the separate kernels)
constexpr int PSTEPS = 4 * PLEV + 6;
constexpr int CHUNK = BS * ILP;  // rows of a separate kernel's block
constexpr int WPB = BS / 32;     // its warps

// an operator in sliced ELL (ptr: slice pointers): a row to a lane (lg == 0), or dealt out over 1 << lg lanes
// (upload_lanes)
template <class T>
struct POp {
  int n, lg;
  const int* ptr;
  const int* col;
  const T* val;
};

// kinds of step.  Rows: PS_RESID y = b - A x; PS_RESTRICT y = A x and the coarse pre-smoothing y2 = s .* y
// (y2 may be null); PS_PROLONG y = b + A x; PS_SMOOTH y = x + s .* (b - A x).
enum PStepKind { PS_START, PS_DIR, PS_STEP, PS_SMOOTH0, PS_FOLD0, PS_RESID, PS_RESTRICT, PS_PROLONG, PS_SMOOTH, PS_COARSE_A,
                 PS_COARSE_B, PS_DENSE };

template <class T>
struct PStep {
  int kind;
  int units;  // its warps' units, or its partials, shared out evenly among the blocks
  POp<T> A;
  const T *x, *b, *s;
  T *y, *y2;
};

struct PBar {
  unsigned arrived;  // blocks arrived since the launch began
  unsigned left;     // blocks that have left the kernel; the last one clears both
};

// TP: the PCG's vectors and finest operator; TV: the V-cycle's (TP = double, TV = float: the FP64 PCG
// with the FP32 V-cycle, its product with A0 from the operator split into FP32 pairs)
template <class TP, class TV>
struct PcgArgs {
  int n;            // rows
  int G, Gdot;      // reduction blocks of the fused kernels and of the plain inner product
  int kshift;       // warps of one of the former's partials (log2)
  int cluster;      // the grid is one cluster
  int n_steps;      // PS_START, the V-cycle, PS_DIR, PS_STEP
  int nc, zr;       // coarsest rows (fused correction, dense solve); rows of Z
  POp<TP> A0;
  SellDF A0s;
  const TP* b;
  TP *x, *r, *p, *Ap;
  const TV* s0;  // level 0: smoother, pre-smoothed iterate, the V-cycle's input (r or its FP32 copy), output
  TV *xv, *rv, *z;
  const TV *M, *Z;  // W (fused correction) or the coarsest inverse; Z
  TV* zvec;
  double tol;
  int maxiter;
  Scalars* sc;
  double* part;
  PBar* bar;
  PStep<TV> steps[PSTEPS];
};

// All blocks of the grid meet; what they wrote before is visible to all after.  As one cluster the
// hardware barrier; else a counter in L2 (the launch is cooperative, so every block is resident).  The
// wait is bounded: after ~2^21 polls (about a second) the block records the failure in sc->bar_err, and
// every block that sees it leaves the kernel.  Returns false then.
__device__ __forceinline__ bool grid_meet(PBar* bar, bool cluster, unsigned& target, Scalars* sc) {
  if (cluster) {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    return true;
  }
  __shared__ int s_ok;
  __syncthreads();
  target += gridDim.x;
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&bar->arrived) : "memory");
    int ok = 1;
    for (unsigned polls = 0;; ++polls) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&bar->arrived) : "memory");
      if ((int)(v - target) >= 0) break;
      if ((polls & 255u) == 255u) {
        cuda::atomic_ref<int, cuda::thread_scope_device> err(sc->bar_err);
        if (polls > (1u << 21)) err.store(1, cuda::memory_order_relaxed);
        if (err.load(cuda::memory_order_relaxed) != 0) {
          ok = 0;
          break;
        }
      }
    }
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// the last block to leave clears the barrier for the next launch
__device__ __forceinline__ void grid_leave(PBar* bar, bool cluster) {
  if (cluster || threadIdx.x != 0) return;
  cuda::atomic_ref<unsigned, cuda::thread_scope_device> left(bar->left);
  if (left.fetch_add(1u, cuda::memory_order_acq_rel) == gridDim.x - 1) {
    bar->arrived = 0u;
    bar->left = 0u;
  }
}

// ------------------------------------------------------------------------------------------
// row products.  Vectors are read with plain loads (they change between phases); operators through
// the read-only path.  A block holds half the threads of the separate kernels' SMs, so each keeps more
// loads in flight: two rows of two entry pairs (sliced rows), four pairs of a lane (dealt-out rows).
// ------------------------------------------------------------------------------------------
constexpr int PPF = 2;

template <class T>
__device__ __forceinline__ void psell2(const POp<T>& A, const T* x, int r0, int r1, T (&acc)[2]) {
  using P2 = typename Pair<T>::type;
  const int rows[2] = {r0, r1};
  int base[2], wp[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int s = rows[q] >> 5;  // the same slice for the whole warp
    acc[q] = T(0);
    wp[q] = 0;
    base[q] = 0;
    if ((s << 5) < A.n) {
      const int b0 = __ldg(A.ptr + s);
      wp[q] = (__ldg(A.ptr + s + 1) - b0) >> 6;
      base[q] = b0 + 2 * (rows[q] & 31);
    }
  }
  const int wmax = max(wp[0], wp[1]);
#pragma unroll 1
  for (int j0 = 0; j0 < wmax; j0 += PPF) {
    int2 c[2][PPF] = {};
    P2 v[2][PPF] = {};
    T g[2][PPF][2] = {};
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int u = 0; u < PPF; ++u)
        if (j0 + u < wp[q]) {
          c[q][u] = __ldg(reinterpret_cast<const int2*>(A.col + base[q] + 64 * (j0 + u)));
          v[q][u] = __ldg(reinterpret_cast<const P2*>(A.val + base[q] + 64 * (j0 + u)));
        }
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int u = 0; u < PPF; ++u)
        if (j0 + u < wp[q]) {
          g[q][u][0] = x[c[q][u].x];
          g[q][u][1] = x[c[q][u].y];
        }
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int u = 0; u < PPF; ++u)
        if (j0 + u < wp[q]) {
          acc[q] = fmaT<T>(v[q][u].x, g[q][u][0], acc[q]);
          acc[q] = fmaT<T>(v[q][u].y, g[q][u][1], acc[q]);
        }
  }
}

__device__ __forceinline__ void psell2_df(const SellDF& A, const float* z, int r0, int r1, float (&sh)[2],
                                          float (&sl)[2]) {
  const int rows[2] = {r0, r1};
  int base[2], wp[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int s = rows[q] >> 5;
    sh[q] = 0.0f;
    sl[q] = 0.0f;
    wp[q] = 0;
    base[q] = 0;
    if ((s << 5) < A.n) {
      const int b0 = __ldg(A.sptr + s);
      wp[q] = (__ldg(A.sptr + s + 1) - b0) >> 6;
      base[q] = b0 + 2 * (rows[q] & 31);
    }
  }
  const int wmax = max(wp[0], wp[1]);
#pragma unroll 1
  for (int j0 = 0; j0 < wmax; j0 += PPF) {
    int2 c[2][PPF] = {};
    float2 vh[2][PPF] = {}, vl[2][PPF] = {};
    float g[2][PPF][2] = {};
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int u = 0; u < PPF; ++u)
        if (j0 + u < wp[q]) {
          const int e = base[q] + 64 * (j0 + u);
          c[q][u] = __ldg(reinterpret_cast<const int2*>(A.col + e));
          vh[q][u] = __ldg(reinterpret_cast<const float2*>(A.hi + e));
          vl[q][u] = __ldg(reinterpret_cast<const float2*>(A.lo + e));
        }
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int u = 0; u < PPF; ++u)
        if (j0 + u < wp[q]) {
          g[q][u][0] = z[c[q][u].x];
          g[q][u][1] = z[c[q][u].y];
        }
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int u = 0; u < PPF; ++u)
        if (j0 + u < wp[q]) {
          df_madd(vh[q][u].x, vl[q][u].x, g[q][u][0], sh[q], sl[q]);
          df_madd(vh[q][u].y, vl[q][u].y, g[q][u][1], sh[q], sl[q]);
        }
  }
}

// A slice of a row dealt out over 1 << lg lanes, eight entries of a lane in flight; the row's sum in all its lanes.
// FP64 products leave by branches on the slice's width: a predicated-off FP64 operation still holds the FP64 pipe
// for its 16 clocks, eight of them for the two or three entries of a prolongation's lane.
template <class T>
__device__ __forceinline__ T planes(const POp<T>& A, const T* x, int s) {
  using P2 = typename Pair<T>::type;
  constexpr int U = 4;
  const int lane = threadIdx.x & 31;
  int at = __ldg(A.ptr + s);
  int left = (__ldg(A.ptr + s + 1) - at) >> 6;
  at += 2 * lane;
  T acc = T(0);
#pragma unroll 1
  for (; left > 0; left -= U, at += 64 * U) {
    int2 c[U] = {};  // defined on every path: a register that only predicated loads write stays live
    P2 v[U] = {};    // through the whole kernel
    T g[U][2] = {};
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u < left) {
        c[u] = __ldg(reinterpret_cast<const int2*>(A.col + at + 64 * u));
        v[u] = __ldg(reinterpret_cast<const P2*>(A.val + at + 64 * u));
      }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u < left) {
        g[u][0] = x[c[u].x];
        g[u][1] = x[c[u].y];
      }
    do {
#define PMADD(K)                             \
  if (K >= left) break;                     \
  acc = fmaT<T>(v[K].x, g[K][0], acc);       \
  acc = fmaT<T>(v[K].y, g[K][1], acc);
      PMADD(0) PMADD(1) PMADD(2) PMADD(3)
#undef PMADD
    } while (false);
  }
#pragma unroll 1
  for (int o = 1 << A.lg >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  return acc;
}

// The separate kernels' product with dealt-out rows.  MODE 0: y = A x; 1: y = b - A x; 2: y = x + s .* (b - A x); 3: y = b + A x;
// 4: y = A x and, with s, y2 = s .* y (a restriction and the coarse pre-smoothing).  The lanes are those that suit the one
// launch, fewer than these kernels would take, and a row's sum is the same bits in both forms; from compressed rows so
// few lanes load in separate pieces.  Eight threads' FP64 solves of 262,144 rows, us a solve: 1007 from compressed rows, 825
// from dealt-out ones, 867 from compressed rows with their own lanes.
template <int MODE, class T>
__global__ void __launch_bounds__(BS) k_dealt(SellT<T> M, int tpr, const T* x, const T* b, const T* __restrict__ s, T* y,
                                              T* y2, const int* __restrict__ done) {
  pdl_entry();
  if (done && *done) return;
  const POp<T> A{M.n, 31 - __clz(tpr), M.sptr, M.col, M.val};
  const int lane = threadIdx.x & 31, per = 32 >> A.lg;
#pragma unroll 1
  for (int u = blockIdx.x * WPB + (threadIdx.x >> 5); u * per < A.n; u += gridDim.x * WPB) {
    const T ax = planes<T>(A, x, u);
    const int row = u * per + (lane >> A.lg);
    if (row >= A.n || (lane & (tpr - 1)) != 0) continue;
    if (MODE == 1) y[row] = b[row] - ax;
    else if (MODE == 2) y[row] = x[row] + s[row] * (b[row] - ax);
    else if (MODE == 3) y[row] = b[row] + ax;
    else y[row] = ax;
    if (MODE == 4 && s) y2[row] = s[row] * ax;
  }
}

// the rows of one step (PS_RESID .. PS_SMOOTH)
template <class T>
__device__ __forceinline__ void prow_out(const PStep<T>& st, int i, T ax) {
  if (st.kind == PS_RESTRICT) {
    st.y[i] = ax;
    if (st.y2) st.y2[i] = st.s[i] * ax;
  } else if (st.kind == PS_PROLONG) st.y[i] = st.b ? st.b[i] + ax : ax;
  else if (st.kind == PS_SMOOTH) st.y[i] = st.x[i] + st.s[i] * (st.b[i] - ax);
  else st.y[i] = st.b[i] - ax;
}

template <class T>
__device__ __forceinline__ void prows(const PStep<T>& st, int lo, int hi) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const POp<T> A = st.A;
  const T* x = st.x;
  if (A.lg == 0) {  // units of two slices
#pragma unroll 1
    for (int u = lo + wid; u < hi; u += PW) {
      const int r0 = 64 * u + lane, r1 = r0 + 32;
      T ax[2];
      psell2<T>(A, x, r0, r1, ax);
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if ((q ? r1 : r0) < A.n) prow_out<T>(st, q ? r1 : r0, ax[q]);
    }
  } else {  // units of a warp's rows
#pragma unroll 1
    for (int u = lo + wid; u < hi; u += PW) {
      const T ax = planes<T>(A, x, u);
      const int row = (u << (5 - A.lg)) + (lane >> A.lg);
      if (row < A.n && (lane & ((1 << A.lg) - 1)) == 0) prow_out<T>(st, row, ax);
    }
  }
}

// ------------------------------------------------------------------------------------------
// reductions in the separate kernels' order (chunk_finish): unit u is what warp u % 8 of their block
// u / 8 takes, the rows w*32 + lane and w*32 + lane + BS of the block's chunks; 1 << kshift units make a
// partial.  Here a warp takes a unit, and a block's share of the partials is folded from shared memory.
// ------------------------------------------------------------------------------------------
extern __shared__ double s_unit[];

// The iteration's scalars, formed by one thread of every block alike and kept in shared memory: an FP64
// division or comparison by every warp would hold the SM's FP64 pipe (16 clocks a warp instruction) for
// microseconds.
struct PScal {
  double bb, tol2, rr, rz, alpha, beta;
  int done;
  double red[2][BS];
};

// One meeting of the block's threads inside a phase: every warp calls it before it uses a scalar that the
// first warps are forming meanwhile, and at the latest after its units.
struct PMeet {
  bool met;
  __device__ __forceinline__ void operator()() {
    if (met) return;
    met = true;
    asm volatile("barrier.sync 2, %0;" ::"n"(PT) : "memory");
  }
};

// The grid total of a slot's G partials (after a barrier) in grid_total's order, and the scalar that follows
// from it (grid_total's POST_*), by the block's first BS threads.  The others go on: the scalar is theirs
// after a meeting or a barrier.
__device__ __noinline__ void ptotal(PScal& ps, const double* part, int slot, int G, int it, int maxiter, double tol) {
  const int tid = threadIdx.x;
  if (tid >= BS) return;
  // b.b's total is followed by another without a barrier between them: a buffer and a barrier of its own
  double* s_red = ps.red[slot == R_BB];
  const int bar = slot == R_BB ? 3 : 1;
  const double* pa = part + (size_t)slot * MAXG;
  double a = 0.0;
#pragma unroll 4
  for (int i = tid; i < G; i += BS) a += __ldcg(pa + i);
  s_red[tid] = a;
  if (tid >= 32) {
    asm volatile("barrier.arrive %0, %1;" ::"r"(bar), "n"(BS) : "memory");
    return;
  }
  asm volatile("barrier.sync %0, %1;" ::"r"(bar), "n"(BS) : "memory");
  double u[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) u[k] = s_red[tid + 32 * k];
  a = warp_sum(fold8<false>(u));
  if (tid == 0) {
    if (slot == R_BB) {
      ps.bb = a;
      ps.tol2 = tol * tol * a;
      ps.rz = ps.alpha = ps.beta = 0.0;
    } else if (slot == R_R2) {
      ps.rr = a;
      ps.done = a <= ps.tol2 || it >= maxiter;
    } else {
      const double num = slot == R_RZ ? a : ps.rz, den = slot == R_RZ ? ps.rz : a;
      const double quot = num / (den + 1e-30);
      if (slot == R_RZ) {
        ps.beta = it > 0 ? quot : 0.0;  // the first direction is z
        ps.rz = a;
      } else {
        ps.alpha = quot;
      }
    }
  }
  __syncwarp();
}

// A unit's sum: a partial of its own, or kept in shared memory for pparts_out, which folds a partial of eight units.
template <class T>
__device__ __forceinline__ void punit_out(Acc<T>& acc, double* pa, int kshift, int u) {
  const int lane = threadIdx.x & 31;
  if (kshift == 0) {
    const double t = acc.warp_total();
    if (lane == 0) pa[u] = t;
  } else if constexpr (std::is_same<T, double>::value) {
    s_unit[32 * u + lane] = acc.s;
  } else {
    const double t = acc.warp_total();
    if (lane == 0) s_unit[u] = t;
  }
}

template <class T>
__device__ __forceinline__ void pparts_out(double* pa, int kshift, int nc) {
  if (kshift == 0) return;
  const int lane = threadIdx.x & 31;
  __syncthreads();
#pragma unroll 1
  for (int c = threadIdx.x >> 5; c < nc; c += PW) {
    double t;
    if constexpr (std::is_same<T, double>::value) {
      double u[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) u[j] = s_unit[32 * (8 * c + j) + lane];
      t = warp_sum(fold8<false>(u));
    } else {
      t = 0.0;
#pragma unroll 1
      for (int j = 0; j < WPB; ++j) t += s_unit[WPB * c + j];
    }
    if (lane == 0) pa[c] = t;
  }
}

// The steps with a reduction over level 0's rows, on vectors of T.  kind PS_START: r = b - A x, r.r;
// PS_DIR: p = z + beta p, Ap = A z + beta Ap, p.Ap; PS_STEP: x += alpha p, r -= alpha Ap, r.r (both with
// the V-cycle's input and its pre-smoothing xv = s0 .* r); PS_SMOOTH0: z = x + s0 .* (r - A x), r.z.
// The warps that ptotal leaves free take the first units; every warp passes `meet` after its loads.
template <class T, class TP, class TV>
__device__ __forceinline__ void preduce(const PcgArgs<TP, TV>& a, int kind, PScal& ps, bool first, int c0, int nc) {
  constexpr bool MP = !std::is_same<TP, TV>::value;
  constexpr bool OUTER = std::is_same<T, TP>::value;  // START, DIR, STEP here
  constexpr bool INNER = std::is_same<T, TV>::value;  // SMOOTH0 here
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int n = a.n, kshift = a.kshift;
  const int slot = kind == PS_DIR ? R_PAP : kind == PS_SMOOTH0 ? R_RZ : R_R2;
  double* const pa = a.part + (size_t)slot * MAXG + c0;
  PMeet meet{kind != PS_DIR && kind != PS_STEP};
#pragma unroll 1
  for (int u = wid >= WPB ? wid - WPB : wid + PW - WPB; u < (nc << kshift); u += PW) {
    const int ug = (c0 << kshift) + u;
    Acc<T> acc;
#pragma unroll 1
    for (int rb = (ug / WPB) * CHUNK; rb < n; rb += a.G * CHUNK) {
      const int r0 = rb + 32 * (ug % WPB) + lane, r1 = r0 + BS;
      T ax[2] = {}, e0[2] = {}, e1[2] = {}, e2[2] = {}, e3[2] = {};
      float sl[2] = {};
      TV e4[2] = {};
      // the rows' vector entries, in flight with the product's loads
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int i = q ? r1 : r0;
        if (i >= n) continue;
        if (OUTER && kind == PS_START) {
          e0[q] = (T)a.b[i];
        } else if (OUTER && kind == PS_DIR) {
          e0[q] = (T)a.z[i];
          if (!first) {
            e1[q] = (T)a.p[i];
            e2[q] = (T)a.Ap[i];
          }
        } else if (OUTER && kind == PS_STEP) {
          e0[q] = (T)a.x[i];
          e1[q] = (T)a.p[i];
          e2[q] = (T)a.Ap[i];
          e3[q] = (T)a.r[i];
          if (a.xv) e4[q] = a.s0[i];
        } else if (INNER) {
          e0[q] = (T)a.xv[i];
          e1[q] = (T)a.s0[i];
          e2[q] = (T)a.rv[i];
        }
      }
      if (kind != PS_STEP) {
        if constexpr (MP && OUTER) {
          if (kind == PS_DIR) {
            float sh[2];
            psell2_df(a.A0s, a.z, r0, r1, sh, sl);
            ax[0] = (T)sh[0] + (T)sl[0];
            ax[1] = (T)sh[1] + (T)sl[1];
          } else {
            psell2<T>(a.A0, a.x, r0, r1, ax);
          }
        } else if constexpr (MP) {
          psell2<T>(a.steps[a.n_steps - 3].A, a.xv, r0, r1, ax);
        } else {
          psell2<T>(a.A0, kind == PS_DIR ? a.z : kind == PS_START ? a.x : a.xv, r0, r1, ax);
        }
      }
      meet();
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int i = q ? r1 : r0;
        if (i >= n) continue;
        if (OUTER && kind == PS_DIR) {
          const T beta = (T)ps.beta;
          const T pn = first ? e0[q] : e0[q] + beta * e1[q];
          const T apn = first ? ax[q] : ax[q] + beta * e2[q];
          a.p[i] = (TP)pn;
          a.Ap[i] = (TP)apn;
          acc.add(pn, apn);
        } else if (OUTER && (kind == PS_STEP || kind == PS_START)) {
          T ri;
          if (kind == PS_STEP) {
            const T alpha = (T)ps.alpha;
            a.x[i] = (TP)(e0[q] + alpha * e1[q]);
            ri = e3[q] - alpha * e2[q];
          } else {
            ri = e0[q] - ax[q];
          }
          a.r[i] = (TP)ri;
          acc.add(ri, ri);
          const TV rf = (TV)ri;
          if (MP) a.rv[i] = rf;
          if (a.xv) a.xv[i] = (kind == PS_STEP ? e4[q] : a.s0[i]) * rf;
        } else if (INNER) {
          const T yi = e0[q] + e1[q] * (e2[q] - ax[q]);
          a.z[i] = (TV)yi;
          acc.add(e2[q], yi);
        }
      }
    }
    punit_out(acc, pa, kshift, u);
  }
  meet();
  pparts_out<T>(pa, kshift, nc);
}

// The folded prolongation on level 0, z = A [r; e] (e behind r in memory), and r.z.  The rows may be dealt out over lanes
// (below 16Ki rows), and a block takes those of its partials, whose sums it then forms in k_rz's order from shared
// memory.  Small problems only (folded()): a partial is one warp's unit of 64 rows, with no second round of a grid's
// blocks.
template <class TP, class TV>
__device__ __forceinline__ void pfold0(const PcgArgs<TP, TV>& a, const PStep<TV>& st, int c0, int nc) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const POp<TV> A = st.A;
  const int n = A.n, lg = A.lg;
  double* const pa = a.part + (size_t)R_RZ * MAXG + c0;
  TV* const s_z = reinterpret_cast<TV*>(s_unit);
  auto row0 = [&](int u, int q) {
    const int ug = c0 + u;
    return ug / WPB * CHUNK + 32 * (ug % WPB) + q * BS;
  };
#pragma unroll 1
  for (int k = wid; k < nc << (lg + 1); k += PW) {
    const int g = k >> lg, sub = k & ((1 << lg) - 1), r0 = row0(g >> 1, g & 1) + (sub << (5 - lg));
    if (r0 >= n) continue;
    const TV ax = planes<TV>(A, st.x, r0 >> (5 - lg));
    const int j = lane >> lg;
    if (r0 + j < n && (lane & ((1 << lg) - 1)) == 0) {
      st.y[r0 + j] = ax;
      s_z[32 * g + (sub << (5 - lg)) + j] = ax;
    }
  }
  TV r[2] = {};  // the first unit's, in flight over the barrier
#pragma unroll
  for (int q = 0; q < 2; ++q)
    if (wid < nc && row0(wid, q) + lane < n) r[q] = st.x[row0(wid, q) + lane];
  __syncthreads();
#pragma unroll 1
  for (int u = wid; u < nc; u += PW) {
    Acc<TV> acc;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int i = row0(u, q) + lane;
      if (i < n) acc.add(u == wid ? r[q] : st.x[i], s_z[64 * u + 32 * q + lane]);
    }
    punit_out(acc, pa, 0, u);
  }
}

// b.b -> R_BB with k_dot's blocks (a partial of eight warps each)
template <class TP, class TV>
__device__ __forceinline__ void pdot_bb(const PcgArgs<TP, TV>& a) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int c0 = a.Gdot * (int)blockIdx.x / (int)gridDim.x, nc = a.Gdot * (int)(blockIdx.x + 1) / (int)gridDim.x - c0;
#pragma unroll 1
  for (int u = wid; u < nc * WPB; u += PW) {
    Acc<TP> acc;
#pragma unroll 1
    for (int rb = (c0 + u / WPB) * CHUNK; rb < a.n; rb += a.Gdot * CHUNK)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int i = rb + q * BS + 32 * (u % WPB) + lane;
        if (i < a.n) {
          const TP bi = a.b[i];
          acc.add(bi, bi);
        }
      }
    punit_out(acc, nullptr, 3, u);
  }
  pparts_out<TP>(a.part + (size_t)R_BB * MAXG + c0, 3, nc);
  __syncthreads();
}

// ------------------------------------------------------------------------------------------
// the coarsest levels
// ------------------------------------------------------------------------------------------
// k_coarse_a: z = Z x, a row of Z by the block's first BS threads (block_reduce's order), and y = A x, a warp
// per row, by the other warps
template <class TP, class TV>
__device__ __forceinline__ void pcoarse_a(const PcgArgs<TP, TV>& a, const PStep<TV>& st, double* s_red, int lo, int hi) {
  const TV* b = st.x;
  const int n = st.A.n, tb = threadIdx.x;
  if (tb < BS) {
#pragma unroll 1
    for (int r = blockIdx.x; r < a.zr; r += gridDim.x) {
      const TV* zr = a.Z + (size_t)r * n;
      double acc = 0.0;
#pragma unroll 1
      for (int k = tb; k < n; k += 8 * BS) {
        TV m[8] = {}, v[8] = {};
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (k + j * BS < n) {
            m[j] = __ldg(zr + k + j * BS);
            v[j] = b[k + j * BS];
          }
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (k + j * BS < n) acc = fma((double)m[j], (double)v[j], acc);
      }
      s_red[tb] = acc;
      asm volatile("barrier.sync 1, %0;" ::"n"(BS) : "memory");
      if (tb < 32) {
        double u[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) u[k] = s_red[tb + 32 * k];
        acc = warp_sum(fold8<false>(u));
        if (tb == 0) a.zvec[r] = (TV)acc;
      }
      asm volatile("barrier.sync 1, %0;" ::"n"(BS) : "memory");
    }
  } else {
    const int lane = tb & 31;
#pragma unroll 1
    for (int row = lo + (tb - BS) / 32; row < hi; row += PW - WPB) {
      const TV acc = planes<TV>(st.A, b, row);
      if (lane == 0) st.y[row] = acc;
    }
  }
}

// rows of a dense matrix M (nc columns) times v, 1 << lg lanes per row: k_coarse_b (y = b + M v, 8 lanes) and
// k_dense_mv (y = M v, a warp)
template <class TP, class TV>
__device__ __forceinline__ void pdense(const PcgArgs<TP, TV>& a, const PStep<TV>& st, int lo, int hi) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int lg = st.A.lg, nc = a.nc, q = lane & ((1 << lg) - 1);
  const TV* v = st.x;
#pragma unroll 1
  for (int u = lo + wid; u < hi; u += PW) {
    const int row = (u << (5 - lg)) + (lane >> lg);
    TV acc = TV(0);
    if (row < st.A.n) {
      const TV* mr = a.M + (size_t)row * nc;
#pragma unroll 1
      for (int k = q; k < nc; k += 8 << lg) {
        TV m[8] = {}, g[8] = {};
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (k + (j << lg) < nc) {
            m[j] = __ldg(mr + k + (j << lg));
            g[j] = v[k + (j << lg)];
          }
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (k + (j << lg) < nc) acc = fmaT<TV>(m[j], g[j], acc);
      }
    }
#pragma unroll 1
    for (int o = 1 << lg >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (row < st.A.n && q == 0) st.y[row] = st.b ? st.b[row] + acc : acc;
  }
}

// The PCG of enqueue_pcg_start and the loop body (k_dot, k_pcg_init_scalars, k_init_residual, V-cycle;
// then k_pcg_dir, k_pcg_step, V-cycle until done); every block forms the scalars alike.  The stopping test
// is formed beside the V-cycle's first phase, which goes to waste when it ends the solve.
template <class TP, class TV>
__device__ __forceinline__ void pcg_run(const PcgArgs<TP, TV>& a, PScal& ps, const int2* share) {
  const int parts = (a.G * WPB) >> a.kshift;
  unsigned target = 0;
  int it = 0;
#pragma unroll 1
  for (int i = 0;;) {
    const PStep<TV>& st = a.steps[i];
    const int kind = st.kind, lo = share[i].x, hi = share[i].y;
    if (i == 1 && it == 0) ptotal(ps, a.part, R_BB, a.Gdot, it, a.maxiter, a.tol);
    if (i == 1 || kind == PS_DIR || kind == PS_STEP)
      ptotal(ps, a.part, i == 1 ? R_R2 : kind == PS_DIR ? R_RZ : R_PAP, parts, it, a.maxiter, a.tol);
    if (kind >= PS_RESID && kind <= PS_SMOOTH) {
      prows<TV>(st, lo, hi);
    } else if (kind == PS_FOLD0) {
      pfold0(a, st, lo, hi - lo);
    } else if (kind == PS_COARSE_A) {
      pcoarse_a(a, st, ps.red[0], lo, hi);
    } else if (kind >= PS_COARSE_B) {
      pdense(a, st, lo, hi);
    } else {
      if (kind == PS_START) pdot_bb(a);
      if constexpr (std::is_same<TP, TV>::value) {
        preduce<TP>(a, kind, ps, it == 0, lo, hi - lo);
      } else {
        if (kind == PS_SMOOTH0) preduce<TV>(a, kind, ps, it == 0, lo, hi - lo);
        else preduce<TP>(a, kind, ps, it == 0, lo, hi - lo);
      }
    }
    if (!grid_meet(a.bar, a.cluster, target, a.sc)) return;
    if (i == 1 && ps.done) break;
    if (++i == a.n_steps) {
      i = 1;
      ++it;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    Scalars* const sc = a.sc;
    sc->tol2 = ps.tol2;
    sc->rz = ps.rz;
    sc->alpha = ps.alpha;
    sc->beta = ps.beta;
    sc->it = it;
    sc->done = 1;
    sc->maxiter = a.maxiter;
    sc->loops = 0;  // no trips of a loop graph
    sc->red[R_BB] = ps.bb;
    sc->red[R_R2] = ps.rr;
  }
}

template <class TP, class TV>
__global__ void __launch_bounds__(PT, 1) k_pcg_persistent(const __grid_constant__ PcgArgs<TP, TV> args) {
  __shared__ PScal ps;
  __shared__ PcgArgs<TP, TV> a;  // where the phases read their operands
  __shared__ int2 share[PSTEPS];
  for (int i = threadIdx.x; i < (int)(sizeof(a) / 4); i += PT)
    reinterpret_cast<int*>(&a)[i] = reinterpret_cast<const int*>(&args)[i];
  if (threadIdx.x < args.n_steps) {
    const int units = args.steps[threadIdx.x].units;
    share[threadIdx.x] = make_int2((int)((long long)units * blockIdx.x / gridDim.x),
                                   (int)((long long)units * (blockIdx.x + 1) / gridDim.x));
  }
  __syncthreads();
  pcg_run<TP, TV>(a, ps, share);
  grid_leave(a.bar, a.cluster);
}

}  // namespace mmk
