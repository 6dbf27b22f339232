// kernels.cuh -- sm_100a kernels of the face-addressed Krylov solvers.
//
// Storage (built on the host by solv_gpu.cu):
//   * cells live in an internal order: wavefront level of the lower-
//     triangular DAG first, then the caller's index, so every level of the
//     DIC/DILU sweeps is one contiguous range and "neighbour j is below
//     cell i in the caller's order" is exactly "j < i" internally;
//   * each cell's interior faces form one row of a sliced ELL (32 cells per
//     slice, slot-major inside a slice, so a warp reads 32 consecutive
//     words per slot); slots keep the cell's faces in ascending face order,
//     which is the order the reference's face loop adds them in;
//   * vectors with V components are cell-interleaved: x[i*V + v].
// FP64 arithmetic uses explicit _rn intrinsics (no FMA contraction), so
// matrix products, residuals and sweeps are bit-identical to the in-order
// CPU restatement; reductions use a fixed tree and are run-to-run
// deterministic.
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>
#include <type_traits>

namespace sg {

constexpr double kSmall = 1e-20;  // spray-simulation/precision.f90:8
constexpr double kLarge = 1e20;   // spray-simulation/precision.f90:9
constexpr int kWarp = 32;

// ---- precision helpers ---------------------------------------------------
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float mul(float a, float b) { return a * b; }
__device__ __forceinline__ float add(float a, float b) { return a + b; }
__device__ __forceinline__ float sub(float a, float b) { return a - b; }
// Reduction term: always formed and accumulated in FP64.
__device__ __forceinline__ double prod(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double prod(float a, float b) { return __dmul_rn((double)a, (double)b); }

// ---- per (system, component) Krylov state ---------------------------------
struct Lane {
  double s, beta, alpha, pq;           // CG: s = r.z, beta, alpha
  double rho, beta0, gam, omeg;        // BiCGSTAB (alpha shared)
  double res0_n, ratio, reduc, l1;
  double gs;                           // FCG: residual scale fed to the network
  double s_prev;                       // CG: r.z of the previous iteration
  double l1_stop;                      // FP32 inner iterations: stop for a reliable
                                       // update once |r|_1 falls below this (0: never)
  int iter, n_iter, active, status;
};
enum : int { kLaneRunning = 0, kLaneConverged = 1, kLaneMaxIter = 2, kLaneNaN = 3,
             kLaneStall = 4, kLaneRefine = 5 };

// Flexible-CG beta = -(z.q)/(p.q) for the next direction p = z + beta p,
// restarted (beta = 0) each time the lane has taken a multiple of n
// iterations on its n-cell system.  CG ends within n steps in exact
// arithmetic; past them the old direction only cancels the new one (on a
// one-cell system z + beta p is exactly zero and the iteration stops
// moving).  Systems with more cells than iterations never restart.
__device__ __forceinline__ double flex_beta(const Lane& L, double zq, int n) {
  return (L.pq > 0.0 && L.iter % n != 0) ? -zq / L.pq : 0.0;
}

// The step scalars of the FP32 inner iterations (mixed precision) divide
// without the reference's absolute guard `+ small` (precision.f90:8): after
// a reliable update the residual of a small or weakly driven system, and
// with it every inner product, can lie far below 1e-20, where the guard
// would shrink each step towards zero and the iteration would stall.  A
// zero denominator gives a zero step.  The FP64 kernels keep the
// reference's expressions unchanged.
__device__ __forceinline__ double div0(double num, double den) {
  return den != 0.0 ? num / den : 0.0;
}

template <typename T>
struct Rows {
  const int* __restrict__ slice_ptr;    // element offset of each slice
  const uint8_t* __restrict__ slice_w;  // slots in each slice
  const int* __restrict__ col;          // internal column, -1 = padding
  const T* __restrict__ val;            // A(i, col) for the matrix product
  const T* __restrict__ sval;           // sweep coefficient (ng%n below, ng%p above)
  const T* __restrict__ diag;           // pl
};

// Reduction geometry: each block works on one segment (system) and strides
// through that segment's cells; partial sums go to part[], and the last
// block of a segment to finish (ticket) combines them in block order.
struct SegMap {
  const int* __restrict__ blk_seg;
  const int* __restrict__ blk_rank;
  const int* __restrict__ seg_nblk;
  const int* __restrict__ seg_blk0;
  const int* __restrict__ seg_c0;
  const int* __restrict__ seg_c1;
  unsigned int* ticket;
  int* n_active;  // lanes still iterating (host polls this)
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Block-wide sum of NR values; result valid in thread 0.  Fixed order.
template <int NR>
__device__ __forceinline__ void block_sum(double (&v)[NR]) {
  __shared__ double sh[NR][32];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  const int nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int k = 0; k < NR; ++k) v[k] = warp_sum(v[k]);
  if (l == 0) {
#pragma unroll
    for (int k = 0; k < NR; ++k) sh[k][w] = v[k];
  }
  __syncthreads();
  if (w == 0) {
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      double t = l < nw ? sh[k][l] : 0.0;
      v[k] = warp_sum(t);
    }
  }
  __syncthreads();
}

// Commit this block's partials; returns true in the segment's last block,
// with the segment totals in tot[] (valid in every thread of that block).
template <int NR>
__device__ __forceinline__ bool seg_commit(const SegMap& sm, int b, int s,
                                           double* __restrict__ part,
                                           double (&v)[NR], double (&tot)[NR]) {
  __shared__ bool last;
  __shared__ double tsh[NR];
  block_sum<NR>(v);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NR; ++k) part[(size_t)b * NR + k] = v[k];
    __threadfence();
    unsigned t = atomicAdd(&sm.ticket[s], 1u);
    last = (t == (unsigned)sm.seg_nblk[s] - 1u);
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  const int nb = sm.seg_nblk[s], b0 = sm.seg_blk0[s];
  double acc[NR];
#pragma unroll
  for (int k = 0; k < NR; ++k) acc[k] = 0.0;
  for (int j = threadIdx.x; j < nb; j += blockDim.x) {
#pragma unroll
    for (int k = 0; k < NR; ++k) acc[k] += __ldcg(&part[(size_t)(b0 + j) * NR + k]);
  }
  block_sum<NR>(acc);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NR; ++k) tsh[k] = acc[k];
    sm.ticket[s] = 0u;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NR; ++k) tot[k] = tsh[k];
  return true;
}

__device__ __forceinline__ void lane_stop(Lane& L, int status, int* n_active) {
  if (L.active) {
    L.active = 0;
    L.status = status;
    atomicSub(n_active, 1);
  }
}

// The kernels of an iteration are launched as a chain of programmatic
// dependents (chain_launch in solv_gpu.cu): the next one is set up while this
// one drains, and waits here, before it touches anything, until the one before
// is complete.  Every kernel of a chain has to wait, also one with nothing to
// do: its completion stands for all before it.  (Letting the next one's blocks
// start early as well, griddepcontrol.launch_dependents, cost 3-9% on systems
// of 0.5-0.9M cells, where they came to stand in the way of blocks at work.)
__device__ __forceinline__ void chain_enter() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Kernels on the reduction grid (SegMap) are meant to run every block of the
// grid at once: the grid holds at most 2048 threads per SM (blocks of at
// most 256 threads), and the register budget of the one-component kernels
// is capped at 32 so that all of them are resident -- a block left for a
// second wave would run the tail of every reduction at a fraction of the
// occupancy.  Several components (V > 1) get 64 registers and run in two
// full waves.
constexpr int kMaxBlock = 256;
#define SG_BOUNDS(V) __launch_bounds__(sg::kMaxBlock, ((V) == 1 ? 8 : 4))

// Row walk helpers ---------------------------------------------------------
template <typename T>
struct RowIt {
  int base, w;
  __device__ __forceinline__ RowIt(const Rows<T>& R, int i) {
    const int sl = i >> 5;
    base = __ldg(&R.slice_ptr[sl]) + (i & 31);
    w = __ldg(&R.slice_w[sl]);
  }
};

// y = A x for V interleaved components.
// FP64: y_i = pl_i x_i + sum in face order (the reference's arithmetic).
// FP32: difference form y_i = rs_i x_i + sum_j a_ij (x_j - x_i), where the
// FP32 "diagonal" holds the row sum rs_i = pl_i + sum_j a_ij (formed in
// FP64).  For the smooth vectors late Krylov iterations produce, x_j - x_i
// is exact and small, so the product keeps its relative accuracy instead of
// losing log10(cond) digits to cancellation; same bytes moved.
// Rows are walked a chunk of slots at a time: the column indices, the
// coefficients and the gathered x of a chunk are all loaded before any of
// them is used, so a warp keeps several independent gathers in flight; the
// sums still run slot by slot in face order, so the FP64 product stays bit
// for bit the reference's.  FP32 takes 4 slots at a time (0.52 -> 0.69 of
// copy bandwidth); FP64 one: two slots spilled under the reduction
// kernels' 32-register cap and made the FP64 products slower at 256^3
// (0.30 -> 0.38 ms for y = A x, 0.289 -> 0.306 ms for the CG product).
#ifndef SG_ROW_CHUNK64
#define SG_ROW_CHUNK64 1
#endif
constexpr int kRowChunk = 4;
constexpr int kRowChunk64 = SG_ROW_CHUNK64;

template <typename T, int V, int CH = kRowChunk>
__device__ __forceinline__ void row_apply(const Rows<T>& R, int i,
                                          const T* __restrict__ x, T (&y)[V]) {
  RowIt<T> it(R, i);
  const T d = R.diag[i];
  if constexpr (sizeof(T) == 4) {
    T xi[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
      xi[v] = x[(size_t)i * V + v];
      y[v] = d * xi[v];
    }
    for (int k0 = 0; k0 < it.w; k0 += CH) {
      int j[CH];
      T a[CH], xv[CH][V];
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        j[u] = -1;
        a[u] = T(0);
        if (k0 + u < it.w) {
          const int e = it.base + (k0 + u) * kWarp;
          j[u] = __ldg(&R.col[e]);
          a[u] = R.val[e];
        }
      }
#pragma unroll
      for (int u = 0; u < CH; ++u)
#pragma unroll
        for (int v = 0; v < V; ++v) xv[u][v] = j[u] >= 0 ? x[(size_t)j[u] * V + v] : xi[v];
#pragma unroll
      for (int u = 0; u < CH; ++u)
        if (j[u] >= 0) {
#pragma unroll
          for (int v = 0; v < V; ++v) y[v] = fmaf(a[u], xv[u][v] - xi[v], y[v]);
        }
    }
  } else {
#pragma unroll
    for (int v = 0; v < V; ++v) y[v] = mul(d, x[(size_t)i * V + v]);
    constexpr int C = V == 1 ? kRowChunk64 : 1;
    for (int k0 = 0; k0 < it.w; k0 += C) {
      int j[C];
      T a[C], xv[C][V];
#pragma unroll
      for (int u = 0; u < C; ++u) {
        j[u] = -1;
        a[u] = T(0);
        if (k0 + u < it.w) {
          const int e = it.base + (k0 + u) * kWarp;
          j[u] = __ldg(&R.col[e]);
          a[u] = R.val[e];
        }
      }
#pragma unroll
      for (int u = 0; u < C; ++u)
#pragma unroll
        for (int v = 0; v < V; ++v) xv[u][v] = j[u] >= 0 ? x[(size_t)j[u] * V + v] : T(0);
#pragma unroll
      for (int u = 0; u < C; ++u)
        if (j[u] >= 0) {
#pragma unroll
          for (int v = 0; v < V; ++v) y[v] = add(y[v], mul(a[u], xv[u][v]));
        }
    }
  }
}

// FP32 row-sum "diagonal" for the difference-form product: rs_i = pl_i +
// sum_j a_ij, formed in FP64 then rounded once.
__global__ void k_rowsum_diag(int n, Rows<double> R, float* __restrict__ rs) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    RowIt<double> it(R, i);
    double s = R.diag[i];
    for (int k = 0; k < it.w; ++k) {
      const int e = it.base + k * kWarp;
      if (R.col[e] >= 0) s += R.val[e];
    }
    rs[i] = (float)s;
  }
}

// ---- layout conversion ---------------------------------------------------
// caller phi (cell-major [N][V], caller order) -> internal interleaved
template <typename T>
__global__ void k_phi_in(int n, int V, const int* __restrict__ old_of_new,
                         const double* __restrict__ src, T* __restrict__ dst) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int o = old_of_new[i];
    for (int v = 0; v < V; ++v) dst[(size_t)i * V + v] = (T)src[(size_t)o * V + v];
  }
}
template <typename T>
__global__ void k_phi_out(int n, int V, const int* __restrict__ old_of_new,
                          const T* __restrict__ src, double* __restrict__ dst) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int o = old_of_new[i];
    for (int v = 0; v < V; ++v) dst[(size_t)o * V + v] = (double)src[(size_t)i * V + v];
  }
}
// caller res0 (column-major [V][N]) <-> internal interleaved
__global__ void k_col_in(int n, int V, const int* __restrict__ old_of_new,
                         const double* __restrict__ src, double* __restrict__ dst) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int o = old_of_new[i];
    for (int v = 0; v < V; ++v) dst[(size_t)i * V + v] = src[(size_t)v * n + o];
  }
}
__global__ void k_col_out(int n, int V, const int* __restrict__ old_of_new,
                          const double* __restrict__ src, double* __restrict__ dst) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int o = old_of_new[i];
    for (int v = 0; v < V; ++v) dst[(size_t)v * n + o] = src[(size_t)i * V + v];
  }
}

// ---- matrix values ---------------------------------------------------------
// slot_src = 2*face + (1 if the row's cell is the face neighbour), -1 pad.
// val: the coefficient the face loop multiplies x(other cell) by for this
// row (ng%p for the owner's row, ng%n for the neighbour's row);
// sval: the sweep coefficient, ng%n for a lower neighbour, ng%p for an
// upper one (solv_direct.f90:19,33).
template <typename T>
__global__ void k_fill_values(int n, const int* __restrict__ slice_ptr,
                              const uint8_t* __restrict__ slice_w,
                              const int* __restrict__ slot_src, const int* __restrict__ col,
                              const double* __restrict__ p, const double* __restrict__ nn,
                              T* __restrict__ val, T* __restrict__ sval) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int sl = i >> 5, base = slice_ptr[sl] + (i & 31), w = slice_w[sl];
    for (int k = 0; k < w; ++k) {
      const int e = base + k * kWarp;
      const int s = slot_src[e];
      if (s < 0) {
        val[e] = (T)0;
        if (sval) sval[e] = (T)0;
        continue;
      }
      const int f = s >> 1;
      val[e] = (T)((s & 1) ? nn[f] : p[f]);
      if (sval) sval[e] = (T)(col[e] < i ? nn[f] : p[f]);
    }
  }
}
template <typename T>
__global__ void k_fill_diag(int n, const int* __restrict__ old_of_new,
                            const double* __restrict__ pl, T* __restrict__ diag) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    diag[i] = (T)pl[old_of_new[i]];
}
template <typename Tsrc, typename Tdst>
__global__ void k_convert(long long n, const Tsrc* __restrict__ a, Tdst* __restrict__ b) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x)
    b[e] = (Tdst)a[e];
}

// ---- residual: solv_res.f90:12-29 ----------------------------------------
// r_i = ((b_i - pl_i phi_i) - a_1 phi_j1) - ...; L1 norm per component.
template <int V>
__global__ void SG_BOUNDS(V) k_res(Rows<double> R, SegMap sm, const double* __restrict__ phi,
                      double* __restrict__ r, int not_r0, double* __restrict__ part,
                      double* __restrict__ l1_out) {
  const int b = blockIdx.x, s = sm.blk_seg[b];
  const int c0 = sm.seg_c0[s], c1 = sm.seg_c1[s];
  const int stride = sm.seg_nblk[s] * blockDim.x;
  double l1[V];
#pragma unroll
  for (int v = 0; v < V; ++v) l1[v] = 0.0;
  for (int i = c0 + sm.blk_rank[b] * blockDim.x + threadIdx.x; i < c1; i += stride) {
    double y[V];
    if (!not_r0) {
      RowIt<double> it(R, i);
      const double d = R.diag[i];
#pragma unroll
      for (int v = 0; v < V; ++v) y[v] = sub(r[(size_t)i * V + v], mul(d, phi[(size_t)i * V + v]));
      for (int k = 0; k < it.w; ++k) {
        const int e = it.base + k * kWarp;
        const int j = __ldg(&R.col[e]);
        if (j >= 0) {
          const double a = R.val[e];
#pragma unroll
          for (int v = 0; v < V; ++v) y[v] = sub(y[v], mul(a, phi[(size_t)j * V + v]));
        }
      }
#pragma unroll
      for (int v = 0; v < V; ++v) r[(size_t)i * V + v] = y[v];
    } else {
#pragma unroll
      for (int v = 0; v < V; ++v) y[v] = r[(size_t)i * V + v];
    }
#pragma unroll
    for (int v = 0; v < V; ++v) l1[v] += fabs(y[v]);
  }
  double tot[V];
  if (seg_commit<V>(sm, b, s, part, l1, tot) && threadIdx.x == 0) {
#pragma unroll
    for (int v = 0; v < V; ++v) l1_out[s * V + v] = tot[v];
  }
}

__global__ void k_set_res0n(Lane* lanes, int nl, const double* __restrict__ l1) {
  for (int l = threadIdx.x; l < nl; l += blockDim.x) lanes[l].res0_n = l1[l];
}

// ---- mixed precision: FP32 inner solve inside FP64 refinement --------------
// inner right-hand side r_f = (float) r, shadow r0_f = r_f, correction d = 0
template <int V>
__global__ void k_mp_start(long long nv, const double* __restrict__ r, float* __restrict__ rf,
                           float* __restrict__ r0f, float* __restrict__ d) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nv;
       e += (long long)gridDim.x * blockDim.x) {
    const float t = (float)r[e];
    rf[e] = t;
    r0f[e] = t;
    d[e] = 0.0f;
  }
}
__global__ void k_add(long long n, double* __restrict__ x, const double* __restrict__ y) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x)
    x[e] += y[e];
}
// phi += (double) d for the (system, component) lanes flagged in mask
// (FP64 solution accumulation)
template <int V>
__global__ void SG_BOUNDS(V) k_mp_accum(SegMap sm, const int* __restrict__ mask, double* __restrict__ phi,
                           const float* __restrict__ d) {
  const int b = blockIdx.x, s = sm.blk_seg[b];
  bool on[V];
  bool any = false;
#pragma unroll
  for (int v = 0; v < V; ++v) { on[v] = mask[s * V + v] != 0; any |= on[v]; }
  if (!any) return;
  const int c0 = sm.seg_c0[s], c1 = sm.seg_c1[s];
  const int stride = sm.seg_nblk[s] * blockDim.x;
  for (int i = c0 + sm.blk_rank[b] * blockDim.x + threadIdx.x; i < c1; i += stride) {
#pragma unroll
    for (int v = 0; v < V; ++v)
      if (on[v]) phi[(size_t)i * V + v] += (double)d[(size_t)i * V + v];
  }
}

// ---- sync-free triangular recurrences ---------------------------------------
// solv_precond (the DIC/DILU factorisation) and solv_direct (the two
// triangular sweeps) are recurrences over the cells: in the internal order
// every lower neighbour of a cell has a lower index (and every upper one a
// higher index), so a cell can be computed as soon as the values of its
// lower (forward) or upper (backward) neighbours exist.  One cooperative
// launch does a whole recurrence: warp w of W owns the 32-cell slices
// w, w + W, w + 2W, ... (backward: counted from the top) and takes them in
// that order; the output array starts out filled with a signalling-NaN
// pattern ("pending"), which arithmetic never produces (it returns quiet
// NaNs), and a cell reads a neighbour's value with a relaxed load until it
// is no longer pending.  All warps are resident at once (cooperative
// launch), so the lowest unfinished slice always has its owner running and
// its inputs done: the recurrence cannot deadlock.  Each cell still adds its
// neighbour terms one by one in slot (face) order, with the reference's
// operations, so the results are bit for bit those of the sequential loops.
// Every wait is bounded (kSweepPolls polls): a wait that runs out sets
// SweepCtl::err, every warp then stops waiting, and the host reports the
// error and refills the pending state before the next sweep.
struct SweepCtl {
  int err;      // a wait ran out (sticky until the host clears it)
  int pad[3];
};
constexpr int kSweepPolls = 1 << 20;
constexpr int kSweepThreads = 256;

template <typename T> struct Pending;
template <> struct Pending<double> {
  using U = unsigned long long;
  static constexpr U bits = 0x7ff5a5a5a5a5a5a5ull;  // signalling NaN
  static __device__ __forceinline__ double value() { return __longlong_as_double((long long)bits); }
  static __device__ __forceinline__ double from(U u) { return __longlong_as_double((long long)u); }
};
template <> struct Pending<float> {
  using U = unsigned int;
  static constexpr U bits = 0x7fa5a5a5u;  // signalling NaN
  static __device__ __forceinline__ float value() { return __int_as_float((int)bits); }
  static __device__ __forceinline__ float from(U u) { return __int_as_float((int)u); }
};

__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned int ld_relaxed(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed(double* p, double v) {
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(__double_as_longlong(v))
               : "memory");
}
__device__ __forceinline__ void st_relaxed(float* p, float v) {
  asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(__float_as_int(v)) : "memory");
}
__device__ __forceinline__ int ld_err(const SweepCtl* ctl) {
  return (int)ld_relaxed(reinterpret_cast<const unsigned int*>(&ctl->err));
}

// *p into bits where on
__device__ __forceinline__ void ld_relaxed_if(bool on, const unsigned long long* p,
                                              unsigned long long& bits) {
  asm volatile(
      "{ .reg .pred q; setp.ne.u32 q, %2, 0; @q ld.relaxed.gpu.global.b64 %0, [%1]; }"
      : "+l"(bits) : "l"(p), "r"((unsigned)on) : "memory");
}
__device__ __forceinline__ void ld_relaxed_if(bool on, const unsigned int* p, unsigned int& bits) {
  asm volatile(
      "{ .reg .pred q; setp.ne.u32 q, %2, 0; @q ld.relaxed.gpu.global.b32 %0, [%1]; }"
      : "+r"(bits) : "l"(p), "r"((unsigned)on) : "memory");
}

// Where a recurrence's values are: global memory (relaxed, at the GPU's
// scope) or this block's shared memory (one system a block, cells from base).
template <typename T>
struct GlobalVals {
  using U = typename Pending<T>::U;
  const U* p;
  __device__ __forceinline__ void get(bool on, int j, int V, int v, U& bits) const {
    ld_relaxed_if(on, &p[(size_t)j * V + v], bits);
  }
  __device__ __forceinline__ U peek(int j, int V) const { return ld_relaxed(&p[(size_t)j * V]); }
};
struct SharedVals {
  using U = unsigned long long;
  unsigned at;  // shared-memory address of cell base's first value
  int base;
  __device__ __forceinline__ void get(bool on, int j, int V, int v, U& bits) const {
    asm volatile(
        "{ .reg .pred q; setp.ne.u32 q, %2, 0; @q ld.relaxed.cta.shared.b64 %0, [%1]; }"
        : "+l"(bits) : "r"(at + (unsigned)((j - base) * V + v) * 8u), "r"((unsigned)on) : "memory");
  }
  __device__ __forceinline__ U peek(int j, int V) const {
    U bits = 0;
    get(true, j, V, 0, bits);
    return bits;
  }
  __device__ __forceinline__ void put(int j, int V, int v, double x) const {
    asm volatile("st.relaxed.cta.shared.b64 [%0], %1;" ::"r"(at + (unsigned)((j - base) * V + v) * 8u),
                 "l"(__double_as_longlong(x)) : "memory");
  }
};

// x[0 .. n) = pending
template <typename T>
__global__ void k_fill_pending(long long n, T* __restrict__ x) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x)
    x[e] = Pending<T>::value();
}

// Warp-level driver of one recurrence: each lane takes one cell of the
// warp's slice.  A cell's slots are taken C at a time (one chunk for rows of
// up to C slots), their indices and coefficients (`coef(e)`, read-only data)
// in registers, so that a poll is one batch of loads of the neighbour values
// and nothing else.  In an order of many levels (GATE) the dependencies are
// first packed to the front, while the warp waits anyway, so that the sum
// runs over them alone (0.93 -> 0.74 us a level); in an order of a few
// levels, where bandwidth counts, the packing would only delay the
// coefficients.
// Once the values are all there, the products (`term`, side by side) are
// folded in in slot order (`fold`), the sequential loop's arithmetic;
// `finish` stores the cell.  A lane stores
// as soon as its own inputs are there, because a slice that spans two levels
// holds cells that wait for cells of the same slice.
//
// What bounds a level-by-level order is the step from one level's store to
// the next level's load, through L2 (0.24-0.45 us one way between two SMs,
// within a die and across).  Two things had made that step 1.65 us: a
// second, serial round trip for slots past the fourth, and the polls of all
// the resident warps -- dozens of levels ahead of the front, each re-reading
// every neighbour value -- which kept L2 busy.  So, where the order has
// levels to wait for (GATE), a warp first waits on ONE value, with one
// sector per poll: the last dependency of the last cell its slice depends
// on, an ancestor two steps back (one step back was 4% slower).  Only the
// slices next to the front then poll their own inputs.
// A batch's systems are recurrences of their own, one after the other in the
// internal order; in index order the front would pass through them one by
// one, so with GATE the blocks are dealt out to the systems (SweepMap), and
// a slice that holds the end of one system and the start of the next is
// visited for each.
constexpr int kSweepSpin = 64;
constexpr int kSweepSleep = 64;  // ns
constexpr int kGateSleep = 32;   // ns

struct SweepMap {
  const int* __restrict__ c0;  // the systems' cell ranges
  const int* __restrict__ c1;
  int n_sys;
};

template <bool UP>
__device__ __forceinline__ bool sweep_dep(int j, int i) {
  return j >= 0 && (UP ? j > i : j < i);
}

// One slice of a recurrence over the cells c0 .. c1 (n: those of the matrix).
template <bool UP, bool GATE, int C, int V, typename A, typename T, typename Vals, typename Start,
          typename Coef, typename Term, typename Fold, typename Finish>
__device__ __forceinline__ void sweep_slice(int n, const Rows<T>& R, int s, int c0, int c1,
                                            const Vals& vals, SweepCtl* ctl, Start&& start,
                                            Coef&& coef, Term&& term, Fold&& fold,
                                            Finish&& finish) {
  using P = Pending<T>;
  using U = typename P::U;
  constexpr unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int i = s * 32 + lane;
  const int w = __ldg(&R.slice_w[s]);
  const int base = __ldg(&R.slice_ptr[s]) + lane;
  int dj[C];  // the chunk's dependencies in slot order: the first nd (GATE), or
  A a[C];     // those of the slots in mask
  U bits[C][V];
  int nd = 0, k0 = 0;
  unsigned mask = 0;
  bool done = i < c0 || i >= c1;
  auto on = [&](int q) { return GATE ? q < nd : ((mask >> q) & 1u) != 0; };
  auto load = [&]() {
    int j[C], du[C];
#pragma unroll
    for (int u = 0; u < C; ++u) {
      j[u] = -1;
      if (k0 + u < w) j[u] = __ldg(&R.col[base + (k0 + u) * kWarp]);
    }
    if constexpr (GATE) {
      nd = 0;
#pragma unroll
      for (int u = 0; u < C; ++u) {
        dj[u] = du[u] = 0;
        const bool dep = sweep_dep<UP>(j[u], i);
#pragma unroll
        for (int q = 0; q <= u; ++q)
          if (dep && nd == q) {
            dj[q] = j[u];
            du[q] = u;
          }
        nd += dep;
      }
    } else {
      mask = 0;
#pragma unroll
      for (int u = 0; u < C; ++u) {
        dj[u] = j[u];
        du[u] = u;
        if (sweep_dep<UP>(j[u], i)) mask |= 1u << u;
      }
    }
#pragma unroll
    for (int q = 0; q < C; ++q) {
      if (on(q)) a[q] = coef(base + (k0 + du[q]) * kWarp);
#pragma unroll
      for (int v = 0; v < V; ++v) bits[q][v] = 0;
    }
  };
  if (!done) {
    start(i);
    load();
  }
  if constexpr (GATE) {
    // the last cell of an earlier slice that this chunk depends on, then
    // the last dependency of that cell (indices offset so that 0 is none;
    // backward, counted from the top)
    unsigned last = 0;
#pragma unroll
    for (int q = 0; q < C; ++q)
      if (q < nd && (UP ? (dj[q] >> 5) > s : (dj[q] >> 5) < s))
        last = max(last, (unsigned)(UP ? n - dj[q] : dj[q] + 1));
    last = __reduce_max_sync(full, last);
    if (last) {
      const int jl = UP ? n - (int)last : (int)last - 1;
      const int wl = __ldg(&R.slice_w[jl >> 5]);
      const int bl = __ldg(&R.slice_ptr[jl >> 5]) + (jl & 31);
      const int c = lane < wl ? __ldg(&R.col[bl + lane * kWarp]) : -1;
      unsigned far = sweep_dep<UP>(c, jl) ? (unsigned)(UP ? n - c : c + 1) : 0u;
      far = __reduce_max_sync(full, far);
      if (far) {
        const int g = UP ? n - (int)far : (int)far - 1;
        for (int poll = 0; vals.peek(g, V) == P::bits; ++poll) {
          if (poll >= kSweepPolls || ((poll & 63) == 63 && ld_err(ctl))) {
            if (lane == 0) atomicExch(&ctl->err, 1);
            break;
          }
          __nanosleep(kGateSleep);
        }
        __syncwarp();
      }
    }
  }
  for (int poll = 0;; ++poll) {
    if (!done) {
#pragma unroll
      for (int q = 0; q < C; ++q) {
#pragma unroll
        for (int v = 0; v < V; ++v) vals.get(on(q), dj[q], V, v, bits[q][v]);
      }
      bool ready = true;
#pragma unroll
      for (int q = 0; q < C; ++q) {
#pragma unroll
        for (int v = 0; v < V; ++v) ready &= bits[q][v] != P::bits;
      }
      if (ready) {
        T m[C][V];
#pragma unroll
        for (int q = 0; q < C; ++q) {
          T xv[V];
#pragma unroll
          for (int v = 0; v < V; ++v) xv[v] = P::from(bits[q][v]);
          term(a[q], xv, m[q]);
        }
#pragma unroll
        for (int q = 0; q < C; ++q) {
          if (GATE && q >= nd) break;
          if (on(q)) fold(m[q]);
        }
        k0 += C;
        if (k0 < w) {
          load();
        } else {
          finish(i);
          done = true;
        }
      }
    }
    if (__all_sync(full, done)) break;
    if (poll >= kSweepPolls || ((poll & 63) == 63 && ld_err(ctl))) {
      if (lane == 0) atomicExch(&ctl->err, 1);
      break;
    }
    if (poll >= kSweepSpin) __nanosleep(kSweepSleep);
  }
}

// The slices of all the systems, a block's warps taking turns.
template <bool UP, bool GATE, int C, int V, typename A, typename T, typename Start, typename Coef,
          typename Term, typename Fold, typename Finish>
__device__ __forceinline__ void sweep_rows(int n, const Rows<T>& R, const SweepMap& sm,
                                           const T* values, SweepCtl* ctl, Start&& start,
                                           Coef&& coef, Term&& term, Fold&& fold,
                                           Finish&& finish) {
  const GlobalVals<T> vals{reinterpret_cast<const typename Pending<T>::U*>(values)};
  // this block's systems (sys, sys + step, ...), its rank among theirs
  int sys = 0, step = 1, rank = blockIdx.x, nblk = gridDim.x;
  const bool by_sys = GATE && sm.n_sys > 1;
  if (by_sys && sm.n_sys >= (int)gridDim.x) {
    sys = blockIdx.x;
    step = gridDim.x;
    rank = 0;
    nblk = 1;
  } else if (by_sys) {
    step = sm.n_sys;
    const int per = gridDim.x / sm.n_sys, more = gridDim.x % sm.n_sys;
    const int cut = more * (per + 1), b = blockIdx.x;
    nblk = b < cut ? per + 1 : per;
    sys = b < cut ? b / nblk : more + (b - cut) / nblk;
    rank = (b < cut ? b : b - cut) % nblk;
  }
  const int warps = blockDim.x >> 5;
  int c0 = 0, c1 = n;
  int r = rank * warps + (threadIdx.x >> 5);
  const int r0 = r, W = nblk * warps;
  if (by_sys) {
    c0 = sm.c0[sys];
    c1 = sm.c1[sys];
  }
  for (;; r += W) {
    const int s_lo = c0 >> 5, ns = ((c1 + 31) >> 5) - s_lo;
    if (r >= ns) {  // this system is done: the block's next
      sys += step;
      if (!by_sys || sys >= sm.n_sys) break;
      c0 = sm.c0[sys];
      c1 = sm.c1[sys];
      r = r0 - W;
      continue;
    }
    const int s = s_lo + (UP ? ns - 1 - r : r);
    sweep_slice<UP, GATE, C, V, A>(n, R, s, c0, c1, vals, ctl, start, coef, term, fold, finish);
  }
}

// solv_precond.f90:10-29: d_i = pl_i - sum_{j<i} n^2 c_j (DIC, imat 1) or
// - (p c_j) n (DILU, imat 2) in face order; c_r = d; c = 1/(d + small).
// imat <= 0 is Jacobi (no recurrence; k_precond_jacobi), imat >= 3 keeps
// d = pl (the reference's fall-through).  c must start out pending.  A lower
// neighbour's ng%n is the slot's sweep coefficient; DILU also takes ng%p,
// from its face.
template <int IMAT, bool GATE>
__global__ void __launch_bounds__(kSweepThreads, 1) k_precond_sf(
    int n, Rows<double> R, SweepMap sm, const int* __restrict__ slot_src,
    const double* __restrict__ fp, double* c, double* __restrict__ c_r, SweepCtl* ctl) {
  double d = 0.0;
  sweep_rows<false, GATE, 8, 1, double2>(
      n, R, sm, c, ctl, [&](int i) { d = R.diag[i]; },
      [&](int e) {
        return make_double2(IMAT == 2 ? __ldg(&fp[__ldg(&slot_src[e]) >> 1]) : 0.0,
                            __ldg(&R.sval[e]));
      },
      [&](const double2& a, const double (&cj)[1], double (&m)[1]) {
        m[0] = IMAT == 1 ? mul(mul(a.y, a.y), cj[0]) : mul(mul(a.x, cj[0]), a.y);
      },
      [&](const double (&m)[1]) { d = sub(d, m[0]); },
      [&](int i) {
        c_r[i] = d;
        st_relaxed(&c[i], 1.0 / add(d, kSmall));
      });
}

// Jacobi diagonal (solv_precond.f90:13 with imat <= 0): c_r = pl, c = 1/(pl+small)
__global__ void k_precond_jacobi(int n, const double* __restrict__ diag, double* __restrict__ c,
                                 double* __restrict__ c_r) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double d = diag[i];
    c_r[i] = d;
    c[i] = 1.0 / add(d, kSmall);
  }
}

// Slots per chunk and blocks per SM (what the registers are held to) of the
// sweeps.  In an order of many levels (GATE) a step's latency counts, not the
// blocks; in one of a few levels bandwidth does, so as many warps as hold a
// chunk of 6 slots, a hex row, without a spill: FP64 rows of two components
// take 72 registers for it, of four 112.  With 8 slots in 64 and 6 in 80
// registers they spilled 16-34 words a thread: BiCGSTAB + DILU in multicolour
// order, ms at 72x73x71 and 100x101x99, two components 1.95 and 4.18, now 1.69
// and 3.55 (8 slots at 3 blocks 1.71 and 3.65, 4 at 4 blocks 1.77 and 3.71);
// four components 3.61 and 7.65, now 3.26 and 7.02 (4 slots at 3 blocks 3.44
// and 7.05).
template <typename T, int V, bool GATE> struct SweepShape {
  static constexpr bool wide = sizeof(T) == 8 && !GATE;
  static constexpr int chunk = V == 1 || (V == 2 && !wide) ? 8 : 6;
  static constexpr int blocks = GATE ? 1 : V == 1 || (V == 2 && !wide) ? 4 : V == 4 && wide ? 2 : 3;
};

// solv_direct.f90:12-24 forward sweep, x_i = (b_i - sum_{j<i} n x_j) c_i, into
// t (which starts out pending); the backward sweep's output x is reset to
// pending on the way.
template <typename T, int V, bool GATE>
__global__ void __launch_bounds__(kSweepThreads, (SweepShape<T, V, GATE>::blocks)) k_fwd_sf(
    int n, Rows<T> R, SweepMap sm, const T* __restrict__ c, const T* __restrict__ bvec, T* t, T* x,
    SweepCtl* ctl, const int* __restrict__ n_active) {
  if (n_active && *n_active == 0) return;
  T acc[V], ci = T(0);
  sweep_rows<false, GATE, SweepShape<T, V, GATE>::chunk, V, T>(
      n, R, sm, t, ctl,
      [&](int i) {
        ci = __ldg(&c[i]);
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] = bvec[(size_t)i * V + v];
      },
      [&](int e) { return __ldg(&R.sval[e]); },
      [&](const T a, const T (&xv)[V], T (&m)[V]) {
#pragma unroll
        for (int v = 0; v < V; ++v) m[v] = mul(a, xv[v]);
      },
      [&](const T (&m)[V]) {
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] = sub(acc[v], m[v]);
      },
      [&](int i) {
#pragma unroll
        for (int v = 0; v < V; ++v) {
          st_relaxed(&t[(size_t)i * V + v], mul(acc[v], ci));
          x[(size_t)i * V + v] = Pending<T>::value();
        }
      });
}

// solv_direct.f90:26-38 backward sweep with the x = x c_r scaling of :26:
// x_i = (t_i c_r_i - sum_{j>i} p x_j) c_i; x starts out pending, and each
// t_i is reset to pending once read, ready for the next forward sweep.
template <typename T, int V, bool GATE>
__global__ void __launch_bounds__(kSweepThreads, (SweepShape<T, V, GATE>::blocks)) k_bwd_sf(
    int n, Rows<T> R, SweepMap sm, const T* __restrict__ c, const T* __restrict__ c_r, T* t, T* x,
    SweepCtl* ctl, const int* __restrict__ n_active) {
  if (n_active && *n_active == 0) return;
  T acc[V], ci = T(0);
  sweep_rows<true, GATE, SweepShape<T, V, GATE>::chunk, V, T>(
      n, R, sm, x, ctl,
      [&](int i) {
        ci = __ldg(&c[i]);
        const T cr = c_r[i];
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] = mul(t[(size_t)i * V + v], cr);
      },
      [&](int e) { return __ldg(&R.sval[e]); },
      [&](const T a, const T (&xv)[V], T (&m)[V]) {
#pragma unroll
        for (int v = 0; v < V; ++v) m[v] = mul(a, xv[v]);
      },
      [&](const T (&m)[V]) {
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] = sub(acc[v], m[v]);
      },
      [&](int i) {
#pragma unroll
        for (int v = 0; v < V; ++v) {
          st_relaxed(&x[(size_t)i * V + v], mul(acc[v], ci));
          t[(size_t)i * V + v] = Pending<T>::value();
        }
      });
}

// Jacobi: x = b*c (solv_direct.f90:41)
template <typename T, int V>
__global__ void k_jacobi(int n, const T* __restrict__ c, const T* __restrict__ bvec,
                         T* __restrict__ x) {
  chain_enter();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const T ci = c[i];
#pragma unroll
    for (int v = 0; v < V; ++v) x[(size_t)i * V + v] = mul(bvec[(size_t)i * V + v], ci);
  }
}

// ---- plain matrix product (benchmarks / solv_gpu_spmv) ---------------------
template <typename T, int V>
__global__ void k_spmv(int n, Rows<T> R, const T* __restrict__ x, T* __restrict__ y) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    T t[V];
    row_apply<T, V>(R, i, x, t);
#pragma unroll
    for (int v = 0; v < V; ++v) y[(size_t)i * V + v] = t[v];
  }
}

// ======================= CG: solv_cg.f90:26-84 =============================
// Lane init for CG: s = large, iter = 0, active = 1.
__global__ void k_lane_init(Lane* lanes, int nl, int n_iter, double reduc, int* n_active) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= nl) return;
  Lane L;
  L.s = kLarge; L.beta = 0.0; L.alpha = 1.0; L.pq = 0.0;   // solv_cg.f90:29
  L.rho = 0.0; L.beta0 = 1.0; L.gam = 1.0; L.omeg = 0.0;   // solv_bicg.f90:31-33
  L.res0_n = lanes[l].res0_n;
  L.ratio = 0.0; L.reduc = reduc; L.l1 = 0.0;
  L.iter = 0; L.n_iter = n_iter; L.active = 1; L.status = kLaneRunning; L.l1_stop = 0.0;
  if (n_iter <= 0) { L.active = 0; L.status = kLaneMaxIter; }  // n_active set by the host
  lanes[l] = L;
}

// s = r.z with z = M^-1 r (Jacobi: z = c r, computed here); then
// beta = (1/s_old) s, s_old = s  (solv_cg.f90:44-50).
// FLEX (the FP32 inner iteration, not the reference's): beta = -(z.q)/(p.q)
// with q = A p of the previous step, the flexible-CG formula that
// A-orthogonalises the new direction against the last one explicitly.
template <typename T, int V, bool JAC, bool FLEX = false>
__global__ void SG_BOUNDS(V) k_cg_rz(SegMap sm, const T* __restrict__ c, const T* __restrict__ r,
                        const T* __restrict__ z, double* __restrict__ part,
                        Lane* __restrict__ lanes, const T* __restrict__ q = nullptr) {
  chain_enter();
  const int b = blockIdx.x, s = sm.blk_seg[b];
  bool any = false;
#pragma unroll
  for (int v = 0; v < V; ++v) any |= lanes[s * V + v].active != 0;
  if (!any) return;
  const int c0 = sm.seg_c0[s], c1 = sm.seg_c1[s];
  const int stride = sm.seg_nblk[s] * blockDim.x;
  double acc[V];
#pragma unroll
  for (int v = 0; v < V; ++v) acc[v] = 0.0;
  for (int i = c0 + sm.blk_rank[b] * blockDim.x + threadIdx.x; i < c1; i += stride) {
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const T ri = r[(size_t)i * V + v];
      const T zi = JAC ? mul(ri, c[i]) : z[(size_t)i * V + v];
      acc[v] += FLEX ? prod(zi, q[(size_t)i * V + v]) : prod(ri, zi);
    }
  }
  double tot[V];
  if (seg_commit<V>(sm, b, s, part, acc, tot) && threadIdx.x == 0) {
#pragma unroll
    for (int v = 0; v < V; ++v) {
      Lane& L = lanes[s * V + v];
      if (!L.active) continue;
      if (FLEX) {
        L.beta = flex_beta(L, tot[v], c1 - c0);
        continue;
      }
      double beta = 1.0 / L.s;   // :44
      L.s_prev = L.s;
      L.s = tot[v];              // :47
      L.beta = beta * L.s;       // :50
    }
  }
}

// p = z + beta p  (solv_cg.f90:53).  FLEX: also s = p.r, so that the step
// alpha = (p.r)/(p.q) of k_cg_spmv makes the new residual orthogonal to p
// in the arithmetic actually done (flexible CG).
template <typename T, int V, bool JAC, bool FLEX = false>
__global__ void SG_BOUNDS(V) k_cg_p(SegMap sm, const T* __restrict__ c, const T* __restrict__ r,
                       const T* __restrict__ z, T* __restrict__ p,
                       Lane* __restrict__ lanes, double* __restrict__ part = nullptr) {
  chain_enter();
  const int b = blockIdx.x, s = sm.blk_seg[b];
  bool act[V];
  T beta[V];
  bool any = false;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    act[v] = lanes[s * V + v].active != 0;
    beta[v] = (T)lanes[s * V + v].beta;
    any |= act[v];
  }
  if (!any) return;
  const int c0 = sm.seg_c0[s], c1 = sm.seg_c1[s];
  const int stride = sm.seg_nblk[s] * blockDim.x;
  double acc[V];
#pragma unroll
  for (int v = 0; v < V; ++v) acc[v] = 0.0;
  for (int i = c0 + sm.blk_rank[b] * blockDim.x + threadIdx.x; i < c1; i += stride) {
#pragma unroll
    for (int v = 0; v < V; ++v) {
      if (!act[v]) continue;
      const size_t k = (size_t)i * V + v;
      const T ri = (JAC || FLEX) ? r[k] : T(0);
      const T zi = JAC ? mul(ri, c[i]) : z[k];
      const T pn = add(zi, mul(beta[v], p[k]));
      p[k] = pn;
      if (FLEX) acc[v] += prod(pn, ri);
    }
  }
  if constexpr (FLEX) {
    double tot[V];
    if (seg_commit<V>(sm, b, s, part, acc, tot) && threadIdx.x == 0) {
#pragma unroll
      for (int v = 0; v < V; ++v)
        if (act[v]) lanes[s * V + v].s = tot[v];
    }
  }
}

// q = A p and p.q; alpha = s / (p.q + small)   (solv_cg.f90:56-68; the FP32
// instantiation divides without the guard, div0)
template <typename T, int V, int CH = kRowChunk>
__global__ void SG_BOUNDS(V) k_cg_spmv(Rows<T> R, SegMap sm, const T* __restrict__ p, T* __restrict__ q,
                          double* __restrict__ part, Lane* __restrict__ lanes) {
  chain_enter();
  const int b = blockIdx.x, s = sm.blk_seg[b];
  bool any = false;
#pragma unroll
  for (int v = 0; v < V; ++v) any |= lanes[s * V + v].active != 0;
  if (!any) return;
  const int c0 = sm.seg_c0[s], c1 = sm.seg_c1[s];
  const int stride = sm.seg_nblk[s] * blockDim.x;
  double acc[V];
#pragma unroll
  for (int v = 0; v < V; ++v) acc[v] = 0.0;
  for (int i = c0 + sm.blk_rank[b] * blockDim.x + threadIdx.x; i < c1; i += stride) {
    T y[V];
    row_apply<T, V, CH>(R, i, p, y);
#pragma unroll
    for (int v = 0; v < V; ++v) {
      q[(size_t)i * V + v] = y[v];
      acc[v] += prod(p[(size_t)i * V + v], y[v]);
    }
  }
  double tot[V];
  if (seg_commit<V>(sm, b, s, part, acc, tot) && threadIdx.x == 0) {
#pragma unroll
    for (int v = 0; v < V; ++v) {
      Lane& L = lanes[s * V + v];
      if (!L.active) continue;
      L.pq = tot[v];
      if constexpr (sizeof(T) == 4) L.alpha = div0(L.s, tot[v]);
      else L.alpha = L.s / (tot[v] + kSmall);  // :67-68
    }
  }
}

// phi += alpha p; r -= alpha q; L1 = sum|r|; stop test (solv_cg.f90:73-82).
// With JAC, also s_next = r.(c r) and beta for the next iteration; with
// JAC and FLEX, beta = -(z.q)/(p.q) instead, z = c r of the new residual.
template <typename T, int V, bool JAC, bool FLEX = false>
__global__ void SG_BOUNDS(V) k_cg_update(SegMap sm, const T* __restrict__ c, T* __restrict__ phi,
                            T* __restrict__ r, const T* __restrict__ p,
                            const T* __restrict__ q, double* __restrict__ part,
                            Lane* __restrict__ lanes) {
  chain_enter();
  const int b = blockIdx.x, s = sm.blk_seg[b];
  bool act[V];
  T alpha[V];
  bool any = false;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    act[v] = lanes[s * V + v].active != 0;
    alpha[v] = (T)lanes[s * V + v].alpha;
    any |= act[v];
  }
  if (!any) return;
  const int c0 = sm.seg_c0[s], c1 = sm.seg_c1[s];
  const int stride = sm.seg_nblk[s] * blockDim.x;
  constexpr int NR = JAC ? 2 * V : V;
  double acc[NR];
#pragma unroll
  for (int k = 0; k < NR; ++k) acc[k] = 0.0;
  for (int i = c0 + sm.blk_rank[b] * blockDim.x + threadIdx.x; i < c1; i += stride) {
#pragma unroll
    for (int v = 0; v < V; ++v) {
      if (!act[v]) continue;
      const size_t k = (size_t)i * V + v;
      phi[k] = add(phi[k], mul(alpha[v], p[k]));
      const T rn = sub(r[k], mul(alpha[v], q[k]));
      r[k] = rn;
      acc[v] += (double)fabs(rn);
      if (JAC) acc[V + v] += FLEX ? prod(mul(rn, c[i]), q[k]) : prod(rn, mul(rn, c[i]));
    }
  }
  double tot[NR];
  if (seg_commit<NR>(sm, b, s, part, acc, tot) && threadIdx.x == 0) {
#pragma unroll
    for (int v = 0; v < V; ++v) {
      Lane& L = lanes[s * V + v];
      if (!L.active) continue;
      L.iter += 1;
      L.l1 = tot[v];
      const double ratio = tot[v] / (L.res0_n + kSmall);  // :81
      L.ratio = ratio;
      if (!(ratio == ratio) || isinf(ratio)) lane_stop(L, kLaneNaN, sm.n_active);
      else if (ratio < L.reduc) lane_stop(L, kLaneConverged, sm.n_active);  // :82
      else if (L.iter >= L.n_iter) lane_stop(L, kLaneMaxIter, sm.n_active);
      else if (tot[v] < L.l1_stop) lane_stop(L, kLaneRefine, sm.n_active);
      if (JAC && FLEX && L.active) {
        L.beta = flex_beta(L, tot[V + v], c1 - c0);
      } else if (JAC && L.active) {
        double beta = 1.0 / L.s;
        L.s_prev = L.s;
        L.s = tot[V + v];
        L.beta = beta * L.s;
      }
    }
  }
}

// ===================== BiCGSTAB: solv_bicg.f90:27-118 ======================
// rho = r.r0; omeg = rho*gam/(alpha*beta0+small); beta0 = rho  (:48-50;
// FP32 without the guard, div0)
template <typename T, int V>
__global__ void SG_BOUNDS(V) k_bi_rho(SegMap sm, const T* __restrict__ r, const T* __restrict__ r0,
                         double* __restrict__ part, Lane* __restrict__ lanes) {
  const int b = blockIdx.x, s = sm.blk_seg[b];
  bool any = false;
#pragma unroll
  for (int v = 0; v < V; ++v) any |= lanes[s * V + v].active != 0;
  if (!any) return;
  const int c0 = sm.seg_c0[s], c1 = sm.seg_c1[s];
  const int stride = sm.seg_nblk[s] * blockDim.x;
  double acc[V];
#pragma unroll
  for (int v = 0; v < V; ++v) acc[v] = 0.0;
  for (int i = c0 + sm.blk_rank[b] * blockDim.x + threadIdx.x; i < c1; i += stride) {
#pragma unroll
    for (int v = 0; v < V; ++v) acc[v] += prod(r[(size_t)i * V + v], r0[(size_t)i * V + v]);
  }
  double tot[V];
  if (seg_commit<V>(sm, b, s, part, acc, tot) && threadIdx.x == 0) {
#pragma unroll
    for (int v = 0; v < V; ++v) {
      Lane& L = lanes[s * V + v];
      if (!L.active) continue;
      L.rho = tot[v];
      if constexpr (sizeof(T) == 4) L.omeg = div0(L.rho * L.gam, L.alpha * L.beta0);
      else L.omeg = L.rho * L.gam / (L.alpha * L.beta0 + kSmall);
      L.beta0 = L.rho;
    }
  }
}

// p = r + omeg (p - alpha u); with JAC also z = c p  (:54-58)
template <typename T, int V, bool JAC>
__global__ void SG_BOUNDS(V) k_bi_p(SegMap sm, const T* __restrict__ c, const T* __restrict__ r,
                       T* __restrict__ p, const T* __restrict__ u, T* __restrict__ z,
                       const Lane* __restrict__ lanes) {
  chain_enter();
  const int b = blockIdx.x, s = sm.blk_seg[b];
  bool act[V];
  T om[V], al[V];
  bool any = false;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    act[v] = lanes[s * V + v].active != 0;
    om[v] = (T)lanes[s * V + v].omeg;
    al[v] = (T)lanes[s * V + v].alpha;
    any |= act[v];
  }
  if (!any) return;
  const int c0 = sm.seg_c0[s], c1 = sm.seg_c1[s];
  const int stride = sm.seg_nblk[s] * blockDim.x;
  for (int i = c0 + sm.blk_rank[b] * blockDim.x + threadIdx.x; i < c1; i += stride) {
#pragma unroll
    for (int v = 0; v < V; ++v) {
      if (!act[v]) continue;
      const size_t k = (size_t)i * V + v;
      const T pn = add(r[k], mul(om[v], sub(p[k], mul(al[v], u[k]))));
      p[k] = pn;
      if (JAC) z[k] = mul(pn, c[i]);
    }
  }
}

// y = A z, and dots: MODE 0 -> y.r0 (gam = rho/(y.r0+small), :72-73)
//                    MODE 1 -> y.r, y.y (alpha = (y.r)/(y.y+small), :98-100)
// (FP32: the same quotients without the guard, div0)
template <typename T, int V, int MODE, int CH = kRowChunk>
__global__ void SG_BOUNDS(V) k_bi_spmv(Rows<T> R, SegMap sm, const T* __restrict__ z, T* __restrict__ y,
                          const T* __restrict__ w, double* __restrict__ part,
                          Lane* __restrict__ lanes) {
  chain_enter();
  const int b = blockIdx.x, s = sm.blk_seg[b];
  bool any = false;
#pragma unroll
  for (int v = 0; v < V; ++v) any |= lanes[s * V + v].active != 0;
  if (!any) return;
  const int c0 = sm.seg_c0[s], c1 = sm.seg_c1[s];
  const int stride = sm.seg_nblk[s] * blockDim.x;
  constexpr int NR = MODE == 0 ? V : 2 * V;
  double acc[NR];
#pragma unroll
  for (int k = 0; k < NR; ++k) acc[k] = 0.0;
  for (int i = c0 + sm.blk_rank[b] * blockDim.x + threadIdx.x; i < c1; i += stride) {
    T t[V];
    row_apply<T, V, CH>(R, i, z, t);
#pragma unroll
    for (int v = 0; v < V; ++v) {
      y[(size_t)i * V + v] = t[v];
      acc[v] += prod(t[v], w[(size_t)i * V + v]);
      if (MODE == 1) acc[V + v] += prod(t[v], t[v]);
    }
  }
  double tot[NR];
  if (seg_commit<NR>(sm, b, s, part, acc, tot) && threadIdx.x == 0) {
#pragma unroll
    for (int v = 0; v < V; ++v) {
      Lane& L = lanes[s * V + v];
      if (!L.active) continue;
      if (MODE == 0) {
        if constexpr (sizeof(T) == 4) L.gam = div0(L.rho, tot[v]);
        else L.gam = L.rho / (tot[v] + kSmall);
      } else {
        if constexpr (sizeof(T) == 4) L.alpha = div0(tot[v], tot[V + v]);
        else L.alpha = tot[v] / (tot[V + v] + kSmall);
      }
    }
  }
}

// phi += gam z; r -= gam u; with JAC also z = c r   (:77-84)
template <typename T, int V, bool JAC>
__global__ void SG_BOUNDS(V) k_bi_half(SegMap sm, const T* __restrict__ c, T* __restrict__ phi,
                          T* __restrict__ r, T* __restrict__ z, const T* __restrict__ u,
                          const Lane* __restrict__ lanes) {
  chain_enter();
  const int b = blockIdx.x, s = sm.blk_seg[b];
  bool act[V];
  T g[V];
  bool any = false;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    act[v] = lanes[s * V + v].active != 0;
    g[v] = (T)lanes[s * V + v].gam;
    any |= act[v];
  }
  if (!any) return;
  const int c0 = sm.seg_c0[s], c1 = sm.seg_c1[s];
  const int stride = sm.seg_nblk[s] * blockDim.x;
  for (int i = c0 + sm.blk_rank[b] * blockDim.x + threadIdx.x; i < c1; i += stride) {
#pragma unroll
    for (int v = 0; v < V; ++v) {
      if (!act[v]) continue;
      const size_t k = (size_t)i * V + v;
      phi[k] = add(phi[k], mul(g[v], z[k]));
      const T rn = sub(r[k], mul(g[v], u[k]));
      r[k] = rn;
      if (JAC) z[k] = mul(rn, c[i]);
    }
  }
}

// phi += alpha z; r -= alpha v; L1; stop test; rho_next = r.r0 with the
// omeg / beta0 update of the next iteration's head (:105-116, :48-50).
template <typename T, int V>
__global__ void SG_BOUNDS(V) k_bi_update(SegMap sm, T* __restrict__ phi, T* __restrict__ r,
                            const T* __restrict__ z, const T* __restrict__ vv,
                            const T* __restrict__ r0, double* __restrict__ part,
                            Lane* __restrict__ lanes) {
  chain_enter();
  const int b = blockIdx.x, s = sm.blk_seg[b];
  bool act[V];
  T al[V];
  bool any = false;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    act[v] = lanes[s * V + v].active != 0;
    al[v] = (T)lanes[s * V + v].alpha;
    any |= act[v];
  }
  if (!any) return;
  const int c0 = sm.seg_c0[s], c1 = sm.seg_c1[s];
  const int stride = sm.seg_nblk[s] * blockDim.x;
  double acc[2 * V];
#pragma unroll
  for (int k = 0; k < 2 * V; ++k) acc[k] = 0.0;
  for (int i = c0 + sm.blk_rank[b] * blockDim.x + threadIdx.x; i < c1; i += stride) {
#pragma unroll
    for (int v = 0; v < V; ++v) {
      if (!act[v]) continue;
      const size_t k = (size_t)i * V + v;
      phi[k] = add(phi[k], mul(al[v], z[k]));
      const T rn = sub(r[k], mul(al[v], vv[k]));
      r[k] = rn;
      acc[v] += (double)fabs(rn);
      acc[V + v] += prod(rn, r0[k]);
    }
  }
  double tot[2 * V];
  if (seg_commit<2 * V>(sm, b, s, part, acc, tot) && threadIdx.x == 0) {
#pragma unroll
    for (int v = 0; v < V; ++v) {
      Lane& L = lanes[s * V + v];
      if (!L.active) continue;
      L.iter += 1;
      L.l1 = tot[v];
      const double ratio = tot[v] / (L.res0_n + kSmall);
      L.ratio = ratio;
      if (!(ratio == ratio) || isinf(ratio)) lane_stop(L, kLaneNaN, sm.n_active);
      else if (ratio < L.reduc) lane_stop(L, kLaneConverged, sm.n_active);
      else if (L.iter >= L.n_iter) lane_stop(L, kLaneMaxIter, sm.n_active);
      else if (tot[v] < L.l1_stop) lane_stop(L, kLaneRefine, sm.n_active);
      if (L.active) {
        L.rho = tot[V + v];
        if constexpr (sizeof(T) == 4) L.omeg = div0(L.rho * L.gam, L.alpha * L.beta0);
        else L.omeg = L.rho * L.gam / (L.alpha * L.beta0 + kSmall);
        L.beta0 = L.rho;
      }
    }
  }
}

// ================ reliable updates for the mixed-precision CG =================
// d (FP32 correction since the last update) -> x (FP64) for every lane
// flagged in mask, and d = 0.
template <int V>
__global__ void SG_BOUNDS(V) k_mp_flush(SegMap sm, const int* __restrict__ mask, double* __restrict__ x,
                           float* __restrict__ d) {
  const int b = blockIdx.x, s = sm.blk_seg[b];
  bool on[V];
  bool any = false;
#pragma unroll
  for (int v = 0; v < V; ++v) { on[v] = mask[s * V + v] != 0; any |= on[v]; }
  if (!any) return;
  const int c0 = sm.seg_c0[s], c1 = sm.seg_c1[s];
  const int stride = sm.seg_nblk[s] * blockDim.x;
  for (int i = c0 + sm.blk_rank[b] * blockDim.x + threadIdx.x; i < c1; i += stride) {
#pragma unroll
    for (int v = 0; v < V; ++v)
      if (on[v]) {
        const size_t k = (size_t)i * V + v;
        x[k] += (double)d[k];
        d[k] = 0.0f;
      }
  }
}

// The FP64 residual b - A x (solv_res.f90:12-29, k_res's operations) straight
// into the FP32 one, r_f = (float)(b - A x), for the lanes in mask, and its L1
// norm: one pass where a copy of b, the residual and the conversion took
// three.
template <int V>
__global__ void SG_BOUNDS(V) k_mp_res(Rows<double> R, SegMap sm, const int* __restrict__ mask,
                         const double* __restrict__ bvec, const double* __restrict__ phi,
                         float* __restrict__ rf, double* __restrict__ part,
                         double* __restrict__ l1_out) {
  const int b = blockIdx.x, s = sm.blk_seg[b];
  const int c0 = sm.seg_c0[s], c1 = sm.seg_c1[s];
  const int stride = sm.seg_nblk[s] * blockDim.x;
  double l1[V];
#pragma unroll
  for (int v = 0; v < V; ++v) l1[v] = 0.0;
  for (int i = c0 + sm.blk_rank[b] * blockDim.x + threadIdx.x; i < c1; i += stride) {
    double y[V];
    RowIt<double> it(R, i);
    const double d = R.diag[i];
#pragma unroll
    for (int v = 0; v < V; ++v)
      y[v] = sub(bvec[(size_t)i * V + v], mul(d, phi[(size_t)i * V + v]));
    for (int k = 0; k < it.w; ++k) {
      const int e = it.base + k * kWarp;
      const int j = __ldg(&R.col[e]);
      if (j >= 0) {
        const double a = R.val[e];
#pragma unroll
        for (int v = 0; v < V; ++v) y[v] = sub(y[v], mul(a, phi[(size_t)j * V + v]));
      }
    }
#pragma unroll
    for (int v = 0; v < V; ++v) {
      if (mask[s * V + v]) rf[(size_t)i * V + v] = (float)y[v];
      l1[v] += fabs(y[v]);
    }
  }
  double tot[V];
  if (seg_commit<V>(sm, b, s, part, l1, tot) && threadIdx.x == 0) {
#pragma unroll
    for (int v = 0; v < V; ++v) l1_out[s * V + v] = tot[v];
  }
}

// ================ flexible CG, FCG(1), for a nonlinear preconditioner ==========
// z = M(r); beta = -(z.q_old)/(p_old.q_old); p = z + beta p; q = A p;
// alpha = (p.r)/(p.q); x += alpha p; r -= alpha q.  One system, V = 1.

// gs = sum |r_i| rsd_i / N: the residual scale the network normalises by.
template <typename T>
__global__ void SG_BOUNDS(1) k_fcg_scale(SegMap sm, const T* __restrict__ r, const float* __restrict__ rsd,
                            double* __restrict__ part, Lane* __restrict__ lanes) {
  const int b = blockIdx.x, s = sm.blk_seg[b];
  if (!lanes[s].active) return;
  const int c0 = sm.seg_c0[s], c1 = sm.seg_c1[s];
  const int stride = sm.seg_nblk[s] * blockDim.x;
  double acc[1] = {0.0};
  for (int i = c0 + sm.blk_rank[b] * blockDim.x + threadIdx.x; i < c1; i += stride)
    acc[0] += fabs((double)r[i]) * rsd[i];
  double tot[1];
  if (seg_commit<1>(sm, b, s, part, acc, tot) && threadIdx.x == 0)
    lanes[s].gs = tot[0] / (double)(c1 - c0);
}

// (for the one-level operator; the V-cycle's last kernel takes z.q itself)
template <typename T>
__global__ void SG_BOUNDS(1) k_fcg_beta(SegMap sm, const T* __restrict__ z, const T* __restrict__ q,
                           double* __restrict__ part, Lane* __restrict__ lanes) {
  chain_enter();
  const int b = blockIdx.x, s = sm.blk_seg[b];
  if (!lanes[s].active) return;
  const int c0 = sm.seg_c0[s], c1 = sm.seg_c1[s];
  const int stride = sm.seg_nblk[s] * blockDim.x;
  double acc[1] = {0.0};
  for (int i = c0 + sm.blk_rank[b] * blockDim.x + threadIdx.x; i < c1; i += stride)
    acc[0] += prod(z[i], q[i]);
  double tot[1];
  if (seg_commit<1>(sm, b, s, part, acc, tot) && threadIdx.x == 0) {
    Lane& L = lanes[s];
    L.beta = flex_beta(L, tot[0], c1 - c0);
  }
}

template <typename T, int CH = kRowChunk>
__global__ void SG_BOUNDS(1) k_fcg_spmv(Rows<T> R, SegMap sm, const T* __restrict__ p, T* __restrict__ q,
                           const T* __restrict__ r, double* __restrict__ part,
                           Lane* __restrict__ lanes) {
  chain_enter();
  const int b = blockIdx.x, s = sm.blk_seg[b];
  if (!lanes[s].active) return;
  const int c0 = sm.seg_c0[s], c1 = sm.seg_c1[s];
  const int stride = sm.seg_nblk[s] * blockDim.x;
  double acc[2] = {0.0, 0.0};
  for (int i = c0 + sm.blk_rank[b] * blockDim.x + threadIdx.x; i < c1; i += stride) {
    T y[1];
    row_apply<T, 1, CH>(R, i, p, y);
    q[i] = y[0];
    acc[0] += prod(p[i], y[0]);
    acc[1] += prod(p[i], r[i]);
  }
  double tot[2];
  if (seg_commit<2>(sm, b, s, part, acc, tot) && threadIdx.x == 0) {
    Lane& L = lanes[s];
    if (!(tot[0] > 0.0) || !(tot[1] == tot[1])) {  // not SPD-like: hand over to PCG
      L.alpha = 0.0;
      lane_stop(L, kLaneStall, sm.n_active);
    } else {
      L.pq = tot[0];
      L.alpha = tot[1] / tot[0];
    }
  }
}

template <typename T>
__global__ void SG_BOUNDS(1) k_fcg_update(SegMap sm, T* __restrict__ phi, T* __restrict__ r,
                             const T* __restrict__ p, const T* __restrict__ q,
                             double* __restrict__ part, Lane* __restrict__ lanes) {
  chain_enter();
  const int b = blockIdx.x, s = sm.blk_seg[b];
  if (!lanes[s].active) return;
  const T alpha = (T)lanes[s].alpha;
  const int c0 = sm.seg_c0[s], c1 = sm.seg_c1[s];
  const int stride = sm.seg_nblk[s] * blockDim.x;
  double acc[1] = {0.0};
  for (int i = c0 + sm.blk_rank[b] * blockDim.x + threadIdx.x; i < c1; i += stride) {
    phi[i] = add(phi[i], mul(alpha, p[i]));
    const T rn = sub(r[i], mul(alpha, q[i]));
    r[i] = rn;
    acc[0] += fabs((double)rn);
  }
  double tot[1];
  if (seg_commit<1>(sm, b, s, part, acc, tot) && threadIdx.x == 0) {
    Lane& L = lanes[s];
    L.iter += 1;
    L.l1 = tot[0];
    const double ratio = tot[0] / (L.res0_n + kSmall);
    L.ratio = ratio;
    if (!(ratio == ratio) || isinf(ratio)) lane_stop(L, kLaneNaN, sm.n_active);
    else if (ratio < L.reduc) lane_stop(L, kLaneConverged, sm.n_active);
    else if (L.iter >= L.n_iter) lane_stop(L, kLaneMaxIter, sm.n_active);
    else if (tot[0] < L.l1_stop) lane_stop(L, kLaneRefine, sm.n_active);
  }
}

// ============ resident Jacobi PCG: the whole GPU on one loop, matrix in shared memory ============
// The Krylov loop of solv_cg.f90:37-84 with imat = 0 as one cooperative
// launch, for systems (one, or a batch of at most one per SM) whose matrix
// fits the SMs' shared memory: as a graph of step kernels an iteration of a
// small system is three launches and three reduction tails (14-16 us at
// 32^3), none of it bandwidth.  Each block owns a run of consecutive cells
// of one system, one block per SM: their slots in shared memory (slot-major,
// so the reads are free of bank conflicts; slots past the capacity stay in
// global memory), their r, c, phi, p and q in registers.  Two block-to-block
// exchanges an iteration are left: p.q, and |r|_1 with r.z.  The p kernel's
// exchange goes because a block forms its neighbours' p itself: every cell
// publishes the pair {z, p} once r is updated, one 16-byte gather per slot,
// and p_j = z_j + beta p_j is the owner's own operation, bit for bit.
// In an exchange a block pushes its partials into every block's inbox, and
// the value is the flag (an entry holds the pending pattern until it is
// written): no counter, no atomic, one trip through L2, and nobody polls a
// line that others poll (148 blocks polling one shared array took 3 000 -
// 4 000 cycles a time, an inbox each about 1 000).  Every block sums its
// inbox in the same fixed tree, so all hold the same scalars and stop
// together, and the sums are deterministic.  The second exchange also
// publishes the pairs: release before the push, acquire after the poll.
// Before that release each block puts its inbox of the other parity back to
// pending: it has read it already, and the next to write there has to pass
// this exchange first.  The acquire also drops the L1's old pairs, so the
// gathers of one iteration may share lines there.
// Measured: see kGridShapes (solv_gpu.cu).
constexpr int kGridMaxCells = 6144;  // cells a block owns
constexpr int kGridMaxBlocks = 160;  // inbox entries: five a lane

__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ void st_bits(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// Fixed-order warp sum, the result in every lane.
__device__ __forceinline__ double warp_sum_all(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// One warp: push this block's NV partials t into the inboxes of the system's
// nb blocks (entry `rank` of each; `stride` words from one block's inbox to
// the next) and return all the blocks' sums in t.  False when the wait ran
// out.
template <int NV>
__device__ __forceinline__ bool push_and_total(unsigned long long* inbox0, size_t stride, int rank,
                                               int nb, double (&t)[NV], SweepCtl* ctl) {
  using P = Pending<double>;
  constexpr int Q = kGridMaxBlocks / 32;
  const int l = threadIdx.x & 31;
#pragma unroll
  for (int q = 0; q < Q; ++q)
    if (l + 32 * q < nb)
#pragma unroll
      for (int v = 0; v < NV; ++v)
        st_bits(inbox0 + (l + 32 * q) * stride + (size_t)v * kGridMaxBlocks + rank,
                (unsigned long long)__double_as_longlong(t[v]));
  const unsigned long long* mine = inbox0 + rank * stride;
  unsigned long long bits[Q][NV];
#pragma unroll
  for (int q = 0; q < Q; ++q)
#pragma unroll
    for (int v = 0; v < NV; ++v) bits[q][v] = 0;
  for (int poll = 0;; ++poll) {
    bool ready = true;
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
      for (int v = 0; v < NV; ++v)
        ld_relaxed_if(l + 32 * q < nb, mine + (size_t)v * kGridMaxBlocks + l + 32 * q, bits[q][v]);
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
      for (int v = 0; v < NV; ++v) ready &= bits[q][v] != P::bits;
    if (__all_sync(0xffffffffu, ready)) break;
    if (poll >= kSweepPolls || ((poll & 63) == 63 && ld_err(ctl))) {
      if (l == 0) atomicExch(&ctl->err, 1);
      return false;
    }
  }
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    t[v] = 0.0;
#pragma unroll
    for (int q = 0; q < Q; ++q) t[v] += P::from(bits[q][v]);  // 0 past the last block
  }
#pragma unroll
  for (int v = 0; v < NV; ++v) t[v] = warp_sum_all(t[v]);
  return true;
}

// inbox: per block, per parity, three rows of kGridMaxBlocks words (p.q;
// |r|_1; r.z), all pending.
constexpr int kInboxWords = 3 * kGridMaxBlocks;

template <int B, int RPT, bool BIG>
__global__ void __launch_bounds__(B, 1) k_pcg_grid(
    Rows<double> R, SegMap sm, int W, int resident, const double* __restrict__ c,
    double* __restrict__ phi, const double* __restrict__ r_in, double2* zp,
    unsigned long long* inbox, Lane* __restrict__ lanes, SweepCtl* ctl) {
  constexpr int NW = B / 32;
  extern __shared__ __align__(16) unsigned char dyn[];
  double* val_s = reinterpret_cast<double*>(dyn);
  int* col_s = reinterpret_cast<int*>(val_s + (size_t)resident * W * B);
  __shared__ double red[2][32];
  __shared__ double tot_s[2];
  __shared__ int fail_s;
  const int b = blockIdx.x, sys = sm.blk_seg[b], nb = sm.seg_nblk[sys], b0 = sm.seg_blk0[sys];
  const int rank = sm.blk_rank[b];
  const int c0 = sm.seg_c0[sys], c1 = sm.seg_c1[sys];
  const int chunk = (((c1 - c0) + nb - 1) / nb + 31) & ~31;
  const int lo = c0 + rank * chunk, hi = min(lo + chunk, c1);
  const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
  const Lane L0 = lanes[sys];
  if (!L0.active) return;  // uniform over the system's blocks
  if (tid == 0) fail_s = 0;
  constexpr int NR = BIG ? 1 : RPT;  // BIG: c and phi stay in global memory
  double rr[RPT], pp[RPT], qq[RPT], cc[NR], ph[NR];
#pragma unroll
  for (int k = 0; k < RPT; ++k) {
    const int i = lo + k * B + tid;
    const bool h = i < hi;
    rr[k] = h ? r_in[i] : 0.0;
    if constexpr (!BIG) {
      cc[k] = h ? c[i] : 0.0;
      ph[k] = h ? phi[i] : 0.0;
    }
    pp[k] = qq[k] = 0.0;
    if (k < resident) {
      int base = 0, wi = 0;
      if (h) {
        RowIt<double> it(R, i);
        base = it.base;
        wi = it.w;
      }
      for (int u = 0; u < W; ++u) {
        const int e = base + u * kWarp;
        val_s[(k * W + u) * B + tid] = u < wi ? R.val[e] : 0.0;
        col_s[(k * W + u) * B + tid] = u < wi ? R.col[e] : -1;
      }
    }
  }
  auto c_of = [&](int k, int i) { return BIG ? __ldg(&c[i]) : cc[BIG ? 0 : k]; };
  // The sums over the system's blocks of every thread's t[], in parity par's
  // inbox; two values: the exchange that also publishes the pairs.
  auto exchange = [&](auto& t, int par) -> bool {
    constexpr int NV = sizeof(t) / sizeof(double);
#pragma unroll
    for (int v = 0; v < NV; ++v) t[v] = warp_sum(t[v]);
    if (l == 0)
#pragma unroll
      for (int v = 0; v < NV; ++v) red[v][w] = t[v];
    if (NV == 2 && nb > 1 && w == NW - 1) {  // this block's other inbox back to pending
      unsigned long long* o = inbox + ((size_t)b * 2 + (par ^ 1)) * kInboxWords;
      for (int q = l; q < nb; q += 32)
#pragma unroll
        for (int v = 0; v < 3; ++v) st_bits(o + v * kGridMaxBlocks + q, Pending<double>::bits);
    }
    __syncthreads();
    if (w == 0) {
#pragma unroll
      for (int v = 0; v < NV; ++v) t[v] = l < NW ? red[v][l] : 0.0;
#pragma unroll
      for (int v = 0; v < NV; ++v) t[v] = warp_sum_all(t[v]);
      bool ok = true;
      if (nb > 1) {
        if (NV == 2) fence_gpu();
        ok = push_and_total<NV>(inbox + ((size_t)b0 * 2 + par) * kInboxWords +
                                    (NV == 2 ? kGridMaxBlocks : 0),
                                2 * (size_t)kInboxWords, rank, nb, t, ctl);
        if (NV == 2) fence_gpu();
      }
      if (l == 0) {
#pragma unroll
        for (int v = 0; v < NV; ++v) tot_s[v] = t[v];
        if (!ok) fail_s = 1;
      }
    }
    __syncthreads();
#pragma unroll
    for (int v = 0; v < NV; ++v) t[v] = tot_s[v];
    return fail_s == 0;
  };
  const double res0_n = L0.res0_n, reduc = L0.reduc;
  const int n_iter = L0.n_iter;
  double s_cur = L0.s, s_prev = L0.s_prev, beta = 0.0, alpha = L0.alpha, pq = L0.pq;
  double l1v = L0.l1, ratio = L0.ratio;
  int iter = L0.iter, status = kLaneRunning, par = 1;
  {  // s = r.(c r), beta = (1/s_old) s (k_cg_rz with JAC); the first pairs, p = 0
    double t[2] = {0.0, 0.0};
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
      const int i = lo + k * B + tid;
      if (i < hi) {
        const double z = mul(rr[k], c_of(k, i));
        t[1] += prod(rr[k], z);
        __stcg(&zp[i], make_double2(z, 0.0));
      }
    }
    if (!exchange(t, par)) return;
    const double b0s = 1.0 / s_cur;
    s_prev = s_cur;
    s_cur = t[1];
    beta = b0s * s_cur;
  }
  while (true) {
    par ^= 1;
    // p = z + beta p here and at the neighbours; q = A p, p.q
    double a[1] = {0.0};
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
      const int i = lo + k * B + tid;
      if (i >= hi) continue;
      pp[k] = add(mul(rr[k], c_of(k, i)), mul(beta, pp[k]));
      double y = mul(__ldg(&R.diag[i]), pp[k]);
      const bool here = k < resident;
      const RowIt<double> it(R, i);
      const int wi = here ? W : it.w;
      for (int u0 = 0; u0 < wi; u0 += 6) {
        int j[6];
        double av[6];
        double2 x[6];
#pragma unroll
        for (int u = 0; u < 6; ++u) {
          j[u] = -1;
          av[u] = 0.0;
          if (u0 + u < wi) {
            const int at = (k * W + u0 + u) * B + tid, e = it.base + (u0 + u) * kWarp;
            j[u] = here ? col_s[at] : __ldg(&R.col[e]);
            av[u] = here ? val_s[at] : __ldg(&R.val[e]);
          }
        }
#pragma unroll
        for (int u = 0; u < 6; ++u) x[u] = j[u] >= 0 ? zp[j[u]] : make_double2(0.0, 0.0);
#pragma unroll
        for (int u = 0; u < 6; ++u)
          if (j[u] >= 0) y = add(y, mul(av[u], add(x[u].x, mul(beta, x[u].y))));
      }
      qq[k] = y;
      a[0] += prod(pp[k], y);
    }
    if (!exchange(a, par)) return;
    pq = a[0];
    alpha = s_cur / (pq + kSmall);  // solv_cg.f90:67-68
    // phi += alpha p; r -= alpha q; |r|_1; r.(c r) (k_cg_update with JAC)
    double t[2] = {0.0, 0.0};
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
      const int i = lo + k * B + tid;
      if (i >= hi) continue;
      if constexpr (BIG) phi[i] = add(phi[i], mul(alpha, pp[k]));
      else ph[k] = add(ph[k], mul(alpha, pp[k]));
      const double rn = sub(rr[k], mul(alpha, qq[k]));
      const double z = mul(rn, c_of(k, i));
      rr[k] = rn;
      t[0] += fabs(rn);
      t[1] += prod(rn, z);
      __stcg(&zp[i], make_double2(z, pp[k]));
    }
    if (!exchange(t, par)) return;
    iter += 1;
    l1v = t[0];
    ratio = l1v / (res0_n + kSmall);  // solv_cg.f90:81
    if (!(ratio == ratio) || isinf(ratio)) status = kLaneNaN;
    else if (ratio < reduc) status = kLaneConverged;  // :82
    else if (iter >= n_iter) status = kLaneMaxIter;
    if (status != kLaneRunning) break;
    const double b1 = 1.0 / s_cur;
    s_prev = s_cur;
    s_cur = t[1];
    beta = b1 * s_cur;
  }
  if constexpr (!BIG) {
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
      const int i = lo + k * B + tid;
      if (i < hi) phi[i] = ph[k];
    }
  }
  if (rank == 0 && tid == 0) {
    Lane L = L0;
    L.s = s_cur;
    L.s_prev = s_prev;
    L.beta = beta;
    L.alpha = alpha;
    L.pq = pq;
    L.iter = iter;
    L.l1 = l1v;
    L.ratio = ratio;
    L.active = 0;
    L.status = status;
    lanes[sys] = L;
    atomicSub(sm.n_active, 1);
  }
}

// ============ small systems: the whole call in one launch, a block per system ============
// solv_res, solv_precond and the loop of solv_cg.f90:26-84 (SOLVER 0) or
// solv_bicg.f90:27-118 (SOLVER 1), FP64, with the layout conversions, for
// systems whose gathered vectors fit one block's shared memory.  A call on a
// few hundred or thousand cells spent its time in 20 launches before the loop,
// 5-9 per iteration (1.5-3 us each, and the graph's remaining iterations as
// early exits) and the host's round trips; here it is one launch.  What
// neighbours read (p, or z, and the sweeps' t) is in shared memory, so a step
// of a DIC/DILU recurrence is a store and a poll on the SM (SharedVals; 0.74
// us through L2); a cell's own values stay in global memory (L1, L2), its
// thread the only one to touch them.  Per-cell arithmetic and the order of
// the updates are the step kernels'; the sums run in this block's fixed tree.
// A system's slices go to the warps in turn: cell i always to warp
// (i / 32 - first slice) % warps.
struct SmallArgs {
  Rows<double> R;
  const int *seg_c0, *seg_c1, *old_of_new, *slot_src;
  const double* fp;
  double *phi_dev, *res_dev;                       // caller layouts
  double *phi, *r, *r0, *p, *q, *v, *c, *cr;       // internal order
  Lane* lanes;
  double* l1;
  SweepCtl* ctl;
  int N, not_r0, imat, n_iter;
  double reduc;
};
constexpr int kSmallThreads = 512;
enum : int { kSmallResidual = 1, kSmallLoop = 2 };  // the parts of a launch

// gathered vectors in shared memory: t and z of the sweeps, p of CG
template <int SOLVER, bool SW>
constexpr int kSmallVectors = (SW ? 2 : 0) + (SOLVER == 0 || !SW ? 1 : 0);

// z = M^-1 b: the two sweeps of solv_direct.f90 over the cells c0 .. c1, one
// block (ends with a barrier).  Not inlined: BiCGSTAB's two calls would
// otherwise spill each other's addresses around every wait.
template <int V>
__device__ __noinline__ void small_direct(const SmallArgs& A, int c0, int c1, const double* b,
                                          double* t_s, double* z_s) {
  constexpr int NW = kSmallThreads / 32, C = V <= 2 ? 8 : 6;
  const Rows<double>& R = A.R;
  const int s_lo = c0 >> 5, ns = ((c1 + 31) >> 5) - s_lo, first = s_lo * 32;
  const int wid = threadIdx.x >> 5;
  const SharedVals tv{(unsigned)__cvta_generic_to_shared(t_s), first};
  const SharedVals zv{(unsigned)__cvta_generic_to_shared(z_s), first};
  double acc[V], ci = 0.0;
  auto coef = [&](int e) { return __ldg(&R.sval[e]); };
  auto term = [](const double a, const double (&xv)[V], double (&m)[V]) {
#pragma unroll
    for (int v = 0; v < V; ++v) m[v] = mul(a, xv[v]);
  };
  auto fold = [&](const double (&m)[V]) {
#pragma unroll
    for (int v = 0; v < V; ++v) acc[v] = sub(acc[v], m[v]);
  };
  for (int r = wid; r < ns; r += NW)
    sweep_slice<false, true, C, V, double>(
        A.N, R, s_lo + r, c0, c1, tv, A.ctl,
        [&](int i) {
          ci = A.c[i];
#pragma unroll
          for (int v = 0; v < V; ++v) acc[v] = b[(size_t)i * V + v];
        },
        coef, term, fold,
        [&](int i) {
#pragma unroll
          for (int v = 0; v < V; ++v) {
            tv.put(i, V, v, mul(acc[v], ci));
            zv.put(i, V, v, Pending<double>::value());
          }
        });
  __syncthreads();
  for (int r = wid; r < ns; r += NW)
    sweep_slice<true, true, C, V, double>(
        A.N, R, s_lo + ns - 1 - r, c0, c1, zv, A.ctl,
        [&](int i) {
          ci = A.c[i];
          const double cr = A.cr[i];
#pragma unroll
          for (int v = 0; v < V; ++v) acc[v] = mul(t_s[(i - first) * V + v], cr);
        },
        coef, term, fold,
        [&](int i) {
#pragma unroll
          for (int v = 0; v < V; ++v) {
            zv.put(i, V, v, mul(acc[v], ci));
            t_s[(i - first) * V + v] = Pending<double>::value();
          }
        });
  __syncthreads();
}

template <int SOLVER, int V, bool SW>
__global__ void __launch_bounds__(kSmallThreads, 1)
k_small_solve(const __grid_constant__ SmallArgs A, int parts) {
  constexpr int NW = kSmallThreads / 32;
  extern __shared__ __align__(16) double dyn_s[];
  __shared__ double red[2][2 * V][NW];
  __shared__ Lane L_s[V];     // the lanes as reported
  __shared__ double rn_s[V];  // their |r0|_1
  const Rows<double>& R = A.R;
  const int sys = blockIdx.x, c0 = A.seg_c0[sys], c1 = A.seg_c1[sys];
  const int s_lo = c0 >> 5, ns = ((c1 + 31) >> 5) - s_lo, first = s_lo * 32;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* t_s = dyn_s;                             // SW: forward sweeps
  double* z_s = dyn_s + (SW ? ns * 32 * V : 0);    // SW: backward sweeps; BiCGSTAB: z
  double* p_s = SOLVER == 0 && SW ? z_s + ns * 32 * V : z_s;  // CG: p
  double* x_s = SOLVER == 0 ? p_s : z_s;           // what the matrix product gathers
  auto vals_of = [&](double* a) {
    return SharedVals{(unsigned)__cvta_generic_to_shared(a), first};
  };
  auto each = [&](auto&& f) {  // f(i) for this thread's cells
    for (int r = wid; r < ns; r += NW) {
      const int i = first + r * 32 + lane;
      if (i >= c0 && i < c1) f(i);
    }
  };
  auto li = [&](int i, int v) { return (i - first) * V + v; };
  int buf = 0;
  auto sums = [&](auto& t) {  // block sums of t[], in every thread (and a barrier)
    constexpr int NR = sizeof(t) / sizeof(double);
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      const double x = warp_sum(t[k]);
      if (lane == 0) red[buf][k][wid] = x;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NR; ++k) t[k] = warp_sum_all(lane < NW ? red[buf][k][lane] : 0.0);
    buf ^= 1;
  };
  // y = b - A x (RES) or y = A x for row i, x gathered from x_s
  auto row = [&](int i, const double* x, auto res, double (&y)[V]) {
    constexpr bool RES = decltype(res)::value;
    RowIt<double> it(R, i);
    const double d = __ldg(&R.diag[i]);
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const double m = mul(d, x[li(i, v)]);
      y[v] = RES ? sub(y[v], m) : m;
    }
    for (int u0 = 0; u0 < it.w; u0 += 6) {
      int j[6];
      double a[6];
#pragma unroll
      for (int u = 0; u < 6; ++u) {
        j[u] = -1;
        if (u0 + u < it.w) {
          const int e = it.base + (u0 + u) * kWarp;
          j[u] = __ldg(&R.col[e]);
          a[u] = __ldg(&R.val[e]);
        }
      }
#pragma unroll
      for (int u = 0; u < 6; ++u)
        if (j[u] >= 0) {
#pragma unroll
          for (int v = 0; v < V; ++v) {
            const double m = mul(a[u], x[li(j[u], v)]);
            y[v] = RES ? sub(y[v], m) : add(y[v], m);
          }
        }
    }
  };
  using True = std::true_type;
  using False = std::false_type;

  if (parts & kSmallResidual) {  // solv_res.f90:12-29
    each([&](int i) {
      const int o = A.old_of_new[i];
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const double f = A.phi_dev[(size_t)o * V + v];
        A.phi[(size_t)i * V + v] = f;
        x_s[li(i, v)] = f;
      }
    });
    __syncthreads();
    double l1[V];
#pragma unroll
    for (int v = 0; v < V; ++v) l1[v] = 0.0;
    each([&](int i) {
      const int o = A.old_of_new[i];
      double y[V];
#pragma unroll
      for (int v = 0; v < V; ++v) y[v] = A.res_dev[(size_t)v * A.N + o];
      if (!A.not_r0) row(i, x_s, True(), y);
#pragma unroll
      for (int v = 0; v < V; ++v) {
        A.res_dev[(size_t)v * A.N + o] = y[v];
        A.r0[(size_t)i * V + v] = y[v];
        l1[v] += fabs(y[v]);
      }
    });
    sums(l1);
    if (threadIdx.x == 0)
#pragma unroll
      for (int v = 0; v < V; ++v) A.l1[sys * V + v] = l1[v];
    if (gridDim.x == 1) {  // solv_cg.f90:21 (a batch: the host looks at all its systems)
      double mx = -HUGE_VAL;
#pragma unroll
      for (int v = 0; v < V; ++v) mx = mx < l1[v] ? l1[v] : mx;
      if (mx < kSmall) return;
    }
    __syncthreads();
  }
  if (!(parts & kSmallLoop)) return;

  // the lanes' scalars (every thread's own copy), bit v of act: still running
  struct Scalars {
    double s, alpha, beta, beta0, gam;  // BiCGSTAB: s is rho, beta is omeg
  };
  Scalars L[V];
  unsigned act = 0;
  int iter = 0;
#pragma unroll
  for (int v = 0; v < V; ++v) {  // as k_lane_init
    L[v] = {SOLVER == 0 ? kLarge : 0.0, 1.0, 0.0, 1.0, 1.0};
    if (A.n_iter > 0) act |= 1u << v;
    if (threadIdx.x == 0) {
      L_s[v] = Lane{};
      L_s[v].status = A.n_iter > 0 ? kLaneRunning : kLaneMaxIter;
      rn_s[v] = A.l1[sys * V + v];  // this block's own, or the launch's before
    }
  }
  auto on = [&](int v) { return ((act >> v) & 1u) != 0; };
  auto pending = [&](double* a, int per) {  // whole slices
    for (int k = threadIdx.x; k < ns * 32 * per; k += kSmallThreads) a[k] = Pending<double>::value();
  };
  // solv_precond
  if constexpr (SW) {
    pending(t_s, 1);
    __syncthreads();
    const SharedVals cv = vals_of(t_s);
    double d = 0.0;
    const bool dilu = A.imat == 2;
    for (int r = wid; r < ns; r += NW)
      sweep_slice<false, true, 8, 1, double2>(
          A.N, R, s_lo + r, c0, c1, cv, A.ctl, [&](int i) { d = __ldg(&R.diag[i]); },
          [&](int e) {
            return make_double2(dilu ? __ldg(&A.fp[__ldg(&A.slot_src[e]) >> 1]) : 0.0,
                                __ldg(&R.sval[e]));
          },
          [&](const double2& a, const double (&cj)[1], double (&m)[1]) {
            m[0] = dilu ? mul(mul(a.x, cj[0]), a.y) : mul(mul(a.y, a.y), cj[0]);
          },
          [&](const double (&m)[1]) { d = sub(d, m[0]); },
          [&](int i) {
            const double ci = 1.0 / add(d, kSmall);
            A.cr[i] = d;
            A.c[i] = ci;
            cv.put(i, 1, 0, ci);
          });
    __syncthreads();
    pending(t_s, V);
  }
  each([&](int i) {
    if constexpr (!SW) A.c[i] = 1.0 / add(__ldg(&R.diag[i]), kSmall);
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const size_t k = (size_t)i * V + v;
      A.r[k] = A.r0[k];
      if (SOLVER == 0) p_s[li(i, v)] = 0.0;
      else A.p[k] = A.q[k] = 0.0;
    }
  });
  __syncthreads();
  auto direct = [&](const double* b) {
    if constexpr (SW) small_direct<V>(A, c0, c1, b, t_s, z_s);
  };
  // the stopping test of a lane whose |r|_1 is l1 (solv_cg.f90:78-82)
  auto stop = [&](int v, double l1) {
    const double ratio = l1 / (rn_s[v] + kSmall);
    int status = kLaneRunning;
    if (!(ratio == ratio) || isinf(ratio)) status = kLaneNaN;
    else if (ratio < A.reduc) status = kLaneConverged;
    else if (iter >= A.n_iter) status = kLaneMaxIter;
    if (status == kLaneRunning) return;
    act &= ~(1u << v);
    if (threadIdx.x == 0) {
      L_s[v].iter = iter;
      L_s[v].l1 = l1;
      L_s[v].ratio = ratio;
      L_s[v].status = status;
    }
  };
  if constexpr (SOLVER == 0) {
    while (act) {
      ++iter;
      direct(A.r);
      double rz[V];
#pragma unroll
      for (int v = 0; v < V; ++v) rz[v] = 0.0;
      auto z_of = [&](int i, int v, double ri) {
        return SW ? z_s[li(i, v)] : mul(ri, A.c[i]);
      };
      each([&](int i) {
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const double ri = A.r[(size_t)i * V + v];
          rz[v] += prod(ri, z_of(i, v, ri));
        }
      });
      sums(rz);
#pragma unroll
      for (int v = 0; v < V; ++v)
        if (on(v)) {
          const double b = 1.0 / L[v].s;
          L[v].s = rz[v];
          L[v].beta = b * L[v].s;
        }
      each([&](int i) {
#pragma unroll
        for (int v = 0; v < V; ++v)
          if (on(v))
            p_s[li(i, v)] = add(z_of(i, v, A.r[(size_t)i * V + v]), mul(L[v].beta, p_s[li(i, v)]));
      });
      __syncthreads();
      double pq[V];
#pragma unroll
      for (int v = 0; v < V; ++v) pq[v] = 0.0;
      each([&](int i) {
        double y[V];
        row(i, p_s, False(), y);
#pragma unroll
        for (int v = 0; v < V; ++v) {
          A.q[(size_t)i * V + v] = y[v];
          pq[v] += prod(p_s[li(i, v)], y[v]);
        }
      });
      sums(pq);
      double l1[V];
#pragma unroll
      for (int v = 0; v < V; ++v) {
        if (on(v)) L[v].alpha = L[v].s / (pq[v] + kSmall);
        l1[v] = 0.0;
      }
      each([&](int i) {
#pragma unroll
        for (int v = 0; v < V; ++v)
          if (on(v)) {
            const size_t k = (size_t)i * V + v;
            A.phi[k] = add(A.phi[k], mul(L[v].alpha, p_s[li(i, v)]));
            const double rn = sub(A.r[k], mul(L[v].alpha, A.q[k]));
            A.r[k] = rn;
            l1[v] += fabs(rn);
          }
      });
      sums(l1);
#pragma unroll
      for (int v = 0; v < V; ++v)
        if (on(v)) stop(v, l1[v]);
    }
  } else {
    auto head = [&](Scalars& X, double rho) {  // solv_bicg.f90:48-50
      X.s = rho;
      X.beta = X.s * X.gam / (X.alpha * X.beta0 + kSmall);
      X.beta0 = X.s;
    };
    double rho[V];
#pragma unroll
    for (int v = 0; v < V; ++v) rho[v] = 0.0;
    each([&](int i) {
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const size_t k = (size_t)i * V + v;
        rho[v] += prod(A.r[k], A.r0[k]);
      }
    });
    sums(rho);
#pragma unroll
    for (int v = 0; v < V; ++v)
      if (on(v)) head(L[v], rho[v]);
    while (act) {
      ++iter;
      each([&](int i) {  // p = r + omeg (p - alpha u)
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const size_t k = (size_t)i * V + v;
          if (on(v))
            A.p[k] = add(A.r[k], mul(L[v].beta, sub(A.p[k], mul(L[v].alpha, A.q[k]))));
          if (!SW) z_s[li(i, v)] = mul(A.p[k], A.c[i]);
        }
      });
      if (SW) direct(A.p);
      else __syncthreads();
      double g[V];
#pragma unroll
      for (int v = 0; v < V; ++v) g[v] = 0.0;
      each([&](int i) {  // u = A z, u.r0
        double y[V];
        row(i, z_s, False(), y);
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const size_t k = (size_t)i * V + v;
          A.q[k] = y[v];
          g[v] += prod(y[v], A.r0[k]);
        }
      });
      sums(g);
#pragma unroll
      for (int v = 0; v < V; ++v)
        if (on(v)) L[v].gam = L[v].s / (g[v] + kSmall);
      each([&](int i) {  // phi += gam z; r -= gam u
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const size_t k = (size_t)i * V + v;
          if (on(v)) {
            A.phi[k] = add(A.phi[k], mul(L[v].gam, z_s[li(i, v)]));
            A.r[k] = sub(A.r[k], mul(L[v].gam, A.q[k]));
          }
          if (!SW) z_s[li(i, v)] = mul(A.r[k], A.c[i]);
        }
      });
      __syncthreads();
      if (SW) direct(A.r);
      double d[2 * V];
#pragma unroll
      for (int k = 0; k < 2 * V; ++k) d[k] = 0.0;
      each([&](int i) {  // v = A z, v.r, v.v
        double y[V];
        row(i, z_s, False(), y);
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const size_t k = (size_t)i * V + v;
          A.v[k] = y[v];
          d[v] += prod(y[v], A.r[k]);
          d[V + v] += prod(y[v], y[v]);
        }
      });
      sums(d);
#pragma unroll
      for (int v = 0; v < V; ++v)
        if (on(v)) L[v].alpha = d[v] / (d[V + v] + kSmall);
#pragma unroll
      for (int k = 0; k < 2 * V; ++k) d[k] = 0.0;
      each([&](int i) {  // phi += alpha z; r -= alpha v; |r|_1, r.r0
#pragma unroll
        for (int v = 0; v < V; ++v)
          if (on(v)) {
            const size_t k = (size_t)i * V + v;
            A.phi[k] = add(A.phi[k], mul(L[v].alpha, z_s[li(i, v)]));
            const double rn = sub(A.r[k], mul(L[v].alpha, A.v[k]));
            A.r[k] = rn;
            d[v] += fabs(rn);
            d[V + v] += prod(rn, A.r0[k]);
          }
      });
      sums(d);
#pragma unroll
      for (int v = 0; v < V; ++v)
        if (on(v)) {
          stop(v, d[v]);
          if (on(v)) head(L[v], d[V + v]);
        }
    }
  }
  each([&](int i) {
    const int o = A.old_of_new[i];
#pragma unroll
    for (int v = 0; v < V; ++v) A.phi_dev[(size_t)o * V + v] = A.phi[(size_t)i * V + v];
  });
  if (threadIdx.x == 0)
#pragma unroll
    for (int v = 0; v < V; ++v) A.lanes[sys * V + v] = L_s[v];
}

// ============ persistent fused Jacobi PCG: one thread-block cluster per system ============
// The whole Krylov loop of solv_cg.f90:37-84 with imat = 0 in one launch:
// each cluster of CTAs (kPcgCluster, or kPcgClusterMax where the GPU holds
// a cluster that large at once) owns one system (segment) and iterates it
// to its stopping test, fusing the Jacobi step into the direction update,
// the product with p.q, and the solution / residual update with |r|_1 and
// r.z.  Per iteration three cluster barriers (after p; after the p.q
// partials; after the update's partials); each CTA reduces its cells in a
// fixed tree, puts its partials in shared memory, and in every CTA one warp
// reads the cluster's partials over distributed shared memory (a lane per
// rank) and sums them in a fixed tree -- so all CTAs hold the same scalars
// and take the same branch, and the sums are deterministic.  Per-cell arithmetic is the graph path's (k_cg_p,
// k_cg_spmv, k_cg_update with JAC), so a solve differs from it only in the
// reduction trees.  The loop is bounded by the lane's n_iter.
constexpr int kPcgCluster = 8;      // portable cluster size
constexpr int kPcgClusterMax = 16;  // non-portable, one system's whole GPC
constexpr int kPcgThreads = 1024;

__device__ __forceinline__ double cluster_block_sum(double v, double* red) {
  // fixed-order block sum; result in every thread
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  v = warp_sum(v);
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double t = 0.0;
  if (w == 0) {
    t = l < (int)(blockDim.x >> 5) ? red[l] : 0.0;
    t = warp_sum(t);
    if (l == 0) red[32] = t;
  }
  __syncthreads();
  return red[32];
}

// Two fixed-order block sums in one pass (red holds 2 x 33 doubles).
__device__ __forceinline__ void cluster_block_sum2(double& a, double& b, double* red) {
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  a = warp_sum(a);
  b = warp_sum(b);
  __syncthreads();
  if (l == 0) {
    red[w] = a;
    red[33 + w] = b;
  }
  __syncthreads();
  if (w == 0) {
    const bool in = l < (int)(blockDim.x >> 5);
    double ta = warp_sum(in ? red[l] : 0.0);
    double tb = warp_sum(in ? red[33 + l] : 0.0);
    if (l == 0) {
      red[32] = ta;
      red[65] = tb;
    }
  }
  __syncthreads();
  a = red[32];
  b = red[65];
}

// y_i = (A p)_i for two rows at once (i1 < 0: none), each summed in slot
// order as row_apply does; slot k of both rows is loaded before either is
// added, so two independent gathers are in flight (two slots a row spilled
// under the 64 registers a 1024-thread block allows).
__device__ __forceinline__ void row_pair_apply(const Rows<double>& R, int i0, int i1,
                                               const double* p, double& y0, double& y1) {
  RowIt<double> r0(R, i0);
  RowIt<double> r1(R, i1 >= 0 ? i1 : i0);
  const int w0 = r0.w, w1 = i1 >= 0 ? r1.w : 0;
  y0 = mul(R.diag[i0], __ldcg(&p[i0]));
  y1 = i1 >= 0 ? mul(R.diag[i1], __ldcg(&p[i1])) : 0.0;
  const int wm = max(w0, w1);
  for (int k = 0; k < wm; ++k) {
    int j0 = -1, j1 = -1;
    double a0 = 0.0, a1 = 0.0;
    if (k < w0) {
      const int e = r0.base + k * kWarp;
      j0 = __ldg(&R.col[e]);
      a0 = __ldg(&R.val[e]);
    }
    if (k < w1) {
      const int e = r1.base + k * kWarp;
      j1 = __ldg(&R.col[e]);
      a1 = __ldg(&R.val[e]);
    }
    const double x0 = j0 >= 0 ? __ldcg(&p[j0]) : 0.0;
    const double x1 = j1 >= 0 ? __ldcg(&p[j1]) : 0.0;
    if (j0 >= 0) y0 = add(y0, mul(a0, x0));
    if (j1 >= 0) y1 = add(y1, mul(a1, x1));
  }
}

__global__ void __launch_bounds__(kPcgThreads) k_pcg_cluster(
    Rows<double> R, const int* __restrict__ seg_c0, const int* __restrict__ seg_c1,
    const double* __restrict__ c, double* __restrict__ phi, double* __restrict__ r,
    double* __restrict__ p, double* __restrict__ q, Lane* __restrict__ lanes,
    int* __restrict__ n_active) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  __shared__ double red[66];
  __shared__ double part[2][2];  // this CTA's partials: [product][update]
  __shared__ double tot_s[2];
  const int rank = (int)cl.block_rank(), cs = (int)cl.num_blocks();
  const int sys = blockIdx.x / cs;
  const int c0 = seg_c0[sys], c1 = seg_c1[sys];
  const int stride = cs * blockDim.x;
  const int first = c0 + rank * blockDim.x + threadIdx.x;
  // the lane's scalars, in registers (the Lane itself is written back once)
  const Lane L0 = lanes[sys];
  if (!L0.active) return;  // uniform over the cluster
  const double res0_n = L0.res0_n, reduc = L0.reduc;
  const int n_iter = L0.n_iter;
  double s_cur = L0.s, s_prev = L0.s_prev, beta = 0.0, alpha = L0.alpha, pq = L0.pq;
  double l1v = L0.l1, ratio = L0.ratio;
  int iter = L0.iter;
  // the cluster's totals of one partial slot: lane q of warp 0 reads rank
  // q's pair over distributed shared memory, the warp sums them in a fixed
  // tree (the same in every CTA), and the block takes the pair from there
  auto cluster_totals = [&](int slot, double& t0, double& t1) {
    if (threadIdx.x < 32) {
      const int l = threadIdx.x;
      double a = 0.0, b = 0.0;
      if (l < cs) {
        const double* pp = cl.map_shared_rank(&part[slot][0], l);
        a = pp[0];
        b = pp[1];
      }
      a = warp_sum(a);
      b = warp_sum(b);
      if (l == 0) {
        tot_s[0] = a;
        tot_s[1] = b;
      }
    }
    __syncthreads();
    t0 = tot_s[0];
    t1 = tot_s[1];
  };
  // s = r.(c r), beta = (1/s_old) s (k_cg_rz with JAC)
  {
    double a = 0.0;
    for (int i = first; i < c1; i += stride) {
      const double ri = r[i];
      a += prod(ri, mul(ri, c[i]));
    }
    a = cluster_block_sum(a, red);
    if (threadIdx.x == 0) {
      part[1][0] = a;
      part[1][1] = 0.0;
    }
    cl.sync();
    double s_new, unused;
    cluster_totals(1, s_new, unused);
    const double b0 = 1.0 / s_cur;
    s_prev = s_cur;
    s_cur = s_new;
    beta = b0 * s_cur;
  }
  int status = kLaneRunning;
  while (true) {
    // (a partial slot is rewritten only two barriers after its last read)
    // p = z + beta p, z = c r (k_cg_p with JAC)
    for (int i = first; i < c1; i += stride) {
      const double zi = mul(r[i], c[i]);
      p[i] = add(zi, mul(beta, p[i]));
    }
    cl.sync();  // p complete in the cluster
    // q = A p, p.q (k_cg_spmv); neighbours' p read past L1; two rows at a time
    double a = 0.0;
    for (int i = first; i < c1; i += 2 * stride) {
      const int i1 = i + stride < c1 ? i + stride : -1;
      double y0, y1;
      row_pair_apply(R, i, i1, p, y0, y1);
      q[i] = y0;
      a += prod(__ldcg(&p[i]), y0);
      if (i1 >= 0) {
        q[i1] = y1;
        a += prod(__ldcg(&p[i1]), y1);
      }
    }
    a = cluster_block_sum(a, red);
    if (threadIdx.x == 0) {
      part[0][0] = a;
      part[0][1] = 0.0;
    }
    cl.sync();
    double unused2;
    cluster_totals(0, pq, unused2);
    alpha = s_cur / (pq + kSmall);  // solv_cg.f90:67-68
    // phi += alpha p; r -= alpha q; |r|_1; r.(c r) (k_cg_update with JAC)
    double l1 = 0.0, rz = 0.0;
    for (int i = first; i < c1; i += stride) {
      phi[i] = add(phi[i], mul(alpha, p[i]));
      const double rn = sub(r[i], mul(alpha, q[i]));
      r[i] = rn;
      l1 += fabs(rn);
      rz += prod(rn, mul(rn, c[i]));
    }
    cluster_block_sum2(l1, rz, red);
    if (threadIdx.x == 0) {
      part[1][0] = l1;
      part[1][1] = rz;
    }
    cl.sync();
    double t1, t2;
    cluster_totals(1, t1, t2);
    iter += 1;
    l1v = t1;
    ratio = t1 / (res0_n + kSmall);  // solv_cg.f90:81
    if (!(ratio == ratio) || isinf(ratio)) status = kLaneNaN;
    else if (ratio < reduc) status = kLaneConverged;  // :82
    else if (iter >= n_iter) status = kLaneMaxIter;
    if (status != kLaneRunning) break;
    const double b1 = 1.0 / s_cur;
    s_prev = s_cur;
    s_cur = t2;
    beta = b1 * s_cur;
  }
  cl.sync();  // no CTA leaves while others may still read its partials
  if (rank == 0 && threadIdx.x == 0) {
    Lane L = L0;
    L.s = s_cur;
    L.s_prev = s_prev;
    L.beta = beta;
    L.alpha = alpha;
    L.pq = pq;
    L.iter = iter;
    L.l1 = l1v;
    L.ratio = ratio;
    L.active = 0;
    L.status = status;
    lanes[sys] = L;
    atomicSub(n_active, 1);
  }
}

// The same loop for a system small enough for one cluster to hold
// (at most cs x 1024 x RPT cells): each CTA owns a contiguous block of
// B = 1024 x RPT cells, keeps their r, c, phi, p and q in registers (RPT
// cells a thread) and their p in shared memory, and the product reads a
// neighbour's p over distributed shared memory from the CTA that owns it
// -- no vector goes through L2 inside the loop, only the matrix slots
// (read-only, L1-resident after the first pass).  Per-cell arithmetic and
// the slot order of the sums are the global-memory kernel's.
template <int RPT>
__global__ void __launch_bounds__(kPcgThreads) k_pcg_cluster_res(
    Rows<double> R, const int* __restrict__ seg_c0, const int* __restrict__ seg_c1,
    const double* __restrict__ c, double* __restrict__ phi, double* __restrict__ r,
    double* __restrict__ p, double* __restrict__ q, Lane* __restrict__ lanes,
    int* __restrict__ n_active) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  constexpr int B = kPcgThreads * RPT;
  constexpr int LOGB = RPT == 1 ? 10 : 11;
  static_assert(RPT == 1 || RPT == 2, "one or two cells a thread");
  __shared__ double p_s[B];
  __shared__ double red[66];
  __shared__ double part[2][2];
  __shared__ double tot_s[2];
  const int rank = (int)cl.block_rank(), cs = (int)cl.num_blocks();
  const int sys = blockIdx.x / cs;
  const int c0 = seg_c0[sys], c1 = seg_c1[sys];
  const Lane L0 = lanes[sys];
  if (!L0.active) return;  // uniform over the cluster
  int row[RPT];
  double rr[RPT], cc[RPT], ph[RPT], pp[RPT], qq[RPT];
#pragma unroll
  for (int u = 0; u < RPT; ++u) {
    row[u] = c0 + rank * B + u * kPcgThreads + (int)threadIdx.x;
    const bool h = row[u] < c1;
    rr[u] = h ? r[row[u]] : 0.0;
    cc[u] = h ? c[row[u]] : 0.0;
    ph[u] = h ? phi[row[u]] : 0.0;
    pp[u] = h ? p[row[u]] : 0.0;
    qq[u] = 0.0;
    if (!h) row[u] = -1;
  }
  const double res0_n = L0.res0_n, reduc = L0.reduc;
  const int n_iter = L0.n_iter;
  double s_cur = L0.s, s_prev = L0.s_prev, beta = 0.0, alpha = L0.alpha, pq = L0.pq;
  double l1v = L0.l1, ratio = L0.ratio;
  int iter = L0.iter;
  auto cluster_totals = [&](int slot, double& t0, double& t1) {
    if (threadIdx.x < 32) {
      const int l = threadIdx.x;
      double a = 0.0, b = 0.0;
      if (l < cs) {
        const double* pr = cl.map_shared_rank(&part[slot][0], l);
        a = pr[0];
        b = pr[1];
      }
      a = warp_sum(a);
      b = warp_sum(b);
      if (l == 0) {
        tot_s[0] = a;
        tot_s[1] = b;
      }
    }
    __syncthreads();
    t0 = tot_s[0];
    t1 = tot_s[1];
  };
  // s = r.(c r), beta = (1/s_old) s
  {
    double a = 0.0;
#pragma unroll
    for (int u = 0; u < RPT; ++u)
      if (row[u] >= 0) a += prod(rr[u], mul(rr[u], cc[u]));
    a = cluster_block_sum(a, red);
    if (threadIdx.x == 0) {
      part[1][0] = a;
      part[1][1] = 0.0;
    }
    cl.sync();
    double s_new, unused;
    cluster_totals(1, s_new, unused);
    const double b0 = 1.0 / s_cur;
    s_prev = s_cur;
    s_cur = s_new;
    beta = b0 * s_cur;
  }
  int status = kLaneRunning;
  while (true) {
    // p = z + beta p, z = c r; this CTA's p into shared memory
#pragma unroll
    for (int u = 0; u < RPT; ++u) {
      if (row[u] >= 0) pp[u] = add(mul(rr[u], cc[u]), mul(beta, pp[u]));
      p_s[u * kPcgThreads + threadIdx.x] = pp[u];
    }
    cl.sync();  // every CTA's p visible in the cluster
    // q = A p, p.q: neighbours' p from their owners' shared memory
    double a = 0.0;
#pragma unroll
    for (int u = 0; u < RPT; ++u) {
      if (row[u] < 0) continue;
      RowIt<double> it(R, row[u]);
      double y = mul(__ldg(&R.diag[row[u]]), pp[u]);
      for (int k0 = 0; k0 < it.w; k0 += 4) {
        int j[4];
        double av[4], xv[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          j[v] = -1;
          av[v] = 0.0;
          if (k0 + v < it.w) {
            const int e = it.base + (k0 + v) * kWarp;
            j[v] = __ldg(&R.col[e]);
            av[v] = __ldg(&R.val[e]);
          }
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          xv[v] = 0.0;
          if (j[v] >= 0) {
            const int o = j[v] - c0;
            xv[v] = *cl.map_shared_rank(&p_s[o & (B - 1)], o >> LOGB);
          }
        }
#pragma unroll
        for (int v = 0; v < 4; ++v)
          if (j[v] >= 0) y = add(y, mul(av[v], xv[v]));
      }
      qq[u] = y;
      a += prod(pp[u], y);
    }
    a = cluster_block_sum(a, red);
    if (threadIdx.x == 0) {
      part[0][0] = a;
      part[0][1] = 0.0;
    }
    cl.sync();
    double unused2;
    cluster_totals(0, pq, unused2);
    alpha = s_cur / (pq + kSmall);  // solv_cg.f90:67-68
    double l1 = 0.0, rz = 0.0;
#pragma unroll
    for (int u = 0; u < RPT; ++u) {
      if (row[u] < 0) continue;
      ph[u] = add(ph[u], mul(alpha, pp[u]));
      const double rn = sub(rr[u], mul(alpha, qq[u]));
      rr[u] = rn;
      l1 += fabs(rn);
      rz += prod(rn, mul(rn, cc[u]));
    }
    cluster_block_sum2(l1, rz, red);
    if (threadIdx.x == 0) {
      part[1][0] = l1;
      part[1][1] = rz;
    }
    cl.sync();
    double t1, t2;
    cluster_totals(1, t1, t2);
    iter += 1;
    l1v = t1;
    ratio = t1 / (res0_n + kSmall);  // solv_cg.f90:81
    if (!(ratio == ratio) || isinf(ratio)) status = kLaneNaN;
    else if (ratio < reduc) status = kLaneConverged;  // :82
    else if (iter >= n_iter) status = kLaneMaxIter;
    if (status != kLaneRunning) break;
    const double b1 = 1.0 / s_cur;
    s_prev = s_cur;
    s_cur = t2;
    beta = b1 * s_cur;
  }
#pragma unroll
  for (int u = 0; u < RPT; ++u) {
    if (row[u] < 0) continue;
    phi[row[u]] = ph[u];
    r[row[u]] = rr[u];
    p[row[u]] = pp[u];
    q[row[u]] = qq[u];
  }
  cl.sync();  // no CTA leaves while others may still read its shared memory
  if (rank == 0 && threadIdx.x == 0) {
    Lane L = L0;
    L.s = s_cur;
    L.s_prev = s_prev;
    L.beta = beta;
    L.alpha = alpha;
    L.pq = pq;
    L.iter = iter;
    L.l1 = l1v;
    L.ratio = ratio;
    L.active = 0;
    L.status = status;
    lanes[sys] = L;
    atomicSub(n_active, 1);
  }
}

// How local a structure is for k_pcg_cluster_res: over all slots, how many
// have their neighbour in the same block of 2^logb cells of the system as
// the row (cnt[0] slots, cnt[1] local ones).  seg_c0/seg_c1 are sorted.
__global__ void k_block_locality(int n, Rows<double> R, const int* __restrict__ seg_c0,
                                 const int* __restrict__ seg_c1, int n_seg, int logb,
                                 unsigned long long* __restrict__ cnt) {
  unsigned long long tot = 0, loc = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int lo = 0, hi = n_seg - 1;  // the system of row i
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (seg_c0[mid] <= i) lo = mid;
      else hi = mid - 1;
    }
    const int c0 = seg_c0[lo];
    RowIt<double> it(R, i);
    for (int k = 0; k < it.w; ++k) {
      const int j = R.col[it.base + k * kWarp];
      if (j < 0) continue;
      ++tot;
      loc += ((j - c0) >> logb) == ((i - c0) >> logb);
    }
  }
  tot = (unsigned long long)warp_sum((double)tot);
  loc = (unsigned long long)warp_sum((double)loc);
  if ((threadIdx.x & 31) == 0 && tot) {
    atomicAdd(&cnt[0], tot);
    atomicAdd(&cnt[1], loc);
  }
}

// How well a warp's gathers share lines: over all pairs of neighbouring cells
// of a slice and each slot, how many read columns at most two apart (cnt[0]
// pairs, cnt[1] near ones).
__global__ void k_near_slots(int n, Rows<double> R, unsigned long long* __restrict__ cnt) {
  const int lane = threadIdx.x & 31, ns = (n + 31) >> 5;
  const int W = gridDim.x * (blockDim.x >> 5);
  unsigned tot = 0, near = 0;
  for (int s = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); s < ns; s += W) {
    const int w = R.slice_w[s], base = R.slice_ptr[s] + lane;
    for (int k = 0; k < w; ++k) {
      const int j = s * 32 + lane < n ? R.col[base + k * kWarp] : -1;
      const int before = __shfl_up_sync(0xffffffffu, j, 1);
      if (lane == 0 || j < 0 || before < 0) continue;
      ++tot;
      near += abs(j - before) <= 2;
    }
  }
  tot = __reduce_add_sync(0xffffffffu, tot);
  near = __reduce_add_sync(0xffffffffu, near);
  if (lane == 0) {
    atomicAdd(&cnt[0], (unsigned long long)tot);
    atomicAdd(&cnt[1], (unsigned long long)near);
  }
}

// Loop control of a WHILE graph of Krylov iterations: one pass per
// iteration, on until every lane has stopped or the budget is spent.
__global__ void k_loop_ctl(cudaGraphConditionalHandle h, const int* __restrict__ n_active,
                           int* __restrict__ budget) {
  chain_enter();
  if (threadIdx.x == 0) {
    const int b = *budget - 1;
    *budget = b;
    cudaGraphSetConditional(h, (b > 0 && *n_active > 0) ? 1u : 0u);
  }
}

// Self-test of the recurrences' bounded wait: a two-cell slice whose second
// cell depends on the first one's value, which nothing ever writes, through
// the same driver (sweep_rows) as the sweeps, so the wait runs out after
// kSweepPolls polls and sets ctl->err.  R holds slice_ptr {0}, slice_w {1}
// and col {-1, 0}; never holds two pending values.
__global__ void k_sweep_selftest(Rows<double> R, const double* never, SweepCtl* ctl) {
  sweep_rows<false, false, 1, 1, int>(
      2, R, SweepMap{nullptr, nullptr, 1}, never, ctl, [](int) {}, [](int) { return 0; },
      [](int, const double (&)[1], double (&)[1]) {}, [](const double (&)[1]) {}, [](int) {});
}

}  // namespace sg
