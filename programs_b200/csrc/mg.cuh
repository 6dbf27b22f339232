// mg.cuh -- aggregation multigrid around the learned preconditioner.
//
// A preconditioner that acts on one row at a time (the network's operator
// M^-1 = D^-1/2 S (I + E) S D^-1/2 reaches one neighbour) cannot change how
// the CG iteration count grows with the mesh: smooth error spans the whole
// domain.  Here the network's operator is the smoother on the finest level
// of an aggregation hierarchy, and one symmetric V-cycle is the
// preconditioner of flexible CG:
//
//   level l+1 cells = aggregates of about 8 level-l cells (three passes of
//                     pairwise matching along the strongest coupling),
//   P_l            = piecewise-constant prolongation (cell -> its aggregate),
//   A_{l+1}        = P^T A_l P (Galerkin: coefficients of the faces between
//                     two aggregates summed, row sums summed),
//   V-cycle on b:  x = w K b;  t = b - A x;  x += a P V(P^T t);
//                  x += w K (b - A x),
//   K              = the network's operator on level 0 (or its diagonal
//                     S^2 D^-1 alone -- learned Jacobi weights, fused like
//                     Jacobi -- or D^-1), D^-1 below,
//   coarsest level = at most kCoarsest cells, solved with its dense inverse.
//
// With a symmetric positive definite K on level 0 and Jacobi below, the
// V-cycle is a symmetric linear operator; flexible CG tolerates it being
// indefinite in rare cases, and hands over to Jacobi-PCG if a step loses
// positive curvature.
//
// Every level keeps the fine level's layout: sliced ELL rows (32 cells per
// slice, slot-major), FP32 coefficients and the FP32 row sum in place of the
// diagonal, so the product is taken in difference form
// (A x)_i = rs_i x_i + sum_j a_ij (x_j - x_i) on every level.
//
// The aggregation (structure) is computed on the host once per matrix
// structure, from the coefficients present then; the coarse coefficients
// are recomputed on the device for every solve (gathers in a fixed order,
// FP64 sums, deterministic).
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <numeric>
#include <thread>
#include <vector>

#include "kernels.cuh"

namespace mg {

constexpr int kCoarsest = 256;   // dense inverse at or below this many cells
constexpr int kMaxLevels = 12;   // coarse levels at most

// ---- host: graphs and aggregation ---------------------------------------------
// Undirected graph in CSR with positive coupling strengths (|a_ij|).
struct Graph {
  int n = 0;
  std::vector<long long> ptr;  // n + 1
  std::vector<int> adj;
  std::vector<float> w;
};

// One pass of pairwise matching: each cell still free, in index order, is
// paired with its free neighbour of strongest coupling (ties: lowest index),
// or stays alone.  agg[i] = new index (numbered in order of creation, so
// locality of the input numbering is kept); returns the number of aggregates.
inline int match_pass(const Graph& g, std::vector<int>& agg) {
  agg.assign(g.n, -1);
  int nc = 0;
  for (int i = 0; i < g.n; ++i) {
    if (agg[i] >= 0) continue;
    int best = -1;
    float bw = 0.0f;
    for (long long k = g.ptr[i]; k < g.ptr[i + 1]; ++k) {
      const int j = g.adj[k];
      if (j == i || agg[j] >= 0) continue;
      if (g.w[k] > bw || (g.w[k] == bw && best >= 0 && j < best)) {
        bw = g.w[k];
        best = j;
      }
    }
    agg[i] = nc;
    if (best >= 0 && bw > 0.0f) agg[best] = nc;
    ++nc;
  }
  return nc;
}

// Members of each aggregate, in increasing cell index (counting sort).
inline void members(const std::vector<int>& agg, int nc, std::vector<int>& ptr,
                    std::vector<int>& cells) {
  ptr.assign(nc + 1, 0);
  for (int a : agg) ptr[a + 1]++;
  for (int k = 0; k < nc; ++k) ptr[k + 1] += ptr[k];
  cells.resize(agg.size());
  std::vector<int> pos(ptr.begin(), ptr.end() - 1);
  for (int i = 0; i < (int)agg.size(); ++i) cells[pos[agg[i]]++] = i;
}

// Run f(begin, end, thread) over [0, n) in contiguous chunks on up to 16
// host threads (one for small n).  Callers write disjoint outputs per index,
// so results do not depend on the number of threads.
template <typename F>
inline void parallel_rows(int n, F f) {
  const unsigned hc = std::thread::hardware_concurrency();
  int T = (int)std::max(1u, std::min(hc ? hc : 1u, 16u));
  if (n < 65536) T = 1;
  const int chunk = (n + T - 1) / T;
  std::vector<std::thread> th;
  for (int t = 1; t < T; ++t) {
    const int b = t * chunk, e = std::min(n, b + chunk);
    if (b < e) th.emplace_back(f, b, e, t);
  }
  f(0, std::min(n, chunk), 0);
  for (auto& x : th) x.join();
}

// Graph of the aggregates: strengths of the couplings between two
// aggregates summed (in member order, then row order), couplings inside an
// aggregate dropped; each row lists its neighbours in order of first
// appearance.
inline Graph coarsen(const Graph& g, const std::vector<int>& agg, int nc) {
  std::vector<int> mp, mc;
  members(agg, nc, mp, mc);
  Graph out;
  out.n = nc;
  out.ptr.assign(nc + 1, 0);
  const int T = 16;
  std::vector<std::vector<int>> tadj(T);
  std::vector<std::vector<float>> tw(T);
  std::vector<int> deg(nc, 0), first(T, 0);
  parallel_rows(nc, [&](int b, int e, int t) {
    std::vector<int> mark(nc, -1), pos(nc, 0);
    auto& A = tadj[t];
    auto& W = tw[t];
    first[t] = b;
    for (int I = b; I < e; ++I) {
      const size_t r0 = A.size();
      for (int m = mp[I]; m < mp[I + 1]; ++m) {
        const int i = mc[m];
        for (long long k = g.ptr[i]; k < g.ptr[i + 1]; ++k) {
          const int J = agg[g.adj[k]];
          if (J == I) continue;
          if (mark[J] != I) {
            mark[J] = I;
            pos[J] = (int)(A.size() - r0);
            A.push_back(J);
            W.push_back(g.w[k]);
          } else {
            W[r0 + pos[J]] += g.w[k];
          }
        }
      }
      deg[I] = (int)(A.size() - r0);
    }
  });
  for (int I = 0; I < nc; ++I) out.ptr[I + 1] = out.ptr[I] + deg[I];
  out.adj.resize(out.ptr[nc]);
  out.w.resize(out.ptr[nc]);
  for (int t = 0; t < T; ++t) {
    if (tadj[t].empty()) continue;
    std::copy(tadj[t].begin(), tadj[t].end(), out.adj.begin() + out.ptr[first[t]]);
    std::copy(tw[t].begin(), tw[t].end(), out.w.begin() + out.ptr[first[t]]);
  }
  return out;
}

// Aggregates of about 2^passes cells: passes of matching, composed.  A cell
// left alone by every pass (its neighbours were all taken before its turn)
// then joins the aggregate of its most strongly coupled neighbour: left
// alone, such cells carry over from level to level and, on the small
// levels, stall the coarsening.  Aggregates keep the order of their first
// member.
inline int aggregate(const Graph& g, int passes, std::vector<int>& agg) {
  agg.resize(g.n);
  std::iota(agg.begin(), agg.end(), 0);
  Graph cur;
  const Graph* gp = &g;
  int nc = g.n;
  for (int p = 0; p < passes; ++p) {
    std::vector<int> a;
    const int n2 = match_pass(*gp, a);
    for (int& x : agg) x = a[x];
    if (p + 1 < passes) {
      cur = coarsen(*gp, a, n2);
      gp = &cur;
    }
    nc = n2;
  }
  std::vector<int> size(nc, 0);
  for (int x : agg) size[x]++;
  for (int i = 0; i < g.n; ++i) {
    if (size[agg[i]] != 1) continue;
    int best = -1;
    float bw = 0.0f;
    for (long long k = g.ptr[i]; k < g.ptr[i + 1]; ++k) {
      const int j = g.adj[k];
      if (j != i && size[agg[j]] > 1 && g.w[k] > bw) {
        bw = g.w[k];
        best = j;
      }
    }
    if (best >= 0) {
      size[agg[i]] = 0;
      agg[i] = agg[best];
      size[agg[i]]++;
    }
  }
  std::vector<int> renum(nc, -1);
  int m = 0;
  for (int i = 0; i < g.n; ++i)
    if (renum[agg[i]] < 0) renum[agg[i]] = m++;
  for (int& x : agg) x = renum[x];
  return m;
}

// Sliced-ELL structure of one coarse level and, per coarse slot, the list of
// finer-level slots whose coefficients sum into it.
struct CoarseHost {
  int n = 0;
  std::vector<int> slice_ptr;
  std::vector<uint8_t> slice_w;
  std::vector<int> col;         // -1 = padding
  std::vector<int> gptr, gsrc;  // slot e sums finer slots gsrc[gptr[e] .. gptr[e+1])
  std::vector<int> agg_ptr, agg_cells, agg_of;
  long long n_slots = 0;
};

// Fine level given by its sliced-ELL arrays (n cells) and aggregation agg.
// Coarse row I lists its neighbours J in order of first appearance over
// I's members and their slots; slot (I, J) sums the finer slots listed for
// it, in the same order.
inline bool build_coarse(int n, const std::vector<int>& sp, const std::vector<uint8_t>& sw,
                         const std::vector<int>& col, const std::vector<int>& agg, int nc,
                         CoarseHost& C) {
  C.n = nc;
  C.agg_of = agg;
  members(agg, nc, C.agg_ptr, C.agg_cells);
  const std::vector<int>& mp = C.agg_ptr;
  const std::vector<int>& mc = C.agg_cells;
  // walk the finer slots of coarse row I: visit(J, finer slot, k of J)
  auto walk = [&](int I, std::vector<int>& mark, std::vector<int>& pos, auto&& visit) {
    int d = 0;
    for (int m = mp[I]; m < mp[I + 1]; ++m) {
      const int i = mc[m];
      const int s = i >> 5, l = i & 31;
      for (int k = 0; k < sw[s]; ++k) {
        const long long e = (long long)sp[s] + (long long)k * 32 + l;
        const int j = col[e];
        if (j < 0) continue;
        const int J = agg[j];
        if (J == I) continue;
        if (mark[J] != I) {
          mark[J] = I;
          pos[J] = d++;
        }
        visit(J, (int)e, pos[J]);
      }
    }
    return d;
  };
  std::vector<int> deg(nc, 0);
  parallel_rows(nc, [&](int b, int e, int) {
    std::vector<int> mark(nc, -1), pos(nc, 0);
    for (int I = b; I < e; ++I) deg[I] = walk(I, mark, pos, [](int, int, int) {});
  });
  const int ns = (nc + 31) / 32;
  C.slice_ptr.assign(ns + 1, 0);
  C.slice_w.assign(ns, 0);
  long long total = 0;
  for (int s = 0; s < ns; ++s) {
    int w = 0;
    for (int l = 0; l < 32; ++l)
      if (s * 32 + l < nc) w = std::max(w, deg[s * 32 + l]);
    if (w > 255) return false;
    C.slice_w[s] = (uint8_t)w;
    C.slice_ptr[s] = (int)total;
    total += 32LL * w;
    if (total > (1LL << 31) - 1) return false;
  }
  C.slice_ptr[ns] = (int)total;
  C.n_slots = total;
  C.col.assign(total, -1);
  std::vector<int> cnt(total, 0);
  parallel_rows(nc, [&](int b, int e, int) {
    std::vector<int> mark(nc, -1), pos(nc, 0);
    for (int I = b; I < e; ++I) {
      const long long base = (long long)C.slice_ptr[I >> 5] + (I & 31);
      walk(I, mark, pos, [&](int J, int, int k) {
        C.col[base + (long long)k * 32] = J;
        cnt[base + (long long)k * 32]++;
      });
    }
  });
  C.gptr.assign(total + 1, 0);
  for (long long e = 0; e < total; ++e) C.gptr[e + 1] = C.gptr[e] + cnt[e];
  C.gsrc.assign(C.gptr[total], 0);
  parallel_rows(nc, [&](int b, int e, int) {
    std::vector<int> mark(nc, -1), pos(nc, 0);
    for (int I = b; I < e; ++I) {
      const long long base = (long long)C.slice_ptr[I >> 5] + (I & 31);
      std::vector<int> fill;
      walk(I, mark, pos, [&](int, int ef, int k) {
        if ((int)fill.size() <= k) fill.resize(k + 1, 0);
        const long long ec = base + (long long)k * 32;
        C.gsrc[C.gptr[ec] + fill[k]++] = ef;
      });
    }
  });
  (void)n;
  return true;
}

// Coupling graph of a level given by its sliced-ELL arrays and coefficients.
inline Graph graph_of(int n, const std::vector<int>& sp, const std::vector<uint8_t>& sw,
                      const std::vector<int>& col, const std::vector<float>& val) {
  Graph g;
  g.n = n;
  g.ptr.assign(n + 1, 0);
  std::vector<int> deg(n, 0);
  parallel_rows(n, [&](int b, int e, int) {
    for (int i = b; i < e; ++i) {
      const int s = i >> 5, l = i & 31;
      int d = 0;
      for (int k = 0; k < sw[s]; ++k) d += col[(long long)sp[s] + (long long)k * 32 + l] >= 0;
      deg[i] = d;
    }
  });
  for (int i = 0; i < n; ++i) g.ptr[i + 1] = g.ptr[i] + deg[i];
  g.adj.resize(g.ptr[n]);
  g.w.resize(g.ptr[n]);
  parallel_rows(n, [&](int b, int e, int) {
    for (int i = b; i < e; ++i) {
      const int s = i >> 5, l = i & 31;
      long long o = g.ptr[i];
      for (int k = 0; k < sw[s]; ++k) {
        const long long q = (long long)sp[s] + (long long)k * 32 + l;
        if (col[q] >= 0) {
          g.adj[o] = col[q];
          g.w[o++] = std::fabs(val[q]);
        }
      }
    }
  });
  return g;
}

// ---- device: coefficients of the coarse levels ---------------------------------
// v[e] = sum of the finer coefficients listed for slot e (FP64 sum, in list order).
__global__ void k_mg_gather_slots(long long ns, const int* __restrict__ gptr,
                                  const int* __restrict__ gsrc, const float* __restrict__ vf,
                                  float* __restrict__ v) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < ns;
       e += (long long)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int k = gptr[e]; k < gptr[e + 1]; ++k) s += (double)vf[gsrc[k]];
    v[e] = (float)s;
  }
}

// rs[I] = sum of the finer row sums of I's members (the Galerkin row sum).
__global__ void k_mg_rowsum(int nc, const int* __restrict__ aptr, const int* __restrict__ acell,
                            const float* __restrict__ rsf, float* __restrict__ rs) {
  for (int I = blockIdx.x * blockDim.x + threadIdx.x; I < nc; I += gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int m = aptr[I]; m < aptr[I + 1]; ++m) s += (double)rsf[acell[m]];
    rs[I] = (float)s;
  }
}

// dinv = 1 / (rs - sum_j a_ij): the inverse diagonal (0 where it is not > 0).
__global__ void k_mg_dinv(int n, sg::Rows<float> R, float* __restrict__ dinv) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    sg::RowIt<float> it(R, i);
    double d = R.diag[i];
    for (int k = 0; k < it.w; ++k) {
      const int e = it.base + k * sg::kWarp;
      if (R.col[e] >= 0) d -= (double)R.val[e];
    }
    dinv[i] = d > 0.0 ? (float)(1.0 / d) : 0.0f;
  }
}

// Dense FP64 copy of the coarsest matrix (row-major n x n, zeroed before).
__global__ void k_mg_dense(int n, sg::Rows<float> R, double* __restrict__ A) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    sg::RowIt<float> it(R, i);
    double d = R.diag[i];
    for (int k = 0; k < it.w; ++k) {
      const int e = it.base + k * sg::kWarp;
      const int j = R.col[e];
      if (j >= 0) {
        A[(size_t)i * n + j] += (double)R.val[e];
        d -= (double)R.val[e];
      }
    }
    A[(size_t)i * n + i] += d;
  }
}

// Gauss-Jordan inverse of the symmetric positive definite coarsest matrix
// (no pivoting needed); a pivot below 1e-13 of the largest diagonal (a
// singular, all-Neumann system) drops that row and column, which leaves a
// generalised inverse.  Result rounded to FP32.
// The n steps are a serial chain, so what counts is the step: the matrix
// stays in registers of CS blocks (one, or a cluster of 8 above 128 cells) --
// a thread owns one column of kInvRows consecutive rows -- and a step is the
// pivot row, shared by its owner, the pivot column, shared by each block for
// its own rows, one barrier, and kInvRows updates.  Through global memory in
// one block the step swept n^2 entries through L2 (252 us at n = 67, 3.77 ms
// at n = 242, a tenth of a 160^3 solve).
constexpr int kInvRows = 16;
template <int COLS, int CS>
__global__ void __launch_bounds__(CS == 1 ? 1024 : 512)
k_mg_invert(int n, const double* __restrict__ A, float* __restrict__ Ainv) {
  namespace cg = cooperative_groups;
  constexpr int NT = CS == 1 ? 1024 : 512, GRP = NT / COLS;  // row groups in this block
  static_assert(CS * GRP * kInvRows >= COLS, "every row has an owner");
  __shared__ double row_s[2][COLS + 1];                // the pivot row and 1 / pivot, in its owner's block
  __shared__ double col_s[2][GRP][kInvRows];           // the pivot column of this block's rows
  __shared__ double dmax_s;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = CS == 1 ? 0 : (int)cl.block_rank();
  const int j = threadIdx.x % COLS, g = threadIdx.x / COLS;
  const int i0 = (rank * GRP + g) * kInvRows;  // this thread's rows i0 .. i0 + kInvRows
  double a[kInvRows];
#pragma unroll
  for (int r = 0; r < kInvRows; ++r)
    a[r] = i0 + r < n && j < n ? A[(size_t)(i0 + r) * n + j] : 0.0;
  if (threadIdx.x < 32) {
    double m = 0.0;
    for (int i = threadIdx.x; i < n; i += 32) m = fmax(m, fabs(A[(size_t)i * n + i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (threadIdx.x == 0) dmax_s = m;
  }
  __syncthreads();
  const double dmax = dmax_s;
  for (int k0 = 0; k0 < n; k0 += kInvRows) {
    const int owner = k0 / kInvRows / GRP;
    const bool mine = i0 == k0;  // the pivot rows of this round are this group's
#pragma unroll
    for (int kk = 0; kk < kInvRows; ++kk) {
      const int k = k0 + kk, par = kk & 1;  // buffers alternate: kInvRows is even
      if (k < n) {
        if (mine) row_s[par][j] = a[kk];
        if (mine && j == k) row_s[par][COLS] = 1.0 / a[kk];
        if (j == k) {
#pragma unroll
          for (int r = 0; r < kInvRows; ++r) col_s[par][g][r] = a[r];
        }
        if (CS == 1) __syncthreads();
        else cl.sync();
        const double* rs = CS == 1 ? row_s[par] : cl.map_shared_rank(&row_s[par][0], owner);
        const double piv = rs[k], rj = rs[j], ip = rs[COLS];
        if (!(fabs(piv) > 1e-13 * dmax)) {
#pragma unroll
          for (int r = 0; r < kInvRows; ++r)
            if (j == k || i0 + r == k) a[r] = 0.0;
        } else {
          const double pr = j == k ? ip : rj * ip;
#pragma unroll
          for (int r = 0; r < kInvRows; ++r) {
            const double f = col_s[par][g][r];
            const double v = (j == k ? 0.0 : a[r]) - f * pr;
            a[r] = i0 + r == k ? pr : v;
          }
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < kInvRows; ++r)
    if (i0 + r < n && j < n) Ainv[(size_t)(i0 + r) * n + j] = (float)a[r];
  if (CS > 1) cl.sync();  // no block leaves while others may still read its pivot row
}

// ---- device: the V-cycle ---------------------------------------------------------
// x = w D^-1 b and t = b - A x (pre-smoothing from zero, then its residual;
// x_j at the neighbours is recomputed from b_j).
template <int CH = sg::kRowChunk>
__global__ void k_mg_pre(int n, sg::Rows<float> R, const float* __restrict__ dinv, float w,
                         const float* __restrict__ b, float* __restrict__ x,
                         float* __restrict__ t, const int* __restrict__ n_active) {
  sg::chain_enter();
  if (n_active && *n_active == 0) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    sg::RowIt<float> it(R, i);
    const float bi = b[i];
    const float xi = w * dinv[i] * bi;
    float y = R.diag[i] * xi;
    for (int k0 = 0; k0 < it.w; k0 += CH) {
      int j[CH];
      float a[CH], xj[CH];
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        j[u] = -1;
        a[u] = 0.0f;
        if (k0 + u < it.w) {
          const int e = it.base + (k0 + u) * sg::kWarp;
          j[u] = __ldg(&R.col[e]);
          a[u] = R.val[e];
        }
      }
#pragma unroll
      for (int u = 0; u < CH; ++u) xj[u] = j[u] >= 0 ? w * dinv[j[u]] * b[j[u]] : xi;
#pragma unroll
      for (int u = 0; u < CH; ++u)
        if (j[u] >= 0) y = fmaf(a[u], xj[u] - xi, y);
    }
    x[i] = xi;
    t[i] = bi - y;
  }
}

// The coarse levels' rows hold 17-27 slots, and from the second level on
// there are too few rows to fill the SMs with one thread each, so G lanes
// share a row: lane = part * (32/G) + row, so a load still reads 32/G
// consecutive words per slot.  Returns y + sum_j a_ij (x(j) - xi) in every
// lane.  ORD keeps the sum slot by slot (values by shuffle), as in row_apply:
// the training's loss gradient, a difference of nearly equal terms, moves by
// 2e-5 when the V-cycle's rounding does, so its V-cycle keeps the order the
// network was trained with; a solve takes the lanes' partial sums (V-cycle
// at 64^3 86 us, ordered 101).
template <int G, bool ORD, typename X>
__device__ __forceinline__ float row_diff(const sg::Rows<float>& R, int i, int part, float xi,
                                          float y0, X&& x) {
  constexpr int CH = 4, RW = 32 / G;
  sg::RowIt<float> it(R, i);
  const int rl = (threadIdx.x & 31) % RW;
  float y = ORD ? y0 : 0.0f;
  for (int k0 = 0; k0 < it.w; k0 += CH * G) {  // w is the slice's, the same for the whole warp
    int j[CH];
    float a[CH], dx[CH];
#pragma unroll
    for (int u = 0; u < CH; ++u) {
      j[u] = -1;
      a[u] = 0.0f;
      if (k0 + u * G + part < it.w) {
        const int e = it.base + (k0 + u * G + part) * sg::kWarp;
        j[u] = __ldg(&R.col[e]);
        a[u] = __ldg(&R.val[e]);
      }
    }
#pragma unroll
    for (int u = 0; u < CH; ++u) dx[u] = (j[u] >= 0 ? x(j[u]) : xi) - xi;
#pragma unroll
    for (int u = 0; u < CH; ++u) {
      if (!ORD) {
        if (j[u] >= 0) y = fmaf(a[u], dx[u], y);
        continue;
      }
      if (k0 + u * G >= it.w) break;
      const float v = j[u] >= 0 ? a[u] : 0.0f;
#pragma unroll
      for (int q = 0; q < G; ++q)  // padding and slots past w add 0
        y = fmaf(__shfl_sync(0xffffffffu, v, q * RW + rl),
                 __shfl_sync(0xffffffffu, dx[u], q * RW + rl), y);
    }
  }
  if (!ORD) {
#pragma unroll
    for (int o = 16; o >= RW; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
    y = y0 + y;
  }
  return y;
}

// Calls f(row, part, store) for every row of n, G lanes a row (whole warps at
// a time; rows past n repeat the last one with store off).
template <int G, typename F>
__device__ __forceinline__ void rows_by_group(int n, int thread, int n_threads, F&& f) {
  constexpr int RW = 32 / G;  // rows a warp
  const int lane = thread & 31, part = lane / RW, rl = lane % RW;
  for (int i0 = (thread >> 5) * RW; i0 < n; i0 += (n_threads >> 5) * RW)
    f(min(i0 + rl, n - 1), part, part == 0 && i0 + rl < n);
}

// pre- and post-smoothing (k_mg_pre, k_mg_post) of a coarse level of at most
// kCoarseCells rows, 4 lanes a row.
constexpr int kCoarseLanes = 4;
constexpr int kCoarseCells = 100000;
template <bool ORD>
__global__ void k_mg_pre_coarse(int n, sg::Rows<float> R, const float* __restrict__ dinv, float w,
                                const float* __restrict__ b, float* __restrict__ x,
                                float* __restrict__ t, const int* __restrict__ n_active) {
  sg::chain_enter();
  if (n_active && *n_active == 0) return;
  rows_by_group<kCoarseLanes>(
      n, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x,
      [&](int i, int part, bool store) {
        const float bi = b[i], xi = w * dinv[i] * bi;
        const float y = row_diff<kCoarseLanes, ORD>(R, i, part, xi, R.diag[i] * xi,
                                               [&](int j) { return w * dinv[j] * b[j]; });
        if (store) {
          x[i] = xi;
          t[i] = bi - y;
        }
      });
}
template <bool ORD>
__global__ void k_mg_post_coarse(int n, sg::Rows<float> R, const float* __restrict__ dinv, float w,
                                 const float* __restrict__ b, const float* __restrict__ x,
                                 float* __restrict__ y, const int* __restrict__ n_active) {
  sg::chain_enter();
  if (n_active && *n_active == 0) return;
  rows_by_group<kCoarseLanes>(
      n, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x,
      [&](int i, int part, bool store) {
        const float xi = x[i];
        const float ax = row_diff<kCoarseLanes, ORD>(R, i, part, xi, R.diag[i] * xi,
                                                [&](int j) { return x[j]; });
        if (store) y[i] = xi + w * dinv[i] * (b[i] - ax);
      });
}

// The V-cycle's bottom in one launch: from the finer level's residual t to
// the correction y of level 0 here (the first of at most kFuseCells cells),
// one thread-block cluster over all the levels below.  As a kernel per step
// these levels are four dependent launches each on a few hundred to a few
// thousand rows, 5-12 us apiece; here a step ends with a cluster barrier
// (0.4-0.7 us with its stores).  More lanes share a row the fewer rows there
// are.  The vectors pass between the blocks through L2 (loads that skip L1).
// A whole V-cycle, before / after, us: 32^3 67 / 53, 64^3 99 / 86, 100^3
// 182 / 153, 160^3 413 / 386, 200^3 666 / 634; with levels of up to 16k cells
// in here, more than 16 SMs are good for, 160^3 took 420.
struct FuseLevel {
  int n;
  sg::Rows<float> R;
  const float* dinv;
  const int *agg_ptr, *agg_cells, *agg_of;  // members on the finer level; finer cell -> cell
  float *x, *b, *t, *y;
};
struct FuseArgs {
  int n_level;
  FuseLevel lv[kMaxLevels];
  const float* t_fine;  // residual of the level above lv[0]
  const float* ainv;    // dense inverse of the last level
};
constexpr int kFuseCells = 6000;
constexpr int kFuseThreads = 1024;
constexpr int kFuseCluster = 16;

template <int G, bool ORD>
__device__ __forceinline__ void fuse_pre(const FuseLevel& L, float w, int t, int nt) {
  rows_by_group<G>(L.n, t, nt, [&](int i, int part, bool store) {
    const float bi = __ldcg(&L.b[i]), xi = w * __ldg(&L.dinv[i]) * bi;
    const float y = row_diff<G, ORD>(L.R, i, part, xi, __ldg(&L.R.diag[i]) * xi, [&](int j) {
      return w * __ldg(&L.dinv[j]) * __ldcg(&L.b[j]);
    });
    if (store) {
      __stcg(&L.x[i], xi);
      __stcg(&L.t[i], bi - y);
    }
  });
}
template <int G, bool ORD>
__device__ __forceinline__ void fuse_post(const FuseLevel& L, float w, int t, int nt) {
  rows_by_group<G>(L.n, t, nt, [&](int i, int part, bool store) {
    const float xi = __ldcg(&L.x[i]);
    const float ax = row_diff<G, ORD>(L.R, i, part, xi, __ldg(&L.R.diag[i]) * xi,
                                 [&](int j) { return __ldcg(&L.x[j]); });
    if (store) __stcg(&L.y[i], xi + w * __ldg(&L.dinv[i]) * (__ldcg(&L.b[i]) - ax));
  });
}

template <bool ORD>
__global__ void __launch_bounds__(kFuseThreads) k_mg_bottom(FuseArgs A, float w, float alpha,
                                                            const int* __restrict__ n_active) {
  sg::chain_enter();
  if (n_active && *n_active == 0) return;  // the same for every block
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  __shared__ float sb[kCoarsest];
  const int nt = (int)cl.num_blocks() * kFuseThreads;
  const int t = (int)cl.block_rank() * kFuseThreads + threadIdx.x;
  const int last = A.n_level - 1;
  for (int l = 0; l <= last; ++l) {
    const FuseLevel& L = A.lv[l];
    const float* tf = l == 0 ? A.t_fine : A.lv[l - 1].t;
    for (int I = t; I < L.n; I += nt) {  // restriction, members in list order
      float s = 0.0f;
      for (int m = __ldg(&L.agg_ptr[I]); m < __ldg(&L.agg_ptr[I + 1]); ++m)
        s += __ldcg(&tf[__ldg(&L.agg_cells[m])]);
      __stcg(&L.b[I], s);
    }
    cl.sync();
    if (l == last) break;
    if (L.n * 2 > nt) fuse_pre<2, ORD>(L, w, t, nt);
    else if (L.n * 8 > nt) fuse_pre<8, ORD>(L, w, t, nt);
    else fuse_pre<16, ORD>(L, w, t, nt);
    cl.sync();
  }
  {  // x = Ainv b, a warp a row
    const FuseLevel& L = A.lv[last];
    for (int i = threadIdx.x; i < L.n; i += kFuseThreads) sb[i] = __ldcg(&L.b[i]);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int i = t >> 5; i < L.n; i += nt >> 5) {
      float s = 0.0f;
      for (int j0 = 0; j0 < L.n; j0 += 32) {
        const float a = j0 + lane < L.n ? __ldg(&A.ainv[(size_t)i * L.n + j0 + lane]) : 0.0f;
        if (!ORD) {
          if (j0 + lane < L.n) s = fmaf(a, sb[j0 + lane], s);
          continue;
        }
#pragma unroll
        for (int q = 0; q < 32; ++q)
          if (j0 + q < L.n) s = fmaf(__shfl_sync(0xffffffffu, a, q), sb[j0 + q], s);
      }
      if (!ORD) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      }
      if (lane == 0) __stcg(&L.y[i], s);
    }
  }
  for (int l = last - 1; l >= 0; --l) {
    const FuseLevel& L = A.lv[l];
    const FuseLevel& C = A.lv[l + 1];
    cl.sync();
    for (int i = t; i < L.n; i += nt)
      __stcg(&L.x[i], __ldcg(&L.x[i]) + alpha * __ldcg(&C.y[__ldg(&C.agg_of[i])]));
    cl.sync();
    if (L.n * 2 > nt) fuse_post<2, ORD>(L, w, t, nt);
    else if (L.n * 8 > nt) fuse_post<8, ORD>(L, w, t, nt);
    else fuse_post<16, ORD>(L, w, t, nt);
  }
}

// t = b - A x
template <int CH = sg::kRowChunk>
__global__ void k_mg_resid(int n, sg::Rows<float> R, const float* __restrict__ b,
                           const float* __restrict__ x, float* __restrict__ t,
                           const int* __restrict__ n_active) {
  sg::chain_enter();
  if (n_active && *n_active == 0) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    float y[1];
    sg::row_apply<float, 1, CH>(R, i, x, y);
    t[i] = b[i] - y[0];
  }
}

// y = x + w D^-1 (b - A x)  (post-smoothing; y and x are different arrays)
template <typename TO, int CH = sg::kRowChunk>
__global__ void k_mg_post(int n, sg::Rows<float> R, const float* __restrict__ dinv, float w,
                          const float* __restrict__ b, const float* __restrict__ x,
                          TO* __restrict__ y, const int* __restrict__ n_active) {
  sg::chain_enter();
  if (n_active && *n_active == 0) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    float ax[1];
    sg::row_apply<float, 1, CH>(R, i, x, ax);
    y[i] = (TO)(x[i] + w * dinv[i] * (b[i] - ax[0]));
  }
}

// The network's operator as smoother: out = [out +] w K in,
// K in = q (q in + E (q in)) (the learned preconditioner's application).
template <bool ADD, typename TO>
__global__ void k_mg_net(int n, sg::Rows<float> R, const float* __restrict__ gE,
                         const float* __restrict__ q, float w, const float* __restrict__ in,
                         const float* __restrict__ base, TO* __restrict__ out,
                         const int* __restrict__ n_active) {
  sg::chain_enter();
  if (n_active && *n_active == 0) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    sg::RowIt<float> it(R, i);
    const float qi = q[i];
    float t = qi * in[i];
    for (int k0 = 0; k0 < it.w; k0 += sg::kRowChunk) {
      int j[sg::kRowChunk];
      float g[sg::kRowChunk], qj[sg::kRowChunk], vj[sg::kRowChunk];
#pragma unroll
      for (int u = 0; u < sg::kRowChunk; ++u) {
        j[u] = -1;
        g[u] = 0.0f;
        if (k0 + u < it.w) {
          const int e = it.base + (k0 + u) * sg::kWarp;
          j[u] = __ldg(&R.col[e]);
          g[u] = gE[e];
        }
      }
#pragma unroll
      for (int u = 0; u < sg::kRowChunk; ++u) {
        qj[u] = j[u] >= 0 ? q[j[u]] : 0.0f;
        vj[u] = j[u] >= 0 ? in[j[u]] : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < sg::kRowChunk; ++u)
        if (j[u] >= 0) t = fmaf(g[u] * qj[u], vj[u], t);
    }
    const float v = w * qi * t;
    out[i] = (TO)(ADD ? base[i] + v : v);
  }
}

// The last kernel of a V-cycle inside flexible CG: z = x + w K t (NET, as
// k_mg_net<true>) or z = x + w D^-1 (b - A x) (as k_mg_post), and beta =
// -(z.q)/(p.q) with it, on the reduction grid -- k_fcg_beta's pass over z and
// q and its reduction tail in a kernel of their own were 7.6 us of a 64^3
// iteration.  in: t, or b; dq: q, or D^-1.
template <bool NET, int CH>
__global__ void SG_BOUNDS(1) k_mg_last(sg::SegMap sm, sg::Rows<float> R, const float* __restrict__ gE,
                          const float* __restrict__ dq, float w, const float* __restrict__ in,
                          const float* __restrict__ x, float* __restrict__ z,
                          const float* __restrict__ qv, double* __restrict__ part,
                          sg::Lane* __restrict__ lanes) {
  sg::chain_enter();
  const int b = blockIdx.x, s = sm.blk_seg[b];
  if (!lanes[s].active) return;
  const int c0 = sm.seg_c0[s], c1 = sm.seg_c1[s];
  const int stride = sm.seg_nblk[s] * blockDim.x;
  double acc[1] = {0.0};
  for (int i = c0 + sm.blk_rank[b] * blockDim.x + threadIdx.x; i < c1; i += stride) {
    float zi;
    if (NET) {
      sg::RowIt<float> it(R, i);
      const float qi = dq[i];
      float t = qi * in[i];
      for (int k0 = 0; k0 < it.w; k0 += CH) {
        int j[CH];
        float g[CH], vj[CH];
#pragma unroll
        for (int u = 0; u < CH; ++u) {
          j[u] = -1;
          g[u] = 0.0f;
          if (k0 + u < it.w) {
            const int e = it.base + (k0 + u) * sg::kWarp;
            j[u] = __ldg(&R.col[e]);
            g[u] = gE[e];
          }
        }
#pragma unroll
        for (int u = 0; u < CH; ++u) {
          if (j[u] >= 0) g[u] *= dq[j[u]];
          vj[u] = j[u] >= 0 ? in[j[u]] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < CH; ++u)
          if (j[u] >= 0) t = fmaf(g[u], vj[u], t);
      }
      zi = x[i] + w * qi * t;
    } else {
      float ax[1];
      sg::row_apply<float, 1, CH>(R, i, x, ax);
      zi = x[i] + w * dq[i] * (in[i] - ax[0]);
    }
    z[i] = zi;
    acc[0] += sg::prod(zi, qv[i]);
  }
  double tot[1];
  if (sg::seg_commit<1>(sm, b, s, part, acc, tot) && threadIdx.x == 0)
    lanes[s].beta = sg::flex_beta(lanes[s], tot[0], c1 - c0);
}

// ---- device: bounding the network smoother -----------------------------------------
// v_i = a fixed pseudo-random value in [-1, 1) (power-iteration start)
__global__ void k_mg_hashfill(int n, float* __restrict__ v) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    unsigned int h = (unsigned int)i * 2654435761u + 0x9e3779b9u;
    h ^= h >> 16;
    h *= 0x85ebca6bu;
    h ^= h >> 13;
    v[i] = (float)(h & 0xFFFFFF) * (2.0f / 16777216.0f) - 1.0f;
  }
}

// out += x.x (FP64, one atomic per block)
__global__ void __launch_bounds__(256) k_mg_norm2(int n, const float* __restrict__ x,
                                                  double* __restrict__ out) {
  __shared__ double sh[8];
  double acc = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    acc += (double)x[i] * x[i];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += sh[k];
    atomicAdd(out, t);
  }
}

// One step of the power iteration for lambda_max(w K A): v = (w / |v|) K y,
// y = A v taken before, |v|^2 = norm2[0], the new |v|^2 added to norm2[1]
// (zeroed before).  The norms stay on the device until the last step: the
// scaling and the norm as passes of their own, with the host reading each
// norm, were 250 us of a 64^3 solve.
__global__ void __launch_bounds__(256)
k_mg_power(int n, sg::Rows<float> R, const float* __restrict__ gE, const float* __restrict__ q,
           float w, const float* __restrict__ y, float* __restrict__ v,
           double* __restrict__ norm2) {
  __shared__ double sh[8];
  const float f = (float)(1.0 / sqrt(norm2[0]));
  double acc = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    sg::RowIt<float> it(R, i);
    const float qi = q[i];
    float t = qi * y[i];
    for (int k0 = 0; k0 < it.w; k0 += sg::kRowChunk) {
      int j[sg::kRowChunk];
      float g[sg::kRowChunk], yj[sg::kRowChunk];
#pragma unroll
      for (int u = 0; u < sg::kRowChunk; ++u) {
        j[u] = -1;
        g[u] = 0.0f;
        if (k0 + u < it.w) {
          const int e = it.base + (k0 + u) * sg::kWarp;
          j[u] = __ldg(&R.col[e]);
          g[u] = gE[e];
        }
      }
#pragma unroll
      for (int u = 0; u < sg::kRowChunk; ++u) {
        if (j[u] >= 0) g[u] *= q[j[u]];
        yj[u] = j[u] >= 0 ? y[j[u]] : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < sg::kRowChunk; ++u)
        if (j[u] >= 0) t = fmaf(g[u], yj[u], t);
    }
    const float x = f * (w * qi * t);
    v[i] = x;
    acc += (double)x * x;
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) s += sh[k];
    atomicAdd(&norm2[1], s);
  }
}

// q_i = max(q_i, f rsd_i): the network's per-cell scale s = q / rsd held at
// or above f, so no cell is left (almost) unsmoothed.  A NaN stays NaN: a
// broken network must reach flexible CG's hand-over to plain PCG, not be
// quietly repaired here.
__global__ void k_mg_floor(int n, float f, const float* __restrict__ rsd, float* __restrict__ q) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float lo = f * rsd[i];
    if (q[i] < lo) q[i] = lo;
  }
}

// x *= c
__global__ void k_mg_scale(int n, float c, float* __restrict__ x) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    x[i] *= c;
}

// dq = q^2: the network's per-cell scale as a Jacobi weight (smoother 2)
__global__ void k_mg_square(int n, const float* __restrict__ q, float* __restrict__ dq) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    dq[i] = q[i] * q[i];
}

// bc[I] = sum of t over I's members (restriction P^T)
__global__ void k_mg_restrict(int nc, const int* __restrict__ aptr,
                              const int* __restrict__ acell, const float* __restrict__ t,
                              float* __restrict__ bc, const int* __restrict__ n_active) {
  sg::chain_enter();
  if (n_active && *n_active == 0) return;
  for (int I = blockIdx.x * blockDim.x + threadIdx.x; I < nc; I += gridDim.x * blockDim.x) {
    float s = 0.0f;
    for (int m = aptr[I]; m < aptr[I + 1]; ++m) s += t[acell[m]];
    bc[I] = s;
  }
}

// x[i] += a xc[agg_of[i]]  (prolongation P, scaled)
__global__ void k_mg_prolong(int n, const int* __restrict__ agg_of, float a,
                             const float* __restrict__ xc, float* __restrict__ x,
                             const int* __restrict__ n_active) {
  sg::chain_enter();
  if (n_active && *n_active == 0) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    x[i] += a * xc[agg_of[i]];
}

// ---- device: training the network through the V-cycle ----------------------------
// Loss per sample b (original space, z = V(b)): L = -log((z.b)^2 / (z.A z)).
// (z.b)^2/(z.Az) is twice the energy one CG step along z removes -- free of
// z's overall scale; the logarithm makes every sample count alike whatever
// its own energy, which varies by orders of magnitude between smooth and
// rough residuals.

// b = r / gs (the sample at unit mean scaled magnitude; gs in lane 0)
__global__ void k_mg_normalise(int n, const float* __restrict__ r, const sg::Lane* __restrict__ lanes,
                               float* __restrict__ b) {
  const double gs = lanes[0].gs > 0 ? lanes[0].gs : 1.0;
  const float inv = (float)(1.0 / gs);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    b[i] = r[i] * inv;
}

// az = A z; sums[0] += z.b, sums[1] += z.az (FP64; one atomic per block)
__global__ void __launch_bounds__(256)
k_mg_loss_sums(int n, sg::Rows<float> R, const float* __restrict__ z, const float* __restrict__ b,
               float* __restrict__ az, double* __restrict__ sums) {
  __shared__ double sh[2][8];
  double zb = 0.0, zaz = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    float y[1];
    sg::row_apply<float, 1>(R, i, z, y);
    az[i] = y[0];
    zb += (double)z[i] * b[i];
    zaz += (double)z[i] * y[0];
  }
  for (int o = 16; o > 0; o >>= 1) {
    zb += __shfl_down_sync(0xffffffffu, zb, o);
    zaz += __shfl_down_sync(0xffffffffu, zaz, o);
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) { sh[0][w] = zb; sh[1][w] = zaz; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, c = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) { a += sh[0][k]; c += sh[1][k]; }
    atomicAdd(&sums[0], a);
    atomicAdd(&sums[1], c);
  }
}

// g = dL/dz = 2 (A z / (z.Az) - b / (z.b)); jsum += L (once)
__global__ void k_mg_loss_grad(int n, const float* __restrict__ az, const float* __restrict__ b,
                               const double* __restrict__ sums, float* __restrict__ g,
                               double* __restrict__ jsum) {
  const double zb = sums[0], zaz = sums[1];
  // a sample whose z is (numerically) orthogonal to b or not finite has no
  // usable gradient (2/z.b explodes): it is skipped
  const bool ok = zaz > 0.0 && isfinite(zaz) && isfinite(zb) && zb * zb > 1e-20 * zaz;
  const float ca = ok ? (float)(2.0 / zaz) : 0.0f, cb = ok ? (float)(2.0 / zb) : 0.0f;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    g[i] = ca * az[i] - cb * b[i];
  if (blockIdx.x == 0 && threadIdx.x == 0 && ok) *jsum += -log(zb * zb / zaz);
}

// One application x -> w K x of the smoother, K = D^-1/2 S (I+E) S D^-1/2,
// seen from the scaled-space backward kernels: input u = rsd x and output
// gradient gh = w rsd g (g the gradient with respect to w K x).
__global__ void k_mg_scaled_pair(int n, const float* __restrict__ rsd, float w,
                                 const float* __restrict__ x, const float* __restrict__ g,
                                 float* __restrict__ u, float* __restrict__ gh) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    u[i] = rsd[i] * x[i];
    gh[i] = w * rsd[i] * g[i];
  }
}

}  // namespace mg
