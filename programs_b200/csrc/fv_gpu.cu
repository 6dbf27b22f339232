// fv_gpu.cu -- the SIMPLE outer-loop pieces on the GPU (include/fv_gpu.h).
//
// The reference assembles the momentum and pressure-correction matrices,
// the Green-Gauss gradients and the corrections in face loops over
// ng(:)%{ip,in} (cfd_setup.f90:178-431, 473-518, 604-646, 765-866).  A face
// loop scatters into both of its cells; on the GPU the face terms are
// computed one thread per face, and each cell then gathers its faces in
// ascending face order (a cell -> face list built once), which is the order
// the face loop adds them in -- so the sums, and every output, are bit-for-
// bit the host restatement's in fvmesh.cpp.  All double arithmetic below is
// written with explicit round-to-nearest operations (no fused multiply-add),
// as a compiler without FMA contraction evaluates the host code.
#include <cuda_runtime.h>

#include <algorithm>
#include <new>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/fv_gpu.h"
#include "../../include/solv_gpu.h"

namespace {

__device__ __forceinline__ double dm(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double da(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double ds(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dd(double a, double b) { return __ddiv_rn(a, b); }
// w a_N + (1 - w) a_P: linear interpolation to the face
__device__ __forceinline__ double lerp(double w, double an, double ap) {
  return da(dm(w, an), dm(ds(1.0, w), ap));
}

// What bounds the cell kernels is the number of gather requests L1 can take
// (60-77% of its throughput at 80^3, DRAM at 30%), so everything gathered
// stands in aligned 32-byte records and moves in 256-bit loads: two per face
// (unit normal and area; centre and weight), one per cell (centre and volume),
// one per gradient carried from sweep to sweep.  As arrays of single values
// the same visit took 18 requests.  The face kernels that need a few of these
// values, in face order, read them as plain arrays (sw, w, vol).  A cell's
// faces stand in a sliced ELL (32 cells a slice, slot-major, faces ascending)
// with the cell on the face's other side beside them, so a warp reads
// consecutive words and the neighbour's values need no trip through the face.
struct alignas(32) D4 {
  double x, y, z, w;
};
__device__ __forceinline__ D4 ld4(const D4* p) {  // read-only data
  D4 v;
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
      : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
  return v;
}

struct Geo {
  int n_cell, n_face;
  const int2* ab;              // owner and neighbour cell, 0-based (-1 on boundary faces)
  const D4 *fn, *fc;           // per face {unit normal, area}; {centre, w_fp}
  const D4* cr;                // per cell {centre, volume}
  const double2* sw;           // per face {area, w_fp}
  const double *l, *w, *vol;   // l_pn, w_fp; cell volumes
  const int* cs_row;           // first row of 32 slots of each slice of 32 cells
  const int2* cs;              // slots: {2 face + (1 for the neighbour's side), other cell};
                               // {-1, -1} padding, other cell -1 on boundary faces
};

struct Face {
  double nx, ny, nz, s, x, y, z, w;
};
// CENTRE off: the centre is not needed, the weight comes without it
template <bool CENTRE = true>
__device__ __forceinline__ Face face_of(const Geo& g, int f) {
  const D4 a = ld4(g.fn + f);
  if (!CENTRE) return {a.x, a.y, a.z, a.w, 0.0, 0.0, 0.0, g.w[f]};
  const D4 b = ld4(g.fc + f);
  return {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
}
struct Cell {
  double x, y, z, vol;
};
__device__ __forceinline__ Cell cell_of(const Geo& g, int c) {
  const D4 a = ld4(g.cr + c);
  return {a.x, a.y, a.z, a.w};
}
// A cell's slots, S at a time and before the faces are looked at: on a mesh
// of a few thousand cells a kernel is one wave whose time is the chain of its
// loads, and with a test for the list's end between them each slot waited for
// the face before it (9x9x9, us: two sweeps 12.1, now 9.3; the imbalance's
// sums 5.2, now 3.6).  S = 6, a hex cell's faces, where the registers allow.
template <int S>
__device__ __forceinline__ void chunk_of(const Geo& g, int c, int r, int end, int2 (&t)[S]) {
  const int2* p = g.cs + (32ll * r + (c & 31));
#pragma unroll
  for (int k = 0; k < S; ++k) t[k] = r + k < end ? p[32 * k] : make_int2(-1, -1);
}
__device__ __forceinline__ int face_in(int2 t) { return (int)((unsigned)t.x >> 1); }
__device__ __forceinline__ bool own_side(int2 t) { return (t.x & 1) == 0; }
// f(face, owner side, other cell) for the faces of cell c, ascending
template <int S, typename F>
__device__ __forceinline__ void faces_of(const Geo& g, int c, F&& f) {
  const int end = g.cs_row[(c >> 5) + 1];
  for (int r = g.cs_row[c >> 5]; r < end; r += S) {
    int2 t[S];
    chunk_of(g, c, r, end, t);
#pragma unroll
    for (int k = 0; k < S; ++k)
      if (t[k].x != -1) f(face_in(t[k]), own_side(t[k]), t[k].y);
  }
}
// The same where a face gives a value or a few, load(face, owner side): the
// chunk's are loaded side by side, then folded in by f(value, face, owner
// side, other cell) in order.
template <int S, typename L, typename F>
__device__ __forceinline__ void fold_faces(const Geo& g, int c, L&& load, F&& f) {
  const int end = g.cs_row[(c >> 5) + 1];
  for (int r = g.cs_row[c >> 5]; r < end; r += S) {
    int2 t[S];
    decltype(load(0, true)) v[S];
    chunk_of(g, c, r, end, t);
#pragma unroll
    for (int k = 0; k < S; ++k)
      if (t[k].x != -1) v[k] = load(face_in(t[k]), own_side(t[k]));
#pragma unroll
    for (int k = 0; k < S; ++k)
      if (t[k].x != -1) f(v[k], face_in(t[k]), own_side(t[k]), t[k].y);
  }
}

// std::min / std::max as the host evaluates them (ties and NaN included)
__device__ __forceinline__ double smin(double a, double b) { return (b < a) ? b : a; }
__device__ __forceinline__ double smax(double a, double b) { return (a < b) ? b : a; }

// displacement from a cell centre xc to its auxiliary point on the face:
// (x_f - n ((x_f - x_c).n)) - x_c, the host's V3 operations in order
struct Dx {
  double x, y, z;
};
__device__ __forceinline__ double dot3(double ax, double ay, double az, double bx, double by,
                                       double bz) {
  return da(da(dm(ax, bx), dm(ay, by)), dm(az, bz));
}
__device__ __forceinline__ Dx aux_dx(const Face& F, const Cell& C) {
  const double t = dot3(ds(F.x, C.x), ds(F.y, C.y), ds(F.z, C.z), F.nx, F.ny, F.nz);
  return {ds(ds(F.x, dm(F.nx, t)), C.x), ds(ds(F.y, dm(F.ny, t)), C.y),
          ds(ds(F.z, dm(F.nz, t)), C.z)};
}

constexpr int kBlock = 256;
constexpr int kRedBlocks = 1024;

// Above these many cells a vector field's components are one thread's work
// (K = 3 of each()); below, a thread for each has the shorter chain.  us, one
// thread a cell against three, in RCM order: two sweeps at 11.5k cells 17.3 /
// 10.3, 28k 15.0 / 11.6, 64k 19.7 / 19.9, 125k 32.6 / 35.6, 942k 226 / 266;
// deferred terms at 2.2k 5.6 / 5.2, 11.5k 5.9 / 5.9, 28k 7.2 / 8.8, 64k 10.4 /
// 13.3; gradient at 64k 8.8 / 8.0, 238k 20.4 / 19.4, 512k 47.5 / 52.1
// (unordered 80.6 / 65.4), 942k 76.6 / 87.2.
constexpr int kSweepVector = 64000;
constexpr int kDeferredVector = 16000;
constexpr int kGradientVector = 600000;

int grid(long long n) { return (int)std::max(1LL, std::min((n + kBlock - 1) / kBlock, 148LL * 16)); }

// d = rho (1/a_P)_f area V_f / l_pn (cfd_setup.f90:604-634)
__device__ __forceinline__ double pc_coef(double w, double s, double l, double vb, double va,
                                          double apb, double apa, double rho) {
  const double p_r = da(dd(w, da(apb, 1e-20)), dd(ds(1.0, w), da(apa, 1e-20)));
  const double v = lerp(w, vb, va);
  return dd(dm(dm(dm(rho, p_r), s), v), l);
}

// ---- momentum ---------------------------------------------------------------------
__global__ void k_fv_mom_faces(Geo g, const double* __restrict__ u, const double* __restrict__ flux,
                               double rho, double mu, double* __restrict__ p, double* __restrict__ n,
                               double* __restrict__ flux_out) {
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < g.n_face; f += gridDim.x * blockDim.x) {
    const int2 ab = g.ab[f];
    const int a = ab.x, b = ab.y;
    const D4 F = flux ? D4{0.0, 0.0, 0.0, g.sw[f].x} : ld4(g.fn + f);
    const double d = dd(dm(mu, F.w), g.l[f]);
    if (b >= 0) {
      double c;
      if (flux) {
        c = flux[f];
      } else {
        const double w = g.w[f];
        const double uf = lerp(w, u[3 * b], u[3 * a]);
        const double vf = lerp(w, u[3 * b + 1], u[3 * a + 1]);
        const double wf = lerp(w, u[3 * b + 2], u[3 * a + 2]);
        const double un = da(da(dm(uf, F.x), dm(vf, F.y)), dm(wf, F.z));
        c = dm(dm(rho, F.w), un);
      }
      if (flux_out) flux_out[f] = c;
      const double mn = (0.0 < c) ? 0.0 : c;  // std::min(c, 0.0)
      const double mx = (c < 0.0) ? 0.0 : c;  // std::max(c, 0.0)
      p[f] = da(-d, mn);
      n[f] = ds(-d, mx);
    } else {
      if (flux_out) flux_out[f] = 0.0;
      p[f] = -d;
      n[f] = 0.0;
    }
  }
}

__global__ void k_fv_mom_cells(Geo g, const double* __restrict__ u, const double* __restrict__ p,
                               const double* __restrict__ n, double u_lid, double urf,
                               double* __restrict__ pl, double* __restrict__ rhs) {
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < g.n_cell; c += gridDim.x * blockDim.x) {
    double s = 0.0, rx = 0.0;
    fold_faces<6>(
        g, c, [&](int f, bool own) { return own ? p[f] : n[f]; },
        [&](double v, int f, bool, int other) {
          if (other < 0) {
            const double d = -v;
            s = da(s, d);
            // the moving lid: the y = 1 wall (outward normal +y)
            const Face F = face_of(g, f);
            if (F.ny > 0.9 && F.y > 1.0 - 1e-9) rx = da(rx, dm(d, u_lid));
          } else {
            s = ds(s, v);
          }
        });
    s = dd(s, urf);
    pl[c] = s;
    if (rhs) {
      const double k = dm(ds(1.0, urf), s);
      rhs[3 * c] = da(rx, dm(k, u[3 * c]));
      rhs[3 * c + 1] = da(0.0, dm(k, u[3 * c + 1]));
      rhs[3 * c + 2] = da(0.0, dm(k, u[3 * c + 2]));
    }
  }
}

// ---- pressure correction ----------------------------------------------------------
__global__ void k_fv_pc_faces(Geo g, const double* __restrict__ ap, double rho, int pc,
                              double* __restrict__ dface, double* __restrict__ p,
                              double* __restrict__ n) {
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < g.n_face; f += gridDim.x * blockDim.x) {
    const int2 ab = g.ab[f];
    const int a = ab.x, b = ab.y;
    double d = 0.0, off = 0.0;
    if (b >= 0) {
      const double2 sw = g.sw[f];
      d = pc_coef(sw.y, sw.x, g.l[f], g.vol[b], g.vol[a], ap[b], ap[a], rho);
      if (a != pc && b != pc) off = -d;
    }
    dface[f] = d;
    p[f] = off;
    n[f] = off;
  }
}

__global__ void k_fv_pc_cells(Geo g, const double* __restrict__ dface, double* __restrict__ pl) {
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < g.n_cell; c += gridDim.x * blockDim.x) {
    double s = 0.0;
    fold_faces<6>(
        g, c, [&](int f, bool) { return dface[f]; },
        [&](double d, int, bool, int other) {
          if (other >= 0) s = da(s, d);
        });
    pl[c] = s;
  }
}

// ---- Green-Gauss gradient -----------------------------------------------------------
// The kernels over components come in three forms: K = 1, a scalar; K = 3,
// a vector field's components in one thread (the geometry is read and the
// auxiliary points are formed once); K = 0, one of nc components a thread, a
// cell's components in neighbouring lanes, which then read the geometry
// together (apart, in blocks of their own, four components of an 80^3
// gradient took 163 us; 66 like this).  each() gives a thread its cells (or
// faces) i, the first of their M components that is its own, and M.
template <int K, typename F>
__device__ __forceinline__ void each(int n, int nc, F&& f) {
  if constexpr (K != 0) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
      f(i, 0, K);
  } else {
    const long long tot = (long long)n * nc;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < tot;
         t += (long long)gridDim.x * blockDim.x) {
      const int i = tot <= 0xffffffffll ? (int)((unsigned)t / (unsigned)nc) : (int)(t / nc);
      f(i, (int)(t - (long long)i * nc), nc);
    }
  }
}
template <int K>
__global__ void k_fv_gradient(Geo g, int nc, const double* __restrict__ phi,
                              double* __restrict__ grad) {
  constexpr int NC = K == 3 ? 3 : 1;
  each<K>(g.n_cell, nc, [&](int c, int k0, int M) {
    double gx[NC], gy[NC], gz[NC], own_phi[NC];
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      gx[k] = gy[k] = gz[k] = 0.0;
      own_phi[k] = phi[(size_t)c * M + k0 + k];
    }
    faces_of<6>(g, c, [&](int f, bool own, int other) {
      const Face F = face_of<false>(g, f);
#pragma unroll
      for (int k = 0; k < NC; ++k) {
        double pf = own_phi[k];
        if (other >= 0) {
          const double po = phi[(size_t)other * M + k0 + k];
          pf = own ? lerp(F.w, po, pf) : lerp(F.w, pf, po);
        }
        const double ps = dm(pf, F.s);
        const double tx = dm(ps, F.nx), ty = dm(ps, F.ny), tz = dm(ps, F.nz);
        gx[k] = own ? da(gx[k], tx) : ds(gx[k], tx);
        gy[k] = own ? da(gy[k], ty) : ds(gy[k], ty);
        gz[k] = own ? da(gz[k], tz) : ds(gz[k], tz);
      }
    });
    const double v = g.cr[c].w;
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      double* o = grad + ((size_t)c * M + k0 + k) * 3;
      o[0] = dd(gx[k], v);
      o[1] = dd(gy[k], v);
      o[2] = dd(gz[k], v);
    }
  });
}

// ---- solv_grad in full: corrected Green-Gauss sweeps ---------------------------------
// One sweep of fvm_gradient_sweeps (cfd_setup.f90:765-866): the face value
// of each face (previous sweep's gradient g0 at the auxiliary points after
// the first sweep; walls by neu), its term ((phi_f s) n) / V added by each
// of the face's cells in ascending face order, 1/V (vr) formed once per
// cell.  bval[f*nc + k] are the wall values for neu = 0.  The gradients
// between sweeps (g0, and grad where PAD) are records of four.
template <int K, bool CORR, bool PAD>
__global__ void __launch_bounds__(kBlock, !CORR || K == 1 ? 4 : K == 0 ? 3 : 2)
k_fv_grad_sweep(Geo g, int nc, const double* __restrict__ phi, const double* __restrict__ bval,
                int neu, const double* __restrict__ vr, const D4* __restrict__ g0,
                double* __restrict__ grad) {
  constexpr int NC = K == 3 ? 3 : 1;
  each<K>(g.n_cell, nc, [&](int c, int k0, int M) {
    double gx[NC], gy[NC], gz[NC], pc[NC];
    D4 gc[NC];
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      const size_t q = (size_t)c * M + k0 + k;
      gx[k] = gy[k] = gz[k] = 0.0;
      pc[k] = phi[q];
      gc[k] = CORR ? ld4(g0 + q) : D4{};
    }
    const double v = vr[c];
    const Cell C = CORR ? cell_of(g, c) : Cell{};
    faces_of<K == 1 && CORR ? 3 : 6>(g, c, [&](int f, bool own, int other) {
      const Face F = face_of<CORR>(g, f);
      Dx xc{}, xo{};  // this cell's auxiliary point and the other's
      if (CORR && other >= 0) {
        xc = aux_dx(F, C);
        xo = aux_dx(F, cell_of(g, other));
      }
#pragma unroll
      for (int k = 0; k < NC; ++k) {
        double pf;
        if (other >= 0) {
          const size_t q = (size_t)other * M + k0 + k;
          double me = pc[k], po = phi[q];
          if (CORR) {
            const D4 go = ld4(g0 + q);
            me = da(me, dot3(gc[k].x, gc[k].y, gc[k].z, xc.x, xc.y, xc.z));
            po = da(po, dot3(go.x, go.y, go.z, xo.x, xo.y, xo.z));
          }
          pf = own ? lerp(F.w, po, me) : lerp(F.w, me, po);
        } else if (neu > 0) {
          pf = pc[k];
          if (CORR && neu == 2)
            pf = da(pf, dot3(gc[k].x, gc[k].y, gc[k].z, ds(F.x, C.x), ds(F.y, C.y),
                             ds(F.z, C.z)));
        } else {
          pf = bval[(size_t)f * M + k0 + k];
        }
        const double ps = dm(pf, F.s);
        const double tx = dm(dm(ps, F.nx), v), ty = dm(dm(ps, F.ny), v), tz = dm(dm(ps, F.nz), v);
        gx[k] = own ? da(gx[k], tx) : ds(gx[k], tx);
        gy[k] = own ? da(gy[k], ty) : ds(gy[k], ty);
        gz[k] = own ? da(gz[k], tz) : ds(gz[k], tz);
      }
    });
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      const size_t q = (size_t)c * M + k0 + k;
      if (PAD) {
        reinterpret_cast<D4*>(grad)[q] = {gx[k], gy[k], gz[k], 0.0};
      } else {
        grad[3 * q] = gx[k];
        grad[3 * q + 1] = gy[k];
        grad[3 * q + 2] = gz[k];
      }
    }
  });
}

__global__ void k_fv_recip(int n, const D4* __restrict__ cr, double* __restrict__ vr) {
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x)
    vr[c] = dd(1.0, cr[c].w);  // cfd_grid.f90:546
}

// ---- explicit momentum terms: fvm_momentum_deferred ------------------------------------
// Per interior face and component (cfd_setup.f90:185-272, 306-328):
// cor = c_bl c (phi_up - phi_f) + d ((phi_N' - phi_P') - (phi_N - phi_P)),
// the face value by `scheme` (0 central, 1 min-mod, 2 van Leer, 3 superbee
// on the auxiliary-point values); then each cell adds +cor (owner) or
// -cor (neighbour) of its faces in ascending face order.
template <int K>
__global__ void __launch_bounds__(kBlock, K == 3 ? 3 : 4)
k_fv_deferred_faces(Geo g, int nc, const double* __restrict__ phi, const double* __restrict__ grad,
                    const double* __restrict__ flux, double mu, double c_bl, int scheme,
                    double* __restrict__ cor) {
  constexpr int NC = K == 3 ? 3 : 1;
  each<K>(g.n_face, nc, [&](int f, int k0, int M) {
    const int2 ab = g.ab[f];
    const int a = ab.x, b = ab.y;
    if (b < 0) {
#pragma unroll
      for (int k = 0; k < NC; ++k) cor[(size_t)f * M + k0 + k] = 0.0;
      return;
    }
    const Face F = face_of(g, f);
    const Cell A = cell_of(g, a), B = cell_of(g, b);
    const double w = F.w;
    const Dx xa = aux_dx(F, A), xb = aux_dx(F, B);
    const double c = flux[f], d = dd(dm(mu, F.s), g.l[f]);
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      const size_t qa = (size_t)a * M + k0 + k, qb = (size_t)b * M + k0 + k;
      const double pa = phi[qa], pb = phi[qb];
      const double ga[3] = {grad[3 * qa], grad[3 * qa + 1], grad[3 * qa + 2]};
      const double gb[3] = {grad[3 * qb], grad[3 * qb + 1], grad[3 * qb + 2]};
      const double pa_aux = da(pa, dot3(ga[0], ga[1], ga[2], xa.x, xa.y, xa.z));
      const double pb_aux = da(pb, dot3(gb[0], gb[1], gb[2], xb.x, xb.y, xb.z));
      double r_cor = 0.0;
      if (c != 0.0) {
        double pf;
        if (scheme == 0) {
          pf = lerp(w, pb_aux, pa_aux);
        } else {
          const bool fwd = c > 0.0;
          const double pc = fwd ? pa_aux : pb_aux, pd = fwd ? pb_aux : pa_aux;
          const double xpa[3] = {da(A.x, xa.x), da(A.y, xa.y), da(A.z, xa.z)};
          const double xpb[3] = {da(B.x, xb.x), da(B.y, xb.y), da(B.z, xb.z)};
          double dx[3], gc[3];
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            dx[q] = fwd ? ds(xpb[q], xpa[q]) : ds(xpa[q], xpb[q]);
            gc[q] = fwd ? ga[q] : gb[q];
          }
          const double pu = ds(pd, dm(2.0, dot3(gc[0], gc[1], gc[2], dx[0], dx[1], dx[2])));
          double r = dd(ds(pc, pu), da(ds(pd, pc), 1e-20));
          if (scheme == 1) {
            r = smax(0.0, smin(1.0, r));
          } else if (scheme == 2) {
            r = dd(da(r, fabs(r)), da(da(1.0, fabs(r)), 1e-20));
          } else {  // std::max({0, min(1, 2r), min(2, r)}): the first largest
            double m = 0.0;
            const double c1 = smin(1.0, dm(2.0, r)), c2 = smin(2.0, r);
            if (m < c1) m = c1;
            if (m < c2) m = c2;
            r = m;
          }
          pf = da(pc, dm(dm(0.5, r), ds(pd, pc)));
        }
        const double up = c > 0.0 ? pa : pb;
        r_cor = dm(dm(c_bl, c), ds(up, pf));
      }
      cor[(size_t)f * M + k0 + k] = da(r_cor, dm(d, ds(ds(pb_aux, pa_aux), ds(pb, pa))));
    }
  });
}

template <int K>
__global__ void __launch_bounds__(kBlock, K == 3 ? 3 : 4)
k_fv_deferred_cells(Geo g, int nc, const double* __restrict__ cor, double* __restrict__ rhs) {
  constexpr int NC = K == 3 ? 3 : 1;
  struct Cor {
    double x[NC];
  };
  each<K>(g.n_cell, nc, [&](int c, int k0, int M) {
    double acc[NC];
#pragma unroll
    for (int k = 0; k < NC; ++k) acc[k] = rhs[(size_t)c * M + k0 + k];
    fold_faces<6>(
        g, c,
        [&](int f, bool) {
          Cor v;
#pragma unroll
          for (int k = 0; k < NC; ++k) v.x[k] = cor[(size_t)f * M + k0 + k];
          return v;
        },
        [&](const Cor& v, int, bool own, int other) {
          if (other < 0) return;
#pragma unroll
          for (int k = 0; k < NC; ++k) acc[k] = own ? da(acc[k], v.x[k]) : ds(acc[k], v.x[k]);
        });
#pragma unroll
    for (int k = 0; k < NC; ++k) rhs[(size_t)c * M + k0 + k] = acc[k];
  });
}

// ---- Rhie-Chow face fluxes ------------------------------------------------------------
__global__ void k_fv_face_flux(Geo g, const double* __restrict__ u, const double* __restrict__ pr,
                               const double* __restrict__ gp, const double* __restrict__ ap,
                               double rho, int aux, double* __restrict__ flux) {
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < g.n_face; f += gridDim.x * blockDim.x) {
    const int2 ab = g.ab[f];
    const int a = ab.x, b = ab.y;
    if (b < 0) {
      flux[f] = 0.0;
      continue;
    }
    const Face F = face_of(g, f);
    const Cell A = cell_of(g, a), B = cell_of(g, b);
    const double w = F.w;
    const double ufx = lerp(w, u[3 * b], u[3 * a]), ufy = lerp(w, u[3 * b + 1], u[3 * a + 1]),
                 ufz = lerp(w, u[3 * b + 2], u[3 * a + 2]);
    const double d = pc_coef(w, F.s, g.l[f], B.vol, A.vol, ap[b], ap[a], rho);
    const double gx = lerp(w, gp[3 * b], gp[3 * a]), gy = lerp(w, gp[3 * b + 1], gp[3 * a + 1]),
                 gz = lerp(w, gp[3 * b + 2], gp[3 * a + 2]);
    const double dx = ds(B.x, A.x), dy = ds(B.y, A.y), dz = ds(B.z, A.z);
    double pa = pr[a], pb = pr[b];
    if (aux) {  // cfd_setup.f90:611-614
      const Dx xa = aux_dx(F, A), xb = aux_dx(F, B);
      pa = da(pa, dot3(gp[3 * a], gp[3 * a + 1], gp[3 * a + 2], xa.x, xa.y, xa.z));
      pb = da(pb, dot3(gp[3 * b], gp[3 * b + 1], gp[3 * b + 2], xb.x, xb.y, xb.z));
    }
    const double dp = ds(ds(pb, pa), da(da(dm(gx, dx), dm(gy, dy)), dm(gz, dz)));
    const double un = da(da(dm(ufx, F.nx), dm(ufy, F.ny)), dm(ufz, F.nz));
    flux[f] = ds(dm(dm(rho, F.s), un), dm(d, dp));
  }
}

// ---- mass imbalance -------------------------------------------------------------------
__global__ void k_fv_imbalance(Geo g, const double* __restrict__ flux, int pc,
                               double* __restrict__ bvec, double* __restrict__ part) {
  __shared__ double sh[kBlock / 32];
  double acc = 0.0;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < g.n_cell; c += gridDim.x * blockDim.x) {
    double s = 0.0;
    fold_faces<6>(
        g, c, [&](int f, bool) { return flux[f]; },
        [&](double d, int, bool own, int other) {
          if (other >= 0) s = own ? ds(s, d) : da(s, d);
        });
    if (c == pc) s = 0.0;
    bvec[c] = s;
    acc += fabs(s);
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < kBlock / 32; ++k) t += sh[k];
    part[blockIdx.x] = t;
  }
}

__global__ void k_fv_sum(int n, const double* __restrict__ part, double* __restrict__ out) {
  __shared__ double sh[kBlock / 32];
  double acc = 0.0;
  for (int k = threadIdx.x; k < n; k += blockDim.x) acc += part[k];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < kBlock / 32; ++k) t += sh[k];
    *out = t;
  }
}

// ---- SIMPLE corrections -------------------------------------------------------------------
__global__ void k_fv_correct_cells(Geo g, const double* __restrict__ pp,
                                   const double* __restrict__ gpp, const double* __restrict__ ap,
                                   double urf_p, double* __restrict__ u, double* __restrict__ p) {
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < g.n_cell; c += gridDim.x * blockDim.x) {
    p[c] = da(p[c], dm(urf_p, pp[c]));
    const double k = dd(g.vol[c], da(ap[c], 1e-20));
    for (int d = 0; d < 3; ++d) u[3 * c + d] = ds(u[3 * c + d], dm(k, gpp[3 * c + d]));
  }
}

__global__ void k_fv_correct_faces(Geo g, const double* __restrict__ pp,
                                   const double* __restrict__ ap, double rho,
                                   double* __restrict__ flux) {
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < g.n_face; f += gridDim.x * blockDim.x) {
    const int2 ab = g.ab[f];
    const int a = ab.x, b = ab.y;
    if (b < 0) continue;
    const double2 sw = g.sw[f];
    const double d = pc_coef(sw.y, sw.x, g.l[f], g.vol[b], g.vol[a], ap[b], ap[a], rho);
    flux[f] = ds(flux[f], dm(d, ds(pp[b], pp[a])));
  }
}

struct DBuf {
  void* p = nullptr;
  ~DBuf() { if (p) cudaFree(p); }
  template <typename T> T* as() const { return static_cast<T*>(p); }
};

}  // namespace

struct fv_gpu {
  int dev = 0;
  cudaStream_t stream = nullptr;
  Geo g{};
  DBuf ab, fn, fc, cr, sw, l, w, vol, vr, cs_row, cs, dface, part, total, tmp;
  size_t tmp_bytes = 0;
};

namespace {

template <typename T>
cudaError_t up(DBuf& b, const T* h, size_t count) {
  cudaError_t e = cudaMalloc(&b.p, std::max<size_t>(count, 1) * sizeof(T));
  if (e != cudaSuccess || count == 0) return e;
  return cudaMemcpy(b.p, h, count * sizeof(T), cudaMemcpyHostToDevice);
}

// The context's scratch of at least `bytes` (grown in order on its stream).
double* scratch(fv_gpu* fv, size_t bytes) {
  if (fv->tmp_bytes >= bytes && fv->tmp.p) return fv->tmp.as<double>();
  if (cudaStreamSynchronize(fv->stream) != cudaSuccess) return nullptr;
  if (fv->tmp.p) cudaFree(fv->tmp.p);
  fv->tmp.p = nullptr;
  fv->tmp_bytes = 0;
  if (cudaMalloc(&fv->tmp.p, bytes) != cudaSuccess) return nullptr;
  fv->tmp_bytes = bytes;
  return fv->tmp.as<double>();
}

// First row of each slice, and the rows in all, from the cells' face counts:
// a slice has as many rows of 32 slots as its widest cell has faces.  (Rows
// fit 32 bits where the counts' sum does; slots need not, with one cell of
// very many faces.)
std::vector<int> slice_rows(int n_cell, const int* deg) {
  std::vector<int> r(((long long)n_cell + 31) / 32 + 1, 0);
  for (int c = 0; c < n_cell; ++c) r[c / 32 + 1] = std::max(r[c / 32 + 1], deg[c]);
  for (size_t k = 1; k < r.size(); ++k) r[k] += r[k - 1];
  return r;
}

int enter(fv_gpu* fv) {
  if (!fv) return SOLV_GPU_BAD_INPUT;
  return cudaSetDevice(fv->dev) == cudaSuccess ? SOLV_GPU_OK : SOLV_GPU_DEVICE_ERROR;
}

// f(the form of the component kernels for this call: each(), kSweepVector)
template <typename F>
void with_form(const Geo& g, int ncomp, int vector_cells, F&& f) {
  if (ncomp == 1)
    f(std::integral_constant<int, 1>());
  else if (ncomp == 3 && g.n_cell > vector_cells)
    f(std::integral_constant<int, 3>());
  else
    f(std::integral_constant<int, 0>());
}
// Blocks for n cells or faces in form K
template <int K>
int grid_of(int n, int ncomp) {
  return grid(K == 0 ? (long long)n * ncomp : n);
}

int done() {
  return cudaGetLastError() == cudaSuccess ? SOLV_GPU_OK : SOLV_GPU_DEVICE_ERROR;
}

int create(fv_gpu** out, int device, int n_cell, int n_face, const int* ip, const int* in,
           const double* area, const double* nrm, const double* xf, const double* l_pn,
           const double* w_fp, const double* xc, const double* vol) {
  std::vector<int2> ab(n_face);
  std::vector<int> deg(n_cell, 0);
  for (int f = 0; f < n_face; ++f) {
    const int a = ip[f] - 1, b = in[f] - 1;
    if (a < 0 || a >= n_cell || b < -1 || b >= n_cell || a == b) return SOLV_GPU_BAD_INPUT;
    ab[f] = make_int2(a, b);
    deg[a]++;
    if (b >= 0) deg[b]++;
  }
  const std::vector<int> cs_row = slice_rows(n_cell, deg.data());
  std::vector<int2> cs((size_t)cs_row.back() * 32, make_int2(-1, -1));
  std::vector<int> pos(n_cell, 0);
  for (int f = 0; f < n_face; ++f) {  // ascending faces: each cell's slots come out sorted
    auto put = [&](int c, unsigned side, int other) {
      const size_t row = cs_row[c >> 5] + pos[c]++;
      cs[row * 32 + (c & 31)] = make_int2((int)(2u * f + side), other);
    };
    put(ab[f].x, 0, ab[f].y);
    if (ab[f].y >= 0) put(ab[f].y, 1, ab[f].x);
  }
  std::vector<D4> fn(n_face), fc(n_face), cr(n_cell);
  std::vector<double2> sw(n_face);
  for (size_t f = 0; f < (size_t)n_face; ++f) {
    fn[f] = {nrm[3 * f], nrm[3 * f + 1], nrm[3 * f + 2], area[f]};
    fc[f] = {xf[3 * f], xf[3 * f + 1], xf[3 * f + 2], w_fp[f]};
    sw[f] = make_double2(area[f], w_fp[f]);
  }
  for (size_t c = 0; c < (size_t)n_cell; ++c)
    cr[c] = {xc[3 * c], xc[3 * c + 1], xc[3 * c + 2], vol[c]};
  if (cudaSetDevice(device) != cudaSuccess) return SOLV_GPU_DEVICE_ERROR;
  fv_gpu* fv = new fv_gpu;
  fv->dev = device;
  const size_t F = n_face, N = n_cell;
  cudaError_t e = cudaSuccess;
  auto chk = [&](cudaError_t r) { if (e == cudaSuccess) e = r; };
  chk(up(fv->ab, ab.data(), F));
  chk(up(fv->fn, fn.data(), F));
  chk(up(fv->fc, fc.data(), F));
  chk(up(fv->cr, cr.data(), N));
  chk(up(fv->sw, sw.data(), F));
  chk(up(fv->l, l_pn, F));
  chk(up(fv->w, w_fp, F));
  chk(up(fv->vol, vol, N));
  chk(up(fv->cs_row, cs_row.data(), cs_row.size()));
  chk(up(fv->cs, cs.data(), cs.size()));
  chk(cudaMalloc(&fv->dface.p, std::max<size_t>(F, 1) * sizeof(double)));
  chk(cudaMalloc(&fv->part.p, kRedBlocks * sizeof(double)));
  chk(cudaMalloc(&fv->total.p, sizeof(double)));
  chk(cudaMalloc(&fv->vr.p, std::max<size_t>(N, 1) * sizeof(double)));
  if (e == cudaSuccess) {
    k_fv_recip<<<grid(n_cell), kBlock>>>(n_cell, fv->cr.as<D4>(), fv->vr.as<double>());
    chk(cudaGetLastError());
    chk(cudaDeviceSynchronize());
  }
  if (e != cudaSuccess) {
    delete fv;
    return SOLV_GPU_DEVICE_ERROR;
  }
  Geo& g = fv->g;
  g.n_cell = n_cell;
  g.n_face = n_face;
  g.ab = fv->ab.as<int2>();
  g.fn = fv->fn.as<D4>();
  g.fc = fv->fc.as<D4>();
  g.sw = fv->sw.as<double2>();
  g.vol = fv->vol.as<double>();
  g.cr = fv->cr.as<D4>();
  g.l = fv->l.as<double>();
  g.w = fv->w.as<double>();
  g.cs_row = fv->cs_row.as<int>();
  g.cs = fv->cs.as<int2>();
  *out = fv;
  return SOLV_GPU_OK;
}

}  // namespace

extern "C" {

int fv_gpu_create(fv_gpu** out, int device, int n_cell, int n_face, const int* ip, const int* in,
                  const double* area, const double* nrm, const double* xf, const double* l_pn,
                  const double* w_fp, const double* xc, const double* vol) {
  if (!out) return SOLV_GPU_BAD_INPUT;
  *out = nullptr;
  if (n_cell <= 0 || n_face < 0 || !ip || !in || !area || !nrm || !xf || !l_pn || !w_fp || !xc ||
      !vol)
    return SOLV_GPU_BAD_INPUT;
  try {
    return create(out, device, n_cell, n_face, ip, in, area, nrm, xf, l_pn, w_fp, xc, vol);
  } catch (const std::bad_alloc&) {
    return SOLV_GPU_TOO_LARGE;
  }
}

int fv_gpu_destroy(fv_gpu* fv) {
  if (!fv) return SOLV_GPU_BAD_INPUT;
  cudaSetDevice(fv->dev);
  cudaStreamSynchronize(fv->stream);
  delete fv;
  return SOLV_GPU_OK;
}

int fv_gpu_set_stream(fv_gpu* fv, void* stream) {
  if (!fv) return SOLV_GPU_BAD_INPUT;
  fv->stream = static_cast<cudaStream_t>(stream);
  return SOLV_GPU_OK;
}

int fv_gpu_momentum(fv_gpu* fv, const double* u, const double* flux, double rho, double mu,
                    double u_lid, double urf, double* p, double* n, double* pl, double* rhs,
                    double* flux_out) {
  int rc = enter(fv);
  if (rc) return rc;
  if (!u || !p || !n || !pl || !(urf > 0.0)) return SOLV_GPU_BAD_INPUT;
  const Geo& g = fv->g;
  k_fv_mom_faces<<<grid(g.n_face), kBlock, 0, fv->stream>>>(g, u, flux, rho, mu, p, n, flux_out);
  k_fv_mom_cells<<<grid(g.n_cell), kBlock, 0, fv->stream>>>(g, u, p, n, u_lid, urf, pl, rhs);
  return done();
}

int fv_gpu_pressure_correction(fv_gpu* fv, const double* ap, double rho, int pin, double* p,
                               double* n, double* pl) {
  int rc = enter(fv);
  if (rc) return rc;
  if (!ap || !p || !n || !pl || pin < 0 || pin > fv->g.n_cell) return SOLV_GPU_BAD_INPUT;
  const Geo& g = fv->g;
  k_fv_pc_faces<<<grid(g.n_face), kBlock, 0, fv->stream>>>(g, ap, rho, pin - 1,
                                                           fv->dface.as<double>(), p, n);
  k_fv_pc_cells<<<grid(g.n_cell), kBlock, 0, fv->stream>>>(g, fv->dface.as<double>(), pl);
  return done();
}

int fv_gpu_gradient(fv_gpu* fv, int ncomp, const double* phi, double* grad) {
  int rc = enter(fv);
  if (rc) return rc;
  if (ncomp < 1 || ncomp > 16 || !phi || !grad) return SOLV_GPU_BAD_INPUT;
  const Geo& g = fv->g;
  with_form(g, ncomp, kGradientVector, [&](auto form) {
    constexpr int K = decltype(form)::value;
    k_fv_gradient<K><<<grid_of<K>(g.n_cell, ncomp), kBlock, 0, fv->stream>>>(g, ncomp, phi, grad);
  });
  return done();
}

int fv_gpu_face_flux(fv_gpu* fv, const double* u, const double* p, const double* gradp,
                     const double* ap, double rho, double* flux) {
  int rc = enter(fv);
  if (rc) return rc;
  if (!u || !p || !gradp || !ap || !flux) return SOLV_GPU_BAD_INPUT;
  const Geo& g = fv->g;
  k_fv_face_flux<<<grid(g.n_face), kBlock, 0, fv->stream>>>(g, u, p, gradp, ap, rho, 0, flux);
  return done();
}

int fv_gpu_face_flux_aux(fv_gpu* fv, const double* u, const double* p, const double* gradp,
                         const double* ap, double rho, double* flux) {
  int rc = enter(fv);
  if (rc) return rc;
  if (!u || !p || !gradp || !ap || !flux) return SOLV_GPU_BAD_INPUT;
  const Geo& g = fv->g;
  k_fv_face_flux<<<grid(g.n_face), kBlock, 0, fv->stream>>>(g, u, p, gradp, ap, rho, 1, flux);
  return done();
}

int fv_gpu_gradient_sweeps(fv_gpu* fv, int ncomp, const double* phi, const double* bval,
                           int n_iter, int neu, double* grad) {
  int rc = enter(fv);
  if (rc) return rc;
  if (ncomp < 1 || ncomp > 16 || !phi || !grad || n_iter < 1 || n_iter > 64 || neu < 0 ||
      neu > 2 || (neu == 0 && !bval))
    return SOLV_GPU_BAD_INPUT;
  const Geo& g = fv->g;
  const size_t G = (size_t)4 * ncomp * g.n_cell;  // a sweep's gradients, in records of four
  double* t = scratch(fv, std::max<size_t>(std::min(n_iter - 1, 2) * G, 1) * sizeof(double));
  if (!t) return SOLV_GPU_DEVICE_ERROR;
  const double* g0 = nullptr;
  for (int it = 1; it <= n_iter; ++it) {
    const bool pad = it < n_iter;
    double* out = pad ? t + ((it & 1) ? 0 : G) : grad;
    with_form(g, ncomp, kSweepVector, [&](auto form) {
      constexpr int K = decltype(form)::value;
      auto kern = !g0 ? (pad ? k_fv_grad_sweep<K, false, true> : k_fv_grad_sweep<K, false, false>)
                      : (pad ? k_fv_grad_sweep<K, true, true> : k_fv_grad_sweep<K, true, false>);
      kern<<<grid_of<K>(g.n_cell, ncomp), kBlock, 0, fv->stream>>>(
          g, ncomp, phi, bval, neu, fv->vr.as<double>(), reinterpret_cast<const D4*>(g0), out);
    });
    g0 = out;
  }
  return done();
}

int fv_gpu_momentum_deferred(fv_gpu* fv, int ncomp, const double* phi, const double* grad,
                             const double* flux, double mu, double c_bl, int scheme,
                             double* rhs) {
  int rc = enter(fv);
  if (rc) return rc;
  if (ncomp < 1 || ncomp > 16 || !phi || !grad || !flux || !rhs || scheme < 0 || scheme > 3)
    return SOLV_GPU_BAD_INPUT;
  const Geo& g = fv->g;
  double* cor = scratch(fv, std::max<size_t>((size_t)g.n_face * ncomp, 1) * sizeof(double));
  if (!cor) return SOLV_GPU_DEVICE_ERROR;
  with_form(g, ncomp, kDeferredVector, [&](auto form) {
    constexpr int K = decltype(form)::value;
    k_fv_deferred_faces<K><<<grid_of<K>(g.n_face, ncomp), kBlock, 0, fv->stream>>>(
        g, ncomp, phi, grad, flux, mu, c_bl, scheme, cor);
    k_fv_deferred_cells<K><<<grid_of<K>(g.n_cell, ncomp), kBlock, 0, fv->stream>>>(g, ncomp, cor,
                                                                                  rhs);
  });
  return done();
}

int fv_gpu_mass_imbalance(fv_gpu* fv, const double* flux, int pin, double* b, double* total) {
  int rc = enter(fv);
  if (rc) return rc;
  if (!flux || !b || pin < 0 || pin > fv->g.n_cell) return SOLV_GPU_BAD_INPUT;
  const Geo& g = fv->g;
  const int nb = std::min(grid(g.n_cell), kRedBlocks);
  k_fv_imbalance<<<nb, kBlock, 0, fv->stream>>>(g, flux, pin - 1, b, fv->part.as<double>());
  k_fv_sum<<<1, kBlock, 0, fv->stream>>>(nb, fv->part.as<double>(), fv->total.as<double>());
  if ((rc = done())) return rc;
  if (total) {
    if (cudaMemcpyAsync(total, fv->total.p, sizeof(double), cudaMemcpyDeviceToHost, fv->stream) !=
            cudaSuccess ||
        cudaStreamSynchronize(fv->stream) != cudaSuccess)
      return SOLV_GPU_DEVICE_ERROR;
  }
  return SOLV_GPU_OK;
}

int fv_gpu_simple_correct(fv_gpu* fv, const double* pp, const double* gradpp, const double* ap,
                          double rho, double urf_p, double* u, double* p, double* flux) {
  int rc = enter(fv);
  if (rc) return rc;
  if (!pp || !gradpp || !ap || !u || !p || !flux) return SOLV_GPU_BAD_INPUT;
  const Geo& g = fv->g;
  k_fv_correct_cells<<<grid(g.n_cell), kBlock, 0, fv->stream>>>(g, pp, gradpp, ap, urf_p, u, p);
  k_fv_correct_faces<<<grid(g.n_face), kBlock, 0, fv->stream>>>(g, pp, ap, rho, flux);
  return done();
}

}  // extern "C"
