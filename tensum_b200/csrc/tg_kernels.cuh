// tg_kernels.cuh -- device kernels of the FP64 single-solve path.
//
// One launch per reference phase; every accumulation is a fixed-order gather
// over per-vertex lists built on the host (tg_mesh.cc), so results are
// bitwise reproducible from run to run.
#pragma once

#include <cstdint>

#include "tg_physics.cuh"

namespace tg {

constexpr int kBlock = 256;

struct MeshView {
  int nv, ne, nb, nvu, n_int_cells;
  const double *dcarea, *inv6mc, *pweight;
  const double *inv_area;             // 1 / dcarea
  // local time step: sum of |n| over a vertex's gather list (boundary faces half), and of
  // |n| / |x_b - x_a| over its edges (viscous runs)
  const double *lam_area, *lam_visc;
  const int *e_a, *e_b;
  const double *e_nx, *e_ny, *e_dx, *e_dy;
  const int *ce_off, *ce_ent;
  const int *cb_off, *cb_ent;
  const int *b_v0, *b_v1, *b_kind, *b_adiab, *b_cell;
  const double *b_nx, *b_ny, *b_val;
  const double *bf_face_nx, *bf_face_ny;
  const int *bf_face_v0, *bf_face_v1;
  const int* u_cell;
  const int* c_v;
  const double *c_n, *c_inv2a;
  const int *c_bf_off, *c_bf, *c_nbr_off, *c_nbr;
  // bc_scheme strong: per vertex bit 0 = a boundary condition resets its state,
  // bit 1 = on a no-slip face; the reset list (vertex, then (face << 1 | slot)
  // entries in reference face order)
  const int* sflag;
  int nsb;
  const int *sb_v, *sb_off, *sb_ent;
  // axisymmetric radii (src/grid_preproc.cc:750-777): per vertex and per viscous unit
  const double *v_r, *u_r;
};

// Vertex radius of an axisymmetric run (1 when planar): update_solution divides
// by radius x dual area (src/fv.cc:1646, 1671, 1685).
__device__ __forceinline__ double vertex_radius(const Params& k, const MeshView& m, int v) {
  return k.axi ? m.v_r[v] : 1.0;
}

// Dependent launches.  The kernels of a step are launched with programmatic stream
// serialization: a kernel's CTAs may start once every CTA of its predecessor has called
// pdl_trigger (or ended) and an SM has room, and pdl_wait returns when the predecessor has
// completed and its writes are visible.  Nothing else makes them visible: a trigger orders
// the launch in time and no memory.  So every such kernel waits before it reads or writes
// anything a step changes -- its own completion then implies that of all kernels before it --
// and reads mesh data only ahead of that, behind the predecessor's tail.  A kernel may be
// resident while its predecessor writes what it will read, so none of its parameters is
// declared __restrict__ (read-only data the compiler may fetch at any time).  Launched
// without the attribute both calls do nothing.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// A 32-byte record: one sector, moved by one 256-bit access per thread.
struct alignas(32) D4 {
  double x, y, z, w;
};
__device__ __forceinline__ D4 ld4(const D4* p) {
  D4 v;
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void st4(D4* p, double x, double y, double z, double w) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(x), "d"(y), "d"(z), "d"(w) : "memory");
}

// Device state.  What the flux of a vertex reads is one 32-byte record
// S = (u, v, p, V5), so a gather of a neighbour touches one sector and one owned vertex
// is one access; the temperature and V1 are arrays of their own (the central fluxes read
// neither).  V2 = -V5 u and V3 = -V5 v are not stored: with V5 = -2 beta they are the
// products prim2ent forms.  Strong boundary conditions reset u, v, p and T after an update
// and leave the entropy variables, so their runs keep V2, V3 in W23.
struct StateView {
  D4* S;          // nv    u, v, p, V5
  double* T;      // nv
  double* V1;     // nv
  double2* W23;   // nv    V2, V3 (bc_scheme strong only)
  const D4* S0;   // the state the step started from: U_old is formed from it (not for strong
  const double* T0;   // conditions' reset vertices: their density comes from T0)
  D4* G;          // 2*nv  (dV1/dx, dV1/dy, dV2/dx, dV2/dy), (dV3/dx, dV3/dy, dV5/dx, dV5/dy)
  double* R;      // 4*nv  component-major
  double* Uold;   // 4*nv  store_conserved_old for the single-phase calls
  double* dt;     // nv
  double* Fb;     // 4*2*nb
  double* Fv;     // 3*3*nvu  (x-mom, y-mom, energy)
  double* Fvb;    // 3*nb
  double* part;   // block partial sums
  double* R2;     // 4*nv  RK4 residual accumulator (residual2 of src/fv.h)
  int* ssw;       // nv    Liou shock switch (src/fv.h:160)
};

// Step bookkeeping kept on the device so that whole steps replay from a CUDA graph.
struct Scalars {
  double dt_global;
  double elapsed;
  double rtotal;
  double rtotal0;
  double rnorm[4];
  long long iter;
  int counter;
  int reached;
  int done;
  int bad;
  unsigned long long dtmin_bits;
  int stop_counter;    // steps stop once counter exceeds it (output-time stepping)
  // Set by a last-stage update that also formed dt and its minimum
  // (dtmin_next) for the state it wrote; cleared whenever the state changes by
  // any other route, so the next step then forms them itself.
  int dt_next;
  unsigned long long dtmin_next;
  unsigned int blocks_done;   // blocks of the last stage's launch that have written their norm partials
  double rsq[4];              // a partition's residual-norm sums of its last step, before the exchange
};

struct Control {
  int time_mode;       // 0 steady, 1 unsteady
  int n_rks;           // stages per step: 3 (ssprk3) or 4 (rk4)
  int scheme;          // 0 ssprk3, 1 rk4
  int ntinst;
  double time_step;
  double min_residue;
  long long max_iter;
  double final_time;
  const double* tinst;
  int part;            // a partition of a decomposed mesh: norms wait for the other partitions' sums
};

__device__ __forceinline__ Prim load_prim(const StateView& s, int i) {
  const D4 r = ld4(s.S + i);
  Prim q;
  q.T = s.T[i]; q.u = r.x; q.v = r.y; q.p = r.z;
  return q;
}
// The stored entropy variables of a vertex.
__device__ __forceinline__ Ent load_ent(const Params& k, const StateView& s, int i) {
  const D4 r = ld4(s.S + i);
  Ent e;
  e.f = s.V1[i]; e.l = r.w;
  if (k.strong) {
    const double2 w = s.W23[i];
    e.vx = w.x; e.vy = w.y;
  } else {
    e.vx = -r.w * r.x; e.vy = -r.w * r.y;
  }
  return e;
}
__device__ __forceinline__ void store_state(const Params& k, const StateView& s, int i, const Prim& q, const Ent& e) {
  st4(s.S + i, q.u, q.v, q.p, e.l);
  s.T[i] = q.T;
  s.V1[i] = e.f;
  if (k.strong) s.W23[i] = make_double2(e.vx, e.vy);
}

// Entropy variables of a vertex after a boundary condition's single-state form
// (src/bc.h:615-654).  A condition that changes nothing returns the stored variables; one
// that keeps T and p (slip, adiabatic no-slip) moves V1 by beta (|u|^2 - |u'|^2) exactly;
// the others, and strong runs (whose stored variables lag the reset state), form them anew.
// Without the logarithms a boundary vertex's thread no longer holds its tile's gradient
// pass back as long (17.7 -> 15.5 us on the 128 x 256 cylinder).
__device__ __forceinline__ Ent bc_ent(const Params& k, const StateView& s, int kind, int adiabatic, const double* val,
                                      double nx, double ny, int v) {
  if (!k.strong && (kind == BC_NONE || kind == BC_FARFIELD || kind == BC_OUTLET || kind == BC_PERIODIC))
    return load_ent(k, s, v);
  Prim q = load_prim(s, v);
  if (!k.strong && (kind == BC_SLIP || (kind == BC_NOSLIP && adiabatic))) {
    const double q2 = q.u * q.u + q.v * q.v, V5 = s.S[v].w;
    bc_apply1(kind, adiabatic, val, nx, ny, q);
    Ent e;
    e.f = s.V1[v] - 0.5 * V5 * (q2 - (q.u * q.u + q.v * q.v));
    e.vx = -V5 * q.u; e.vy = -V5 * q.v; e.l = V5;
    return e;
  }
  bc_apply1(kind, adiabatic, val, nx, ny, q);
  return prim2ent(k, q);
}

// Boundary correction n_b * (W_b0 + W_b1 - W_0 - W_1)/2 of one boundary face
// (src/fv.cc:926-966): states after the single-state BC at each face vertex.
__device__ __forceinline__ void bface_grad_corr(const Params& k, const MeshView& m, const StateView& s, int d,
                                                double* dW /*4*/) {
  const int v0 = m.b_v0[d], v1 = m.b_v1[d], kind = m.b_kind[d], ad = m.b_adiab[d];
  const double nx = m.b_nx[d], ny = m.b_ny[d];
  const Ent e0 = bc_ent(k, s, kind, ad, m.b_val + (size_t)d * 10, nx, ny, v0);
  const Ent e1 = bc_ent(k, s, kind, ad, m.b_val + (size_t)d * 10 + 5, nx, ny, v1);
  const Ent w0 = load_ent(k, s, v0), w1 = load_ent(k, s, v1);
  dW[0] = (e0.f + e1.f - w0.f - w1.f) * 0.5;
  dW[1] = (e0.vx + e1.vx - w0.vx - w1.vx) * 0.5;
  dW[2] = (e0.vy + e1.vy - w0.vy - w1.vy) * 0.5;
  dW[3] = (e0.l + e1.l - w0.l - w1.l) * 0.5;
}

// ------------------------------------------------------------------ kernels

// Entropy variables of a state from its primitive one; bad (may be NULL): only when clear.
__global__ void k_prim2ent(Params k, int nv, StateView s, const int* __restrict__ bad) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nv || (bad && *bad)) return;
  const Prim q = load_prim(s, i);
  store_state(k, s, i, q, prim2ent(k, q));
}

// A caller state arrives as PrimVar records (T, p, u, v, w; src/primvar.h:17-18) in the caller's
// vertex order.  k_state_check flags any vertex the reference would refuse at
// initialisation (src/fv.cc:388-389: T > 0 and p > 0, NaN refused too);
// k_state_in then reorders into the device SoA only when nothing was flagged,
// so a refused state leaves the previous one in place.
__global__ void k_state_check(int nv, const double* __restrict__ raw, int* __restrict__ bad) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nv) return;
  const double* q = raw + 5 * (size_t)i;
  if (!(q[0] > 0.0) || !(q[1] > 0.0)) atomicOr(bad, 1);
}

__global__ void k_state_in(int nv, const double* __restrict__ raw, const int* __restrict__ old_of_new,
                           const int* __restrict__ bad, D4* __restrict__ S, double* __restrict__ T) {
  if (*bad) return;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nv) return;
  const double* q = raw + 5 * (size_t)old_of_new[i];
  st4(S + i, q[2], q[3], q[1], 0.0);   // V5 and V1 follow (k_prim2ent)
  T[i] = q[0];
}

// Device records -> PrimVar records in the caller's order (w = 0 in 2D).
__global__ void k_state_out(int nv, StateView s, const int* __restrict__ old_of_new,
                            double* __restrict__ raw) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nv) return;
  double* q = raw + 5 * (size_t)old_of_new[i];
  const Prim r = load_prim(s, i);
  q[0] = r.T; q[1] = r.p; q[2] = r.u; q[3] = r.v; q[4] = 0.0;
}

// A state handed in asynchronously (tg_set_state_async) becomes current, with fresh step
// bookkeeping, only if k_state_check accepted it.
__global__ void k_scalars_set(Scalars* sc, Scalars s0, const int* __restrict__ bad) {
  if (*bad) return;
  *sc = s0;
}

// Device gradients G (V1, V2, V3, V5) x (x, y) -> the reference's dE records,
// 5 variables x (x, y, z) per vertex in the caller's order (src/fv.h:148),
// zero for the z components and for the fourth (z-momentum) variable.
// zero_unstepped: all zero while no step has run since the state was set (the
// reference zeroes dE when a sample starts, src/fv.cc:207-212).
__global__ void k_grad_out(int nv, const D4* __restrict__ G, const int* __restrict__ old_of_new,
                           double* __restrict__ out, const Scalars* __restrict__ sc, int zero_unstepped) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nv) return;
  double* d = out + 15 * (size_t)old_of_new[i];
#pragma unroll
  for (int q = 0; q < 15; ++q) d[q] = 0.0;
  if (zero_unstepped && sc->iter == 0) return;
  const D4 a = ld4(G + 2 * (size_t)i), b = ld4(G + 2 * (size_t)i + 1);
  d[0] = a.x; d[1] = a.y; d[3] = a.z; d[4] = a.w;       // variables 0, 1, 2 and 4 of five
  d[6] = b.x; d[7] = b.y; d[12] = b.z; d[13] = b.w;
}

// store_conserved_old (src/fv.cc:1626-1630)
__global__ void k_store_old(Params k, MeshView m, StateView s, const int* __restrict__ done) {
  if (*done) return;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m.nv) return;
  Cons c = prim2con(k, load_prim(s, i));
  s.Uold[i] = c.r; s.Uold[m.nv + i] = c.mx; s.Uold[2 * m.nv + i] = c.my; s.Uold[3 * m.nv + i] = c.E;
}

// Boundary-face inviscid fluxes (src/fv.cc:1100-1188): one thread per (face, vertex).
template <int FLUX, int RECON>
__device__ __forceinline__ void bflux_one(const Params& k, const MeshView& m, const StateView& s, int t) {
  int d = t >> 1, q = t & 1;
  int c = q ? m.b_v1[d] : m.b_v0[d];
  Prim s0 = load_prim(s, c), s1 = s0;
  double nx = m.b_nx[d], ny = m.b_ny[d];
  int kind = m.b_kind[d];
  bc_apply2(kind, m.b_adiab[d], m.b_val + (size_t)d * 10 + 5 * q, nx, ny, s0, s1);
  Flx F;
  if (kind == BC_FARFIELD) {
    double z[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    F = num_flux<FLUX, RECON>(k, make_vrec<FLUX>(k, s0), make_vrec<FLUX>(k, s1), nx, ny, 0.0, 0.0, z, z);
  } else {
    F = inviscid_bflux(k, s0, s1, nx, ny);
  }
  const int n2 = 2 * m.nb;
  s.Fb[t] = F.m; s.Fb[n2 + t] = F.x; s.Fb[2 * n2 + t] = F.y; s.Fb[3 * n2 + t] = F.e;
}
template <int FLUX, int RECON>
__global__ void k_bflux(Params k, MeshView m, StateView s, const int* done) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < 2 * m.nb && !*done) bflux_one<FLUX, RECON>(k, m, s, t);
}

// Viscous residual units (src/fv.cc:1197-1320): interior cells and boundary faces.
__device__ __forceinline__ void viscous_one(const Params& k, const MeshView& m, const StateView& s, int u) {
  int c = m.u_cell[u];
  int v[3] = {m.c_v[3 * c], m.c_v[3 * c + 1], m.c_v[3 * c + 2]};
  const double* n = m.c_n + 6 * (size_t)c;
  // cell gradient: P1 sum, boundary corrections in face order, / (2 area)
  const Ent w0 = load_ent(k, s, v[0]), w1 = load_ent(k, s, v[1]), w2 = load_ent(k, s, v[2]);
  double dE[8];
  {
    const double a[4][3] = {{w0.f, w1.f, w2.f}, {w0.vx, w1.vx, w2.vx}, {w0.vy, w1.vy, w2.vy}, {w0.l, w1.l, w2.l}};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      dE[2 * q] = n[0] * a[q][0] + n[2] * a[q][1] + n[4] * a[q][2];
      dE[2 * q + 1] = n[1] * a[q][0] + n[3] * a[q][1] + n[5] * a[q][2];
    }
  }
  for (int j = m.c_bf_off[c]; j < m.c_bf_off[c + 1]; ++j) {
    int d = m.c_bf[j];
    double dW[4];
    bface_grad_corr(k, m, s, d, dW);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      dE[2 * q] += m.b_nx[d] * dW[q];
      dE[2 * q + 1] += m.b_ny[d] * dW[q];
    }
  }
  double f = m.c_inv2a[c];
#pragma unroll
  for (int q = 0; q < 8; ++q) dE[q] *= f;

  Ent avg;
  if (u < m.n_int_cells) {
    const double t3 = 1.0 / 3.0;
    avg.f = w0.f * t3 + w1.f * t3 + w2.f * t3;
    avg.vx = w0.vx * t3 + w1.vx * t3 + w2.vx * t3;
    avg.vy = w0.vy * t3 + w1.vy * t3 + w2.vy * t3;
    avg.l = w0.l * t3 + w1.l * t3 + w2.l * t3;
  } else {
    avg.f = avg.vx = avg.vy = avg.l = 0.0;
    int cnt = m.c_nbr_off[c + 1] - m.c_nbr_off[c];
    for (int j = m.c_nbr_off[c]; j < m.c_nbr_off[c + 1]; ++j) {
      int d = m.c_nbr[j];
      for (int q = 0; q < 2; ++q) {
        int vb = q ? m.bf_face_v1[d] : m.bf_face_v0[d];
        const double* val = m.b_val + (size_t)d * 10 + (vb == m.b_v0[d] ? 0 : 5);
        const Ent e = bc_ent(k, s, m.b_kind[d], m.b_adiab[d], val, m.bf_face_nx[d], m.bf_face_ny[d], vb);
        avg.f += e.f; avg.vx += e.vx; avg.vy += e.vy; avg.l += e.l;
      }
    }
    double sc = (0.5 * 1.0 / cnt);
    avg.f *= sc; avg.vx *= sc; avg.vy *= sc; avg.l *= sc;
  }
  ViscK K = viscous_K(k, avg, dE);
  const int n3 = 3 * m.nvu;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    Flx F = viscous_apply(K, n[2 * q], n[2 * q + 1]);
    s.Fv[3 * u + q] = F.x; s.Fv[n3 + 3 * u + q] = F.y; s.Fv[2 * n3 + 3 * u + q] = F.e;
  }
  if (u >= m.n_int_cells) {
    int d = u - m.n_int_cells;
    double nbx = m.b_nx[d], nby = m.b_ny[d];
    double Cor = m.b_adiab[d] ? -1.0 * (0.0 + K.c2 * K.e4 * K.e4 * (dE[6] * nbx + dE[7] * nby)) : 0.0;
    Flx F = viscous_apply(K, nbx, nby);
    s.Fvb[d] = F.x; s.Fvb[m.nb + d] = F.y; s.Fvb[2 * m.nb + d] = F.e - Cor;
  }
}
__global__ void k_viscous(Params k, MeshView m, StateView s, const int* __restrict__ done) {
  const int u = blockIdx.x * blockDim.x + threadIdx.x;
  if (u < m.nvu && !*done) viscous_one(k, m, s, u);
}

// |n| and the face spectral radius |u.n| + c |n| of the local time step
// (src/fv.cc:1512-1580), with their multiply-adds written out so that every
// kernel forming them rounds them the same way.
__device__ __forceinline__ double face_area(double nx, double ny) { return sqrt(fma(nx, nx, ny * ny)); }
__device__ __forceinline__ double face_radius(double u, double v, double nx, double ny, double c, double area) {
  return fma(c, area, fabs(fma(u, nx, v * ny)));
}

// The spectral radius sum of a vertex whose copies all hold its state q, from the sum of
// |u.n| over its faces: + c sum |n| + (mu / rho) sum |n| / |d|, the geometric sums formed
// once per mesh.  The last stage's update and k_dt both use it, so a step whose dt is
// formed either way is the same bit for bit.
__device__ __forceinline__ double spectral_sum(const Params& k, const MeshView& m, int v, const Prim& q, double un) {
  double lam = fma(sound_speed(k, q), m.lam_area[v], un);
  if (k.model == 1) lam = fma(viscosity(k, q.T) * (k.R * q.T) / q.p, m.lam_visc[v], lam);
  return lam;
}

__device__ __forceinline__ unsigned long long warp_min_u64(unsigned long long x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long y = __shfl_xor_sync(0xffffffffu, x, o);
    x = y < x ? y : x;
  }
  return x;
}

// Local time step (src/fv.cc:1499-1598): spectral-radius gather, dt = cfl A / sum,
// block minimum by warp shuffles, then one atomicMin on the (positive) bit pattern.
__global__ void k_dt(Params k, MeshView m, StateView s, Scalars* sc, const int* done, int in_step) {
  pdl_trigger();
  pdl_wait();
  if (*done) return;
  if (in_step && k.fuse_dt && sc->dt_next) return;   // the previous step's last update formed it
  int v = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long bits = 0x7ff0000000000000ull;  // +inf
  if (v < m.nv) {
    const Prim q0 = load_prim(s, v);
    double lam = 0.0;
    bool same = true;    // every periodic copy holds this vertex's state, as after any update
    for (int j = m.ce_off[v]; j < m.ce_off[v + 1]; ++j) {
      const int ent = m.ce_ent[j], e = ent >> 1;
      const int self = (ent & 1) ? m.e_b[e] : m.e_a[e];
      if (self != v) {
        const Prim q = load_prim(s, self);
        same = same && q.u == q0.u && q.v == q0.v && q.T == q0.T && q.p == q0.p;
      }
      lam += fabs(fma(q0.u, m.e_nx[e], q0.v * m.e_ny[e]));
    }
    if (same) {
      for (int j = m.cb_off[v]; j < m.cb_off[v + 1]; ++j) {
        const int ent = m.cb_ent[j];
        if ((ent & 3) != 0) continue;
        const int d = ent >> 3;
        lam += 0.5 * fabs(fma(q0.u, m.b_nx[d], q0.v * m.b_ny[d]));
      }
      lam = spectral_sum(k, m, v, q0, lam);
    } else {   // an initial state whose copies differ: each contribution from its own copy
      lam = 0.0;
      for (int j = m.ce_off[v]; j < m.ce_off[v + 1]; ++j) {
        const int ent = m.ce_ent[j], e = ent >> 1;
        const Prim q = load_prim(s, (ent & 1) ? m.e_b[e] : m.e_a[e]);
        const double nx = m.e_nx[e], ny = m.e_ny[e];
        lam += face_radius(q.u, q.v, nx, ny, sound_speed(k, q), face_area(nx, ny));
      }
      for (int j = m.cb_off[v]; j < m.cb_off[v + 1]; ++j) {
        const int ent = m.cb_ent[j];
        if ((ent & 3) != 0) continue;
        const int idx = ent >> 2, d = idx >> 1;
        const Prim q = load_prim(s, (idx & 1) ? m.b_v1[d] : m.b_v0[d]);
        const double nx = m.b_nx[d], ny = m.b_ny[d];
        lam += 0.5 * face_radius(q.u, q.v, nx, ny, sound_speed(k, q), face_area(nx, ny));
      }
      if (k.model == 1)
        for (int j = m.ce_off[v]; j < m.ce_off[v + 1]; ++j) {
          const int ent = m.ce_ent[j], e = ent >> 1;
          const Prim q = load_prim(s, (ent & 1) ? m.e_b[e] : m.e_a[e]);
          const double area = face_area(m.e_nx[e], m.e_ny[e]), dl = face_area(m.e_dx[e], m.e_dy[e]);
          lam += viscosity(k, q.T) * area / dl / density(k, q);
        }
    }
    double dtv = k.cfl * m.dcarea[v] / lam;
    s.dt[v] = dtv;
    bits = (unsigned long long)__double_as_longlong(dtv);
    if (!(dtv > 0.0)) bits = 0x7ff0000000000000ull;  // NaN / non-positive: flagged by the update
  }
  bits = warp_min_u64(bits);
  __shared__ unsigned long long wmin[kBlock / 32];
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) wmin[w] = bits;
  __syncthreads();
  if (w == 0) {
    bits = lane < (int)(blockDim.x >> 5) ? wmin[lane] : 0x7ff0000000000000ull;
    bits = warp_min_u64(bits);
    if (lane == 0) atomicMin(&sc->dtmin_bits, bits);
  }
}

// Start of a solve-loop iteration (src/fv.cc:2273-2276): loop condition and dt reset.
// compute_ssw (src/compute_ssw.cc:7-38): flags both endpoints of every edge
// (all faces, boundary ones included) across which u.n - a|n| or u.n + a|n|
// changes sign from positive to negative.  Writers only ever store 1.
__global__ void k_ssw(Params k, MeshView m, StateView s, const int* done) {
  pdl_trigger();
  pdl_wait();
  if (*done) return;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m.ne) return;
  const int a = m.e_a[e], b = m.e_b[e];
  const Prim qa = load_prim(s, a), qb = load_prim(s, b);
  const double nx = m.e_nx[e], ny = m.e_ny[e];
  const double ui = qa.u * nx + qa.v * ny, uj = qb.u * nx + qb.v * ny;
  const double ai = sound_speed(k, qa), aj = sound_speed(k, qb);
  const double area = sqrt(nx * nx + ny * ny);
  const double l1i = ui - ai * area, l1j = uj - aj * area;
  const double l5i = ui + ai * area, l5j = uj + aj * area;
  if ((l1i > 0 && l1j < 0) || (l5i > 0 && l5j < 0)) {
    s.ssw[a] = 1;
    s.ssw[b] = 1;
  }
}

// bc_scheme strong, after each stage update (src/fv.cc:1694-1704): every
// boundary face's condition applied to its vertices' primitive state in face
// order; the entropy variables keep their values (the reference does not
// recompute them), so gradients see the pre-condition state.
__global__ void k_strong_bc(MeshView m, StateView s, const int* done) {
  pdl_trigger();
  pdl_wait();
  if (*done) return;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m.nsb) return;
  const int v = m.sb_v[j];
  Prim q = load_prim(s, v);
  for (int e = m.sb_off[j]; e < m.sb_off[j + 1]; ++e) {
    const int d = m.sb_ent[e] >> 1, slot = m.sb_ent[e] & 1;
    bc_apply1(m.b_kind[d], m.b_adiab[d], m.b_val + (size_t)d * 10 + 5 * slot, m.b_nx[d], m.b_ny[d], q);
  }
  st4(s.S + v, q.u, q.v, q.p, s.S[v].w);
  s.T[v] = q.T;
}

// bc_scheme strong, in compute_residual_norm (src/fv.cc:1805-1819): the momentum
// residual of no-slip vertices is zeroed (the update then uses it).
__global__ void k_strong_zero_res(MeshView m, StateView s) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= m.nv || !(m.sflag[v] & 2)) return;
  s.R[m.nv + v] = 0.0;
  s.R[2 * (size_t)m.nv + v] = 0.0;
}

// Global dt and the unsteady clamp to the next output time (src/fv.cc:1584-1618).
__device__ __forceinline__ void dt_final(const Control& ctl, Scalars* sc) {
  double dtg;
  if (ctl.time_step > 0.0) {
    dtg = ctl.time_step;
  } else {
    dtg = 1.0e20;
    double m = __longlong_as_double((long long)sc->dtmin_bits);
    dtg = dmin_(dtg, m);
    if (ctl.time_mode == 1) {
      int c = sc->counter < ctl.ntinst ? sc->counter : ctl.ntinst - 1;
      if (sc->elapsed + dtg > ctl.tinst[c]) {
        dtg = ctl.tinst[c] - sc->elapsed;
        sc->reached = 1;
      }
    }
  }
  sc->dt_global = dtg;
}

__global__ void k_dt_final(Control ctl, Scalars* sc, const int* done) {
  pdl_trigger();
  pdl_wait();
  if (*done) return;
  dt_final(ctl, sc);
}

// Start of a solve-loop iteration: the loop condition, and the running dt
// minimum -- the previous step's last update already formed it for this state
// when dt_next is set.  warm (a step captured without the first-stage dt pass,
// launched only when dt_next is set): the dt clamp happens here too.
__global__ void k_step_begin(Control ctl, Scalars* sc, int* done, int warm) {
  pdl_trigger();
  pdl_wait();
  // unsteady runs never advance the iteration bound (term_iter stays 0, src/fv.cc:2266-2268)
  bool go = sc->rtotal > ctl.min_residue && (ctl.time_mode == 1 || sc->iter < ctl.max_iter) &&
            sc->elapsed < ctl.final_time && sc->counter <= sc->stop_counter;
  *done = go ? 0 : 1;
  if (!go) return;
  sc->dtmin_bits = sc->dt_next ? sc->dtmin_next : 0x7ff0000000000000ull;
  sc->dtmin_next = 0x7ff0000000000000ull;
  if (warm) dt_final(ctl, sc);
}

// Residual norms from the weighted squared sums of the whole mesh (src/fv.cc:1846-1876);
// the first iteration's total becomes the reference for the relative residual.
__device__ __forceinline__ void set_norms(Scalars* sc, const double* sum4, int nv_total, bool first) {
  double n0 = sqrt(sum4[0]) / nv_total, n1 = sqrt(sum4[1]) / nv_total;
  double n2 = sqrt(sum4[2]) / nv_total, n3 = sqrt(sum4[3]) / nv_total;
  double total = sqrt(n0 * n0 + (n1 * n1 + n2 * n2 + 0.0) + n3 * n3);
  if (first) {
    sc->rtotal0 = total;
    if (sc->rtotal0 == 0.0) sc->rtotal0 = 1.0;
  }
  sc->rnorm[0] = n0; sc->rnorm[1] = n1; sc->rnorm[2] = n2; sc->rnorm[3] = n3;
  sc->rtotal = total / sc->rtotal0;
}

// Residual norms from the per-block partials (src/fv.cc:1846-1876) and the end
// of the solve-loop iteration (src/fv.cc:2307-2343), by one block of `threads`
// threads (red: 4 * threads doubles of shared memory).
__device__ __forceinline__ void norm_and_step_end(const StateView& s, int nblocks, int nv_total, Scalars* sc,
                                                  const Control& ctl, double* red, int threads) {
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 8
  for (int b = threadIdx.x; b < nblocks; b += threads)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[c] += __ldcg(s.part + (size_t)b * 4 + c);
#pragma unroll
  for (int c = 0; c < 4; ++c) red[c * threads + threadIdx.x] = acc[c];
  __syncthreads();
  for (int o = threads / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o)
#pragma unroll
      for (int c = 0; c < 4; ++c) red[c * threads + threadIdx.x] += red[c * threads + threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double sum4[4] = {red[0], red[threads], red[2 * threads], red[3 * threads]};
    if (ctl.part) {
#pragma unroll
      for (int c = 0; c < 4; ++c) sc->rsq[c] = sum4[c];
    } else {
      set_norms(sc, sum4, nv_total, sc->iter == 0);
    }
    sc->iter += 1;
    sc->elapsed += sc->dt_global;
    if (sc->reached && ctl.time_mode == 1) {
      sc->counter += 1;
      sc->reached = 0;
    }
  }
}

// update_solution for SSP-RK3 (src/fv.cc:1641-1652), fused with the residual-norm
// partial sums of compute_residual_norm (src/fv.cc:1822-1841) at the last stage.
// New conserved state of vertex v at stage r from its residual: the Shu-Osher
// SSP-RK3 stage (src/fv.cc:1635-1658, src/constants.h:4-6) or the classical RK4
// stage (src/fv.cc:1667-1679, src/constants.h:9), which accumulates
// sum_r R_r / rks_r in R2 (zero before the first stage, src/fv.cc:2287-2293).
// c is the stage's input state (conserved), uo U_old, factor = dt / area.
__device__ __forceinline__ Cons rk_stage(const Control& ctl, const StateView& s, int nv, int v, int r, Cons c,
                                         const double* uo, double factor, double r0, double r1, double r2, double r3) {
  if (ctl.scheme == 1) {
    // selects, not an indexed table: the stage is a run-time value and a table would live in
    // local memory
    const double inv = (r == 1 || r == 2) ? 2.0 : 1.0;   // 1 / rks[r], rks = (1, 1/2, 1/2, 1)
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    if (r > 0) { a0 = s.R2[v]; a1 = s.R2[nv + v]; a2 = s.R2[2 * nv + v]; a3 = s.R2[3 * nv + v]; }
    a0 += r0 * inv; a1 += r1 * inv; a2 += r2 * inv; a3 += r3 * inv;
    if (r < 3) { s.R2[v] = a0; s.R2[nv + v] = a1; s.R2[2 * nv + v] = a2; s.R2[3 * nv + v] = a3; }
    const bool fin = (r == 3);
    const double c2 = fin ? -factor / 6.0 : -factor * (r == 2 ? 1.0 : 0.5);
    c.r = uo[0] * 1.0 + (fin ? a0 : r0) * c2;
    c.mx = uo[1] * 1.0 + (fin ? a1 : r1) * c2;
    c.my = uo[2] * 1.0 + (fin ? a2 : r2) * c2;
    c.E = uo[3] * 1.0 + (fin ? a3 : r3) * c2;
    return c;
  }
  const double ar = r == 0 ? 0.0 : (r == 1 ? 3.0 / 4.0 : 1.0 / 3.0);
  const double br = r == 0 ? 1.0 : (r == 1 ? 1.0 / 4.0 : 2.0 / 3.0);
  const double c2 = -factor * br;
  c.r *= br; c.mx *= br; c.my *= br; c.E *= br;
  c.r += uo[0] * ar + r0 * c2;
  c.mx += uo[1] * ar + r1 * c2;
  c.my += uo[2] * ar + r2 * c2;
  c.E += uo[3] * ar + r3 * c2;
  return c;
}

__global__ void k_update(Params k, MeshView m, StateView s, Control ctl, Scalars* sc, int r, int do_norm,
                         const int* __restrict__ done) {
  if (*done) return;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int nv = m.nv;
  double nrm[4] = {0.0, 0.0, 0.0, 0.0};
  if (i < nv) {
    double R0 = s.R[i], R1 = s.R[nv + i], R2 = s.R[2 * nv + i], R3 = s.R[3 * nv + i];
    const double ia = m.inv_area[i];
    if (do_norm) {
      double w = m.pweight[i];
      double q0 = R0 * ia, q1 = R1 * ia, q2 = R2 * ia, q3 = R3 * ia;
      nrm[0] = q0 * q0 * w; nrm[1] = q1 * q1 * w; nrm[2] = q2 * q2 * w; nrm[3] = q3 * q3 * w;
    }
    double dtv = (ctl.time_mode == 1 || ctl.time_step > 0.0) ? sc->dt_global : s.dt[i];
    const double factor = dtv * ia / vertex_radius(k, m, i);
    const double uo[4] = {s.Uold[i], s.Uold[nv + i], s.Uold[2 * nv + i], s.Uold[3 * nv + i]};
    Cons c = rk_stage(ctl, s, nv, i, r, prim2con(k, load_prim(s, i)), uo, factor, R0, R1, R2, R3);
    Prim q = con2prim(k, c);
    Ent e = prim2ent(k, q);
    store_state(k, s, i, q, e);
    bool ok = isfinite(q.T) && isfinite(q.u) && isfinite(q.v) && isfinite(q.p) && q.p > 0.0 && c.r > 0.0;
    if (!ok) atomicOr(&sc->bad, 1);
  }
  if (do_norm) {
    // fixed-shape block reduction -> per-block partials, summed in block order later
    __shared__ double red[4][kBlock];
#pragma unroll
    for (int c = 0; c < 4; ++c) red[c][threadIdx.x] = nrm[c];
    __syncthreads();
    for (int o = kBlock / 2; o > 0; o >>= 1) {
      if ((int)threadIdx.x < o)
#pragma unroll
        for (int c = 0; c < 4; ++c) red[c][threadIdx.x] += red[c][threadIdx.x + o];
      __syncthreads();
    }
    if (threadIdx.x == 0)
#pragma unroll
      for (int c = 0; c < 4; ++c) s.part[(size_t)blockIdx.x * 4 + c] = red[c][0];
  }
}

// Residual-norm partial sums alone (src/fv.cc:1822-1841), same reduction shape as k_update.
__global__ void k_norm_part(MeshView m, StateView s, const int* __restrict__ done) {
  if (*done) return;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int nv = m.nv;
  double nrm[4] = {0.0, 0.0, 0.0, 0.0};
  if (i < nv) {
    const double ia = m.inv_area[i], w = m.pweight[i];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      double q = s.R[c * nv + i] * ia;
      nrm[c] = q * q * w;
    }
  }
  __shared__ double red[4][kBlock];
#pragma unroll
  for (int c = 0; c < 4; ++c) red[c][threadIdx.x] = nrm[c];
  __syncthreads();
  for (int o = kBlock / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o)
#pragma unroll
      for (int c = 0; c < 4; ++c) red[c][threadIdx.x] += red[c][threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0)
#pragma unroll
    for (int c = 0; c < 4; ++c) s.part[(size_t)blockIdx.x * 4 + c] = red[c][0];
}

// Norm finalisation (src/fv.cc:1846-1876): one block sums the partials in a fixed order.
__global__ void k_norm_final(StateView s, int nblocks, int nv_total, Scalars* sc, int use_sc_iter, long long iter,
                             const int* __restrict__ done) {
  if (*done) return;
  __shared__ double red[4][kBlock];
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  // unrolled so that several partials' loads are in flight before the ordered adds
#pragma unroll 8
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[c] += s.part[(size_t)b * 4 + c];
#pragma unroll
  for (int c = 0; c < 4; ++c) red[c][threadIdx.x] = acc[c];
  __syncthreads();
  for (int o = kBlock / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o)
#pragma unroll
      for (int c = 0; c < 4; ++c) red[c][threadIdx.x] += red[c][threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    double n0 = sqrt(red[0][0]) / nv_total, n1 = sqrt(red[1][0]) / nv_total;
    double n2 = sqrt(red[2][0]) / nv_total, n3 = sqrt(red[3][0]) / nv_total;
    double total = sqrt(n0 * n0 + (n1 * n1 + n2 * n2 + 0.0) + n3 * n3);
    long long it = use_sc_iter ? sc->iter : iter;
    if (it == 0) {
      sc->rtotal0 = total;
      if (sc->rtotal0 == 0.0) sc->rtotal0 = 1.0;
    }
    sc->rnorm[0] = n0; sc->rnorm[1] = n1; sc->rnorm[2] = n2; sc->rnorm[3] = n3;
    sc->rtotal = total / sc->rtotal0;
  }
}

// End of a solve-loop iteration (src/fv.cc:2307-2343).
__global__ void k_step_end(Control ctl, Scalars* sc, const int* __restrict__ done) {
  if (*done) return;
  sc->iter += 1;
  sc->elapsed += sc->dt_global;
  if (sc->reached && ctl.time_mode == 1) {
    sc->counter += 1;
    sc->reached = 0;
  }
}

// Kinetic-energy and entropy integrals (src/fv.cc:2186-2203), block partials.
__global__ void k_global(Params k, MeshView m, StateView s) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  double ke = 0.0, en = 0.0;
  if (i < m.nv) {
    Prim q = load_prim(s, i);
    double w = m.pweight[i], A = m.dcarea[i];
    double rho = density(k, q);
    ke = (0.5 * rho * (q.u * q.u + q.v * q.v) * A) * w;
    en = (-rho * entropy_fn(k, q) / (k.gamma - 1.0)) * A * w;
  }
  __shared__ double red[2][kBlock];
  red[0][threadIdx.x] = ke;
  red[1][threadIdx.x] = en;
  __syncthreads();
  for (int o = kBlock / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) {
      red[0][threadIdx.x] += red[0][threadIdx.x + o];
      red[1][threadIdx.x] += red[1][threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) { s.part[(size_t)blockIdx.x * 4] = red[0][0]; s.part[(size_t)blockIdx.x * 4 + 1] = red[1][0]; }
}

// ------------------------------------------------------------ forces
// compute_forces (src/force.cc:116-219) for the force of block f: pressure
// force sum over faces of 0.5 (p0 + p1) n and, for Navier-Stokes, the viscous
// stress from the vertex gradients of u and v recovered from those of the
// entropy variables.  Face record (d, dq, k0, k1): the face's device index, and
// -- as the reference applies the condition of bface[f] with f the force
// index -- the device index of bface[f] (-1: no condition) with the value
// slots its evaluation uses.  Fixed-order block reduction.
__global__ void k_forces(Params k, MeshView m, StateView s, const int4* __restrict__ faces,
                         const int* __restrict__ off, double* __restrict__ out) {
  const int f = blockIdx.x;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (int j = off[f] + threadIdx.x; j < off[f + 1]; j += blockDim.x) {
    const int4 r = faces[j];
    const int d = r.x, dq = r.y;
    const int v0 = m.b_v0[d], v1 = m.b_v1[d];
    const double nx = m.b_nx[d], ny = m.b_ny[d];
    Prim s0 = load_prim(s, v0), s1 = load_prim(s, v1);
    if (dq >= 0) {
      bc_apply1(m.b_kind[dq], m.b_adiab[dq], m.b_val + (size_t)dq * 10 + 5 * r.z, m.b_nx[dq], m.b_ny[dq], s0);
      bc_apply1(m.b_kind[dq], m.b_adiab[dq], m.b_val + (size_t)dq * 10 + 5 * r.w, m.b_nx[dq], m.b_ny[dq], s1);
    }
    const double pr = 0.5 * (s0.p + s1.p);
    acc[0] += nx * pr;
    acc[1] += ny * pr;
    if (k.model == 1) {
      const Ent e0 = prim2ent(k, s0), e1 = prim2ent(k, s1);
      const double T = (s0.T + s1.T) / 2.0;
      const double mu = viscosity(k, T);
      const double f0 = 1.0 / e0.l, f1 = 1.0 / e1.l;
      const D4 ga[2] = {ld4(s.G + 2 * (size_t)v0), ld4(s.G + 2 * (size_t)v1)};
      const D4 gb[2] = {ld4(s.G + 2 * (size_t)v0 + 1), ld4(s.G + 2 * (size_t)v1 + 1)};
      auto g = [&](int c, int w) {   // c = 2 .. 7
        const D4 &a = ga[w], &b = gb[w];
        return c == 2 ? a.z : c == 3 ? a.w : c == 4 ? b.x : c == 5 ? b.y : c == 6 ? b.z : b.w;
      };
      // u = -V2 / V5: grad u = -grad V2 / V5 + V2 grad V5 / V5^2 (src/force.cc:169-179)
      const double ux0 = g(2, 0) * -f0 + g(6, 0) * (f0 * e0.vx / e0.l), uy0 = g(3, 0) * -f0 + g(7, 0) * (f0 * e0.vx / e0.l);
      const double ux1 = g(2, 1) * -f1 + g(6, 1) * (f1 * e1.vx / e1.l), uy1 = g(3, 1) * -f1 + g(7, 1) * (f1 * e1.vx / e1.l);
      const double vx0 = g(4, 0) * -f0 + g(6, 0) * (f0 * e0.vy / e0.l), vy0 = g(5, 0) * -f0 + g(7, 0) * (f0 * e0.vy / e0.l);
      const double vx1 = g(4, 1) * -f1 + g(6, 1) * (f1 * e1.vy / e1.l), vy1 = g(5, 1) * -f1 + g(7, 1) * (f1 * e1.vy / e1.l);
      const double gux = ux0 * 0.5 + ux1 * 0.5, guy = uy0 * 0.5 + uy1 * 0.5;
      const double gvx = vx0 * 0.5 + vx1 * 0.5, gvy = vy0 * 0.5 + vy1 * 0.5;
      const double div = gux + gvy;
      const double sxx = 2.0 * mu * (gux - (1.0 / 3.0) * div);
      const double syy = 2.0 * mu * (gvy - (1.0 / 3.0) * div);
      const double sxy = mu * (guy + gvx);
      acc[2] += -(sxx * nx + sxy * ny);
      acc[3] += -(sxy * nx + syy * ny);
    }
  }
  __shared__ double red[4][kBlock];
#pragma unroll
  for (int c = 0; c < 4; ++c) red[c][threadIdx.x] = acc[c];
  __syncthreads();
  for (int o = kBlock / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o)
#pragma unroll
      for (int c = 0; c < 4; ++c) red[c][threadIdx.x] += red[c][threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0)
#pragma unroll
    for (int c = 0; c < 4; ++c) out[4 * f + c] = red[c][0];
}

// ------------------------------------------------------------ MC moments
// increment_moments (src/fv.cc:595-694) for the k-th sample of a group, one
// thread per vertex.  Moment arrays are [var][vertex] with the per-vertex
// record of the reference's reduce_moments packing: PrimVar (T, p, u, v, w)
// then density, mach, entropy, vorticity as selected by `extras` (bits 0-3).
// Vorticity (src/material.h:623-627) reads the entropy-variable gradients G of
// the last gradient pass: V2 = 2 beta u, V3 = 2 beta v, V5 = -2 beta.
__global__ void k_moments_increment(Params k, int nv, StateView s, int extras, int nvar, long long kk,
                                    double* __restrict__ fm, double* __restrict__ sm, double* __restrict__ m2) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nv) return;
  Prim q = load_prim(s, i);
  double x[9];
  x[0] = q.T; x[1] = q.p; x[2] = q.u; x[3] = q.v; x[4] = 0.0;
  int j = 5;
  if (extras & 1) x[j++] = density(k, q);
  if (extras & 2) x[j++] = sqrt(q.u * q.u + q.v * q.v) / sound_speed(k, q);
  if (extras & 4) x[j++] = entropy_fn(k, q);
  if (extras & 8) {
    const D4 a = ld4(s.G + 2 * (size_t)i), b = ld4(s.G + 2 * (size_t)i + 1);
    x[j++] = k.R * q.T * (b.x + q.v * b.z - a.w - q.u * b.w);
  }
  const double K = (double)kk, c1 = 1.0 / K, c2 = (K - 1.0) / K;
  for (int c = 0; c < nvar; ++c) {
    const size_t o = (size_t)c * nv + i;
    const double xc = x[c];
    if (kk == 1) {
      fm[o] = xc; sm[o] = xc * xc; m2[o] = 0.0;
    } else {
      const double mkm1 = fm[o];
      const double mk = c < 5 ? xc * c1 + mkm1 * c2 : mkm1 + (xc - mkm1) / K;   // PrimVar::equ / scalar form
      fm[o] = mk;
      sm[o] += xc * xc;
      m2[o] += (xc - mkm1) * (xc - mk);
    }
  }
}

// The three moment arrays [nvar][nv] of an instance -> [vertex][nvar] in the caller's order.
__global__ void k_moments_out(int nv, int nvar, const double* __restrict__ mom, const int* __restrict__ old_of_new,
                              double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nv) return;
  const size_t n = (size_t)nvar * nv * blockIdx.y;
  double* o = out + n + (size_t)nvar * old_of_new[i];
  for (int c = 0; c < nvar; ++c) o[c] = mom[n + (size_t)c * nv + i];
}

// One received group of reduce_moments (src/reduce_moments.cc:36-113).
__global__ void k_moments_merge(size_t n, double fact1, double fact2, double* __restrict__ fm,
                                double* __restrict__ sm, double* __restrict__ m2, const double* __restrict__ fo,
                                const double* __restrict__ so, const double* __restrict__ mo) {
  size_t j = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (j >= n) return;
  const double diff = fo[j] - fm[j];
  fm[j] += diff * fact1;
  m2[j] += mo[j] + (diff * diff) * fact2;
  sm[j] += so[j];
}

// Final scaling of reduce_moments (src/reduce_moments.cc:115-141).
__global__ void k_moments_scale(size_t n, double fact3, double fact4, double* __restrict__ sm,
                                double* __restrict__ m2) {
  size_t j = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (j >= n) return;
  m2[j] *= fact3;
  sm[j] *= fact4;
}

// ---- domain decomposition (tg_part_*): halo exchange and the exchanged step scalars

// Packs 8 doubles per listed vertex into out[8 * i + c]: a state's record S, T and V1 (the
// last two unused), or the gradient's two records.
__global__ void k_halo_pack(int n, const int* __restrict__ idx, StateView s, int grad, double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 2 * n) return;
  const int v = idx[i >> 1];
  D4 q{0.0, 0.0, 0.0, 0.0};
  if (grad) q = ld4(s.G + 2 * (size_t)v + (i & 1));
  else if ((i & 1) == 0) q = ld4(s.S + v);
  else { q.x = s.T[v]; q.y = s.V1[v]; }
  double* o = out + 4 * (size_t)i;     // a caller's buffer: 8-byte aligned
  o[0] = q.x; o[1] = q.y; o[2] = q.z; o[3] = q.w;
}

__global__ void k_halo_unpack(int n, const int* __restrict__ idx, StateView s, int grad, const double* __restrict__ in) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 2 * n) return;
  const int v = idx[i >> 1];
  const double* q = in + 4 * (size_t)i;
  if (grad) st4(s.G + 2 * (size_t)v + (i & 1), q[0], q[1], q[2], q[3]);
  else if ((i & 1) == 0) st4(s.S + v, q[0], q[1], q[2], q[3]);
  else { s.T[v] = q[0]; s.V1[v] = q[1]; }
}

// After the first-stage dt pass of tg_part_prime: its minimum is the next step's.
__global__ void k_part_primed(Scalars* sc) {
  sc->dtmin_next = sc->dtmin_bits;
  sc->dtmin_bits = 0x7ff0000000000000ull;
  sc->dt_next = 1;
}

// A partition's contribution to the step exchange: its running dt minimum (as
// bits; positive doubles order like their bit patterns) and its residual-norm sums.
__global__ void k_part_export(const Scalars* sc, unsigned long long* out) {
  out[0] = sc->dtmin_next;
#pragma unroll
  for (int c = 0; c < 4; ++c) out[1 + c] = (unsigned long long)__double_as_longlong(sc->rsq[c]);
}

// All partitions' contributions, combined in partition order so every partition
// forms the same dt and norms: the dt minimum of the whole mesh and, after a
// step, the norms over the whole mesh with nv_total its vertex count (the
// reference's MPI reductions, src/fv.cc:1602, src/reduce_res_norm.cc:25).
__global__ void k_part_import(Scalars* sc, const unsigned long long* __restrict__ all, int n_parts, int nv_total,
                              int norms) {
  unsigned long long m = all[0];
  double sum4[4] = {0.0, 0.0, 0.0, 0.0};
  for (int q = 0; q < n_parts; ++q) {
    m = all[5 * q] < m ? all[5 * q] : m;
#pragma unroll
    for (int c = 0; c < 4; ++c) sum4[c] += __longlong_as_double((long long)all[5 * q + 1 + c]);
  }
  sc->dtmin_next = m;
  if (norms) set_norms(sc, sum4, nv_total, sc->iter == 1);
}

// Owned vertices of a partition -> PrimVar records in local order (tg_get_state).
__global__ void k_part_state_out(int n, StateView s, double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double* q = out + 5 * (size_t)i;
  const Prim r = load_prim(s, i);
  q[0] = r.T; q[1] = r.p; q[2] = r.u; q[3] = r.v; q[4] = 0.0;
}

}  // namespace tg
