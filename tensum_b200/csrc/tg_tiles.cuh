// tg_tiles.cuh -- tiled stage kernels of the FP64 single-solve path.
//
// A tile is a contiguous range of owned vertices (Hilbert order) plus every
// vertex one edge away (periodic copies' neighbourhoods included).  A CTA
// gathers a tile's vertex records and gather lists into shared memory,
// computes each edge flux of the tile once, and every owned vertex sums its
// edge fluxes in a fixed order (deterministic; no flux buffer in HBM).
//
// The gathers are a chain of dependent memory accesses (tile record -> vertex
// indices -> records), and with one tile per CTA a warp spent 60 % of its life
// waiting on them.  So a CTA walks tiles blockIdx.x, blockIdx.x + gridDim.x, ...
// (the grid fills the chip once) and runs the chain of the next tile behind the
// current one: its record and indices are read into registers during the edge
// loop, its vertex records are copied while the owned vertices gather and
// update.
//
// k_tile_grad   compute_gradients (src/fv.cc:699-1059) for the owned vertices.
// k_tile_flux   compute_inviscid_residual + residual assembly
//               (src/fv.cc:1066-1192, 1467-1494) and, in MODE_UPDATE, the
//               RK update (src/fv.cc:1641-1652); the last stage also forms the
//               next step's local time step (src/fv.cc:1499-1598) and the
//               residual norm; writes the new state into the next buffer.
#pragma once

#include "tg_kernels.cuh"

#ifndef TG_TILE_OWNED
#define TG_TILE_OWNED 128      // most owned vertices per tile (<= kTileThreads)
#endif
#ifndef TG_TILE_LCAP
#define TG_TILE_LCAP 256       // local (owned + halo) vertices per tile
#endif
#ifndef TG_TILE_ECAP
#define TG_TILE_ECAP 512       // edges per tile
#endif
// resident flux CTAs per SM the register budget is sized for: TeCNO fluxes / central fluxes,
// and gradient CTAs.  With the next tile's loads behind the current one, fewer CTAs with
// more registers win: KH 1025^2 steps of TeCNO-Rusanov / KEPEC / KEP in us with
// (TeCNO, central, gradient) CTAs (4, 7, 7): 732 / 274 / 246, (4, 6, 5): 678 / 256 / 246,
// (4, 5, 6): 724 / 271 / 264, (3, 5, 5): 706 / 271 / 266; gradient pass 78 / 68 / 60 / 59 us
// with 7 (spills) / 3 / 5 / 4.  With the central fluxes' normals staged too,
// CTAs of a step's earlier / last updates 6 / 6, 6 / 5, 5 / 5: KEPEC 240 / 227 / 243, KEP 236 /
// 234 / 236, Roe-EC 259 / 248 / 251.
#ifndef TG_FLUX_MINB
#define TG_FLUX_MINB 4
#endif
#ifndef TG_FLUX_MINB_CENTRAL
#define TG_FLUX_MINB_CENTRAL 6
#endif
#ifndef TG_FLUX_MINB_CENTRAL_LAST
#define TG_FLUX_MINB_CENTRAL_LAST 5
#endif
#ifndef TG_GRAD_MINB
#define TG_GRAD_MINB 5
#endif

namespace tg {

// One tile: its ranges in the local vertex table (L vertices, nown of them owned, packed
// L | nown << 16), the edge arrays, the owned vertices, the list offsets and the gather
// lists (start a multiple of 8); bit 30 of nent: some owned vertex has boundary or viscous
// entries.  A partition's records are in its tile order: frontier tiles first.
struct alignas(32) TileRec {
  int l0, sizes, e0, NE, vb, rel, cb, nent;
  __host__ __device__ int L() const { return sizes & 0xffff; }
  __host__ __device__ int nown() const { return sizes >> 16; }
};
constexpr int kTileBnd = 1 << 30;

struct TileView {
  const TileRec* rec;
  const int* lv;                // local vertex table (owned vertices first)
  const unsigned int* ab;       // local endpoints per tile edge
  const double2* u;             // unit normal per tile edge
  const double2* n;             // normal
  const double* ar;             // |n|
  const double* r;              // radius per tile edge (axisymmetric runs)
  const unsigned short* crel;   // per tile (owned + 1) offsets into its lists, at rel
  const unsigned short* cent;   // (tile edge << 1) | side
  const double2* gjg;           // the same entries in lane order for the gradients: weights,
  const unsigned int* gji;      // and other | self << 16 (local vertices)
  const double2* xy;            // vertex coordinates (device order)
  // a launch works on tiles base .. base + count; total is the number of CTAs of every
  // launch of the pass and pbase this launch's first one (norm partials)
  int base, count, pbase, total;
};

__device__ __forceinline__ TileRec load_rec(const TileView& t, int i) {
  const int4* p = reinterpret_cast<const int4*>(t.rec + t.base + i);
  const int4 a = __ldg(p), b = __ldg(p + 1);
  return TileRec{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
}
// Global index of local vertex i of a tile (0 past its end): only the halo is tabled.
__device__ __forceinline__ int local_vertex(const TileView& t, const TileRec& R, int i) {
  return i < R.nown() ? R.vb + i : (i < R.L() ? t.lv[R.l0 + i] : 0);
}

#ifndef TG_TILE_THREADS
#define TG_TILE_THREADS 128    // threads per tile CTA (>= TG_TILE_OWNED)
#endif
constexpr int kTileThreads = TG_TILE_THREADS;

// Owned vertices per tile of a mesh of nv vertices on a chip that holds `ctas` flux CTAs at
// once.  A large mesh takes full tiles (the smallest halo).  Where full tiles would fill
// the chip less than twice, they are made smaller so that its one or two rounds are full:
// a CTA's time is a chain of latencies and grows with its edges per thread, so a chip half
// filled with full tiles, or a nearly empty second round, costs as much as a full one.
// Below 32 the halo outweighs the edges.  Steps in us on n^2 vertices with 32 / 64 / 96 / 112 / 128
// owned, the rule's choice last.  TeCNO-Roe: 65^2 31.8 / 31.5 / 33.8 / 37.0 / 37.3, 32; 129^2 37.6 /
// 41.4 / 51.5 / 43.8 / 43.6, 32; 193^2 62.1 / 46.4 / 53.3 / 55.9 / 54.5, 64; 225^2 81.5 / 70.1 / 54.0 /
// 58.2 / 60.6, 96; 257^2 92.9 / 74.4 / 70.4 / 66.0 / 63.6, 112; 300^2 109 / 88.8 / 83.4 / 88.5 / 82.8,
// 80 (86.5); 321^2 129 / 100 / 92.5 / 91.4 / 94.5, 96; 387^2 173 / 132 / 122 / 118 / 109, 128.
// Where it is not the best, the chip is filled but the halo larger.  The central fluxes are sized
// for their earlier updates (6 CTAs per SM); the last one runs 5, so its last round can be nearly
// empty (257^2, 387^2).  KEPEC: 65^2 19.2 / 18.8 / 19.7 / 21.1 / 20.8, 32; 300^2 47.7 / 37.8 / 37.1 /
// 35.8 / 33.3, 112; 387^2 66.9 / 50.4 / 47.0 / 46.4 / 46.6, 96; 450^2 85.3 / 63.3 / 57.3 / 55.6 / 55.2,
// 128.  Roe-EC: 257^2 24.8 / 21.9 / 20.2 / 20.9 / 21.0, 80 (21.4); 387^2 68.8 / 52.2 / 48.4 / 47.9 /
// 48.2, 96; 450^2 87.6 / 65.0 / 59.1 / 57.9 / 60.6, 128.
inline int tile_owned(long nv, int ctas) {
  const long full = (long)ctas * TG_TILE_OWNED, rounds = (nv + full - 1) / full;
  if (rounds > 2) return TG_TILE_OWNED;
  const long want = (nv + ctas * rounds - 1) / (ctas * rounds);
  return (int)(want <= 32 ? 32 : want >= TG_TILE_OWNED ? TG_TILE_OWNED : (want + 15) / 16 * 16);
}

// ---- asynchronous global -> shared copies (sm_80+ cp.async)
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// ---------------------------------------------------------------- gradients
// Entropy-variable gradients of the owned vertices.  The next tile's S and V1 are read
// into registers and its gather entries (weights and local indices in lane order, so
// copies and reads are consecutive words) into the other half of a double buffer while
// this tile is summed; the records go to shared memory as the pairs (V2, V3), (V1, V5).
__host__ __device__ inline size_t tile_grad_smem(int lmax, int cmax) {
  return (size_t)lmax * 2 * sizeof(double2) + 2 * (size_t)cmax * (sizeof(double2) + sizeof(unsigned int));
}

struct GradVertex {
  D4 q;
  double V1;
  double2 w;     // V2, V3 (strong conditions)
};
__device__ __forceinline__ GradVertex load_grad_vertex(const Params& k, const StateView& s, int g) {
  GradVertex x;
  x.q = ld4(s.S + g);
  x.V1 = s.V1[g];
  x.w = k.strong ? s.W23[g] : make_double2(0.0, 0.0);
  return x;
}

// The pass over a launch's tiles by its first `ctas` CTAs.
__device__ __forceinline__ void tile_grad(const Params& k, const MeshView& m, const TileView& t, const StateView& s,
                                          int lmax, int cmax, const int* done, int ctas) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x;
  double2* sA = reinterpret_cast<double2*>(smem);             // (V2, V3)
  double2* sB = sA + lmax;                                    // (V1, V5)
  double2* sE0 = sB + lmax;                                   // weights per entry, two buffers
  unsigned int* sI0 = reinterpret_cast<unsigned int*>(sE0 + 2 * (size_t)cmax);   // local indices per entry
  int at = blockIdx.x;
  TileRec R = load_rec(t, at);
  auto entries = [&](const TileRec& r, int buf) {
    const int n = r.nent & ~kTileBnd;
    double2* e = sE0 + (size_t)buf * cmax;
    unsigned int* i4 = sI0 + (size_t)buf * cmax;
    for (int i = tid; i < n; i += kTileThreads) cp_async16(e + i, t.gjg + r.cb + i);
    for (int i = tid; 4 * i < n; i += kTileThreads) cp_async16(i4 + 4 * i, t.gji + r.cb + 4 * i);
    cp_async_commit();
  };
  entries(R, 0);
  const int v0 = local_vertex(t, R, tid), v1 = local_vertex(t, R, tid + kTileThreads);
  pdl_wait();
  const int stop = *done;
  GradVertex x0 = load_grad_vertex(k, s, v0);
  GradVertex x1 = load_grad_vertex(k, s, v1);
  if (stop) {
    cp_async_wait<0>();
    return;
  }
  for (int buf = 0;; buf ^= 1) {
    const unsigned short* rel = t.crel + R.rel;
    const int j0 = tid < R.nown() ? rel[tid] : 0, deg = tid < R.nown() ? rel[tid + 1] - j0 : 0;
    const double f = tid < R.nown() ? m.inv6mc[R.vb + tid] : 0.0;
    at += ctas;
    const bool more = at < t.count;
    const TileRec N = more ? load_rec(t, at) : R;
    auto put = [&](int i, const GradVertex& x) {
      if (i >= R.L()) return;
      sA[i] = k.strong ? x.w : make_double2(-x.q.w * x.q.x, -x.q.w * x.q.y);
      sB[i] = make_double2(x.V1, x.q.w);
    };
    put(tid, x0);
    put(tid + kTileThreads, x1);
    for (int i = tid + 2 * kTileThreads; i < R.L(); i += kTileThreads)
      put(i, load_grad_vertex(k, s, local_vertex(t, R, i)));
    const double2 *sE = sE0 + (size_t)buf * cmax;
    const unsigned int* sI = sI0 + (size_t)buf * cmax;
    cp_async_wait<0>();
    __syncthreads();
    if (more) {
      entries(N, buf ^ 1);
      x0 = load_grad_vertex(k, s, local_vertex(t, N, tid));
      x1 = load_grad_vertex(k, s, local_vertex(t, N, tid + kTileThreads));
    }
    else pdl_trigger();   // this late, so that the flux pass's CTAs do not take this pass's place
    const double2 wa = sA[tid < R.nown() ? tid : 0], wb = sB[tid < R.nown() ? tid : 0];
    double acc[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[c] = 0.0;
    int p = __shfl_sync(0xffffffffu, j0, 0);       // the warp's first entry
    const unsigned below = (1u << (tid & 31)) - 1u;
    for (int n = 0;; ++n) {
      const unsigned have = __ballot_sync(0xffffffffu, n < deg);
      if (!have) break;
      if (n < deg) {
        const int e = p + __popc(have & below);
        const unsigned idx = sI[e];
        const double2 g = sE[e];
        const int o = idx & 0xffff, self = idx >> 16;
        const double2 oa = sA[o], ob = sB[o];
        double2 ca = wa, cb = wb;
        if (self != tid) { ca = sA[self]; cb = sB[self]; }   // a periodic copy's entry
        const double d1 = ob.x - cb.x, d2 = oa.x - ca.x, d3 = oa.y - ca.y, d5 = ob.y - cb.y;
        acc[0] += g.x * d1; acc[1] += g.y * d1;
        acc[2] += g.x * d2; acc[3] += g.y * d2;
        acc[4] += g.x * d3; acc[5] += g.y * d3;
        acc[6] += g.x * d5; acc[7] += g.y * d5;
      }
      p += __popc(have);
    }
    if (tid < R.nown()) {
      const int v = R.vb + tid;
      if (R.nent & kTileBnd)
        for (int j = m.cb_off[v]; j < m.cb_off[v + 1]; ++j) {
          const int ent = m.cb_ent[j];
          if ((ent & 3) != 1) continue;
          const int idx = ent >> 2;
          double dW[4];
          bface_grad_corr(k, m, s, idx, dW);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            acc[2 * c] += m.b_nx[idx] * dW[c];
            acc[2 * c + 1] += m.b_ny[idx] * dW[c];
          }
        }
      st4(s.G + 2 * (size_t)v, acc[0] * f, acc[1] * f, acc[2] * f, acc[3] * f);
      st4(s.G + 2 * (size_t)v + 1, acc[4] * f, acc[5] * f, acc[6] * f, acc[7] * f);
    }
    if (!more) break;
    R = N;
    __syncthreads();      // the records are rewritten for the next tile
  }
}

__global__ void __launch_bounds__(kTileThreads, TG_GRAD_MINB)
    k_tile_grad(Params k, MeshView m, TileView t, StateView s, int lmax, int cmax, const int* done) {
  tile_grad(k, m, t, s, lmax, cmax, done, gridDim.x);
}

// The gradients of a mesh that fills the chip at most once, with the boundary faces and
// viscous units of the same state (nvu, 0 in inviscid runs) by the CTAs from `ctas` on.  They
// depend on nothing but the state, take the places that the tiles leave, and wait for it like
// the tiles: launches of their own would either start after the gradients or read the state
// without a wait that makes it visible to them.  64 steps and four wall forces on the 128 x 256
// cylinder 7.00 (own launches, no wait) -> 6.38 ms.
template <int FLUX, int RECON>
__global__ void __launch_bounds__(kTileThreads, TG_GRAD_MINB)
    k_stage_head(Params k, MeshView m, TileView t, StateView s, int lmax, int cmax, const int* done,
                 int ctas, int nvu) {
  if (blockIdx.x < ctas) {
    tile_grad(k, m, t, s, lmax, cmax, done, ctas);
    return;
  }
  const int i = (blockIdx.x - ctas) * kTileThreads + threadIdx.x;
  pdl_wait();
  if (*done) return;
  if (i < 2 * m.nb) bflux_one<FLUX, RECON>(k, m, s, i);
  else if (i - 2 * m.nb < nvu) viscous_one(k, m, s, i - 2 * m.nb);
}

// --------------------------------------------------------------------- fluxes
// MODE_LAST is a step's last update: it also forms the residual norm and the next local time
// step.  It is a kernel of its own, except for TeCNO-Roe, whose every update runs it (norm
// tells the last one): without that code the others spill less, but Roe's earlier stages
// come out slower.  Steps on 1025^2 in us, one kernel / two: TeCNO-Rusanov 651 / 638, KEPEC
// 246 / 227, Roe-EC 261 / 248 (both with the staged normals), TeCNO-Roe 657 / 677.
enum : int { MODE_RESIDUAL = 0, MODE_UPDATE = 1, MODE_LAST = 2 };
template <int FLUX>
__host__ __device__ constexpr bool own_last() {
  return FLUX != FLUX_TECNO_ROE;
}


template <int FLUX>
__host__ __device__ constexpr bool is_tecno() {
  return FLUX == FLUX_TECNO_ROE || FLUX == FLUX_TECNO_RUSANOV;
}
template <int FLUX, int RECON>
__host__ __device__ constexpr bool flux_needs_grad() {
  return is_tecno<FLUX>() && RECON != RECON_FIRST;
}

// Shared memory of a staged vertex: the pairs (u, v) and (p, V5), one single (V1 for the
// TeCNO fluxes, T for KEP, sqrt(-V5) for Roe-EC), and for the gradient fluxes four pairs of
// the gradient and the coordinates.
template <int FLUX>
__host__ __device__ constexpr int vertex_singles() {
  return is_tecno<FLUX>() || FLUX == FLUX_KEP || FLUX == FLUX_ROE_EC ? 1 : 0;
}
template <int FLUX, int RECON>
__host__ __device__ constexpr int vertex_pairs() {
  return 2 + (flux_needs_grad<FLUX, RECON>() ? 5 : 0);
}

template <int FLUX>
__device__ __forceinline__ VRec load_vrec(const double2* sA, const double2* sB, const double* s1, int i) {
  VRec q;
  const double2 a = sA[i], b = sB[i];
  q.u = a.x; q.v = a.y; q.p = b.x; q.V5 = b.y;
  q.V1 = is_tecno<FLUX>() ? s1[i] : 0.0;
  q.x = (FLUX == FLUX_KEP || FLUX == FLUX_ROE_EC) ? s1[i] : 0.0;
  return q;
}

// Whether a stage update forms V5 alone of the entropy variables: the central fluxes
// read no other, and an inviscid run forms no gradients inside its steps.  Strong
// conditions keep all four: they reset the primitive state after the update and leave the
// entropy variables of the reset vertices as the update formed them, as the reference does.
template <int FLUX>
__device__ __forceinline__ bool w3_only(const Params& k) {
  return !is_tecno<FLUX>() && k.model == 0 && !k.strong;
}

// Sums of four values and a minimum over the block's warps, valid in thread 0
// (fixed order).
__device__ __forceinline__ void block_sum4_min(double* x, unsigned long long& lo) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int c = 0; c < 4; ++c) x[c] += __shfl_xor_sync(0xffffffffu, x[c], o);
  lo = warp_min_u64(lo);
  __shared__ double ws[kTileThreads / 32][4];
  __shared__ unsigned long long wl[kTileThreads / 32];
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int c = 0; c < 4; ++c) ws[w][c] = x[c];
    wl[w] = lo;
  }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int i = 1; i < kTileThreads / 32; ++i) {
#pragma unroll
      for (int c = 0; c < 4; ++c) x[c] += ws[i][c];
      lo = wl[i] < lo ? wl[i] : lo;
    }
}

// Shared-memory layout of k_tile_flux, in bytes (host and device agree on it).
template <int FLUX, int RECON>
struct FluxSmem {
  size_t xy, g, f, n, ab, single, list, ssw, bytes;
  static constexpr bool kStage = !is_tecno<FLUX>();
  __host__ __device__ FluxSmem(int lmax, int emax, int cmax, bool dt) {
    size_t o = 2 * (size_t)lmax * sizeof(double2);            // (u, v), (p, V5)
    g = o;
    if (flux_needs_grad<FLUX, RECON>()) o += 4 * (size_t)lmax * sizeof(double2);
    xy = o;
    if (flux_needs_grad<FLUX, RECON>()) o += (size_t)lmax * sizeof(double2);
    f = o;                                                    // (mass, x), (y, energy) per edge
    o += 2 * (size_t)emax * sizeof(double2);
    n = o;                                                    // normals (TeCNO: where dt is fused)
    if (dt || kStage) o += (size_t)emax * sizeof(double2);
    ab = o;                                                   // central fluxes: endpoints
    if (kStage) o += (((size_t)emax + 3) & ~(size_t)3) * sizeof(unsigned int);
    list = o;                                                 // gather lists, two buffers
    o += 2 * (size_t)cmax * sizeof(unsigned short);
    single = o;
    o += (size_t)(vertex_singles<FLUX>() * lmax) * sizeof(double);
    ssw = o;
    if (FLUX == FLUX_TECNO_ROE) o += (size_t)lmax * sizeof(int);
    const size_t red = 4 * kTileThreads * sizeof(double);     // norm_and_step_end's buffer
    bytes = o > red ? o : red;
  }
};

template <int FLUX, int RECON, int MODE>
__global__ void __launch_bounds__(kTileThreads, is_tecno<FLUX>()    ? TG_FLUX_MINB
                                                : MODE == MODE_LAST ? TG_FLUX_MINB_CENTRAL_LAST
                                                                    : TG_FLUX_MINB_CENTRAL)
    k_tile_flux(Params k, MeshView m, TileView t, StateView s, Control ctl, Scalars* sc, int r, int norm,
                StateView out, int lmax, int emax, int cmax, const int* done) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr bool kGrad = flux_needs_grad<FLUX, RECON>();
  // The central fluxes are short and linear in the normal: a tile's normals (no |n|) and
  // endpoints are copied with its records, 20 bytes an edge instead of 28, and the next dt
  // finds them there.  The TeCNO fluxes leave no shared memory for that and read an edge
  // ahead into registers.
  constexpr bool kStage = !is_tecno<FLUX>();
  constexpr bool kRoe = (FLUX == FLUX_TECNO_ROE);
  constexpr bool kUpdate = MODE != MODE_RESIDUAL;
  const bool do_norm = MODE == MODE_LAST && (own_last<FLUX>() || norm);
  const int nv = m.nv, tid = threadIdx.x;
  const FluxSmem<FLUX, RECON> lay(lmax, emax, cmax, MODE == MODE_LAST && k.fuse_dt);
  double2* sA = reinterpret_cast<double2*>(smem);
  double2* sB = sA + lmax;
  double2* sG = reinterpret_cast<double2*>(smem + lay.g);              // 4 * lmax
  double2* sX = reinterpret_cast<double2*>(smem + lay.xy);
  double2* sF = reinterpret_cast<double2*>(smem + lay.f);
  double2* sF2 = sF + emax;
  double2* sN = reinterpret_cast<double2*>(smem + lay.n);
  unsigned int* sAB = reinterpret_cast<unsigned int*>(smem + lay.ab);
  double* s1 = reinterpret_cast<double*>(smem + lay.single);
  unsigned short* sC = reinterpret_cast<unsigned short*>(smem + lay.list);
  int* sS = reinterpret_cast<int*>(smem + lay.ssw);                    // Liou switch of the local vertices

  int at = blockIdx.x;
  TileRec R = load_rec(t, at);
  auto stage_vertex = [&](int i, int g) {
    const double2* q = reinterpret_cast<const double2*>(s.S + g);
    cp_async16(sA + i, q);
    cp_async16(sB + i, q + 1);
    if (is_tecno<FLUX>()) cp_async8(s1 + i, s.V1 + g);
    if (FLUX == FLUX_KEP) cp_async8(s1 + i, s.T + g);
    if (kGrad) {
      const double2* q = reinterpret_cast<const double2*>(s.G + 2 * (size_t)g);
#pragma unroll
      for (int c = 0; c < 4; ++c) cp_async16(sG + c * lmax + i, q + c);
      cp_async16(sX + i, t.xy + g);
    }
    if (kRoe && k.liou) cp_async4(sS + i, s.ssw + g);
  };
  auto stage_normals = [&](const TileRec& T) {
    for (int le = tid; le < T.NE; le += kTileThreads) cp_async16(sN + le, t.n + T.e0 + le);
  };
  // copies a tile's vertex records (global ids of the thread's first two given), endpoints
  // and lists
  auto stage = [&](const TileRec& T, int g0, int g1, int buf) {
    if (kStage)
      for (int le = tid; le < T.NE; le += kTileThreads) cp_async4(sAB + le, t.ab + T.e0 + le);
    if (tid < T.L()) stage_vertex(tid, g0);
    if (tid + kTileThreads < T.L()) stage_vertex(tid + kTileThreads, g1);
    for (int i = tid + 2 * kTileThreads; i < T.L(); i += kTileThreads) stage_vertex(i, local_vertex(t, T, i));
    unsigned short* c = sC + (size_t)buf * cmax;
    for (int i = tid; 8 * i < (T.nent & ~kTileBnd); i += kTileThreads) cp_async16(c + 8 * i, t.cent + T.cb + 8 * i);
    if (!kStage) cp_async_commit();
  };
  {
    const int g0 = local_vertex(t, R, tid), g1 = local_vertex(t, R, tid + kTileThreads);
    if (kStage) stage_normals(R);
    pdl_wait();
    const int stop = *done;
    stage(R, g0, g1, 0);
    if (kStage) cp_async_commit();
    if (stop) {
      cp_async_wait<0>();
      return;
    }
  }

  // last stage with fuse_dt: the next step's local dt from the new state
  const bool next_dt = do_norm && k.fuse_dt;
  double nrm[4] = {0.0, 0.0, 0.0, 0.0};
  unsigned long long dbits = 0x7ff0000000000000ull;
  const double dtg = kUpdate && (ctl.time_mode == 1 || ctl.time_step > 0.0) ? sc->dt_global : 0.0;

  for (int buf = 0;; buf ^= 1) {
    at += gridDim.x;
    const bool more = at < t.count;
    const TileRec N = more ? load_rec(t, at) : R;
    const int e0 = R.e0, NE = R.NE;
    // the thread's first edge (TeCNO) and its list's range, read while the copies are in flight
    double2 un = make_double2(0.0, 0.0);
    double ar = 0.0;
    unsigned ab = 0;
    if (!kStage && tid < NE) { un = t.u[e0 + tid]; ar = t.ar[e0 + tid]; ab = t.ab[e0 + tid]; }
    const bool own = tid < R.nown();
    const int v = R.vb + (own ? tid : 0);
    const unsigned short* rel = t.crel + R.rel;
    const int j0 = own ? rel[tid] : 0, j1 = own ? rel[tid + 1] : 0;
    cp_async_wait<0>();
    __syncthreads();
    if (FLUX == FLUX_ROE_EC || k.strong) {
      for (int i = tid; i < R.L(); i += kTileThreads) {
        if (FLUX == FLUX_ROE_EC) s1[i] = sqrt_nr(-sB[i].y);
        const int g = k.strong ? local_vertex(t, R, i) : 0;
        if (k.strong && (m.sflag[g] & 1)) {
          // a strong condition reset this vertex's primitive state but not its entropy
          // variables: the flux reads the primitive state, as the reference does
          Prim q;
          q.T = s.T[g]; q.u = sA[i].x; q.v = sA[i].y; q.p = sB[i].x;
          const VRec x = make_vrec<FLUX>(k, q);
          sB[i] = make_double2(x.p, x.V5);
          if (is_tecno<FLUX>()) s1[i] = x.V1;
          if (FLUX == FLUX_ROE_EC) s1[i] = x.x;
        }
      }
      __syncthreads();
    }
    const int g0 = more ? local_vertex(t, N, tid) : 0, g1 = more ? local_vertex(t, N, tid + kTileThreads) : 0;

    // ---- edge fluxes
    for (int le = tid; le < NE; le += kTileThreads) {
      if (kStage) ab = sAB[le];
      const int la = ab & 0xffff, lb = ab >> 16;
      const double2 u = kStage ? sN[le] : un;
      const double area = ar;
      const int nx = le + kTileThreads;
      if (!kStage && nx < NE) { un = t.u[e0 + nx]; ar = t.ar[e0 + nx]; ab = t.ab[e0 + nx]; }
      const VRec A = load_vrec<FLUX>(sA, sB, s1, la), B = load_vrec<FLUX>(sA, sB, s1, lb);
      double gl[8], gr[8], dx = 0.0, dy = 0.0;
      if (kGrad) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const double2 x = sG[c * lmax + la], y = sG[c * lmax + lb];
          gl[2 * c] = x.x; gl[2 * c + 1] = x.y;
          gr[2 * c] = y.x; gr[2 * c + 1] = y.y;
        }
        const double2 xa = sX[la], xb = sX[lb];
        dx = xb.x - xa.x;
        dy = xb.y - xa.y;
      }
      Flx F = kStage ? central_flux<FLUX>(k, A, B, u.x, u.y)
                     : num_flux_unit<FLUX, RECON>(k, A, B, u.x, u.y, area, dx, dy, gl, gr,
                                                  kRoe && k.liou ? sS[la] + sS[lb] : 0);
      if (k.axi) {   // residual[cl] += flux * r_f, residual[cr] -= flux * r_f (src/fv.cc:1095-1096)
        const double rf = t.r[e0 + le];
        F.m *= rf; F.x *= rf; F.y *= rf; F.e *= rf;
      }
      sF[le] = make_double2(F.m, F.x);
      sF2[le] = make_double2(F.y, F.e);
    }
    // what the update reads, in flight across the barrier; the vertex's own record is staged
    D4 q0{0.0, 0.0, 0.0, 0.0}, qo = q0;
    double ia = 0.0, w = 0.0, dtl = dtg;
    const bool old = kUpdate && (ctl.scheme == 1 || r > 0);   // the stage adds U_old
    if (kUpdate && own) {
      const double2 a = sA[tid], b = sB[tid];
      q0 = D4{a.x, a.y, b.x, b.y};
      if (old) qo = ld4(s.S0 + v);
      ia = m.inv_area[v];
      if (do_norm) w = m.pweight[v];
      if (!(ctl.time_mode == 1 || ctl.time_step > 0.0)) dtl = s.dt[v];
    }
    __syncthreads();
    if (!kStage && next_dt) {
      for (int le = tid; le < NE; le += kTileThreads) cp_async16(sN + le, t.n + e0 + le);
      cp_async_commit();
    }
    if (more) {
      stage(N, g0, g1, buf ^ 1);
      if (kStage && !next_dt) stage_normals(N);
    }
    else pdl_trigger();   // this late, the next pass starts behind the last update only

    // ---- owned vertices: fixed-order sum, then residual or RK update
    const unsigned short* list = sC + (size_t)buf * cmax;
    Prim qn{0.0, 0.0, 0.0, 0.0};               // the owned vertex's new state
    if (own) {
      double r0 = 0.0, r1 = 0.0, r2 = 0.0, r3 = 0.0;
      for (int j = j0; j < j1; ++j) {
        const int ent = list[j], le = ent >> 1;
        const double sg = (ent & 1) ? -1.0 : 1.0;
        const double2 f = sF[le], f2 = sF2[le];
        r0 += f.x * sg; r1 += f.y * sg; r2 += f2.x * sg; r3 += f2.y * sg;
      }
      if (R.nent & kTileBnd) {
        const int n2 = 2 * m.nb, n3 = 3 * m.nvu;
        for (int j = m.cb_off[v]; j < m.cb_off[v + 1]; ++j) {
          int ent = m.cb_ent[j];
          int type = ent & 3, idx = ent >> 2;
          // axisymmetric weights (src/fv.cc:1151, 1187, 1226-1228, 1280-1282, 1315-1316): half the
          // radius of the boundary-face vertex, of the viscous unit's cell, of the vertex
          if (type == 0) {
            const double w = k.axi ? 0.5 * m.v_r[(idx & 1) ? m.b_v1[idx >> 1] : m.b_v0[idx >> 1]] : 0.5;
            r0 += s.Fb[idx] * w; r1 += s.Fb[n2 + idx] * w; r2 += s.Fb[2 * n2 + idx] * w; r3 += s.Fb[3 * n2 + idx] * w;
          } else if (type == 2 && k.model == 1) {
            const double w = k.axi ? -(0.5 * m.u_r[idx / 3]) : -(0.5 * 1.0);
            r1 += s.Fv[idx] * w; r2 += s.Fv[n3 + idx] * w; r3 += s.Fv[2 * n3 + idx] * w;
          } else if (type == 3 && k.model == 1) {
            const double w = k.axi ? 0.5 * m.v_r[v] : 0.5;
            r1 += s.Fvb[idx] * w; r2 += s.Fvb[m.nb + idx] * w; r3 += s.Fvb[2 * m.nb + idx] * w;
          }
        }
      }
      // strong conditions: compute_residual_norm zeroes the no-slip momentum residual
      // before the last stage's update (src/fv.cc:1805-1819)
      if (do_norm && k.strong && (m.sflag[v] & 2)) { r1 = 0.0; r2 = 0.0; }
      if (MODE == MODE_RESIDUAL) {
        s.R[v] = r0; s.R[nv + v] = r1; s.R[2 * nv + v] = r2; s.R[3 * nv + v] = r3;
      } else {
        if (do_norm) {
          const double a0 = r0 * ia, a1 = r1 * ia, a2 = r2 * ia, a3 = r3 * ia;
          nrm[0] += a0 * a0 * w; nrm[1] += a1 * a1 * w; nrm[2] += a2 * a2 * w; nrm[3] += a3 * a3 * w;
        }
        double factor = dtl * ia;
        if (k.axi) factor /= m.v_r[v];
        // conserved records from the stored ones: rho = -V5 p, no division; strong runs read
        // T, since V5 lags a reset state
        auto conserved = [&](const D4& q, const double* T) {
          const double rho = k.strong ? density(k, Prim{T[v], q.x, q.y, q.z}) : -q.w * q.z;
          return Cons{rho, q.x * rho, q.y * rho, fma(0.5 * fma(q.x, q.x, q.y * q.y), rho, q.z * k.inv_gm1)};
        };
        double uo[4] = {0.0, 0.0, 0.0, 0.0};
        if (old) {
          const Cons c = conserved(qo, s.T0);
          uo[0] = c.r; uo[1] = c.mx; uo[2] = c.my; uo[3] = c.E;
        }
        const Cons c = rk_stage(ctl, s, nv, v, r, conserved(q0, s.T), uo, factor, r0, r1, r2, r3);
        qn = con2prim(k, c);
        if (w3_only<FLUX>(k)) {
          // inviscid central fluxes read only V5 = -2 beta: V1 (two logarithms) is formed
          // from the state by whatever later needs it (refresh_w)
          st4(out.S + v, qn.u, qn.v, qn.p, prim2ent_v5(k, qn));
          out.T[v] = qn.T;
        } else {
          store_state(k, out, v, qn, prim2ent(k, qn));
        }
        bool ok = isfinite(qn.T) && isfinite(qn.u) && isfinite(qn.v) && isfinite(qn.p) && qn.p > 0.0 && c.r > 0.0;
        if (!ok) atomicOr(&sc->bad, 1);
      }
    }
    if (next_dt) {
      // compute_dt (src/fv.cc:1499-1598) of the coming step, as k_dt forms it
      if (!kStage) {
        if (more) cp_async_wait<1>();
        else cp_async_wait<0>();
        __syncthreads();
      }
      if (own) {
        double lam = 0.0;
        for (int j = j0; j < j1; ++j) {
          const double2 n = sN[list[j] >> 1];
          lam += fabs(fma(qn.u, n.x, qn.v * n.y));
        }
        if (R.nent & kTileBnd)
          for (int j = m.cb_off[v]; j < m.cb_off[v + 1]; ++j) {
            const int ent = m.cb_ent[j];
            if ((ent & 3) != 0) continue;
            const int d = ent >> 3;
            lam += 0.5 * fabs(fma(qn.u, m.b_nx[d], qn.v * m.b_ny[d]));
          }
        lam = spectral_sum(k, m, v, qn, lam);
        const double dtn = k.cfl * m.dcarea[v] / lam;
        if (ctl.time_mode == 0) s.dt[v] = dtn;     // unsteady runs read the minimum only
        unsigned long long bits = (unsigned long long)__double_as_longlong(dtn);
        if (!(dtn > 0.0)) bits = 0x7ff0000000000000ull;
        dbits = bits < dbits ? bits : dbits;
      }
      if (kStage && more) {
        __syncthreads();      // the normals are read until here
        stage_normals(N);
      }
    }
    if (!more) break;
    if (kStage) cp_async_commit();
    R = N;
  }
  if (do_norm) {
    block_sum4_min(nrm, dbits);
    __shared__ int last;
    if (tid == 0) {
      if (next_dt) {
        atomicMin(&sc->dtmin_next, dbits);
        if (blockIdx.x == 0) sc->dt_next = 1;
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) s.part[(size_t)(t.pbase + blockIdx.x) * 4 + c] = nrm[c];
      // the last block to finish forms the norms and ends the step
      __threadfence();
      last = atomicAdd(&sc->blocks_done, 1u) == (unsigned)t.total - 1;
    }
    __syncthreads();
    if (last) {
      __threadfence();
      norm_and_step_end(s, t.total, nv, sc, ctl, reinterpret_cast<double*>(smem), kTileThreads);
      if (tid == 0) sc->blocks_done = 0;
    }
  }
}

}  // namespace tg
