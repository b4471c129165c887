// wx3d_kernels.cuh -- sm_100a kernels of the per-block Godunov update.
//
// Stages of the Godunov step, one CTA per (block, z-slab) marching up the
// slab's k-planes: predictor_kernel and corrector_kernel for the hydro
// equations, stage_kernel (either order) for MHD.  All are persistent: items
// past the first wave are handed out on demand.
//
// stage_kernel: 320 threads (10 warps); a 4-plane shared-memory ring holds
// the primitives of each plane together with its ORDER-deep x/y ghost frame,
// so every x-, y- and z-interface flux is computed exactly once and the
// conservative update (godunov.f90:259-271) reads the two fluxes of each
// face from shared memory (x, y) or from the thread's registers (z).
#pragma once

#include "wx3d_device.cuh"
#include "wx3d_wind.cuh"

namespace wx {


// stage_kernel: 17*16 x- and y-interfaces per plane on the first 272 threads,
// the plane loads (320 cells at first order, 384 at second) over all 320.
// predictor_kernel, corrector_kernel: 256 columns and 64 block-face cells of
// a plane; two CTAs per SM put five warps on every sub-partition.
constexpr int STAGE_THREADS = 320;
static_assert(STAGE_THREADS >= 17 * NC, "one thread per x- and y-interface of a plane");
static_assert(STAGE_THREADS >= PLANE + 4 * NC, "the viscous step's UP frame is gathered by threads PLANE..PLANE+63");
constexpr int RING = 4;             // planes p-1..p+2 of the second-order stencil

struct StageParams {
  const double* __restrict__ src;   // array whose primitives feed the fluxes (physical cells)
  const double* __restrict__ base;  // array the update starts from (U; src itself at first order)
  double* __restrict__ out;         // result (UP for stage 1, W for stage 2)
  const DevBlock* __restrict__ blocks;
  const int32_t* __restrict__ work; // occupied slots
  int32_t nwork;                    // number of (block, slab) items
  int32_t zsplit;                   // slabs per block (1, 2, 4 or 8)
  DevCtl* ctl;
  double dt_factor;                 // 0.5 for the predictor, 1 otherwise
  PhysParams ph;
  int32_t do_dt;                    // fused viscous step: fold the CFL minimum of the result
  const double* __restrict__ gsrc;  // array the ghost cells are gathered from (src, or the
                                    // wind-imposed copy of U in the first stage of a wind run)
  double* __restrict__ gframe;      // first-order stage: where to leave the ghost primitives
                                    // markByPhysical reads (nullptr: not wanted)
};

// markByPhysical's ghost primitives (rho, p) of one block, left behind by the
// first-order stage, which gathers and converts exactly these cells anyway:
// entry (kk-1)*64 + h for entry h of the one-deep x/y frame of plane kk
// (1..16), 1024 + c for cell c of the bottom ghost plane (kk = 0) and
// 1280 + c for the top one (kk = 17).  Two doubles per entry.
constexpr int GFRAME = 16 * 64 + 2 * PLANE;

__device__ __forceinline__ int gframe_entry(int kk, int c) {
  if (c >= PLANE) return (kk >= 1 && kk <= NC) ? (kk - 1) * 64 + (c - PLANE) : -1;
  if (kk == 0) return 16 * 64 + c;
  if (kk == NC + 1) return 16 * 64 + PLANE + c;
  return -1;
}


// Ring plane geometry: 16x16 cells with the ORDER-deep x/y ghost frame.
template <int ORDER>
struct Geo {
  static constexpr int W = NC + 2 * ORDER;   // 20 for the corrector, 18 for the predictor
  static constexpr int PL = W * W;
};

constexpr int VPLANE = (NC + 2) * (NC + 2);  // a plane with its one-deep x/y frame

// Per-block constants and status counters of a stage CTA, kept in shared
// memory rather than in registers: dt/dx, dt/dy, dt/dz of the update, the
// inverse cell sizes of the CFL fold, and the counts of pressure floors,
// density floors, zero densities and non-finite results.
struct StageConsts {
  double dtdx, dtdy, dtdz, idx, idy, idz;
  unsigned cnt[4];
  int next;   // the CTA's next work item
  int pad_;
};

template <int NEQ, int ORDER, bool VISC = false>
__host__ __device__ constexpr size_t stage_smem_bytes() {
  return sizeof(double) * ((size_t)RING * NEQ * Geo<ORDER>::PL + 2 * (size_t)NEQ * 17 * NC +
                           (VISC ? 2 * (size_t)NEQ * VPLANE : 0)) +
         sizeof(DevBlock) + sizeof(StageConsts);
}

template <int ORDER>
__device__ __forceinline__ int hidx(int i, int j) { return (i + ORDER - 1) + Geo<ORDER>::W * (j + ORDER - 1); }
__device__ __forceinline__ int ring_slot(int kk) { return (kk + 64) & (RING - 1); }

// Copies the (rho, p) just stored in ring plane pl at (i, j) to entry e of
// the block's ghost-primitive record.
template <int ORDER>
__device__ __forceinline__ void put_gframe(double* g, int slot, int e, const double* pl, int i, int j) {
  double2 v;
  v.x = pl[hidx<ORDER>(i, j)];
  v.y = pl[4 * Geo<ORDER>::PL + hidx<ORDER>(i, j)];
  reinterpret_cast<double2*>(g)[(size_t)slot * GFRAME + e] = v;
}

// Warp minimum of a positive time step folded into ctl->dtmin_bits.
__device__ __forceinline__ void block_min_dt(double v, DevCtl* ctl) {
  v = fmin(v, __shfl_xor_sync(0xffffffffu, v, 16));
  v = fmin(v, __shfl_xor_sync(0xffffffffu, v, 8));
  v = fmin(v, __shfl_xor_sync(0xffffffffu, v, 4));
  v = fmin(v, __shfl_xor_sync(0xffffffffu, v, 2));
  v = fmin(v, __shfl_xor_sync(0xffffffffu, v, 1));
  if ((threadIdx.x & 31) == 0) atomic_min_pos(&ctl->dtmin_bits, v);
}

// One interface flux in direction DIR from ring cells c0..c3 (pointers to
// equation 0 of cells l-1, l, r, r+1; stride Geo<ORDER>::PL between channels).
// With CARRY (the z-interfaces, which a thread visits in order along its
// column) the limited slope of the lower cell is the upper cell's slope of
// the previous interface -- the limiter sees the same two differences -- and
// is taken from `carry` instead of being evaluated again, unless `first`;
// the upper cell's slope is left in `carry` for the next interface.
template <int NEQ, int SOLVER, int ORDER, int LIM, int DIR, bool CARRY = false>
__device__ __forceinline__ void iface_flux(const double* c0, const double* c1, const double* c2, const double* c3,
                                           const PhysParams& ph, double* f, double* carry = nullptr,
                                           bool first = true) {
  double pl[NEQ], pr[NEQ], fx[NEQ];
#pragma unroll
  for (int e = 0; e < NEQ; ++e) {
    const int q = perm<DIR, true>(e);
    pl[e] = c1[q * Geo<ORDER>::PL];
    pr[e] = c2[q * Geo<ORDER>::PL];
  }
  if (ORDER == 2) {  // limiter (hydro_core.f90:613-636) on permuted primitives
#pragma unroll
    for (int e = 0; e < NEQ; ++e) {
      const int q = perm<DIR, true>(e);
      const double prr = c3[q * Geo<ORDER>::PL];
      const double dm = pr[e] - pl[e], dr = prr - pr[e];
      double al;
      if (!CARRY || first) al = average_t<LIM>(pl[e] - c0[q * Geo<ORDER>::PL], dm, ph.limiter);
      else al = carry[e];
      const double ar = average_t<LIM>(dm, dr, ph.limiter);
      if (CARRY) carry[e] = ar;
      pl[e] = pl[e] + 0.5 * al;
      pr[e] = pr[e] - 0.5 * ar;
    }
  }
#pragma unroll
  for (int e = 0; e < NEQ; ++e) fx[e] = 0.0;
  riemann_mhd<NEQ, SOLVER>(pl, pr, fx, ph.gamma, ph.cv);
#pragma unroll
  for (int e = 0; e < NEQ; ++e) f[perm<DIR, true>(e)] = fx[e];
}

// Stores the result of the fused viscous step for one cell, counts
// non-finite values and folds the cell's CFL time step.
template <int NEQ, bool MHD>
__device__ __forceinline__ void visc_store(const StageParams& P, const double* un, size_t o,
                                           Cfl<NEQ, MHD>& cfl, StageConsts& K) {
  unsigned nonfinite = 0;
#pragma unroll
  for (int e = 0; e < NEQ; ++e) {
    P.out[o + (size_t)e * BCELLS] = un[e];
    nonfinite += !isfinite(un[e]);
  }
  if (nonfinite) atomicAdd(&K.cnt[3], nonfinite);
  if (P.do_dt) {
    double p[NEQ], rinv;
    flow2prim<NEQ, MHD>(un, p, P.ph.inv_cv, &rinv);
    cfl.fold(p, rinv, K.idx, K.idy, K.idz, P.ph.gamma);
  }
}

// Loads plane kk of the slab into its ring slot as primitives: the 16x16
// physical cells, plus -- for the planes that get x/y fluxes -- the x/y ghost
// frame (two deep for the second-order stage), gathered from the neighbours.
// Converts one cell's conserved variables to primitives into ring plane pl,
// counting the flow2prim floors of physical cells when `count`.
template <int NEQ, int ORDER>
__device__ __forceinline__ void store_cell(const PhysParams& ph, double* pl, int i, int j, const double* u, bool count,
                                           unsigned* cnt) {
  double p[NEQ];
  const int st = flow2prim<NEQ, true>(u, p, ph.inv_cv);
  if (count && st != 0) atomicAdd(&cnt[st == 1 ? 0 : (st == 2 ? 1 : 2)], 1u);
#pragma unroll
  for (int e = 0; e < NEQ; ++e) pl[e * Geo<ORDER>::PL + hidx<ORDER>(i, j)] = p[e];
}

template <int NEQ, int ORDER>
__device__ __forceinline__ void load_plane(const StageParams& P, const DevBlock& B, int slot, int kk, int z0, int z1,
                                           double* ring, unsigned* cnt, bool skip_interior = false) {
  const int t = threadIdx.x;
  const PhysParams& ph = P.ph;
  double* pl = ring + ring_slot(kk) * NEQ * Geo<ORDER>::PL;
  const bool inner = (kk >= 1 && kk <= NC);
  const bool frame = (kk >= z0 && kk <= z1);  // plane gets x/y fluxes
  const int nframe = frame ? (ORDER == 2 ? 128 : 64) : 0;
  for (int c = skip_interior && t < PLANE ? t + STAGE_THREADS : t; c < PLANE + nframe; c += STAGE_THREADS) {
    int i, j;
    if (c < PLANE) { i = (c & 15) + 1; j = (c >> 4) + 1; }
    else {
      const int h = c - PLANE;
      const int per = ORDER == 2 ? 32 : 16;         // cells per side
      const int side = h / per, r = (h % 16) + 1;
      const int d = (ORDER == 2) ? ((h % 32) >> 4) : 1;   // 0: outer, 1: inner ghost layer
      if (side == 0) { i = d - 1; j = r; }
      else if (side == 1) { i = NC + 2 - d; j = r; }
      else if (side == 2) { i = r; j = d - 1; }
      else { i = r; j = NC + 2 - d; }
    }
    double u[NEQ];
    if (inner && c < PLANE) load_cell<NEQ>(P.src, slot, i, j, kk, u);
    else gather_ghost<NEQ>(P.gsrc ? P.gsrc : P.src, B, slot, i, j, kk, u);
    store_cell<NEQ, ORDER>(ph, pl, i, j, u, c < PLANE && inner && frame, cnt);
    if (ORDER == 1 && P.gframe) {
      const int e = gframe_entry(kk, c);
      if (e >= 0) put_gframe<ORDER>(P.gframe, slot, e, pl, i, j);
    }
  }
}

// Per slab the planes are walked with two barriers each.  Phase A of update
// plane m loads plane m+ORDER+1 into the slot of plane m-1 (no longer read:
// the z-interface slope of plane m is carried in registers) while the same
// threads compute the z-flux m+1/2 and the x/y fluxes of plane m; phase B
// applies the update.  The loads of one warp overlap the flux arithmetic of
// the others.
//
// VISC (second stage, whole blocks) fuses doViscousStep
// (hydro_solver.f90:217-250): the stage result W of plane m goes to a
// two-plane shared buffer whose one-deep x/y frame holds the half-step UP
// ghosts, and phase B of plane m applies U = W + eta (sum of the six
// neighbours - 6 W) to plane m-1, whose z-neighbours are W(m-2) (still in
// the buffer slot that W(m) replaces, read first by the same thread) and
// W(m) (in registers).  The block-face z-neighbours are UP ghosts as well.
// One CTA per SM (168 registers, 105-200 KB of shared memory): bound by the
// FP64 chains of HLLD.  Refined reciprocals and roots in place of its nine
// divisions and seven roots per interface, and minmod compiled in as for
// hydro: 440 blocks (HLLD) predictor 0.394 -> 0.266 ms, corrector with the
// viscous step 0.912 -> 0.434 ms; 16 blocks in 8 slabs 29 + 50 -> 20 + 24 us.

// Cell-centred electric field E = -v x B of the stage primitives at one ring
// cell: the field-interpolated E of the field-CD scheme (Toth 2000, J. Comput.
// Phys. 161, 605), which brio-wu/flux_cd.f90:37 declares as efield(3,...).
template <int ORDER>
__device__ __forceinline__ void efield(const double* c, double* E) {
  constexpr int PL = Geo<ORDER>::PL;
  const double v1 = c[1 * PL], v2 = c[2 * PL], v3 = c[3 * PL];
  const double b1 = c[5 * PL], b2 = c[6 * PL], b3 = c[7 * PL];
  E[0] = v3 * b2 - v2 * b3;
  E[1] = v1 * b3 - v3 * b1;
  E[2] = v2 * b1 - v1 * b2;
}

template <int NEQ, int SOLVER, int ORDER, int LIM, bool VISC = false>
__global__ void __launch_bounds__(STAGE_THREADS, 1) stage_kernel(StageParams P) {
  extern __shared__ __align__(16) double smem[];
  double* ring = smem;                                   // [RING][NEQ][Geo<ORDER>::PL]
  double* fxs = ring + RING * NEQ * Geo<ORDER>::PL;               // [NEQ][16 rows][17]
  double* fys = fxs + NEQ * 17 * NC;                     // [NEQ][17][16 cols]
  double* wpl = fys + NEQ * 17 * NC;                     // VISC: [2][NEQ][VPLANE]
  DevBlock& B = *reinterpret_cast<DevBlock*>(wpl + (VISC ? 2 * NEQ * VPLANE : 0));
  StageConsts& K = *reinterpret_cast<StageConsts*>(&B + 1);
  auto vq = [](int i, int j) { return i + (NC + 2) * j; };
  Cfl<NEQ, true> cfl;
  const int t = threadIdx.x;
  const int planes = NC / P.zsplit;
  const PhysParams& ph = P.ph;
  if (t < 4) K.cnt[t] = 0;

  for (int w = blockIdx.x; w < P.nwork;) {
    const int slot = P.work[w / P.zsplit];
    const int z0 = 1 + (w % P.zsplit) * planes, z1 = z0 + planes - 1;
    __syncthreads();
    if (t < (int)(sizeof(DevBlock) / 4)) reinterpret_cast<int*>(&B)[t] = reinterpret_cast<const int*>(P.blocks + slot)[t];
    __syncthreads();
    if (t == 0) {  // read after the prologue's barriers
      const double dtp = P.ctl->dt * P.dt_factor;
      K.dtdx = dtp / B.dx;
      K.dtdy = dtp / B.dy;
      K.dtdz = dtp / B.dz;
      K.idx = 1.0 / B.dx;
      K.idy = 1.0 / B.dy;
      K.idz = 1.0 / B.dz;
    }
    const int ci = (t & (NC - 1)) + 1, cj = (t >> 4) + 1;   // column of threads t < 256
    const int hc = hidx<ORDER>(ci, cj);
    double zprev[NEQ], znew[NEQ], zslope[NEQ];
#pragma unroll
    for (int e = 0; e < NEQ; ++e) { zprev[e] = 0.0; znew[e] = 0.0; zslope[e] = 0.0; }
    double bz_below = 0.0;  // B_z of plane m-1 in this thread's column (Powell source)
    double e_below[3] = {0.0, 0.0, 0.0};  // E of plane m-1 in this thread's column (field-CD)

    // ---- prologue: planes z0-ORDER .. z0+ORDER-1, the z-interface z0-1/2,
    // then plane z0+ORDER into the slot of plane z0-ORDER ------------------
    for (int kk = z0 - ORDER; kk <= z0 + ORDER - 1; ++kk) load_plane<NEQ, ORDER>(P, B, slot, kk, z0, z1, ring, K.cnt);
    __syncthreads();
    if (t < PLANE) {
      const int m = z0 - 1;
      const double* c0 = ring + ring_slot(m - 1) * NEQ * Geo<ORDER>::PL + hc;
      const double* c1 = ring + ring_slot(m) * NEQ * Geo<ORDER>::PL + hc;
      const double* c2 = ring + ring_slot(m + 1) * NEQ * Geo<ORDER>::PL + hc;
      const double* c3 = ring + ring_slot(m + 2) * NEQ * Geo<ORDER>::PL + hc;
      iface_flux<NEQ, SOLVER, ORDER, LIM, 2, true>(c0, c1, c2, c3, ph, znew, zslope, true);
      bz_below = c1[7 * Geo<ORDER>::PL];
      if (ph.flux_cd) efield<ORDER>(c1, e_below);
    }
#pragma unroll
    for (int e = 0; e < NEQ; ++e) zprev[e] = znew[e];
    if (VISC && t < PLANE) {  // W(z0-1) of the column: the bottom UP ghost
      double g[NEQ];
      gather_ghost<NEQ>(P.src, B, slot, ci, cj, z0 - 1, g);
#pragma unroll
      for (int e = 0; e < NEQ; ++e) wpl[((z0 - 1) & 1) * NEQ * VPLANE + e * VPLANE + vq(ci, cj)] = g[e];
    }
    __syncthreads();
    load_plane<NEQ, ORDER>(P, B, slot, z0 + ORDER, z0, z1, ring, K.cnt);
    __syncthreads();

    for (int m = z0; m <= z1; ++m) {
      // ---- phase A: load plane m+ORDER+1; z-flux m+1/2; x/y fluxes of m ---
      {
        // L2 prefetch, one plane period ahead, of the physical cells of the
        // plane the next phase A loads and of the base plane the next phase B
        // reads (16 lines of 128 bytes per equation and plane)
        const int kq = t < 16 * NEQ ? m + ORDER + 2 : m + 1;
        const double* arr = t < 16 * NEQ ? P.src : P.base;
        const int r = t < 16 * NEQ ? t : t - 16 * NEQ;
        if (r < 16 * NEQ && kq >= 1 && kq <= NC && kq <= z1 + ORDER && (t < 16 * NEQ || kq <= z1))
          prefetch_l2(arr + cell_off(slot, NEQ, r >> 4, 1, 1, kq) + (size_t)(r & 15) * 16);
      }
      // the physical cell of each thread t < 256 is fetched here and
      // converted into the ring after the fluxes, so its load latency
      // overlaps them; the ghost frame is gathered and stored first
      const int kl = m + ORDER + 1;
      const bool late = t < PLANE && kl <= z1 + ORDER;
      double ul[NEQ];
      if (late) {
        if (kl >= 1 && kl <= NC) load_cell<NEQ>(P.src, slot, ci, cj, kl, ul);
        else gather_ghost<NEQ>(P.gsrc ? P.gsrc : P.src, B, slot, ci, cj, kl, ul);
      }
      if (kl <= z1 + ORDER) load_plane<NEQ, ORDER>(P, B, slot, kl, z0, z1, ring, K.cnt, true);
      // one-deep x/y frame of W(m): UP ghosts of plane m, on threads 256..319,
      // which compute no z-flux and at most one x/y interface pair
      if (VISC && t >= PLANE && t < PLANE + 4 * NC) {
        {
          const int f = t - PLANE;
          const int side = f >> 4, r = (f & 15) + 1;
          const int gi = side == 0 ? 0 : (side == 1 ? NC + 1 : r);
          const int gj = side == 2 ? 0 : (side == 3 ? NC + 1 : r);
          double g[NEQ];
          gather_ghost<NEQ>(P.src, B, slot, gi, gj, m, g);
#pragma unroll
          for (int e = 0; e < NEQ; ++e) wpl[(m & 1) * NEQ * VPLANE + e * VPLANE + vq(gi, gj)] = g[e];
        }
      }
      if (t < 17 * NC) {
        const double* pp = ring + ring_slot(m) * NEQ * Geo<ORDER>::PL;
        // x-interface between ii and ii+1 in row jx: a half-warp takes 16
        // consecutive interfaces of one row (conflict-free shared loads),
        // threads 256..271 the last interface of each row; y-interface
        // between jj and jj+1 in column iy
        const int ii = t < PLANE ? (t & 15) : NC, jx = t < PLANE ? (t >> 4) + 1 : t - PLANE + 1;
        const int iy = (t & 15) + 1, jj = t >> 4;
        {
          double f[NEQ];
          iface_flux<NEQ, SOLVER, ORDER, LIM, 0>(pp + hidx<ORDER>(ii - 1, jx), pp + hidx<ORDER>(ii, jx), pp + hidx<ORDER>(ii + 1, jx),
                                                 pp + hidx<ORDER>(ii + 2, jx), ph, f);
#pragma unroll
          for (int e = 0; e < NEQ; ++e) fxs[(e * NC + (jx - 1)) * 17 + ii] = f[e];
        }
        {
          double f[NEQ];
          iface_flux<NEQ, SOLVER, ORDER, LIM, 1>(pp + hidx<ORDER>(iy, jj - 1), pp + hidx<ORDER>(iy, jj), pp + hidx<ORDER>(iy, jj + 1),
                                                 pp + hidx<ORDER>(iy, jj + 2), ph, f);
#pragma unroll
          for (int e = 0; e < NEQ; ++e) fys[(e * 17 + jj) * NC + (iy - 1)] = f[e];
        }
      }
      if (t < PLANE) {  // z-flux m+1/2 last: znew is live only from here to phase B
        const double* c1 = ring + ring_slot(m) * NEQ * Geo<ORDER>::PL + hc;
        const double* c2 = ring + ring_slot(m + 1) * NEQ * Geo<ORDER>::PL + hc;
        const double* c3 = ring + ring_slot(m + 2) * NEQ * Geo<ORDER>::PL + hc;
        iface_flux<NEQ, SOLVER, ORDER, LIM, 2, true>(nullptr, c1, c2, c3, ph, znew, zslope, false);
      }
      if (late) {
        double* pl = ring + ring_slot(kl) * NEQ * Geo<ORDER>::PL;
        store_cell<NEQ, ORDER>(ph, pl, ci, cj, ul, kl >= 1 && kl <= NC && kl >= z0 && kl <= z1, K.cnt);
        if (ORDER == 1 && P.gframe && kl == NC + 1) put_gframe<ORDER>(P.gframe, slot, gframe_entry(kl, t), pl, ci, cj);
      }
      __syncthreads();
      // ---- phase B: conservative update of plane m (godunov.f90:259-271) --
      if (t < PLANE) {
        double s[NEQ];
#pragma unroll
        for (int e = 0; e < NEQ; ++e) s[e] = 0.0;
        if (ph.eight_wave) {  // Powell source (sources.f90:38-95) on the stage primitives
          const double* pm = ring + ring_slot(m) * NEQ * Geo<ORDER>::PL;
          const double* pu = ring + ring_slot(m + 1) * NEQ * Geo<ORDER>::PL;
          const int h = hc;
          const double divB = (pm[5 * Geo<ORDER>::PL + h + 1] - pm[5 * Geo<ORDER>::PL + h - 1]) * (0.5 * K.idx) +
                              (pm[6 * Geo<ORDER>::PL + h + Geo<ORDER>::W] - pm[6 * Geo<ORDER>::PL + h - Geo<ORDER>::W]) * (0.5 * K.idy) +
                              (pu[7 * Geo<ORDER>::PL + h] - bz_below) * (0.5 * K.idz);
          const double v1 = pm[1 * Geo<ORDER>::PL + h], v2 = pm[2 * Geo<ORDER>::PL + h], v3 = pm[3 * Geo<ORDER>::PL + h];
          const double b1 = pm[5 * Geo<ORDER>::PL + h], b2 = pm[6 * Geo<ORDER>::PL + h], b3 = pm[7 * Geo<ORDER>::PL + h];
          s[1] = -divB * b1;
          s[2] = -divB * b2;
          s[3] = -divB * b3;
          s[4] = -divB * (v1 * b1 + v2 * b2 + v3 * b3);
          s[5] = -divB * v1;
          s[6] = -divB * v2;
          s[7] = -divB * v3;
        }
        bz_below = ring[ring_slot(m) * NEQ * Geo<ORDER>::PL + 7 * Geo<ORDER>::PL + hc];
        const size_t o = cell_off(slot, NEQ, 0, ci, cj, m);
        // field-CD (brio-wu/flux_cd.f90:74-84): B from the central differences
        // of E over the six face neighbours; E of plane m-1 is carried
        double bcd[3] = {0.0, 0.0, 0.0};
        if (ph.flux_cd) {
          constexpr int PL = Geo<ORDER>::PL, W = Geo<ORDER>::W;
          const double* pm = ring + ring_slot(m) * NEQ * PL + hc;
          double xl[3], xr[3], yl[3], yr[3], zu[3], ec[3];
          efield<ORDER>(pm - 1, xl);
          efield<ORDER>(pm + 1, xr);
          efield<ORDER>(pm - W, yl);
          efield<ORDER>(pm + W, yr);
          efield<ORDER>(ring + ring_slot(m + 1) * NEQ * PL + hc, zu);
          efield<ORDER>(pm, ec);
          const double hx = 0.5 * K.dtdx, hy = 0.5 * K.dtdy, hz = 0.5 * K.dtdz;
          bcd[0] = __ldg(P.base + o + 5 * (size_t)BCELLS) - hy * (yr[2] - yl[2]) - hz * (-zu[1] + e_below[1]);
          bcd[1] = __ldg(P.base + o + 6 * (size_t)BCELLS) - hx * (-xr[2] + xl[2]) - hz * (zu[0] - e_below[0]);
          bcd[2] = __ldg(P.base + o + 7 * (size_t)BCELLS) - hx * (xr[1] - xl[1]) - hy * (-yr[0] + yl[0]);
#pragma unroll
          for (int d = 0; d < 3; ++d) e_below[d] = ec[d];
        }
        double wv[NEQ];
        const double dtdx = K.dtdx, dtdy = K.dtdy, dtdz = K.dtdz;
#pragma unroll
        for (int e = 0; e < NEQ; ++e) {
          const double fxl = fxs[(e * NC + (cj - 1)) * 17 + ci - 1], fxr = fxs[(e * NC + (cj - 1)) * 17 + ci];
          const double fyl = fys[(e * 17 + cj - 1) * NC + ci - 1], fyr = fys[(e * 17 + cj) * NC + ci - 1];
          double v = __ldg(P.base + o + (size_t)e * BCELLS) + dtdx * (fxl - fxr) + dtdy * (fyl - fyr) +
                     dtdz * (zprev[e] - znew[e]);
          if (ph.eight_wave) v = v + P.ctl->dt * P.dt_factor * s[e];
          if (ph.flux_cd && e >= 5 && e <= 7) v = bcd[e - 5];
          if (VISC) wv[e] = v;
          else P.out[o + (size_t)e * BCELLS] = v;
        }
        if constexpr (VISC) {
          double* wb = wpl + (m & 1) * NEQ * VPLANE;          // W(m-2) of the column, then W(m)
          const double* wc = wpl + ((m - 1) & 1) * NEQ * VPLANE;  // W(m-1) with its frame
          if (m > z0) {
            double un[NEQ];
#pragma unroll
            for (int e = 0; e < NEQ; ++e) {
              const double* pe = wc + e * VPLANE;
              const double c = pe[vq(ci, cj)];
              un[e] = c + ph.eta * (+pe[vq(ci + 1, cj)] + pe[vq(ci - 1, cj)] + pe[vq(ci, cj + 1)] + pe[vq(ci, cj - 1)] +
                                    wv[e] + wb[e * VPLANE + vq(ci, cj)] - 6.0 * c);
            }
            visc_store<NEQ, true>(P, un, o - NC * NC, cfl, K);
          }
#pragma unroll
          for (int e = 0; e < NEQ; ++e) wb[e * VPLANE + vq(ci, cj)] = wv[e];
        }
      }
#pragma unroll
      for (int e = 0; e < NEQ; ++e) zprev[e] = znew[e];
      __syncthreads();
    }
    if (VISC && t < PLANE) {  // viscous step of plane z1: above it, the top UP ghost
      double g[NEQ], un[NEQ];
      gather_ghost<NEQ>(P.src, B, slot, ci, cj, z1 + 1, g);
      const double* wc = wpl + (z1 & 1) * NEQ * VPLANE;
      const double* wb = wpl + ((z1 - 1) & 1) * NEQ * VPLANE;
#pragma unroll
      for (int e = 0; e < NEQ; ++e) {
        const double* pe = wc + e * VPLANE;
        const double c = pe[vq(ci, cj)];
        un[e] = c + ph.eta * (+pe[vq(ci + 1, cj)] + pe[vq(ci - 1, cj)] + pe[vq(ci, cj + 1)] + pe[vq(ci, cj - 1)] + g[e] +
                              wb[e * VPLANE + vq(ci, cj)] - 6.0 * c);
      }
      visc_store<NEQ, true>(P, un, cell_off(slot, NEQ, 0, ci, cj, z1), cfl, K);
    }
    // items past the first wave go, in list order, to whichever CTA
    // finishes first (the counter is zeroed before each launch): blocks at
    // coarse/fine faces cost more, and a static stride left SMs idle
    if (t == 0) K.next = (int)gridDim.x + (int)atomicAdd(&P.ctl->work_next[ORDER - 1], 1u);
    __syncthreads();
    w = K.next;
  }
  if (VISC && P.do_dt) block_min_dt(cfl.dt(), P.ctl);
  __syncthreads();
  if (t < 4 && K.cnt[t]) atomicAdd(&P.ctl->cnt[t], (unsigned long long)K.cnt[t]);
}

// ---------------------------------------------------------------------------
// First-order stage of the hydro equations (the predictor, and the single
// stage of HLL1): one CTA per (block, z-slab), marching up the z-planes.
//
// What bounds the stage is the shared-memory/L1 data path (67 % busy in the
// stage kernel that staged every operand and every flux through shared
// memory), then instruction issue, so as little as possible travels:
//  - a thread t < 256 owns a column and keeps the primitives (and sound
//    speed) of its cell of plane m in registers for its three interfaces;
//  - it solves the x-interface to the next cell and the y-interface to the
//    next row, reading only that neighbour's primitives from the plane in
//    shared memory; the x-flux goes to the next lane by a shuffle, the
//    y-flux to the next row through shared memory;
//  - the frame cells never reach shared memory: each of the 64 threads of
//    warps 8 and 9 gathers the ghost of one (side, row), keeps it in
//    registers and solves the block-face interface it belongs to (x on
//    warp 8, y on warp 9), so no warp has a partly filled solve.
// The plane and the flux buffers are doubled, which leaves one barrier per
// plane: the update of plane m and the fluxes of plane m+1 run between the
// same two barriers.  Conserved cells arrive by 8-byte asynchronous copies a
// plane ahead and stay in shared memory until they are the base of the
// update (P.base is P.src), so no load holds registers across the fluxes:
// with 96 registers two CTAs share an SM (no spills up to six equations, 12 to
// 40 bytes of stores at seven).  Loading them into
// registers instead, or late, spilled or exposed the loads (1.71 and 1.95 ms
// against 1.51 on the 11,600-block AMR blast at five equations; the kernel
// that staged everything took 1.75); three CTAs at 64 registers: 2.06 ms.
// Six equations, 5,496 blocks of the winds mesh: 0.945 -> 0.848 ms.
template <int NEQ>
struct PredSmem {
  static constexpr int W = NC + 1;               // padded row: a column read is conflict-free
  double pl[2][NEQ + 1][W * NC];                 // primitives and sound speed of a plane
  double raw[3][NEQ][PLANE];                     // conserved variables of planes m, m+1, m+2
  double fy[2][NEQ][(NC + 1) * NC];              // y-flux below row j (rows 0 and 16: block faces)
  double ex[2][2][NEQ][NC];                      // x-flux of the low and the high block face
  DevBlock B;
  StageConsts K;
};

// Barrier of all threads of a stage CTA, met by the roles at different places.
__device__ __forceinline__ void plane_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(STAGE_THREADS) : "memory"); }
// Barrier of all threads of the CTA's cluster.
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ void copy_async8(double* smem, const double* g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(g) : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <int NEQ, int SOLVER, int DIR>
__device__ __forceinline__ void cell_flux(const double* a, const double* b, const PhysParams& ph, double* f) {
  double pl[NEQ], pr[NEQ], fx[NEQ];
#pragma unroll
  for (int e = 0; e < NEQ; ++e) {
    pl[e] = a[perm<DIR, false>(e)];
    pr[e] = b[perm<DIR, false>(e)];
  }
  if constexpr (SOLVER == WX_SOLVER_HLLC) riemann_hllc_c<NEQ>(pl, pr, a[NEQ], b[NEQ], fx, ph.cv);
  else riemann_hll_c<NEQ>(pl, pr, a[NEQ], b[NEQ], fx, ph.cv);
#pragma unroll
  for (int e = 0; e < NEQ; ++e) f[perm<DIR, false>(e)] = fx[e];
}

// Primitives and sound speed of a cell; physical cells count their floors.
template <int NEQ>
__device__ __forceinline__ void prim_and_sound(const PhysParams& ph, const double* u, double* p, bool count,
                                               unsigned* cnt) {
  double rinv;
  const int st = flow2prim<NEQ, false>(u, p, ph.inv_cv, &rinv);
  p[NEQ] = sqrt_nr(ph.gamma * p[4] * rinv);
  if (count && st != 0) atomicAdd(&cnt[st == 1 ? 0 : (st == 2 ? 1 : 2)], 1u);
}

template <int NEQ, int SOLVER>
__global__ void __launch_bounds__(STAGE_THREADS, 2) predictor_kernel(StageParams P) {
  extern __shared__ __align__(16) unsigned char smraw[];
  PredSmem<NEQ>& S = *reinterpret_cast<PredSmem<NEQ>*>(smraw);
  constexpr int W = PredSmem<NEQ>::W;
  DevBlock& B = S.B;
  StageConsts& K = S.K;
  const int t = threadIdx.x, lane = t & (NC - 1);
  const PhysParams& ph = P.ph;
  const int planes = NC / P.zsplit;
  const bool column = t < PLANE;
  const int ci = lane + 1, cj = (t >> 4) + 1;                  // column threads
  const int side = (t - PLANE) >> 4;                           // face threads: 0, 1 x; 2, 3 y
  const int gi = side == 0 ? 0 : (side == 1 ? NC + 1 : lane + 1);
  const int gj = side == 2 ? 0 : (side == 3 ? NC + 1 : lane + 1);
  const double* gsrc = P.gsrc ? P.gsrc : P.src;
  if (t < 4) K.cnt[t] = 0;

  for (int w = blockIdx.x; w < P.nwork;) {
    const int slot = P.work[w / P.zsplit];
    const int z0 = 1 + (w % P.zsplit) * planes, z1 = z0 + planes - 1;
    __syncthreads();
    if (t < (int)(sizeof(DevBlock) / 4)) reinterpret_cast<int*>(&B)[t] = reinterpret_cast<const int*>(P.blocks + slot)[t];
    __syncthreads();
    if (t == 0) {  // read after the prologue's barrier
      const double dtp = P.ctl->dt * P.dt_factor;
      K.dtdx = dtp / B.dx;
      K.dtdy = dtp / B.dy;
      K.dtdz = dtp / B.dz;
    }
    // conserved variables of the column's cell of plane kk into the raw ring
    // (an asynchronous copy; each thread reads back its own cell only)
    auto fetch = [&](int kk) {
      double* d = &S.raw[(unsigned)(kk + 3) % 3u][0][t];
      if (kk >= 1 && kk <= NC) {
        const double* g = P.src + cell_off(slot, NEQ, 0, ci, cj, kk);
#pragma unroll
        for (int e = 0; e < NEQ; ++e) copy_async8(d + e * PLANE, g + (size_t)e * BCELLS);
      } else {
        double u[NEQ];
        gather_ghost<NEQ>(gsrc, B, slot, ci, cj, kk, u);
#pragma unroll
        for (int e = 0; e < NEQ; ++e) d[e * PLANE] = u[e];
      }
    };
    // primitives and sound speed of the column's cell of plane kk
    auto convert = [&](int kk, double* p) {
      const double* d = &S.raw[(unsigned)(kk + 3) % 3u][0][t];
      double u[NEQ];
#pragma unroll
      for (int e = 0; e < NEQ; ++e) u[e] = d[e * PLANE];
      prim_and_sound<NEQ>(ph, u, p, kk >= z0 && kk <= z1, K.cnt);
    };
    auto put_plane = [&](int kk, const double* p) {
      double* d = &S.pl[kk & 1][0][(cj - 1) * W + lane];
#pragma unroll
      for (int e = 0; e <= NEQ; ++e) d[e * (W * NC)] = p[e];
    };
    auto put_mark = [&](int e, const double* p) {  // (rho, p) of a ghost cell for markByPhysical
      double2 v;
      v.x = p[0];
      v.y = p[4];
      reinterpret_cast<double2*>(P.gframe)[(size_t)slot * GFRAME + e] = v;
    };
    double pc[NEQ + 1], zf[NEQ];
    if (column) {
      double pn[NEQ + 1];
      fetch(z0 - 1);
      fetch(z0);
      fetch(z0 + 1);
      copy_async_wait();
      convert(z0 - 1, pn);
      if (P.gframe && z0 == 1) put_mark(gframe_entry(0, t), pn);
      if (z0 + 2 <= z1 + 1) fetch(z0 + 2);   // into the slot of plane z0-1
      convert(z0, pc);
      put_plane(z0, pc);
      cell_flux<NEQ, SOLVER, 2>(pn, pc, ph, zf);
      convert(z0 + 1, pn);
      if (P.gframe && z0 + 1 == NC + 1) put_mark(gframe_entry(NC + 1, t), pn);
      put_plane(z0 + 1, pn);
    } else {
      double u[NEQ];
      gather_ghost<NEQ>(gsrc, B, slot, gi, gj, z0, u);
      prim_and_sound<NEQ>(ph, u, pc, false, K.cnt);
      if (P.gframe) put_mark(gframe_entry(z0, t), pc);
    }
    __syncthreads();

    for (int m = z0; m <= z1; ++m) {
      const int b = m & 1;
      if (column) {
        double dx[NEQ], dz[NEQ], f[NEQ];
        const double* pl = &S.pl[b][0][(cj - 1) * W + lane];
        {  // y-interface to row cj+1 (the last row's flux is a face thread's)
          double pr[NEQ + 1];
          const int o = cj < NC ? W : 0;
#pragma unroll
          for (int e = 0; e <= NEQ; ++e) pr[e] = pl[e * (W * NC) + o];
          cell_flux<NEQ, SOLVER, 1>(pc, pr, ph, f);
          if (cj < NC) {
#pragma unroll
            for (int e = 0; e < NEQ; ++e) S.fy[b][e][cj * NC + lane] = f[e];
          }
        }
        {  // x-interface to cell ci+1 (the last lane's flux is a face thread's)
          double pr[NEQ + 1];
          const int o = lane < NC - 1 ? 1 : 0;
#pragma unroll
          for (int e = 0; e <= NEQ; ++e) pr[e] = pl[e * (W * NC) + o];
          cell_flux<NEQ, SOLVER, 0>(pc, pr, ph, f);
#pragma unroll
          for (int e = 0; e < NEQ; ++e) {
            const double xl = __shfl_up_sync(0xffffffffu, f[e], 1, NC);
            dx[e] = lane == 0 ? -f[e] : (lane == NC - 1 ? xl : xl - f[e]);
          }
        }
        {  // z-interface m+1/2: the column's own cells
          const double* pu = &S.pl[b ^ 1][0][(cj - 1) * W + lane];
          double pn[NEQ + 1];
#pragma unroll
          for (int e = 0; e <= NEQ; ++e) pn[e] = pu[e * (W * NC)];
          cell_flux<NEQ, SOLVER, 2>(pc, pn, ph, f);
#pragma unroll
          for (int e = 0; e < NEQ; ++e) {
            dz[e] = zf[e] - f[e];
            zf[e] = f[e];
          }
#pragma unroll
          for (int e = 0; e <= NEQ; ++e) pc[e] = pn[e];
        }
        const size_t o = cell_off(slot, NEQ, 0, ci, cj, m);
        plane_barrier();
        // conservative update of plane m (godunov.f90:259-271); each
        // direction's two fluxes are subtracted before they are scaled, so
        // equal fluxes cancel exactly
        const double dtdx = K.dtdx, dtdy = K.dtdy, dtdz = K.dtdz;
        const bool xedge = lane == 0 || lane == NC - 1;
        const double* ex = &S.ex[b][lane >> 3][0][cj - 1];
        const double* v = &S.raw[(unsigned)m % 3u][0][t];
#pragma unroll
        for (int e = 0; e < NEQ; ++e) {
          const double xe = xedge ? ex[e * NC] : 0.0;
          const double ddx = dx[e] + (lane == 0 ? xe : -xe);
          const double dy = S.fy[b][e][(cj - 1) * NC + lane] - S.fy[b][e][cj * NC + lane];
          P.out[o + (size_t)e * BCELLS] = v[e * PLANE] + dtdx * ddx + dtdy * dy + dtdz * dz[e];
        }
        if (m < z1) {  // plane m+2 into the buffer of plane m, which no one reads any more
          double pn[NEQ + 1];
          copy_async_wait();
          convert(m + 2, pn);
          if (P.gframe && m + 2 == NC + 1) put_mark(gframe_entry(NC + 1, t), pn);
          put_plane(m + 2, pn);
          if (m + 3 <= z1 + 1) fetch(m + 3);
        }
      } else {
        double u[NEQ], pr[NEQ + 1], f[NEQ];
        if (m < z1) gather_ghost<NEQ>(gsrc, B, slot, gi, gj, m + 1, u);
        if (side < 2) {
          const double* c = &S.pl[b][0][lane * W + (side ? NC - 1 : 0)];
#pragma unroll
          for (int e = 0; e <= NEQ; ++e) pr[e] = c[e * (W * NC)];
          double l[NEQ + 1], r[NEQ + 1];
#pragma unroll
          for (int e = 0; e <= NEQ; ++e) { l[e] = side ? pr[e] : pc[e]; r[e] = side ? pc[e] : pr[e]; }
          cell_flux<NEQ, SOLVER, 0>(l, r, ph, f);
#pragma unroll
          for (int e = 0; e < NEQ; ++e) S.ex[b][side][e][lane] = f[e];
        } else {
          const double* c = &S.pl[b][0][(side == 3 ? NC - 1 : 0) * W + lane];
#pragma unroll
          for (int e = 0; e <= NEQ; ++e) pr[e] = c[e * (W * NC)];
          double l[NEQ + 1], r[NEQ + 1];
#pragma unroll
          for (int e = 0; e <= NEQ; ++e) { l[e] = side == 3 ? pr[e] : pc[e]; r[e] = side == 3 ? pc[e] : pr[e]; }
          cell_flux<NEQ, SOLVER, 1>(l, r, ph, f);
#pragma unroll
          for (int e = 0; e < NEQ; ++e) S.fy[b][e][(side == 3 ? NC * NC : 0) + lane] = f[e];
        }
        plane_barrier();
        if (m < z1) {
          prim_and_sound<NEQ>(ph, u, pc, false, K.cnt);
          if (P.gframe) put_mark(gframe_entry(m + 1, t), pc);
        }
      }
    }
    // items past the first wave go, in list order, to whichever CTA
    // finishes first (the counter is zeroed before each launch)
    if (t == 0) K.next = (int)gridDim.x + (int)atomicAdd(&P.ctl->work_next[0], 1u);
    __syncthreads();
    w = K.next;
  }
  __syncthreads();
  if (t < 4 && K.cnt[t]) atomicAdd(&P.ctl->cnt[t], (unsigned long long)K.cnt[t]);
}

// ---------------------------------------------------------------------------
// Second-order stage of the hydro equations (the corrector), laid out as the
// predictor above: columns on 256 threads, block-face interfaces on warps 8
// and 9, one barrier per plane.  Shared memory holds a ring of three planes
// with their one-deep x/y frame: primitives of planes m and m+1, and plane
// m+2, which arrives as conserved variables.  A column thread
//  - limits its own x-slope and passes the state at its left face to the
//    lane below by a shuffle, so every x-slope is computed once;
//  - limits its own and the next row's y-slope;
//  - converts its cell of plane m+2 in place, limits the z-slope of the cell
//    above, and carries that cell's upper-face state to the next plane's
//    interface;
//  - copies its cell of plane m+3 over plane m asynchronously once the
//    barrier has passed, and loads its base cell, whose plane was brought
//    into L2 a plane ahead.
// A face thread leaves the inner ghost of its (side, row) in the frame for the
// slopes next to the face, keeps the outer one in registers, and solves the
// block-face interface.
//
// VISC (whole blocks) fuses doViscousStep (hydro_solver.f90:217-250): the
// result W of plane m goes to one of two shared planes framed by the
// half-step UP ghosts, and the update of plane m applies
// U = W + eta (sum of the six neighbours - 6 W) to plane m-1, whose
// z-neighbours are W(m-2) (in the place that W(m) takes, read first by the
// same thread) and W(m).
//
// Bound, as the predictor, by the shared-memory data path (60 % busy) and
// instruction issue (50 %) at five warps per scheduler.  Up to six equations
// two CTAs share an SM: 96 registers, which the conversion in place keeps
// almost free of spills (minmod at five equations none, the fused form at six
// 48 bytes of stores and 124 of loads), and at most 113 KB, for which the
// frame rows are unpadded.  At seven the unfused form still pairs CTAs, with
// 48 to 124 bytes of spill stores (1,128 blocks, HLLC and minmod, with the
// predictor and the viscous kernel: 1.11 -> 0.83 ms against the staged kernel
// at one CTA), and the fused form runs one at 168 registers (0.98 -> 0.81).
// 11,600-block AMR blast, five equations: fused 3.44 -> 2.83 ms, unfused
// 2.72 -> 2.45 ms; 5,496-block winds mesh, six equations: fused (one CTA per
// SM before) 2.37 -> 1.79 ms, unfused 1.55 -> 1.36 ms.  The prefetch of the
// next base plane is 4 % of it; keeping the base in a shared plane instead
// cost 15 % (less L1 for the ghost gathers).
template <int NEQ, bool VISC>
struct CorrSmem {
  static constexpr int W = NC + 2;               // row of an 18-cell framed plane
  static constexpr int PL = W * W;
  double pl[3][NEQ][PL];                         // primitives of planes m, m+1; conserved, then
                                                 // primitive variables of plane m+2
  double fy[2][NEQ][(NC + 1) * NC];              // y-flux below row j (rows 0 and 16: block faces)
  double ex[2][2][NEQ][NC];                      // x-flux of the low and the high block face
  double w[VISC ? 2 : 1][VISC ? NEQ : 1][VISC ? PL : 1];  // W of planes m, m-1, framed by UP ghosts
  double wg[VISC ? 2 : 1][NEQ][VISC ? 4 * NC : 1];  // the frame's UP ghosts, a plane ahead
  DevBlock B;
  StageConsts K;
};

template <int D>
struct Dir { static constexpr int value = D; };
template <int NEQ>
struct Flux {
  double v[NEQ];
  __device__ __forceinline__ explicit Flux(const double* f) {
#pragma unroll
    for (int e = 0; e < NEQ; ++e) v[e] = f[e];
  }
};

// Flux between two face states already permuted to direction DIR.
template <int NEQ, int SOLVER, int DIR>
__device__ __forceinline__ void state_flux(const double* l, const double* r, const PhysParams& ph, double* f) {
  const double cl = sound_nr(ph.gamma * l[4], l[0]);
  const double cr = sound_nr(ph.gamma * r[4], r[0]);
  double fx[NEQ];
  if constexpr (SOLVER == WX_SOLVER_HLLC) riemann_hllc_c<NEQ>(l, r, cl, cr, fx, ph.cv);
  else riemann_hll_c<NEQ>(l, r, cl, cr, fx, ph.cv);
#pragma unroll
  for (int e = 0; e < NEQ; ++e) f[perm<DIR, false>(e)] = fx[e];
}

template <int NEQ, bool VISC>
__host__ __device__ constexpr int corr_ctas_per_sm() {
  return 2 * (sizeof(CorrSmem<NEQ, VISC>) + 1024) <= 228 * 1024 ? 2 : 1;
}

template <int NEQ, int SOLVER, int LIM, bool VISC>
__global__ void __launch_bounds__(STAGE_THREADS, (corr_ctas_per_sm<NEQ, VISC>())) corrector_kernel(StageParams P) {
  extern __shared__ __align__(16) unsigned char smraw[];
  CorrSmem<NEQ, VISC>& S = *reinterpret_cast<CorrSmem<NEQ, VISC>*>(smraw);
  constexpr int W = CorrSmem<NEQ, VISC>::W, PL = CorrSmem<NEQ, VISC>::PL;
  DevBlock& B = S.B;
  StageConsts& K = S.K;
  const int t = threadIdx.x, lane = t & (NC - 1);
  const PhysParams& ph = P.ph;
  const int planes = NC / P.zsplit;
  const bool column = t < PLANE;
  const int ci = lane + 1, cj = (t >> 4) + 1;                  // column threads
  const int q = t - PLANE, side = q >> 4;                      // face threads: 0, 1 x; 2, 3 y
  const bool high = side & 1;
  const int gi = side == 0 ? 0 : (side == 1 ? NC + 1 : lane + 1);   // inner ghost
  const int gj = side == 2 ? 0 : (side == 3 ? NC + 1 : lane + 1);
  const int oi = side == 0 ? -1 : (side == 1 ? NC + 2 : lane + 1);  // outer ghost
  const int oj = side == 2 ? -1 : (side == 3 ? NC + 2 : lane + 1);
  const int h = column ? ci + W * cj : gi + W * gj;            // place in a framed plane
  const double* gsrc = P.gsrc ? P.gsrc : P.src;
  Cfl<NEQ, false> cfl;
  if (t < 4) K.cnt[t] = 0;

  for (int w = blockIdx.x; w < P.nwork;) {
    const int slot = P.work[w / P.zsplit];
    const int z0 = 1 + (w % P.zsplit) * planes, z1 = z0 + planes - 1;
    __syncthreads();
    if (t < (int)(sizeof(DevBlock) / 4)) reinterpret_cast<int*>(&B)[t] = reinterpret_cast<const int*>(P.blocks + slot)[t];
    __syncthreads();
    if (t == 0) {  // read after the prologue's barrier
      const double dtp = P.ctl->dt * P.dt_factor;
      K.dtdx = dtp / B.dx;
      K.dtdy = dtp / B.dy;
      K.dtdz = dtp / B.dz;
      K.idx = 1.0 / B.dx;
      K.idy = 1.0 / B.dy;
      K.idz = 1.0 / B.dz;
    }
    if (column) {
      // conserved variables of the column's cell in plane kk
      auto load = [&](int kk, double* u) {
        if (kk >= 1 && kk <= NC) load_cell<NEQ>(P.src, slot, ci, cj, kk, u);
        else gather_ghost<NEQ>(gsrc, B, slot, ci, cj, kk, u);
      };
      // the same into the plane's place in shared memory, asynchronously where
      // it is a plain copy; the thread itself converts it (to_plane)
      auto fetch = [&](int kk) {
        double* d = &S.pl[(unsigned)(kk + 3) % 3u][0][h];
        if (kk >= 1 && kk <= NC) {
          const double* g = P.src + cell_off(slot, NEQ, 0, ci, cj, kk);
#pragma unroll
          for (int e = 0; e < NEQ; ++e) copy_async8(d + e * PL, g + (size_t)e * BCELLS);
        } else {
          double u[NEQ];
          gather_ghost<NEQ>(gsrc, B, slot, ci, cj, kk, u);
#pragma unroll
          for (int e = 0; e < NEQ; ++e) d[e * PL] = u[e];
        }
      };
      auto to_prim = [&](int kk, const double* u, double* p) {
        const int st = flow2prim<NEQ, false>(u, p, ph.inv_cv);
        if (st != 0 && kk >= z0 && kk <= z1) atomicAdd(&K.cnt[st == 1 ? 0 : (st == 2 ? 1 : 2)], 1u);
      };
      auto to_plane = [&](int kk, double* p) {
        double* d = &S.pl[(unsigned)(kk + 3) % 3u][0][h];
        double u[NEQ];
#pragma unroll
        for (int e = 0; e < NEQ; ++e) u[e] = d[e * PL];
        to_prim(kk, u, p);
#pragma unroll
        for (int e = 0; e < NEQ; ++e) d[e * PL] = p[e];
      };
      double lz[NEQ], zf[NEQ];
      {  // planes z0-2 .. z0+1 and the z-interface z0-1/2; plane z0+2 on its way
        double u[NEQ], p0[NEQ], p1[NEQ], pc[NEQ], pu[NEQ], l[NEQ], r[NEQ];
        fetch(z0);
        fetch(z0 + 1);
        fetch(z0 + 2);
        load(z0 - 2, u);
        to_prim(z0 - 2, u, p0);
        load(z0 - 1, u);
        if (VISC) {  // W(z0-1) of the column: the bottom UP ghost
#pragma unroll
          for (int e = 0; e < NEQ; ++e) S.w[(z0 - 1) & 1][e][h] = u[e];
        }
        to_prim(z0 - 1, u, p1);
        copy_async_wait();
        to_plane(z0, pc);
        to_plane(z0 + 1, pu);
#pragma unroll
        for (int e = 0; e < NEQ; ++e) {
          const int k = perm<2, false>(e);
          const double dm = pc[k] - p1[k];
          l[e] = p1[k] + 0.5 * average_t<LIM>(p1[k] - p0[k], dm, ph.limiter);
          const double s = average_t<LIM>(dm, pu[k] - pc[k], ph.limiter);
          r[e] = pc[k] - 0.5 * s;
          lz[e] = pc[k] + 0.5 * s;
        }
        state_flux<NEQ, SOLVER, 2>(l, r, ph, zf);
      }
      plane_barrier();

      for (int m = z0; m <= z1; ++m) {
        const int b = m & 1;
        double dx[NEQ], dz[NEQ], f[NEQ], v[NEQ], pc[NEQ];
        // the base plane after this one into L2 (16 lines per equation)
        if (t < 16 * NEQ && m < z1) prefetch_l2(P.base + cell_off(slot, NEQ, t >> 4, 1, 1, m + 1) + (size_t)(t & 15) * 16);
        const double* pp = &S.pl[(unsigned)m % 3u][0][h];
#pragma unroll
        for (int e = 0; e < NEQ; ++e) pc[e] = pp[e * PL];
        {  // y-interface to row cj+1 (the last row's flux is a face thread's)
          double l[NEQ], r[NEQ];
          const int o2 = cj < NC ? 2 * W : W;
#pragma unroll
          for (int e = 0; e < NEQ; ++e) {
            const int k = perm<1, false>(e);
            const double a = pp[k * PL + W], dm = a - pc[k];
            l[e] = pc[k] + 0.5 * average_t<LIM>(pc[k] - pp[k * PL - W], dm, ph.limiter);
            r[e] = a - 0.5 * average_t<LIM>(dm, pp[k * PL + o2] - a, ph.limiter);
          }
          state_flux<NEQ, SOLVER, 1>(l, r, ph, f);
          if (cj < NC) {
#pragma unroll
            for (int e = 0; e < NEQ; ++e) S.fy[b][e][cj * NC + lane] = f[e];
          }
        }
        {  // x-interface to cell ci+1 (the last lane's flux is a face thread's)
          double l[NEQ], r[NEQ];
#pragma unroll
          for (int e = 0; e < NEQ; ++e) {
            const double s = average_t<LIM>(pc[e] - pp[e * PL - 1], pp[e * PL + 1] - pc[e], ph.limiter);
            l[e] = pc[e] + 0.5 * s;
            r[e] = __shfl_down_sync(0xffffffffu, pc[e] - 0.5 * s, 1, NC);
          }
          state_flux<NEQ, SOLVER, 0>(l, r, ph, f);
#pragma unroll
          for (int e = 0; e < NEQ; ++e) {
            const double xl = __shfl_up_sync(0xffffffffu, f[e], 1, NC);
            dx[e] = lane == 0 ? -f[e] : (lane == NC - 1 ? xl : xl - f[e]);
          }
        }
        {  // z-interface m+1/2: the column's own cells
          const double* pa = &S.pl[(unsigned)(m + 1) % 3u][0][h];
          double l[NEQ], r[NEQ], pu[NEQ];
          if (m > z0) copy_async_wait();
          to_plane(m + 2, pu);
#pragma unroll
          for (int e = 0; e < NEQ; ++e) {
            const int k = perm<2, false>(e);
            const double a = pa[k * PL];
            const double s = average_t<LIM>(a - pc[k], pu[k] - a, ph.limiter);
            r[e] = a - 0.5 * s;
            l[e] = lz[e];
            lz[e] = a + 0.5 * s;
          }
          state_flux<NEQ, SOLVER, 2>(l, r, ph, f);
#pragma unroll
          for (int e = 0; e < NEQ; ++e) {
            dz[e] = zf[e] - f[e];
            zf[e] = f[e];
          }
        }
        const size_t o = cell_off(slot, NEQ, 0, ci, cj, m);
#pragma unroll
        for (int e = 0; e < NEQ; ++e) v[e] = __ldg(P.base + o + (size_t)e * BCELLS);
        plane_barrier();
        // conservative update of plane m (godunov.f90:259-271); each
        // direction's two fluxes are subtracted before they are scaled, so
        // equal fluxes cancel exactly
        const double dtdx = K.dtdx, dtdy = K.dtdy, dtdz = K.dtdz;
        const bool xedge = lane == 0 || lane == NC - 1;
        const double* ex = &S.ex[b][lane >> 3][0][cj - 1];
#pragma unroll
        for (int e = 0; e < NEQ; ++e) {
          const double xe = xedge ? ex[e * NC] : 0.0;
          const double ddx = dx[e] + (lane == 0 ? xe : -xe);
          const double dy = S.fy[b][e][(cj - 1) * NC + lane] - S.fy[b][e][cj * NC + lane];
          v[e] = v[e] + dtdx * ddx + dtdy * dy + dtdz * dz[e];
          if (!VISC) P.out[o + (size_t)e * BCELLS] = v[e];
        }
        if (VISC) {  // W(m) over W(m-2) of the column, and the viscous step of plane m-1
#pragma unroll
          for (int e = 0; e < NEQ; ++e) {
            const double* pw = &S.w[b ^ 1][e][h];
            const double below = S.w[b][e][h];
            S.w[b][e][h] = v[e];
            v[e] = pw[0] + ph.eta * ((pw[1] + pw[-1]) + (pw[W] + pw[-W]) + (v[e] + below) - 6.0 * pw[0]);
          }
          if (m > z0) visc_store<NEQ, false>(P, v, o - NC * NC, cfl, K);
        }
        if (m < z1) fetch(m + 3);  // over plane m, which no one reads any more
      }
      if (VISC) {  // plane z1: above it, the top UP ghost
        double g[NEQ], un[NEQ];
        gather_ghost<NEQ>(gsrc, B, slot, ci, cj, z1 + 1, g);
        plane_barrier();
#pragma unroll
        for (int e = 0; e < NEQ; ++e) {
          const double* pw = &S.w[z1 & 1][e][h];
          un[e] = pw[0] + ph.eta * ((pw[1] + pw[-1]) + (pw[W] + pw[-W]) + (g[e] + S.w[(z1 - 1) & 1][e][h]) - 6.0 * pw[0]);
        }
        visc_store<NEQ, false>(P, un, cell_off(slot, NEQ, 0, ci, cj, z1), cfl, K);
      }
    } else {
      double g2[NEQ];  // primitives of the outer ghost; the inner one's are in the frame
      auto take = [&](int kk, const double* u1, const double* u2) {
        double g1[NEQ];
        flow2prim<NEQ, false>(u1, g1, ph.inv_cv);
        flow2prim<NEQ, false>(u2, g2, ph.inv_cv);
#pragma unroll
        for (int e = 0; e < NEQ; ++e) {
          S.pl[(unsigned)kk % 3u][e][h] = g1[e];
          if (VISC) S.wg[kk & 1][e][q] = u1[e];
        }
      };
      // face state of the block-face interface from its four cells in order
      auto faces = [&](const double* pg, int step, auto dir) {
        constexpr int DIR = decltype(dir)::value;
        double l[NEQ], r[NEQ], f[NEQ];
#pragma unroll
        for (int e = 0; e < NEQ; ++e) {
          const int k = perm<DIR, false>(e);
          const double g = pg[k * PL], a = pg[k * PL + step], a2 = pg[k * PL + 2 * step];
          const double c0 = high ? a2 : g2[k], c1 = high ? a : g, c2 = high ? g : a, c3 = high ? g2[k] : a2;
          const double dm = c2 - c1;
          l[e] = c1 + 0.5 * average_t<LIM>(c1 - c0, dm, ph.limiter);
          r[e] = c2 - 0.5 * average_t<LIM>(dm, c3 - c2, ph.limiter);
        }
        state_flux<NEQ, SOLVER, DIR>(l, r, ph, f);
        return Flux<NEQ>(f);
      };
      // both ghost layers of plane kk; across an x face to a same-level block
      // they are two adjacent cells of a row, one 16-byte load per equation
      // (each of the 32 lanes reads another line there)
      const bool pair = side < 2 && B.ftype[side] == WX_NEIGH_SAME;
      const double* row = pair ? gsrc + cell_off(B.fnb[side][0], NEQ, 0, high ? 1 : NC - 1, gj, 1) : nullptr;
      auto fetch = [&](int kk) {
        double u1[NEQ], u2[NEQ];
        if (pair) {
#pragma unroll
          for (int e = 0; e < NEQ; ++e) {
            const double2 v = __ldg(reinterpret_cast<const double2*>(row + (size_t)e * BCELLS + (kk - 1) * PLANE));
            u1[e] = high ? v.x : v.y;
            u2[e] = high ? v.y : v.x;
          }
        } else {
          gather_ghost<NEQ>(gsrc, B, slot, gi, gj, kk, u1);
          gather_ghost<NEQ>(gsrc, B, slot, oi, oj, kk, u2);
        }
        take(kk, u1, u2);
      };
      fetch(z0);
      plane_barrier();
      for (int m = z0; m <= z1; ++m) {
        const int b = m & 1;
        if (side < 2) {
          const Flux<NEQ> f = faces(&S.pl[(unsigned)m % 3u][0][h], high ? -1 : 1, Dir<0>());
#pragma unroll
          for (int e = 0; e < NEQ; ++e) S.ex[b][side][e][lane] = f.v[e];
        } else {
          const Flux<NEQ> f = faces(&S.pl[(unsigned)m % 3u][0][h], high ? -W : W, Dir<1>());
#pragma unroll
          for (int e = 0; e < NEQ; ++e) S.fy[b][e][(high ? NC * NC : 0) + lane] = f.v[e];
        }
        if (m < z1) fetch(m + 1);
        plane_barrier();
        if (VISC) {
#pragma unroll
          for (int e = 0; e < NEQ; ++e) S.w[b][e][h] = S.wg[b][e][q];
        }
      }
      if (VISC) plane_barrier();
    }
    // items past the first wave go, in list order, to whichever CTA
    // finishes first (the counter is zeroed before each launch)
    if (t == 0) K.next = (int)gridDim.x + (int)atomicAdd(&P.ctl->work_next[1], 1u);
    __syncthreads();
    w = K.next;
  }
  if (VISC && P.do_dt) block_min_dt(cfl.dt(), P.ctl);
  __syncthreads();
  if (t < 4 && K.cnt[t]) atomicAdd(&P.ctl->cnt[t], (unsigned long long)K.cnt[t]);
}

// ---------------------------------------------------------------------------
// Lax-Friedrichs (lax.f90:39-99): first order, from U with one-deep ghosts.
struct LaxParams {
  const double* __restrict__ u;
  double* __restrict__ out;
  const DevBlock* __restrict__ blocks;
  const int32_t* __restrict__ work;
  int32_t nwork;
  DevCtl* ctl;
  PhysParams ph;
};

template <int NEQ, bool MHD>
__global__ void __launch_bounds__(256) lax_kernel(LaxParams P) {
  __shared__ DevBlock B;
  const int t = threadIdx.x;
  const int i = (t & 15) + 1, j = (t >> 4) + 1;
  for (int w = blockIdx.x; w < P.nwork; w += gridDim.x) {
    const int slot = P.work[w];
    __syncthreads();
    if (t < (int)(sizeof(DevBlock) / 4)) reinterpret_cast<int*>(&B)[t] = reinterpret_cast<const int*>(P.blocks + slot)[t];
    __syncthreads();
    const double dt = P.ctl->dt;
    const double cx = 0.5 * dt / B.dx, cy = 0.5 * dt / B.dy, cz = 0.5 * dt / B.dz;
    for (int k = 1; k <= NC; ++k) {
      double un[6][NEQ], fl[NEQ], fr[NEQ], pv[NEQ], tmp[NEQ];
      const int di[6] = {1, -1, 0, 0, 0, 0}, dj[6] = {0, 0, 1, -1, 0, 0}, dk[6] = {0, 0, 0, 0, 1, -1};
#pragma unroll
      for (int q = 0; q < 6; ++q) get_cell<NEQ>(P.u, B, slot, i + di[q], j + dj[q], k + dk[q], un[q]);
      double res[NEQ];
#pragma unroll
      for (int e = 0; e < NEQ; ++e)
        res[e] = (un[0][e] + un[1][e] + un[2][e] + un[3][e] + un[4][e] + un[5][e]) / 6.0;
      // physical fluxes of the neighbour primitives, direction by direction
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const double cc = d == 0 ? cx : (d == 1 ? cy : cz);
        flow2prim<NEQ, MHD>(un[2 * d], pv, P.ph.inv_cv);
#pragma unroll
        for (int e = 0; e < NEQ; ++e) tmp[e] = pv[d == 0 ? e : (d == 1 ? perm<1, MHD>(e) : perm<2, MHD>(e))];
        xflux<NEQ, MHD>(tmp, fr, P.ph.cv);
        flow2prim<NEQ, MHD>(un[2 * d + 1], pv, P.ph.inv_cv);
#pragma unroll
        for (int e = 0; e < NEQ; ++e) tmp[e] = pv[d == 0 ? e : (d == 1 ? perm<1, MHD>(e) : perm<2, MHD>(e))];
        xflux<NEQ, MHD>(tmp, fl, P.ph.cv);
#pragma unroll
        for (int e = 0; e < NEQ; ++e) {
          const int q = d == 0 ? e : (d == 1 ? perm<1, MHD>(e) : perm<2, MHD>(e));
          res[q] = res[q] - cc * (fr[e] - fl[e]);
        }
      }
      const size_t o = cell_off(slot, NEQ, 0, i, j, k);
#pragma unroll
      for (int e = 0; e < NEQ; ++e) P.out[o + (size_t)e * BCELLS] = res[e];
    }
  }
}

// ---------------------------------------------------------------------------
// doViscousStep (hydro_solver.f90:217-250) with the next step's CFL minimum
// (hydro_solver.f90:150-182) of the new state fused into the epilogue.
struct ViscParams {
  double* __restrict__ w;              // stage result, overwritten in place by U^{n+1}
  const double* __restrict__ up;       // predictor state: source of the face ghosts
  const DevBlock* __restrict__ blocks;
  const int32_t* __restrict__ work;
  int32_t zsplit;                      // CTAs per block, one cluster (1, 2, 4 or 8)
  int32_t zero_ghost;                  // single-stage solvers: UP ghosts are never filled (0)
  int32_t do_dt;                       // fold the CFL minimum of the new state
  DevCtl* ctl;
  PhysParams ph;
};

// One CTA per block, or a cluster of S CTAs that split its planes where the
// mesh has too few blocks (launch_viscous).  HBM-bound: W is read and written
// once, the ghosts of UP once.  Columns copy their cells a few planes ahead
// into a ring of shared planes (no registers held while a load is in flight)
// and warps 8 and 9 gather the frame from UP a plane ahead, so three CTAs per
// SM keep about 60 KB of loads in flight; one barrier per plane.  The update
// is in place: the planes just outside a slab are read before the cluster's
// barrier, and the first write follows it.  11,600 blocks of five equations:
// 1.57 -> 1.02 ms (the x-face ghosts cost a 32-byte sector per cell: with
// them 5.1 GB, 0.79 ms at the copy rate); 20,896 blocks of six: 2.87 -> 2.32
// ms.  64 blocks in clusters of eight: 26 -> 16 us; 16 MHD blocks: 54 -> 14.
constexpr int VRING = 4;
template <int NEQ>
struct ViscSmem {
  double pl[VRING][NEQ][VPLANE];   // planes of W with the one-deep ghost frame from UP
  double dt[8];
  DevBlock B;
};

template <int NEQ, bool MHD>
__global__ void __launch_bounds__(STAGE_THREADS, NEQ <= 6 ? 3 : 2) viscous_kernel(ViscParams P) {
  extern __shared__ __align__(16) unsigned char smraw[];
  ViscSmem<NEQ>& S = *reinterpret_cast<ViscSmem<NEQ>*>(smraw);
  DevBlock& B = S.B;
  const int t = threadIdx.x, lane = t & (NC - 1);
  const int slot = P.work[blockIdx.x / P.zsplit];
  const int planes = NC / P.zsplit, z0 = 1 + (blockIdx.x % P.zsplit) * planes, z1 = z0 + planes - 1;
  const double eta = P.ph.eta;
  if (t < (int)(sizeof(DevBlock) / 4)) reinterpret_cast<int*>(&B)[t] = reinterpret_cast<const int*>(P.blocks + slot)[t];
  __syncthreads();
  unsigned nonfinite = 0;
  if (t < PLANE) {
    const int i = lane + 1, j = (t >> 4) + 1, h = i + (NC + 2) * j;
    double* d0 = &S.pl[0][0][h];
    double* w0 = P.w + cell_off(slot, NEQ, 0, i, j, 1);
    auto fetch = [&](int k) {
      double* d = d0 + (k & (VRING - 1)) * (NEQ * VPLANE);
      const double* g = w0 + (k - 1) * PLANE;
#pragma unroll
      for (int e = 0; e < NEQ; ++e) copy_async8(d + e * VPLANE, g + (size_t)e * BCELLS);
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // the column's cells below and above the slab
    auto outside = [&](int k, double* u) {
      if (k >= 1 && k <= NC) {
        load_cell_rw<NEQ>(P.w, slot, i, j, k, u);
      } else if (P.zero_ghost) {
#pragma unroll
        for (int e = 0; e < NEQ; ++e) u[e] = 0.0;
      } else {
        gather_ghost<NEQ>(P.up, B, slot, i, j, k, u);
      }
    };
    // one group per plane, empty past the slab, so the group counts match
    for (int k = z0; k < z0 + 3; ++k) {
      if (k <= z1) fetch(k);
      else asm volatile("cp.async.commit_group;" ::: "memory");
    }
    double wm[NEQ], wt[NEQ];
    outside(z0 - 1, wm);
    outside(z1 + 1, wt);
    Cfl<NEQ, MHD> cfl;
    cfl.block(B);
    if (P.zsplit > 1) cluster_barrier();
    for (int k = z0; k <= z1; ++k) {
      asm volatile("cp.async.wait_group 1;" ::: "memory");   // planes up to k+1
      plane_barrier();
      if (k + 3 <= z1) fetch(k + 3);                          // over plane k-1
      else asm volatile("cp.async.commit_group;" ::: "memory");
      const double* p = d0 + (k & (VRING - 1)) * (NEQ * VPLANE);
      const double* pn = d0 + ((k + 1) & (VRING - 1)) * (NEQ * VPLANE);
      double un[NEQ];
      double* o = w0 + (k - 1) * PLANE;
#pragma unroll
      for (int e = 0; e < NEQ; ++e) {
        const double* q = p + e * VPLANE;
        const double c = q[0], up = k < z1 ? pn[e * VPLANE] : wt[e];
        un[e] = c + eta * (+q[1] + q[-1] + q[NC + 2] + q[-(NC + 2)] + up + wm[e] - 6.0 * c);
        wm[e] = c;
        o[(size_t)e * BCELLS] = un[e];
        nonfinite += !isfinite(un[e]);
      }
      if (P.do_dt) {
        double v[NEQ], rinv;
        flow2prim<NEQ, MHD>(un, v, P.ph.inv_cv, &rinv);
        cfl.fold(v, rinv, P.ph.gamma);
      }
    }
    if (P.do_dt) {
      double v = cfl.dt();
      for (int s = 16; s > 0; s >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, s));
      if ((t & 31) == 0) S.dt[t >> 5] = v;
    }
    nonfinite = __reduce_add_sync(0xffffffffu, nonfinite);
    if ((t & 31) == 0 && nonfinite) atomicAdd(&P.ctl->cnt[3], (unsigned long long)nonfinite);
  } else {  // the frame cell of one (side, row) from UP
    const int side = (t - PLANE) >> 4;
    const int gi = side == 0 ? 0 : (side == 1 ? NC + 1 : lane + 1);
    const int gj = side == 2 ? 0 : (side == 3 ? NC + 1 : lane + 1);
    double* d0 = &S.pl[0][0][gi + (NC + 2) * gj];
    double u[NEQ];
    auto take = [&](int k) {
      if (P.zero_ghost) {
#pragma unroll
        for (int e = 0; e < NEQ; ++e) u[e] = 0.0;
      } else {
        gather_ghost<NEQ>(P.up, B, slot, gi, gj, k, u);
      }
    };
    take(z0);
    if (P.zsplit > 1) cluster_barrier();
    for (int k = z0; k <= z1; ++k) {
      double* d = d0 + (k & (VRING - 1)) * (NEQ * VPLANE);
#pragma unroll
      for (int e = 0; e < NEQ; ++e) d[e * VPLANE] = u[e];
      if (k < z1) take(k + 1);
      plane_barrier();
    }
  }
  if (P.do_dt) {
    __syncthreads();
    if (t == 0) {
      double v = S.dt[0];
      for (int k = 1; k < 8; ++k) v = fmin(v, S.dt[k]);
      atomic_min_pos(&P.ctl->dtmin_bits, v);
    }
  }
}

// CFL minimum of an arbitrary state (getTimestep's loop, hydro_solver.f90:150-182).
struct DtParams {
  const double* __restrict__ u;
  const DevBlock* __restrict__ blocks;
  const int32_t* __restrict__ work;
  int32_t nwork;
  DevCtl* ctl;
  PhysParams ph;
};

// Items of two planes, so that a mesh of a few blocks still spreads over the
// SMs (8 blocks: 10 -> 4 us).
constexpr int DT_PLANES = 2;
template <int NEQ, bool MHD>
__global__ void __launch_bounds__(256) dt_kernel(DtParams P) {
  const int t = threadIdx.x;
  Cfl<NEQ, MHD> cfl;
  for (int w = blockIdx.x; w < P.nwork * (NC / DT_PLANES); w += gridDim.x) {
    const int slot = P.work[w / (NC / DT_PLANES)], k0 = w % (NC / DT_PLANES) * DT_PLANES;
    const DevBlock& B = P.blocks[slot];
    double u[DT_PLANES][NEQ], p[NEQ], rinv;
#pragma unroll
    for (int k = 0; k < DT_PLANES; ++k) load_cell<NEQ>(P.u, slot, (t & 15) + 1, (t >> 4) + 1, k0 + k + 1, u[k]);
    cfl.block(B);
#pragma unroll
    for (int k = 0; k < DT_PLANES; ++k) {
      flow2prim<NEQ, MHD>(u[k], p, P.ph.inv_cv, &rinv);
      cfl.fold(p, rinv, P.ph.gamma);
    }
  }
  block_min_dt(cfl.dt(), P.ctl);
}

__global__ void ctl_reset_dtmin_kernel(DevCtl* ctl) {
  if (threadIdx.x == 0) ctl->dtmin_bits = (unsigned long long)__double_as_longlong(1.0e30);
}

// getTimestep's scalar tail (hydro_solver.f90:185-207) and the iteration
// counter of main.f90:81.  Single thread.
__global__ void step_begin_kernel(DevCtl* ctl, double cfl, int cooling_on, double dtout, double t_sc, int bump_it) {
  if (threadIdx.x != 0) return;
  if (bump_it) ctl->it = ctl->it + 1;
  const double dt_hydro = __longlong_as_double((long long)ctl->dtmin_bits);
  const double dt_cool = 1.0e30;
  double dt_loc = cooling_on ? dmin(dt_hydro, dt_cool) * cfl : dt_hydro * cfl;
  if (ctl->it <= 10) dt_loc = exp2(-(double)(11 - ctl->it)) * dt_loc;
  double dt_glob = dt_loc;
  const double tnext = (double)ctl->nextout * dtout / t_sc;
  if (ctl->time + dt_glob >= tnext) {
    dt_glob = tnext - ctl->time;
    ctl->dumpout = 1;
  }
  ctl->dt = dt_glob;
  ctl->work_next[0] = ctl->work_next[1] = 0;
  ctl->dtmin_bits = (unsigned long long)__double_as_longlong(1.0e30);
}

// time += dt (hydro_solver.f90:225) and, when the call stands for a whole
// main-loop iteration, the output bookkeeping of main.f90:109-114 (the
// output itself belongs to the host).
__global__ void step_end_kernel(DevCtl* ctl, int finish_output) {
  if (threadIdx.x != 0) return;
  ctl->time = ctl->time + ctl->dt;
  if (finish_output && ctl->dumpout) {
    ctl->nextout = ctl->nextout + 1;
    ctl->dumpout = 0;
    ctl->dumps = ctl->dumps + 1;
  }
}

// ---------------------------------------------------------------------------
// userBoundary of the wind problems: imposes the wind on the physical cells
// of `u` inside the spheres (blocks flagged in the neighbour table only).
// A ghost in a sphere is then gathered from a same-level neighbour whose
// cell at the same position carries the same imposed value
// (wx3d_set_winds refuses meshes where a coarse/fine face's ghost layer
// meets a sphere).
struct WindParams {
  double* __restrict__ u;
  const DevBlock* __restrict__ blocks;
  const int32_t* __restrict__ work;
  int32_t nwork;
  PhysParams ph;
};

// Copies whole blocks within one array: slot pairs (from, to), one row of
// CTAs per pair.
__global__ void copy_slots_kernel(double* u, const int2* __restrict__ pairs, int neq) {
  const int2 pr = pairs[blockIdx.y];
  const size_t n = (size_t)neq * BCELLS;
  const double* from = u + (size_t)pr.x * n;
  double* to = u + (size_t)pr.y * n;
  for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x)
    to[c] = from[c];
}

template <int NEQ, bool MHD>
__global__ void __launch_bounds__(256) wind_kernel(WindParams P) {
  for (int w = blockIdx.x; w < P.nwork; w += gridDim.x) {
    const int slot = P.work[w];
    const DevBlock& B = P.blocks[slot];
    if (!B.wind) continue;
    for (int c = threadIdx.x; c < BCELLS; c += blockDim.x) {
      const int i = (c & 15) + 1, j = ((c >> 4) & 15) + 1, k = (c >> 8) + 1;
      double u[NEQ];
      if (wind_state<NEQ, MHD>(P.ph, B, i, j, k, u)) {
        const size_t o = cell_off(slot, NEQ, 0, i, j, k);
#pragma unroll
        for (int e = 0; e < NEQ; ++e) P.u[o + (size_t)e * BCELLS] = u[e];
      }
    }
  }
}

}  // namespace wx
