// Kernel templates of the LBM step.  Included by one translation unit per
// population storage type (lbm_inst_*.cu), which instantiates Ops<PopT>.
//
// Two execution forms share one device state:
//  * phase-by-phase kernels that mirror the reference's seven Sim methods one
//    to one (src/sim.js:176-582), for callers that invoke them individually;
//  * the fused step: a z-marching kernel that, per cell, pulls the 27 + 7
//    populations of its neighbours, applies each source cell's BGK collision on
//    the fly from per-cell collision coefficients staged in shared memory,
//    streams with halfway bounce-back / moving-wall correction, and writes the
//    new populations and macros -- one read and one write of every state array
//    per step.
#pragma once

#include <stdio.h>

#include "lbm_core.cuh"

namespace lbm {

template <class PopT>
struct Prec {
  using Real = float;
};
template <>
struct Prec<double> {
  using Real = double;
};

inline unsigned nblocks(long long n, int t) { return (unsigned)((n + t - 1) / t); }

__device__ __forceinline__ long long cell_index(int x, int y, int z, int nx, int ny) {
  return ((long long)z * ny + y) * nx + x;
}

// The reference's phase loops run over 1..n-2 on every axis (src/sim.js:334-338);
// cells on the boundary are never collided or streamed, whatever their tag.
__device__ __forceinline__ bool interior_cell(long long i, int nx, int ny, int nz) {
  int x = (int)(i % nx);
  long long t = i / nx;
  int y = (int)(t % ny);
  int z = (int)(t / ny);
  return x >= 1 && x <= nx - 2 && y >= 1 && y <= ny - 2 && z >= 1 && z <= nz - 2;
}

// Weight tables usable with a runtime index (generic kernels, host code).
__host__ __device__ inline float w27_of(int k) {
  int nnz = (dcomp(k, 0) != 0) + (dcomp(k, 1) != 0) + (dcomp(k, 2) != 0);
  return (float)(nnz == 0 ? 8.0 / 27.0 : nnz == 1 ? 2.0 / 27.0 : nnz == 2 ? 1.0 / 54.0 : 1.0 / 216.0);
}
__host__ __device__ inline float w7_of(int k) { return (float)(k == 0 ? 0.25 : 0.125); }
__host__ __device__ inline int opp_of(int k) { return k == 0 ? 0 : ((k & 1) ? k + 1 : k - 1); }

__device__ __forceinline__ void flush_impulse(const SolidSet &ss, int owner, int x, int y, int z,
                                              double acc[6]) {
  if (owner < 0) return;
  const ImpulseTarget &t = ss.imp[owner];
  int lx = x - t.lo[0], ly = y - t.lo[1], lz = z - t.lo[2];
  if (lx < 0 || ly < 0 || lz < 0 || lx >= t.dim[0] || ly >= t.dim[1] || lz >= t.dim[2]) return;
  double *slot = t.acc + 6 * (((long long)lz * t.dim[1] + ly) * t.dim[0] + lx);
#pragma unroll
  for (int j = 0; j < 6; j++) {
    slot[j] = __dadd_rn(slot[j], acc[j]);
    acc[j] = 0.0;
  }
}

// =====================================================================================
// init (src/sim.js:112-134): both ping-pong halves receive identical values so
// that walls, which are never rewritten, read the same from either half.
template <class PopT>
__global__ void k_init_flat(Scene<PopT, typename Prec<PopT>::Real> s, const double *phiCol) {
  using Real = typename Prec<PopT>::Real;
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= s.n) return;
  int x = (int)(i % s.nx);
  long long t = i / s.nx;
  int y = (int)(t % s.ny);
  int z = (int)(t / s.ny);
  double pc = phiCol[y];
  bool wall = x == 0 || x == s.nx - 1 || y == 0 || y == s.ny - 1 || z == 0 || z == s.nz - 1;
  Real phiR = (Real)pc;
  for (int c = 0; c < 2; c++) {
    s.phi[c][i] = phiR;
    s.rho[c][i] = (Real)1.0;
    s.set_ux(c, i, (Real)0);
    s.set_uy(c, i, (Real)0);
    s.uz[c][i] = (Real)0;
    for (int k = 0; k < Q27; k++) {
      Real w = (Real)w27_of(k);
      s.F[c][pidx<27>(k, i)] = Codec<PopT>::enc(w, w);
    }
    for (int k = 0; k < Q7; k++) {
      Real hv = (Real)((double)w7_of(k) * pc);
      s.H[c][pidx<7>(k, i)] = Codec<PopT>::enc(hv, (Real)w7_of(k) * phiR);
    }
  }
  uint8_t tg = wall ? TAG_WALL : TAG_FLUID;
  s.tag[i] = tg;
  s.tagPrev[i] = tg;
}

// seedHydrostatic (src/sim.js:144-173): one thread per (z, x) column, y
// ascending, FP64 arithmetic; writes rho and f into both halves.
template <class PopT>
__global__ void k_seed_hydrostatic(Scene<PopT, typename Prec<PopT>::Real> s, int cur, double rhoL,
                                   double rhoG, double gravity) {
  using Real = typename Prec<PopT>::Real;
  long long col = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (col >= (long long)s.nx * s.nz) return;
  int x = (int)(col % s.nx);
  int z = (int)(col / s.nx);
  const double dRho = rhoL - rhoG;
  const double gOverCs2 = gravity * 3.0;
  const double uLatY = -0.5 * gravity;
  const double uLat2 = uLatY * uLatY;
  double pCs2 = 1.0;
  for (int y = 0; y < s.ny; y++) {
    long long i = cell_index(x, y, z, s.nx, s.ny);
    double rhoPhase = rhoG + (double)s.phi[cur][i] * dRho;
    for (int c = 0; c < 2; c++) s.rho[c][i] = (Real)pCs2;
    for (int k = 0; k < Q27; k++) {
      double eu = dcomp(k, 1) * uLatY;
      double Qi = eu * (3.0 + 4.5 * eu) - 1.5 * uLat2;
      double fk = (double)w27_of(k) * (pCs2 + rhoPhase * Qi);
      Real w = (Real)w27_of(k);
      PopT e = Codec<PopT>::enc((Real)fk, w);
      s.F[0][pidx<27>(k, i)] = e;
      s.F[1][pidx<27>(k, i)] = e;
    }
    pCs2 += rhoPhase * gOverCs2;
  }
}

// retagCells over the whole grid (src/sim.js:214-244): tagPrev <- tag,
// phiPrev <- phi, classification with FP64 contains, us = float(surfaceVelocity).
template <class PopT>
__global__ void k_retag_full(Scene<PopT, typename Prec<PopT>::Real> s, int cur,
                             const SolidSet *__restrict__ ssp) {
  const SolidSet &ss = *ssp;
  using Real = typename Prec<PopT>::Real;
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= s.n) return;
  const int nx = s.nx, ny = s.ny, nz = s.nz;
  const unsigned t = (unsigned)i / (unsigned)nx;  // (n < 2^31 cells)
  const int x = (int)((unsigned)i - t * (unsigned)nx), z = (int)(t / (unsigned)ny), y = (int)(t - (unsigned)z * (unsigned)ny);
  s.tagPrev[i] = s.tag[i];
  s.phi[1 - cur][i] = s.phi[cur][i];
  if (x == 0 || x == nx - 1 || y == 0 || y == ny - 1 || z == 0 || z == nz - 1) {
    s.tag[i] = TAG_WALL;
    s.usx[i] = s.usy[i] = s.usz[i] = (Real)0;
    return;
  }
  int b = owner_of<LBM_MAX_SPHERES>(ss.sph, ss.nsph, x, y, z);
  if (b >= 0) {
    double ox, oy, oz;
    sphere_surface_velocity(ss.sph[b], x, y, z, ox, oy, oz);
    s.tag[i] = TAG_SOLID;
    // stored like the reference's Float32Array us (double in the FP64 form)
    s.usx[i] = (Real)ox;
    s.usy[i] = (Real)oy;
    s.usz[i] = (Real)oz;
  } else {
    s.tag[i] = TAG_FLUID;
    s.usx[i] = s.usy[i] = s.usz[i] = (Real)0;
  }
}

// =====================================================================================
// Sparse passes around the spheres.

// Cells of a box in its linear (scan) order are worked on in chunks.
constexpr int COMPACT_CHUNK = 2048;
// Most CTAs a box sweep launches: the kernels stride over the box's chunks, so
// a step whose planned box is small does not pay for the empty CTAs of a
// launch sized for the largest possible box.
constexpr unsigned SWEEP_CTAS = 148 * 4;

__device__ __forceinline__ void box_cell(const Box &bx, long long l, int &x, int &y, int &z) {
  int dx = bx.hi[0] - bx.lo[0] + 1, dy = bx.hi[1] - bx.lo[1] + 1;
  x = bx.lo[0] + (int)(l % dx);
  y = bx.lo[1] + (int)((l / dx) % dy);
  z = bx.lo[2] + (int)(l / ((long long)dx * dy));
}

// handleFreshCells over the scan-ordered fresh list (src/sim.js:257-310): the
// FLUID neighbours' phi, rho and u averaged in the reference's neighbour order
// (dz, dy, dx ascending), then phi, phiPrev, rho, u and the equilibrium
// populations written.  The reference fills in scan order, in place: a fresh
// cell sees the filled values of fresh neighbours before it in scan order and
// the old values of those after it.
//
// FILL_GROUP cells of the list at a time: a lane per neighbour stages its five
// values, all in one memory latency; a thread per cell and value adds them in
// neighbour order; a lane per direction writes the populations.  The order
// between the cells of a group is kept by rounds: a cell is filled in the first
// round in which its fresh neighbours before it have been filled.  A z slab
// fills its own planes only (its copied planes receive the neighbouring slab's
// filled values).
// Latency-bound: with a thread per cell that went from neighbour to neighbour,
// one fresh cell took 31,000 cycles and twenty 75,000 to 118,000 (256^3, one
// sphere of radius 24); now 6,600, and 10,000 to 15,000.
constexpr int FILL_GROUP = 32;

template <class PopT, int THREADS>
__device__ __forceinline__ void fresh_fill_body(const Scene<PopT, typename Prec<PopT>::Real> &s, int cur,
                                                const int *fresh, int nf, double rhoL, double rhoG, int zlo,
                                                int zend) {
  using Real = typename Prec<PopT>::Real;
  constexpr int WARPS = THREADS / 32, OWN = 13;  // (neighbour 13 is the cell itself)
  static_assert(FILL_GROUP == 32 && FILL_GROUP % WARPS == 0 && THREADS >= 5 * FILL_GROUP, "");
  __shared__ Real sVal[FILL_GROUP][5][Q27];  // phi, rho, u of the neighbours (0 where not FLUID) and the cell's own
  __shared__ double sMean[FILL_GROUP][5];
  __shared__ int sRaw[FILL_GROUP], sIdx[FILL_GROUP];  // the cell; -1 where it is another slab's
  __shared__ int sCnt[FILL_GROUP];                    // its FLUID neighbours
  __shared__ uint32_t sNeed[FILL_GROUP], sDone;       // cells of the group it waits for; those filled
  __shared__ int8_t sDep[FILL_GROUP][OWN];            // place in the group of each neighbour before it, or -1
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nxny = s.nx * s.ny;
  const int dz = lane / 9 - 1, dy = lane / 3 % 3 - 1, dx = lane % 3 - 1;
  const int k = min(lane, Q27 - 1);  // the lane's direction
  const double ex = dcomp(k, 0), ey = dcomp(k, 1), ez = dcomp(k, 2);
  const float w = w27_of(k), w7 = w7_of(min(k, Q7 - 1));
  for (int g0 = 0; g0 < nf; g0 += FILL_GROUP) {
    const int m = min(FILL_GROUP, nf - g0);
    if (threadIdx.x < FILL_GROUP) {
      int i = -1;
      if (lane < m) {
        i = sRaw[lane] = fresh[g0 + lane];
        const int z = i / nxny;
        if (zend > 0 && (z < zlo || z >= zend)) i = -1;
      }
      sIdx[lane] = i;
      sNeed[lane] = 0;
      if (lane == 0) sDone = 0;
    }
    __syncthreads();
#pragma unroll 1
    for (int e = threadIdx.x; e < m * OWN; e += THREADS) {
      const int q = e / OWN, n = e - q * OWN, i = sIdx[q];
      const int j = i + (n / 9 - 1) * nxny + (n / 3 % 3 - 1) * s.nx + n % 3 - 1;
      int lo = 0, hi = q - 1, dep = -1;  // (the list is sorted by cell index)
      while (lo <= hi) {
        const int mid = (lo + hi) >> 1, at = sRaw[mid];
        if (at == j) dep = mid;
        if (at < j) lo = mid + 1;
        else hi = mid - 1;
      }
      if (i < 0 || dep >= 0 && sIdx[dep] < 0) dep = -1;
      sDep[q][n] = (int8_t)dep;
      if (dep >= 0) atomicOr(&sNeed[q], 1u << dep);
    }
#pragma unroll
    for (int t = 0; t < FILL_GROUP / WARPS; t++) {
      const int q = warp + t * WARPS, i = sIdx[q], j = i + dz * nxny + dy * s.nx + dx;
      if (i < 0 || lane >= Q27) continue;
      // (the tag from L2: other blocks of the same launch may have written it)
      const bool fluid = __ldcg(s.tag + j) == TAG_FLUID;
      const Real v[5] = {s.phi[cur][j], s.rho[cur][j], s.ux_at(cur, j), s.uy_at(cur, j), s.uz[cur][j]};
      for (int c = 0; c < 5; c++) sVal[q][c][lane] = fluid ? v[c] : (Real)0;
      if (lane == OWN) sVal[q][0][OWN] = v[0];
      const unsigned fl = __ballot_sync((1u << Q27) - 1, fluid && lane != OWN);
      if (lane == 0) sCnt[q] = __popc(fl);
    }
    __syncthreads();
    const int q = threadIdx.x / 5, c = threadIdx.x % 5;
    const int i = q < FILL_GROUP ? sIdx[q] : -1;
    bool waiting = i >= 0;
    while (__syncthreads_or(waiting)) {
      const uint32_t done = sDone;
      __syncthreads();
      if (waiting && !(sNeed[q] & ~done)) {
        double sum = 0;
#pragma unroll
        for (int n = 0; n < Q27; n++) {  // (a zero changes no sum)
          if (n == OWN) continue;
          const int dep = n < OWN ? sDep[q][n] : -1;
          sum += (double)(dep >= 0 ? sVal[dep][c][OWN] : sVal[q][c][n]);
        }
        const int cnt = sCnt[q];
        const double mean = cnt > 0 ? sum / cnt : c == 0 ? (double)sVal[q][0][OWN] : c == 1 ? 1.0 : 0.0;
        sMean[q][c] = mean;
        sVal[q][c][OWN] = (Real)mean;
        if (c == 0) s.phi[cur][i] = s.phi[1 - cur][i] = (Real)mean;  // phi and phiPrev
        if (c == 1) s.rho[cur][i] = (Real)mean;
        if (c == 2) s.set_ux(cur, i, (Real)mean);
        if (c == 3) s.set_uy(cur, i, (Real)mean);
        if (c == 4) s.uz[cur][i] = (Real)mean;
        if (c == 0) atomicOr(&sDone, 1u << q);
        waiting = false;
      }
    }
#pragma unroll 1
    for (int e = warp; e < m; e += WARPS) {
      const int at = sIdx[e];
      if (at < 0 || lane >= Q27) continue;
      const double p = sMean[e][0], r = sMean[e][1], vx = sMean[e][2], vy = sMean[e][3], vz = sMean[e][4];
      const double rhoPhase = rhoG + p * (rhoL - rhoG);
      const double u2 = vx * vx + vy * vy + vz * vz;
      const double eu = ex * vx + ey * vy + ez * vz;
      const double Qi = eu * (3.0 + 4.5 * eu) - 1.5 * u2;
      const double fk = (double)w * (r + rhoPhase * Qi);
      s.F[cur][pidx<27>(k, at)] = Codec<PopT>::enc((Real)fk, (Real)w);
      if (k < Q7) {
        const double hk = (double)w7 * p * (1 + 4.0 * eu);
        s.H[cur][pidx<7>(k, at)] = Codec<PopT>::enc((Real)hk, (Real)w7 * (Real)p);
      }
    }
    __syncthreads();
  }
}

// The same as the reference's loop, in place by one thread in list order: the
// test hook's fill (lbm_test_sequential_fill), which shares nothing with the
// one above.
template <class PopT>
__device__ __forceinline__ void fresh_fill_in_order(const Scene<PopT, typename Prec<PopT>::Real> &s, int cur,
                                                    const int *fresh, int nf, double rhoL, double rhoG, int zlo,
                                                    int zend) {
  using Real = typename Prec<PopT>::Real;
  const long long nxny = (long long)s.nx * s.ny;
  for (int q = 0; q < nf; q++) {
    const long long i = fresh[q], z = i / nxny;
    if (zend > 0 && (z < zlo || z >= zend)) continue;
    double ps = 0, rs = 0, xs = 0, ys = 0, zs = 0;
    int cnt = 0;
    for (int dz = -1; dz <= 1; dz++)
      for (int dy = -1; dy <= 1; dy++)
        for (int dx = -1; dx <= 1; dx++) {
          const long long j = i + dz * nxny + (long long)dy * s.nx + dx;
          if (j == i || s.tag[j] != TAG_FLUID) continue;
          ps += (double)s.phi[cur][j];
          rs += (double)s.rho[cur][j];
          xs += (double)s.ux_at(cur, j);
          ys += (double)s.uy_at(cur, j);
          zs += (double)s.uz[cur][j];
          cnt++;
        }
    const double p = cnt ? ps / cnt : (double)s.phi[cur][i], r = cnt ? rs / cnt : 1.0;
    const double vx = cnt ? xs / cnt : 0.0, vy = cnt ? ys / cnt : 0.0, vz = cnt ? zs / cnt : 0.0;
    s.phi[0][i] = s.phi[1][i] = (Real)p;
    s.rho[cur][i] = (Real)r;
    s.set_ux(cur, i, (Real)vx);
    s.set_uy(cur, i, (Real)vy);
    s.uz[cur][i] = (Real)vz;
    const double rhoPhase = rhoG + p * (rhoL - rhoG), u2 = vx * vx + vy * vy + vz * vz;
    for (int k = 0; k < Q27; k++) {
      const double eu = dcomp(k, 0) * vx + dcomp(k, 1) * vy + dcomp(k, 2) * vz;
      const double fk = (double)w27_of(k) * (r + rhoPhase * (eu * (3.0 + 4.5 * eu) - 1.5 * u2));
      s.F[cur][pidx<27>(k, i)] = Codec<PopT>::enc((Real)fk, (Real)w27_of(k));
      if (k < Q7)
        s.H[cur][pidx<7>(k, i)] =
            Codec<PopT>::enc((Real)((double)w7_of(k) * p * (1 + 4.0 * eu)), (Real)w7_of(k) * (Real)p);
    }
  }
}

// ---------------------------------------------------------------- SOLID cells
// The step updates FLUID cells only; a SOLID cell keeps its values in both
// halves.  It gets them into the half that the step writes when it turns SOLID
// (k_sets), and the tiles pass it by: copying every SOLID cell in every step
// made the warps inside a sphere wait nine memory latencies a plane (160x112x160
// with one sphere 227 -> 193 us a launch on a B200).
template <class PopT>
__device__ __forceinline__ void carry_cell(const Scene<PopT, typename Prec<PopT>::Real> &s, int cur, long long i) {
  using Real = typename Prec<PopT>::Real;
  struct alignas(4 * sizeof(PopT) > 16 ? 16 : 4 * sizeof(PopT)) Group {
    PopT v[4];
  };
  const int nxt = 1 - cur;
  Group f[PopGroups<Q27>::G], h[PopGroups<Q7>::G];
  const long long F = pidx<27>(0, i), H = pidx<7>(0, i);
  for (int g = 0; g < PopGroups<Q27>::G; g++) f[g] = *reinterpret_cast<const Group *>(s.F[cur] + F + 32 * g);
  for (int g = 0; g < PopGroups<Q7>::G; g++) h[g] = *reinterpret_cast<const Group *>(s.H[cur] + H + 32 * g);
  const Real p = s.phi[cur][i], r = s.rho[cur][i], z = s.uz[cur][i];
  for (int g = 0; g < PopGroups<Q27>::G; g++) *reinterpret_cast<Group *>(s.F[nxt] + F + 32 * g) = f[g];
  for (int g = 0; g < PopGroups<Q7>::G; g++) *reinterpret_cast<Group *>(s.H[nxt] + H + 32 * g) = h[g];
  s.phi[nxt][i] = p;
  s.rho[nxt][i] = r;
  s.uz[nxt][i] = z;
  if constexpr (!Scene<PopT, Real>::UPAD) {  // (in the pads, copied with the groups)
    s.ux[nxt][i] = s.ux[cur][i];
    s.uy[nxt][i] = s.uy[cur][i];
  }
}
// every cell of [c0, c1) that the step does not update (SOLID, written WALL, the
// domain's faces), after calls that may have changed one half alone
template <class PopT>
__global__ void k_carry_solid(Scene<PopT, typename Prec<PopT>::Real> s, int cur, long long c0, long long c1) {
  for (long long i = c0 + blockIdx.x * (long long)blockDim.x + threadIdx.x; i < c1; i += (long long)gridDim.x * blockDim.x)
    if (s.tag[i] != TAG_FLUID || !interior_cell(i, s.nx, s.ny, s.nz)) carry_cell<PopT>(s, cur, i);
}

// ---------------------------------------------------------------- retag, fresh / dead sets, fresh fill
// Arguments of a scene's sparse kernels (by value for one scene; a batch reads
// one block per scene from device memory).
template <class PopT>
struct SmallArgs {
  Scene<PopT, typename Prec<PopT>::Real> s;
  int cur, listCap, zlo, zend, seqFill;
  const Plan *plan;
  int2 *counts;     // per chunk of the box: fresh, dead cells; then their offsets
  uint32_t *bits;   // per chunk: [64] pairs of fresh / dead ballot words
  unsigned *ticket;
  int *fresh, *dead, *totals;
  double rhoL, rhoG;
};

// The first three parts of a step around the spheres in one launch: retagCells
// on the plan's box (RETAG; src/sim.js:214-244: every cell outside the union of
// the current and the two previous sphere boxes keeps tag == tagPrev; a cell
// that turns SOLID is copied into the half that the step writes), the
// scan-ordered lists of fresh (FLUID, was SOLID) and dead (SOLID, was FLUID)
// cells, and handleFreshCells (FILL).
//
// Blocks stride over the box's 2,048-cell chunks and leave one fresh and one
// dead ballot word per 32 cells and the chunk's counts; the block that takes
// the last ticket scans the counts, writes the lists in scan order from the
// ballots, one warp per chunk, and fills the fresh cells.
// Latency-bound: the boxes hold 10^3 to 10^5 cells, so what counts is the
// number of dependent launches.  This one launch takes the place of five
// (retag, count, scan, emit, fill).
constexpr int SETS_THREADS = 256;
constexpr int SETS_WORDS = COMPACT_CHUNK / 32;

template <class PopT, bool RETAG, bool FILL>
__device__ __forceinline__ void sets_body(const SmallArgs<PopT> &a, unsigned bid, unsigned gdim) {
  using Real = typename Prec<PopT>::Real;
  static_assert(SETS_THREADS == 256 && COMPACT_CHUNK == 2048, "eight cells per thread and chunk");
  __shared__ int2 sw[SETS_THREADS / 32];
  __shared__ bool last;
  const Scene<PopT, Real> &s = a.s;
  const SolidSet &ss = a.plan->ss;
  const Box bx = a.plan->U;
  const unsigned total = (unsigned)a.plan->ucells;
  const int nch = a.plan->nchunks;
  const unsigned nb = min(gdim, (unsigned)max(nch, 1));
  if (bid >= nb) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned dx = bx.hi[0] - bx.lo[0] + 1, dy = bx.hi[1] - bx.lo[1] + 1;
  for (int c = bid; c < nch; c += gdim) {
    int cell[8];
    int3 at[8];
    uint8_t t[8], p[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const unsigned l = (unsigned)c * COMPACT_CHUNK + j * SETS_THREADS + threadIdx.x;
      cell[j] = -1;
      if (l < total) {
        const unsigned q = l / dx;
        const int x = bx.lo[0] + (int)(l - q * dx), y = bx.lo[1] + (int)(q % dy), z = bx.lo[2] + (int)(q / dy);
        cell[j] = (z * s.ny + y) * s.nx + x;
        at[j] = make_int3(x, y, z);
        t[j] = s.tag[cell[j]];
        if (!RETAG) p[j] = s.tagPrev[cell[j]];
      }
    }
    int nf = 0, nd = 0;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      bool isF = false, isD = false;
      if (cell[j] >= 0) {
        if (RETAG) {
          const int x = at[j].x, y = at[j].y, z = at[j].z;
          p[j] = t[j];
          if (x == 0 || x == s.nx - 1 || y == 0 || y == s.ny - 1 || z == 0 || z == s.nz - 1) {
            t[j] = TAG_WALL;
          } else {
            t[j] = owner_of<LBM_MAX_SPHERES>(ss.sph, ss.nsph, x, y, z) >= 0 ? TAG_SOLID : TAG_FLUID;
          }
          s.tagPrev[cell[j]] = p[j];
          s.tag[cell[j]] = t[j];
        }
        isF = t[j] == TAG_FLUID && p[j] == TAG_SOLID;
        isD = t[j] == TAG_SOLID && p[j] == TAG_FLUID;
        // (also a cell that a written tag made WALL, which is no dead cell)
        if (RETAG && t[j] == TAG_SOLID && p[j] != TAG_SOLID) carry_cell<PopT>(s, a.cur, cell[j]);
      }
      const unsigned bf = __ballot_sync(0xffffffffu, isF), bd = __ballot_sync(0xffffffffu, isD);
      if (lane == 0)
        reinterpret_cast<uint2 *>(a.bits)[(long long)c * SETS_WORDS + j * (SETS_THREADS / 32) + warp] =
            make_uint2(bf, bd);
      nf += __popc(bf);
      nd += __popc(bd);
    }
    if (lane == 0) sw[warp] = make_int2(nf, nd);
    __syncthreads();
    if (threadIdx.x == 0) {
      int2 v = make_int2(0, 0);
      for (int w = 0; w < SETS_THREADS / 32; w++) v.x += sw[w].x, v.y += sw[w].y;
      a.counts[c] = v;
    }
    __syncthreads();
  }
  if (nb > 1) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(a.ticket, 1u) == nb - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x == 0) *a.ticket = 0;
  }

  // Per 256 chunks: exclusive scan of the counts, a queue of the chunks that
  // hold any, then one warp per such chunk: lane l's two pairs of words (32
  // cells each) in order, the next chunk's words on the way.  (Chunks given to
  // the warps by place kept five of eight warps idle at 65 chunks: 28,000
  // cycles where this takes 9,000.)
  __shared__ int3 queue[SETS_THREADS];
  __shared__ int queued;
  int2 all = make_int2(0, 0);
  for (int t0 = 0; t0 < nch; t0 += SETS_THREADS) {
    const int mine = t0 + threadIdx.x;
    const int2 cnt = mine < nch ? __ldcg(a.counts + mine) : make_int2(0, 0);
    int2 inc = cnt;
    for (int o = 1; o < 32; o <<= 1) {
      const int fx = __shfl_up_sync(0xffffffffu, inc.x, o), fy = __shfl_up_sync(0xffffffffu, inc.y, o);
      if (lane >= o) inc.x += fx, inc.y += fy;
    }
    if (lane == 31) sw[warp] = inc;
    if (threadIdx.x == 0) queued = 0;
    __syncthreads();
    int2 run = make_int2(all.x + inc.x - cnt.x, all.y + inc.y - cnt.y);
    for (int w = 0; w < SETS_THREADS / 32; w++) {
      const int2 v = sw[w];
      if (w < warp) run.x += v.x, run.y += v.y;
      all.x += v.x, all.y += v.y;
    }
    if (cnt.x | cnt.y) queue[atomicAdd(&queued, 1)] = make_int3(mine, run.x, run.y);
    __syncthreads();
    const int n = queued;
    const uint4 *words = reinterpret_cast<const uint4 *>(a.bits) + lane;
    uint4 next = make_uint4(0, 0, 0, 0);
    if (warp < n) next = __ldcg(words + (long long)queue[warp].x * (SETS_WORDS / 2));
#pragma unroll 1
    for (int e = warp; e < n; e += SETS_THREADS / 32) {
      const int3 at = queue[e];
      const uint4 w = next;
      if (e + SETS_THREADS / 32 < n)
        next = __ldcg(words + (long long)queue[e + SETS_THREADS / 32].x * (SETS_WORDS / 2));
      // fresh cells in the low half of a word, dead ones in the high half
      const int m = __popc(w.x) + __popc(w.z) + ((__popc(w.y) + __popc(w.w)) << 16);
      int pre = m;
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, pre, o);
        if (lane >= o) pre += x;
      }
      pre -= m;
      int of = at.y + (pre & 0xffff), od = at.z + (pre >> 16);
      unsigned l0 = (unsigned)at.x * COMPACT_CHUNK + 2 * lane * 32;
#pragma unroll 1
      for (int part = 0; part < 4; part++) {
        const bool dead = part & 1;
        unsigned bits = part == 0 ? w.x : part == 1 ? w.y : part == 2 ? w.z : w.w;
        int *list = dead ? a.dead : a.fresh;
        int pos = dead ? od : of;
        for (; bits; bits &= bits - 1, pos++) {
          const unsigned l = l0 + (part & 2) * 16 + (__ffs(bits) - 1), q = l / dx;
          const int x = bx.lo[0] + (int)(l - q * dx), y = bx.lo[1] + (int)(q % dy), z = bx.lo[2] + (int)(q / dy);
          if (pos < a.listCap) list[pos] = (z * s.ny + y) * s.nx + x;
        }
        if (dead) od = pos;
        else of = pos;
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    a.totals[0] = all.x;
    a.totals[1] = all.y;
  }
  if constexpr (FILL) {
    if (all.x == 0 || a.seqFill) return;
    fresh_fill_body<PopT, SETS_THREADS>(s, a.cur, a.fresh, min(all.x, a.listCap), a.rhoL, a.rhoG, a.zlo, a.zend);
  }
}
template <class PopT, bool RETAG, bool FILL>
__global__ void __launch_bounds__(SETS_THREADS) k_sets(const __grid_constant__ SmallArgs<PopT> a) {
  sets_body<PopT, RETAG, FILL>(a, blockIdx.x, gridDim.x);
}
// every scene of a batch: grid row s is scene s
template <class PopT>
__global__ void __launch_bounds__(SETS_THREADS) kb_sets(const SmallArgs<PopT> *__restrict__ A) {
  sets_body<PopT, true, true>(A[blockIdx.y], blockIdx.x, gridDim.x);
}

// with the test hook on, after k_sets / kb_sets; scene b in block b
template <class PopT>
__device__ __forceinline__ void fill_in_order_body(const SmallArgs<PopT> &a) {
  if (a.seqFill && threadIdx.x == 0)
    fresh_fill_in_order<PopT>(a.s, a.cur, a.fresh, min(a.totals[0], a.listCap), a.rhoL, a.rhoG, a.zlo, a.zend);
}
template <class PopT>
__global__ void k_fill_in_order(const __grid_constant__ SmallArgs<PopT> a) {
  fill_in_order_body<PopT>(a);
}
template <class PopT>
__global__ void kb_fill_in_order(const SmallArgs<PopT> *__restrict__ A) {
  fill_in_order_body<PopT>(A[blockIdx.x]);
}

// ---------------------------------------------------------------- generic solids
// retagCells(solid) for any duck-typed solid (src/sim.js:214-244): the host
// has evaluated solid.contains / solid.surfaceVelocity per cell into mask
// (non-zero = inside) and us (3 floats per cell, x y z; null = at rest).
template <class PopT>
__global__ void k_retag_mask(Scene<PopT, typename Prec<PopT>::Real> s, int cur, const uint8_t *__restrict__ mask,
                             const float *__restrict__ us) {
  using Real = typename Prec<PopT>::Real;
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= s.n) return;
  const int nx = s.nx, ny = s.ny, nz = s.nz;
  int x = (int)(i % nx);
  long long t = i / nx;
  int y = (int)(t % ny);
  int z = (int)(t / ny);
  s.tagPrev[i] = s.tag[i];
  s.phi[1 - cur][i] = s.phi[cur][i];
  if (x == 0 || x == nx - 1 || y == 0 || y == ny - 1 || z == 0 || z == nz - 1) {
    s.tag[i] = TAG_WALL;
    s.usx[i] = s.usy[i] = s.usz[i] = (Real)0;
  } else if (mask[i]) {
    s.tag[i] = TAG_SOLID;
    s.usx[i] = us ? (Real)us[3 * i] : (Real)0;
    s.usy[i] = us ? (Real)us[3 * i + 1] : (Real)0;
    s.usz[i] = us ? (Real)us[3 * i + 2] : (Real)0;
  } else {
    s.tag[i] = TAG_FLUID;
    s.usx[i] = s.usy[i] = s.usz[i] = (Real)0;
  }
}

// Momentum-exchange links of the last hydro stream (after
// k_stream_hydro_macro, while F[1 - cur] still holds the post-collision f2):
// for every interior FLUID cell i in scan order and every direction k whose
// source i - e_k is SOLID, the link (i, k, m) with m = f2_opp(i) + f_k(i), the
// value src/sim.js:529-531 hands to solid.applyImpulseAtCell (as
// -m e_k at the solid cell).  Three passes: count per chunk, scan, emit.
constexpr int LINK_CHUNK = 1024;  // cells per chunk = threads per block

__device__ __forceinline__ uint32_t solid_links(const uint8_t *tag, long long i, int nx, int ny, int nz) {
  if (tag[i] != TAG_FLUID || !interior_cell(i, nx, ny, nz)) return 0u;
  uint32_t m = 0;
  for (int k = 1; k < Q27; k++) {
    const long long src = i - (((long long)dcomp(k, 2) * ny + dcomp(k, 1)) * nx + dcomp(k, 0));
    if (tag[src] == TAG_SOLID) m |= 1u << k;
  }
  return m;
}

__device__ __forceinline__ int block_exclusive_scan(int v, int *sh, int &total) {
  // Hillis-Steele over one block of LINK_CHUNK threads
  const int t = threadIdx.x;
  sh[t] = v;
  __syncthreads();
  for (int d = 1; d < LINK_CHUNK; d <<= 1) {
    const int a = t >= d ? sh[t - d] : 0;
    __syncthreads();
    sh[t] += a;
    __syncthreads();
  }
  total = sh[LINK_CHUNK - 1];
  const int excl = sh[t] - v;
  __syncthreads();
  return excl;
}

static __global__ void __launch_bounds__(LINK_CHUNK) k_link_count(const uint8_t *tag, int nx, int ny, int nz,
                                                                 long long n, int *chunkCount) {
  __shared__ int sh[LINK_CHUNK];
  const long long i = (long long)blockIdx.x * LINK_CHUNK + threadIdx.x;
  const int c = i < n ? __popc(solid_links(tag, i, nx, ny, nz)) : 0;
  int total;
  block_exclusive_scan(c, sh, total);
  if (threadIdx.x == 0) chunkCount[blockIdx.x] = total;
}

// exclusive scan of the chunk counts in place; total into chunkCount[nchunks]
static __global__ void k_link_scan(int *chunkCount, int nchunks) {
  __shared__ int part[1024];
  const int per = (nchunks + blockDim.x - 1) / blockDim.x;
  const int b0 = threadIdx.x * per, b1 = min(b0 + per, nchunks);
  int sum = 0;
  for (int b = b0; b < b1; b++) sum += chunkCount[b];
  part[threadIdx.x] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    int run = 0;
    for (int t = 0; t < (int)blockDim.x; t++) {
      const int v = part[t];
      part[t] = run;
      run += v;
    }
    chunkCount[nchunks] = run;
  }
  __syncthreads();
  int run = part[threadIdx.x];
  for (int b = b0; b < b1; b++) {
    const int v = chunkCount[b];
    chunkCount[b] = run;
    run += v;
  }
}

template <class PopT>
__global__ void __launch_bounds__(LINK_CHUNK) k_link_emit(Scene<PopT, typename Prec<PopT>::Real> s, int cur,
                                                         const int *chunkOff, int cap, int *cells,
                                                         int8_t *dirs, double *mom) {
  __shared__ int sh[LINK_CHUNK];
  const long long i = (long long)blockIdx.x * LINK_CHUNK + threadIdx.x;
  const uint32_t m = i < s.n ? solid_links(s.tag, i, s.nx, s.ny, s.nz) : 0u;
  int total;
  int pos = chunkOff[blockIdx.x] + block_exclusive_scan(__popc(m), sh, total);
  const PopT *f2 = s.F[1 - cur];
  const PopT *f = s.F[cur];
  for (uint32_t r = m; r; r &= r - 1, pos++) {
    const int k = __ffs(r) - 1;
    if (pos >= cap) break;
    const double fopp = (double)Codec<PopT>::dec(f2[pidx<27>(opp_of(k), i)], 0);
    const double fk = (double)Codec<PopT>::dec(f[pidx<27>(k, i)], 0);
    cells[pos] = (int)i;
    dirs[pos] = (int8_t)k;
    mom[pos] = fopp + fk;
  }
}

// absorbDeadCells (src/solid.js:87-101): impulse rho(phi)*u of every cell on
// the scan-ordered dead list, in FP64, to the sphere owning the cell.  One CTA
// per sphere; thread t sums the contiguous t-th share of the list in scan
// order, then a fixed shared-memory tree adds the shares -- deterministic,
// and independent of how many dead cells there are per step.
constexpr int DEAD_THREADS = 256;

// (static: Real = float is instantiated by several translation units)
// the dead-cell sweep reads phi and u through one of these: plain arrays
// (the allocation-free entry's caller arrays) or a scene's current half
template <class Real>
struct ArrayFields {
  const Real *phi, *ux, *uy, *uz;
  __device__ __forceinline__ double p(long long i) const { return (double)phi[i]; }
  __device__ __forceinline__ double vx(long long i) const { return (double)ux[i]; }
  __device__ __forceinline__ double vy(long long i) const { return (double)uy[i]; }
  __device__ __forceinline__ double vz(long long i) const { return (double)uz[i]; }
};
template <class PopT>
struct SceneFields {
  const Scene<PopT, typename Prec<PopT>::Real> &s;
  int cur;
  __device__ __forceinline__ double p(long long i) const { return (double)s.phi[cur][i]; }
  __device__ __forceinline__ double vx(long long i) const { return (double)s.ux_at(cur, i); }
  __device__ __forceinline__ double vy(long long i) const { return (double)s.uy_at(cur, i); }
  __device__ __forceinline__ double vz(long long i) const { return (double)s.uz[cur][i]; }
};

template <class Fields>
__device__ __forceinline__ void absorb_dead_body(const Fields &fd, int nx, int ny, const int *__restrict__ dead,
                                                 const int *__restrict__ totals, int cap, double rhoL,
                                                 double rhoG, const SolidSet *__restrict__ ssp, double *out,
                                                 int b, double (*sh)[DEAD_THREADS]) {
  const SolidSet &ss = *ssp;
  if (b >= ss.nsph) return;
  int nd = totals[1];
  if (nd > cap) nd = cap;
  if (nd == 0) {
    if (threadIdx.x < 6) out[6 * b + threadIdx.x] = 0.0;
    return;
  }
  const double dRho = rhoL - rhoG;
  const int per = (nd + DEAD_THREADS - 1) / DEAD_THREADS;
  const int q0 = threadIdx.x * per, q1 = min(q0 + per, nd);
  double acc[6] = {0, 0, 0, 0, 0, 0};
  for (int q = q0; q < q1; q++) {
    const long long i = dead[q];
    const int x = (int)(i % nx);
    const long long t = i / nx;
    const int y = (int)(t % ny);
    const int z = (int)(t / ny);
    if (ss.zend > 0 && (z < ss.zlo || z >= ss.zend)) continue;
    if (owner_of<LBM_MAX_SPHERES>(ss.sph, ss.nsph, x, y, z) != b) continue;
    const double rhoPhase = __dadd_rn(rhoG, __dmul_rn(fd.p(i), dRho));
    impulse_terms(ss.sph[b], x, y, z, __dmul_rn(rhoPhase, fd.vx(i)), __dmul_rn(rhoPhase, fd.vy(i)),
                  __dmul_rn(rhoPhase, fd.vz(i)), acc);
  }
  for (int j = 0; j < 6; j++) sh[j][threadIdx.x] = acc[j];
  __syncthreads();
  for (int st = DEAD_THREADS / 2; st > 0; st >>= 1) {
    if ((int)threadIdx.x < st)
      for (int j = 0; j < 6; j++) sh[j][threadIdx.x] = __dadd_rn(sh[j][threadIdx.x], sh[j][threadIdx.x + st]);
    __syncthreads();
  }
  if (threadIdx.x < 6) out[6 * b + threadIdx.x] = sh[threadIdx.x][0];
  __syncthreads();
}
template <class Real>
static __global__ void __launch_bounds__(DEAD_THREADS)
    k_absorb_dead(const Real *__restrict__ phi, const Real *__restrict__ ux,
                  const Real *__restrict__ uy, const Real *__restrict__ uz, int nx, int ny,
                  const int *__restrict__ dead, const int *__restrict__ totals, int cap, double rhoL,
                  double rhoG, const SolidSet *__restrict__ ssp, double *out) {
  __shared__ double sh[6][DEAD_THREADS];
  absorb_dead_body(ArrayFields<Real>{phi, ux, uy, uz}, nx, ny, dead, totals, cap, rhoL, rhoG, ssp, out,
                   blockIdx.x, sh);
}
// the same over a scene's current half
template <class PopT>
static __global__ void __launch_bounds__(DEAD_THREADS)
    k_absorb_dead_scene(Scene<PopT, typename Prec<PopT>::Real> s, int cur, const int *__restrict__ dead,
                        const int *__restrict__ totals, int cap, double rhoL, double rhoG,
                        const SolidSet *__restrict__ ssp, double *out) {
  __shared__ double sh[6][DEAD_THREADS];
  absorb_dead_body(SceneFields<PopT>{s, cur}, s.nx, s.ny, dead, totals, cap, rhoL, rhoG, ssp, out, blockIdx.x,
                   sh);
}

// Deterministic reduction of the phase-by-phase path's impulse slots (cleared
// before every hydro stream) in one launch.  Block (c, b) sums chunk c (1024
// cells) of sphere b's slots -- the threads stride the chunk, then a
// shared-memory tree -- and stores its partial; the block that takes the last
// ticket of sphere b adds the partials in chunk order and resets the ticket.
// Which block finishes last does not change the result, nor does how the stream
// kernel was tiled.  Every slot counts: tags written by the caller may put FLUID
// cells, and so links, anywhere in the box.
constexpr int RED_CHUNK = 1024;
constexpr int RED_THREADS = 256;

__device__ __forceinline__ void impulse_reduce_body(const SolidSet *__restrict__ ssp, double *partials,
                                                    int maxChunks, double *out, unsigned *tickets, int cx,
                                                    int b) {
  const SolidSet &ss = *ssp;
  if (b >= ss.nsph) return;
  const ImpulseTarget &t = ss.imp[b];
  const long long cells = (long long)t.dim[0] * t.dim[1] * t.dim[2];
  int nch = (int)((cells + RED_CHUNK - 1) / RED_CHUNK);
  if (nch < 1) nch = 1;  // an empty box still gives its zero
  if (nch > maxChunks) nch = maxChunks;
  if (cx >= nch) return;
  const long long c0 = (long long)cx * RED_CHUNK;
  __shared__ double sh[6][RED_THREADS];
  __shared__ bool last;
  double a[6] = {0, 0, 0, 0, 0, 0};
  for (int j = threadIdx.x; j < RED_CHUNK; j += RED_THREADS) {
    const long long c = c0 + j;
    if (c >= cells) break;
    const double *p = t.acc + 6 * c;
    for (int q = 0; q < 6; q++) a[q] = __dadd_rn(a[q], p[q]);
  }
  for (int q = 0; q < 6; q++) sh[q][threadIdx.x] = a[q];
  __syncthreads();
  for (int st = RED_THREADS / 2; st > 0; st >>= 1) {
    if ((int)threadIdx.x < st)
      for (int q = 0; q < 6; q++) sh[q][threadIdx.x] = __dadd_rn(sh[q][threadIdx.x], sh[q][threadIdx.x + st]);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    for (int q = 0; q < 6; q++) partials[((long long)b * maxChunks + cx) * 6 + q] = sh[q][0];
    __threadfence();
    last = atomicAdd(&tickets[b], 1u) == (unsigned)nch - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (threadIdx.x < 6) {
    double s = 0;
    for (int c = 0; c < nch; c++) s = __dadd_rn(s, __ldcg(&partials[((long long)b * maxChunks + c) * 6 + threadIdx.x]));
    out[6 * b + threadIdx.x] = s;
  }
  if (threadIdx.x == 0) tickets[b] = 0;
}
static __global__ void __launch_bounds__(RED_THREADS)
    k_impulse_reduce(const SolidSet *__restrict__ ssp, double *partials, int maxChunks, double *out,
                     unsigned *tickets) {
  impulse_reduce_body(ssp, partials, maxChunks, out, tickets, blockIdx.x, blockIdx.y);
}

// Device-side plan P of a step of the device-resident loop, from the sphere
// state and the previous step's plan (the same object for the first step):
// sphere descriptors, the retag box (current and two previous sphere boxes),
// compaction chunking, and impulse slots of slotCells cells per sphere.
__device__ __forceinline__ void plan_body(Plan *P, const Plan *prev, const lbm_sphere *sph, int nsph, int nx, int ny,
                                          int nz, double *impBase, long long slotCells, long long maxUCells) {
  SolidSet &ss = P->ss;
  const Box boxLast = prev->boxLast, boxLastLast = prev->boxLastLast;
  const int fullRetag = prev->fullRetag;
  int overflow = prev->overflow;
  Box stale = prev->stale;
  ss.nsph = nsph;
  ss.zlo = ss.zend = 0;
  Box now{{1, 1, 1}, {0, 0, 0}};
  for (int b = 0; b < nsph; b++) {
    SphereDesc &d = ss.sph[b];
    const double cx = sph[b].cx, cy = sph[b].cy, cz = sph[b].cz, r = sph[b].r;
    d.cx = cx;
    d.cy = cy;
    d.cz = cz;
    d.r = r;
    d.vx = sph[b].vx;
    d.vy = sph[b].vy;
    d.vz = sph[b].vz;
    d.wx = sph[b].wx;
    d.wy = sph[b].wy;
    d.wz = sph[b].wz;
    const Box sb = sphere_box(cx, cy, cz, r, nx, ny, nz);
    now = box_union(now, sb);
    Box tb = box_grow(sb, 1, nx, ny, nz);
    ImpulseTarget &t = ss.imp[b];
    t.acc = impBase + (long long)b * slotCells * 6;
    long long cells = box_cells(tb);
    if (cells > slotCells) {
      overflow = 1;
      cells = 0;
      tb = Box{{1, 1, 1}, {0, 0, 0}};
    }
    for (int a = 0; a < 3; a++) {
      t.lo[a] = box_empty(tb) ? 0 : tb.lo[a];
      t.dim[a] = box_empty(tb) ? 0 : tb.hi[a] - tb.lo[a] + 1;
    }
  }
  Box U;
  if (fullRetag > 0) {
    U = Box{{0, 0, 0}, {nx - 1, ny - 1, nz - 1}};
    P->fullRetag = fullRetag - 1;
  } else {
    U = box_union(box_union(now, boxLast), boxLastLast);
    P->fullRetag = 0;
  }
  long long uc = box_cells(U);
  if (uc > maxUCells) {
    overflow = 1;
    stale = box_union(stale, boxLast);
    uc = 0;
    U = Box{{1, 1, 1}, {0, 0, 0}};
  }
  P->overflow = overflow;
  P->stale = stale;
  P->U = U;
  P->ucells = uc;
  P->nchunks = (int)((uc + COMPACT_CHUNK - 1) / COMPACT_CHUNK);
  P->boxLastLast = boxLast;
  P->boxLast = now;
}
static __global__ void k_plan(Plan *P, const lbm_sphere *sph, int nsph, int nx, int ny, int nz, double *impBase,
                              long long slotCells, long long maxUCells) {
  if (blockIdx.x == 0 && threadIdx.x == 0)
    plan_body(P, P, sph, nsph, nx, ny, nz, impBase, slotCells, maxUCells);
}

// packVolume's two bytes of cell i (src/sim.js:586-600): R = clamp01(phi) *
// 255 truncated (a NaN gives 0), G = 255 for a SOLID cell, else 0
template <class Real>
__device__ __forceinline__ void pack_rg8(uint8_t *out, long long i, Real phi, bool solid) {
  double p = (double)phi;
  if (p < 0.0) p = 0.0;
  else if (p > 1.0) p = 1.0;
  const double v = p * 255.0;
  uchar2 o;
  o.x = (uint8_t)((v == v) ? (int)v : 0);
  o.y = solid ? 255 : 0;
  reinterpret_cast<uchar2 *>(out)[i] = o;
}

// packVolume (src/sim.js:586-600)
template <class PopT>
__global__ void k_pack(Scene<PopT, typename Prec<PopT>::Real> s, int cur, uint8_t *out) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= s.n) return;
  pack_rg8(out, i, s.phi[cur][i], s.tag[i] == TAG_SOLID);
}

// packVolume of the planes z = 0 and z = nz - 1 only: the fused step packs
// every other cell on a frame step
template <class PopT>
__global__ void k_pack_end_planes(Scene<PopT, typename Prec<PopT>::Real> s, int cur, uint8_t *out) {
  const long long plane = (long long)s.nx * s.ny;
  long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (j >= 2 * plane) return;
  const long long i = j < plane ? j : (long long)(s.nz - 1) * plane + (j - plane);
  pack_rg8(out, i, s.phi[cur][i], s.tag[i] == TAG_SOLID);
}

// NaN/Inf watchdog: the lowest index of a cell whose phi, rho or u is not
// finite is min-ed into *first, which the caller sets to ~0 beforehand (rho
// alone would not do: rho = sum f > 0.01 ? sum f : 0.01 turns a NaN sum into
// 0.01, src/sim.js:546).  The loop strides by whole blocks, so every warp
// takes the same trips and one lane per warp that sees such a cell does the
// atomic.
template <class PopT>
__global__ void k_watch_finite(Scene<PopT, typename Prec<PopT>::Real> s, int cur, unsigned long long *first) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i0 = blockIdx.x * (long long)blockDim.x; i0 < s.n; i0 += stride) {
    const long long i = i0 + threadIdx.x;
    bool bad = false;
    if (i < s.n)
      bad = !isfinite((double)s.phi[cur][i]) || !isfinite((double)s.rho[cur][i]) ||
            !isfinite((double)s.ux_at(cur, i)) || !isfinite((double)s.uy_at(cur, i)) ||
            !isfinite((double)s.uz[cur][i]);
    const unsigned m = __ballot_sync(0xffffffffu, bad);
    if (m && (int)(threadIdx.x & 31) == __ffs(m) - 1) atomicMin(first, (unsigned long long)i);
  }
}

}  // namespace lbm
