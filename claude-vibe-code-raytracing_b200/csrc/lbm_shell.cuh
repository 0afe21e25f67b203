// The shell launch: everything of a step that hangs on the spheres' surfaces,
// after the fused tiles.  It finishes the cells next to a sphere (Ladd
// moving-wall links, src/sim.js:517-528), sums the momentum exchange
// (src/sim.js:529-536) and the dead-cell impulses (src/solid.js:87-101) in
// FP64 and, in the device-resident loop, runs RigidSphere.step
// (src/solid.js:104-210) and plans the next step.
//
// A link needs the cell's own post-collision values; the launch collides the
// shell's cells once more from the half that the step read, with the tiles'
// collide_cell, so it gets the same bits without the tiles storing anything.
// The cells it finishes are those next to a SOLID cell that a sphere of the plan
// contains; where the tags can hold other SOLID cells a sweep finishes the rest
// (finish_unowned).
// Latency-bound: the shells hold 10^2 to 10^4 cells.  What counts is the
// number of dependent launches and the length of each thread's chain: this one
// launch takes the place of three (impulse reduction, dead-cell impulses,
// sphere step) and of the links in the tiles.  Measured on a B200, a step with
// one sphere before and after (with lbm_kernels.cuh's k_sets in place of five
// launches, the same fused tile shape): 12^3 95 -> 43 us, 61x47x83 208 -> 92,
// 160x112x160 311 -> 243, 256^3 1199 -> 1127 (FP32) and 1202 -> 1044 (FP16).
// The tiles alone, FP16 at 256^3 without a sphere: 1038 -> 987 us.
#pragma once

#include "lbm_fused.cuh"
#include "lbm_sphere.cuh"

namespace lbm {

template <class PopT>
struct ShellArgs {
  FusedArgs<PopT> f;  // the step's fused arguments
  const Plan *plan;   // this step's
  double rhoL;
  int ns, redChunks, listCap;  // chunks per sphere: redChunks blocks each
  int anyTag;                  // the tags may not be the plan's: links anywhere in the spheres' boxes
  unsigned *ticket;
  double *partials, *impulse;  // per chunk; fluid [MAX][6], then dead-cell [MAX][6]
  const int *dead, *totals;
  // the device-resident loop: spheres to step and the next step's plan to make
  // (null in a host-driven step)
  lbm_sphere *sph;
  Plan *next;
  double *impBase;
  long long slotCells, maxU;
};

// RigidSphere.step(1.0, gravity) of sphere b: the momentum-exchange and
// dead-cell impulses of the step are added first, as
// RigidSphere.applyImpulseAtCell would have.
__device__ __forceinline__ void sphere_step_body(lbm_sphere *sph, int b, double gravity, const double *fluid,
                                                 const double *dead, int nx, int ny, int nz) {
  lbm_sphere s = sph[b];
  double *F[6] = {&s.Fx, &s.Fy, &s.Fz, &s.Tx, &s.Ty, &s.Tz};
  for (int j = 0; j < 6; j++) {
    *F[j] = __dadd_rn(*F[j], fluid[6 * b + j]);
    *F[j] = __dadd_rn(*F[j], dead[6 * b + j]);
  }
  sphere_step_fp64(s, 1.0, gravity, nx, ny, nz);
  sph[b] = s;
}

// Direction k as one word: e + 1 in two bits each, then the number of non-zero
// components, then the opposite direction.  (A table of these lies in shared
// memory: constant memory serialises lanes that ask for different directions.)
__device__ __forceinline__ int link_dir(int k) {
  const int ex = dcomp(k, 0), ey = dcomp(k, 1), ez = dcomp(k, 2);
  return (ex + 1) | (ey + 1) << 2 | (ez + 1) << 4 | ((ex != 0) + (ey != 0) + (ez != 0)) << 6 | opp_of(k) << 8;
}

// the phi stencil of cell i (interior) from the half that the step read
template <class PopT>
__device__ __forceinline__ void load_stencil(const Scene<PopT, typename Prec<PopT>::Real> &s, int cur, long long i,
                                             CellLoad<PopT> &L) {
  const long long nx = s.nx, nxny = nx * s.ny;
  const auto *phi = s.phi[cur] + i;
  L.p = phi[0];
  L.pxp = phi[1];
  L.pxm = phi[-1];
  L.pyp = phi[nx];
  L.pym = phi[-nx];
  L.pzp = phi[nxny];
  L.pzm = phi[-nxny];
}

// The tiles leave the raw sums of every FLUID cell with a SOLID source; the
// blocks below finish those with a source that a sphere of the plan contains.
// Where the tags are not the plan's (written since the step's retag, or left by
// a plan that ran out of room) there may be others: their SOLID sources are
// walls at rest, so their populations are right and only the macros remain.
template <class PopT>
__device__ __forceinline__ void finish_unowned(const FusedArgs<PopT> &f, const SolidSet &ss, int x, int y, int z) {
  using Real = typename Prec<PopT>::Real;
  const auto &s = f.s;
  const int cur = f.cur, nxt = 1 - cur;
  const long long i = ((long long)z * s.ny + y) * s.nx + x;
  if (s.tag[i] != TAG_FLUID) return;
  bool raw = false;
#pragma unroll 1
  for (int k = 1; k < Q27; k++) {
    const int sx = x - dcomp(k, 0), sy = y - dcomp(k, 1), sz = z - dcomp(k, 2);
    if (s.tag[((long long)sz * s.ny + sy) * s.nx + sx] != TAG_SOLID) continue;
    raw = true;
    if (owner_of<LBM_MAX_SPHERES>(ss.sph, ss.nsph, sx, sy, sz) >= 0) return;
  }
  if (!raw) return;
  CellLoad<PopT> L;
  load_stencil(s, cur, i, L);
  Real gx, gy, gz, lap, rho, ux, uy, uz;
  phi_stencil(L, gx, gy, gz, lap);
  finish_macros(coll_consts(f), s.phi[nxt][i], gx, gy, gz, lap, s.rho[nxt][i], s.ux_at(nxt, i), s.uy_at(nxt, i),
                s.uz[nxt][i], rho, ux, uy, uz);
  s.rho[nxt][i] = rho;
  s.set_ux(nxt, i, ux);
  s.set_uy(nxt, i, uy);
  s.uz[nxt][i] = uz;
}
// the whole grid, after a step whose tags were written since its retag
template <class PopT>
__global__ void k_finish_unowned(const __grid_constant__ FusedArgs<PopT> f, const Plan *__restrict__ plan) {
  const int nx = f.s.nx, ny = f.s.ny, nz = f.s.nz;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < f.s.n; i += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(i / nx), x = (int)(i - (long long)t * nx), z = t / ny, y = t - z * ny;
    if (x >= 1 && x <= nx - 2 && y >= 1 && y <= ny - 2 && z >= 1 && z <= nz - 2) finish_unowned(f, plan->ss, x, y, z);
  }
}

constexpr int SHELL_THREADS = 256;
static_assert(SHELL_THREADS == RED_THREADS && SHELL_THREADS == DEAD_THREADS && SHELL_THREADS >= Q27, "");

// A plan without room for the retag (the run is reported as failed): the fields
// stay those of a step next to walls at rest where the old SOLID cells are.
// (Not inlined: in the shell's body it cost 0.5 us of 41 a step at 40x28x40.)
template <class PopT>
__device__ __noinline__ void finish_stale(const ShellArgs<PopT> &a) {
  const auto &s = a.f.s;
  const Box w = box_grow(a.plan->stale, 1, s.nx, s.ny, s.nz);
  const int dx = w.hi[0] - w.lo[0] + 1, dy = w.hi[1] - w.lo[1] + 1, n = (int)box_cells(w);
  for (int c = threadIdx.x; c < n; c += SHELL_THREADS) {
    const int q = c / dx, x = w.lo[0] + c - q * dx, y = w.lo[1] + q % dy, z = w.lo[2] + q / dy;
    if (x >= 1 && x <= s.nx - 2 && y >= 1 && y <= s.ny - 2 && z >= 1 && z <= s.nz - 2)
      finish_unowned(a.f, a.plan->ss, x, y, z);
  }
}

// Block (chunk cx of sphere b): 1,024 cells of the sphere's box in scan order.
//   1. the cells with links to a SOLID cell are listed: where the tags are the
//      plan's, only cells within sqrt(3) outside the sphere can have any;
//   2. each listed cell is collided, one thread per cell; its momentum exchange
//      with this sphere is summed in direction order into its slot, and the
//      block of the first sphere that it has a link to adds the links'
//      moving-wall terms to the sums the tile left in its macros, rewrites the
//      linked populations and finishes the macros;
//   3. the slots are summed in a fixed order: share t takes cells t, t + 256,
//      ..., then a tree, then the chunks in order by the block that finishes
//      last.  That block also sums the dead-cell impulses, steps the spheres
//      and plans the next step.
template <class PopT>
__device__ __forceinline__ void shell_body(const ShellArgs<PopT> &a, int cx, int b) {
  using Real = typename Prec<PopT>::Real;
  using C = Codec<PopT>;
  constexpr int BLK27 = PopGroups<Q27>::BLOCK, BLK7 = PopGroups<Q7>::BLOCK;
  __shared__ double sh[6][SHELL_THREADS];
  // threads that collide a cell (FP64: as many as the static shared memory holds)
  constexpr int CELLS = sizeof(Real) == 4 ? SHELL_THREADS : 96;
  __shared__ Real fo[Q27][CELLS];        // post-collision populations of each thread's cell
  __shared__ uint32_t sMask[RED_CHUNK];  // SOLID sources of each listed cell
  __shared__ uint16_t sList[RED_CHUNK];  // the chunk's cells with links, in any order
  __shared__ uint8_t sHas[RED_CHUNK];    // whether a cell has links
  __shared__ int sDir[Q27], sCount, sLast;
  const SolidSet &ss = a.plan->ss;
  const auto &s = a.f.s;
  const int tid = threadIdx.x;
  const int nx = s.nx, ny = s.ny, nz = s.nz, nxny = nx * ny, cur = a.f.cur, nxt = 1 - cur;
  const int ns = ss.nsph, over = a.plan->overflow;
  auto chunks_of = [&](int j) {
    const ImpulseTarget &t = ss.imp[j];
    const long long cells = (long long)t.dim[0] * t.dim[1] * t.dim[2];
    return min(max((int)((cells + RED_CHUNK - 1) / RED_CHUNK), 1), a.redChunks);  // an empty box gives its zero
  };
  if (ns > 0) {
    if (b >= ns || cx >= chunks_of(b)) return;
    const ImpulseTarget &t = ss.imp[b];
    const SphereDesc sp = ss.sph[b];
    const int cells = (int)((long long)t.dim[0] * t.dim[1] * t.dim[2]), c0 = cx * RED_CHUNK;
    const int dxb = t.dim[0], dyb = t.dim[1], lo0 = t.lo[0], lo1 = t.lo[1], lo2 = t.lo[2];
    const double rad = fabs(sp.r), rIn = rad > 1.0 ? rad - 1.0 : 0.0, rOut = rad + 2.0;
    const bool anyTag = a.anyTag || over;
    const double in2 = anyTag ? 0 : rIn * rIn, out2 = anyTag ? INFINITY : rOut * rOut;
    if (tid == 0) sCount = 0;
    if (tid < Q27) sDir[tid] = link_dir(tid);
    __syncthreads();
    for (int j = tid; j < RED_CHUNK; j += SHELL_THREADS) {
      const int c = c0 + j;
      uint32_t m = 0;
      if (c < cells) {
        const int q = c / dxb, x = lo0 + c - q * dxb, z = lo2 + q / dyb, y = lo1 + q % dyb;
        const double ex = x + 0.5 - sp.cx, ey = y + 0.5 - sp.cy, ez = z + 0.5 - sp.cz;
        const double d2 = ex * ex + ey * ey + ez * ez;
        if (!(d2 < in2 || d2 > out2) && x >= 1 && x <= nx - 2 && y >= 1 && y <= ny - 2 && z >= 1 && z <= nz - 2) {
          const uint8_t *tg = s.tag + ((long long)z * ny + y) * nx + x;
          uint8_t v[Q27];
          static_for<0, Q27>([&](auto KK) {
            using D = D27<decltype(KK)::value>;
            v[decltype(KK)::value] = __ldg(tg - (D::ez * nxny + D::ey * nx + D::ex));
          });
          if (v[0] == TAG_FLUID)
            static_for<1, Q27>([&](auto KK) {
              if (v[decltype(KK)::value] == TAG_SOLID) m |= 1u << decltype(KK)::value;
            });
        }
      }
      sHas[j] = m != 0;
      if (m) {
        const int pos = atomicAdd(&sCount, 1);
        sList[pos] = (uint16_t)j;
        sMask[pos] = m;
      }
    }
    __syncthreads();
    const CollK<Real> K = coll_consts(a.f);
    for (int e = tid; e < sCount && tid < CELLS; e += CELLS) {
      const int c = c0 + sList[e];
      const uint32_t m = sMask[e];
      const int q = c / dxb, x = lo0 + c - q * dxb, z = lo2 + q / dyb, y = lo1 + q % dyb;
      const long long i = ((long long)z * ny + y) * nx + x;
      CellLoad<PopT> L;
      const PopT *f = s.F[cur] + (i >> 3) * BLK27 + (i & 7) * 4, *h = s.H[cur] + (i >> 3) * BLK7 + (i & 7) * 4;
      static_for<0, PopGroups<Q27>::G>([&](auto GG) {
        constexpr int g = decltype(GG)::value;
        PopT v[4];
        ld4_global(f + 32 * g, v);
        static_for<4 * g, (4 * g + 4 < Q27 ? 4 * g + 4 : Q27)>([&](auto KK) {
          L.fv[decltype(KK)::value] = v[decltype(KK)::value & 3];
        });
        if constexpr (g < PopGroups<Q7>::G) {
          ld4_global(h + 32 * g, v);
          static_for<4 * g, (4 * g + 4 < Q7 ? 4 * g + 4 : Q7)>([&](auto KK) {
            L.hv[decltype(KK)::value] = v[decltype(KK)::value & 3];
          });
        }
      });
      load_stencil(s, cur, i, L);
      L.sumF = s.rho[cur][i];
      L.ux = s.ux_at(cur, i);
      L.uy = s.uy_at(cur, i);
      L.uz = s.uz[cur][i];
      L.tg = TAG_FLUID;
      // what the tile left: phi, and the populations' sums in the macros
      const Real p = s.phi[nxt][i];
      Real rhoA = s.rho[nxt][i], mx = s.ux_at(nxt, i), my = s.uy_at(nxt, i), mz = s.uz[nxt][i];
      CellOut<PopT> o;
      Real gx, gy, gz, lap;
      collide_cell<PopT, 0, 0, 0>(K, L, o, gx, gy, gz, lap);
      static_for<1, Q27>([&](auto KK) { fo[decltype(KK)::value][tid] = o.f[decltype(KK)::value]; });
      const Real rhoPhOld = rfma(L.p, K.dRho, K.rhoG);
      const bool counts = ss.zend <= 0 || (z >= ss.zlo && z < ss.zend);
      double acc[6] = {0, 0, 0, 0, 0, 0}, tot[6] = {0, 0, 0, 0, 0, 0};
      int owner = -1, first = LBM_MAX_SPHERES;
      // the sums restart where the owner of the links changes
      auto flush = [&]() {
        for (int j = 0; j < 6; j++) {
          if (owner == b) tot[j] = __dadd_rn(tot[j], acc[j]);
          acc[j] = 0.0;
        }
      };
#pragma unroll 1
      for (uint32_t r = m; r; r &= r - 1) {
        const int k = __ffs(r) - 1, v = sDir[k];
        const int ex = (v & 3) - 1, ey = (v >> 2 & 3) - 1, ez = (v >> 4 & 3) - 1, nz_ = v >> 6 & 3;
        const Real w = nz_ == 1 ? (Real)D27<1>::w : nz_ == 2 ? (Real)D27<7>::w : (Real)D27<19>::w;
        const int sx = x - ex, sy = y - ey, sz = z - ez;
        const int own = owner_of<LBM_MAX_SPHERES>(ss.sph, ns, sx, sy, sz);
        if (own < 0) continue;
        first = min(first, own);
        if (own != owner) {
          flush();
          owner = own;
        }
        double ox, oy, oz;
        sphere_surface_velocity(own == b ? sp : ss.sph[own], sx, sy, sz, ox, oy, oz);
        // surface velocity rounded as the reference stores it (Float32Array us)
        const Real eus = radd(radd(rmul((Real)ex, (Real)ox), rmul((Real)ey, (Real)oy)), rmul((Real)ez, (Real)oz));
        const Real corr = rmul(rmul(rmul(rmul((Real)2, w), rhoPhOld), eus), (Real)3);
        const Real fopp = fo[v >> 8][tid], fk = radd(fopp, corr);
        fo[v >> 8][tid] = fk;  // (each opposite value is used once)
        rhoA = radd(rhoA, corr);
        mx = radd(mx, rmul((Real)ex, corr));
        my = radd(my, rmul((Real)ey, corr));
        mz = radd(mz, rmul((Real)ez, corr));
        const double mom = __dadd_rn((double)fopp, (double)fk);
        if (own == b) impulse_terms(sp, sx, sy, sz, -mom * ex, -mom * ey, -mom * ez, acc);
      }
      flush();
      double *slot = t.acc + 6 * (long long)c;
      for (int j = 0; j < 6; j++) slot[j] = counts ? tot[j] : 0.0;
      if (first == b) {
#pragma unroll 1
        for (uint32_t r = m; r; r &= r - 1) {
          const int k = __ffs(r) - 1, v = sDir[k], nz_ = v >> 6 & 3;
          const Real w = nz_ == 1 ? (Real)D27<1>::w : nz_ == 2 ? (Real)D27<7>::w : (Real)D27<19>::w;
          s.F[nxt][pidx<27>(k, i)] = C::enc(fo[v >> 8][tid], w);
        }
        Real rhoN, ux, uy, uz;
        finish_macros(K, p, gx, gy, gz, lap, rhoA, mx, my, mz, rhoN, ux, uy, uz);
        s.rho[nxt][i] = rhoN;
        s.set_ux(nxt, i, ux);
        s.set_uy(nxt, i, uy);
        s.uz[nxt][i] = uz;
      }
    }
    __syncthreads();
    double v[6] = {0, 0, 0, 0, 0, 0};
    for (int c = tid; c < RED_CHUNK; c += SHELL_THREADS)
      if (sHas[c])
        for (int j = 0; j < 6; j++) v[j] = __dadd_rn(v[j], t.acc[6 * (long long)(c0 + c) + j]);
    for (int j = 0; j < 6; j++) sh[j][tid] = v[j];
    __syncthreads();
    for (int st = SHELL_THREADS / 2; st > 0; st >>= 1) {
      if (tid < st)
        for (int j = 0; j < 6; j++) sh[j][tid] = __dadd_rn(sh[j][tid], sh[j][tid + st]);
      __syncthreads();
    }
    int blocks = 0;
    for (int j = 0; j < ns; j++) blocks += chunks_of(j);
    if (blocks > 1) {
      if (tid < 6) {
        a.partials[((long long)b * a.redChunks + cx) * 6 + tid] = sh[tid][0];
        __threadfence();
      }
      __syncthreads();
      if (tid == 0) sLast = atomicAdd(a.ticket, 1u) == (unsigned)blocks - 1;
      __syncthreads();
      if (!sLast) return;
      __threadfence();
      if (tid == 0) *a.ticket = 0;
      double *stage = &sh[0][0];
      for (int sb = 0; sb < ns; sb++) {
        const int n = 6 * chunks_of(sb);
        const double *part = a.partials + (long long)sb * a.redChunks * 6;
        double sum = 0;
        for (int p0 = 0; p0 < n; p0 += 6 * SHELL_THREADS) {
          const int take = min(n - p0, 6 * SHELL_THREADS);
          for (int j = tid; j < take; j += SHELL_THREADS) stage[j] = __ldcg(part + p0 + j);
          __syncthreads();
          if (tid < 6)
            for (int j = tid; j < take; j += 6) sum = __dadd_rn(sum, stage[j]);
          __syncthreads();
        }
        if (tid < 6) a.impulse[6 * sb + tid] = sum;
      }
    } else if (tid < 6) {
      a.impulse[tid] = __dadd_rn(0.0, sh[tid][0]);
    }
    __syncthreads();
    // dead cells are SOLID and keep their values through the step: the half
    // that the step read holds what the new one holds
    for (int sb = 0; sb < ns; sb++)
      absorb_dead_body(SceneFields<PopT>{s, cur}, nx, ny, a.dead, a.totals, a.listCap, a.rhoL, a.f.rhoG, &ss,
                       a.impulse + LBM_MAX_SPHERES * 6, sb, sh);
    if (over) finish_stale(a);
    __syncthreads();
    if (a.sph && tid < ns)
      sphere_step_body(a.sph, tid, a.f.gravity, a.impulse, a.impulse + LBM_MAX_SPHERES * 6, nx, ny, nz);
    __syncthreads();
  } else if (cx != 0 || b != 0) {
    return;
  }
  if (a.next && tid == 0) plan_body(a.next, a.plan, a.sph, ns, nx, ny, nz, a.impBase, a.slotCells, a.maxU);
}
template <class PopT>
__global__ void __launch_bounds__(SHELL_THREADS) k_shell(const __grid_constant__ ShellArgs<PopT> a) {
  shell_body(a, blockIdx.x, blockIdx.y);
}
// every scene of a batch: grid plane s is scene s
template <class PopT>
__global__ void __launch_bounds__(SHELL_THREADS) kb_shell(const ShellArgs<PopT> *__restrict__ A) {
  shell_body(A[blockIdx.z], blockIdx.x, blockIdx.y);
}
// first plan of a batch's device-resident steps, scene s in block s
template <class PopT>
__global__ void kb_plan(const ShellArgs<PopT> *__restrict__ A) {
  const ShellArgs<PopT> &a = A[blockIdx.x];
  if (threadIdx.x == 0)
    plan_body(const_cast<Plan *>(a.plan), a.plan, a.sph, a.ns, a.f.s.nx, a.f.s.ny, a.f.s.nz, a.impBase, a.slotCells,
              a.maxU);
}

}  // namespace lbm
