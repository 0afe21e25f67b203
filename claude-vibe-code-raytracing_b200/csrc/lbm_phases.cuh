// Phase-by-phase kernels (FP32 and FP64 storage), for programs that call the
// reference's Sim methods one by one.  Reference semantics: f = F[cur],
// f2 = F[1-cur]; h = H[cur], h2 = H[1-cur]; macros in place in [cur];
// phiPrev = phi[1-cur].
//
// One thread per cell.  What bounds them is memory: each phase reads and writes
// its arrays once, and no phase may leave work to the next.  A cell's
// populations move as the layout's groups of four (one 16-byte access instead
// of four that touch the same sectors), the directions are unrolled with their
// components known to the compiler, so that all loads of a cell are in flight
// together, and the cell's coordinates come from 32-bit divisions.  With a
// rolled loop of scalar accesses and 64-bit divisions ten steps at 112x96x120
// (FP32, one sphere, the fields read at the end) took 6.19 ms on a B200, now
// 4.43 to 4.66.  Each phase alone at 256^3 (beyond L2; bytes an interior cell
// cannot do without): collidePhase 266 us (89 bytes), streamPhase 218 (65),
// collideHydro 658 (257: 6.4 TB/s, the copy rate is 6.55), streamHydroAndMacro
// with its impulse read-back 1,026 (297: 4.7 TB/s).
#pragma once

#include "lbm_fused.cuh"

namespace lbm {

constexpr int PHASE_THREADS = 256;

struct PhaseCell {
  long long i;
  int x, y, z;
};
// this thread's cell (n < 2^31 cells: lbm_create)
__device__ __forceinline__ PhaseCell phase_cell(int nx, int ny) {
  const unsigned i = blockIdx.x * (unsigned)PHASE_THREADS + threadIdx.x;
  const unsigned t = i / (unsigned)nx, z = t / (unsigned)ny;
  return PhaseCell{(long long)i, (int)(i - t * (unsigned)nx), (int)(t - z * (unsigned)ny), (int)z};
}
// The reference's phase loops run over 1..n-2 on every axis (src/sim.js:334-338);
// cells on the boundary are never collided or streamed, whatever their tag.
__device__ __forceinline__ bool phase_interior(const PhaseCell &c, int nx, int ny, int nz) {
  return c.x >= 1 && c.x <= nx - 2 && c.y >= 1 && c.y <= ny - 2 && c.z >= 1 && c.z <= nz - 2;
}
// cell i's part of a Q-direction half
template <int Q>
__device__ __forceinline__ long long pop_base(long long i) {
  return (long long)((unsigned)i >> 3) * PopGroups<Q>::BLOCK + (i & 7) * 4;
}
// every group of a cell, the pad included
template <int Q, class PopT>
__device__ __forceinline__ void load_groups(const PopT *p, PopT (&v)[PopGroups<Q>::G * 4]) {
  static_for<0, PopGroups<Q>::G>([&](auto GG) {
    constexpr int g = decltype(GG)::value;
    PopT t[4];
    ld4_global(p + 32 * g, t);
    v[4 * g] = t[0], v[4 * g + 1] = t[1], v[4 * g + 2] = t[2], v[4 * g + 3] = t[3];
  });
}
template <int Q, class PopT>
__device__ __forceinline__ void store_groups(PopT *p, const PopT (&v)[PopGroups<Q>::G * 4]) {
  static_for<0, PopGroups<Q>::G>([&](auto GG) {
    constexpr int g = decltype(GG)::value;
    const PopT t[4] = {v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]};
    st4_global(p + 32 * g, t);
  });
}

// e.X with every term, as the reference has it: 0 * X is NaN where X is not
// finite, so a blow-up in one component reaches every direction (edot skips
// those terms)
template <int ex, int ey, int ez, class Real>
__device__ __forceinline__ Real edot_all(Real X, Real Y, Real Z) {
  return rfma((Real)ez, Z, rfma((Real)ey, Y, rmul((Real)ex, X)));
}

// computePhiGradients (src/sim.js:176-199)
template <class PopT>
__global__ void __launch_bounds__(PHASE_THREADS) k_gradients(Scene<PopT, typename Prec<PopT>::Real> s, int cur) {
  using Real = typename Prec<PopT>::Real;
  const int nx = s.nx, ny = s.ny, nz = s.nz;
  const PhaseCell t = phase_cell(nx, ny);
  const long long i = t.i, sz = (long long)nx * ny;
  if (i >= s.n) return;
  const Real *phi = s.phi[cur] + i;
  const Real c = phi[0];
  const Real px = phi[t.x < nx - 1 ? 1 : 0], mx = phi[t.x > 0 ? -1 : 0];
  const Real py = phi[t.y < ny - 1 ? nx : 0], my = phi[t.y > 0 ? -nx : 0];
  const Real pz = phi[t.z < nz - 1 ? sz : 0], mz = phi[t.z > 0 ? -sz : 0];
  s.gx[i] = (Real)0.5 * (px - mx);
  s.gy[i] = (Real)0.5 * (py - my);
  s.gz[i] = (Real)0.5 * (pz - mz);
  s.lap[i] = px + mx + py + my + pz + mz - (Real)6 * c;
}

// collidePhase (src/sim.js:324-364)
template <class PopT>
__global__ void __launch_bounds__(PHASE_THREADS)
    k_collide_phase(Scene<PopT, typename Prec<PopT>::Real> s, int cur, StepConst k) {
  using Real = typename Prec<PopT>::Real;
  const PhaseCell t = phase_cell(s.nx, s.ny);
  const long long i = t.i;
  if (i >= s.n || !phase_interior(t, s.nx, s.ny, s.nz)) return;
  const long long b = pop_base<Q7>(i);
  const uint8_t tag = s.tag[i];
  PopT h[8];  // (h[7]: uy)
  load_groups<Q7>(s.H[cur] + b, h);
  const Real p = s.phi[cur][i];
  const Real uxi = s.ux_at(cur, i), uyi = (Real)h[7], uzi = s.uz[cur][i];
  const Real ggx = s.gx[i], ggy = s.gy[i], ggz = s.gz[i];
  if (tag != TAG_FLUID) return;
  const Real invTau = (Real)k.invTauPhi, sharpC = (Real)k.sharpC, sharpFac = (Real)4.0;
  // (rounded as written, whatever the compiler would contract)
  const Real gmag = sqrt(rfma(ggz, ggz, rfma(ggx, ggx, rmul(ggy, ggy)))) + (Real)1e-12;
  const Real sharpen = sharpC * p * ((Real)1 - p);
  const Real Sx = sharpen * sharpFac * ggx / gmag;
  const Real Sy = sharpen * sharpFac * ggy / gmag;
  const Real Sz = sharpen * sharpFac * ggz / gmag;
  static_for<0, Q7>([&](auto KK) {
    constexpr int q = decltype(KK)::value;
    using D = D7<q>;
    const Real wk = (Real)D::w;
    const Real eu = edot_all<D::ex, D::ey, D::ez>(uxi, uyi, uzi);
    const Real heq = wk * p * ((Real)1 + (Real)4 * eu);
    const Real Fk = wk * edot_all<D::ex, D::ey, D::ez>(Sx, Sy, Sz);
    const Real hk = (Real)h[q];
    h[q] = (PopT)(hk - invTau * (hk - heq) + Fk);
  });
  // (the pad takes the cell's uy: whole sectors are written; a FLUID cell's pad
  // of the other half is read by nothing before it is written again)
  store_groups<Q7>(s.H[1 - cur] + b, h);
}

// streamPhase (src/sim.js:376-397): pull with plain bounce-back.
template <class PopT>
__global__ void __launch_bounds__(PHASE_THREADS)
    k_stream_phase(Scene<PopT, typename Prec<PopT>::Real> s, int cur) {
  const PhaseCell t = phase_cell(s.nx, s.ny);
  const long long i = t.i;
  if (i >= s.n || !phase_interior(t, s.nx, s.ny, s.nz)) return;
  const int nx = s.nx, nxny = s.nx * s.ny;
  const long long b = pop_base<Q7>(i);
  const PopT *h2 = s.H[1 - cur];
  const uint8_t *tag = s.tag + i;
  uint8_t tg[Q7];
  static_for<0, Q7>([&](auto KK) {
    using D = D7<decltype(KK)::value>;
    tg[decltype(KK)::value] = __ldg(tag - (D::ez * nxny + D::ey * nx + D::ex));
  });
  if (tg[0] != TAG_FLUID) return;
  PopT v[8];
  v[7] = s.H[cur][b + pofs(7)];  // uy stays
  static_for<0, Q7>([&](auto KK) {
    constexpr int q = decltype(KK)::value;
    using D = D7<q>;
    const long long src = i - (D::ez * nxny + D::ey * nx + D::ex);
    v[q] = __ldg(h2 + (tg[q] == TAG_FLUID ? pop_base<Q7>(src) + pofs(q) : b + pofs(D::opp)));
  });
  store_groups<Q7>(s.H[cur] + b, v);
}

// collideHydro (src/sim.js:406-464)
template <class PopT>
__global__ void __launch_bounds__(PHASE_THREADS)
    k_collide_hydro(Scene<PopT, typename Prec<PopT>::Real> s, int cur, StepConst k) {
  using Real = typename Prec<PopT>::Real;
  const PhaseCell t = phase_cell(s.nx, s.ny);
  const long long i = t.i;
  if (i >= s.n || !phase_interior(t, s.nx, s.ny, s.nz)) return;
  const long long b = pop_base<Q27>(i);
  const uint8_t tag = s.tag[i];
  PopT f[28];  // (f[27]: ux)
  load_groups<Q27>(s.F[cur] + b, f);
  const Real sumF = s.rho[cur][i], p = s.phi[cur][i], lap = s.lap[i];
  const Real ggx = s.gx[i], ggy = s.gy[i], ggz = s.gz[i];
  const Real uxe = (Real)f[27], uye = s.uy_at(cur, i), uze = s.uz[cur][i];
  if (tag != TAG_FLUID) return;
  const Real invTau = (Real)k.invTau;
  const Real beta = (Real)k.beta, kappa = (Real)k.kappa, dRho = (Real)k.dRho;
  const Real A = (Real)k.A, rhoG = (Real)k.rhoG, gravity = (Real)k.gravity;
  const Real rhoPhase = rhoG + p * dRho;
  const Real mu = (Real)4 * beta * p * (p - (Real)1) * ((Real)2 * p - (Real)1) - kappa * lap;
  const Real bx = s.bfx ? s.bfx[i] : (Real)0, by = s.bfy ? s.bfy[i] : (Real)0, bz = s.bfz ? s.bfz[i] : (Real)0;
  const Real fx = bx + mu * ggx;
  const Real fy = by + mu * ggy + rhoPhase * gravity;
  const Real fz = bz + mu * ggz;
  const Real u2 = uxe * uxe + uye * uye + uze * uze;
  const Real negU2half = (Real)-1.5 * u2;
  const Real uF = uxe * fx + uye * fy + uze * fz;
  static_for<0, Q27>([&](auto KK) {
    constexpr int q = decltype(KK)::value;
    using D = D27<q>;
    const Real wk = (Real)D::w;
    const Real eu = edot_all<D::ex, D::ey, D::ez>(uxe, uye, uze);
    const Real Qi = negU2half + eu * ((Real)3 + (Real)4.5 * eu);
    const Real feq = wk * (sumF + rhoPhase * Qi);
    const Real ekF = edot_all<D::ex, D::ey, D::ez>(fx, fy, fz);
    const Real Sk = A * wk * (ekF * ((Real)1 + (Real)3 * eu) - uF);
    const Real fk = (Real)f[q];
    f[q] = (PopT)(fk - invTau * (fk - feq) + Sk);
  });
  store_groups<Q27>(s.F[1 - cur] + b, f);  // (ux in the pad, as in k_collide_phase)
}

// streamHydroAndMacro (src/sim.js:484-582).  A cell next to a SOLID cell takes
// a rolled loop over the directions (moving-wall term, momentum exchange).
template <class PopT>
__global__ void __launch_bounds__(PHASE_THREADS)
    k_stream_hydro_macro(Scene<PopT, typename Prec<PopT>::Real> s, int cur, StepConst kc,
                         const SolidSet *__restrict__ ssp) {
  using Real = typename Prec<PopT>::Real;
  const PhaseCell t = phase_cell(s.nx, s.ny);
  const long long i = t.i;
  if (i >= s.n || !phase_interior(t, s.nx, s.ny, s.nz)) return;
  const int x = t.x, y = t.y, z = t.z, nx = s.nx, nxny = s.nx * s.ny;
  const long long b = pop_base<Q27>(i), bH = pop_base<Q7>(i);
  const PopT *f2 = s.F[1 - cur];
  PopT *f = s.F[cur] + b;
  const uint8_t *tag = s.tag + i;
  uint8_t tg[Q27];
  static_for<0, Q27>([&](auto KK) {
    using D = D27<decltype(KK)::value>;
    tg[decltype(KK)::value] = __ldg(tag - (D::ez * nxny + D::ey * nx + D::ex));
  });
  if (tg[0] != TAG_FLUID) return;
  PopT h[8];
  load_groups<Q7>(s.H[cur] + bH, h);
  const Real phiOld = s.phi[cur][i], lap = s.lap[i];
  const Real ggx = s.gx[i], ggy = s.gy[i], ggz = s.gz[i];
  uint8_t any = 0;
  static_for<1, Q27>([&](auto KK) { any |= tg[decltype(KK)::value]; });
  const Real beta = (Real)kc.beta, kappa = (Real)kc.kappa, dRho = (Real)kc.dRho;
  const Real rhoG = (Real)kc.rhoG, gravity = (Real)kc.gravity;
  Real pSumF = 0, mx = 0, my = 0, mz = 0;
  PopT last[4];  // f's last group: it waits for ux, its pad
  static_assert(TAG_FLUID == 0 && (TAG_SOLID & TAG_WALL) == 0, "tag bits");
  if (!(any & TAG_SOLID)) {
    PopT v[Q27];
    static_for<0, Q27>([&](auto KK) {
      constexpr int q = decltype(KK)::value;
      using D = D27<q>;
      const long long src = i - (D::ez * nxny + D::ey * nx + D::ex);
      v[q] = __ldg(f2 + (tg[q] == TAG_FLUID ? pop_base<Q27>(src) + pofs(q) : b + pofs(D::opp)));
    });
    static_for<0, Q27>([&](auto KK) {
      constexpr int q = decltype(KK)::value;
      using D = D27<q>;
      const Real fk = (Real)v[q];
      last[q & 3] = v[q];
      if constexpr ((q & 3) == 3) st4_global(f + 32 * (q >> 2), last);
      pSumF += fk;
      mx = rfma((Real)D::ex, fk, mx);
      my = rfma((Real)D::ey, fk, my);
      mz = rfma((Real)D::ez, fk, mz);
    });
  } else {
    const SolidSet &ss = *ssp;
    const Real rhoPhaseOld = rhoG + phiOld * dRho;
    double acc[6] = {0, 0, 0, 0, 0, 0};
    int owner = -1;
#pragma unroll 1
    for (int q = 0; q < Q27; q++) {
      const int ex = dcomp(q, 0), ey = dcomp(q, 1), ez = dcomp(q, 2);
      const long long src = i - (ez * nxny + ey * nx + ex);
      const uint8_t sTag = s.tag[src];
      Real fk;
      if (sTag == TAG_FLUID) {
        fk = (Real)f2[pop_base<Q27>(src) + pofs(q)];
      } else {
        const Real fopp = (Real)f2[b + pofs(opp_of(q))];
        Real corr = 0;
        if (sTag == TAG_SOLID) {
          const Real eu = (Real)ex * s.usx[src] + (Real)ey * s.usy[src] + (Real)ez * s.usz[src];
          corr = (Real)2 * (Real)w27_of(q) * rhoPhaseOld * eu * (Real)3;
        }
        fk = fopp + corr;
        if (sTag == TAG_SOLID && ss.nsph > 0) {
          const int sx = x - ex, sy = y - ey, sz = z - ez;
          const int o = owner_of<LBM_MAX_SPHERES>(ss.sph, ss.nsph, sx, sy, sz);
          if (o >= 0) {
            if (o != owner) {
              flush_impulse(ss, owner, x, y, z, acc);
              owner = o;
            }
            const double m = __dadd_rn((double)fopp, (double)fk);
            impulse_terms(ss.sph[o], sx, sy, sz, -m * ex, -m * ey, -m * ez, acc);
          }
        }
      }
      if (q < 24) f[pofs(q)] = (PopT)fk;
      else if (q == 24) last[0] = (PopT)fk;
      else if (q == 25) last[1] = (PopT)fk;
      else last[2] = (PopT)fk;
      pSumF += fk;
      mx += (Real)ex * fk;
      my += (Real)ey * fk;
      mz += (Real)ez * fk;
    }
    flush_impulse(ss, owner, x, y, z, acc);
  }
  s.rho[cur][i] = pSumF > (Real)0.01 ? pSumF : (Real)0.01;
  Real phiSum = 0;
  static_for<0, Q7>([&](auto KK) { phiSum += (Real)h[decltype(KK)::value]; });
  const Real p = phiSum < (Real)0 ? (Real)0 : phiSum > (Real)1 ? (Real)1 : phiSum;
  s.phi[cur][i] = p;
  const Real rhoPhaseNew = rhoG + p * dRho;
  const Real mu = (Real)4 * beta * p * (p - (Real)1) * ((Real)2 * p - (Real)1) - kappa * lap;
  const Real bx = s.bfx ? s.bfx[i] : (Real)0, by = s.bfy ? s.bfy[i] : (Real)0, bz = s.bfz ? s.bfz[i] : (Real)0;
  const Real fx = bx + mu * ggx;
  const Real fy = by + mu * ggy + rhoPhaseNew * gravity;
  const Real fz = bz + mu * ggz;
  const Real invRho = (Real)1 / rhoPhaseNew;
  Real uxn = (mx + (Real)0.5 * fx) * invRho;
  Real uyn = (my + (Real)0.5 * fy) * invRho;
  Real uzn = (mz + (Real)0.5 * fz) * invRho;
  const Real u2 = uxn * uxn + uyn * uyn + uzn * uzn;
  const Real UMAX = (Real)0.2, UMAX2 = (Real)(0.2 * 0.2);
  if (u2 > UMAX2) {
    const Real sc = UMAX / sqrt(u2);
    uxn *= sc;
    uyn *= sc;
    uzn *= sc;
  }
  last[3] = (PopT)uxn;
  st4_global(f + 32 * 6, last);
  const PopT hl[4] = {h[4], h[5], h[6], (PopT)uyn};
  st4_global(s.H[cur] + bH + 32, hl);
  s.uz[cur][i] = uzn;
}

}  // namespace lbm
