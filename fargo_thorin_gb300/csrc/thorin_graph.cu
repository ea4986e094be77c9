// thorin_graph.cu -- the control kernels of a device-resident DT.
//
// One DT of AlgoGas (SourceEuler.c:210-317) runs as one CUDA graph: a WHILE
// node whose body is one substep, with the SOR sweep loop a WHILE node inside
// it.  Everything the host path decides between launches is decided here on
// the device, by one-thread kernels that run the host path's own source
// (thorin_planet.cuh): the substep interval and MinStepForRebound before the
// CFL, the pebble accretion set-up and Heating1 for each planet, the
// per-planet force constants and the indirect term, the planet kick, the
// N-body step and the frame rotation, the SOR omega schedule around each
// solve, and the loop condition.  This file is compiled without FMA
// contraction, so these kernels round like the host code.
//
// Bounded loops: the substep loop stops after GRAPH_MAX_SUBSTEPS substeps or
// on a non-positive dt (with an error flag the host reads); the SOR loop
// stops at the iteration cap (its completion step, k_sor_pass).
#include "thorin_graph.cuh"

__global__ void k_g_dt_begin(StepDev S)
{
  pdl_wait();
  if (threadIdx.x != 0) return;
  S.g.ctl[CTL_DTEMP] = 0.0;
  GraphStats *st = S.st;
  st->nsub = 0;
  st->crashed = 0;
  st->sor_calls = 0;
  st->sor_sweeps = 0;
  st->capped = 0;
  st->error = 0;
}

// SourceEuler.c:230-244 up to ConditionCFL: MassTaper, MinStepForRebound and
// the remaining interval of the DT.
__global__ void k_g_sub_begin(StepDev S)
{
  pdl_wait();
  if (threadIdx.x != 0) return;
  double *ctl = S.g.ctl;
  ctl[CTL_MASS_TAPER] = pl_mass_taper(ctl[CTL_TIME], S.c.mass_taper_param);
  ctl[CTL_INVDTREB] = pl_min_step_for_rebound(S.sys);
  ctl[CTL_DELTAT] = S.DT - ctl[CTL_DTEMP];
}

// InitHeating (Planet.c:251) and EvaporatePebbles' fraction of this dt.
__device__ void acc_init(const StepDev &S)
{
  for (int k = 0; k < S.npl; k++) { S.heat_val[k] = 0.0; S.heat_idx[k] = -1; }
  double facc = S.evaporation_rate * S.g.ctl[CTL_DT];
  if (facc > 1.0) facc = 1.0;
  S.g.ctl[CTL_FACC_EVAP] = facc;
}

__global__ void k_g_acc_init(StepDev S)
{
  pdl_wait();
  if (threadIdx.x == 0) acc_init(S);
}

// AccretePebblesOntoPlanets' set-up for planet k (the first: InitHeating too).
__global__ void k_g_acc_prep(StepDev S, int k)
{
  pdl_wait();
  if (threadIdx.x != 0) return;
  if (k == 0) acc_init(S);
  AccArgs a = *S.acc;
  pl_pebble_acc_prep(S.c, S.g.r.Rinf, S.g.r.Rsup, S.g.r.Rmed, S.sys, k, S.g.ctl[CTL_OMEGA_FRAME], S.g.ctl[CTL_DT],
                     ACC_BX, &a);
  *S.acc = a;
}

// dtemp += dt (SourceEuler.c:249), then FillForcesArrays' per-planet
// constants, the planets' indirect term and each planet's ring for
// DampingTW04.
__device__ void force_prep(const StepDev &S)
{
  S.iscal[IS_CRASH] = 0;
  double *ctl = S.g.ctl;
  ctl[CTL_DTEMP] += ctl[CTL_DT];
  double axs = 0.0, ays = 0.0;
  for (int k = 0; k < S.npl; k++) {
    pl_force_planet(S.c, S.g.r.Rsup, S.g.r.csmean, S.g.r.OmegaInv, S.sys, k, ctl[CTL_MASS_TAPER], &S.pl[k], &axs,
                    &ays);
    const double x = S.sys->x[k], y = S.sys->y[k];
    const double r = sqrt(x * x + y * y);
    const int i = (r >= S.c.rin && r <= S.c.rout) ? pl_ring_of(S.g.r.Rsup, S.c.nr, r) : -1;
    S.ring_info[k] = i;
    // the planet step runs beside the hydro substep, which rewrites the
    // ring means of c_s at its end: DampingTW04's value is taken now
    S.scal[SC_RCS + k] = (i >= 0) ? S.g.r.csmean[i] : 0.0;
  }
  ctl[CTL_INDX_PL] = S.indirect_term ? -axs : 0.0;
  ctl[CTL_INDY_PL] = S.indirect_term ? -ays : 0.0;
}

__global__ void k_g_force_prep(StepDev S)
{
  pdl_wait();
  if (threadIdx.x == 0) force_prep(S);
}

// Heating1 and the planet's new mass and velocity after the accretion; after
// the last planet's the forces' set-up.
__global__ void k_g_acc_finish(StepDev S, int k)
{
  pdl_wait();
  if (threadIdx.x != 0) return;
  const AccArgs &a = *S.acc;
  double dMp = 0.0, dPx = 0.0, dPy = 0.0;
  if (a.nb > 0) { dMp = S.scal[SC_ACC_DM]; dPx = S.scal[SC_ACC_DPX]; dPy = S.scal[SC_ACC_DPY]; }
  if (S.accret_heating) {
    int idx;
    double add;
    if (pl_heating1(S.c, S.g.r.Rsup, S.g.r.Surf, S.g.ctl[CTL_TIME], a.Mp, dMp, a.Xp, a.Yp, S.g.ctl[CTL_DT], &idx, &add)) {
      S.heat_idx[k] = idx;
      S.heat_val[k] += add;
    }
  }
  pl_pebble_acc_finish(S.sys, k, a, dMp, dPx, dPy);
  if (k == S.npl - 1) force_prep(S);
}

// The N-body step of thorin_planet.cuh (pl_nbody_step_n) by two warps.  Lane
// 3 i + c holds component c of body i's position and velocity (N <= 9 bodies,
// 27 lanes), so an update of the state is one FP64 instruction instead of 3 N,
// and a body's distance to another is formed from its three lanes' squares by
// shuffles.  Every sum keeps the order of the host's loops (a body's partners
// in ascending order, the star first), and 2 k and 1 k are exact products, so
// the results are the host's bits.
// A warp alone on its sub-partition gets one FP64 instruction per 64 cycles
// whatever the lanes do, and 1024 accelerations in line were longer than the
// hydro substep of a small disk.  But of a step's four only two are in line: a0
// and a1 need no other, a2 needs a0 and a3 needs a1.  So one warp (on another sub-partition) takes a0, a2 and
// the new positions, the other one a1, a3 and the new velocities, 39 FP64
// instructions each with two bodies, where one warp had 84: a DT of one substep of
// a 24x72 disk as a graph 866 -> 518 us.

// Acceleration of the lane's component at positions xt.
__device__ __forceinline__ double nbody_acc(double xt, double m, int N, int body, int c)
{
  const int b0 = 3 * body;                         // the body's first lane
  double a = 0.0;
  for (int k = 1; k < N; k++) {
    // partner k - 1 of the other bodies in ascending order; lanes of one
    // body take the same one, and every lane stays in the loop
    const int p = (k <= body) ? k - 1 : k;
    const double d = __shfl_sync(TH_FULL, xt, 3 * p + c) - xt;
    const double q = d * d;
    const double r2 = (__shfl_sync(TH_FULL, q, b0) + __shfl_sync(TH_FULL, q, b0 + 1)) + __shfl_sync(TH_FULL, q, b0 + 2);
    const double ir3 = div_fast(1.0, r2 * sqrt_fast(r2));
    const double f = __shfl_sync(TH_FULL, m, 3 * p) * d * ir3;
    a = (k == 1) ? f : a + f;
  }
  return a;
}

// By a block of two warps; ends with a barrier.
__device__ void nbody_step_pair(thorin_planets *sys, double dt)
{
  __shared__ double sa0[32], sa2[32], sv2[32], sxn[32], svn[32];
  const int N = sys->nb + 1;
  const int lane = threadIdx.x & 31, body = min(lane / 3, N - 1), c = lane - 3 * (lane / 3);
  const double *px = (c == 0) ? sys->x : (c == 1) ? sys->y : sys->z;
  const double *pv = (c == 0) ? sys->vx : (c == 1) ? sys->vy : sys->vz;
  double x = body > 0 ? px[body - 1] : 0.0, v = body > 0 ? pv[body - 1] : 0.0;
  const double m = body > 0 ? sys->mass[body - 1] : 1.0;
  // to the barycentre
  double M = 0.0, cx = 0.0, cv = 0.0;
  for (int i = 0; i < N; i++) {
    const double mi = __shfl_sync(TH_FULL, m, 3 * i);
    M += mi;
    cx += mi * __shfl_sync(TH_FULL, x, 3 * i + c);
    cv += mi * __shfl_sync(TH_FULL, v, 3 * i + c);
  }
  x -= cx / M;
  v -= cv / M;
  __syncthreads();                                 // both have read the state
  const int nsteps = 256;
  const double h = dt / nsteps, h6 = h / 6.0, hh = 0.5 * h;
  if (threadIdx.x < 32) {
    for (int s = 0; s < nsteps; s++) {
      const double a0 = nbody_acc(x, m, N, body, c);
      sa0[lane] = a0;
      const double v1 = v + hh * a0, x2 = x + hh * v1;
      const double a2 = nbody_acc(x2, m, N, body, c);
      sa2[lane] = a2;
      const double v3 = v + h * a2;
      __syncthreads();                             // a0, a2 and v2
      x += h6 * (__fma_rn(2.0, sv2[lane], __fma_rn(2.0, v1, v)) + v3);
      sxn[lane] = x;
      __syncthreads();                             // the new x and v
      v = svn[lane];
    }
  } else {
    for (int s = 0; s < nsteps; s++) {
      const double x1 = x + hh * v;
      const double a1 = nbody_acc(x1, m, N, body, c);
      const double v2 = v + hh * a1;
      sv2[lane] = v2;
      const double x3 = x + h * v2;
      const double a3 = nbody_acc(x3, m, N, body, c);
      __syncthreads();
      v += h6 * (__fma_rn(2.0, sa2[lane], __fma_rn(2.0, a1, sa0[lane])) + a3);
      svn[lane] = v;
      __syncthreads();
      x = sxn[lane];
    }
  }
  const double xh = x - __shfl_sync(TH_FULL, x, c), vh = v - __shfl_sync(TH_FULL, v, c);
  if (threadIdx.x >= 3 && threadIdx.x < 3 * N) {   // of the first warp
    double *ox = (c == 0) ? sys->x : (c == 1) ? sys->y : sys->z;
    double *ov = (c == 0) ? sys->vx : (c == 1) ? sys->vy : sys->vz;
    ox[body - 1] = xh;
    ov[body - 1] = vh;
  }
  __syncthreads();
}

// AdvanceSystemFromDisk with DampingTW04, the N-body step and RotatePsys
// (SourceEuler.c:251-268), two warps.
__global__ void __launch_bounds__(64) k_g_planet_step(StepDev S)
{
  pdl_wait();
  thorin_planets *sys = S.sys;
  const double dt = S.g.ctl[CTL_DT];
  if (threadIdx.x == 0) {
    double rrho[MAXPL_DEV], rcs[MAXPL_DEV];
    for (int k = 0; k < S.npl; k++) {
      sys->ax[k] = S.scal[SC_PLANET_A + 2 * k];
      sys->ay[k] = S.scal[SC_PLANET_A + 2 * k + 1];
      const int i = S.ring_info[k];
      rrho[k] = (i >= 0) ? S.scal[SC_PLANET_A + 2 * MAXPL_DEV + k] : 0.0;
      rcs[k] = (i >= 0) ? S.scal[SC_RCS + k] : 0.0;
    }
    const double ind[2] = {S.scal[SC_INDX], S.scal[SC_INDY]};
    pl_advance_from_disk(S.c, sys, dt, ind, rrho, rcs);
  }
  __syncthreads();
  if (sys->nb > 0) nbody_step_pair(sys, dt);
  if (threadIdx.x == 0) pl_rotate(sys, S.g.ctl[CTL_OMEGA_FRAME] * dt);
}

// The omega schedule before a solve (EnergySources.c:298-305); arms the
// sweep loop's condition, whose default is applied only once per launch of
// the whole graph.
__global__ void k_g_sor_begin(StepDev S)
{
  pdl_wait();
  if (threadIdx.x != 0) return;
  double *ctl = S.g.ctl;
  double omega = ctl[CTL_SOR_OMEGA] + ctl[CTL_SOR_DOMEGA], domega = ctl[CTL_SOR_DOMEGA];
  if (omega > TH_OMEGAUPPER) { omega = TH_OMEGAUPPER; domega = -domega; }
  if (omega < 1.0) { omega = 1.0; domega = -domega; }
  ctl[CTL_SOR_OMEGA] = omega;
  ctl[CTL_SOR_DOMEGA] = domega;
  if (S.sor_loop) cudaGraphSetConditional(S.h_sor, 1u);
}

// After a solve (EnergySources.c:306-317): counters, and the schedule's
// reversal when the solve took more sweeps than the last.
__global__ void k_g_sor_end(StepDev S)
{
  pdl_wait();
  if (threadIdx.x != 0) return;
  GraphStats *st = S.st;
  const int done = *S.sor.done, n = *S.sor.niter;
  if (!done || n < 1) st->error = 1;
  if (*S.sor.abort) st->error = 4;                 // the solve is void, whatever done says
  if (done == 2) st->capped = 1;
  st->sor_calls++;
  st->sor_sweeps += n;
  st->sor_last_niter = n;
  st->omega_used = S.g.ctl[CTL_SOR_OMEGA];
  if (n > st->niterlast) S.g.ctl[CTL_SOR_DOMEGA] = -S.g.ctl[CTL_SOR_DOMEGA];
  st->niterlast = n;
}

// End of a substep: the clock, the counters and the loop condition
// (dtemp < 0.999999999 DT, SourceEuler.c:229).
__global__ void k_g_sub_end(StepDev S)
{
  pdl_wait();
  if (threadIdx.x != 0) return;
  double *ctl = S.g.ctl;
  GraphStats *st = S.st;
  const double dt = ctl[CTL_DT];
  ctl[CTL_TIME] += dt;
  st->nsub++;
  st->crashed = S.iscal[IS_CRASH];
  unsigned more = (ctl[CTL_DTEMP] < 0.999999999 * S.DT) ? 1u : 0u;
  if (!(dt > 0.0)) { st->error = 3; more = 0u; }
  if (st->nsub >= GRAPH_MAX_SUBSTEPS) { st->error = 2; more = 0u; }
  if (st->error) more = 0u;
  cudaGraphSetConditional(S.h_sub, more);
}

void graph_dt_begin(const StepDev &S, cudaStream_t s) { launch(k_g_dt_begin, 1, 32, 0, s, S); g_thorin_launches++; }
void graph_sub_begin(const StepDev &S, cudaStream_t s) { launch(k_g_sub_begin, 1, 32, 0, s, S); g_thorin_launches++; }
void graph_acc_init(const StepDev &S, cudaStream_t s) { launch(k_g_acc_init, 1, 32, 0, s, S); g_thorin_launches++; }
void graph_acc_prep(const StepDev &S, int k, cudaStream_t s) { launch(k_g_acc_prep, 1, 32, 0, s, S, k); g_thorin_launches++; }
void graph_acc_finish(const StepDev &S, int k, cudaStream_t s) { launch(k_g_acc_finish, 1, 32, 0, s, S, k); g_thorin_launches++; }
void graph_force_prep(const StepDev &S, cudaStream_t s) { launch(k_g_force_prep, 1, 32, 0, s, S); g_thorin_launches++; }
void graph_planet_step(const StepDev &S, cudaStream_t s) { launch(k_g_planet_step, 1, 64, 0, s, S); g_thorin_launches++; }
void graph_sor_begin(const StepDev &S, cudaStream_t s) { launch(k_g_sor_begin, 1, 32, 0, s, S); g_thorin_launches++; }
void graph_sor_end(const StepDev &S, cudaStream_t s) { launch(k_g_sor_end, 1, 32, 0, s, S); g_thorin_launches++; }
void graph_sub_end(const StepDev &S, cudaStream_t s) { launch(k_g_sub_end, 1, 32, 0, s, S); g_thorin_launches++; }
