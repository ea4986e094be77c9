// kernels_hydro.cu -- source terms, viscosity, energy equation, SOR and
// transport of the AlgoGas substep (src_main/SourceEuler.c:319-586,
// Viscosity.c:85-260, EnergySources.c:75-856, TransportEuler.c:34-505).
//
// The kernels are bound by the FP64 pipe, so their arithmetic is regrouped for
// few FP64 instructions (each says how); results agree with the reference's
// operation order to rounding, and integer decisions are exact.
#include <cstdio>
#include <type_traits>
#include "thorin_kernels.cuh"

#define CELL_LOOP_2D                                                        \
  const int j = blockIdx.x * blockDim.x + threadIdx.x;                      \
  const int i = blockIdx.y;                                                 \
  if (j >= ns) return;                                                      \
  const int l = j + i * ns;

static inline dim3 grid2d(int ns, int rows, int bx) { return dim3((ns + bx - 1) / bx, rows); }
static const int BX = 128;

// Rings per block of a kernel whose threads walk the rings of a column: the
// chunk length with the least work on the busiest multiprocessor, which runs
// its blocks `slots` at a time and uses 1 - (1 - n / slots)^2 of the FP64 pipe
// with n of them left; `extra` is the work at a chunk's start, in rings.
static int chunk_rings(int nr, int ns, int nsm, int most, double extra, int slots = 4)
{
  const long long nbx = (ns + BX - 1) / BX;
  int best = 1;
  double bestw = 1e300;
  for (int r = 1; r <= most; r++) {
    const long long n = (nbx * ((nr + r - 1) / r) + nsm - 1) / nsm;
    const double full = (double)(n / slots * slots), part = (double)(n % slots), q = 1.0 - part / slots;
    const double w = (full + (part > 0.0 ? part / (1.0 - q * q) : 0.0)) * (r + extra);
    if (w < bestw) { bestw = w; best = r; }
  }
  return best;
}

// ---------------------------------------------------------------------------
// SubStep1 velocity predictor (SourceEuler.c:319-407), pressure from the
// energy (ComputePressureField, SourceEuler.c:740-762) or, in isothermal
// runs, the pressure field formed at the start of the substep; with pebbles
// also SourceTermsPebbles (Pebbles.c:550-613), SubStep1Pebbles (:617-652) and
// ParticleDiffusion (:656-698), whose new velocities go to pvrn, pvtn (the
// neighbours' old ones are read here).  Their accelerations and drags are used
// at the cell that forms them, so they stay in registers: six fields written
// and read less, and three launches in one.
//
// A thread walks the rings of a column and keeps what the next ring shares
// (pressure, half of the velocity average, the pebble-to-gas ratio); quotients
// by the same sums of densities share a reciprocal; the difference of the
// ratios of two columns is one quotient.  FP64-bound: about 30 FP64
// instructions a cell for the gas (40 before) and 98 with pebbles (135 in three
// kernels).  512x1536: 157 us, 213 us in three kernels.
#define SRC_MAXRINGS 24

struct SrcRing { double inv2, invrinf, ro, invdx2, supp, omega, oinv, cr, ct; };

template <bool PEB>
__global__ void __launch_bounds__(BX) k_sources(DevGrid g, SourceIO io)
{
  pdl_wait();
  __shared__ SrcRing ring[SRC_MAXRINGS];
  __shared__ double tab[128];
  const double dt = g.ctl[CTL_DT];
  const int ns = g.ns, nr = g.nr;
  const int i0 = blockIdx.y * io.rings, i1 = min(i0 + io.rings, nr);
  if ((int)threadIdx.x < i1 - i0) {
    const int i = i0 + threadIdx.x;
    SrcRing &R = ring[threadIdx.x];
    R.inv2 = 2.0 * g.r.InvDiffRmed[i];
    R.invrinf = g.r.InvRinf[i];
    R.ro = g.r.Rinf[i] * g.ctl[CTL_OMEGA_FRAME];
    R.invdx2 = 2.0 * io.invdxtheta[i];
    R.supp = io.supp_torque[i];
    if (PEB) {
      R.omega = g.r.Omega[i];
      R.oinv = g.r.OmegaInv[i];
      R.cr = div_fast(-g.r.nu_inf[i], io.schmidt) * g.r.InvDiffRmed[i];
      R.ct = div_fast(-g.r.nu_med[i], io.schmidt) * io.invdxtheta[i];
    }
  }
  if (PEB) tab[threadIdx.x] = c_exp64[threadIdx.x];
  __syncthreads();
  const int j = blockIdx.x * BX + threadIdx.x;
  if (j >= ns) return;
  const int jm = (j == 0) ? ns - 1 : j - 1, jp = (j == ns - 1) ? 0 : j + 1;
  const double colr = io.col[j], colt = io.col[ns + j];
  const double *pres = io.press ? io.press : io.energy;
  const double pscale = io.press ? 1.0 : io.gm1;
  // of the ring below: density, pressure, v_theta sum, acceleration
  double rho_m = 1.0, p_m = 0.0, vts_m = 0.0, ag_m = 0.0;
  double pd_m = 1.0, ratio_m = 0.0, pvts_m = 0.0, pag_m = 0.0;
  if (i0 > 0) {
    const int l = j + (i0 - 1) * ns, lp = jp + (i0 - 1) * ns;
    rho_m = io.rho[l];
    p_m = pscale * pres[l];
    vts_m = io.vt[l] + io.vt[lp];
    ag_m = io.agr[l];
    if (PEB) {
      pd_m = io.pd[l];
      ratio_m = div_fast(pd_m, rho_m);
      pvts_m = io.pvt[l] + io.pvt[lp];
      pag_m = io.pagr[l];
    }
  }
  for (int i = i0; i < i1; i++) {
    const SrcRing &R = ring[i - i0];
    const int row = i * ns, l = j + row, ljm = jm + row, ljp = jp + row;
    const double rho = io.rho[l], rho_jm = io.rho[ljm], p = pscale * pres[l], vr = io.vr[l], vt = io.vt[l];
    const double vts = vt + io.vt[ljp], ag = io.agr[l];
    double pd = 0.0, ratio = 0.0, pvts = 0.0, pag = 0.0, otau = 0.0, toinv = 0.0, ef = 0.0, ef1 = 0.0, pvr = 0.0,
           pvt = 0.0;
    if (PEB) {
      const double tau = io.tau[l];
      pd = io.pd[l];
      pvr = io.pvr[l];
      pvt = io.pvt[l];
      pvts = pvt + io.pvt[ljp];
      pag = io.pagr[l];
      otau = div_fast(R.omega, tau);
      toinv = tau * R.oinv;
      ef = exp_fast(-dt * otau, tab);
      ef1 = 1.0 - ef;
      if (io.diffusion) ratio = div_fast(pd, rho);
    }
    if (i >= 1) {
      const double den = rho + rho_m, ir = div_fast(1.0, den);
      double w = __fma_rn(vts + vts_m, 0.25, R.ro);
      double acc = __fma_rn(w * w, R.invrinf, -((p - p_m) * ir * R.inv2));
      acc = __fma_rn(0.5, ag + ag_m, acc) + colr;
      double v = __fma_rn(dt, acc, vr);
      if (PEB) {
        const double pds = pd + pd_m;
        if (io.back_reaction) {
          const double drag = (pvr - vr) * otau * (pds * ir);
          v = __fma_rn(dt, drag, v);
          acc += drag;
        }
        w = __fma_rn(pvts + pvts_m, 0.25, R.ro);
        const double pacc = __fma_rn(0.5, pag + pag_m, w * w * R.invrinf) + colr;
        double a = __fma_rn(__fma_rn(pacc - acc, toinv, vr), ef1, __fma_rn(acc, dt, pvr * ef));
        if (io.diffusion) a += div_fast(R.cr * (ratio - ratio_m) * den, pds);
        io.pvrn[l] = a;
      }
      io.vrint[l] = v;
    } else if (PEB) {
      io.pvrn[l] = pvr;
    }
    {
      const double den = rho + rho_jm, it = div_fast(1.0, den);
      double acc = __fma_rn(0.5, io.agt[l] + io.agt[ljm], -((p - pscale * pres[ljm]) * it * R.invdx2)) + colt;
      double v = __fma_rn(dt, acc, vt);
      if (R.supp != 0.0) {
        v = __fma_rn(dt, R.supp, v);
        acc += R.supp;
      }
      if (PEB) {
        const double pd_jm = io.pd[ljm], pds = pd + pd_jm;
        if (io.back_reaction) {
          const double drag = (pvt - vt) * otau * (pds * it);
          v = __fma_rn(dt, drag, v);
          acc += drag;
        }
        const double pacc = __fma_rn(0.5, io.pagt[l] + io.pagt[ljm], colt);
        double b = __fma_rn(__fma_rn(pacc - acc, toinv, vt), ef1, __fma_rn(acc, dt, pvt * ef));
        // (pd/rho - pd_jm/rho_jm) (rho + rho_jm) / (pd + pd_jm) as one quotient
        if (io.diffusion)
          b += div_fast(R.ct * __fma_rn(-pd_jm, rho, pd * rho_jm) * den, rho * rho_jm * pds);
        io.pvtn[l] = b;
      }
      io.vtint[l] = v;
    }
    if (PEB && i == nr - 1) io.pvrn[l + ns] = io.pvr[l + ns];     // row nrad as it was
    rho_m = rho; p_m = p; vts_m = vts; ag_m = ag;
    if (PEB) { pd_m = pd; ratio_m = ratio; pvts_m = pvts; pag_m = pag; }
  }
}

// UpdateDivVelocAndStressTensor (Viscosity.c:85-162): divergence and the
// three stress components of a cell from the staggered velocities, with the
// ring's constants folded into its coefficients.
struct StressRing { double cr, cp, cv, rsup, rinf, cd, nu2, t1, t2; };

__device__ __forceinline__ void stress_ring(const DevGrid &g, int i, double invdphi, StressRing &R)
{
  const double ir = g.r.InvRmed[i];
  R.cr = g.r.InvDiffRsup[i];
  R.cp = invdphi * ir;                       // (v_theta(j+1) - v_theta(j)) cp
  R.cv = 0.5 * ir;                           // (v_r(i+1) + v_r(i)) cv
  R.rsup = g.r.Rsup[i];
  R.rinf = g.r.Rinf[i];
  R.cd = R.cr * ir;
  R.nu2 = 2.0 * g.r.nu_med[i];
  // tau_rp = 2 rho_4/4 nu (r dOmega/dr + (v_r(j) - v_r(j-1)) / (r dphi)) / 2
  const double n = 0.25 * g.r.nu_inf[i];
  R.t1 = n * g.r.Rinf[i] * g.r.InvDiffRmed[i];
  R.t2 = n * invdphi * g.r.InvRinf[i];
}

struct Stress { double divv, trr, tpp, trp; };

// om, om_m: v_theta / r of the cell and of the one below; rs, rs_m: the
// densities of the cell and its left neighbour added, and those below.
__device__ __forceinline__ Stress stress_cell(const StressRing &R, int i, double vr, double vr_ip, double vr_jm,
                                              double vt, double vt_jp, double om, double om_m, double rho, double rs,
                                              double rs_m)
{
  Stress s;
  const double dt = (vt_jp - vt) * R.cp;
  const double Drr = (vr_ip - vr) * R.cr;
  const double Dpp = __fma_rn(vr_ip + vr, R.cv, dt);
  s.divv = __fma_rn(__fma_rn(vr_ip, R.rsup, -(vr * R.rinf)), R.cd, dt);
  const double n = R.nu2 * rho;
  s.trr = n * __fma_rn(-1.0 / 3.0, s.divv, Drr);
  s.tpp = n * __fma_rn(-1.0 / 3.0, s.divv, Dpp);
  s.trp = (i >= 1) ? (rs + rs_m) * __fma_rn(vr - vr_jm, R.t2, (om - om_m) * R.t1) : 0.0;
  return s;
}

// The viscous terms and SubStep2 in one kernel: the stress tensor,
// UpdateVelocityWithViscousTerms (Viscosity.c:165-218), ImposeKeplerianEdges
// (:221-260) and the von Neumann-Richtmyer artificial viscosity with its
// velocity and energy updates (SourceEuler.c:417-504).
//
// A thread walks the rings of a column; at ring k it forms the stress of ring
// k, v_r of ring k, v_theta of ring k-1 and writes ring k-1.  Neighbours in
// azimuth pass stress, v_theta and the artificial pressure through shared
// memory, so a block of 128 threads covers 125 columns (two on the left and one
// on the right only feed their neighbours).  The sums of densities and their reciprocals are
// shared by both parts.  FP64-bound: about 58 FP64 instructions a cell plus 1.8
// rings a chunk, where the three kernels took 103 and kept three fields between
// them; 512x1536: 166 -> 133 us.
#define VI_MAXRINGS 40
#define VI_COLS (BX - 3)

struct ViscRing { StressRing s; double irm, a, b, c, ra, rm, rc, rt, sr, st, er, et; };

__global__ void __launch_bounds__(BX) k_viscous(DevGrid g, ViscousIO io)
{
  pdl_wait();
  __shared__ ViscRing ring[VI_MAXRINGS + 3];
  __shared__ double s_tpp[2][BX], s_trp[2][BX], s_vt[BX], s_q[BX];
  const double dt = g.ctl[CTL_DT];
  const int ns = g.ns, nr = g.nr;
  const int i0 = blockIdx.y * io.rings, i1 = min(i0 + io.rings, nr);
  const int k0 = max(i0 - 2, 0);
  for (int q = threadIdx.x; q <= min(i1, nr - 1) - k0; q += BX) {
    const int i = k0 + q;
    ViscRing &R = ring[q];
    stress_ring(g, i, io.invdphi, R.s);
    R.irm = g.r.InvRmed[i];
    // v_theta += 2 dt / r (...) / (rho + rho_jm), v_r += 2 dt / r (...) / (rho + rho_im)
    const double ct = 2.0 * dt * g.r.InvRmed[i], cr = 2.0 * dt * g.r.InvRinf[i];
    R.a = ct * __fma_rn(g.r.Rsup[i], g.r.InvDiffRsup[i], 0.5);            // tau_rp(i+1)
    R.b = ct * __fma_rn(-g.r.Rinf[i], g.r.InvDiffRsup[i], 0.5);           // tau_rp(i)
    R.c = ct * io.invdphi;                                                // tau_pp - tau_pp(j-1)
    R.ra = cr * g.r.Rmed[i] * g.r.InvDiffRmed[i];                         // tau_rr
    R.rm = (i >= 1) ? -(cr * g.r.Rmed[i - 1] * g.r.InvDiffRmed[i]) : 0.0; // tau_rr(i-1)
    R.rc = cr * io.invdphi;                                               // tau_rp(j+1) - tau_rp
    R.rt = -0.5 * cr;                                                     // tau_pp + tau_pp(i-1)
    R.sr = -2.0 * dt * g.r.InvDiffRmed[i];                                // q_r - q_r(i-1)
    R.st = -2.0 * dt * io.invdxtheta[i];                                  // q_t - q_t(j-1)
    R.er = -dt * g.r.InvDiffRsup[i];
    R.et = -dt * io.invdxtheta[i];
  }
  __syncthreads();
  const int t = threadIdx.x, x = blockIdx.x * VI_COLS + t - 2;
  const bool out = t >= 2 && t < BX - 1 && x < ns;
  int j = x;                                       // wrapped column (ns >= 4)
  if (j < 0) j += ns;
  j %= ns;
  const int jm = (j == 0) ? ns - 1 : j - 1, jp = (j == ns - 1) ? 0 : j + 1;
  const int tm = (t == 0) ? 0 : t - 1, tp = (t == BX - 1) ? t : t + 1;
  // of ring k-1: stress, rotation rate, density sums, old v_theta; of ring k-1 and k-2 after the viscous update
  double trr_m = 0.0, tpp_m = 0.0, trp_m = 0.0, dtp_m = 0.0, om_m = 0.0, rs_m = 0.0, rho_m = 0.0, vt_m = 0.0;
  double vr_m = 0.0, qr_m = 0.0, ir_m = 0.0;
  if (k0 > 0) {
    const int l = j + (k0 - 1) * ns;
    om_m = io.vt[l] * g.r.InvRmed[k0 - 1];
    rho_m = io.rho[l];
    rs_m = rho_m + io.rho[jm + (k0 - 1) * ns];
  }
  double vr = io.vr[j + k0 * ns];
  const int k1 = i1;                               // ring k1 closes ring i1 - 1
  for (int k = k0; k <= k1; k++) {
    const int row = k * ns, l = j + row;
    const bool body = k < nr;
    double trr = 0.0, tpp = 0.0, trp = 0.0, om = 0.0, rs = 0.0, rho = 0.0, vt = 0.0, vr_ip = 0.0;
    if (body) {
      const ViscRing &R = ring[k - k0];
      vr_ip = io.vr[l + ns];
      vt = io.vt[l];
      rho = io.rho[l];
      rs = rho + io.rho[jm + row];
      om = vt * R.irm;
      const Stress s = stress_cell(R.s, k, vr, vr_ip, io.vr[jm + row], vt, io.vt[jp + row], om, om_m, rho, rs, rs_m);
      trr = s.trr; tpp = s.tpp; trp = s.trp;
      if (io.divv && out && k >= i0 && k < i1) io.divv[l] = s.divv;
    }
    s_tpp[k & 1][t] = tpp;
    s_trp[k & 1][t] = trp;
    __syncthreads();
    // v_r of ring k
    double vrn = vr, ir = 0.0;
    if (body && k >= 1) {
      const ViscRing &R = ring[k - k0];
      ir = div_fast(1.0, rho + rho_m);
      const double w = __fma_rn(trr, R.ra, __fma_rn(trr_m, R.rm, __fma_rn(s_trp[k & 1][tp] - trp, R.rc, (tpp + tpp_m) * R.rt)));
      vrn = __fma_rn(w, ir, vr);
    }
    // v_theta of ring k-1, then SubStep2 of ring k-1
    const int m = k - 1;
    if (m >= i0 - 1 && m >= k0) {
      const ViscRing &R = ring[m - k0];
      double vtn = vt_m, it = 0.0;
      if (m >= i0) {
        it = div_fast(1.0, rs_m);
        if (m >= 1 && m < nr - 1) {
          const double w = __fma_rn(trp, R.a, __fma_rn(trp_m, R.b, dtp_m * R.c));
          vtn = __fma_rn(w, it, vt_m);
        }
        if (io.kepler) {
          if (m == 0) vtn = io.vkep_in;
          if (m == nr - 1) vtn = io.vkep_out;
        }
      }
      const double dvr = vrn - vr_m;
      const double cq = (TH_CVNR * TH_CVNR) * rho_m;
      const double qr = (__double_as_longlong(dvr) < 0LL) ? cq * dvr * dvr : 0.0;
      if (m >= i0) {                               // block-uniform
        s_vt[t] = vtn;
        __syncthreads();
        const double dvt = s_vt[tp] - vtn;
        const double qt = (__double_as_longlong(dvt) < 0LL) ? cq * dvt * dvt : 0.0;
        s_q[t] = qt;
        __syncthreads();
        if (out) {
          const int lm = l - ns;
          io.vrnew[lm] = (m >= 1) ? __fma_rn((qr - qr_m) * ir_m, R.sr, vr_m) : 0.0;
          io.vtnew[lm] = __fma_rn((qt - s_q[tm]) * it, R.st, vtn);
          if (io.eint) io.eint[lm] = __fma_rn(qt * dvt, R.et, __fma_rn(qr * dvr, R.er, io.energy[lm]));
        }
      }
      qr_m = qr;
    }
    dtp_m = tpp - s_tpp[k & 1][tm];
    trr_m = trr; tpp_m = tpp; trp_m = trp; om_m = om; rs_m = rs; rho_m = rho; vt_m = vt;
    vr_m = vrn;
    ir_m = ir;
    vr = vr_ip;
  }
  if (i1 == nr && out) {                           // rows the reference never writes stay zero
    io.vrnew[j + nr * ns] = 0.0;
    io.vtnew[j + nr * ns] = 0.0;
  }
}

// SubStep3 viscous heating (SourceEuler.c:541-567) from the stress of the
// updated velocities (the second UpdateDivVelocAndStressTensor call,
// SourceEuler.c:302), with its power-law extrapolation into ring 0, and the
// temperature and sound speed of the energy equation's start
// (ComputeTemperatureField, ComputeSoundSpeed; temper NULL: neither).  A thread
// walks the rings of a column.  FP64-bound: 42 FP64 instructions a cell, 57 in
// the three kernels before; 512x1536: 99 -> 71 us.
#define HT_MAXRINGS 24

__global__ void __launch_bounds__(BX) k_heating(DevGrid g, HeatingIO io)
{
  pdl_wait();
  __shared__ StressRing ring[HT_MAXRINGS];
  const int ns = g.ns, nr = g.nr;
  const int i0 = blockIdx.y * io.rings, i1 = min(i0 + io.rings, nr);
  if ((int)threadIdx.x < i1 - i0) stress_ring(g, i0 + threadIdx.x, io.invdphi, ring[threadIdx.x]);
  __syncthreads();
  const int j = blockIdx.x * BX + threadIdx.x;
  if (j >= ns) return;
  const int jm = (j == 0) ? ns - 1 : j - 1, jp = (j == ns - 1) ? 0 : j + 1;
  double om_m = 0.0, rs_m = 0.0, q1 = 0.0;
  if (i0 > 0) {
    const int l = j + (i0 - 1) * ns;
    om_m = io.vt[l] * g.r.InvRmed[i0 - 1];
    rs_m = io.rho[l] + io.rho[jm + (i0 - 1) * ns];
  }
  double vr = io.vr[j + i0 * ns];
  for (int i = i0; i < i1; i++) {
    const StressRing &R = ring[i - i0];
    const int row = i * ns, l = j + row;
    const double vr_ip = io.vr[l + ns], vt = io.vt[l], rho = io.rho[l];
    const double rs = rho + io.rho[jm + row], om = vt * g.r.InvRmed[i];
    const Stress s = stress_cell(R, i, vr, vr_ip, io.vr[jm + row], vt, io.vt[jp + row], om, om_m, rho, rs, rs_m);
    io.divv[l] = s.divv;
    if (i >= 1) {
      double q = 0.0;
      if (R.nu2 != 0.0) {
        const double n = R.nu2 * rho;                          // 2 nu rho
        q = div_fast(__fma_rn(s.trr, s.trr, __fma_rn(s.tpp, s.tpp, 2.0 * s.trp * s.trp)), n);
        q = __fma_rn((1.0 / 9.0) * n * s.divv, s.divv, q);
      }
      io.qplus[l] = q;
      if (i == 1) q1 = q;
      if (i == 2)
        io.qplus[j] = (g.r.nu_med[0] != 0.0) ? q1 * exp(log(q1 / q) * io.lr01 / io.lr12) : 0.0;
    }
    if (io.temper) {
      const double T = div_fast(io.energy[l] * io.gm1, rho);
      io.temper[l] = T;
      io.cs[l] = sqrt_fast(io.gamma * abs_i(T));               // gamma (gamma - 1) e / rho = gamma T
    }
    om_m = om; rs_m = rs;
    vr = vr_ip;
  }
}

// ---------------------------------------------------------------------------
// Energy equation (EnergySources.c)
// ComputeTemperatureField + ComputeSoundSpeed (SourceEuler.c:715-792).
__global__ void k_eos(DevGrid g, const double *__restrict__ rho, const double *__restrict__ energy,
                      double *__restrict__ temper, double *__restrict__ cs, double gm1, double gamma)
{
  pdl_wait();
  const int ns = g.ns;
  CELL_LOOP_2D
  // c_s = sqrt(gamma (gamma - 1) |e| / rho) = sqrt(gamma |T|)
  const double t = div_fast(energy[l] * gm1, rho[l]);
  if (temper) temper[l] = t;                // NULL: ComputeSoundSpeed alone
  cs[l] = sqrt_fast(gamma * abs_i(t));
}

// Opacity laws, Opacity.c.
// Bell & Lin (Opacity.c:31-75).  The thresholds T(i,j) solve
// kappa_i rho^a_i T^b_i = kappa_j rho^a_j T^b_j.  The first branch
// (T <= T(2,3), grains) covers almost the whole disk; its test
// T <= (kappa_3/kappa_2 rho)^(1/24.5) is decided by FP32 logarithms unless the
// two sides are within 0.01 of each other in log2, then as T^49 <=
// (kappa_3/kappa_2 rho)^2 unless those are within 1e-12, when the threshold
// itself is evaluated with pow as in the reference.  The grain branch's integer
// and half powers are products, quotients and roots (each within a few ulp of
// pow); it does not use rho, so rho = vd * rho2cgs is formed only where it is
// needed.
__device__ __forceinline__ double pow_int_pos(double x, int n)
{
  double r = 1.0, b = x;
  while (n) { if (n & 1) r *= b; b *= b; n >>= 1; }
  return r;
}

__device__ double opacity_BL94(double vd, double rho2cgs, double T)
{
  const double kappa[8] = {2.0e-4, 2.0e16, 0.1, 2.0e81, 1.0e-8, 1.0e-36, 1.5e20, 0.348};
  const double a[8] = {0.0, 0.0, 0.0, 1.0, 2.0 / 3.0, 1.0 / 3.0, 1.0, 0.0};
  const double b[8] = {2.0, -7.0, 0.5, -24.0, 3.0, 10.0, -2.5, 0.0};
#define TEMPB(i, j) pow(kappa[j] / kappa[i] * pow(rho, a[j] - a[i]), 1.0 / (b[i] - b[j]))
  bool grains;
  // 49 log2 T against 2 log2(kappa_3/kappa_2 rho), each within 1e-4
  const float Tf = to_float_pos(T), rf = to_float_pos(vd) * (float)rho2cgs;
  const float d = (Tf > 0.0f && rf > 0.0f)
                      ? 49.0f * __log2f(Tf) - 2.0f * (__log2f(rf) + 273.39788f) : 0.0f;    // log2(2e82)
  double rho = 0.0;
  if (fabsf(d) > 0.01f) {
    grains = d < 0.0f;
    if (!grains) rho = vd * rho2cgs;
  } else {
    rho = vd * rho2cgs;
    const double c23 = kappa[3] / kappa[2] * rho;          // (kappa_3/kappa_2) rho^(a_3-a_2), a_3-a_2 = 1
    if (T > 0.0 && T < 1.0e5 && c23 > 0.0 && c23 < 1.0e150) {
      const double lhs = pow_int_pos(T, 49), rhs = c23 * c23;
      if (lhs < rhs * (1.0 - 1e-12)) grains = true;
      else if (lhs > rhs * (1.0 + 1e-12)) grains = false;
      else grains = (T <= TEMPB(2, 3));
    } else {
      grains = (T <= TEMPB(2, 3));
      if (grains && T < 0.0) return sqrt(T);                 // not a number, as the reference's T^(1/2)
    }
  }
  double k;
  if (grains) {
    // k1 = kappa0 T^2, k2 = kappa1 T^-7, k3 = kappa2 T^0.5;
    // t1 = (k1^-2 + k2^-2)^-2, x = k3 / (1 + 1e22 T^-10), k = (t1 + x^4)^(1/4),
    // rearranged to two divisions; x only enters squared, so without the root
    const double T2 = T * T, T4 = T2 * T2, T5 = T4 * T, T10 = T5 * T5, T14 = T10 * T4;
    const double ik = div_fast(T4, __fma_rn(2.5e-33 * T14, T4, 2.5e7));         // 1 / (k1^-2 + k2^-2) = T^4 / (2.5e7 + 2.5e-33 T^18)
    const double u = div_fast(T10, T10 + 1.0e22);
    const double x2 = (kappa[2] * kappa[2]) * T * (u * u);
    k = root4(__fma_rn(ik, ik, x2 * x2));
  } else if (T > 0.0 && rho > 0.0) {
    // T <= TEMPB(i, j) compared as logarithms: ln T <= (ln(kappa_j / kappa_i)
    // + (a_j - a_i) ln rho) / (b_i - b_j), one log each of rho and T; the
    // regimes' power laws with integer powers, cbrt and sqrt
    const double lr = log(rho), lT = log(T);
    const double t34 = __fma_rn(-0.33333333333333337, lr, -205.62322045703002) * -0.037037037037037035;
    const double t45 = __fma_rn(-0.3333333333333333, lr, -64.47238260383328) * -0.14285714285714285;
    const double t56 = __fma_rn(0.6666666666666667, lr, 129.35023031577472) * 0.08;
    const double t67 = __fma_rn(-1.0, lr, -47.51271976719674) * -0.4;
    const double T2 = T * T;
    if (lT <= t34) {
      const double T3 = T2 * T, T6 = T3 * T3, T12 = T6 * T6;
      k = div_fast(kappa[3] * rho, T12 * T12);                 // rho T^-24
    } else if (lT <= t45) {
      const double c = cbrt(rho);
      k = kappa[4] * (c * c) * (T2 * T);                       // rho^(2/3) T^3
    } else if (lT <= t56) {
      const double T5 = T2 * T2 * T;
      k = kappa[5] * cbrt(rho) * (T5 * T5);                    // rho^(1/3) T^10
    } else if (lT <= t67) {
      k = div_fast(kappa[6] * rho, T2 * sqrt(T));              // rho T^-2.5
    } else {
      k = kappa[7];
    }
  } else if (T <= TEMPB(3, 4)) {
    k = kappa[3] * pow(rho, a[3]) * pow(T, b[3]);
  } else if ((T > TEMPB(3, 4)) && (T <= TEMPB(4, 5))) {
    k = kappa[4] * pow(rho, a[4]) * pow(T, b[4]);
  } else if ((T > TEMPB(4, 5)) && (T <= TEMPB(5, 6))) {
    k = kappa[5] * pow(rho, a[5]) * pow(T, b[5]);
  } else if ((T > TEMPB(5, 6)) && (T <= TEMPB(6, 7))) {
    k = kappa[6] * pow(rho, a[6]) * pow(T, b[6]);
  } else {
    k = kappa[7];
  }
#undef TEMPB
  return k;
}

// The two ice and silicate regimes, which hold most of a disk (T below about
// 600 K but for a narrow band at the ice line), are kappa = C T^1.5: no logarithm
// and no power.  FP32 logarithms (within 1e-5) decide the regime unless a
// threshold is within 1e-3 of it.  214 FP64 instructions a cell of k_diffcoef
// with the logarithms everywhere, 105 with this; 384x1152: 195 -> 116 us.
__device__ double opacity_ZHU12(double vd, double rho2cgs, double T)
{
  const float Tf = to_float_pos(T), rf = to_float_pos(vd) * (float)rho2cgs;
  if (Tf > 0.0f && rf > 0.0f && Tf < 1e30f && rf < 1e30f) {
    const float lt = 0.30103f * __log2f(Tf), lp = 0.30103f * __log2f(rf) + lt + 7.5395978f;   // log10(8.3144598e7 / 2.4)
    const float d1 = lt - (2.23567f + 0.01899f * (lp - 5.0f)), d2 = lt - (2.30713f + 0.01899f * (lp - 5.0f));
    const bool ice = d1 < -1e-3f, silicate = d1 > 1e-3f && d2 > 1e-3f && lt < 2.8015132f - 1e-3f;      // (17.08 + 1.5 2.30713) / 7.332
    // the last rule's floor 3.586 lt - 16.85 is far below either
    if ((ice || silicate) && lt < 3.0f) return (ice ? 0.0033011936420003054 : 0.001443128488200116) * (T * sqrt_fast(T));  // 10^-2.481329, 10^-2.840695
  }
  const double rho = vd * rho2cgs;
  double xlop, pre = 8.3144598 * 1.0e7 / 2.4 * rho * T;
  double xlp = log10(pre), xlt = log10(T);
  if (xlt < 2.23567 + 0.01899 * (xlp - 5.)) xlop = 1.5 * (xlt - 1.16331) - 0.736364;
  else if (xlt < 2.30713 + 0.01899 * (xlp - 5.)) xlop = -3.53154212 * xlt + 8.767726 - (7.24786 - 8.767726) * (xlp - 5.) / 16.;
  else if (xlt < (17.7 - 0.62 + 1.5 * 2.30713) / (1.5 + 5.832)) xlop = 1.5 * (xlt - 2.30713) + 0.62;
  else if (xlt < (5.9398 + 17.7) / (5.832 + 2.129)) xlop = -5.832 * xlt + 17.7;
  else if (xlt < (129.88071 + 5.9398 + (142.996475 - 129.88071) * 0.1 * (xlp + 4.)) / (2.129 + 42.98075)) xlop = 2.129 * xlt - 5.9398;
  else if (xlt < (129.88071 + 15.0125 + (142.996475 - 129.88071) * 0.1 * (xlp + 4.)) / (4.0625 + 42.98075)) xlop = 129.88071 - 42.98075 * xlt + (142.996475 - 129.88071) * 0.1 * (xlp + 4.0);
  else if (xlt < 3.28 + xlp / 4. * 0.12) xlop = -15.0125 + 4.0625 * xlt;
  else if (xlt < 3.41 + 0.03328 * xlp / 4.) xlop = 58.9294 - 18.4808 * xlt + (61.6346 - 58.9294) * xlp / 4.;
  else if (xlt < 3.76 + (xlp - 4) / 2. * 0.03) xlop = -12.002 + 2.90477 * xlt + (xlp - 4) / 4. * (13.9953 - 12.002);
  else if (xlt < 4.07 + (xlp - 4) / 2. * 0.08) xlop = -39.4077 + 10.1935 * xlt + (xlp - 4) / 2. * (40.1719 - 39.4077);
  else if (xlt < 5.3715 + (xlp - 6) / 2. * 0.5594) xlop = 17.5935 - 3.3647 * xlt + (xlp - 6) / 2. * (17.5935 - 15.7376);
  else xlop = -0.48;
  if (xlop < 3.586 * xlt - 16.85 && xlt < 4.) xlop = 3.586 * xlt - 16.85;
  return exp10(xlop);
}

__device__ double opacity_LP85(double rho, double T)
{
  if (T < pow(2.0e-4 / 2.0e16, -1.0 / 9.0)) return 2.0e-4 * T * T;
  if (T < pow(2.0e16 / 5.0e-3, 1.0 / 8.0)) return 2.0e16 * pow(T, -7.0);
  if (T < pow(5.0e-3 / 2.0e34, -1.0 / 10.0) * pow(rho, 1.0 / 15.0)) return 5.0e-3 * T;
  if (T < pow(2.0e34 / 2.0e-8, 1.0 / 12.0)) return 2.0e34 * pow(rho, 2.0 / 3.0) * pow(T, -9.0);
  if (T < pow(2.0e-8 / 1.0e-36, 1.0 / 7.0) * pow(rho, 1.0 / 21.0)) return 2.0e-8 * pow(rho, 2.0 / 3.0) * T * T * T;
  if (T < pow(1.0e-36 / 1.5e20, -1.0 / 12.5) * pow(rho, 4.0 / 75.0)) return 1.0e-36 * pow(rho, 1.0 / 3.0) * pow(T, 10.0);
  return 1.5e20 * rho * pow(T, -5.0 / 2.0);
}

// Semenov et al. (2003) dust with Malygin et al. (2014) gas, Rosseland
// means (Opacity2.c:25-245): fifth-order polynomials in T per dust regime,
// evaporation temperatures interpolated in log rho, sine smoothing across the
// transitions (tested, as in the reference, on the integer part of
// |T - T_i|), and a bilinear pressure-temperature lookup in the gas table.
__constant__ double c_sm_dust[36] = {
    0.244153190819473e-03, -0.191588103585833e-03, 0.229132294521843e-03, 0.454088516995579e-06,
    -0.389280273285906e-08, 0.319006401785413e-11,
    0.292517586013911e+01, -0.801305197566973e-01, 0.923001367150898e-03, -0.349287851393541e-05,
    0.587151269508960e-08, -0.371333580736933e-11,
    -0.125893536782728e+02, 0.160197849829283e+00, -0.582601311634824e-03, 0.110792133181219e-05,
    -0.105506373600323e-08, 0.404997080931974e-12,
    -0.192550086994197e+01, 0.354301116460647e-01, -0.127355043519226e-03, 0.233773506650911e-06,
    -0.207587683535083e-09, 0.728005983960845e-13,
    0.165244978116957e+01, -0.260479348963077e-02, 0.590717655258634e-05, -0.300202906476749e-08,
    0.803836688553263e-12, -0.916709776405312e-16,
    0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
__constant__ double c_sm_logtt[32] = {
    2.03742650, 2.92168648, 2.95520654, 2.96801571, 2.07188201, 2.95808585, 2.99122608, 2.99869516,
    2.11058971, 2.99738638, 3.02077549, 3.03181227, 2.15533604, 3.04139269, 3.05269394, 3.06744284,
    2.20139712, 3.08990511, 3.08707121, 3.10619090, 2.25527251, 3.14457421, 3.12417806, 3.14860265,
    2.31597035, 3.20736504, 3.16494737, 3.19589965, 2.38738983, 3.28057837, 3.20978301, 3.24895362};

__device__ double opacity_SM03(const DevConst &k, double rho, double T_dust)
{
  if (T_dust <= 0.9) return 0.9;
  const double logrho = log10(rho);
  double T[5], dT[5] = {5.0, 5.0, 15.0, 5.0, 100.0}, T_ev[4];
  for (int c = 0; c < 4; c++) {                  // interp over log rho = -18, -16, ..., -4
    double v;
    if (logrho < -18.0) v = c_sm_logtt[c];
    else if (logrho > -4.0) v = c_sm_logtt[28 + c];
    else {
      int i = 1;
      while ((-18.0 + 2.0 * i < logrho) && (i < 7)) i++;
      const double x0 = -18.0 + 2.0 * (i - 1), x1 = -18.0 + 2.0 * i;
      const double y0 = c_sm_logtt[4 * (i - 1) + c], y1 = c_sm_logtt[4 * i + c];
      v = y0 + (y1 - y0) * (logrho - x0) / (x1 - x0);
    }
    T_ev[c] = pow(10.0, v);
  }
  T[0] = T_ev[0]; T[1] = 275.0; T[2] = 425.0; T[3] = 680.0;
  const double tmax1 = (T_ev[1] > T_ev[2]) ? T_ev[1] : T_ev[2];
  const double tmax2 = (T_ev[2] > T_ev[3]) ? T_ev[2] : T_ev[3];
  T[4] = (tmax1 < tmax2) ? tmax1 : tmax2;
  int KK = 5;
  if (T_dust <= (T[0] + dT[0])) KK = 0;
  for (int i = 1; i < 5; i++)
    if ((T_dust > (T[i - 1] + dT[i - 1])) && (T_dust <= (T[i] + dT[i]))) KK = i;
  double aKext = 0.0;
  if (KK != 5) {
    int smooth = 0;
    for (int i = 0; i < 5; i++)
      if (abs((int)(T_dust - T[i])) < dT[i]) smooth = 1;
    const double *eD = c_sm_dust;
    auto poly = [&](int j, double x) {
      return ((((eD[j - 1] * x + eD[j - 2]) * x + eD[j - 3]) * x + eD[j - 4]) * x + eD[j - 5]) * x + eD[j - 6];
    };
    if (smooth) {
      const double T1 = T[KK] - dT[KK], T2 = T[KK] + dT[KK], TD = T_dust - T[KK];
      const double aKrL = poly((KK + 1) * 6, T1);
      const double aKrR = (KK == 4) ? 0.0 : poly((KK + 2) * 6, T2);
      const double AA = 0.5e0 * (aKrL - aKrR), BB = 0.5e0 * (aKrL + aKrR), FF = TH_PI / 2.0 / dT[KK];
      aKext = BB - AA * sin(FF * TD);
    } else {
      aKext = poly((KK + 1) * 6, T_dust);
    }
  }
  // Malygin gas table (Opacity2.c:45-92)
  const int rows = k.sm_rows, cols = k.sm_cols;
  const double *pg = k.sm_pgrid, *tg = k.sm_tgrid;
  double tP = 8.3144598 * 1.0e7 / 2.4 * rho * T_dust, tT = T_dust, kappa_gas;
  if (tT < tg[0]) {
    kappa_gas = 0.0;
  } else {
    if (tT > tg[cols - 1]) tT = tg[cols - 1];
    if (tP < pg[0]) tP = pg[0];
    else if (tP > pg[rows - 1]) tP = pg[rows - 1];
    int Tlow = 0, Thigh = 1;
    for (int i = 0; i < cols - 2; i++)
      if (tT >= tg[i]) { Tlow = i; Thigh = i + 1; }
    const double fac = ((double)rows) / log10(pg[rows - 1] / pg[0]);
    int Plow = (int)(fac * log10(tP / pg[0]));
    Plow = (Plow > 0) ? Plow : 0;
    Plow = (Plow < rows - 2) ? Plow : rows - 2;
    const int Phigh = Plow + 1;
    const double denom = 1.0 / ((tg[Thigh] - tg[Tlow]) * (pg[Phigh] - pg[Plow]));
    const double mul1 = (tg[Thigh] - tT) * (pg[Phigh] - tP), mul2 = (tT - tg[Tlow]) * (pg[Phigh] - tP);
    const double mul3 = (tg[Thigh] - tT) * (tP - pg[Plow]), mul4 = (tT - tg[Tlow]) * (tP - pg[Plow]);
    const double *a = k.sm_ross;
    kappa_gas = denom * (mul1 * a[Tlow + Plow * cols] + mul2 * a[Thigh + Plow * cols] + mul3 * a[Tlow + Phigh * cols] +
                         mul4 * a[Thigh + Phigh * cols]);
  }
  return (aKext > kappa_gas) ? aKext : kappa_gas;
}

template <int LAW>
__device__ __forceinline__ double opacity_law(const DevConst &k, double vd, double T)
{
  if (LAW == THORIN_OPA_SM03) return opacity_SM03(k, vd * k.rho2cgs, T);
  if (LAW == THORIN_OPA_ZHU12) return opacity_ZHU12(vd, k.rho2cgs, T);
  if (LAW == THORIN_OPA_LP85) return opacity_LP85(vd * k.rho2cgs, T);
  return opacity_BL94(vd, k.rho2cgs, T);
}

// MidplaneVolumeDensity, OpacityProfile, CalculateQminus and the centred
// diffusion coefficient of DiffusionCoefs (EnergySources.c:556-592,
// 658-711, Opacity.c:231-266), and DiffusionTimestep (EnergySources.c:
// 833-856).
//
// A thread walks the rings of a column, so the radial temperature difference
// of a ring is formed once; |grad T|^2 (TemperatureGradient, :609-653) is
// (R^2 + P^2) / 4, R = dT/dr at the two faces added, P the difference across the
// two azimuthal neighbours over the cell width.  The flux limiter
// (FluxLimiterValue, :684-698) of s = 4 |grad T| / (rho kappa T) needs only s^2
// below s = 2, where it is 2 / (3 + sqrt(9 + 10 s^2)); both forms give 1/5 at
// s = 2.  The diffusion coefficient's division and the limiter's are one.
// FP64-bound: 79 FP64 instructions a cell with the Bell & Lin opacity, 120
// before; 512x1536: 182 -> 136 us, with the minimum over the blocks.
// Rings per block: chunks of at most 8, as the inner, hotter rings take the
// longer opacity branches and short chunks spread them (512x1536: 133 / 138 / 157
// us with 3 / 6 / 11 rings; 1024x3072: 486 / 500 / 543 us with 8 / 16 / 21).
#define DC_MAXRINGS 8

struct DcRing { double c1, inv, invp, invdx, deltar2; };

template <int LAW>
__global__ void __launch_bounds__(BX) k_diffcoef(DevGrid g, DiffusionIO io)
{
  pdl_wait();
  __shared__ DcRing ring[DC_MAXRINGS];
  __shared__ unsigned long long smax[BX / 32][DC_MAXRINGS];
  __shared__ bool last;
  const int ns = g.ns, nr = g.nr;
  const int i0 = blockIdx.y * io.rings, i1 = min(i0 + io.rings, nr);
  if ((int)threadIdx.x < i1 - i0) {
    const int i = i0 + threadIdx.x;
    DcRing &R = ring[threadIdx.x];
    R.c1 = div_fast(g.k.sqrt2pi_inv, g.r.OmegaInv[i] * g.k.sqrt_adiabind_inv);   // rho / H / sqrt(2 pi) = rho c1 / c_s
    R.inv = g.r.InvDiffRmed[i];
    R.invp = g.r.InvDiffRmed[i + 1];
    R.invdx = io.invdxtheta[i];
    R.deltar2 = io.deltar2[i];
  }
  __syncthreads();
  const int jt = blockIdx.x * BX + threadIdx.x;
  const bool in = jt < ns;
  const int j = in ? jt : ns - 1;
  const int jm = (j == 0) ? ns - 1 : j - 1, jp = (j == ns - 1) ? 0 : j + 1;
  const double sig2 = 2.0 * g.k.sigma_sb, sig32 = 32.0 * g.k.sigma_sb, drop = io.opacity_drop * 0.5;
  const double *T = io.T;
  // radial difference of ring i with the ring below, over their distance; the
  // edge rings adopt their neighbour's gradient
  double Tl = T[j + i0 * ns], below = 0.0, dtl = 1.0e38;
  if (i0 > 0) below = (Tl - T[j + (i0 - 1) * ns]) * ring[0].inv;
  for (int i = i0; i < i1; i++) {
    const DcRing &R = ring[i - i0];
    const int row = i * ns, l = j + row;
    const double Tn = (i + 1 < nr) ? T[l + ns] : 0.0;
    const double above = (i + 1 < nr) ? (Tn - Tl) * R.invp : 0.0;
    double gr, gp;
    if (i == 0 || i == nr - 1) {
      const int k = (i == 0) ? 1 : nr - 2, lk = j + k * ns;
      gr = (T[lk] - T[lk - ns]) * g.r.InvDiffRmed[k] + (T[lk + ns] - T[lk]) * g.r.InvDiffRmed[k + 1];
      gp = (T[jp + k * ns] - T[jm + k * ns]) * io.invdxtheta[k];
    } else {
      gr = above + below;
      gp = (T[jp + row] - T[jm + row]) * R.invdx;
    }
    const double G = __fma_rn(gr, gr, gp * gp);                // 4 |grad T|^2
    const double rho = io.rho[l];
    const double vd = div_fast(rho * R.c1, io.cs[l]);
    const double kap = (LAW == THORIN_OPA_CONST) ? io.parametric_cu
                                                 : opacity_law<LAW>(g.k, vd, Tl * g.k.t2si) * g.k.opa2cu;
    const double tau = drop * kap * rho;
    const double T3 = cube_rn(Tl);
    // Q- = 2 sigma T^3 / tau_eff, tau_eff = 3/8 tau + c + 1/(4 tau), as one quotient
    const double qm = div_fast(sig2 * T3 * tau, __fma_rn(__fma_rn(0.375, tau, io.taueff_c), tau, 0.25));
    // q = 1 / (rho_mid kappa T); s^2 = 16 |grad T|^2 q^2 = 4 G q^2
    const double q = div_fast(1.0, vd * kap * Tl);
    const double X = q * q * G;
    const double num = sig32 * T3 * (q * Tl);                  // 2 * 16 sigma T^3 / (rho_mid kappa)
    double D;
    if (__double_as_longlong(X) <= __double_as_longlong(1.0)) {      // s <= 2
      D = div_fast(num, 3.0 + sqrt_fast(__fma_rn(40.0, X, 9.0)));
    } else {
      const double s = 2.0 * sqrt_fast(X);
      D = div_fast(5.0 * num, 10.0 * s + 9.0 + sqrt_fast(81.0 + 180.0 * s));
    }
    if (in) {
      io.opacity[l] = kap;
      io.qminus[l] = qm;
      io.dcen[l] = D;
    }
    // DiffusionTimestep's min of deltar2 / D: deltar2 is a ring constant and
    // correctly rounded division is monotone, so for D > 0 the minimum of a
    // ring is deltar2 / max D; other D (which only a crashed state holds) are
    // divided cell by cell as the reference does (a D that is not a number
    // counts for nothing, and must not hide the ring's others)
    unsigned hi = (unsigned)__double2hiint(D), lo = (unsigned)__double2loint(D);
    if ((unsigned long long)__double_as_longlong(D) - 1ULL >= 0x7ff0000000000000ULL) {
      hi = lo = 0u;
      const double t = div_fast(R.deltar2, D);
      if (in && t < dtl) dtl = t;
    }
    const unsigned mh = __reduce_max_sync(TH_FULL, hi);
    const unsigned ml = __reduce_max_sync(TH_FULL, hi == mh ? lo : 0u);
    if ((threadIdx.x & 31) == 0) smax[threadIdx.x >> 5][i - i0] = ((unsigned long long)mh << 32) | ml;
    Tl = Tn;
    below = above;
  }
  __syncthreads();
  const int b = blockIdx.x + blockIdx.y * gridDim.x, nb = gridDim.x * gridDim.y;
  if ((int)threadIdx.x < i1 - i0) {
    unsigned long long m = 0ULL;
#pragma unroll
    for (int w = 0; w < BX / 32; w++) m = max(m, smax[w][threadIdx.x]);
    const double dm = __longlong_as_double((long long)m);
    if (dm > 0.0) {
      const double t = div_fast(ring[threadIdx.x].deltar2, dm);
      if (t < dtl) dtl = t;
    }
  }
  const double m = block_reduce_smem<BX>(dtl, OpMin());
  if (threadIdx.x == 0) {
    io.part[b] = m;
    __threadfence();
    last = (atomicAdd(io.ticket, 1u) == (unsigned)nb - 1u);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double t = 1.0e38;
  for (int k = threadIdx.x; k < nb; k += BX) {
    const double v = __ldcg(io.part + k);
    t = (v < t) ? v : t;
  }
  t = block_reduce_smem<BX>(t, OpMin());
  if (threadIdx.x == 0) {
    *io.dtmin = t;
    *io.ticket = 0u;
  }
}

// Stellar irradiation: CalculateFlaring + CalculateQirr
// (EnergySources.c:103-198).  The flaring sin(atan a - atan b) is
// (a - b) / sqrt((1 + a^2)(1 + b^2)), and the flux over the effective optical depth
// 3/8 tau + c + 1 / (4 tau) one quotient: 38 FP64 instructions a cell, 113 with
// the angles; 384x1152: 99 -> 36 us.
__global__ void k_irradiation(DevGrid g, const double *__restrict__ rho, const double *__restrict__ cs,
                              const double *__restrict__ opacity, double *__restrict__ flaring, double *__restrict__ qirr,
                              double rstar, double tirr4fac, double opacity_drop, double taueff_c,
                              const double *__restrict__ rinf15, const double *__restrict__ rsup15)
{
  pdl_wait();
  const int ns = g.ns, nr = g.nr;
  CELL_LOOP_2D
  const double sqi = g.k.sqrt_adiabind_inv;
  // flaring at (i, j): interior rings use their own derivative, rings 0 and
  // nr-1 adopt the derivative of rings 1 and nr-2.
  int ic = (i == 0) ? 1 : (i == nr - 1 ? nr - 2 : i);
  if (nr >= 3) {
    const int lc = j + ic * ns;
    const double csin = 0.5 * (cs[lc] + cs[lc - ns]);
    const double csout = 0.5 * (cs[lc] + cs[lc + ns]);
    const double Hin = csin * rinf15[ic] * sqi;
    const double Hout = csout * rsup15[ic] * sqi;
    const double a = (Hout - Hin) * g.r.InvDiffRsup[ic];
    const double H = cs[l] * g.r.OmegaInv[i] * sqi;
    const double b = (i == ic) ? (H - 0.4 * rstar) * g.r.InvRmed[i] : div_fast(H - 0.4 * rstar, g.r.Rmed[i]);
    double f = 0.0, q = 0.0;
    if (a - b >= 0.0) f = div_fast(a - b, sqrt_fast(__fma_rn(a, a, 1.0) * __fma_rn(b, b, 1.0)));
    flaring[l] = f;
    if (f > 0.0) {
      const double tau = opacity_drop * 0.5 * opacity[l] * rho[l];
      const double den = __fma_rn(__fma_rn(0.375, tau, taueff_c), tau, 0.25);     // tau_eff tau
      q = div_fast(2.0 * g.k.sigma_sb * tirr4fac * f * tau, g.r.Rmed2[i] * den);
    }
    qirr[l] = q;
  }
}

// ---------------------------------------------------------------------------
// Red-black SOR (SuccessiveOverrelaxation, EnergySources.c:406-511).
// Rings 1 .. nr-2 are updated; pass 1 visits j = (i-1) mod 2, 1 + ..., pass 2
// the other colour (jchess1st = 0, jchess2nd = 1 on one rank, :431-432).
// Per-block partial L1 residual sums and "changed" counts go to scratch; the
// last block of pass 2 (ticketed with an atomic counter, no waiting) sums
// both passes in a fixed order and evaluates the three exit tests.

__device__ __forceinline__ double sor_resid_at(const double *T, const double *ml, const double *mlip,
                                               const double *mlim, const double *mljp, const double *mljm,
                                               const double *rhs, int l, int lip, int lim, int ljp, int ljm, size_t q)
{
  // the reference's sum T ml + T_ip mlip + T_im mlim + T_jp mljp + T_jm mljm - rhs as a chain of five FMAs
  double r = __fma_rn(T[l], ml[q], -rhs[q]);
  r = __fma_rn(T[lip], mlip[q], r);
  r = __fma_rn(T[lim], mlim[q], r);
  r = __fma_rn(T[ljp], mljp[q], r);
  return __fma_rn(T[ljm], mljm[q], r);
}

#define SOR_CPT 4        // cells per thread of the start residual
#define SOR_BX 128       // and its threads per block
#define SOR_PX 256       // threads per block of a colour pass
#define SOR_POCC 4       // and resident blocks per multiprocessor

// Block sums of the pass's L1 residual and "changed" count, result in
// thread 0.  The FP64 pipe bounds the SOR pass, so the first level goes
// through shared memory: warp 0 adds the SOR_PX / 32 values of its lane's
// column, then one shuffle tree finishes.  That is SOR_PX / 32 + 4 warp-wide
// FP64 adds per block instead of 5 (SOR_PX / 32 + 1).  Fixed order.
__device__ __forceinline__ void sor_block_sums(double &a, int &c)
{
  __shared__ double sa[SOR_PX];
  __shared__ int sc[SOR_PX];
  sa[threadIdx.x] = a;
  sc[threadIdx.x] = c;
  __syncthreads();
  if (threadIdx.x < 32) {
    double s = sa[threadIdx.x];
    int t = sc[threadIdx.x];
#pragma unroll
    for (int k = 1; k < SOR_PX / 32; k++) {
      s += sa[threadIdx.x + 32 * k];
      t += sc[threadIdx.x + 32 * k];
    }
    a = warp_reduce(s, OpAdd());
    c = warp_reduce(t, OpAddI());
  }
}

// Sum of the block partials by the block holding the last ticket; every
// block adds its partial first (no block ever waits on another).
__device__ __forceinline__ bool sor_last_block(unsigned int *ticket, unsigned nb)
{
  __shared__ bool last;
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned t = atomicAdd(ticket, 1u);
    last = (t == nb - 1);
  }
  __syncthreads();
  return last;
}

// The start residual's sums over the grid (the L1 norm and the warm start's
// input scale) by the last block, which also resets the solve's counters.
__device__ __forceinline__ void sor_resid_sums(const SorCtl &c, double a, double aj)
{
  a = block_reduce(a, OpAdd(), 0.0);
  aj = block_reduce(aj, OpAdd(), 0.0);
  const unsigned nb = gridDim.x * gridDim.y;
  const int b = blockIdx.x + blockIdx.y * gridDim.x;
  if (threadIdx.x == 0) {
    c.part[b] = a;
    c.part[nb + b] = aj;
  }
  if (sor_last_block(c.ticket, nb)) {
    __threadfence();
    double s = 0.0, sj = 0.0;
    for (unsigned k = threadIdx.x; k < nb; k += blockDim.x) {
      s += __ldcg(c.part + k);                     // L2, past L1
      sj += __ldcg(c.part + nb + k);
    }
    s = block_reduce(s, OpAdd(), 0.0);
    sj = block_reduce(sj, OpAdd(), 0.0);
    if (threadIdx.x == 0) {
      *c.jscale = sj;
      *c.normres0 = s;
      *c.done = 0;
      *c.niter = 0;
      *c.ticket = 0u;
      *c.epoch += 1ULL;
      *c.abort = 0;
    }
  }
}

__global__ void __launch_bounds__(SOR_BX) k_sor_resid0(DevGrid g, const double *__restrict__ T,
                                                    const double *__restrict__ ml, const double *__restrict__ mlip,
                                                    const double *__restrict__ mlim, const double *__restrict__ mljp,
                                                    const double *__restrict__ mljm, const double *__restrict__ rhs,
                                                    double *__restrict__ cw, SorCtl c)
{
  pdl_wait();
  const double omega = g.ctl[CTL_SOR_OMEGA];
  const int ns = g.ns, half = ns >> 1;
  const int i = blockIdx.y + 1;
  double a = 0.0, aj = 0.0;
  for (int m = 0; m < SOR_CPT; m++) {
    const int j = blockIdx.x * blockDim.x * SOR_CPT + m * blockDim.x + threadIdx.x;
    if (j < ns) {
      const int l = j + i * ns;
      const int ljp = (j == ns - 1) ? i * ns : l + 1;
      const int ljm = (j == 0) ? i * ns + ns - 1 : l - 1;
      const size_t q = sor_pidx(i, j, half);
      const double r = abs_i(sor_resid_at(T, ml, mlip, mlim, mljp, mljm, rhs, l, l + ns, l - ns, ljp, ljm, q));
      const double w = div_fast(omega, ml[q]);     // the sweeps' update is resid * omega / ml
      cw[q] = w;
      a += r;
      aj += r * w;                                 // omega |resid / Ml|: the warm start's input scale
    }
  }
  sor_resid_sums(c, a, aj);
}

// Matrix of the linearised implicit energy equation
// (ImplicitRadiativeDiffusion, EnergySources.c:256-297) and, with RESID, the
// start of the SOR solve at the omega of the control block (what
// k_sor_resid0 does for a system that is already in memory): omega/Ml and the
// L1 residual of the start temperature.
//
// A thread walks the rings of a column: the radial face coefficient of a ring's
// outer face is the next ring's inner one, and the azimuthal one of a cell's
// right face comes from the neighbouring thread through shared memory (the
// last thread of a block forms it).  The diagonal is 1 + the heating terms
// minus the four neighbour coefficients.  FP64-bound: 40 FP64 instructions a
// cell with the start residual, 60 in the two kernels before; 512x1536: 107 -> 74
// us.
#define MX_MAXRINGS 24

struct MxRing { double ca, cb, ch; };

template <bool RESID>
__global__ void __launch_bounds__(BX) k_matrix(DevGrid g, MatrixIO io, SorCtl c)
{
  pdl_wait();
  __shared__ MxRing ring[MX_MAXRINGS + 1];
  __shared__ double sB[2][BX];
  const double dt = g.ctl[CTL_DT], omega = RESID ? g.ctl[CTL_SOR_OMEGA] : 0.0;
  const int ns = g.ns, half = ns >> 1;
  const int i0 = 1 + blockIdx.y * io.rings, i1 = min(i0 + io.rings, g.nr - 1);     // rings 1 .. nr-2
  if ((int)threadIdx.x <= i1 - i0) {
    const int i = i0 + threadIdx.x;
    MxRing &R = ring[threadIdx.x];
    const double hc = g.r.OmegaInv[i] * g.k.sqrt_adiabind_inv;                     // H = c_s hc
    R.ca = 0.5 * g.r.Rinf[i] * g.r.InvDiffRmed[i];
    R.cb = io.invdxtheta2[i] * hc;
    R.ch = 2.0 * g.r.InvDiffRsup[i] * g.r.InvRmed[i] * hc;
  }
  __syncthreads();
  const int jt = blockIdx.x * BX + threadIdx.x;
  const bool in = jt < ns;
  const int j = in ? jt : ns - 1;
  const int jm = (j == 0) ? ns - 1 : j - 1, jp = (j == ns - 1) ? 0 : j + 1;
  const bool edge = threadIdx.x == BX - 1 || j == ns - 1;       // the right neighbour is in another block
  const double dtc = div_fast(dt, g.k.cv), dtg = dt * io.gm1;
  const double *T = io.T;
  double D = io.dcen[j + i0 * ns];
  double A = (D + io.dcen[j + (i0 - 1) * ns]) * ring[0].ca;     // inner face of ring i
  double Tm = 0.0, Tl = T[j + i0 * ns], a = 0.0, aj = 0.0;
  if (RESID) Tm = T[j + (i0 - 1) * ns];
  for (int i = i0; i < i1; i++) {
    const MxRing &R = ring[i - i0];
    const int row = i * ns, l = j + row;
    const double cs = io.cs[l];
    const double B = (D + io.dcen[jm + row]) * (cs * R.cb);     // left face
    double *s = sB[i & 1];
    s[threadIdx.x] = B;
    __syncthreads();
    const double Bp = edge ? (io.dcen[jp + row] + D) * (io.cs[jp + row] * R.cb) : s[threadIdx.x + 1];
    const double Dn = io.dcen[l + ns];
    const double Ap = (Dn + D) * ring[i - i0 + 1].ca;           // outer face
    const double bfac = div_fast(dtc, io.rho[l]);
    const double afac = bfac * (cs * R.ch);
    const double bq = bfac * io.qminus[l];
    const double mip = -(afac * Ap), mim = -(afac * A), mjp = -(bfac * Bp), mjm = -(bfac * B);
    const double diag = __fma_rn(4.0, bq, __fma_rn(io.divv[l], dtg, 1.0)) - (mip + mim) - (mjp + mjm);
    double r = __fma_rn(3.0 * bq, Tl, __fma_rn(bfac, io.qplus[l], Tl));
    if (io.qirr) r = __fma_rn(bfac, io.qirr[l], r);
    for (int k = 0; k < io.nheat; k++)
      if (l == io.heat_idx[k]) r = __fma_rn(bfac, io.heat_val[k], r);
    const double Tn = T[l + ns];
    if (in) {
      const size_t q = sor_pidx(i, j, half);
      io.ml[q] = diag;
      io.mlip[q] = mip;
      io.mlim[q] = mim;
      io.mljp[q] = mjp;
      io.mljm[q] = mjm;
      io.rhs[q] = r;
      if (RESID) {
        double e = __fma_rn(Tl, diag, -r);
        e = __fma_rn(Tn, mip, e);
        e = __fma_rn(Tm, mim, e);
        e = __fma_rn(T[jp + row], mjp, e);
        e = __fma_rn(T[jm + row], mjm, e);
        e = abs_i(e);
        const double w = div_fast(omega, diag);
        io.cw[q] = w;
        a += e;
        aj = __fma_rn(e, w, aj);
      }
    }
    D = Dn; A = Ap; Tm = Tl; Tl = Tn;
  }
  if (RESID) sor_resid_sums(c, a, aj);
}

// One colour pass of a sweep.  Each cell costs seven FP64 instructions: the
// residual as five FMAs, its absolute value added to the L1 norm, and the
// update T - resid * (omega/Ml) as one FMA (omega/Ml prepared once per solve
// by k_matrix, or k_sor_resid0); the change test delta > T*SORPRECISION runs
// on the integer pipe (sor_changed).  That is 22 us of the FP64 pipe for a pass of the
// 1024x3072 disk, 17 us of DRAM traffic (seven coefficient arrays and T, 118
// MB), and the latency of a pass's start and end, so:
// * one wave of blocks strides over the colour's cells, 10 a thread on that
//   disk, and a cell's coefficients are loaded while the cell before it is
//   computed (with 1024 threads per multiprocessor and 64 registers a thread;
//   more threads without the prefetch were slower);
// * a pass's blocks start while the pass before drains (programmatic
//   dependent launch) and load their first coefficients, which no pass
//   writes, before they wait for it;
// * the last block sums the block partials in one level.
// 1024x3072: 25.6 us a pass (29.2 us with one cell in flight per thread, full
// launches and a two-level sum; prefetch and launch give 1.5 us each), 512x1536
// 13.2 -> 10.7 us, 128x384 7.6 -> 5.4 us.  Blocks of 512 x 2: 25.7 / 10.7 / 6.0 us,
// 512 x 3 without prefetch 27.3 / 11.3 / 6.4 us, prefetching T too 25.8 us.
// The sweep number is counted on the device (c.niter), so every sweep is the
// same two launches: the body of the sweep loop's WHILE graph node.
// delta > tn * SORPRECISION (SORPRECISION = 1e-15, between 2^-50 and 2^-49)
// with delta = resid * cw, cw = omega / Ml > 0.  When resid, cw and tn are
// positive normal numbers well inside the exponent range, delta lies in
// [2^(a+b), 2^(a+b+2)] for the exponents a, b of resid and cw, so the
// exponents decide the test on the integer pipe unless a + b - t is within
// -51..-49; those cases, and all unusual operands, take the exact sign test.
__device__ __forceinline__ bool sor_changed(double resid, double cw, double tn)
{
  const long long r64 = __double_as_longlong(resid), c64 = __double_as_longlong(cw), t64 = __double_as_longlong(tn);
  const int er = (int)(r64 >> 52), ec = (int)(c64 >> 52), et = (int)(t64 >> 52);
  if (t64 > 0LL && et >= 100 && et < 0x7FF && c64 > 0LL && ec != 0 && ec < 0x7FF) {
    if (r64 <= 0LL) return false;                      // resid <= +0: delta <= 0 < threshold
    if (er != 0 && er != 0x7FF && er + ec - 1023 >= 100 && er + ec - 1023 < 0x7FF - 100) {
      const int diff = er + ec - 1023 - et;
      if (diff >= -48) return true;
      if (diff <= -52) return false;
    }
  }
  return __double_as_longlong(__fma_rn(-tn, TH_SORPRECISION, resid * cw)) > 0LL;
}

struct SorRow { double ml, mlip, mlim, mljp, mljm, rhs, cw; };

__global__ void __launch_bounds__(SOR_PX, SOR_POCC)
k_sor_pass(DevGrid g, double *__restrict__ T, const double *__restrict__ ml, const double *__restrict__ mlip,
           const double *__restrict__ mlim, const double *__restrict__ mljp, const double *__restrict__ mljm,
           const double *__restrict__ rhs, const double *__restrict__ cw, SorCtl c, double eps, int pass, int maxiters)
{
  const int ns = g.ns, half = ns >> 1;
  const int col = pass - 1;
  const int total = half * (g.nr - 2);             // cell idx: ring idx / half + 1, k = idx % half of this colour
  const int stride = gridDim.x * SOR_PX;
  int idx = blockIdx.x * SOR_PX + threadIdx.x;
  int r = idx / half, k = idx - r * half;
  const int dr = stride / half, dk = stride - dr * half;
  auto row_of = [&](int r, int k) {
    const size_t q = (size_t)(((r + 1) << 1) + col) * half + k;
    return SorRow{ml[q], mlip[q], mlim[q], mljp[q], mljm[q], rhs[q], cw[q]};
  };
  SorRow m;
  if (idx < total) m = row_of(r, k);
  // what a block does before this must not touch anything the pass before writes
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (*((volatile int *)c.done)) return;
  double a = 0.0;
  int ch = 0;
  while (idx < total) {
    const int j = 2 * k + ((r + col) & 1);
    const int row = (r + 1) * ns, l = row + j;
    const int ljp = (j == ns - 1) ? row : l + 1;
    const int ljm = (j == 0) ? row + ns - 1 : l - 1;
    const double t = T[l], tip = T[l + ns], tim = T[l - ns], tjp = T[ljp], tjm = T[ljm];
    idx += stride;
    r += dr;
    k += dk;
    if (k >= half) { k -= half; r++; }
    SorRow n;
    if (idx < total) n = row_of(r, k);
    // the reference's sum T ml + T_ip mlip + T_im mlim + T_jp mljp + T_jm mljm - rhs
    double resid = __fma_rn(t, m.ml, -m.rhs);
    resid = __fma_rn(tip, m.mlip, resid);
    resid = __fma_rn(tim, m.mlim, resid);
    resid = __fma_rn(tjp, m.mljp, resid);
    resid = __fma_rn(tjm, m.mljm, resid);
    a += abs_i(resid);
    const double tn = __fma_rn(-resid, m.cw, t);     // T -= omega resid / Ml
    T[l] = tn;
    ch += sor_changed(resid, m.cw, tn) ? 1 : 0;
    m = n;
  }
  sor_block_sums(a, ch);
  const unsigned nb = gridDim.x;
  const int b = blockIdx.x;
  if (threadIdx.x == 0) {
    c.part[col * nb + b] = a;
    c.ipart[col * nb + b] = ch;
  }
  if (pass != 2) return;
  // The last block to finish sums both colours' partials in block order and
  // applies the exit tests.
  if (!sor_last_block(c.ticket, nb)) return;
  __threadfence();
  double s = 0.0;
  int cs = 0;
  for (unsigned q = threadIdx.x; q < 2 * nb; q += SOR_PX) {
    s += __ldcg(c.part + q);
    cs += __ldcg(c.ipart + q);
  }
  s = block_reduce(s, OpAdd(), 0.0);
  cs = block_reduce(cs, OpAddI(), 0);
  if (threadIdx.x == 0) {
    const double r0 = *c.normres0;
    const int n = __ldcg(c.niter) + 1;             // this sweep's number (the start residual set 0)
    *c.normres = s;
    *c.changed = cs;
    *c.niter = n;
    const int dn = (s < eps * r0 || s < TH_SORMIN || cs == 0) ? 1 : (n >= maxiters ? 2 : 0);
    if (dn) *c.done = dn;
    *c.ticket = 0u;
    // the sweep loop of the graph ends with the first sweep that sets done;
    // n >= maxiters always does, so the loop is finite
    if (c.has_cond) cudaGraphSetConditional(c.cond, dn == 0 ? 1u : 0u);
  }
}

// The whole solve in one cooperative launch, one block per multiprocessor.  A
// pass as a launch of its own has 0.1 to 10 us of FP64 work on disks of up to
// 700 x 2100 and takes 5.3 us (96x288) to 15 (700x2100); the rest is launch,
// load latency and completion.  Here a block keeps its cells from sweep to
// sweep (consecutive column pairs of one red and one black cell; temperatures
// and, as far as they fit, coefficients in shared memory, the others streamed
// from L2), and a cell whose neighbour belongs to another block waits for
// that neighbour's value alone: every update goes to x as one 16-byte store of
// the value and a tag (number of the solve, number of the sweep), which a
// relaxed 16-byte load sees whole, so there is no barrier across the grid, no
// fence and no flag.  No slot is written too early: a cell's next value needs
// what every neighbour computed from this one.
// The exit test runs beside the next sweep: a warp of its own in each block
// sums the threads' |resid| of a sweep (in a fixed order, as all sums here),
// that of block 0 adds the blocks' records and posts the verdict, which the
// blocks take up at the end of the next sweep; the result is the sweep before,
// still in the other of x's two buffers.  So a solve runs one sweep more than
// it needs.  The updates are the passes' own, bit for bit.
// All blocks are resident together (cooperative launch); each wait has a
// limit, after which its block ends the solve for all (*abort) and the caller
// reports that, also when the verdict was out already: such a block has not
// written its temperatures.
// us a pass, launches / here: 24x72 6.2 / 2.25, 128x384 5.7 / 1.9, 256x768 6.8 /
// 2.5, 333x1002 8.0 / 3.3, 384x1152 8.6 / 3.9, 512x1536 10.8 / 6.0, 640x1920 12.9 /
// 9.1, 700x2100 15.2 / 11.1, 850x2550 19.3 / 18.9, 1024x3072 25.8 / 28.2: there the
// coefficients no longer fit in L2 beside x, so SOR_GRID_CELLS lies between the
// last two.  Coefficients all streamed: 192x576 2.8 (2.1 in shared memory),
// 333x1002 3.4, 640x1920 9.7.
#define SOR_GRID_CELLS 2400000        // largest disk (cells of rings 1 .. nr-2)

__device__ __forceinline__ void x_load(const ulonglong2 *p, unsigned long long &v, unsigned long long &tag)
{
  asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
               : "=l"(v), "=l"(tag) : "l"(p) : "memory");
}

__device__ __forceinline__ void x_store(ulonglong2 *p, unsigned long long v, unsigned long long tag)
{
  asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}"
               ::"l"(p), "l"(v), "l"(tag) : "memory");
}

// Loads until the tag (shifted right) is there; false when the wait ran out,
// here or in another block.  FEW: a limit of `spin` loads, for the test of this;
// as a comparison of every load it costs 128x384 2.34 -> 2.44 us a pass, so the
// usual limit is looked at once in 1024.
template <bool FEW>
__device__ __forceinline__ bool x_wait(const ulonglong2 *p, unsigned long long want, int shift, int spin, int *abort,
                                       unsigned long long &v, unsigned long long &tag)
{
  for (int n = 1; (tag >> shift) != want; n++) {
    if (FEW ? n >= spin : (n & 1023) == 0 && (n >= SOR_GRID_SPIN || *(volatile int *)abort)) {
      *(volatile int *)abort = 1;
      return false;
    }
    x_load(p, v, tag);
  }
  return true;
}

struct SorSystem { const double *ml, *mlip, *mlim, *mljp, *mljm, *rhs, *cw; };

template <bool FEW>
__global__ void __maxnreg__(64) k_sor_grid(DevGrid g, double *T, SorSystem m, SorCtl c, ulonglong2 *x, double eps,
                                           int maxiters, int R, int res, int spin)
{
  extern __shared__ double sm[];
  __shared__ int sdec[2];
  const int ns = g.ns, half = ns >> 1, nr = g.nr, np = half * (nr - 2);
  const int nb = gridDim.x, b = blockIdx.x, nt = blockDim.x - 32, tid = threadIdx.x;
  const int g0 = (int)((long long)np * b / nb), P = (int)((long long)np * (b + 1) / nb) - g0;
  const int Pm = (np + nb - 1) / nb;
  double *sT = sm, *sA = sT + 2 * Pm, *sco = sA + 2 * nt;
  int *sC = (int *)(sco + 14 * res), *sJ = sC + 2 * nt;
  ulonglong2 *rec = x + 4 * (size_t)np, *verdict = rec + nb;
  if (*(volatile int *)c.done) return;             // the same for all blocks: set at the end of a solve only
  const unsigned long long ep = *(volatile unsigned long long *)c.epoch << 24;   // tag: solve, sweep
  if (tid < 2) sdec[tid] = 0;

  if (tid >= nt) {                                 // the exit test's warp
    const int lane = tid - nt;
    const double r0 = *c.normres0;
    __syncthreads();
    bool dead = false;
    for (int n = 1;; n++) {
      if (__syncthreads_or(dead)) return;          // end of sweep n
      if (n > 1 && sdec[(n - 1) & 1]) return;
      double s = 0.0;
      int ch = 0;
      for (int t = lane; t < nt; t += 32) {
        s += sA[(n & 1) * nt + t];
        ch += sC[(n & 1) * nt + t];
      }
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(TH_FULL, s, o);
      ch = __reduce_add_sync(TH_FULL, ch);
      if (lane == 0)
        x_store(rec + b, (unsigned long long)__double_as_longlong(s), ((ep | (unsigned)n) << 13) | (unsigned)min(ch, 8191));
      const unsigned long long want = ((ep | (unsigned)n) << 13) >> 13;
      unsigned long long v, tag = ~want << 13;
      int dec = 0;
      if (b == 0) {
        s = 0.0;
        ch = 0;
        for (int k = lane; k < nb; k += 32) {
          tag = ~want << 13;
          if (!x_wait<FEW>(rec + k, want, 13, spin, c.abort, v, tag)) { dead = true; break; }
          s += __longlong_as_double((long long)v);
          ch += (int)(tag & 8191u);
        }
        dead = __any_sync(TH_FULL, dead);
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(TH_FULL, s, o);
        ch = __reduce_add_sync(TH_FULL, ch);
        if (dead) continue;
        dec = (s < eps * r0 || s < TH_SORMIN || ch == 0) ? 1 : (n >= maxiters ? 2 : 0);
        if (lane == 0) {
          if (dec) {
            *c.normres = s;
            *c.changed = ch;
            *c.niter = n;
            *c.done = dec;
          }
          x_store(verdict, (unsigned long long)dec, ep | (unsigned)n);
        }
      } else {
        tag = ~(ep | (unsigned)n);
        if (lane == 0) dead = !x_wait<FEW>(verdict, ep | (unsigned)n, 0, spin, c.abort, v, tag);
        dead = __any_sync(TH_FULL, dead);
        dec = dead ? 0 : (int)__shfl_sync(TH_FULL, (unsigned)v, 0);
      }
      if (lane == 0) sdec[n & 1] = dec;
    }
  }

  // Row q of the thread is the block's pair p = q nt + tid; sJ: 2 k of its ring
  // plus the ring's parity, so that colour c sits in column sJ ^ c.  x: two
  // buffers (sweep & 1) of the red and the black cells.
  for (int q = 0; q < R; q++) {
    const int p = q * nt + tid;
    if (p >= P) break;
    const int gg = g0 + p, r = gg / half, k = gg - r * half, j = 2 * k + (r & 1);
    sJ[p] = j;
    double t = 0.0;
    for (int col = 0; col < 2; col++) {
      t = T[(size_t)(r + 1) * ns + (j ^ col)];
      sT[col * Pm + p] = t;
      if (p < res) {
        const size_t e = (size_t)2 * (gg + half) - k + col * half;             // sor_pidx
        double *w = sco + col * 7 * res + p;
        w[0] = m.ml[e]; w[res] = m.mlip[e]; w[2 * res] = m.mlim[e]; w[3 * res] = m.mljp[e];
        w[4 * res] = m.mljm[e]; w[5 * res] = m.rhs[e]; w[6 * res] = m.cw[e];
      }
    }
    x_store(x + np + gg, (unsigned long long)__double_as_longlong(t), ep);      // the black cells before sweep 1
  }
  __syncthreads();
  bool dead = false;
  int dec = 0, n = 0;
  while (!dec) {
    n++;
    double a = 0.0;
    int ch = 0;
    for (int col = 0; col < 2; col++) {
      const int nw = n - 1 + col;                  // sweep of the neighbours' values
      const unsigned long long want = ep | (unsigned)nw;
      const ulonglong2 *xo = x + (size_t)(2 * (nw & 1) + 1 - col) * np + g0;    // by pair of the block
      ulonglong2 *xn = x + (size_t)(2 * (n & 1) + col) * np + g0;
      const double *so = sT + (1 - col) * Pm;
      // the rows at the block's ends first: their values are what the other
      // blocks wait for, and the rows between cover the way there
      for (int z = 0; z < R; z++) {
        const int q = (z & 1) ? R - 1 - (z >> 1) : (z >> 1), p = q * nt + tid;
        if (p >= P) continue;
        const int jr = sJ[p], k = jr >> 1;
        const bool odd = (jr ^ col) & 1;
        // the neighbour on the side away from the other cell of the pair
        const int sd = odd ? (k == half - 1 ? p - half + 1 : p + 1) : (k == 0 ? p + half - 1 : p - 1);
        const bool xup = p + half >= P && g0 + p + half < np, xdn = p < half && g0 + p >= half;
        const bool xsd = (unsigned)sd >= (unsigned)P;
        unsigned long long v0, v1, v2, t0, t1, t2;
        if (xup) x_load(xo + p + half, v0, t0);
        if (xdn) x_load(xo + p - half, v1, t1);
        if (xsd) x_load(xo + sd, v2, t2);
        SorRow w;
        if (p < res) {
          const double *s = sco + col * 7 * res + p;
          w = SorRow{s[0], s[res], s[2 * res], s[3 * res], s[4 * res], s[5 * res], s[6 * res]};
        } else {
          const size_t e = (size_t)2 * (g0 + p + half) - k + col * half;
          w = SorRow{m.ml[e], m.mlip[e], m.mlim[e], m.mljp[e], m.mljm[e], m.rhs[e], m.cw[e]};
        }
        const double own = so[p], tc = sT[col * Pm + p];
        double tip, tim, ts;
        if (xup) {
          if (!x_wait<FEW>(xo + p + half, want, 0, spin, c.abort, v0, t0)) dead = true;
          tip = __longlong_as_double((long long)v0);
        } else tip = (p + half < P) ? so[p + half] : T[(size_t)(nr - 1) * ns + (jr ^ col)];
        if (xdn) {
          if (!x_wait<FEW>(xo + p - half, want, 0, spin, c.abort, v1, t1)) dead = true;
          tim = __longlong_as_double((long long)v1);
        } else tim = (p >= half) ? so[p - half] : T[jr ^ col];
        if (xsd) {
          if (!x_wait<FEW>(xo + sd, want, 0, spin, c.abort, v2, t2)) dead = true;
          ts = __longlong_as_double((long long)v2);
        } else ts = so[sd];
        double resid = __fma_rn(tc, w.ml, -w.rhs);
        resid = __fma_rn(tip, w.mlip, resid);
        resid = __fma_rn(tim, w.mlim, resid);
        resid = __fma_rn(odd ? ts : own, w.mljp, resid);
        resid = __fma_rn(odd ? own : ts, w.mljm, resid);
        a += abs_i(resid);
        const double tn = __fma_rn(-resid, w.cw, tc);
        x_store(xn + p, (unsigned long long)__double_as_longlong(tn), ep | (unsigned)n);
        sT[col * Pm + p] = tn;
        ch += sor_changed(resid, w.cw, tn) ? 1 : 0;
      }
      if (col == 0) asm volatile("bar.sync 1, %0;" ::"r"(nt) : "memory");
    }
    sA[(n & 1) * nt + tid] = a;
    sC[(n & 1) * nt + tid] = ch;
    if (__syncthreads_or(dead)) return;
    if (n > 1) dec = sdec[(n - 1) & 1];
  }
  // the exit test passed on the sweep before this one
  for (int q = 0; q < R; q++) {
    const int p = q * nt + tid;
    if (p >= P) break;
    const int r = (g0 + p) / half;
    for (int col = 0; col < 2; col++) {
      const unsigned long long v = x[(size_t)(2 * ((n - 1) & 1) + col) * np + g0 + p].x;
      T[(size_t)(r + 1) * ns + (sJ[p] ^ col)] = __longlong_as_double((long long)v);
    }
  }
}

// After SOR: boundary rings adopt their neighbours' temperature and the
// energy is rebuilt, E = rho T c_v (EnergySources.c:319-334).  EFT_CPT cells a
// thread, their loads in flight together; 1024x3072: 28 -> 17 us (75 MB at copy
// speed: 11).
#define EFT_CPT 4
__global__ void k_energy_from_t(DevGrid g, const double *__restrict__ rho, double *T, double *__restrict__ enew)
{
  pdl_wait();
  const int ns = g.ns, nr = g.nr, i = blockIdx.y, j0 = blockIdx.x * (BX * EFT_CPT) + threadIdx.x;
  const int row = i * ns, from = (i == 0) ? row + ns : (i == nr - 1) ? row - ns : row;
  double t[EFT_CPT], r[EFT_CPT];
#pragma unroll
  for (int m = 0; m < EFT_CPT; m++) {
    const int j = j0 + m * BX;
    const bool in = j < ns && i < nr;
    t[m] = in ? T[from + j] : 0.0;
    r[m] = in ? rho[row + j] : 0.0;
  }
#pragma unroll
  for (int m = 0; m < EFT_CPT; m++) {
    const int j = j0 + m * BX;
    if (j >= ns) continue;
    if (from != row && i < nr) T[row + j] = t[m];
    enew[row + j] = (i < nr) ? r[m] * t[m] * g.k.cv : 0.0;
  }
}

// ---------------------------------------------------------------------------
// Transport (TransportEuler.c).  Radial step of one fluid in one kernel:
// ComputeLRMomenta and the quotients by the density (TransportEuler.c:
// 318-347), VanLeerRadial's slopes, ComputeStarRad's upwind face values
// (:232-273) and the flux divergence (:384-415).
//
// A thread walks a chunk of rings of one column and keeps the quotients,
// slopes and incoming fluxes of the current and the next ring in registers,
// so the state is read once and the updated quantities are written once (four
// kernels with about 70 field passes between them before this).  Like the
// other stencils it is bound by the FP64 pipe, so the arithmetic is arranged
// for few FP64 instructions (about 50 a cell for the gas, 41 for the pebbles):
// * the quotients Q / (Sigma + 1e-20) of the momenta Sigma v and
//   Sigma (v_theta + Omega r) r are the velocities times unit_quotient(Sigma),
//   which is exactly 1 in all but thin gas;
// * the slope of the quotients with ring spacings h,
//   2 (d- / h-)(d+ / h+) / (d- / h- + d+ / h+) = 2 d- d+ / (h- (rho d- + d+)),
//   rho = h+ / h-, comes from vl_slope without FP64; its 1 / h- goes into the
//   face coefficient, +/-rho - v dt / h-, one FMA;
// * each face's flux is formed once and shared by the two rings.
// Slopes are zero in rings 0 and nr-1, the faces 0 and nr carry no flux.
// Ring constants of the chunk are formed once per block in shared memory.
// 512x1536: 150 us (gas) and 125 us (pebbles) in the four kernels, 90 and 73 us
// here; 1024x3072: 335 and 270 us, 96% of the FP64 pipe's rate.
// Rings per block (chunk_rings): 1.3 rings per chunk are the slopes and the
// face that neighbouring chunks both form.  Measured for the gas: 256x768
// 37 / 39 / 51 us with 4 / 6 / 9 rings, 512x1536 105 / 95 / 90 / 103 us with 7 / 11 /
// 14 / 21, 1024x3072 355 / 335 / 366 / 350 us with 10 / 14 / 20 / 27.
#define RD_MAXRINGS 40

struct RadialIO {
  const double *rho, *vr, *vt, *energy, *label;
  double *out[6];           // the four momenta, the density, the energy
  double *ext;              // Sigma * label
  int rings;                // rings per block
};

struct RdRing { double rm, cu, rho, dtinv, isd, rinf; float wh, wl; };

// The ring's quotients: w[0..3] the momenta's, then energy, tracer.
template <bool E, bool X>
__device__ __forceinline__ void rd_load(const DevGrid &g, const RadialIO &io, const RdRing &c, int i, int j, int jp,
                                        double vr_i, double &vr_ip, double &r, double &wr, double *w)
{
  const int ns = g.ns, l = j + i * ns;
  r = io.rho[l];
  vr_ip = io.vr[l + ns];
  const double u = __fma_rn(io.vt[l], c.rm, c.cu), ujp = __fma_rn(io.vt[jp + i * ns], c.rm, c.cu);
  wr = unit_quotient(r);
  w[0] = vr_ip; w[1] = vr_i; w[2] = ujp; w[3] = u;
  double d = r;
  if (X) w[4 + E] = io.label[l];
  if (__double2hiint(wr) != 0x3ff00000) {          // thin gas
    w[0] *= wr; w[1] *= wr; w[2] *= wr; w[3] *= wr;
    if (X) w[4 + E] *= wr;
    d = r + 1e-20;
  }
  if (E) w[4] = div_fast(io.energy[l], d);
}

template <bool E, bool X>
__global__ void __launch_bounds__(BX, 4) k_radial(DevGrid g, RadialIO io)
{
  pdl_wait();
  constexpr int NW = 4 + E + X;
  __shared__ RdRing ring[RD_MAXRINGS + 4];
  const double dt = g.ctl[CTL_DT];
  const int ns = g.ns, nr = g.nr;
  const int i0 = blockIdx.y * io.rings;
  const int i1 = min(i0 + io.rings, nr);
  // ring constants of rings i0-2 .. i1+1 (entry 0 is ring i0-2)
  {
    const int i = i0 - 2 + (int)threadIdx.x;
    if (i >= 0 && i < nr && i <= i1 + 1) {
      RdRing &c = ring[threadIdx.x];
      c.rm = g.r.Rmed[i];
      c.cu = c.rm * g.ctl[CTL_OMEGA_FRAME] * c.rm;
      const double inv = g.r.InvDiffRmed[i];       // 0 in ring 0
      c.dtinv = dt * inv;
      c.rho = (i >= 1 && i < nr - 1) ? (g.r.Rmed[i + 1] - c.rm) * inv : 0.0;
      c.wh = (float)c.rho;
      c.wl = (float)(c.rho - (double)c.wh);
      c.isd = dt * g.k.dpns * g.r.InvSurf[i];
      c.rinf = g.r.Rinf[i];
    }
  }
  __syncthreads();
  const int j = blockIdx.x * BX + threadIdx.x;
  if (j >= ns) return;
  const int jp = (j == ns - 1) ? 0 : j + 1;
  const RdRing *R = ring + 2 - i0;                  // R[i]: ring i
  // cur: ring i, nxt: ring i+1; ds: differences between them
  double wc[NW], wn[NW], ds[NW], sc[NW], fin[NW + 1];
  double rc, rn, wrc, wrn, dr, srho = 0.0, vn, vf;
  int i;
#pragma unroll
  for (int k = 0; k < NW; k++) sc[k] = 0.0;
  if (i0 == 0) {
    i = 0;
    rd_load<E, X>(g, io, R[0], 0, j, jp, io.vr[j], vf, rc, wrc, wc);
  } else {
    // the face between rings i0-1 and i0 needs the slope of ring i0-1
    i = i0 - 1;
    double w0[NW], r0, wr0;
    if (i >= 1) {
      rd_load<E, X>(g, io, R[i - 1], i - 1, j, jp, io.vr[j + (i - 1) * ns], vf, r0, wr0, w0);
    } else {
      vf = io.vr[j + i * ns];
    }
    rd_load<E, X>(g, io, R[i], i, j, jp, vf, vf, rc, wrc, wc);
    if (i >= 1) {
#pragma unroll
      for (int k = 0; k < NW; k++) sc[k] = wc[k] - w0[k];
      srho = rc - r0;
    }
  }
  // vf: v_r at face i+1
  rd_load<E, X>(g, io, R[i + 1], i + 1, j, jp, vf, vn, rn, wrn, wn);
#pragma unroll
  for (int k = 0; k < NW; k++) ds[k] = wn[k] - wc[k];
  dr = rn - rc;
  if (i0 > 0 && i >= 1) {
    const RdRing &c = R[i];
#pragma unroll
    for (int k = 0; k < NW; k++) sc[k] = vl_slope_t<true>(sc[k], ds[k], c.wh, c.wl, c.rho);
    srho = vl_slope_t<true>(srho, dr, c.wh, c.wl, c.rho);
  }
#pragma unroll
  for (int k = 0; k <= NW; k++) fin[k] = 0.0;
  for (; i < i1; i++) {
    const int l = j + i * ns;
    double sn[NW], fout[NW + 1], sr = 0.0, w2[NW], r2 = 0.0, wr2 = 0.0, v2 = 0.0;
#pragma unroll
    for (int k = 0; k < NW; k++) sn[k] = 0.0;
    if (i + 2 < nr) {                               // ring i+2, and the slope of ring i+1
      rd_load<E, X>(g, io, R[i + 2], i + 2, j, jp, vn, v2, r2, wr2, w2);
      const RdRing &c = R[i + 1];
#pragma unroll
      for (int k = 0; k < NW; k++) {
        const double d2 = w2[k] - wn[k];
        sn[k] = vl_slope_t<true>(ds[k], d2, c.wh, c.wl, c.rho);
        ds[k] = d2;
      }
      const double d2 = r2 - rn;
      sr = vl_slope_t<true>(dr, d2, c.wh, c.wl, c.rho);
      dr = d2;
    }
    if (i + 1 < nr) {                               // the face between rings i and i+1
      const RdRing &a = R[i], &b = R[i + 1];
      const bool up = __double_as_longlong(vf) > 0LL;             // v > 0.0
      const double c = __fma_rn(-vf, up ? a.dtinv : b.dtinv, up ? a.rho : -b.rho);
      const double f = b.rinf * vf * __fma_rn(c, up ? srho : sr, up ? rc : rn);
#pragma unroll
      for (int k = 0; k < NW; k++) fout[k] = __fma_rn(c, up ? sc[k] : sn[k], up ? wc[k] : wn[k]) * f;
      const double wu = up ? wrc : wrn;
      fout[NW] = (__double2hiint(wu) == 0x3ff00000) ? f : wu * f;
    } else {
#pragma unroll
      for (int k = 0; k <= NW; k++) fout[k] = 0.0;
    }
    if (i >= i0) {
      const double isd = R[i].isd;
      const double q = rc + 1e-20;                  // momenta Sigma v = (Sigma + 1e-20) w
#pragma unroll
      for (int k = 0; k < 4; k++) io.out[k][l] = __fma_rn(fin[k] - fout[k], isd, q * wc[k]);
      if (E) io.out[5][l] = __fma_rn(fin[4] - fout[4], isd, io.energy[l]);
      if (X) io.ext[l] = __fma_rn(fin[4 + E] - fout[4 + E], isd, rc * io.label[l]);
      io.out[4][l] = __fma_rn(fin[NW] - fout[NW], isd, rc);
    }
#pragma unroll
    for (int k = 0; k < NW; k++) { wc[k] = wn[k]; wn[k] = w2[k]; sc[k] = sn[k]; fin[k] = fout[k]; }
    fin[NW] = fout[NW];
    rc = rn; rn = r2; wrc = wrn; wrn = wr2; srho = sr; vf = vn; vn = v2;
  }
}

// ComputeSpeQty (TransportEuler.c:197-215): the tracer back from rho*label.
__global__ void k_label_from_ext(DevGrid g, const double *__restrict__ rho, const double *__restrict__ ext,
                                 double *__restrict__ label)
{
  pdl_wait();
  const int ns = g.ns;
  CELL_LOOP_2D
  label[l] = div_fast(ext[l], rho[l]);
}

// Per-ring quantities of ComputeResiduals (TransportEuler.c:70-111): VMed,
// the ring mean of v_theta; the integer FARGO shift Nshift; the uniform
// residual velocity of the second pass.  One block per ring.  The mean is a
// fixed tree sum (ring_sum); when Ntilde + 1/2 lies within 1e-9 of an integer,
// the ring is summed again left to right, the reference's order, so that the
// integer shift is exactly the reference's.
__global__ void __launch_bounds__(RING_T) k_azi_rings(DevGrid g, const double *__restrict__ vt,
                                                      int *__restrict__ nshift, double *__restrict__ vmed,
                                                      double *__restrict__ vtemp)
{
  pdl_wait();
  const double dt = g.ctl[CTL_DT];
  const int i = blockIdx.x;
  const int ns = g.ns;
  const double *row = vt + (size_t)i * ns;
  double vm = ring_sum(row, ns);
  if (threadIdx.x >= 32) return;
  vm /= (double)ns;
  double Ntilde = vm * g.r.InvRmed[i] * dt * (double)ns / 2.0 / TH_PI;
  const double frac = Ntilde + 0.5 - floor(Ntilde + 0.5);
  if (frac < 1e-9 || frac > 1.0 - 1e-9) {
    vm = warp_seq_sum(row, ns) / (double)ns;
    Ntilde = vm * g.r.InvRmed[i] * dt * (double)ns / 2.0 / TH_PI;
  }
  if (threadIdx.x == 0) {
    const double Nround = floor(Ntilde + 0.5);
    const double invdt = 1.0 / dt, dpinvns = 2.0 * TH_PI / (double)ns;
    vmed[i] = vm;
    nshift[i] = (int)(long long)Nround;
    const double v = (Ntilde - Nround) * g.r.Rmed[i] * invdt * dpinvns;
    // of the uniform pass: v, the face coefficient and the flux's ring factor
    vtemp[3 * i] = v;
    vtemp[3 * i + 1] = __fma_rn(-v, dt * g.r.InvDxtheta[i], v > 0.0 ? 1.0 : -1.0);
    vtemp[3 * i + 2] = (g.r.Rsup[i] - g.r.Rinf[i]) * dt * v;
  }
}

// Azimuthal step of the transport (OneWindTheta, QuantitiesAdvection,
// VanLeerTheta, ComputeStarTheta, AdvectSHIFT; TransportEuler.c:70-175,
// 276-347).  A block takes a segment of AZ_S(T) = T - 2*AZ_HALO cells of one
// ring plus AZ_HALO cells on each side, one cell per thread, all transported
// quantities in registers.  Each pass (residual velocity, then the uniform
// one) leaves two fewer valid cells at each end, so after both passes the
// segment itself is exact and is written, cyclically shifted by Nshift, to
// the destination arrays.  Neighbour values move through shared memory.
// The van Leer slope's sign tests read the sign bits as integers: for finite
// values this is the reference's comparison (a NaN, which only a crashed run
// holds, gives NaN instead of a zero slope).  The arithmetic is regrouped to
// save FP64 instructions: Work = Q * (1 / (RhoInt + 1e-20)), the slope's
// 1/dxtheta folded into the face coefficient, the flux as Q* times
// (dxrad RhoStar v); results differ from the reference's grouping in the
// last bits only.  The FP64 pipe bounds it: six FP64 instructions per quantity
// and pass (the quotient, its difference, the face value, the flux and two for
// the update; the slopes run on the FP32 and integer pipes, vl_slope).
// The two passes are separate code: with the choice made per pass at run time
// both passes' FP64 instructions were issued under predicates.
// 1024x3072: 556 us with the gas's six quantities and 87 FP64 instructions a
// cell (588 us and 91 under predicates, 917 us and 151 with the slopes on the
// FP64 pipe).
#define AZ_HALO 4
#define AZ_TMAX 512

template <int NQ>
__global__ void __launch_bounds__(AZ_TMAX) k_azimuthal(DevGrid g, AziIO io, const double *__restrict__ vt,
                                                     int fast, const int *__restrict__ nshift,
                                                     const double *__restrict__ vmed, const double *__restrict__ vtemp)
{
  pdl_wait();
  const double dt = g.ctl[CTL_DT];
  __shared__ double s_a[AZ_TMAX], s_b[AZ_TMAX], s_c[AZ_TMAX];
  const int ns = g.ns, i = blockIdx.y, t = threadIdx.x, T = blockDim.x;
  const int seg = T - 2 * AZ_HALO;
  const int j0 = blockIdx.x * seg;
  const int j = (j0 + t - AZ_HALO + ns) % ns;
  const int tm = (t == 0) ? 0 : t - 1, tp = (t == T - 1) ? t : t + 1;   // edge threads only feed the halo
  const size_t rowo = (size_t)i * ns;
  // ring constants from tables
  const double dtinvdx = dt * g.r.InvDxtheta[i];
  const double dxrad = (g.r.Rsup[i] - g.r.Rinf[i]) * dt;
  const double invsurf = g.r.InvSurf[i];
  double q[NQ];
#pragma unroll
  for (int k = 0; k < NQ; k++) q[k] = io.src[k][rowo + j];
  const double vface = vt[rowo + j];
  const double vsub = fast ? vmed[i] : 0.0;
  // the residual velocity's pass or the uniform one, whose v, face coefficient
  // and flux factor are the ring's
  auto wind = [&](auto uniform) {
    constexpr bool U = decltype(uniform)::value;
    const double v = U ? vtemp[3 * i] : (vface - vsub);
    const bool up = __double_as_longlong(v) > 0LL; // v > 0.0: upwind cell of the left face is j-1
    // face value q* = q_up +/- (dxtheta -/+ v dt) dq_up with the slope dq kept
    // without its 1/dxtheta factor, which goes into csg = +/-1 - v dt/dxtheta
    // instead.  The upwind choice differs between neighbouring cells, so it
    // selects operands (integer moves) and every face value is one FMA,
    // fma(csg, dq_up, q_up), rather than two predicated ones.
    const double csg = U ? vtemp[3 * i + 1] : __fma_rn(-v, dtinvdx, up ? 1.0 : -1.0);
    // RhoStar at the left face (ComputeStarTheta of the density)
    const double rho = q[NQ - 1];
    s_a[t] = rho;
    __syncthreads();
    const double rho_m = s_a[tm];
    const double drm = rho - rho_m;
    s_b[t] = drm;
    __syncthreads();
    const double drho = vl_slope(drm, s_b[tp]);
    s_c[t] = drho;
    __syncthreads();
    const double rs = __fma_rn(csg, up ? s_c[tm] : drho, up ? rho_m : rho);
    const double cf = U ? vtemp[3 * i + 2] * rs : dxrad * rs * v;   // flux = dxrad Q* RhoStar v
    const double rcp = div_fast(1.0, rho + 1e-20); // 1 / (RhoInt + 1e-20)
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NQ; k++) {
      // VanLeerTheta: Work = Q / (RhoInt + 1e-20), its slope, the face value
      const double w = (k < NQ - 1) ? q[k] * rcp : unit_quotient(rho);
      s_a[t] = w;
      __syncthreads();
      const double w_m = s_a[tm];
      double qs;
      if (k < NQ - 1) {
        const double dm = w - w_m;
        s_b[t] = dm;
        __syncthreads();
        const double dq = vl_slope(dm, s_b[tp]);
        s_c[t] = dq;
        __syncthreads();
        qs = __fma_rn(csg, up ? s_c[tm] : dq, up ? w_m : w);
      } else {
        // the density's own quotient rho / (rho + 1e-20) is 1 to within
        // 1e-20 / rho: its slope term is below rounding
        qs = up ? w_m : w;
      }
      const double F = qs * cf;
      s_b[t] = F;                                  // every read of s_b is behind a barrier
      __syncthreads();
      q[k] = __fma_rn(F - s_b[tp], invsurf, q[k]);
    }
  };
  wind(std::false_type());
  if (fast) wind(std::true_type());
  const int x = t - AZ_HALO;
  if (x >= 0 && x < seg && j0 + x < ns) {
    int jo = j;
    if (fast) {
      jo = (j + nshift[i]) % ns;                   // AdvectSHIFT: new[j + Nshift] = old[j]
      if (jo < 0) jo += ns;
    }
#pragma unroll
    for (int k = 0; k < NQ; k++) io.dst[k][rowo + jo] = q[k];
  }
}

// Threads per block for the azimuthal step: the multiple of 32 in
// [128, AZ_TMAX] that needs the fewest warps per ring.
static int azi_block(int ns)
{
  int best = 0, bestw = 1 << 30;
  for (int T = 128; T <= AZ_TMAX; T += 32) {
    const int seg = T - 2 * AZ_HALO;
    const int w = (ns + seg - 1) / seg * (T / 32);
    if (w < bestw) { bestw = w; best = T; }
  }
  return best;
}

// ComputeVelocities (TransportEuler.c:350-381), followed for the gas by the
// damping of v_r (DampingBoundary with DampTowards ZEROVRAD,
// SideEuler.c:368-419) and the EOS refresh (ComputeTemperatureField,
// ComputeSoundSpeed).
__global__ void k_velocities(DevGrid g, const double *__restrict__ rho, const double *__restrict__ rmp,
                             const double *__restrict__ rmm, const double *__restrict__ tmp_,
                             const double *__restrict__ tmm, double *__restrict__ vr, double *__restrict__ vt, int damp_vrad, double drin, double drout,
                             const double *__restrict__ energy, double *__restrict__ temper, double *__restrict__ cs,
                             double gm1, double gamma)
{
  pdl_wait();
  const double dt = g.ctl[CTL_DT], omega_frame = g.ctl[CTL_OMEGA_FRAME];
  const int ns = g.ns;
  CELL_LOOP_2D
  const int ljm = (j == 0) ? i * ns + ns - 1 : l - 1;
  const double rm = g.r.Rmed[i];
  double v;
  if (i == 0) v = 0.0;
  else v = div_fast(rmp[l - ns] + rmm[l], rho[l] + rho[l - ns] + 1e-20);
  if (damp_vrad && (rm < drin || rm > drout)) {
    const double lambda = g.r.WaveKiller[i] * dt;
    v = div_fast(v + lambda * 0.0, 1.0 + lambda);
  }
  vr[l] = v;
  vt[l] = div_fast(tmp_[ljm] + tmm[l], rho[l] + rho[ljm] + 1e-15) * g.r.InvRmed[i] - rm * omega_frame;
  if (temper) {
    const double t = div_fast(energy[l] * gm1, rho[l]);
    temper[l] = t;
    cs[l] = sqrt_fast(gamma * abs_i(t));
  }
}

// ---------------------------------------------------------------------------
// Launch wrappers
void hydro_sources(const DevGrid &g, const SourceIO &io0, cudaStream_t s)
{
  SourceIO io = io0;
  // 0.15 rings a chunk: the ring below is read again, and the ring constants
  io.rings = chunk_rings(g.nr, g.ns, g.nsm, SRC_MAXRINGS, 0.15);
  const dim3 grid((g.ns + BX - 1) / BX, (g.nr + io.rings - 1) / io.rings);
  if (io.pd) launch_fp64(k_sources<true>, grid, BX, 0, s, g, io);
  else launch_fp64(k_sources<false>, grid, BX, 0, s, g, io);
  g_thorin_launches++;
}

void hydro_viscous(const DevGrid &g, const ViscousIO &io0, cudaStream_t s)
{
  ViscousIO io = io0;
  io.rings = chunk_rings(g.nr, g.ns, g.nsm, VI_MAXRINGS, 1.8);
  const dim3 grid((g.ns + VI_COLS - 1) / VI_COLS, (g.nr + io.rings - 1) / io.rings);
  launch_fp64(k_viscous, grid, BX, 0, s, g, io);
  g_thorin_launches++;
}

void hydro_heating(const DevGrid &g, const HeatingIO &io0, cudaStream_t s)
{
  HeatingIO io = io0;
  io.rings = chunk_rings(g.nr, g.ns, g.nsm, HT_MAXRINGS, 0.2);
  if (io.rings < 3) io.rings = 3;                  // ring 0 is extrapolated by the thread of rings 1 and 2
  const dim3 grid((g.ns + BX - 1) / BX, (g.nr + io.rings - 1) / io.rings);
  launch_fp64(k_heating, grid, BX, 0, s, g, io);
  g_thorin_launches++;
}

void hydro_eos(const DevGrid &g, const double *rho, const double *energy, double *temper, double *cs, double gm1,
               double gg1, cudaStream_t s)
{
  launch(k_eos, grid2d(g.ns, g.nr, BX), BX, 0, s, g, rho, energy, temper, cs, gm1, gg1 / gm1);
  g_thorin_launches++;
}

// 0.2 rings a chunk: the difference with the ring below and the ring constants
static int diffcoef_rings(const DevGrid &g) { return chunk_rings(g.nr, g.ns, g.nsm, DC_MAXRINGS, 0.2, 8); }

// Doubles of a disk's reduction scratch that k_diffcoef writes, one a block.
size_t hydro_partials(const DevGrid &g)
{
  const int r = diffcoef_rings(g);
  return (size_t)((g.ns + BX - 1) / BX) * ((g.nr + r - 1) / r);
}

void hydro_diffcoef(const DevGrid &g, const DiffusionIO &io0, int law, cudaStream_t s)
{
  DiffusionIO io = io0;
  io.rings = diffcoef_rings(g);
  const dim3 grid((g.ns + BX - 1) / BX, (g.nr + io.rings - 1) / io.rings);
  switch (law) {
  case THORIN_OPA_SM03: launch_fp64(k_diffcoef<THORIN_OPA_SM03>, grid, BX, 0, s, g, io); break;
  case THORIN_OPA_ZHU12: launch_fp64(k_diffcoef<THORIN_OPA_ZHU12>, grid, BX, 0, s, g, io); break;
  case THORIN_OPA_LP85: launch_fp64(k_diffcoef<THORIN_OPA_LP85>, grid, BX, 0, s, g, io); break;
  case THORIN_OPA_CONST: launch_fp64(k_diffcoef<THORIN_OPA_CONST>, grid, BX, 0, s, g, io); break;
  default: launch_fp64(k_diffcoef<THORIN_OPA_BL94>, grid, BX, 0, s, g, io); break;
  }
  g_thorin_launches++;
}

void hydro_irradiation(const DevGrid &g, const double *rho, const double *cs, const double *opacity, double *flaring,
                       double *qirr, double rstar, double tirr4fac, double opacity_drop, double taueff_c,
                       const double *rinf15, const double *rsup15, cudaStream_t s)
{
  launch_fp64(k_irradiation, grid2d(g.ns, g.nr, BX), BX, 0, s, g, rho, cs, opacity, flaring, qirr, rstar, tirr4fac, opacity_drop,
                                                      taueff_c, rinf15, rsup15);
  g_thorin_launches++;
}

// Rings per block of k_matrix; 0.3 rings a chunk are the first face and the
// ring constants.
static int matrix_rings(const DevGrid &g) { return chunk_rings(g.nr - 2, g.ns, g.nsm, MX_MAXRINGS, 0.3); }

static dim3 matrix_grid(const DevGrid &g)
{
  const int r = matrix_rings(g);
  return dim3((g.ns + BX - 1) / BX, (g.nr - 2 + r - 1) / r);
}

void hydro_matrix(const DevGrid &g, const MatrixIO &io0, const SorCtl *resid, cudaStream_t s)
{
  MatrixIO io = io0;
  io.rings = matrix_rings(g);
  if (resid) launch_fp64(k_matrix<true>, matrix_grid(g), BX, 0, s, g, io, *resid);
  else launch_fp64(k_matrix<false>, matrix_grid(g), BX, 0, s, g, io, SorCtl{});
  g_thorin_launches++;
}

// Resident k_sor_pass blocks per multiprocessor that fit (occupancy API),
// found once.
static int sor_occ_max()
{
  static std::atomic<int> occ_cache{0};
  int occ = occ_cache.load();
  if (occ == 0) {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_sor_pass, SOR_PX, 0) != cudaSuccess || occ < 1) occ = 1;
    occ_cache.store(occ);
  }
  return occ;
}

// One wave of resident blocks striding over the colour's cells, with at most
// g.sor_tpsm threads per multiprocessor (the ensemble autotuner may pick a cap
// per disk; the default is above what the pass's registers allow).
static dim3 sor_grid_pass(const DevGrid &g, bool capped = true)
{
  int occ = sor_occ_max();
  const int tpsm = g.sor_tpsm > 0 ? g.sor_tpsm : 1536;
  if (capped && occ * SOR_PX > tpsm) occ = tpsm / SOR_PX > 0 ? tpsm / SOR_PX : 1;
  const long long nblk = ((long long)(g.ns / 2) * (g.nr - 2) + SOR_PX - 1) / SOR_PX;
  const long long wave = (long long)g.nsm * occ;
  return dim3((unsigned)(nblk < wave ? nblk : wave));
}

int hydro_sor_pass_blocks(const DevGrid &g) { return (int)sor_grid_pass(g).x; }

static dim3 sor_grid_resid(const DevGrid &g)
{
  return dim3((g.ns + SOR_BX * SOR_CPT - 1) / (SOR_BX * SOR_CPT), g.nr - 2);
}

int sor_blocks(const DevGrid &g)
{
  const dim3 a = sor_grid_pass(g, false), b = sor_grid_resid(g), c = matrix_grid(g);
  const int na = a.x * a.y, nb = b.x * b.y, nc = c.x * c.y;
  return na > nb ? (na > nc ? na : nc) : (nb > nc ? nb : nc);
}

void hydro_sor_resid0(const DevGrid &g, const double *T, const double *ml, const double *mlip, const double *mlim,
                      const double *mljp, const double *mljm, const double *rhs, double *cw,
                      const SorCtl &c, cudaStream_t s)
{
  launch(k_sor_resid0, sor_grid_resid(g), SOR_BX, 0, s, g, T, ml, mlip, mlim, mljp, mljm, rhs, cw, c);
  g_thorin_launches++;
}

void hydro_sor_sweeps(const DevGrid &g, double *T, const double *ml, const double *mlip, const double *mlim,
                      const double *mljp, const double *mljm, const double *rhs, const double *cw, const SorCtl &c,
                      double eps, int count, int maxiters, cudaStream_t s)
{
  // numbers of launches are counted by the caller
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = sor_grid_pass(g);
  cfg.blockDim = dim3(SOR_PX);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  for (int n = 0; n < 2 * count; n++) {
    // the first pass waits for whatever wrote its coefficients
    cfg.numAttrs = (n > 0) ? 1 : 0;
    cudaLaunchKernelEx(&cfg, k_sor_pass, g, T, ml, mlip, mlim, mljp, mljm, rhs, cw, c, eps, (n & 1) + 1, maxiters);
  }
}

// k_sor_grid's launch: as many rows R of nt threads as hold a block's pairs,
// the coefficients of its first res pairs (whole warps') in shared memory.
// A solve alone on the GPU takes up to 1024 threads of a multiprocessor and
// 200 KB of its memory; with shared set (disks of an ensemble advanced
// together) it takes three quarters of the multiprocessors and up to 1.15
// million cells at most half of each (above, the temperatures alone fill more
// than 110 KB), so that two solves and the other disks' kernels fit beside each
// other: a DT of eight disks of 128 to 512 rings takes 12.7 ms (13.0 on all
// multiprocessors, 14.2 with the larger blocks); alone the smaller blocks cost
// 333x1002 3.85 us a pass instead of 3.3, 512x1536 6.8 instead of 6.1.
struct SorGridShape { int nb, nt, R, res; size_t smem; };

static SorGridShape sor_grid_shape(const DevGrid &g, int shared)
{
  const int np = (g.ns >> 1) * (g.nr - 2), most = shared ? 480 : 992;
  const int nsm = shared ? (3 * g.nsm + 3) / 4 : g.nsm;
  SorGridShape q;
  q.nb = (np + 31) / 32 < nsm ? (np + 31) / 32 : nsm;
  const int pm = (np + q.nb - 1) / q.nb;
  q.R = (pm + most - 1) / most;
  q.nt = ((pm + q.R - 1) / q.R + 31) / 32 * 32;
  const size_t room = (shared ? 110 : 200) * 1024, fixed = 20 * (size_t)pm + 24 * (size_t)q.nt;
  q.res = fixed < room ? (int)((room - fixed) / (32 * 112)) * 32 : 0;
  if (q.res > pm) q.res = (pm + 31) / 32 * 32;
  q.smem = fixed + 112 * (size_t)q.res;
  return q;
}

// The most dynamic shared memory of a block.
#define SOR_GRID_SMEM (227 * 1024 - 256)

// Whether either shape of a disk is within the kernel's limits; *smem (may be
// NULL): the larger one's shared memory.
bool hydro_sor_grid_within(const DevGrid &g, int maxiters, long long *smem)
{
  if (g.nr < 3 || (g.ns & 1) || (long long)g.ns * (g.nr - 2) > SOR_GRID_CELLS || maxiters >= (1 << 24) - 2) return false;
  size_t most = 0;
  bool ok = true;
  for (int shared = 0; shared < 2; shared++) {
    const SorGridShape q = sor_grid_shape(g, shared);
    most = q.smem > most ? q.smem : most;
    ok = ok && q.smem <= SOR_GRID_SMEM && q.nb < SOR_GRID_RECORDS;
  }
  if (smem) *smem = (long long)most;
  return ok;
}

int hydro_sor_grid_fits(const DevGrid &g, int maxiters)
{
  if (!hydro_sor_grid_within(g, maxiters, nullptr)) return 0;
  int dev = 0, coop = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || !coop ||
      cudaFuncSetAttribute(k_sor_grid<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SOR_GRID_SMEM) != cudaSuccess ||
      cudaFuncSetAttribute(k_sor_grid<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SOR_GRID_SMEM) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  for (int shared = 0; shared < 2; shared++) {
    const SorGridShape q = sor_grid_shape(g, shared);
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_sor_grid<false>, q.nt + 32, q.smem) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    if (n * sms < q.nb) return 0;
  }
  return 1;
}

cudaError_t hydro_sor_grid(const DevGrid &g, double *T, const double *ml, const double *mlip, const double *mlim,
                           const double *mljp, const double *mljm, const double *rhs, const double *cw, const SorCtl &c,
                           void *x, double eps, int maxiters, int shared, int spin, cudaStream_t s)
{
  const SorGridShape q = sor_grid_shape(g, shared);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeCooperative;
  at.val.cooperative = 1;
  cfg.gridDim = dim3(q.nb);
  cfg.blockDim = dim3(q.nt + 32);
  cfg.dynamicSmemBytes = q.smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  const SorSystem m = {ml, mlip, mlim, mljp, mljm, rhs, cw};
  return cudaLaunchKernelEx(&cfg, spin < SOR_GRID_SPIN ? k_sor_grid<true> : k_sor_grid<false>, g, T, m, c,
                            (ulonglong2 *)x, eps, maxiters, q.R, q.res, spin);
}

void hydro_energy_from_t(const DevGrid &g, const double *rho, double *T, double *enew, cudaStream_t s)
{
  launch(k_energy_from_t, grid2d(g.ns, g.nr + 1, BX * EFT_CPT), BX, 0, s, g, rho, T, enew);
  g_thorin_launches++;
}

// Whole transport of one fluid.  q_in: rho, vr, vt, energy (NULL for
// pebbles).  On return the caller's rho/energy pointers
// are swapped with the updated buffers and vr/vt hold the new velocities.

void hydro_transport(const DevGrid &g, double **rho, const double *vr_in, const double *vt_in, double *vr, double *vt,
                     double **energy, double *label, const TransportScratch &S, int fast, int damp_vrad, double drin,
                     double drout, double *temper, double *cs, double gm1, double gg1, cudaStream_t s)
{
  const int ns = g.ns, nr = g.nr;
  // transported quantities in the reference's order: rmp, rmm, tmp, tmm,
  // [e], [rho*label], rho.  Quotient buffers: w[0..3] momenta, w[4] energy,
  // w[6] tracer, w[5] rho.
  int qi[7], nq = 0;
  for (int q = 0; q < 4; q++) qi[nq++] = q;
  if (energy) qi[nq++] = 4;
  if (label) qi[nq++] = 6;
  qi[nq++] = 5;
  // the radially transported quantities go to the w buffers
  RadialIO rd;
  rd.rho = *rho; rd.vr = vr_in; rd.vt = vt_in; rd.energy = energy ? *energy : nullptr; rd.label = label;
  for (int q = 0; q < 4; q++) rd.out[q] = S.w[q];
  rd.out[4] = S.w[5];
  rd.out[5] = S.w[4];
  rd.ext = S.w[6];
  rd.rings = chunk_rings(nr, ns, g.nsm, RD_MAXRINGS, 1.3);
  const dim3 rgrid((ns + BX - 1) / BX, (nr + rd.rings - 1) / rd.rings);
  if (energy && label) launch_fp64(k_radial<true, true>, rgrid, BX, 0, s, g, rd);
  else if (energy) launch_fp64(k_radial<true, false>, rgrid, BX, 0, s, g, rd);
  else if (label) launch_fp64(k_radial<false, true>, rgrid, BX, 0, s, g, rd);
  else launch_fp64(k_radial<false, false>, rgrid, BX, 0, s, g, rd);
  g_thorin_launches++;
  // azimuthal step back into the momenta, the new energy, the tracer and
  // the new density
  launch(k_azi_rings, nr, RING_T, 0, s, g, vt_in, S.nshift, S.vmed, S.vtemp);
  g_thorin_launches++;
  AziIO az;
  for (int k = 0; k < nq; k++) {
    const int q = qi[k];
    az.src[k] = S.w[q];
    az.dst[k] = (q < 4) ? S.mom[q] : (q == 4) ? S.e_new : (q == 6) ? S.ext_new : S.rho_new;
  }
  az.n = nq;
  const int T = azi_block(ns);
  const dim3 grid((ns + T - 2 * AZ_HALO - 1) / (T - 2 * AZ_HALO), nr);
  if (nq == 7) launch_fp64(k_azimuthal<7>, grid, T, 0, s, g, az, vt_in, fast, S.nshift, S.vmed, S.vtemp);
  else if (nq == 6) launch_fp64(k_azimuthal<6>, grid, T, 0, s, g, az, vt_in, fast, S.nshift, S.vmed, S.vtemp);
  else launch_fp64(k_azimuthal<5>, grid, T, 0, s, g, az, vt_in, fast, S.nshift, S.vmed, S.vtemp);
  g_thorin_launches++;
  // velocities from the transported momenta
  launch_fp64(k_velocities, grid2d(ns, nr, BX), BX, 0, s, g, S.rho_new, S.mom[0], S.mom[1], S.mom[2], S.mom[3], vr, vt, damp_vrad, drin, drout,
                                                 energy ? S.e_new : nullptr, energy ? temper : nullptr, cs, gm1, gg1 / gm1);
  g_thorin_launches++;
  if (label) {
    launch(k_label_from_ext, grid2d(ns, nr, BX), BX, 0, s, g, S.rho_new, S.ext_new, label);
    g_thorin_launches++;
  }
}


