// thorin_kernels.cuh -- argument structs and host launchers of the kernels.
#pragma once
#include <atomic>
#include <utility>
#include "thorin_dev.cuh"

#define MAXPL_DEV 8            // planets handled by the force kernel (per-thread arrays)
#define ACC_BX 256             // threads per block of the pebble accretion kernels

// Planet data seen by the kernels (per-planet constants from the host).
struct DevPlanet {
  double x, y, z, m, rhill, Hpl, smoothing2, rst2, rst3, rst4, rsm2, rmorevert2;
  double near_h2, near_hill2;   // (10 Hpl)^2 and (5 rhill)^2: the vertical-quadrature zone
};

// Indices into the small device scalar buffer.
enum {
  SC_NEWDT = 0, SC_INVDTPEB, SC_DTSTELLAR, SC_INDX, SC_INDY, SC_ACC_DM, SC_ACC_DPX, SC_ACC_DPY, SC_RINGRHO,
  SC_MASS, SC_MOM, SC_ENER, SC_PMASS, SC_PMOM, SC_NORMRES0, SC_NORMRES,
  SC_PLANET_A = 32,           // 2 per planet: ax, ay (then the ring means of Sigma for DampingTW04)
  SC_TORQUE = 56,             // 2 per planet: ring means of Sigma either side of the planet (UpdateLog)
  SC_GASACC = 80,             // dM, dPx, dPy of the gas accretion onto one planet
  SC_DRAGCELL = 84,           // 6 values of the planet's cell for the aerodynamic drag
  SC_RCS = 96,                // device-resident DT: ring mean of c_s at each planet, taken before the hydro
  SC_CFLTOP = 104             // bits of the CFL's largest sums of squared rates (gas, pebbles)
};
enum { IS_NSUB = 0, IS_SOR_DONE, IS_SOR_NITER, IS_SOR_CHANGED, IS_CRASH, IS_COUNT, IS_CFL_BOUND = 32,
       IS_SOR_OUT = 40 };         // of the host copy: done, niter, changed, abort of the solve

// Red-black SOR control block (device pointers).
struct SorCtl {
  double *part;           // [2][nblocks] partial |resid| sums
  int *ipart;             // [2][nblocks] partial changed counts
  unsigned int *ticket;
  int *done;              // 1 converged, 2 iteration cap; later sweeps are no-ops
  int *niter;
  double *normres0;
  double *normres;
  int *changed;
  double *jscale;         // sum over the start of |resid| * omega/Ml (with the start residual)
  unsigned long long *epoch;    // number of this solve (k_sor_grid's tags)
  int *abort;             // a wait of k_sor_grid ran out: the solve is void, done or not
  // Condition of the graph's WHILE node around the sweeps: the completion
  // step sets it to 0 together with done (has_cond 0: no such node)
  cudaGraphConditionalHandle cond;
  int has_cond;
};

// Transport scratch (device fields).
struct TransportScratch {
  double *mom[4];          // RadMomP, RadMomM, ThetaMomP, ThetaMomM after the transport
  double *rho_new, *e_new;
  double *ext_new;         // rho * label after the transport (LabelAdvection)
  double *w[7];            // after the radial step: the momenta, energy, density, rho * label
  int *nshift;
  double *vmed, *vtemp;
};

// Arguments of the source step (pd NULL: no pebbles).
struct SourceIO {
  const double *rho, *vr, *vt, *energy, *press, *agr, *agt, *col, *supp_torque, *invdxtheta;
  const double *pd, *pvr, *pvt, *tau, *pagr, *pagt;
  double *vrint, *vtint, *pvrn, *pvtn;
  double gm1, schmidt;
  int back_reaction, diffusion, rings;
};

// Arguments of the viscous terms and SubStep2 (eint NULL: no energy equation;
// divv NULL: formed later, from the updated velocities).
struct ViscousIO {
  const double *rho, *vr, *vt, *energy, *invdxtheta;
  double *vrnew, *vtnew, *eint, *divv;
  double invdphi, vkep_in, vkep_out;
  int kepler, rings;
};

// Arguments of the viscous heating (temper NULL: without the equation of state).
struct HeatingIO {
  const double *rho, *vr, *vt, *energy;
  double *divv, *qplus, *temper, *cs;
  double invdphi, lr01, lr12, gm1, gamma;
  int rings;
};

// Arguments of the opacity and diffusion coefficient step.
struct DiffusionIO {
  const double *rho, *T, *cs, *invdxtheta, *deltar2;
  double *opacity, *qminus, *dcen, *part, *dtmin;   // dtmin: DiffusionTimestep's result
  unsigned int *ticket;
  double parametric_cu, opacity_drop, taueff_c;
  int rings;
};

// Arguments of the implicit energy equation's matrix (qirr NULL: no irradiation).
struct MatrixIO {
  const double *rho, *T, *cs, *dcen, *divv, *qminus, *qplus, *qirr, *invdxtheta2;
  double *ml, *mlip, *mlim, *mljp, *mljm, *rhs, *cw;
  const int *heat_idx;
  const double *heat_val;
  double gm1;
  int nheat, rings;
};

struct AziIO { const double *src[7]; double *dst[7]; int n; };   // index n-1 is the density

struct ViscParams {
  double viscosity, alpha, alpha_mri, alpha_dead, tmri, twidth, t2si;
  double cav_rmin, cav_rmax, cav_ratio, log_cav_ratio;
  int viscosity_alpha, alpha_flock;
};

struct CflRings {
  const double *dxrad, *dxtheta, *mindx, *den5;    // per ring, ConditionCFL's expressions
  double *vmoy, *pvtmed;                           // ring means (scratch)
};

struct CflFinal {
  int pebbles, first_call;
  int own;                     // deltaT and invdtreb_sq are here (else in the control block)
  double deltaT, invdtreb_sq, minimum_step, maximum_step, first_step, twopi_cfl_ns;
};

// The planets and control values that the host path hands to the force
// kernels (n < 0: they are on the device).
struct HostPlanets {
  int n;
  double mass_taper, indx, indy;
  DevPlanet pl[MAXPL_DEV];
};

// Single rings whose means are wanted.
struct RingList {
  int n;
  int ring[3 * MAXPL_DEV];
  double *out[3 * MAXPL_DEV];
};

struct ForceRings {
  double *H_avr, *p_H_avr;     // ring-mean scale heights of the gas and the pebbles
  double *agr0, *pagr0;        // the star's pull averaged over the ring-mean column
  double *starw;               // its weight in the disk's pull on the star, Surf |agr0|
  const double *drsq;          // (Rsup - Rinf)^2
};

// Terms of the star's vertical average as a series in (H/r)^2, and the largest
// (H/r)^2 it is used for: there the first term left out is below 8e-18.
#define FORCE_NC 12
#define FORCE_QMAX 0.0064

struct ForceArgs {
  const double *rho, *cs, *tau, *pdens;
  double *agr, *agt, *pagr, *pagt;
  double *part;               // [2 + 2*npl][nblocks]
  size_t part_size;           // doubles at part
  double *col;                // [2][ns]: the indirect term of each column (radial, and azimuthal between j-1 and j)
  unsigned char *near;        // cells left to k_forces_near
  unsigned int *ticket;       // of k_forces_final
  const DevPlanet *pl;
  DevPlanet *pl_out;           // the same, for the host path's copy
  int npl, pebbles, exclude_hill, pebble_gravity;
  double pebble_alpha, hillcut;   // the mass taper is read from the control block
  // vertical quadrature weights exp(-z_m^2 / 2H^2) at z_m = (m - 1/2) 3H/N,
  // which do not depend on H, the inverses of their sums, and the series
  // sum_k c_k (H/r)^2k of r^3 sum_m w_m (r^2 + z_m^2)^(-3/2) (filled by
  // aux_forces)
  double wq10[10], wq30[30], c10[FORCE_NC], c30[FORCE_NC];
  double isig10, isig30;
  int nba, nbb, nbn;          // blocks of k_forces and of k_forces_near, and those of the latter that walk rings
  int rings_a, rings_b;       // rings per block of the two
};

struct GasAccArgs {           // one planet of AccreteOntoPlanets (Planet.c:34-166)
  double Xp, Yp, Zp, RRoche, facc1, facc2, omega_frame;
  int i_min, i_max, j_min, j_max;
};

struct AccArgs {
  double *pdens, *macc;
  double *part;               // block partials (4 per block)
  double *acc;                // scalars: Reff, vrel, Mt, limiter, ring means of v_theta
  unsigned int *ticket;
  const double *pvr, *pvt, *tau, *cs, *vt;
  double Xp, Yp, Zp, VXp, VYp, VZp, Mp, Rp, Rhill, Omegap, Rp15, omega_frame, dt, pebble_alpha, frac;
  int imin, imax, iflow;
  int nb;                     // blocks over the annulus imin..imax (aux_accrete_blocks)
};

// Number of kernels launched by this library (host-side bookkeeping; every
// launcher below adds the launches it issues).  Atomic: disks of an ensemble
// are advanced from several host threads.
extern std::atomic<long long> g_thorin_launches;

// Kernel launch.  A grid of up to PDL_BLOCKS blocks goes with programmatic
// stream serialization: its blocks are placed while the kernel before it in
// the stream drains, and wait in pdl_wait, the first statement of every kernel
// launched this way, until that one has completed and its writes are visible
// (each kernel's wait keeps the order of the stream as a whole).  A substep is
// some 45 launches in line: 24x72 0.340 -> 0.271 ms, 128x384 with pebbles 0.554 ->
// 0.508, 333x1002 1.12 -> 1.10.  Waiting blocks of larger grids take the places
// that the other stream's kernels (pebble transport) would fill: with a limit
// of 160 / 304 / 608 / 1216 blocks and none, 333x1002 takes 1.095 / 1.095 / 1.137 /
// 1.181 / 1.175 ms, 128x384 0.522 / 0.508 / 0.499 / 0.499 / 0.515.
#define PDL_BLOCKS 304
template <typename... P, typename... A>
inline void launch_upto(size_t most, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A &&...args)
{
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = ((size_t)grid.x * grid.y * grid.z <= most) ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

template <typename... P, typename... A>
inline void launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A &&...args)
{
  launch_upto(PDL_BLOCKS, kernel, grid, block, smem, s, std::forward<A>(args)...);
}

// For the kernels that the FP64 pipe bounds: placed early, their blocks gather
// on the multiprocessors that the kernel before leaves first, and the fullest of
// these sets the time, so only grids of up to half the multiprocessors go
// early.  Limits of 0 / 76 / 152 / 304 blocks, ms a substep: 24x72 0.263 / 0.242 /
// 0.241 / 0.237, 64x192 0.281 / 0.270 / 0.296 / 0.296, 96x288 0.317 / 0.313 / 0.310 /
// 0.333, from 128x384 on the same.
#define PDL_BLOCKS_FP64 76
template <typename... P, typename... A>
inline void launch_fp64(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A &&...args)
{
  launch_upto(PDL_BLOCKS_FP64, kernel, grid, block, smem, s, std::forward<A>(args)...);
}

// kernels_hydro.cu
void hydro_sources(const DevGrid &g, const SourceIO &io, cudaStream_t s);
void hydro_viscous(const DevGrid &g, const ViscousIO &io, cudaStream_t s);
void hydro_heating(const DevGrid &g, const HeatingIO &io, cudaStream_t s);
void hydro_eos(const DevGrid &g, const double *rho, const double *energy, double *temper, double *cs, double gm1,
               double gg1, cudaStream_t s);
size_t hydro_partials(const DevGrid &g);
void hydro_diffcoef(const DevGrid &g, const DiffusionIO &io, int law, cudaStream_t s);
void hydro_irradiation(const DevGrid &g, const double *rho, const double *cs, const double *opacity, double *flaring,
                       double *qirr, double rstar, double tirr4fac, double opacity_drop, double taueff_c,
                       const double *rinf15, const double *rsup15, cudaStream_t s);
// resid: also the start of the SOR solve (NULL: the matrix alone)
void hydro_matrix(const DevGrid &g, const MatrixIO &io, const SorCtl *resid, cudaStream_t s);
int sor_blocks(const DevGrid &g);
int hydro_sor_pass_blocks(const DevGrid &g);     // blocks of a colour pass
void hydro_sor_resid0(const DevGrid &g, const double *T, const double *ml, const double *mlip, const double *mlim,
                      const double *mljp, const double *mljm, const double *rhs, double *cw,
                      const SorCtl &c, cudaStream_t s);
// `count` sweeps (two colour passes each).  The sweep number lives on the
// device, so every call with the same count issues identical launches (the
// caller may capture and replay them as a CUDA graph); the launch counter is
// left to the caller.
void hydro_sor_sweeps(const DevGrid &g, double *T, const double *ml, const double *mlip, const double *mlim,
                      const double *mljp, const double *mljm, const double *rhs, const double *cw, const SorCtl &c,
                      double eps, int count, int maxiters, cudaStream_t s);
// The whole solve in one cooperative launch, where
// hydro_sor_grid_fits; x: 32 bytes a cell of rings 1 .. nr-2 and
// 16 SOR_GRID_RECORDS more, zero at first; shared: other disks are at work on
// the GPU; spin: loads of one wait before it gives up (at most SOR_GRID_SPIN).
#define SOR_GRID_RECORDS 1024
#define SOR_GRID_SPIN (1 << 22)       // about 3 s
int hydro_sor_grid_fits(const DevGrid &g, int maxiters);
bool hydro_sor_grid_within(const DevGrid &g, int maxiters, long long *smem);
cudaError_t hydro_sor_grid(const DevGrid &g, double *T, const double *ml, const double *mlip, const double *mlim,
                           const double *mljp, const double *mljm, const double *rhs, const double *cw, const SorCtl &c,
                           void *x, double eps, int maxiters, int shared, int spin, cudaStream_t s);
void hydro_energy_from_t(const DevGrid &g, const double *rho, double *T, double *enew, cudaStream_t s);
void hydro_transport(const DevGrid &g, double **rho, const double *vr_in, const double *vt_in, double *vr, double *vt,
                     double **energy, double *label, const TransportScratch &S, int fast, int damp_vrad, double drin,
                     double drout, double *temper, double *cs, double gm1, double gg1, cudaStream_t s);

// kernels_aux.cu
size_t aux_partials(const DevGrid &g, int npl);
void aux_ring_means(const DevGrid &g, const double *f0, double *o0, const double *f1, double *o1, int ring0, int nrings,
                    cudaStream_t s);
void aux_ring_mean(const DevGrid &g, const double *f, double *out, cudaStream_t s);
void aux_ring_list(const DevGrid &g, const double *f, const RingList &r, cudaStream_t s);
void aux_sound_rings(const DevGrid &g, const ViscParams &v, const double *cs, const double *temper, double *csmean,
                     double *tempmean, cudaStream_t s);
void aux_stokes(const DevGrid &g, const double *rho, const double *psize, double *tau, cudaStream_t s);
void aux_cfl(const DevGrid &g, const double *vr, const double *vt, const double *cs, const double *pvr, const double *pvt,
             const CflRings &cr, int pebbles, int fast, int viscous, double *part, const CflFinal &f0, double *scal,
             int *iscal, cudaStream_t s);
void aux_evaporate(const DevGrid &g, const double *T, double *pdens, cudaStream_t s);
void aux_damp_gas(const DevGrid &g, double *vrad, double *rho, double *vtheta, double *energy, const int *rings,
                  int nrings, const double *vr0r, int damp_init, int damp_flux, int energy_eq, double *pd, double *pvr,
                  double *pvt, cudaStream_t s);
void aux_open_inner(const DevGrid &g, double *rho, double *vr, double *energy, int energy_eq, int damp_flux,
                    double gasflux, cudaStream_t s);
void aux_open_outer(const DevGrid &g, double *rho, double *vr, double *energy, int energy_eq, int damp_flux,
                    double gasflux, cudaStream_t s);
void aux_nonreflecting(const DevGrid &g, double *rho, double *vr, double *energy, const double *cs, cudaStream_t s);
void aux_outer_source_mass(const DevGrid &g, double *rho, double *vr, double penul_vr, cudaStream_t s);
void aux_parametric_cooling(const DevGrid &g, const double *rho, const double *eint, const double *qplus,
                            const double *divv, const double *coolt, const double *qplusmed, double *enew,
                            double gm1, cudaStream_t s);
void aux_gas_accrete(const DevGrid &g, double *dens, const double *vrad, const double *vtheta, const double *cs,
                     const GasAccArgs &a, double *out, cudaStream_t s);
void aux_drag_cell(const double *rho, const double *cs, const double *vrad, const double *vtheta, int l, int ns,
                   double *out, cudaStream_t s);
void aux_correct_vtheta(const DevGrid &g, double *vt, double domega, cudaStream_t s);
void aux_iso_eos(const DevGrid &g, const double *rho, const double *csr, double *cs, double *press, double *temper,
                 int set_cs, int set_press, int set_temper, cudaStream_t s);
void aux_damp_peb(const DevGrid &g, double *pd, double *pvr, double *pvt, const int *rings, int nrings, cudaStream_t s);
void aux_crash(const DevGrid &g, const double *f, int *flag, cudaStream_t s);
// THORIN_ERR_NOMEM, without a launch, when the block sums do not fit a0.part_size.
int aux_forces(const DevGrid &g, const ForceArgs &a0, const ForceRings &fr, const HostPlanets &hp, double *scal,
               cudaStream_t s);
// Pebble accretion with the arguments a0, which go to a_dev, or, with a0 NULL,
// with those at a_dev; nb: aux_accrete_blocks of the widest annulus possible.
void aux_accrete(const DevGrid &g, const AccArgs *a0, AccArgs *a_dev, int nb, double *scal, cudaStream_t s);
// Control block writes (host path): up to 6 (index, value) pairs; crash (may
// be NULL): cleared.
struct CtlSet { int n; int idx[6]; double val[6]; };
void aux_set_ctl(double *ctl, const CtlSet &v, int *crash, cudaStream_t s);
int aux_accrete_blocks(const DevGrid &g, int imin, int imax);
void aux_integrals(const DevGrid &g, const double *rho, const double *vr, const double *vt, const double *e,
                   const double *pd, const double *pvt, double omega_frame, int pebbles, double *part, double *scal,
                   unsigned int *ticket, cudaStream_t s);
