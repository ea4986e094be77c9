// kernels_aux.cu -- ring means, viscosity per ring, CFL, pebble source terms,
// damping boundaries, disk forces with their reductions, pebble accretion,
// conservation integrals.
#include <algorithm>
#include "thorin_kernels.cuh"
#include "thorin_graph.cuh"

static inline dim3 grid2d(int ns, int rows, int bx) { return dim3((ns + bx - 1) / bx, rows); }
static const int BX = 128;

#define CELL_LOOP_2D                                                        \
  const int j = blockIdx.x * blockDim.x + threadIdx.x;                      \
  const int i = blockIdx.y;                                                 \
  if (j >= ns) return;                                                      \
  const int l = j + i * ns;

// ---------------------------------------------------------------------------
// Ring (azimuthal) means, mpi_make1Dprofile (mpiTasks.c:26-32) and the
// other azimuthal averages of the loop.  One block per ring sums in a fixed
// tree (ring_sum), so results are deterministic; they differ from the
// reference's left-to-right sum in the last bits.  The only integer decision
// fed by a ring mean, the FARGO shift, re-sums its ring in order when the mean
// lands near a rounding tie (see k_azi_rings).  Output index is relative to
// ring0.
__global__ void __launch_bounds__(RING_T) k_ring_means(int ns, const double *__restrict__ f0,
                                                       const double *__restrict__ f1, double *__restrict__ o0,
                                                       double *__restrict__ o1, int ring0, int nf)
{
  pdl_wait();
  const int w = blockIdx.x;
  const size_t base = (size_t)(ring0 + w) * ns;
  const double a0 = ring_sum(f0 + base, ns);
  const double a1 = (nf > 1) ? ring_sum(f1 + base, ns) : 0.0;
  if (threadIdx.x == 0) {
    o0[w] = a0 / (double)ns;
    if (nf > 1) o1[w] = a1 / (double)ns;
  }
}

// The ring mean at a ring chosen on the device (none when *ring is negative).
__global__ void __launch_bounds__(RING_T) k_ring_mean_at(int ns, const double *__restrict__ f, double *__restrict__ o,
                                                         const int *__restrict__ ring)
{
  pdl_wait();
  const int i = *ring;
  if (i < 0) return;
  const double a = ring_sum(f + (size_t)i * ns, ns);
  if (threadIdx.x == 0) *o = a / (double)ns;
}

void graph_ring_mean_at(const DevGrid &g, const double *f, double *out, const int *ring, cudaStream_t s)
{
  launch(k_ring_mean_at, 1, RING_T, 0, s, g.ns, f, out, ring);
  g_thorin_launches++;
}

void aux_ring_means(const DevGrid &g, const double *f0, double *o0, const double *f1, double *o1, int ring0, int nrings,
                    cudaStream_t s)
{
  if (nrings <= 0) return;
  launch(k_ring_means, nrings, RING_T, 0, s, g.ns, f0, f1 ? f1 : f0, o0, o1 ? o1 : o0, ring0, f1 ? 2 : 1);
  g_thorin_launches++;
}

__global__ void k_set_ctl(double *__restrict__ ctl, CtlSet v, int *crash)
{
  pdl_wait();
  if (crash && threadIdx.x == 0) *crash = 0;
  if (threadIdx.x < (unsigned)v.n) ctl[v.idx[threadIdx.x]] = v.val[threadIdx.x];
}

void aux_set_ctl(double *ctl, const CtlSet &v, int *crash, cudaStream_t s)
{
  launch(k_set_ctl, 1, 32, 0, s, ctl, v, crash);
  g_thorin_launches++;
}

void aux_ring_mean(const DevGrid &g, const double *f, double *out, cudaStream_t s)
{
  aux_ring_means(g, f, out, nullptr, nullptr, 0, g.nr, s);
}

// The means of the rings r.ring[] to r.out[].
__global__ void __launch_bounds__(RING_T) k_ring_list(int ns, const double *__restrict__ f, RingList r)
{
  pdl_wait();
  const double a = ring_sum(f + (size_t)r.ring[blockIdx.x] * ns, ns);
  if (threadIdx.x == 0) *r.out[blockIdx.x] = a / (double)ns;
}

void aux_ring_list(const DevGrid &g, const double *f, const RingList &r, cudaStream_t s)
{
  if (r.n <= 0) return;
  launch(k_ring_list, r.n, RING_T, 0, s, g.ns, f, r);
  g_thorin_launches++;
}

// FViscosity at Rmed[i] and Rinf[i] (Viscosity.c:26-54).  The ring index
// found by the reference's linear search is i for both radii; pow(r, 1.5)
// comes precomputed from the host.

__device__ __forceinline__ double fvisc(const ViscParams &v, double rad, double cs, double tmean, double r15)
{
  double nu = v.viscosity;
  if (v.viscosity_alpha) nu = v.alpha * cs * cs * r15;
  if (v.alpha_flock) {
    double a = (v.alpha_mri - v.alpha_dead) * (1.0 - tanh((v.tmri - tmean * v.t2si) / v.twidth)) / 2.0 + v.alpha_dead;
    nu = a * cs * cs * r15;
  }
  if (rad < v.cav_rmin) nu *= v.cav_ratio;
  if ((rad >= v.cav_rmin) && (rad <= v.cav_rmax)) nu *= exp((v.cav_rmax - rad) / (v.cav_rmax - v.cav_rmin) * v.log_cav_ratio);
  return nu;
}

// Ring means of the sound speed (and, with alpha_flock, of the temperature)
// with each ring's viscosity from them, one block per ring.
__global__ void __launch_bounds__(RING_T) k_sound_rings(DevGrid g, ViscParams v, const double *__restrict__ cs,
                                                        const double *__restrict__ temper, double *__restrict__ csmean,
                                                        double *__restrict__ tempmean)
{
  pdl_wait();
  const int i = blockIdx.x, ns = g.ns;
  const double c = ring_sum(cs + (size_t)i * ns, ns) / (double)ns;
  double t = tempmean[i];
  if (temper) t = ring_sum(temper + (size_t)i * ns, ns) / (double)ns;
  if (threadIdx.x != 0) return;
  csmean[i] = c;
  tempmean[i] = t;
  g.r.nu_med[i] = fvisc(v, g.r.Rmed[i], c, t, g.r.Rmed15[i]);
  g.r.nu_inf[i] = fvisc(v, g.r.Rinf[i], c, t, g.r.Rinf15[i]);
}

void aux_sound_rings(const DevGrid &g, const ViscParams &v, const double *cs, const double *temper, double *csmean,
                     double *tempmean, cudaStream_t s)
{
  launch(k_sound_rings, g.nr, RING_T, 0, s, g, v, cs, v.alpha_flock ? temper : nullptr, csmean, tempmean);
  g_thorin_launches++;
}

// ---------------------------------------------------------------------------
// PebbleStokesNumbers (Pebbles.c:280-300).
__global__ void k_stokes(DevGrid g, const double *__restrict__ rho, const double *__restrict__ psize,
                         double *__restrict__ tau, double c)
{
  pdl_wait();
  const int ns = g.ns;
  CELL_LOOP_2D
  tau[l] = div_fast(c * psize[l], rho[l]);
}

void aux_stokes(const DevGrid &g, const double *rho, const double *psize, double *tau, cudaStream_t s)
{
  launch(k_stokes, grid2d(g.ns, g.nr, BX), BX, 0, s, g, rho, psize, tau, 2.0 * g.k.pebbulkdens * g.k.sqrt_adiabind_inv);
  g_thorin_launches++;
}

// ---------------------------------------------------------------------------
// CFL: ConditionCFL (SourceEuler.c:589-712) and CriticalCharTime
// (Pebbles.c:729-767).  Because x -> CFLSECURITY/sqrt((x + a) + b) is
// monotone, the minimum over cells of the per-cell step equals the step of
// the cell with the largest sum of squared rates, so block maxima of that
// sum are reduced (exactly, in any order) and the step is formed once.

// The sums of squared rates are >= 0, so their maxima are taken on the bit
// patterns as 64-bit integers (same order, integer pipe).
struct OpMaxI64 { __device__ long long operator()(long long a, long long b) const { return b > a ? b : a; } };

#define CFL_CPT 4       // cells per thread

// The sums of squared rates of one cell in FP64 (the reference's expressions).
__device__ __forceinline__ void cfl_cell(const DevGrid &g, const double *vr, const double *vt, const double *cs,
                                         const double *pvr, const double *pvt, const CflRings &cr, int pebbles, int fast,
                                         int i, int j, double idxrad, double idxtheta, double imindx, double invdt5,
                                         double &gas, double &peb)
{
  const int ns = g.ns, l = j + i * ns, lip = l + ns;
  const int ljp = (j == ns - 1) ? i * ns : l + 1;
  const double vres = fast ? vt[l] - cr.vmoy[i] : vt[l];
  const double invdt1 = cs[l] * imindx;
  const double invdt2 = fabs(vr[l]) * idxrad;
  const double invdt3 = fabs(vres) * idxtheta;
  double dvr = vr[lip] - vr[l], dvt = vt[ljp] - vt[l];
  dvr = (dvr >= 0.0) ? 1e-10 : -dvr;
  dvt = (dvt >= 0.0) ? 1e-10 : -dvt;
  const double a = dvr * idxrad, b = dvt * idxtheta;
  double invdt4 = (b > a) ? b : a;
  invdt4 *= 4.0 * TH_CVNR * TH_CVNR;
  gas = invdt1 * invdt1 + invdt2 * invdt2 + invdt3 * invdt3 + invdt4 * invdt4 + invdt5 * invdt5;
  peb = 0.0;
  if (pebbles) {
    const double p1 = fabs(pvr[l]) * idxrad;
    const double vrp = fast ? pvt[l] - cr.pvtmed[i] : pvt[l];
    const double p2 = fabs(vrp) * idxtheta;
    const double p3 = fabs(pvr[l] - vr[l]) * idxrad;
    const double p4 = fabs(pvt[l] - vt[l]) * idxtheta;
    peb = p1 * p1 + p2 * p2 + p3 * p3 + p4 * p4;
  }
}

// The sum of squares of lower and upper bounds of |x|, x known to within e.
struct CflBound {
  float lo = 0.0f, hi = 0.0f;
  __device__ void add(float x, float e, float scale)
  {
    const float a = fabsf(x), l = fmaxf(a - e, 0.0f) * scale, h = (a + e) * scale;
    lo = fmaf(l, l, lo);
    hi = fmaf(h, h, hi);
  }
};

// First pass, in FP32: bounds of every cell's sums.  Only the largest sum of
// the disk enters the time step, and it lies in a few rings, so this pass
// keeps the largest upper bound of each block and, over the grid, the largest
// lower bound (bound[0] gas, bound[1] pebbles: maxima of non-negative floats
// taken on their bits, in any order; k_cfl_final clears them), and k_cfl_cells evaluates in FP64 only
// the blocks whose upper bound reaches it: the same maximum, exactly, for a
// tenth of the time (36 FP64 instructions a cell before, 62 us at 512x1536).
// The FP32 values are within 1.3e-7 of |x| of the operands, differences within
// the sum of both, products and sums within 1e-5.
__global__ void __launch_bounds__(256) k_cfl_bounds(DevGrid g, const double *__restrict__ vr,
                                                    const double *__restrict__ vt, const double *__restrict__ cs,
                                                    const double *__restrict__ pvr, const double *__restrict__ pvt,
                                                    CflRings cr, int pebbles, int fast, int viscous,
                                                    float *__restrict__ part, int *__restrict__ bound)
{
  pdl_wait();
  __shared__ float sh[4][8];
  const int ns = g.ns;
  const int i = blockIdx.y + 1;
  const float idxrad = 1.0f / (float)cr.dxrad[i], idxtheta = 1.0f / (float)cr.dxtheta[i],
              imindx = 1.0f / (float)cr.mindx[i];
  const float vm = fast ? (float)cr.vmoy[i] : 0.0f, pvm = (fast && pebbles) ? (float)cr.pvtmed[i] : 0.0f;
  const float eps = 1.5e-7f, c4 = (float)(4.0 * TH_CVNR * TH_CVNR);
  const float x5 = viscous ? (float)(g.r.nu_med[i] * 4.) / (float)cr.den5[i] : 0.0f;
  float mx[4] = {0.0f, 0.0f, 0.0f, 0.0f};          // gas lo, hi, pebbles lo, hi
#pragma unroll
  for (int m = 0; m < CFL_CPT; m++) {
    const int j = (blockIdx.x * CFL_CPT + m) * 256 + threadIdx.x;
    if (j >= ns) break;
    const int l = j + i * ns;
    const int ljp = (j == ns - 1) ? i * ns : l + 1;
    const float r = to_float_trunc(vr[l]), rp = to_float_trunc(vr[l + ns]), t = to_float_trunc(vt[l]),
                tp = to_float_trunc(vt[ljp]);
    const float er = eps * fabsf(r), ert = eps * fabsf(t), em = eps * fabsf(vm);
    CflBound b;
    b.add(x5, 0.0f, 1.0f);
    b.add(to_float_trunc(cs[l]), 0.0f, imindx);
    b.add(r, er, idxrad);
    b.add(t - vm, ert + em + eps * fabsf(t - vm), idxtheta);
    // invdt4: the larger of the two compressions (1e-10 where there is none)
    const float ea = er + eps * fabsf(rp), eb = ert + eps * fabsf(tp);
    const float da = r - rp, db = t - tp;
    const float alo = fmaxf(da - ea, 0.0f) * idxrad, ahi = fmaxf(fmaxf(da, 0.0f) + 1.01f * ea, 1.1e-10f) * idxrad;
    const float blo = fmaxf(db - eb, 0.0f) * idxtheta, bhi = fmaxf(fmaxf(db, 0.0f) + 1.01f * eb, 1.1e-10f) * idxtheta;
    const float lo4 = fmaxf(alo, blo) * c4, hi4 = fmaxf(ahi, bhi) * c4;
    b.lo = fmaf(lo4, lo4, b.lo);
    b.hi = fmaf(hi4, hi4, b.hi);
    // a NaN or infinite bound excludes nothing: the FP64 pass sees the cell
    mx[0] = fmaxf(mx[0], isfinite(b.lo) ? b.lo : 0.0f);
    mx[1] = fmaxf(mx[1], isfinite(b.hi) ? b.hi : __int_as_float(0x7f800000));
    if (pebbles) {
      const float pr = to_float_trunc(pvr[l]), pt = to_float_trunc(pvt[l]);
      const float epr = eps * fabsf(pr), ept = eps * fabsf(pt);
      CflBound p;
      p.add(pr, epr, idxrad);
      p.add(pt - pvm, ept + eps * fabsf(pvm) + eps * fabsf(pt - pvm), idxtheta);
      p.add(pr - r, epr + er + eps * fabsf(pr - r), idxrad);
      p.add(pt - t, ept + ert + eps * fabsf(pt - t), idxtheta);
      mx[2] = fmaxf(mx[2], isfinite(p.lo) ? p.lo : 0.0f);
      mx[3] = fmaxf(mx[3], isfinite(p.hi) ? p.hi : __int_as_float(0x7f800000));
    }
  }
#pragma unroll
  for (int q = 0; q < 4; q++) {
    for (int o = 16; o > 0; o >>= 1) mx[q] = fmaxf(mx[q], __shfl_xor_sync(TH_FULL, mx[q], o));
    if ((threadIdx.x & 31) == 0) sh[q][threadIdx.x >> 5] = mx[q];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < 4; q++)
      for (int w = 0; w < 8; w++) mx[q] = fmaxf(mx[q], sh[q][w]);
    const int b = blockIdx.x + blockIdx.y * gridDim.x;
    part[2 * b] = mx[1] * 1.00001f;
    part[2 * b + 1] = mx[3] * 1.00001f;
    // a block that holds an unbounded cell sets no bound for the others
    if (isfinite(mx[1])) atomicMax(bound, __float_as_int(mx[0] * 0.99999f));
    if (pebbles && isfinite(mx[3])) atomicMax(bound + 1, __float_as_int(mx[2] * 0.99999f));
  }
}

// Second pass: the maxima of the sums in FP64, over the columns that can hold
// the disk's largest (all of them without bounds: upper NULL).  The sums are
// >= 0, so the maxima of the grid are taken on their bits, exactly and in any
// order; a block whose maximum is not a number, as only a crashed state holds,
// does not count.  A block takes a quarter of a block of the first pass: the
// rings that are evaluated fall on several multiprocessors.
__global__ void __launch_bounds__(256) k_cfl_cells(DevGrid g, const double *__restrict__ vr,
                                                   const double *__restrict__ vt, const double *__restrict__ cs,
                                                   const double *__restrict__ pvr, const double *__restrict__ pvt,
                                                   CflRings cr, int pebbles, int fast, int viscous,
                                                   const float *__restrict__ upper, const int *__restrict__ bound,
                                                   unsigned long long *__restrict__ top)
{
  pdl_wait();
  const int ns = g.ns;
  const int i = blockIdx.y + 1;                    // rings One_or_active .. Max_or_active-1
  if (upper) {
    const int b = blockIdx.x / CFL_CPT + blockIdx.y * ((gridDim.x + CFL_CPT - 1) / CFL_CPT);
    if (!(upper[2 * b] >= __int_as_float(bound[0])) && !(pebbles && upper[2 * b + 1] >= __int_as_float(bound[1])))
      return;
  }
  const double dxrad = cr.dxrad[i], dxtheta = cr.dxtheta[i], mindx = cr.mindx[i];
  const double invdt5 = viscous ? div_fast(g.r.nu_med[i] * 4., cr.den5[i]) : 1e-30;
  // the per-cell rates divide by ring constants: multiply by their reciprocals
  const double idxrad = div_fast(1.0, dxrad), idxtheta = div_fast(1.0, dxtheta), imindx = div_fast(1.0, mindx);
  double sg = 0.0, sp = 0.0;
  const int j = blockIdx.x * 256 + threadIdx.x;
  if (j < ns) cfl_cell(g, vr, vt, cs, pvr, pvt, cr, pebbles, fast, i, j, idxrad, idxtheta, imindx, invdt5, sg, sp);
  const long long mg = block_reduce(__double_as_longlong(sg), OpMaxI64(), 0LL);
  const long long mp = pebbles ? block_reduce(__double_as_longlong(sp), OpMaxI64(), 0LL) : 0LL;
  if (threadIdx.x == 0) {
    if (mg <= 0x7ff0000000000000LL) atomicMax(top, (unsigned long long)mg);
    if (pebbles && mp <= 0x7ff0000000000000LL) atomicMax(top + 1, (unsigned long long)mp);
  }
}

// The shear step over the rings, as a 64-bit integer minimum, and the time step.
struct OpMinI64 { __device__ long long operator()(long long a, long long b) const { return b < a ? b : a; } };

__global__ void __launch_bounds__(1024) k_cfl_final(DevGrid g, CflRings cr, CflFinal f, double *__restrict__ scal,
                                                    int *__restrict__ iscal, int *__restrict__ bound,
                                                    unsigned long long *__restrict__ top)
{
  pdl_wait();
  // the remaining part of the DT and MinStepForRebound's rate come from the
  // host (own) or the disk's control block, which receives the substep length
  const double deltaT = f.own ? f.deltaT : g.ctl[CTL_DELTAT], invdtreb_sq = f.own ? f.invdtreb_sq : g.ctl[CTL_INVDTREB],
               dts = scal[SC_DTSTELLAR];
  const unsigned long long mg = top[0], mp = top[1];
  long long shear = __double_as_longlong(1e30);
  for (int i = threadIdx.x; i < g.nr - 1; i += blockDim.x) {
    const double w = fabs(cr.vmoy[i] * g.r.InvRmed[i] - cr.vmoy[i + 1] * g.r.InvRmed[i + 1]);
    const long long dt = __double_as_longlong(div_fast(f.twopi_cfl_ns, w));
    if (dt >= 0 && dt < shear) shear = dt;
  }
  shear = block_reduce(shear, OpMinI64(), __double_as_longlong(1e30));
  if (threadIdx.x < 2) {                           // for the next call
    bound[threadIdx.x] = 0;
    top[threadIdx.x] = 0ULL;
  }
  if (threadIdx.x == 0) {
    const double dmg = __longlong_as_double((long long)mg), dmp = f.pebbles ? __longlong_as_double((long long)mp) : -1.0e30,
                 dshear = __longlong_as_double(shear);
    double newdt;
    if (!f.pebbles) newdt = div_fast(TH_CFLSECURITY, sqrt_fast(dmg + invdtreb_sq));
    else newdt = div_fast(TH_CFLSECURITY, sqrt_fast(dmg + dmp + invdtreb_sq));
    if (newdt > 1e30) newdt = 1e30;
    if (dshear < newdt) newdt = dshear;
    if (newdt > dts) {
      const double m = (1.0 * dts > f.minimum_step) ? 1.0 * dts : f.minimum_step;
      newdt = (newdt < m) ? newdt : m;
    }
    newdt = (newdt < f.maximum_step) ? newdt : f.maximum_step;
    if (f.first_call && f.first_step > 0.0) newdt = f.first_step;
    if (deltaT < newdt) newdt = deltaT;
    scal[SC_NEWDT] = newdt;
    scal[SC_INVDTPEB] = dmp;
    const int n = (int)(ceil(deltaT / newdt));
    iscal[IS_NSUB] = n;
    g.ctl[CTL_DT] = deltaT / (double)n;
  }
}

void aux_cfl(const DevGrid &g, const double *vr, const double *vt, const double *cs, const double *pvr, const double *pvt,
             const CflRings &cr, int pebbles, int fast, int viscous, double *part, const CflFinal &f0, double *scal,
             int *iscal, cudaStream_t s)
{
  if (pebbles && fast) aux_ring_means(g, vt, cr.vmoy, pvt, cr.pvtmed, 0, g.nr, s);
  else aux_ring_means(g, vt, cr.vmoy, nullptr, nullptr, 0, g.nr, s);
  float *upper = (float *)part;
  int *bound = iscal + IS_CFL_BOUND;
  unsigned long long *top = (unsigned long long *)(scal + SC_CFLTOP);
  // on small grids the FP64 of every cell takes less than a launch (128x384:
  // 3.4 us; 256x768: 13 us)
  if ((long long)g.nr * g.ns < (1 << 17)) upper = nullptr;
  if (upper) {
    launch(k_cfl_bounds, grid2d(g.ns, g.nr - 1, 256 * CFL_CPT), 256, 0, s, g, vr, vt, cs, pvr, pvt, cr, pebbles, fast,
                                                                      viscous, upper, bound);
    g_thorin_launches++;
  }
  launch(k_cfl_cells, grid2d(g.ns, g.nr - 1, 256), 256, 0, s, g, vr, vt, cs, pvr, pvt, cr, pebbles, fast, viscous, upper,
                                                          bound, top);
  g_thorin_launches++;
  launch(k_cfl_final, 1, 1024, 0, s, g, cr, f0, scal, iscal, bound, top);
  g_thorin_launches++;
}

// ---------------------------------------------------------------------------
// EvaporatePebbles (Pebbles.c:834-864).  One load and one comparison a cell but
// where it is hot, so a thread takes EVAP_CPT cells with an integer comparison
// (a cell a thread and FP64: 28 us on the 1024x3072 disk, now 11.5).
#define EVAP_CPT 8
__global__ void k_evaporate(DevGrid g, const double *__restrict__ T, double *__restrict__ pdens)
{
  pdl_wait();
  const double facc = g.ctl[CTL_FACC_EVAP];
  const int ns = g.ns, row = blockIdx.y * ns, j0 = blockIdx.x * (BX * EVAP_CPT) + threadIdx.x;
  double t[EVAP_CPT];
#pragma unroll
  for (int m = 0; m < EVAP_CPT; m++) t[m] = (j0 + m * BX < ns) ? T[row + j0 + m * BX] : 0.0;
  // T > evaptemp > 0 on the bits: a negative T is below, a NaN is not above
  const long long e = __double_as_longlong(g.k.evaptemp);
#pragma unroll
  for (int m = 0; m < EVAP_CPT; m++) {
    const int j = j0 + m * BX, l = row + j;
    const long long b = __double_as_longlong(t[m]);
    if (j < ns && (e > 0 ? b > e && b <= 0x7ff0000000000000LL : t[m] > g.k.evaptemp)) {
      asm volatile("" ::: "memory");               // a branch: under predicates the FP64 pipe is busy all the same
      double d = pdens[l] * (1.0 - facc);
      if (d < 1.0e-8) d = 1.0e-8;
      pdens[l] = d;
    }
  }
}

void aux_evaporate(const DevGrid &g, const double *T, double *pdens, cudaStream_t s)
{
  launch(k_evaporate, grid2d(g.ns, g.nr, BX * EVAP_CPT), BX, 0, s, g, T, pdens);
  g_thorin_launches++;
}

// ---------------------------------------------------------------------------
// Damping boundaries (DampingBoundary, SideEuler.c:368-419, and DampPebbles,
// SideEuler.c:423-456).  Only rings inside the damping zones are launched.
// pd: the pebbles in the same launch (NULL: not).
__device__ __forceinline__ void damp_peb_cell(const DevGrid &g, int i, int l, double dt, double omega_frame,
                                              double *pd, double *pvr, double *pvt)
{
  const double lambda = g.r.WaveKiller[i] * dt;
  const double d0 = g.r.PebDensInit[i], vr0 = g.r.PebVradInit[i];
  const double vt0 = g.r.PebVthetaInit[i] - g.r.Rmed[i] * omega_frame;
  pd[l] = div_fast(pd[l] + lambda * d0, 1.0 + lambda);
  pvr[l] = div_fast(pvr[l] + lambda * vr0, 1.0 + lambda);
  pvt[l] = div_fast(pvt[l] + lambda * vt0, 1.0 + lambda);
}

__global__ void k_damp_gas(DevGrid g, double *__restrict__ vrad, double *__restrict__ rho, double *__restrict__ vtheta,
                           double *__restrict__ energy, const int *__restrict__ rings, const double *__restrict__ vr0r,
                           int damp_init, int damp_flux, int energy_eq, double *__restrict__ pd,
                           double *__restrict__ pvr, double *__restrict__ pvt)
{
  pdl_wait();
  const double dt = g.ctl[CTL_DT], omega_frame = g.ctl[CTL_OMEGA_FRAME];
  const int ns = g.ns;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= ns) return;
  const int i = rings[blockIdx.y];
  const int l = j + i * ns;
  const double lambda = g.r.WaveKiller[i] * dt;
  const double vrad0 = damp_flux ? vr0r[i] : 0.0;
  vrad[l] = div_fast(vrad[l] + lambda * vrad0, 1.0 + lambda);
  if (damp_init) {
    const double rho0 = g.r.SigmaMed[i], e0 = g.r.EnergyMed[i];
    const double vt0 = g.r.VthetaMed[i] - g.r.Rmed[i] * omega_frame;
    rho[l] = div_fast(rho[l] + lambda * rho0, 1.0 + lambda);
    vtheta[l] = div_fast(vtheta[l] + lambda * vt0, 1.0 + lambda);
    if (energy_eq) energy[l] = div_fast(energy[l] + lambda * e0, 1.0 + lambda);
  }
  if (damp_flux) rho[l] = div_fast(rho[l] + lambda * g.r.SigmaMed[i], 1.0 + lambda);
  if (pd) damp_peb_cell(g, i, l, dt, omega_frame, pd, pvr, pvt);
}

void aux_damp_gas(const DevGrid &g, double *vrad, double *rho, double *vtheta, double *energy, const int *rings,
                  int nrings, const double *vr0r, int damp_init, int damp_flux, int energy_eq, double *pd, double *pvr,
                  double *pvt, cudaStream_t s)
{
  if (nrings <= 0) return;
  launch(k_damp_gas, grid2d(g.ns, nrings, BX), BX, 0, s, g, vrad, rho, vtheta, energy, rings, vr0r, damp_init, damp_flux,
         energy_eq, pd, pvr, pvt);
  g_thorin_launches++;
}

// Isothermal equation of state (ComputeSoundSpeed, ComputePressureField,
// ComputeTemperatureField without the energy equation, SourceEuler.c:
// 715-792): c_s is the ring profile AspectRatio(r) sqrt(G/r) r^f, P = Sigma
// c_s^2, T = mu P / (Sigma R).  Each part is done only when asked for: the
// reference forms P at the start of a substep and T from that P and the
// transported Sigma at its end.
__global__ void k_iso_eos(DevGrid g, const double *__restrict__ rho, const double *__restrict__ csr,
                          double *__restrict__ cs, double *__restrict__ press, double *__restrict__ temper, int set_cs,
                          int set_press, int set_temper)
{
  pdl_wait();
  const int ns = g.ns;
  CELL_LOOP_2D
  if (set_cs) cs[l] = csr[i];
  if (set_press) press[l] = rho[l] * cs[l] * cs[l];
  if (set_temper) temper[l] = (1.0 * press[l]) * div_fast(1.0, rho[l] * 1.0);
}

void aux_iso_eos(const DevGrid &g, const double *rho, const double *csr, double *cs, double *press, double *temper,
                 int set_cs, int set_press, int set_temper, cudaStream_t s)
{
  launch(k_iso_eos, grid2d(g.ns, g.nr, BX), BX, 0, s, g, rho, csr, cs, press, temper, set_cs, set_press, set_temper);
  g_thorin_launches++;
}

__global__ void k_damp_peb(DevGrid g, double *__restrict__ pd, double *__restrict__ pvr, double *__restrict__ pvt,
                           const int *__restrict__ rings)
{
  pdl_wait();
  const double dt = g.ctl[CTL_DT], omega_frame = g.ctl[CTL_OMEGA_FRAME];
  const int ns = g.ns;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= ns) return;
  const int i = rings[blockIdx.y];
  const int l = j + i * ns;
  damp_peb_cell(g, i, l, dt, omega_frame, pd, pvr, pvt);
}

void aux_damp_peb(const DevGrid &g, double *pd, double *pvr, double *pvt, const int *rings, int nrings, cudaStream_t s)
{
  if (nrings <= 0) return;
  launch(k_damp_peb, grid2d(g.ns, nrings, BX), BX, 0, s, g, pd, pvr, pvt, rings);
  g_thorin_launches++;
}

// DetectCrash (SourceEuler.c:48-66): any negative value in rows 0..nr-1.
__global__ void k_crash(int n, const double *__restrict__ f, int *flag)
{
  pdl_wait();
  int bad = 0;
  for (int l = blockIdx.x * blockDim.x + threadIdx.x; l < n; l += gridDim.x * blockDim.x)
    if (f[l] < 0.0) bad = 1;
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(flag, 1);
}

void aux_crash(const DevGrid &g, const double *f, int *flag, cudaStream_t s)
{
  const int n = g.nr * g.ns;
  int blocks = (n + 255) / 256;
  if (blocks > 1216) blocks = 1216;
  launch(k_crash, blocks, 256, 0, s, n, f, flag);
  g_thorin_launches++;
}

// ---------------------------------------------------------------------------
// FillForcesArrays (Pframeforce.c:43-510) in four kernels.
//
// k_force_rings, one block per ring: the ring-mean Stokes number, the scale
// heights of the ring means and the 10-node vertical average of the star's
// pull for the ring-mean column, one node per lane of the first warp.
// It also leaves the planets and control values of the host path (hp.n >= 0)
// for the kernels after it.
__global__ void __launch_bounds__(RING_T) k_force_rings(DevGrid g, ForceArgs a, ForceRings fr, HostPlanets hp)
{
  pdl_wait();
  if (blockIdx.x == 0 && hp.n >= 0) {
    const double *from = (const double *)hp.pl;
    double *to = (double *)a.pl_out;
    for (int k = threadIdx.x; k < hp.n * (int)(sizeof(DevPlanet) / sizeof(double)); k += RING_T) to[k] = from[k];
    if (threadIdx.x == 0) {
      g.ctl[CTL_MASS_TAPER] = hp.mass_taper;
      g.ctl[CTL_INDX_PL] = hp.indx;
      g.ctl[CTL_INDY_PL] = hp.indy;
    }
  }
  const int i = blockIdx.x, lane = threadIdx.x;
  const double H = g.r.csmean[i] * g.r.OmegaInv[i] * g.k.sqrt_adiabind_inv;
  const double r2 = g.r.Rmed2[i];
  double hc2 = 0.0;
  if (a.pebbles) {
    hc2 = ring_sum(a.tau + (size_t)i * g.ns, g.ns);
    if (lane >= 32) return;
    hc2 = div_fast(a.pebble_alpha, hc2 / (double)g.ns);
  }
  if (lane >= 32) return;
  const int m = lane < 10 ? lane : 9;
  const double z = ((double)m + 0.5) * (3.0 / 10.0) * H, z2 = z * z;
  double s = a.wq10[m] * pow_m32(r2 + z2);
  double p = a.wq10[m] * pow_m32(r2 + z2 * hc2);
  if (lane >= 10) s = p = 0.0;
  s = warp_reduce(s, OpAdd());
  p = warp_reduce(p, OpAdd());
  if (lane == 0) {
    fr.H_avr[i] = H;
    fr.p_H_avr[i] = a.pebbles ? H * sqrt(hc2) : 0.0;
    const double f = s * a.isig10 * g.r.Rmed[i];
    fr.agr0[i] = -f;
    fr.pagr0[i] = a.pebbles ? -(p * a.isig10 * g.r.Rmed[i]) : 0.0;
    fr.starw[i] = g.r.Surf[i] * f;
  }
}

struct ForceRing {
  double rm, surf, starw, agr0, pagr0, hc, H_avr, p_H_avr;
  float hcf, havf, phavf;
};

// Whether |x - m| / m > 0.05, x and m from FP32 when they decide it (the FP32
// values are within 1e-6 of the FP64 ones), else unknown (2).
__device__ __forceinline__ int off_by_5pc(float x, float m)
{
  const float d = fabsf(x - m);
  if (d > 0.05001f * m) return 1;
  if (d < 0.04999f * m) return 0;
  return 2;                                        // NaN as well
}

// k_forces: the accelerations of every cell whose scale height is within 5% of
// the ring mean's and which is not near a planet (s < 10 H_pl or 5 r_Hill):
// the star's pull is the ring's, a planet's is softened.  The other cells are
// marked for k_forces_near.  A thread walks the rings of one column: in the
// frame turned by the column's azimuth a planet lies at (pr, pt), the same for
// all rings, so a cell at radius r sees it at (pr - r, pt); the radial and
// azimuthal pull and the disk's pull on the planet need no rotation per cell,
// and the sums over the column are turned once.  About 28 FP64 instructions a
// cell with pebbles and a planet, where the form that worked in x and y took
// 94; bound by the FP64 pipe.
template <int NP>
__global__ void __launch_bounds__(128) k_forces(DevGrid g, ForceArgs a, ForceRings fr)
{
  pdl_wait();
  extern __shared__ char smem[];
  ForceRing *ring = (ForceRing *)smem;
  const double mass_taper = g.ctl[CTL_MASS_TAPER];
  const int full_mass = (mass_taper == 1.0) ? 1 : 0;
  const int ns = g.ns, peb = a.pebbles;
  const int np = (NP == MAXPL_DEV) ? a.npl : NP;
  const int i0 = blockIdx.y * a.rings_a, i1 = min(i0 + a.rings_a, g.nr);
  for (int q = threadIdx.x; q < i1 - i0; q += 128) {
    const int i = i0 + q;
    ForceRing &R = ring[q];
    R.rm = g.r.Rmed[i]; R.surf = g.r.Surf[i]; R.starw = fr.starw[i]; R.agr0 = fr.agr0[i];
    R.hc = g.r.OmegaInv[i] * g.k.sqrt_adiabind_inv;
    R.H_avr = fr.H_avr[i];
    R.hcf = (float)R.hc; R.havf = (float)R.H_avr;
    if (peb) { R.pagr0 = fr.pagr0[i]; R.p_H_avr = fr.p_H_avr[i]; R.phavf = (float)R.p_H_avr; }
  }
  __syncthreads();
  const int j = blockIdx.x * 128 + threadIdx.x;
  double star = 0.0;
  double W[NP > 0 ? NP : 1], Wu[NP > 0 ? NP : 1], pr[NP > 0 ? NP : 1], pt[NP > 0 ? NP : 1];
  double c = 0.0, s = 0.0;
#pragma unroll
  for (int k = 0; k < NP; k++) W[k] = Wu[k] = pr[k] = pt[k] = 0.0;
  if (j < ns) {
    c = g.r.costab[j];
    s = g.r.sintab[j];
    double m[NP > 0 ? NP : 1], zz[NP > 0 ? NP : 1], sm2[NP > 0 ? NP : 1], sma[NP > 0 ? NP : 1], pt2[NP > 0 ? NP : 1],
        lim[NP > 0 ? NP : 1];
#pragma unroll
    for (int k = 0; k < NP; k++) {
      if (k >= np) continue;
      const DevPlanet &P = a.pl[k];
      pr[k] = c * P.x + s * P.y;
      pt[k] = c * P.y - s * P.x;
      pt2[k] = pt[k] * pt[k];
      m[k] = P.m * mass_taper;
      zz[k] = P.z * P.z;
      sm2[k] = P.smoothing2;
      sma[k] = P.smoothing2 * a.pebble_alpha;
      lim[k] = (P.near_h2 > P.near_hill2) ? P.near_h2 : P.near_hill2;
      if (!full_mass) lim[k] = 0.0;
    }
    const float af = (float)a.pebble_alpha;
    for (int i = i0; i < i1; i++) {
      const ForceRing &R = ring[i - i0];
      const int l = j + i * ns;
      const double cs = a.cs[l], tau = peb ? a.tau[l] : 1.0;
      const float Hf = to_float_pos(cs) * R.hcf;
      int local = off_by_5pc(Hf, R.havf);
      if (local == 2) {
        const double H = cs * R.hc;
        local = (fabs(H - R.H_avr) > 0.05 * R.H_avr) ? 1 : 0;
      }
      if (peb && !local) {
        const float tf = to_float_pos(tau);
        local = (tf > 0.0f) ? off_by_5pc(Hf * sqrtf(__fdividef(af, tf)), R.phavf) : 2;
        if (local == 2) {
          const double pH = cs * R.hc * sqrt(a.pebble_alpha / tau);
          local = (fabs(pH - R.p_H_avr) > 0.05 * R.p_H_avr) ? 1 : 0;
        }
      }
      double u[NP > 0 ? NP : 1], s2[NP > 0 ? NP : 1];
#pragma unroll
      for (int k = 0; k < NP; k++) {
        if (k >= np) continue;
        u[k] = R.rm - pr[k];
        s2[k] = __fma_rn(u[k], u[k], pt2[k]);
        if (__double_as_longlong(s2[k]) < __double_as_longlong(lim[k])) local = 1;   // both >= 0
      }
      a.near[l] = (unsigned char)local;
      if (local) continue;
      const double rho = a.rho[l];
      star = __fma_rn(rho, R.starw, star);
      double ar = R.agr0, at = 0.0, par = 0.0, pat = 0.0;
      if (peb) par = R.pagr0;
      if (NP > 0) {
        const double mcell = rho * R.surf;
        const double itau = peb ? div_fast(1.0, tau) : 0.0;
#pragma unroll
        for (int k = 0; k < NP; k++) {
          if (k >= np) continue;
          const double sz = s2[k] + zz[k];
          const double id3 = pow_m32(sz + sm2[k]);
          const double mi = m[k] * id3, w = mcell * id3;
          ar = __fma_rn(-mi, u[k], ar);
          at = __fma_rn(mi, pt[k], at);
          W[k] += w;
          Wu[k] = __fma_rn(w, u[k], Wu[k]);
          if (peb) {
            const double ip3 = pow_m32(__fma_rn(sma[k], itau, sz));
            const double mp = m[k] * ip3;
            par = __fma_rn(-mp, u[k], par);
            pat = __fma_rn(mp, pt[k], pat);
            if (a.pebble_gravity) {
              const double wp = a.pdens[l] * R.surf * ip3;
              W[k] += wp;
              Wu[k] = __fma_rn(wp, u[k], Wu[k]);
            }
          }
        }
      }
      a.agr[l] = ar;
      a.agt[l] = at;
      if (peb) { a.pagr[l] = par; a.pagt[l] = pat; }
    }
  }
  const int b = blockIdx.x + blockIdx.y * gridDim.x, nb = a.nba + a.nbb;
  double v = block_reduce_smem<128>(star * c, OpAdd());
  if (threadIdx.x == 0) a.part[b] = v;
  v = block_reduce_smem<128>(star * s, OpAdd());
  if (threadIdx.x == 0) a.part[nb + b] = v;
#pragma unroll
  for (int k = 0; k < NP; k++) {
    if (k >= np) continue;
    const double t = W[k] * pt[k];
    v = block_reduce_smem<128>(c * Wu[k] + s * t, OpAdd());
    if (threadIdx.x == 0) a.part[(size_t)(2 + 2 * k) * nb + b] = v;
    v = block_reduce_smem<128>(s * Wu[k] - c * t, OpAdd());
    if (threadIdx.x == 0) a.part[(size_t)(3 + 2 * k) * nb + b] = v;
  }
}

// One quadrature node of a planet's potential (FillForcesArrays,
// Pframeforce.c:300-372): cubic-spline taper inside rst, softened 1/d^3.
__device__ __forceinline__ double planet_node(double s2, double dz, double mx, const DevPlanet &P)
{
  const double d2 = s2 + dz * dz;
  if (d2 < P.rst2) {
    const double dd = sqrt_fast(d2);
    return pow_m32(d2 + mx) * (div_fast(-3.0 * d2 * d2, P.rst4) + div_fast(4.0 * dd * d2, P.rst3));
  }
  return pow_m32(d2 + mx);
}

// Vertical quadrature of a planet's pull on one cell over NV nodes
// z_m = (m - 1/2) 3H/NV (Pframeforce.c:260-372).  A planet in the midplane
// (P.z = 0) outside whose taper the whole column lies needs only
// d2 = s2 + z_m^2 at each node.
template <int NV>
__device__ __forceinline__ double planet_quad(const double *wq, double H, double s2, double mx, const DevPlanet &P)
{
  double sum = 0.0;
  if (P.z == 0.0 && s2 >= P.rst2) {
    const double H2 = H * H, b = s2 + mx;
#pragma unroll
    for (int m = 0; m < NV; m++) {
      const double z = ((double)m + 0.5) * (3.0 / (double)NV);
      sum = __fma_rn(wq[m], pow_m32(__fma_rn(z * z, H2, b)), sum);
    }
    return sum;
  }
  const bool off = (P.z < -0.05 * H || P.z > 0.05 * H);
  const double deltaz = 3.0 * H / (double)NV;
  for (int m = 0; m < NV; m++) {
    const double z = ((double)m + 0.5) * deltaz;
    double f = planet_node(s2, z - P.z, mx, P);
    if (off) f += planet_node(s2, -z - P.z, mx, P);
    sum += wq[m] * f;
  }
  return off ? 0.5 * sum : sum;
}

// The same by a warp, a node per lane; every lane gets the sum.
__device__ __forceinline__ double planet_quad_warp(const double *wq, int nv, double H, double s2, double mx,
                                                   const DevPlanet &P)
{
  const int lane = threadIdx.x & 31;
  const bool off = (P.z < -0.05 * H || P.z > 0.05 * H);
  const double z = ((double)lane + 0.5) * (3.0 * H / (double)nv);
  double f = planet_node(s2, z - P.z, mx, P);
  if (off) f += planet_node(s2, -z - P.z, mx, P);
  f = (lane < nv) ? wq[lane < nv ? lane : 0] * f : 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) f += __shfl_xor_sync(TH_FULL, f, o);
  return off ? 0.5 * f : f;
}

// r^3 times the star's vertical sum over nv nodes as a series in q = (H/r)^2,
// or node by node in columns too thick for it.
__device__ __forceinline__ double star_quad(const double *wq, const double *ck, int nv, double q)
{
  if (q <= FORCE_QMAX) {
    double v = ck[FORCE_NC - 1];
#pragma unroll
    for (int k = FORCE_NC - 2; k >= 0; k--) v = __fma_rn(v, q, ck[k]);
    return v;
  }
  double v = 0.0;
  for (int m = 0; m < nv; m++) {
    const double z = ((double)m + 0.5) * (3.0 / (double)nv);
    v += wq[m] * pow_m32(1.0 + z * z * q);
  }
  return v;
}

// Whether the cell at (x, y) lies within two Hill radii of planet P, where the
// vertical quadrature takes 30 nodes.  Rounded operations, so that every
// kernel decides alike.
__device__ __forceinline__ bool in_hill(double x, double y, const DevPlanet &P)
{
  const double dx = __dsub_rn(x, P.x), dy = __dsub_rn(y, P.y);
  return __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)) < P.rmorevert2;
}

// One of k_forces_near's cells with the NV-node vertical quadrature, by a
// thread (WARP false, NV = 10) or by a warp whose lanes hold the nodes (NV =
// 30; lane 0 writes and adds to acc).
template <int NV, bool WARP>
__device__ __forceinline__ void near_cell(const DevGrid &g, const ForceArgs &a, const ForceRings &fr, int i, int j,
                                          double mass_taper, int full_mass, const double *wq, const double *ck,
                                          double isig, double *acc)
{
  const int l = j + i * g.ns, peb = a.pebbles;
  const bool add = !WARP || (threadIdx.x & 31) == 0;
  const double c = g.r.costab[j], s = g.r.sintab[j], rm = g.r.Rmed[i], ir = g.r.InvRmed[i];
  const double x = rm * c, y = rm * s;
  const double H = a.cs[l] * (g.r.OmegaInv[i] * g.k.sqrt_adiabind_inv), H2 = H * H;
  const double mcell = a.rho[l] * g.r.Surf[i];
  const double hc2 = peb ? div_fast(a.pebble_alpha, a.tau[l]) : 0.0;
  const double q = H2 * (ir * ir), ir2 = ir * ir * isig;
  const double f = star_quad(wq, ck, NV, q) * ir2;             // r sum_m w_m (r^2 + z_m^2)^(-3/2) / sigma
  double ax = 0.0, ay = 0.0, pax = 0.0, pay = 0.0, par = 0.0;
  if (add) {
    acc[0] += mcell * f * c;
    acc[1] += mcell * f * s;
  }
  if (peb) par = -star_quad(wq, ck, NV, q * hc2) * ir2;
  for (int k = 0; k < a.npl; k++) {
    const DevPlanet P = a.pl[k];
    const double dx = x - P.x, dy = y - P.y;
    const double s2 = dx * dx + dy * dy;
    double id3, ip3 = 0.0, mpl = P.m, hillcut = 1.0;
    if (full_mass && (s2 < P.near_h2 || s2 < P.near_hill2)) {
      if (a.exclude_hill) {
        const double d2 = s2 + P.z * P.z;
        hillcut = 1.0 / (exp(-(sqrt(d2) / P.rhill - a.hillcut) / a.hillcut * 10.0) + 1.0);
      }
      const double mx = (P.rsm2 > fr.drsq[i]) ? P.rsm2 : fr.drsq[i];
      if (WARP) {
        id3 = planet_quad_warp(wq, NV, H, s2, mx, P) * isig;
        if (peb) ip3 = planet_quad_warp(wq, NV, H * sqrt_fast(hc2), s2, mx, P) * isig;
      } else {
        id3 = planet_quad<NV>(wq, H, s2, mx, P) * isig;
        if (peb) ip3 = planet_quad<NV>(wq, H * sqrt_fast(hc2), s2, mx, P) * isig;
      }
    } else {
      mpl *= mass_taper;
      const double sz = s2 + P.z * P.z;
      id3 = pow_m32(sz + P.smoothing2);
      if (peb) ip3 = pow_m32(sz + P.smoothing2 * hc2);
    }
    double tx = dx * id3, ty = dy * id3;
    ax -= mpl * tx;
    ay -= mpl * ty;
    if (add) {
      acc[2 + 2 * k] += mcell * (tx * hillcut);
      acc[3 + 2 * k] += mcell * (ty * hillcut);
    }
    if (peb) {
      tx = dx * ip3; ty = dy * ip3;
      pax -= mpl * tx;
      pay -= mpl * ty;
      if (a.pebble_gravity && add) {
        const double pm = a.pdens[l] * g.r.Surf[i];
        acc[2 + 2 * k] += pm * (tx * hillcut);
        acc[3 + 2 * k] += pm * (ty * hillcut);
      }
    }
  }
  if (!add) return;
  a.agr[l] = c * ax + s * ay - f;
  a.agt[l] = c * ay - s * ax;
  if (peb) {
    a.pagr[l] = c * pax + s * pay + par;
    a.pagt[l] = c * pay - s * pax;
  }
}

// k_forces_near: the cells k_forces left out, with the vertical quadrature of
// the star's pull and of the planets near the cell: about 180 FP64
// instructions a cell for 10 nodes and one planet (370 before the star's
// series and the shorter powers).  They lie together around the planets (7% of
// the cells for one planet at r = 1), so the kernel has its own grid, with few
// rings per block.  The cells within two Hill radii take 30 nodes, and the
// taper next to the planet: a few hundred cells whose chains of dependent
// FP64 instructions would hold up the rest, so the last blocks take them, a
// warp per cell and a node per lane (cells w, w + W, ... of the annulus, 32
// tested at a time).  512x1536: 70 us (238 us with two rings per thread and
// the 30-node cells among the others); with k_forces' 66 us, 136 us where one
// kernel for all cells took 340.
__global__ void __launch_bounds__(128) k_forces_near(DevGrid g, ForceArgs a, ForceRings fr)
{
  pdl_wait();
  const double mass_taper = g.ctl[CTL_MASS_TAPER];
  const int full_mass = (mass_taper == 1.0) ? 1 : 0;
  const int ns = g.ns;
  const int nq = 2 + 2 * a.npl, nb = a.nba + a.nbb, b = a.nba + blockIdx.x;
  double acc[2 + 2 * MAXPL_DEV];
  for (int q = 0; q < nq; q++) acc[q] = 0.0;
  int any = 0;
  if ((int)blockIdx.x < a.nbn) {
    const int nbx = (ns + 127) / 128, by = blockIdx.x / nbx;
    const int j = (blockIdx.x - by * nbx) * 128 + threadIdx.x;
    const int i0 = by * a.rings_b, i1 = min(i0 + a.rings_b, g.nr);
    if (j < ns) {
      const double c = g.r.costab[j], s = g.r.sintab[j];
      for (int i = i0; i < i1; i++) {
        if (!a.near[j + i * ns]) continue;
        const double x = __dmul_rn(g.r.Rmed[i], c), y = __dmul_rn(g.r.Rmed[i], s);
        bool hill = false;
        for (int k = 0; k < a.npl; k++) hill = hill || in_hill(x, y, a.pl[k]);
        if (hill) continue;
        any = 1;
        near_cell<10, false>(g, a, fr, i, j, mass_taper, full_mass, a.wq10, a.c10, a.isig10, acc);
      }
    }
  } else {
    const int lane = threadIdx.x & 31, nw = (a.nbb - a.nbn) * 4;
    const int gw = (blockIdx.x - a.nbn) * 4 + (threadIdx.x >> 5);
    for (int k = 0; k < a.npl; k++) {
      const DevPlanet &P = a.pl[k];
      if (!(P.rmorevert2 > 0.0)) continue;
      // rings that reach within two Hill radii of the planet's radius: from the
      // first with Rsup >= rp - rh to the last with Rinf <= rp + rh, counted by the
      // lanes (radii are positive, so their bits compare as integers); two
      // bisections were 20 dependent loads, a third of the kernel on a small disk
      const double rp = sqrt(P.x * P.x + P.y * P.y), rh = 2.001 * P.rhill;
      const long long below = __double_as_longlong(rp - rh), above = __double_as_longlong(rp + rh);
      int imin = 0, lo = 0;
      for (int i = lane; i < g.nr; i += 32) {
        imin += __double_as_longlong(g.r.Rsup[i]) < below ? 1 : 0;
        lo += __double_as_longlong(g.r.Rinf[i]) <= above ? 1 : 0;
      }
      imin = __reduce_add_sync(TH_FULL, imin);
      lo = __reduce_add_sync(TH_FULL, lo);
      const long long ncells = (long long)(lo - imin) * ns;
      for (long long base = gw; base < ncells; base += 32LL * nw) {   // warp-uniform
        const long long q = base + (long long)lane * nw;
        int i = 0, j = 0;
        bool mine = false;
        if (q < ncells) {
          i = imin + (int)(q / ns);
          j = (int)(q - (q / ns) * ns);
          if (a.near[j + i * ns]) {
            const double x = __dmul_rn(g.r.Rmed[i], g.r.costab[j]), y = __dmul_rn(g.r.Rmed[i], g.r.sintab[j]);
            mine = in_hill(x, y, P);
            for (int k2 = 0; k2 < k; k2++) mine = mine && !in_hill(x, y, a.pl[k2]);
          }
        }
        unsigned bal = __ballot_sync(TH_FULL, mine);
        while (bal) {
          const int src = __ffs(bal) - 1;
          bal &= bal - 1u;
          any = 1;
          near_cell<30, true>(g, a, fr, __shfl_sync(TH_FULL, i, src), __shfl_sync(TH_FULL, j, src), mass_taper,
                              full_mass, a.wq30, a.c30, a.isig30, acc);
        }
      }
    }
  }
  if (!__syncthreads_or(any)) {
    if (threadIdx.x < nq) a.part[(size_t)threadIdx.x * nb + b] = 0.0;
    return;
  }
  // a warp per quantity adds the threads' values
  extern __shared__ double near_sums[];              // [nq][128]
  for (int q = 0; q < nq; q++) near_sums[q * 128 + threadIdx.x] = acc[q];
  __syncthreads();
  for (int q = threadIdx.x >> 5; q < nq; q += 4) {
    const double *v = near_sums + q * 128 + (threadIdx.x & 31);
    const double t = warp_reduce((v[0] + v[32]) + (v[64] + v[96]), OpAdd());
    if ((threadIdx.x & 31) == 0) a.part[(size_t)q * nb + b] = t;
  }
}

// The sums over the blocks in a fixed order, one block per quantity, and, by
// the last of them, the indirect term (Pframeforce.c:488-509): in the frame
// of a column it is (c ax + s ay, c ay - s ax) at every radius, so it is kept
// per column, the azimuthal part as the mean of the columns either side of a
// cell's left face, and added where the accelerations are used (a pass over
// four fields and 14 FP64 instructions a cell before).
__global__ void __launch_bounds__(1024) k_forces_final(DevGrid g, ForceArgs a, double *__restrict__ scal)
{
  pdl_wait();
  __shared__ bool last;
  const int q = blockIdx.x, nb = a.nba + a.nbb;
  const double *p = a.part + (size_t)q * nb;
  double s = 0.0;
  for (int b = threadIdx.x; b < nb; b += 1024) s += p[b];
  s = block_reduce_smem<1024>(s, OpAdd());
  if (threadIdx.x == 0) {
    scal[q == 0 ? SC_INDX : q == 1 ? SC_INDY : SC_PLANET_A + (q - 2)] = (q < 2) ? -s : s;
    __threadfence();
    last = (atomicAdd(a.ticket, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (threadIdx.x == 0) *a.ticket = 0u;
  const double axi = __ldcg(scal + SC_INDX) + g.ctl[CTL_INDX_PL], ayi = __ldcg(scal + SC_INDY) + g.ctl[CTL_INDY_PL];
  const int ns = g.ns;
  for (int j = threadIdx.x; j < ns; j += 1024) {
    const double c = g.r.costab[j], sn = g.r.sintab[j];
    const int jm = (j == 0) ? ns - 1 : j - 1;
    a.col[j] = c * axi + sn * ayi;
    a.col[ns + j] = 0.5 * ((c + g.r.costab[jm]) * ayi - (sn + g.r.sintab[jm]) * axi);
  }
}

template <int NP>
static void launch_forces(const DevGrid &g, const ForceArgs &a, const ForceRings &fr, dim3 grid, cudaStream_t s)
{
  launch(k_forces<NP>, grid, 128, a.rings_a * sizeof(ForceRing), s, g, a, fr);
}

// Blocks of the force kernels.
struct ForceShape { int nbx, rings_a, rings_b, nba, nbn, nbb; };

static ForceShape force_shape(const DevGrid &g, int npl)
{
  // rings per block: the chunk with the least work on the busiest
  // multiprocessor, which runs four blocks at a time and uses 1 - (1 - n / 4)^2
  // of the FP64 pipe with n of them left, the ring and planet constants and the
  // block sums counted as two rings.  24x72 16.6 -> 9.4 us, 128x384 17.3 -> 11.5,
  // 512x1536 65.7 -> 61, 1024x3072 243 -> 224 (some six blocks a multiprocessor and
  // at least four rings before).  For the near cells at most four rings, as all
  // their work may lie in a few chunks
  ForceShape q;
  q.nbx = (g.ns + 127) / 128;
  q.rings_a = 1;
  double best = 1e300;
  for (int r = 1; r <= 32; r++) {
    const int n = (q.nbx * ((g.nr + r - 1) / r) + g.nsm - 1) / g.nsm, part = n & 3;
    const double u = 1.0 - 0.25 * part, w = ((n - part) + (part ? part / (1.0 - u * u) : 0.0)) * (r + 2);
    if (w < best) { best = w; q.rings_a = r; }
  }
  const int rb = (int)((long long)g.nr * q.nbx / (g.nsm * 40));
  q.rings_b = rb < 1 ? 1 : (rb > 4 ? 4 : rb);
  q.nba = q.nbx * ((g.nr + q.rings_a - 1) / q.rings_a);
  q.nbn = q.nbx * ((g.nr + q.rings_b - 1) / q.rings_b);
  q.nbb = q.nbn + (npl > 0 ? g.nsm : 0);
  return q;
}

int aux_forces(const DevGrid &g, const ForceArgs &a0, const ForceRings &fr, const HostPlanets &hp, double *scal,
               cudaStream_t s)
{
  ForceArgs a = a0;
  for (int pass = 0; pass < 2; pass++) {
    const int nv = pass ? 30 : 10;
    double *w = pass ? a.wq30 : a.wq10, *ck = pass ? a.c30 : a.c10, sig = 0.0;
    const double deltaz = 3.0 / (double)nv;          // H = 1
    for (int k = 0; k < FORCE_NC; k++) ck[k] = 0.0;
    for (int m = 1; m <= nv; m++) {
      const double z = ((double)m - 0.5) * deltaz;
      w[m - 1] = exp(-(0.5 * (z * z)));
      sig += w[m - 1];
      double t = w[m - 1];
      for (int k = 0; k < FORCE_NC; k++) {           // binomial(-3/2, k) w_m z_m^2k
        ck[k] += t;
        t *= z * z * (-1.5 - k) / (k + 1.0);
      }
    }
    if (pass) a.isig30 = 1.0 / sig;
    else a.isig10 = 1.0 / sig;
  }
  const ForceShape q = force_shape(g, a.npl);
  if ((size_t)(2 + 2 * a.npl) * (q.nba + q.nbb) > a.part_size) return THORIN_ERR_NOMEM;
  a.rings_a = q.rings_a;
  a.rings_b = q.rings_b;
  a.nba = q.nba;
  a.nbn = q.nbn;
  a.nbb = q.nbb;
  const dim3 ga(q.nbx, q.nba / q.nbx);
  launch(k_force_rings, g.nr, RING_T, 0, s, g, a, fr, hp);
  g_thorin_launches++;
  switch (a.npl) {
  case 0: launch_forces<0>(g, a, fr, ga, s); break;
  case 1: launch_forces<1>(g, a, fr, ga, s); break;
  case 2: launch_forces<2>(g, a, fr, ga, s); break;
  case 3: launch_forces<3>(g, a, fr, ga, s); break;
  default: launch_forces<MAXPL_DEV>(g, a, fr, ga, s); break;
  }
  g_thorin_launches++;
  launch(k_forces_near, a.nbb, 128, (2 + 2 * a.npl) * 128 * sizeof(double), s, g, a, fr);
  g_thorin_launches++;
  launch(k_forces_final, 2 + 2 * a.npl, 1024, 0, s, g, a, scal);
  g_thorin_launches++;
  return THORIN_OK;
}

// ---------------------------------------------------------------------------
// AccretePebblesOntoPlanets for one planet (Pebbles.c:353-539).  The annulus
// [imin, imax] holding the Hill sphere is searched; cells within
// the effective accretion radius give up pebbles up to the model rate.

// Trapzd and IntegrateColumnMass (Pebbles.c:302-349) for one cell, evaluated
// by a whole warp.  Levels 2 to 6, before which the reference makes no exit
// test that can pass, have 1, 2, 4, 8 and 16 midpoints: level n's are taken
// at once by the lanes 2^(n-2) to 2^(n-1) - 1 and the lower end by lane 0, so
// five levels cost one exponential a lane and one butterfly (with a pass each
// they were most of the 22 us of this kernel).  From level 7 on the 2^(n-2)
// midpoints are spread over the lanes.  Point j is a + (j + 1/2) spacing and
// a level's sum an xor butterfly over its lanes' partial sums, so every lane
// holds the same bits of the integral and takes the same exit.  The levels,
// the refinement integral = (integral + (b - a) sum / it) / 2 and the exit
// test after level 5 are the reference's (1 / it is exact); only the order of
// the midpoint sum and the rounding of the abscissae differ from its
// sequential loop (x += spacing), by relative amounts of order 1e-16.
__device__ double column_mass_warp(double a, double b, double Hpeb)
{
  const int lane = threadIdx.x & 31;
  const double H2 = Hpeb * Hpeb, w = b - a;
  const int own = (lane == 0) ? 1 : 1 << (31 - __clz(lane));      // points of the lane's level
  double x = (lane == 0) ? a : a + ((double)(lane - own) + 0.5) * (w * (1.0 / own));
  double sum = exp(div_fast(-0.5 * x * x, H2));
  double fb = __shfl_sync(TH_FULL, sum, 0);
  double integral = fb;
  if (a != -b) fb = exp(div_fast(-0.5 * b * b, H2));
  integral = 0.5 * w * (integral + fb);
#pragma unroll
  for (int o = 1; o < 16; o <<= 1) {
    const double t = __shfl_xor_sync(TH_FULL, sum, o);
    if (own > o) sum += t;
  }
  double iold = integral;
#pragma unroll
  for (int n = 2; n <= 6; n++) {
    const double it_inv = 1.0 / (double)(1 << (n - 2));
    iold = integral;
    integral = 0.5 * (integral + w * __shfl_sync(TH_FULL, sum, 1 << (n - 2)) * it_inv);
  }
  for (int n = 7; n <= 17; n++) {
    if (fabs(integral - iold) < 1.0e-4 * fabs(iold) || (integral == 0.0 && iold == 0.0)) return integral;
    if (n > 16) break;
    const int it = 1 << (n - 2);
    const double it_inv = ldexp(1.0, 2 - n), spacing = w * it_inv;
    sum = 0.0;
    for (int j = lane; j < it; j += 32) {
      x = a + ((double)j + 0.5) * spacing;
      sum += exp(div_fast(-0.5 * x * x, H2));
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) sum += __shfl_xor_sync(TH_FULL, sum, o);
    iold = integral;
    integral = 0.5 * (integral + w * sum * it_inv);
  }
  return __longlong_as_double(0x7ff8000000000000ULL);   // the reference aborts here
}

// The annulus work runs in three launches on many blocks (mean Stokes number,
// upper limits per cell, application of the limiter); the block that finishes
// last sums the block partials in a fixed order and does the scalar steps of
// the reference.  A launch on a small disk is mostly latency: the nine
// launches before this, with the arguments, the ring means and each sum a
// launch of its own, took 91 us of a substep at 128x384, these take
// 51 (a third of it the copy of the result and the wait for it).
// acc[] scalars: 0 Reff, 1 vrel, 2 Mt, 3 limiter, 4-5 the ring means.

// Sums of N values over a block of BS threads, valid in every thread: a warp
// per value adds the threads' (the warps' FP64 instructions go side by side,
// where block reductions one after another took 10 N of them in line, 64 cycles
// each in a warp that is alone).
template <int N, int BS>
__device__ __forceinline__ void acc_block_sums(double v[N])
{
  __shared__ double sh[N][BS];
  __shared__ double out[N];
#pragma unroll
  for (int k = 0; k < N; k++) sh[k][threadIdx.x] = v[k];
  __syncthreads();
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (w < N) {
    double a = sh[w][lane];
#pragma unroll
    for (int q = 1; q < BS / 32; q++) a += sh[w][lane + 32 * q];
    a = warp_reduce(a, OpAdd());
    if (lane == 0) out[w] = a;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < N; k++) v[k] = out[k];
}

__device__ __forceinline__ bool acc_last_block(unsigned int *ticket)
{
  __shared__ bool last;
  if (threadIdx.x == 0) {
    __threadfence();
    last = (atomicAdd(ticket, 1u) == gridDim.x - 1);
    if (last) *ticket = 0u;
  }
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// Sum over the annulus of the Stokes number by all blocks but two, which form
// the ring means of v_theta at the two rings bracketing the planet; then the
// effective accretion radius (Pebbles.c:375-437).  With SET the arguments come
// by value and are left for the other two kernels.
template <bool SET>
__global__ void __launch_bounds__(RING_T) k_acc_reff(DevGrid g, AccArgs av, AccArgs *ap)
{
  pdl_wait();
  const AccArgs &a = SET ? av : *ap;
  if (a.nb == 0) return;                         // no annulus (only the device-resident DT launches this)
  const int ns = g.ns, ncells = (a.imax - a.imin + 1) * ns, nb = gridDim.x - 2;
  if (blockIdx.x >= 2) {
    const double *tau = a.tau + (size_t)a.imin * ns;
    double t = 0.0;
    for (int q = (blockIdx.x - 2) * RING_T + threadIdx.x; q < ncells; q += nb * RING_T) t += tau[q];
    acc_block_sums<1, RING_T>(&t);
    if (threadIdx.x == 0) a.part[blockIdx.x - 2] = t;
  } else {
    const int i = a.iflow + blockIdx.x;          // vt1D[nrad] is zero in the reference
    double m = 0.0;
    if (i >= 0 && i < g.nr) m = ring_sum(a.vt + (size_t)i * ns, ns);
    if (threadIdx.x == 0) a.acc[4 + blockIdx.x] = m / (double)ns;
    if (SET && threadIdx.x == 0 && blockIdx.x == 0) *ap = av;
  }
  if (!acc_last_block(a.ticket)) return;
  double ts = 0.0;
  for (int b = threadIdx.x; b < nb; b += RING_T) ts += __ldcg(a.part + b);
  acc_block_sums<1, RING_T>(&ts);
  if (threadIdx.x == 0) {
    const double tau_mean = div_fast(ts, (double)ncells);
    const double flow = __ldcg(a.acc + 4) * (1.0 - a.frac) + __ldcg(a.acc + 5) * a.frac + a.Rp * a.omega_frame;
    const double flowx = div_fast(-flow * a.Yp, a.Rp), flowy = div_fast(flow * a.Xp, a.Rp);
    const double vrel =
        sqrt_fast((a.VXp - flowx) * (a.VXp - flowx) + (a.VYp - flowy) * (a.VYp - flowy) + a.VZp * a.VZp);
    const double Mt = div_fast(sqrt(1.0 / 3.0) * cube_rn(vrel), a.Omegap);
    double Reff;
    if (a.Mp < Mt) {
      const double Rbondi = div_fast(div_fast(a.Mp, vrel), vrel), tbondi = div_fast(Rbondi, vrel);
      Reff = Rbondi * sqrt_fast(div_fast(tau_mean * a.Rp15, tbondi));
    } else {
      Reff = a.Rhill * pow(div_fast(tau_mean, 0.1), 1.0 / 3.0);
    }
    if (Reff > a.Rhill) Reff = a.Rhill;
    a.acc[0] = Reff;
    a.acc[1] = vrel;
    a.acc[2] = Mt;
  }
}

// Annulus cell q (0 .. (imax - imin + 1) ns - 1) of the accretion step: true
// when its midplane distance to the planet is within the effective accretion
// radius, with the pebble scale height and the column's ends inside the
// sphere (Pebbles.c:445-453).
__device__ __forceinline__ bool acc_cell(const DevGrid &g, const AccArgs &a, int q, int &i, int &l, double &Hpeb,
                                         double &zmin, double &zmax)
{
  const int ns = g.ns;
  i = a.imin + q / ns;
  const int j = q - (q / ns) * ns;
  l = j + i * ns;
  const double Reff = a.acc[0], Reff2 = __dmul_rn(Reff, Reff);
  const double dx = __dsub_rn(__dmul_rn(g.r.Rmed[i], g.r.costab[j]), a.Xp);
  const double dy = __dsub_rn(__dmul_rn(g.r.Rmed[i], g.r.sintab[j]), a.Yp);
  const double R2 = __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
  if (!(R2 <= Reff2)) return false;
  const double H = __dmul_rn(__dmul_rn(a.cs[l], g.r.OmegaInv[i]), g.k.sqrt_adiabind_inv);
  Hpeb = __dmul_rn(H, sqrt_fast(div_fast(a.pebble_alpha, a.tau[l])));
  const double h = sqrt_fast(__dsub_rn(Reff2, R2));
  zmin = __dsub_rn(a.Zp, h);
  zmax = __dadd_rn(a.Zp, h);
  return true;
}

// Upper limit of the mass each annulus cell inside the sphere can give up
// (Pebbles.c:454-462) into macc[l] (zero outside the accretion step), with
// its column integral (IntegrateColumnMass of Pebbles.c:456) by one warp per
// cell, and the limiter from the sums of the limit, the scale height, the
// pebble density and the cell count.  Warp w of the grid takes the annulus
// cells w, w + W, w + 2W, ... (W warps in all), 32 of them tested at a time,
// so the cells of the sphere, which lie together around the planet, fall on
// many multiprocessors.
__global__ void __launch_bounds__(ACC_BX) k_acc_upper(DevGrid g, const AccArgs *__restrict__ ap)
{
  pdl_wait();
  const AccArgs &a = *ap;
  if (a.nb == 0) return;                         // no annulus
  const int ncells = (a.imax - a.imin + 1) * g.ns;
  const int lane = threadIdx.x & 31;
  const int nw = gridDim.x * (ACC_BX / 32);
  const int gw = blockIdx.x * (ACC_BX / 32) + (threadIdx.x >> 5);
  double v[4] = {0.0, 0.0, 0.0, 0.0};            // limit, scale height, pebble density, cells
  for (long long base = gw; base < ncells; base += 32LL * nw) {   // warp-uniform
    const long long c = base + (long long)lane * nw;
    int i = 0, l = 0;
    double Hpeb = 0.0, zmin = 0.0, zmax = 0.0, cm = 0.0;
    const bool inside = c < ncells && acc_cell(g, a, (int)c, i, l, Hpeb, zmin, zmax);
    unsigned bal = __ballot_sync(TH_FULL, inside);
    while (bal) {
      const int src = __ffs(bal) - 1;
      bal &= bal - 1u;
      const double m = column_mass_warp(__shfl_sync(TH_FULL, zmin, src), __shfl_sync(TH_FULL, zmax, src),
                                        __shfl_sync(TH_FULL, Hpeb, src));
      if (lane == src) cm = m;
    }
    if (inside) {
      const double pd = a.pdens[l];
      const double mcell = g.r.Surf[i] * pd;
      const double vdp = div_fast(pd, Hpeb) * g.k.sqrt2pi_inv;
      double dM = vdp * g.r.Surf[i] * cm;
      if (dM > mcell) dM = 0.99999999 * mcell;
      a.macc[l] = dM;
      v[0] += dM; v[1] += Hpeb; v[2] += pd; v[3] += 1.0;
    }
  }
  if (__syncthreads_or(v[3] > 0.0)) acc_block_sums<4, ACC_BX>(v);
  if (threadIdx.x == 0)
    for (int k = 0; k < 4; k++) a.part[4 * blockIdx.x + k] = v[k];
  if (!acc_last_block(a.ticket)) return;
  const int nb = gridDim.x;
  for (int k = 0; k < 4; k++) v[k] = 0.0;
  for (int b = threadIdx.x; b < nb; b += ACC_BX)
    for (int k = 0; k < 4; k++) v[k] += __ldcg(a.part + 4 * b + k);
  acc_block_sums<4, ACC_BX>(v);
  if (threadIdx.x == 0) {
    const double dmu = v[0];
    double Hpeb_mean = v[1], pdens_mean = v[2];
    const int nc = (int)v[3];
    if (nc > 0) { Hpeb_mean = div_fast(Hpeb_mean, (double)nc); pdens_mean = div_fast(pdens_mean, (double)nc); }
    const double Reff = a.acc[0], vrel = a.acc[1], Mt = a.acc[2];
    const double veloc = (a.Mp < Mt) ? vrel : Reff * a.Omegap;
    double dM_model;
    if (Hpeb_mean < Reff) dM_model = 2.0 * Reff * veloc * pdens_mean;
    else dM_model = div_fast(TH_PI * Reff * Reff * veloc * pdens_mean, Hpeb_mean) * g.k.sqrt2pi_inv;
    dM_model *= a.dt;
    a.acc[3] = (dmu > dM_model) ? div_fast(dM_model, dmu) : 1.0;
  }
}

// The accreted mass out of the cells (Pebbles.c:479-520) and its sum and
// momentum.
__global__ void __launch_bounds__(ACC_BX) k_acc_apply(DevGrid g, const AccArgs *__restrict__ ap, double *__restrict__ scal)
{
  pdl_wait();
  const AccArgs &a = *ap;
  if (a.nb == 0) return;                         // no annulus
  const int ns = g.ns;
  const int ncells = (a.imax - a.imin + 1) * ns;
  const double limiter = a.acc[3];
  double v[3] = {0.0, 0.0, 0.0};                 // mass and momentum
  for (int q = blockIdx.x * ACC_BX + threadIdx.x; q < ncells; q += gridDim.x * ACC_BX) {
    const int i = a.imin + q / ns, j = q - (q / ns) * ns, l = j + i * ns;
    const double up = a.macc[l];
    if (up > 0.0) {
      const double xc = g.r.Rmed[i] * g.r.costab[j], yc = g.r.Rmed[i] * g.r.sintab[j];
      const double vtcorr = g.r.Rmed[i] * a.omega_frame;
      const double vrc = a.pvr[l], vtc = a.pvt[l] + vtcorr;
      const double vxc = (vrc * xc - vtc * yc) * g.r.InvRmed[i], vyc = (vrc * yc + vtc * xc) * g.r.InvRmed[i];
      const double dM = up * limiter;
      a.macc[l] = 0.0;
      const double mcell = g.r.Surf[i] * a.pdens[l];
      double pd = div_fast(mcell - dM, g.r.Surf[i]);
      if (pd < 0.0) pd = 1.e-20;
      a.pdens[l] = pd;
      v[0] += dM; v[1] += dM * vxc; v[2] += dM * vyc;
    }
  }
  if (__syncthreads_or(v[0] != 0.0)) acc_block_sums<3, ACC_BX>(v);
  if (threadIdx.x == 0)
    for (int k = 0; k < 3; k++) a.part[3 * blockIdx.x + k] = v[k];
  if (!acc_last_block(a.ticket)) return;
  const int nb = gridDim.x;
  for (int k = 0; k < 3; k++) v[k] = 0.0;
  for (int b = threadIdx.x; b < nb; b += ACC_BX)
    for (int k = 0; k < 3; k++) v[k] += __ldcg(a.part + 3 * b + k);
  acc_block_sums<3, ACC_BX>(v);
  if (threadIdx.x == 0) { scal[SC_ACC_DM] = v[0]; scal[SC_ACC_DPX] = v[1]; scal[SC_ACC_DPY] = v[2]; }
}

int aux_accrete_blocks(const DevGrid &g, int imin, int imax)
{
  const int ncells = (imax - imin + 1) * g.ns;
  return (ncells + ACC_BX - 1) / ACC_BX;
}

void aux_accrete(const DevGrid &g, const AccArgs *a0, AccArgs *a_dev, int nb, double *scal, cudaStream_t s)
{
  const int grid = nb < 2 * g.nsm ? nb : 2 * g.nsm;
  if (a0) launch(k_acc_reff<true>, 2 + grid, RING_T, 0, s, g, *a0, a_dev);
  else launch(k_acc_reff<false>, 2 + grid, RING_T, 0, s, g, AccArgs(), a_dev);
  g_thorin_launches++;
  launch(k_acc_upper, 2 * g.nsm, ACC_BX, 0, s, g, a_dev);
  g_thorin_launches++;
  launch(k_acc_apply, grid, ACC_BX, 0, s, g, a_dev, scal);
  g_thorin_launches++;
}

// ---------------------------------------------------------------------------
// Conservation integrals: a block per ring (integral_ring), the rings' sums by
// the block that finishes last.
template <bool PEB>
__global__ void __launch_bounds__(RING_T) k_integrals(DevGrid g, const double *__restrict__ rho, const double *__restrict__ vr,
                                                      const double *__restrict__ vt, const double *__restrict__ e,
                                                      const double *__restrict__ pd, const double *__restrict__ pvt,
                                                      double omega_frame, double *__restrict__ part,
                                                      double *__restrict__ scal, unsigned int *ticket)
{
  pdl_wait();
  __shared__ bool last;
  const int i = blockIdx.x, nr = g.nr, ns = g.ns;
  const size_t row = (size_t)i * ns;
  double sum[5];
  integral_ring<PEB>(rho + row, vr + row, vr + row + ns, vt + row, e + row, pd + row, pvt + row, ns, g.r.Surf[i],
                     g.r.Rmed[i], g.r.Rinf[i], g.r.Rsup[i], omega_frame, sum);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < 5; q++) part[(size_t)q * nr + i] = sum[q];
    __threadfence();
    last = (atomicAdd(ticket, 1u) == (unsigned)nr - 1u);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (threadIdx.x == 0) *ticket = 0u;
  for (int q = threadIdx.x >> 5; q < 5; q += RING_T / 32) {
    const double *p = part + (size_t)q * nr;
    double a = 0.0, b = 0.0;
    int k = threadIdx.x & 31;
    for (; k + 32 < nr; k += 64) {
      a += __ldcg(p + k);
      b += __ldcg(p + k + 32);
    }
    if (k < nr) a += __ldcg(p + k);
    a = warp_reduce(a + b, OpAdd());
    if ((threadIdx.x & 31) == 0) scal[SC_MASS + q] = (q == 1 || q == 4) ? 0.5 * a : a;
  }
}

void aux_integrals(const DevGrid &g, const double *rho, const double *vr, const double *vt, const double *e,
                   const double *pd, const double *pvt, double omega_frame, int pebbles, double *part, double *scal,
                   unsigned int *ticket, cudaStream_t s)
{
  if (pebbles)
    launch(k_integrals<true>, g.nr, RING_T, 0, s, g, rho, vr, vt, e, pd, pvt, omega_frame, part, scal, ticket);
  else
    launch(k_integrals<false>, g.nr, RING_T, 0, s, g, rho, vr, vt, e, pd, pvt, omega_frame, part, scal, ticket);
  g_thorin_launches++;
}

// Doubles that the kernels of this file write to a disk's reduction scratch,
// from the grids they are launched with: the CFL's two floats a block, the
// forces' 2 + 2 npl values a block, the accretion's four values of two blocks
// a multiprocessor, the integrals' five a ring.
size_t aux_partials(const DevGrid &g, int npl)
{
  const ForceShape q = force_shape(g, npl);
  const dim3 c = grid2d(g.ns, g.nr - 1, 256 * CFL_CPT);
  size_t n = (size_t)c.x * c.y;
  n = std::max(n, (size_t)(2 + 2 * npl) * (q.nba + q.nbb));
  n = std::max(n, (size_t)4 * 2 * g.nsm);
  return std::max(n, (size_t)5 * g.nr);
}

// ---------------------------------------------------------------------------
// Open, non-reflecting and source-mass boundaries (ApplyBoundaryCondition,
// SideEuler.c:133-337, 458-486).  The reference's floors of the open inner
// ghost ring (SideEuler.c:15-16):
#define TH_DENSITYFLOOR 1.0e-16
#define TH_ENERGYFLOOR 1.0e-16

// OpenInnerBoundary (SideEuler.c:133-178): ring 0 is the ghost ring.
__global__ void k_open_inner(DevGrid g, double *__restrict__ rho, double *__restrict__ vr,
                             double *__restrict__ energy, int energy_eq, int damp_flux, double gasflux)
{
  pdl_wait();
  const int ns = g.ns, i = 1;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= ns) return;
  const int l = j + i * ns;
  const double a = rho[l] + (rho[l] - rho[l + ns]);
  rho[l - ns] = (a > TH_DENSITYFLOOR) ? a : TH_DENSITYFLOOR;
  if (energy_eq) {
    const double b = energy[l] + (energy[l] - energy[l + ns]);
    energy[l - ns] = (b > TH_ENERGYFLOOR) ? b : TH_ENERGYFLOOR;
  }
  if (vr[l + ns] > 0.0) { vr[l] = 0.0; vr[l - ns] = 0.0; }
  else { vr[l] = vr[l + ns]; vr[l - ns] = vr[l]; }
  if (damp_flux) {
    double rhoinf = 0.5 * (rho[l] + rho[l - ns]);
    vr[l] = div_fast(-gasflux, 2.0 * TH_PI * g.r.Rinf[i] * rhoinf);
    rhoinf = rho[l - ns] - 0.5 * (rho[l] - rho[l - ns]);
    vr[l - ns] = div_fast(-gasflux, 2.0 * TH_PI * g.r.Rinf[i - 1] * rhoinf);
  }
}

// OpenOuterBoundary (SideEuler.c:193-232): ring nrad is the ghost ring.
__global__ void k_open_outer(DevGrid g, double *__restrict__ rho, double *__restrict__ vr,
                             double *__restrict__ energy, int energy_eq, int damp_flux, double gasflux)
{
  pdl_wait();
  const int ns = g.ns, i = g.nr - 1;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= ns) return;
  const int l = j + i * ns;
  rho[l + ns] = rho[l] + (rho[l] - rho[l - ns]);
  if (energy_eq) energy[l + ns] = energy[l] + (energy[l] - energy[l - ns]);
  if (vr[l] > 0.0) { vr[l] = 0.0; vr[l + ns] = 0.0; }
  else { vr[l] = vr[l - ns]; vr[l + ns] = vr[l]; }
  if (damp_flux) {
    double rhoinf = 0.5 * (rho[l] + rho[l + ns]);
    vr[l + ns] = div_fast(-gasflux, 2.0 * TH_PI * g.r.Rinf[i + 1] * rhoinf);
    rhoinf = rho[l + ns] + 0.5 * (rho[l + ns] - rho[l]);
    vr[l + 2 * ns] = div_fast(-gasflux, 2.0 * TH_PI * g.r.Rsup[i + 1] * rhoinf);
  }
}

// Block-wide sum of a ring, valid in every thread (fixed tree order).
__device__ double ring_sum_block(const double *__restrict__ row, int ns)
{
  __shared__ double sh;
  double a = 0.0;
  for (int j = threadIdx.x; j < ns; j += blockDim.x) a += row[j];
  a = block_reduce(a, OpAdd(), 0.0);
  if (threadIdx.x == 0) sh = a;
  __syncthreads();
  a = sh;
  __syncthreads();
  return a;
}

// NonReflectingBoundary (SideEuler.c:234-337): block 0 the inner edge,
// block 1 the outer edge.  Each block copies the ring next to the edge into
// the edge ring rotated by the Keplerian shear over one cell, sets v_r from
// the outgoing characteristic, and restores the edge ring's mean density and
// energy to the initial profile.
__global__ void __launch_bounds__(1024) k_nonreflecting(DevGrid g, double *__restrict__ rho,
                                                        double *__restrict__ vr, double *__restrict__ energy,
                                                        const double *__restrict__ cs)
{
  pdl_wait();
  const int ns = g.ns, nr = g.nr;
  const bool inner = (blockIdx.x == 0);
  const int ia = inner ? 0 : nr - 2, ib = inner ? 1 : nr - 1;     // rings whose c_s are averaged
  const double csin = ring_sum_block(cs + (size_t)ia * ns, ns) / (double)ns;
  const double csout = ring_sum_block(cs + (size_t)ib * ns, ns) / (double)ns;
  double dangle;
  if (inner) dangle = (pow(g.r.Rinf[1], -1.5) - 1.0) / (.5 * (csin + csout)) * (g.r.Rmed[1] - g.r.Rmed[0]);
  else dangle = (pow(g.r.Rinf[nr - 2], -1.5) - 1.0) / (.5 * (csin + csout)) * (g.r.Rmed[nr - 1] - g.r.Rmed[nr - 2]);
  // whole turns are taken off: the reference adds or takes off one, so in thin
  // disks it leaves the ring (and the array), as the shear is longer than that
  const int i_angle = (int)(dangle / 2.0 / TH_PI * (double)ns + .5) % ns;
  const int i = inner ? 1 : nr - 1;
  const int edge = inner ? 0 : nr - 1;
  const double sig = inner ? g.r.SigmaMed[1] : g.r.SigmaMed[nr - 2];
  for (int j = threadIdx.x; j < ns; j += blockDim.x) {
    const int l = j + i * ns;
    int jp = inner ? j + i_angle : j - i_angle;
    if (jp >= ns) jp -= ns;
    if (jp < 0) jp += ns;
    if (inner) {
      const int lp = jp;
      rho[lp] = rho[l];
      energy[lp] = energy[l];
      const double vr_med = div_fast(-cs[l] * (rho[l] - sig), sig);
      vr[l] = 2. * vr_med - vr[l + ns];
    } else {
      const int lp = jp + (i - 1) * ns;
      rho[l] = rho[lp];
      energy[l] = energy[lp];
      const double vr_med = div_fast(cs[l] * (rho[l - ns] - sig), sig);
      vr[l] = 2. * vr_med - vr[l - ns];
    }
  }
  __syncthreads();
  double *re = rho + (size_t)edge * ns, *ee = energy + (size_t)edge * ns;
  const double mr = ring_sum_block(re, ns) / (double)ns;
  for (int j = threadIdx.x; j < ns; j += blockDim.x) re[j] += g.r.SigmaMed[edge] - mr;
  __syncthreads();
  const double me = ring_sum_block(ee, ns) / (double)ns;
  for (int j = threadIdx.x; j < ns; j += blockDim.x) ee[j] += g.r.EnergyMed[edge] - me;
}

// ApplyOuterSourceMass (SideEuler.c:458-486), one block.
__global__ void __launch_bounds__(1024) k_outer_source_mass(DevGrid g, double *__restrict__ rho,
                                                            double *__restrict__ vr, double penul_vr)
{
  pdl_wait();
  const int ns = g.ns, i = g.nr - 1;
  double *row = rho + (size_t)i * ns;
  const double avg = g.r.SigmaMed[i] - ring_sum_block(row, ns) / (double)ns;
  for (int j = threadIdx.x; j < ns; j += blockDim.x) {
    row[j] += avg;
    vr[j + i * ns] = penul_vr;
  }
}

void aux_open_inner(const DevGrid &g, double *rho, double *vr, double *energy, int energy_eq, int damp_flux,
                    double gasflux, cudaStream_t s)
{
  launch(k_open_inner, (g.ns + BX - 1) / BX, BX, 0, s, g, rho, vr, energy, energy_eq, damp_flux, gasflux);
  g_thorin_launches++;
}

void aux_open_outer(const DevGrid &g, double *rho, double *vr, double *energy, int energy_eq, int damp_flux,
                    double gasflux, cudaStream_t s)
{
  launch(k_open_outer, (g.ns + BX - 1) / BX, BX, 0, s, g, rho, vr, energy, energy_eq, damp_flux, gasflux);
  g_thorin_launches++;
}

void aux_nonreflecting(const DevGrid &g, double *rho, double *vr, double *energy, const double *cs, cudaStream_t s)
{
  launch(k_nonreflecting, 2, 1024, 0, s, g, rho, vr, energy, cs);
  g_thorin_launches++;
}

void aux_outer_source_mass(const DevGrid &g, double *rho, double *vr, double penul_vr, cudaStream_t s)
{
  launch(k_outer_source_mass, 1, 1024, 0, s, g, rho, vr, penul_vr);
  g_thorin_launches++;
}

// Parametric cooling of SubStep3 (SourceEuler.c:569-582): the energy relaxes
// towards the initial profile on the cooling time, heated by Q+.
__global__ void k_parametric_cooling(DevGrid g, const double *__restrict__ rho, const double *__restrict__ eint,
                                     const double *__restrict__ qplus, const double *__restrict__ divv,
                                     const double *__restrict__ coolt, const double *__restrict__ qplusmed,
                                     double *__restrict__ enew, double gm1)
{
  pdl_wait();
  const double dt = g.ctl[CTL_DT];
  const int ns = g.ns;
  CELL_LOOP_2D
  const double tc = coolt[i], sm = g.r.SigmaMed[i];
  const double tmp1 = div_fast(g.r.EnergyMed[i] * dt * rho[l], sm) + tc * eint[l] +
                      dt * tc * (qplus[l] - div_fast(qplusmed[i] * rho[l], sm));
  const double tmp2 = dt + tc + gm1 * dt * tc * divv[l];
  enew[l] = div_fast(tmp1, tmp2);
}

void aux_parametric_cooling(const DevGrid &g, const double *rho, const double *eint, const double *qplus,
                            const double *divv, const double *coolt, const double *qplusmed, double *enew,
                            double gm1, cudaStream_t s)
{
  launch(k_parametric_cooling, grid2d(g.ns, g.nr, BX), BX, 0, s, g, rho, eint, qplus, divv, coolt, qplusmed, enew, gm1);
  g_thorin_launches++;
}

// ---------------------------------------------------------------------------
// Gas accretion onto a planet, Kley's prescription (AccreteOntoPlanets,
// Planet.c:34-166): within frac1 = 0.75 and frac2 = 0.45 Roche radii a cell
// loses facc1 times the Gaussian column between the planet's height +/- the
// chord (trapezoid rule refined to 1e-4, at most 16 levels: qtrap,
// Planet.c:172-211) and then the fraction facc2.  One block per planet over
// the window [i_min, i_max] x [j_min, j_max] (narrower than a ring, so no cell
// is visited twice); the mass and momentum taken are block sums written to
// out[0..2].
__device__ double qtrap_gauss(double a, double b)
{
  double s = 0.0, olds = 0.0;
  for (int n = 1; n <= 16; n++) {
    if (n == 1) {
      s = 0.5 * (b - a) * (exp(-a * a) + exp(-b * b));
    } else {
      int it = 1;
      for (int j = 1; j < n - 1; j++) it <<= 1;
      const double tnm = it, del = div_fast(b - a, tnm);
      double x = a + 0.5 * del, sum = 0.0;
      for (int j = 1; j <= it; j++, x += del) sum += exp(-x * x);
      s = 0.5 * (s + div_fast((b - a) * sum, tnm));
    }
    if (n > 5)
      if (fabs(s - olds) < 1.e-4 * fabs(olds) || (s == 0.0 && olds == 0.0)) return s;
    olds = s;
  }
  return s;
}

__global__ void __launch_bounds__(256) k_gas_accrete(DevGrid g, double *__restrict__ dens,
                                                     const double *__restrict__ vrad,
                                                     const double *__restrict__ vtheta,
                                                     const double *__restrict__ cs, GasAccArgs a,
                                                     double *__restrict__ out)
{
  pdl_wait();
  const int ns = g.ns;
  const int nj = a.j_max - a.j_min + 1;
  const int ncell = (a.i_max - a.i_min + 1) * nj;
  double dM = 0.0, dPx = 0.0, dPy = 0.0;
  for (int c = threadIdx.x; c < ncell; c += blockDim.x) {
    const int i = a.i_min + c / nj;
    const int j = a.j_min + c % nj;
    int jf = j;
    while (jf < 0) jf += ns;
    while (jf >= ns) jf -= ns;
    const int l = jf + i * ns, lip = l + ns;
    const int ljp = (jf == ns - 1) ? i * ns : l + 1;
    const double rm = g.r.Rmed[i];
    const double xc = rm * g.r.costab[jf], yc = rm * g.r.sintab[jf];
    const double dx = a.Xp - xc, dy = a.Yp - yc;
    const double distance = sqrt(dx * dx + dy * dy);
    const double vtcell = 0.5 * (vtheta[l] + vtheta[ljp]) + rm * a.omega_frame;
    const double vrcell = 0.5 * (vrad[l] + vrad[lip]);
    const double vxcell = div_fast(vrcell * xc - vtcell * yc, rm);
    const double vycell = div_fast(vrcell * yc + vtcell * xc, rm);
    const double H = cs[l] * g.r.OmegaInv[i] * g.k.sqrt_adiabind_inv;
    const double sq2H = sqrt(2.0) * H;
    for (int pass = 0; pass < 2; pass++) {
      const double fr = pass ? 0.45 : 0.75;
      if (distance < fr * a.RRoche) {
        const double dz = sqrt((fr * a.RRoche) * (fr * a.RRoche) - distance * distance);
        double factor = qtrap_gauss(div_fast(a.Zp - dz, sq2H), div_fast(a.Zp + dz, sq2H));
        factor *= div_fast(1.0, sqrt(2.0 * TH_PI) * H);
        const double fa = pass ? a.facc2 : a.facc1;
        const double deltaM = fa * factor * dens[l] * g.r.Surf[i];
        dens[l] *= pass ? (1.0 - fa) : (1.0 - fa * factor);
        dPx += deltaM * vxcell;
        dPy += deltaM * vycell;
        dM += deltaM;
      }
    }
  }
  dM = block_reduce(dM, OpAdd(), 0.0);
  dPx = block_reduce(dPx, OpAdd(), 0.0);
  dPy = block_reduce(dPy, OpAdd(), 0.0);
  if (threadIdx.x == 0) { out[0] = dM; out[1] = dPx; out[2] = dPy; }
}

void aux_gas_accrete(const DevGrid &g, double *dens, const double *vrad, const double *vtheta, const double *cs,
                     const GasAccArgs &a, double *out, cudaStream_t s)
{
  launch(k_gas_accrete, 1, 256, 0, s, g, dens, vrad, vtheta, cs, a, out);
  g_thorin_launches++;
}

// The gas state of one cell for the planet's aerodynamic drag (StokesDrag,
// Drag.c:17-95): Sigma, c_s, v_r at l and l+nsec, v_theta at l and l+1.
__global__ void k_drag_cell(const double *__restrict__ rho, const double *__restrict__ cs,
                            const double *__restrict__ vrad, const double *__restrict__ vtheta, int l, int ns,
                            double *__restrict__ out)
{
  pdl_wait();
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  out[0] = rho[l];
  out[1] = cs[l];
  out[2] = vrad[l];
  out[3] = vrad[l + ns];
  out[4] = vtheta[l];
  out[5] = vtheta[l + 1];
}

void aux_drag_cell(const double *rho, const double *cs, const double *vrad, const double *vtheta, int l, int ns,
                   double *out, cudaStream_t s)
{
  launch(k_drag_cell, 1, 32, 0, s, rho, cs, vrad, vtheta, l, ns, out);
  g_thorin_launches++;
}

// CorrectVtheta (SideEuler.c:505-519): v_theta -= domega * Rmed when the
// frame's rotation rate changes by domega.
__global__ void k_correct_vtheta(DevGrid g, double *__restrict__ vt, double domega)
{
  pdl_wait();
  const int ns = g.ns;
  CELL_LOOP_2D
  vt[l] -= domega * g.r.Rmed[i];
}

void aux_correct_vtheta(const DevGrid &g, double *vt, double domega, cudaStream_t s)
{
  launch(k_correct_vtheta, grid2d(g.ns, g.nr, BX), BX, 0, s, g, vt, domega);
  g_thorin_launches++;
}
