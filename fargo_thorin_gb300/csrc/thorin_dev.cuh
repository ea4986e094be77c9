// thorin_dev.cuh -- device-side layout and helpers shared by the kernels.
//
// One disk lives on one GPU.  Every 2D field uses the reference's PolarGrid
// layout (src_main/LowTasks.c:73-103): (nrad+1) rows of nsec FP64 values,
// azimuth contiguous, l = j + i*nsec; row nrad is the outer v_rad face.
// Ring (1D) arrays hold nrad+2 values; entries the reference never sets stay
// zero, like its zero-initialised MAX1D globals.
//
// Floating point.  The kernels are compiled with FMA contraction (the FP64
// pipe is the bound on GB300, and a fused multiply-add is one instruction
// instead of two), so per-cell results differ from the reference's
// separately rounded C arithmetic in the last bits; integer decisions
// (FARGO shifts, SOR iteration counts, substep counts) stay exact.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "../../include/thorin_gpu.h"

#define TH_PI 3.14159265358979323844
#define TH_MPI 3.14159265358979323846
#define TH_CFLSECURITY 0.5
#define TH_CVNR 1.41
#define TH_SORMIN 1.0e-15
#define TH_SORPRECISION 1.0e-15
#define TH_OMEGAUPPER 1.9
#define TH_KAPPAFLOOR 1.0e-12
#define TH_FULL 0xffffffffu

// Unit constants of src_main/fondam.h, evaluated once on the host with the
// host libm (so they are the reference's bits) and passed in DevConst.
struct DevConst {
  double opa2cu, t2si, rho2cgs, sigma_sb, sqrt2pi_inv, pebbulkdens, cv, sqrt_adiabind_inv;
  double evaptemp;           // EVAPORATIONTEMPERATURE / T2SI
  double sqrt3;              // sqrt(3.0)
  double dpns;               // 2 pi / nsec, the azimuthal cell width in radians
  // OpacityTable SM03: the Malygin gas table (device copies)
  const double *sm_pgrid, *sm_tgrid, *sm_ross;
  int sm_rows, sm_cols;
};

// Ring arrays (device pointers, nrad+2 entries each).
struct DevRings {
  const double *Rinf, *Rsup, *Rmed, *Surf, *InvRmed, *InvSurf, *InvDiffRmed, *InvDiffRsup, *InvRinf;
  const double *OmegaInv, *Rmed2, *WaveKiller;
  const double *Omega;                  // 1 / OmegaInv
  const double *InvDxtheta;             // 1 / (2 pi / nsec * Rmed)
  const double *Rmed15, *Rinf15;        // pow(Rmed,1.5), pow(Rinf,1.5) (FViscosity)
  const double *costab, *sintab;         // cos/sin(2 pi j / nsec), nsec entries
  const double *SigmaMed, *EnergyMed, *VthetaMed;
  const double *PebDensInit, *PebVradInit, *PebVthetaInit;
  double *csmean;                        // globcsvec   (ring mean of c_s)
  double *tempmean;                      // globtempervec
  double *nu_med, *nu_inf;               // FViscosity(Rmed[i]), FViscosity(Rinf[i])
};

// The disk's control block: scalars that change from one substep to the
// next.  Kernels read them from device memory instead of taking them as
// arguments, so that the launches of a substep do not depend on host values
// and a whole DT can be captured and replayed as one CUDA graph.  The host
// path writes them (k_set_ctl) before the kernels that read them; the graph
// path computes them on the device.
enum {
  CTL_DT = 0,            // substep length dt
  CTL_OMEGA_FRAME,       // OmegaFrame
  CTL_MASS_TAPER,        // MassTaper (SourceEuler.c:230-231)
  CTL_SOR_OMEGA,         // relaxation parameter of the current SOR solve
  CTL_FACC_EVAP,         // EvaporatePebbles' fraction min(EVAPORATIONRATE dt, 1)
  CTL_INDX_PL,           // indirect acceleration of the planets (x, y)
  CTL_INDY_PL,
  CTL_DELTAT,            // the DT's remaining interval DT - dtemp (ConditionCFL)
  CTL_INVDTREB,          // MinStepForRebound's rate invdtreb_sq
  CTL_TIME,              // PhysicalTime
  CTL_DTEMP,             // time advanced so far in this DT
  CTL_SOR_DOMEGA,        // omega schedule step (EnergySources.c:298-317)
  CTL_COUNT = 32
};

struct DevGrid {
  int nr, ns;
  int nsm;                               // multiprocessors of the disk's GPU
  DevRings r;
  DevConst k;
  double *ctl;                           // control block (CTL_*), CTL_COUNT doubles
  int sor_tpsm;                          // SOR pass: resident threads per multiprocessor (0: 1536)
};

// Sum of row[0..n) in strictly left-to-right order (the reference's
// sequential ring sums, e.g. mpi_make1Dprofile, mpiTasks.c:26-32), computed by
// one warp: lanes load coalesced chunks, the running sum walks the chunk in
// order through shuffles.  All lanes return the sum.
__device__ __forceinline__ double warp_seq_sum(const double *row, int n)
{
  const int lane = threadIdx.x & 31;
  double acc = 0.0;
  for (int base = 0; base < n; base += 32) {
    double v = (base + lane < n) ? row[base + lane] : 0.0;
    int cnt = n - base < 32 ? n - base : 32;
    for (int k = 0; k < cnt; k++) acc += __shfl_sync(TH_FULL, v, k);
  }
  return acc;
}

// Start of a kernel launched by launch(): the kernel before it is done, and
// the one after it may be placed.
__device__ __forceinline__ void pdl_wait()
{
  asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;" ::: "memory");
}

// Block-wide reductions (fixed order: warp shuffles then warp partials) -----
template <typename T, typename Op>
__device__ __forceinline__ T warp_reduce(T v, Op op)
{
  for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_down_sync(TH_FULL, v, o));
  return v;
}

struct OpAdd { __device__ double operator()(double a, double b) const { return a + b; } };
struct OpMin { __device__ double operator()(double a, double b) const { return b < a ? b : a; } };
struct OpAddI { __device__ int operator()(int a, int b) const { return a + b; } };

// Result valid in thread 0.  blockDim.x must be a multiple of 32 (<= 1024).
template <typename T, typename Op>
__device__ T block_reduce(T v, Op op, T identity)
{
  __shared__ T sh[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  v = warp_reduce(v, op);
  __syncthreads();
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  v = (threadIdx.x < nw) ? sh[threadIdx.x] : identity;
  if (wid == 0) v = warp_reduce(v, op);
  return v;
}

// Sum of a ring by a block of RING_T threads, valid in the first warp: each
// thread takes every RING_T-th column, the first warp adds the other warps'
// values of its lanes and a butterfly finishes.  A fixed tree, and every lane
// returns the same bits.  (One warp per ring, the form before, left most
// multiprocessors idle: 10 us for the rings of a 512x1536 disk, and the same
// for a single ring.)
#define RING_T 128
__device__ __forceinline__ double ring_sum(const double *__restrict__ row, int ns)
{
  __shared__ double sh[RING_T];
  double a = 0.0, b = 0.0;
  int j = threadIdx.x;
  for (; j + RING_T < ns; j += 2 * RING_T) {
    a += row[j];
    b += row[j + RING_T];
  }
  if (j < ns) a += row[j];
  a += b;
  __syncthreads();
  sh[threadIdx.x] = a;
  __syncthreads();
  if (threadIdx.x < 32) {
#pragma unroll
    for (int w = 1; w < RING_T / 32; w++) a += sh[threadIdx.x + 32 * w];
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(TH_FULL, a, o);
  }
  return a;
}

// Conservation integrals of one ring (GasTotalMass, GasMomentum,
// GasTotalEnergy, SideEuler.c:26-80,523-565, and the pebbles' mass and
// momentum) by a block of RING_T threads: sum[] = mass, twice the momentum,
// energy, pebble mass, twice the pebble momentum, valid in thread 0 (the
// pebbles' only with PEB).  FP64 pipe bound, so what is constant in a ring is
// taken out of its sums, and the momentum sum (rho_j + rho_j-1) w_j is summed
// by parts to rho_j (w_j + w_j+1), whose factor the kinetic energy needs too:
// 14 FP64 instructions a cell with pebbles, where a block reduction of five
// values for every 256 cells and a division per cell took about 75.  A
// 1024x3072 disk, the whole call: 425 -> 127 us (83 us of FP64 pipe; its reads
// at copy speed take 24).
template <bool PEB>
__device__ __forceinline__ void integral_ring(const double *__restrict__ rho, const double *__restrict__ vr,
                                              const double *__restrict__ vrp, const double *__restrict__ vt,
                                              const double *__restrict__ e, const double *__restrict__ pd,
                                              const double *__restrict__ pvt, int ns, double S, double rm, double ri,
                                              double rs, double omega_frame, double sum[5])
{
  __shared__ double sh[5][RING_T];
  const double w2 = 2.0 * (omega_frame * rm), wp = 2.0 * (rm - ri) / (rs - ri), wm = 2.0 * (rs - rm) / (rs - ri);
  double m = 0.0, am = 0.0, ek = 0.0, ei = 0.0, pm = 0.0, pam = 0.0;
#pragma unroll 4
  for (int j = threadIdx.x; j < ns; j += RING_T) {
    const int jp = (j == ns - 1) ? 0 : j + 1;
    const double d = rho[j];
    const double W = (vt[j] + vt[jp]) + w2;        // 2 v_theta of the cell's centre
    const double V = wp * vrp[j] + wm * vr[j];     // 2 v_r
    m += d;
    am += d * W;
    ek += d * (V * V + W * W);
    ei += e[j];
    if (PEB) {
      const double q = pd[j];
      pm += q;
      pam += q * ((pvt[j] + pvt[jp]) + w2);
    }
  }
  double v[5] = {S * m, S * rm * am, S * (0.125 * ek + ei), S * pm, S * rm * pam};
#pragma unroll
  for (int q = 0; q < (PEB ? 5 : 3); q++) sh[q][threadIdx.x] = v[q];
  __syncthreads();
  if (threadIdx.x < 32) {
#pragma unroll
    for (int q = 0; q < (PEB ? 5 : 3); q++) {
      double a = v[q];
#pragma unroll
      for (int w = 1; w < RING_T / 32; w++) a += sh[q][threadIdx.x + 32 * w];
      sum[q] = warp_reduce(a, OpAdd());
    }
    if (!PEB) sum[3] = sum[4] = 0.0;
  }
}

// Reciprocal and reciprocal square root estimates without the FP64 pipe.
// GB300 issues an FP64 warp instruction every 64 cycles of a sub-partition that
// is at it alone and every 76 with all four (1.68 lanes per clock and SM, any
// mix of adds, products and FMAs), and FP32 and integer ones in 1 to 4, so an estimate that takes about 25 of those and
// no FP64 instruction is nearly free beside the FP64 work of any kernel here.
// The mantissa m of the operand is split into a 24-bit FP32 part and an FP32
// remainder, m = mh + ml; one Newton-Raphson step (to second order) from the
// hardware's FP32 estimate y0 gives the correction y - y0 in FP32, which is
// added to the bits of y0 as a 64-bit integer in units of 2^-53 of the
// binade [0.5, 1].  Relative error below 2^-43 even for an FP32 estimate 2 ulp
// off; measured 213 units of 2^-53 (the form before this, the hardware's FP64
// estimate with one FP64 Newton-Raphson step, had 2^-40 and cost two FP64
// instructions).  Operands: normal numbers with exponents in [-500, 500] (the
// callers check).
__device__ __forceinline__ double est_assemble(float y0, float corr, int hi_shift)
{
  const int k = __float2int_rn(corr * 4503599627370496.0f);            // corr * 2^52, |k| < 2^31
  const int b = __float_as_int(y0);
  const long long base = __double_as_longlong(__hiloint2double((b >> 3) + 0x38000000 + hi_shift, b << 29));
  return __longlong_as_double(base + 2LL * (long long)k);
}

// 1 / d, d of either sign.
__device__ __forceinline__ double recip_est(double d)
{
  const int H = __double2hiint(d), L = __double2loint(d);
  const float mh = __int_as_float((__funnelshift_l(L, H, 3) & 0x007fffff) | 0x3f800000);
  const float ml = __int2float_rn(L & 0x1fffffff) * 2.220446049250313e-16f;    // 2^-52
  float y0;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(mh));
  y0 = fminf(fmaxf(y0, 0.5f), 1.0f);                 // m in [1, 2): 1/m in (0.5, 1]
  const float e = __fmaf_rn(-ml, y0, __fmaf_rn(-mh, y0, 1.0f));
  const double y = est_assemble(y0, y0 * __fmaf_rn(e, e, e), 0x3ff00000 - (H & 0x7ff00000));
  return __hiloint2double(__double2hiint(y) | (H & 0x80000000), __double2loint(y));
}

// 1 / sqrt(x), x > 0.
__device__ __forceinline__ double rsqrt_est(double x)
{
  const int H = __double2hiint(x), L = __double2loint(x);
  const int odd = ~(H >> 20) & 1;                    // the exponent's parity goes into the mantissa, m in [1, 4)
  const float mh = __int_as_float((__funnelshift_l(L, H, 3) & 0x007fffff) | ((127 + odd) << 23));
  const float ml = __int2float_rn(L & 0x1fffffff) * __int_as_float((75 + odd) << 23);   // 2^(odd - 52)
  float y0;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(mh));
  y0 = fminf(fmaxf(y0, 0.5f), 1.0f);
  const float t = mh * y0, tl = __fmaf_rn(mh, y0, -t);
  float e = __fmaf_rn(-t, y0, 1.0f);                 // 1 - m y0^2
  e = __fmaf_rn(-tl, y0, e);
  e = __fmaf_rn(-(ml * y0), y0, e);
  const float c = e * __fmaf_rn(0.375f, e, 0.5f);    // (1 - e)^(-1/2) - 1 to second order
  return est_assemble(y0, y0 * c, (1023 + odd - (H >> 20)) << 19);
}

// x / 2 on the integer pipe (x normal, not near the smallest exponent).
__device__ __forceinline__ double half_i(double x)
{
  return __hiloint2double(__double2hiint(x) - 0x00100000, __double2loint(x));
}

// Whether the exponent of x lies in [-500, 500] (zero, subnormals,
// infinities, NaN: no).
__device__ __forceinline__ bool exp_ok(double x)
{
  return (((unsigned)__double2hiint(x) >> 20) & 0x7ffu) - 523u < 1001u;
}

__device__ __forceinline__ bool exp_zero(double x) { return (((unsigned)__double2hiint(x) >> 20) & 0x7ffu) == 0u; }

// Quotient for the van Leer slopes only.  The harmonic-mean slope
// 2 dq- dq+ / (dq- + dq+) enters a face value as a correction of at most
// half a cell width times the slope, beside the cell value itself, so a
// relative error e of the slope moves the face value by at most
// e |dq| dx / |q|.  x times the reciprocal estimate: one FP64 instruction.
// thorin_selftest_slope_division measures its distance from IEEE division
// on the GPU.
__device__ __forceinline__ double div_slope(double x, double d)
{
  if ((exp_ok(x) || exp_zero(x)) && exp_ok(d)) return x * recip_est(d);
  return x / d;
}

// The van Leer slope of the differences a and b on either side of a cell,
// a b / (a + b) where they agree in sign, else 0, without an FP64
// instruction: product, sum and quotient as FP32 pairs.  |a| and |b| are
// scaled by the larger one's power of two and split like recip_est's operand
// (24 bits and the remainder in FP32); the sum is a two-sum, the quotient
// b / (a + b) the hardware's reciprocal estimate with one correction from the
// exact FP32 residual, and the pair's low part is added to the high part's
// bits in units of their last place.  Relative error below 2^-42, measured 441
// units of 2^-53 (963 with a reciprocal estimate one ulp off).  Differences
// more than 2^60 apart, zero, not finite or near the ends of the exponent
// range take the FP64 form (div_slope).  About 60 FP32 and integer
// instructions in place of three FP64 ones (228 cycles of a busy sub-partition).
// With WEIGHTED the sum is w a + b (the radial step's unequal ring spacings),
// w = wh + wl as an FP32 pair, w64 the same in FP64; measured 535 units for w
// within 1.05 of 1, 875 within a factor of 4.
template <bool WEIGHTED>
__device__ __forceinline__ double vl_slope_t(double a, double b, float wh, float wl, double w64)
{
  const int Ha = __double2hiint(a), Hb = __double2hiint(b);
  if ((Ha ^ Hb) < 0) return 0.0;
  const int ea = Ha & 0x7ff00000, eb = Hb & 0x7ff00000;
  const int eM = max(ea, eb), em = min(ea, eb);
  if (em >= (100 << 20) && eM < 0x7ff00000 && eM - em <= (60 << 20)) {
    const int La = __double2loint(a), Lb = __double2loint(b);
    const int sh = eM - (127 << 20);
    const float ah = __int_as_float(__funnelshift_l(La, (Ha & 0x7fffffff) - sh, 3));
    const float bh = __int_as_float(__funnelshift_l(Lb, (Hb & 0x7fffffff) - sh, 3));
    const float al = __int2float_rn(La & 0x1fffffff) * __int_as_float((__float_as_int(ah) & 0x7f800000) - (52 << 23));
    const float bl = __int2float_rn(Lb & 0x1fffffff) * __int_as_float((__float_as_int(bh) & 0x7f800000) - (52 << 23));
    float ch = ah, cl = al;
    if (WEIGHTED) {
      ch = __fmul_rn(ah, wh);
      cl = __fmaf_rn(al, wh, __fmaf_rn(ah, wl, __fmaf_rn(ah, wh, -ch)));
    }
    const float s = __fadd_rn(ch, bh), t = __fsub_rn(s, ch);
    const float sl = __fadd_rn(__fadd_rn(__fsub_rn(ch, __fsub_rn(s, t)), __fsub_rn(bh, t)), __fadd_rn(cl, bl));
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(s));
    const float qh = __fmul_rn(bh, y);
    const float ql = __fmul_rn(__fadd_rn(__fmaf_rn(-qh, s, bh), __fmaf_rn(-qh, sl, bl)), y);
    const float dh = __fmul_rn(ah, qh);
    const float dl = __fmaf_rn(al, qh, __fmaf_rn(ah, ql, __fmaf_rn(ah, qh, -dh)));
    // dh + dl as a float h and a remainder of the same sign, so that adding
    // the remainder to the bits never crosses a power of two downwards
    float h = __fadd_rn(dh, dl), l = __fadd_rn(__fsub_rn(dh, h), dl);
    const int hb = __float_as_int(h) + (__float_as_int(l) >> 31);
    l = __fadd_rn(__fsub_rn(h, __int_as_float(hb)), l);
    const int k = __float2int_rn(l * __int_as_float((306 << 23) - (hb & 0x7f800000)));
    const long long base =
        __double_as_longlong(__hiloint2double(((hb >> 3) + sh) | (Ha & 0x80000000), hb << 29));
    return __longlong_as_double(base + (long long)k);
  }
  const double p = a * b, s = WEIGHTED ? __fma_rn(w64, a, b) : a + b;
  const bool pos = __double_as_longlong(p) > 0LL;                 // p > 0.0
  const bool nz = (__double_as_longlong(s) << 1) != 0LL;          // s != 0.0
  return (pos && nz) ? div_slope(p, s) : 0.0;
}

__device__ __forceinline__ double vl_slope(double a, double b) { return vl_slope_t<false>(a, b, 0.f, 0.f, 0.0); }

// |x| by clearing the sign bit on the integer pipe (same bits as fabs).
__device__ __forceinline__ double abs_i(double x)
{
  return __hiloint2double(__double2hiint(x) & 0x7fffffff, __double2loint(x));
}

// The SOR coefficients (Ml, Mlip, Mlim, Mljp, Mljm, RHS) are stored packed
// by colour: for ring i, the cells of pass 1 (j = i-1 mod 2) then those of
// pass 2, each as k = j/2, so that a colour pass reads them contiguously.
// Every reader of those arrays indexes them through sor_pidx.
__device__ __forceinline__ size_t sor_pidx(int i, int j, int half)
{
  const int c = (j ^ (i - 1)) & 1;
  return (size_t)((i << 1) + c) * half + (j >> 1);
}

// Block reduction for blocks of exactly NT threads through shared memory:
// warp 0 folds the NT / 32 values of its lane's column, then one shuffle
// tree finishes.  On the FP64 pipe that is NT/32 + 4 warp instructions
// instead of the 5 (NT/32 + 1) of block_reduce.  Result valid in thread 0;
// fixed order.  Safe to call repeatedly (the first barrier waits for the
// previous call's readers).
template <int NT, typename T, typename Op>
__device__ __forceinline__ T block_reduce_smem(T v, Op op)
{
  static_assert(NT % 32 == 0 && NT <= 1024, "block of whole warps");
  __shared__ T sh[NT];
  __syncthreads();
  sh[threadIdx.x] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    T s = sh[threadIdx.x];
#pragma unroll
    for (int k = 1; k < NT / 32; k++) s = op(s, sh[threadIdx.x + 32 * k]);
    v = warp_reduce(s, op);
  }
  return v;
}

// x^3 correctly rounded (Dekker two-product with fma): the reference uses
// pow(T, 3.0) (EnergySources.c:95,590), which glibc returns correctly
// rounded in all but vanishingly rare cases.
__device__ __forceinline__ double cube_rn(double x)
{
  double h = x * x;
  double l = __fma_rn(x, x, -h);          // x*x = h + l exactly
  double p = h * x;
  double e = __fma_rn(h, x, -p);          // h*x = p + e exactly
  double t = __fma_rn(l, x, e);           // remaining terms
  return __dadd_rn(p, t);
}

// Division without the IEEE divide sequence, for the hot stencils: the
// quotient q = x y with the reciprocal estimate y gets Markstein's
// correction q + (x - d q) y with the residual formed exactly by an FMA
// (P. W. Markstein, IBM J. Res. Dev. 34(1):111-119, 1990): three FP64
// instructions (two for a reciprocal), where the form with an FP64
// Newton-Raphson step took five.  Operands whose exponents lie in
// [-500, 500] (x may also be zero or subnormal) take this path, anything
// else the IEEE division.  thorin_selftest_division measures it against IEEE
// division on the GPU.
__device__ __forceinline__ double div_fast(double x, double d)
{
  if ((exp_ok(x) || exp_zero(x)) && exp_ok(d)) {
    const double y = recip_est(d);
    const double q = x * y;
    const double r = __fma_rn(-d, q, x);
    return __fma_rn(r, y, q);
  }
  return x / d;
}

// Square root in three FP64 instructions: the estimate y of 1/sqrt(x), then
// s = x y with the residual x - s^2 formed exactly (Markstein's correction as in
// div_fast).  thorin_selftest_sqrt measures it on the GPU.
__device__ __forceinline__ double sqrt_fast(double x)
{
  if (exp_ok(x) && __double2hiint(x) > 0) {
    const double y = rsqrt_est(x);
    const double s = x * y;
    const double r = __fma_rn(-s, s, x);
    return __fma_rn(r, half_i(y), s);
  }
  return sqrt(x);
}

// y (1 + rel) for |rel| below 2^-40: rel in units of y's last place, rounded to
// an integer and added to y's bits (formed in FP32, to 2^-8 of an ulp).
__device__ __forceinline__ double nudge(double y, float rel)
{
  const float mf = __int_as_float(0x3f800000 | ((__double2hiint(y) & 0x000fffff) << 3));
  const int k = __float2int_rn(rel * mf * 4503599627370496.0f);          // 2^52
  return __longlong_as_double(__double_as_longlong(y) + (long long)k);
}

// FP32 value of x, truncated, 0 below 2^-111 in size (x below 2^100).
__device__ __forceinline__ float small_to_float(double x)
{
  const int H = __double2hiint(x), M = H & 0x7fffffff;
  const float f = __int_as_float(__funnelshift_l(__double2loint(x), M - 0x38000000, 3) | (H & 0x80000000));
  return (M < 0x39000000) ? 0.0f : f;
}

// x^(-3/2), x > 0, in three FP64 instructions: y from rsqrt_est, y^2 and y^3
// as rounded products, and the factor 1 + 3/2 (1 - x y^2) by nudge (the
// residual 1 - x y^2 is exact).  Within 2 ulp; the cube of a rounded
// reciprocal square root, five instructions, was within 5.
__device__ __forceinline__ double pow_m32(double x)
{
  if (exp_ok(x) && __double2hiint(x) > 0) {
    const double y = rsqrt_est(x);
    const double y2 = y * y;
    const double e = __fma_rn(-x, y2, 1.0);
    const double y3 = y2 * y;
    return nudge(y3, 1.5f * small_to_float(e));
  }
  return 1.0 / (x * sqrt(x));
}

// x^(1/4), x > 0, in two FP64 instructions: q from two reciprocal square root
// estimates, and the factor 1 + (x - q^4) / (4 x) by nudge.  Within an ulp.
__device__ __forceinline__ double root4(double x)
{
  if (exp_ok(x) && __double2hiint(x) > 0) {
    const double q = rsqrt_est(rsqrt_est(x));
    const double q2 = q * q;
    const double e = __fma_rn(-q2, q2, x);
    // e / x from the two's own exponents: both scaled by x's power of two
    const int sh = (__double2hiint(x) & 0x7ff00000) - 0x3ff00000;
    const float xf = __int_as_float(0x3f800000 | ((__double2hiint(x) & 0x000fffff) << 3));
    const int He = __double2hiint(e), Me = (He & 0x7fffffff) - sh;         // e 2^-E
    const float ef = (Me < 0x39000000 || (He & 0x7ff00000) == 0)
                         ? 0.0f
                         : __int_as_float(__funnelshift_l(__double2loint(e), Me - 0x38000000, 3) | (He & 0x80000000));
    return nudge(q, 0.25f * __fdividef(ef, xf));
  }
  return sqrt(sqrt(x));
}

// r / (r + 1e-20), the density's own transported quotient (the reference
// divides every transported quantity by Sigma + 1e-20): 1 where 1e-20 is
// below half an ulp of r, else 1 - 1e-20 / r with the small quotient in FP32
// (it is below 2^-31, so its FP32 error is below rounding) subtracted from the
// bits of 1; very small, negative or non-finite r divide.
__device__ __forceinline__ double unit_quotient(double r)
{
  const int H = __double2hiint(r);
  if (H >= (1010 << 20) && H < 0x7ff00000) return 1.0;            // r >= 2^-13
  if (H >= (988 << 20) && H < 0x7ff00000) {                       // r >= 2^-35
    const float rf = __int_as_float(__funnelshift_l(__double2loint(r), H - 0x38000000, 3));
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(rf));
    const int k = __float2int_rn(1.0e-20f * y * 9007199254740992.0f);   // units of 2^-53
    return __longlong_as_double(0x3ff0000000000000LL - (long long)k);
  }
  return r * div_fast(1.0, r + 1e-20);
}

// exp(x) by table (P. T. P. Tang, ACM Trans. Math. Softw. 15(2):144-157,
// 1989): n the integer nearest 64 x / ln 2, r = x - n ln 2 / 64 in two steps,
// exp(x) = 2^(n div 64) 2^((n mod 64)/64) (1 + (r + r^2 (1/2 + r/6 + t))) with
// the tail t = r^2/24 + r^3/120 + r^4/720, below 1.3e-6, in FP32.  The powers of
// 2^(1/64) are rounded values and their remainders (c_exp64, copied to shared
// memory: tab): with the rounded ones alone, an FP64 instruction less, the
// largest error was 1.02 ulp, and CUDA's exp has 0.87; with both it is 0.56.
// Nine FP64 instructions.
__constant__ double c_exp64[128] = {
    1.0, 1.0108892860517005, 1.0218971486541166, 1.0330248790212284,
    1.0442737824274138, 1.0556451783605572, 1.0671404006768237, 1.0787607977571199,
    1.0905077326652577, 1.102382583307841, 1.1143867425958924, 1.1265216186082418,
    1.1387886347566916, 1.1511892299529827, 1.1637248587775775, 1.1763969916502812,
    1.189207115002721, 1.202156731452703, 1.215247359980469, 1.22848053610687,
    1.241857812073484, 1.255380757024691, 1.2690509571917332, 1.2828700160787783,
    1.2968395546510096, 1.3109612115247644, 1.3252366431597413, 1.339667524053303,
    1.3542555469368927, 1.3690024229745905, 1.383909881963832, 1.3989796725383112,
    1.4142135623730951, 1.42961333839197, 1.4451808069770467, 1.460917794180647,
    1.4768261459394993, 1.4929077282912648, 1.5091644275934228, 1.5255981507445384,
    1.5422108254079407, 1.559004400237837, 1.5759808451078865, 1.593142151342267,
    1.6104903319492543, 1.6280274218573478, 1.645755478153965, 1.6636765803267364,
    1.681792830507429, 1.7001063537185235, 1.718619298122478, 1.7373338352737062,
    1.7562521603732995, 1.7753764925265212, 1.7947090750031072, 1.8142521755003989,
    1.8340080864093424, 1.8539791250833855, 1.8741676341103, 1.8945759815869656,
    1.9152065613971474, 1.9360617934922943, 1.9571441241754002, 1.978456026387951,
    0.0, -1.5234778603368577e-17, 5.109225028973444e-17, 7.600838874027088e-18,
    8.551889705537965e-17, 1.759325738772092e-18, -7.899853966841582e-17, -6.656660436056593e-17,
    -3.046782079812471e-17, 5.2660368715706944e-17, 1.0410278456845571e-16, 5.165856758795457e-17,
    8.912812676025408e-17, 3.250710218863827e-17, 3.8292048369240935e-17, 5.554203254218079e-17,
    3.982015231465646e-17, 6.644981499252301e-17, -7.712630692681488e-17, -1.89878163130253e-17,
    4.658027591836937e-17, -6.7113898212968784e-18, 2.667932131342186e-18, 1.713594918243561e-17,
    2.5382502794888315e-17, -7.181536135519454e-17, -2.8587312100388614e-17, 8.927282594831732e-17,
    7.70094837980299e-17, 9.593797919118849e-17, -6.770511658794786e-17, -9.614213209051323e-17,
    -9.667293313452913e-17, -1.2031642489053655e-17, -3.0237581349939873e-17, -5.600377186075216e-17,
    -3.483994556892796e-17, 1.4192920154284036e-17, -1.016455327754295e-16, -1.1024941712342561e-16,
    7.949834809697621e-17, 3.7812070533575275e-17, -1.0136916471278304e-17, -1.0094406542311964e-16,
    2.4707192569797888e-17, -6.712955084707084e-17, -1.0125679913674773e-16, 5.8909926967131e-17,
    8.199010020581497e-17, -8.0237193703977e-18, -1.851380418263111e-17, 3.164389299292957e-17,
    2.960140695448873e-17, 6.429731796556572e-17, 1.8227458427912087e-17, -9.969531538920349e-17,
    3.283107224245627e-17, 9.761887490727594e-17, -6.122763413004143e-17, 3.4034035352165297e-17,
    -1.0619946056195963e-16, 1.0332385960676326e-16, 8.960767791036668e-17, 4.0388753109278167e-17};

__device__ __forceinline__ double float_to_double(float f)
{
  const int b = __float_as_int(f);                   // 0 becomes 2^-127
  return __hiloint2double((((b & 0x7fffffff) >> 3) + 0x38000000) | (b & 0x80000000), b << 29);
}

// FP32 value of x, truncated; 0 below 2^-100 in size, infinite above 2^100
// (and for a NaN).
__device__ __forceinline__ float to_float_trunc(double x)
{
  const int H = __double2hiint(x), M = H & 0x7fffffff;
  float f = __int_as_float(__funnelshift_l(__double2loint(x), M - 0x38000000, 3));
  if (M < (923 << 20)) f = 0.0f;
  if (M > (1123 << 20)) f = __int_as_float(0x7f800000);
  return __int_as_float(__float_as_int(f) | (H & 0x80000000));
}

__device__ __forceinline__ double exp_fast(double x, const double *tab)
{
  const float xf = to_float_trunc(x);
  if (fabsf(xf) < 600.0f) {
    const int n = __float2int_rn(xf * 92.332482616893656f);
    const double nd = float_to_double(__int2float_rn(n));
    double r = __fma_rn(nd, -0.01083042469326756, x);
    r = __fma_rn(nd, -2.9815858269852933e-12, r);
    const float rf = to_float_trunc(r);
    const float t = rf * rf * __fmaf_rn(rf, __fmaf_rn(rf, 1.3888889e-3f, 8.3333333e-3f), 4.1666667e-2f);
    const double q = __fma_rn(r, 0.16666666666666666, 0.5) + float_to_double(t);
    const double e = __fma_rn(r * r, q, r);
    const double T = tab[n & 63];
    const double y = T + __fma_rn(T, e, tab[64 + (n & 63)]);
    return __hiloint2double(__double2hiint(y) + ((n >> 6) << 20), __double2loint(y));
  }
  return exp(x);
}

// FP32 value of a positive double of moderate exponent, truncated (0 outside
// [2^-100, 2^100]).
__device__ __forceinline__ float to_float_pos(double x)
{
  const int H = __double2hiint(x);
  const float f = __int_as_float(__funnelshift_l(__double2loint(x), H - 0x38000000, 3));
  return (unsigned)(H - (923 << 20)) < (unsigned)(200 << 20) ? f : 0.0f;
}
