// Force pair loop (K5/K6/K8): cons2prim_everything (cons2prim.f90:326-394,
// eos.f90:184-237), start_cell (force.F90:2172-2514), compute_forces
// (force.F90:914-2060) and finish_cell_and_store_results (force.F90:2649-3330)
// for gas particles: pressure, artificial viscosity and conductivity, ideal MHD
// (anisotropic Lorentz stress, artificial resistivity, div B cleaning) and the
// self-gravity near field; global Courant/force timestep minima.
//
// Decomposition mirrors the density: one warp per leaf cell sweeps the trial
// list, pairs that pass the distance pre-filter are queued per particle and
// evaluated with the lanes dealt out by queue length, and the per-particle sums
// go to k_force_finish (one thread per particle) for
// finish_cell_and_store_results. With self-gravity every trial pair has a
// term: those kernels keep lanes of (particle i, stripe s), which evaluate the
// far pairs where they test them and queue the near ones. The j-side quantities that
// compute_forces recomputes for every pair (rho_j, P_j/rho_j^2, v_wave,j, the
// magnetic stress, ...) are computed once per particle by k_force_prologue and
// read per pair. The neighbour test q_i^2 < 4 .or. q_j^2 < 4 is evaluated with
// the reference's rounding; an FP32 pre-filter skips pairs provably outside
// both kernels.
#include "ph_internal.h"
#include "ph_walk.cuh"

namespace ph {

constexpr int JREC = 16;   // doubles per particle, hydro record
constexpr int JMHD = 16;   // doubles per particle, MHD record
// The pair terms' record: every factor of a pair term that belongs to one
// particle is formed once in the prologue (the particle mass is applied to
// the finished sums). JR_K = -3/4 cnormk h^-4 / Omega (on s of kern_w, giving
// grad W; without the -3/4 in the mixed form, whose kernel is grkernf),
// JR_C = -1/(2 rho) of the viscosity, JR_AVW = alpha v_wave, JR_AU =
// alpha_u / (2 rho) (FP64: with the sqrt(2) of the conductivity's signal
// speed, force.F90:1605-1621), JR_AB = alpha_B / (2 rho^2)
enum { JR_H1 = 0, JR_RHO, JR_C, JR_PRO2, JR_VW, JR_P, JR_AU, JR_K, JR_VX, JR_VY, JR_VZ, JR_U, JR_GS, JR_AB, JR_AVW,
       JR_R21 };
// MHD: B, psi, overcleanfac psi v_wave; B/rho in the finish's slots 10..12
enum { JM_BX = 0, JM_BY, JM_BZ, JM_PSI, JM_CL };
constexpr int NF = 12;     // fsum entries
constexpr int JRECF = 16, JMHDF = 8;  // floats per particle, FP32 records of the mixed form

// get_stress (force.F90:2068-2168) without physical viscosity / radiation: P/rho^2
// with the magnetic pressure and the wave speed (the pair terms form the
// anisotropic stress -(B/rho)(B/rho).n from the Lorentz projections)
__device__ __forceinline__ void get_stress(const Params &p, double pri, double cs, double rhoi, double rho1i,
                                           double bx, double by, double bz, double &pro2, double &vwave) {
  if (p.mhd) {
    double brx = bx * rho1i, bry = by * rho1i, brz = bz * rho1i;
    double bro2 = brx * brx + bry * bry + brz * brz;
    double va2 = bro2 * rhoi;
    vwave = sqrt(cs * cs + va2);
    pro2 = pri * rho1i * rho1i + 0.5 * bro2;
  } else {
    pro2 = pri * rho1i * rho1i;
    vwave = cs;
  }
}

// eos + j-side record per tree position
// shock_capturing.f90:151-177 xi_limiter (dvdx float, arithmetic in FP64)
__device__ __forceinline__ double xi_limiter(const float *dvdxf) {
  double d[9];
  for (int q = 0; q < 9; ++q) d[q] = (double)dvdxf[q];
  const double divv = dadd(dadd(d[0], d[4]), d[8]);
  const double cx = dsub(d[7], d[5]), cy = dsub(d[2], d[6]), cz = dsub(d[3], d[1]);
  const double m = fmax(-divv, 0.0);
  const double fac = dmul(m, m);
  const double traceS = dadd(dadd(dmul(cx, cx), dmul(cy, cy)), dmul(cz, cz));
  if (dadd(fac, traceS) > EPS_D) return ddiv(fac, dadd(fac, traceS));
  return 1.0;
}
// shock_capturing.f90:131-143 get_alphaloc
__device__ __forceinline__ double get_alphaloc(double divvdti, double spsoundi, double hi, double xi,
                                               double alpha_min, double alpha_max) {
  const double source = dmul(dmul(dmul(10.0, dmul(hi, hi)), xi), fmax(-divvdti, 0.0));
  const double temp = dmul(spsoundi, spsoundi);
  if (temp > EPS_D) return fmax(fmin(ddiv(source, temp), alpha_max), alpha_min);
  return alpha_min;
}

// The precision form's prologue: the FP32 particle records formed in FP32
// from the FP64 state rounded on the integer pipe (the FP64 form's exact
// divisions and square roots hold the FP64 pipe; the mixed pair kernels read
// FP32 records only), and of the FP64 ones what the force finish reads: the
// equation of state, u and, with MHD, Bevol and psi. cons2prim
// (cons2prim.f90:326-456) and get_stress (force.F90:2068-2168) as in
// k_force_prologue, in FP32.
__global__ void k_force_prologue_mixed(Params p, int n, const int *perm, const double *th, const double *vel,
                                       const double *Bv, const float *gradh, double *eos_t, double *jrec,
                                       double *jmhd, float *jrecf, float *jmhdf, float4 *txf, const float *alpha1,
                                       const float *ddivvdt_c, const float *dvdx_c, float *alphaloc_t, int *err) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int pid = perm[j];
  const double h = th[j];
  if (h < 0.0) set_error(err, PH_ERR_NEG_H);
  const float pmf = d2f_rn(p.massoftype);
  const float hf = d2f_rn(h);
  const float h1 = 1.0f / hf;
  const float t3 = d2f_rn(p.hfact) * h1;
  const float rho = pmf * (t3 * t3 * t3), rho1 = 1.0f / rho;
  const double *v = vel + 4 * (size_t)pid;
  const float u = p.isothermal ? 0.0f : d2f_rn(v[3]);
  float ponrho, cs;
  if (p.ieos == 1) { ponrho = d2f_rn(p.polyk); cs = sqrtf(ponrho); }
  else {
    ponrho = (p.gamma > 1.0001) ? d2f_rn(p.gamma - 1.0) * u : (2.0f / 3.0f) * u;
    cs = sqrtf(d2f_rn(p.gamma) * ponrho);
  }
  const float P = ponrho * rho;
  eos_t[2 * (size_t)j] = (double)P;
  eos_t[2 * (size_t)j + 1] = (double)cs;
  if (p.nalpha >= 2) {  // cons2prim.f90:413-418 Cullen & Dehnen alphaloc (FP64, as the FP64 form)
    const double xi = xi_limiter(dvdx_c + 9 * (size_t)pid);
    alphaloc_t[j] = (float)get_alphaloc((double)ddivvdt_c[pid], (double)cs, h, xi, p.alpha, p.alphamax);
  }
  float pro2 = P * rho1 * rho1, vwave = cs;
  float *q = jmhdf + JMHDF * (size_t)j;
  if (p.mhd) {
    // B/rho is Bevol; B = Bevol rho; stress -m (B/rho)(B/rho), P/rho^2 + |B/rho|^2/2,
    // v_wave = sqrt(c_s^2 + |B/rho|^2 rho)
    const double *b = Bv + 4 * (size_t)pid;
    const float brx = d2f_rn(b[0]), bry = d2f_rn(b[1]), brz = d2f_rn(b[2]);
    const float bro2 = brx * brx + bry * bry + brz * brz;
    vwave = sqrtf(cs * cs + bro2 * rho);
    pro2 += 0.5f * bro2;
    q[0] = brx * rho; q[1] = bry * rho; q[2] = brz * rho; q[3] = d2f_rn(b[3]);
    q[JM_CL] = d2f_rn(p.overcleanfac) * q[3] * vwave;
    double *m = jmhd + JMHD * (size_t)j;  // the finish's B/rho and psi
    m[3] = b[3]; m[10] = b[0]; m[11] = b[1]; m[12] = b[2];
  }
  const size_t g = p.ind ? (size_t)pid : (size_t)j;
  float *o = jrecf + JRECF * (size_t)j;
  o[JR_H1] = h1; o[JR_RHO] = rho; o[JR_C] = -0.5f * rho1; o[JR_PRO2] = pro2; o[JR_VW] = vwave; o[JR_P] = P;
  o[JR_AU] = 0.5f * rho1 * d2f_rn(p.alphau);
  o[JR_K] = (h1 * h1) * (h1 * h1) * (float)CNORMK * gradh[2 * g];  // on dW/dq (grkernf)
  o[JR_VX] = d2f_rn(v[0]); o[JR_VY] = d2f_rn(v[1]); o[JR_VZ] = d2f_rn(v[2]); o[JR_U] = u;
  o[JR_GS] = gradh[2 * g + 1];
  o[JR_AB] = 0.5f * d2f_rn(p.alphaB) * (rho1 * rho1);
  o[JR_AVW] = (p.nalpha > 0 ? alpha1[pid] : d2f_rn(p.alpha)) * vwave;
  o[JR_R21] = rho1 * rho1;
  jrec[JREC * (size_t)j + 11] = p.isothermal ? 0.0 : v[3];  // the finish's u
  txf[j].w = h1;
}

__global__ void k_force_prologue(Params p, int n, const int *perm, const double *th, const double *vel,
                                 const double *Bv, const float *gradh, double *eos_t, double *jrec, double *jmhd,
                                 float4 *txf, const float *alpha1, const float *ddivvdt_c, const float *dvdx_c,
                                 float *alphaloc_t, int *err) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const double pm = p.massoftype;
  const int pid = perm[j];
  const double h = th[j];
  if (h < 0.0) set_error(err, PH_ERR_NEG_H);
  // cons2prim: rho = rhoh(h) (cons2prim.f90:343), P = (gamma-1) u rho or cs^2 rho
  const double rho_c = rhoh(h, pm, p.hfact);
  const double *v = vel + 4 * (size_t)pid;
  double ponrho, cs;
  if (p.ieos == 1) { ponrho = p.polyk; cs = sqrt(ponrho); }
  else {
    double u = v[3];
    ponrho = (p.gamma > 1.0001) ? (p.gamma - 1.0) * u : 2.0 / 3.0 * u;
    cs = sqrt(p.gamma * ponrho);
  }
  const double P = ponrho * rho_c;
  eos_t[2 * (size_t)j] = P;
  eos_t[2 * (size_t)j + 1] = cs;
  if (p.nalpha >= 2) {  // cons2prim.f90:413-418 Cullen & Dehnen alphaloc
    const double xi = xi_limiter(dvdx_c + 9 * (size_t)pid);
    alphaloc_t[j] = (float)get_alphaloc((double)ddivvdt_c[pid], cs, h, xi, p.alpha, p.alphamax);
  }
  // start_cell and the j-side of compute_forces (force.F90:1428-1511, 2270-2340)
  const double h1 = 1.0 / h;
  const double rho1 = 1.0 / rho_c;
  double bx = 0, by = 0, bz = 0;
  if (p.mhd) {
    const double *b = Bv + 4 * (size_t)pid;
    bx = b[0] * rho_c; by = b[1] * rho_c; bz = b[2] * rho_c;
  }
  double pro2, vwave;
  get_stress(p, P, cs, rho_c, rho1, bx, by, bz, pro2, vwave);
  double *r = jrec + JREC * (size_t)j;
  // gradh in tree order; with individual timesteps in caller order, where
  // inactive particles keep the values of their last density solve
  const size_t g = p.ind ? (size_t)pid : (size_t)j;
  const double h21 = h1 * h1;
  r[JR_H1] = h1; r[JR_RHO] = rho_c; r[JR_C] = -0.5 * rho1; r[JR_PRO2] = pro2;
  r[JR_VW] = vwave; r[JR_P] = P;
  r[JR_AU] = 0.5 * rho1 * p.alphau * (p.gravity ? 1.0 : 1.4142135623730951);
  r[JR_K] = -0.75 * CNORMK * (h21 * h21) * (double)gradh[2 * g];
  r[JR_VX] = v[0]; r[JR_VY] = v[1]; r[JR_VZ] = v[2]; r[JR_U] = p.isothermal ? 0.0 : v[3];
  r[JR_GS] = (double)gradh[2 * g + 1];
  r[JR_AB] = 0.5 * p.alphaB * rho1 * rho1;
  // alphaind(1,j) (force.F90:1478, 2430-2433)
  r[JR_AVW] = (p.nalpha > 0 ? (double)alpha1[pid] : p.alpha) * vwave;
  r[JR_R21] = rho1 * rho1;
  if (p.mhd) {
    double *m = jmhd + JMHD * (size_t)j;
    const double *b = Bv + 4 * (size_t)pid;
    m[JM_BX] = bx; m[JM_BY] = by; m[JM_BZ] = bz; m[JM_PSI] = b[3];
    m[JM_CL] = p.overcleanfac * b[3] * vwave;
    m[10] = b[0]; m[11] = b[1]; m[12] = b[2];
  }
  txf[j].w = (float)h1;  // x, y, z: set by the tree build
}

struct ForceOut {
  double *fxyzu, *dBevol;
  float *divcurlv, *divBsymm, *poten;
  double *dtmin;  // [0] dtcourant, [1] dtforce (atomic min of positive doubles)
  unsigned long long *stats;
  const int *cell_ntrial;
};

// expand_fgrav_in_taylor_series (kdtree.F90:1799-1840): far-field force and
// potential at an offset (dx, dy, dz) from the leaf centre. The potential
// line keeps the reference's dz*dfxy term as written there.
__device__ __forceinline__ void expand_taylor(const double *f, double dx, double dy, double dz, double &fxi,
                                              double &fyi, double &fzi, double &poti) {
  fxi = f[0]; fyi = f[1]; fzi = f[2];
  const double dfxx = f[3], dfxy = f[4], dfxz = f[5], dfyy = f[6], dfyz = f[7], dfzz = f[8];
  const double d2fxxx = f[9], d2fxxy = f[10], d2fxxz = f[11], d2fxyy = f[12], d2fxyz = f[13], d2fxzz = f[14],
               d2fyyy = f[15], d2fyyz = f[16], d2fyzz = f[17], d2fzzz = f[18];
  poti = f[19];
  fxi = fxi + dx * (dfxx + 0.5 * (dx * d2fxxx + dy * d2fxxy + dz * d2fxxz))
            + dy * (dfxy + 0.5 * (dx * d2fxxy + dy * d2fxyy + dz * d2fxyz))
            + dz * (dfxz + 0.5 * (dx * d2fxxz + dy * d2fxyz + dz * d2fxzz));
  fyi = fyi + dx * (dfxy + 0.5 * (dx * d2fxxy + dy * d2fxyy + dz * d2fxyz))
            + dy * (dfyy + 0.5 * (dx * d2fxyy + dy * d2fyyy + dz * d2fyyz))
            + dz * (dfyz + 0.5 * (dx * d2fxyz + dy * d2fyyz + dz * d2fyzz));
  fzi = fzi + dx * (dfxz + 0.5 * (dx * d2fxxz + dy * d2fxyz + dz * d2fxzz))
            + dy * (dfyz + 0.5 * (dx * d2fxyz + dy * d2fyyz + dz * d2fyzz))
            + dz * (dfzz + 0.5 * (dx * d2fxzz + dy * d2fyzz + dz * d2fzzz));
  poti = poti - (dx * (fxi - 0.5 * (dx * dfxx + dy * dfxy + dz * dfxy)) +
                 dy * (fyi - 0.5 * (dx * dfxy + dy * dfyy + dz * dfyz)) +
                 dz * (fzi - 0.5 * (dx * dfxz + dy * dfyz + dz * dfzz)));
}

// gravity far field seen by the finish kernel
struct FarField {
  const double *gleaf;  // LENFG coefficients per leaf index
  const int *leaf_of;   // leaf index per tree position
  const int *leaves;
  const Node *nodes;
  const double *tx, *ty, *tz;
};

// per-particle pair sums written by the force pair kernels (tree order, slot
// major with stride ps): slots 0..NF-1 the fsum entries, slot NF vsigmax
constexpr int FSLOT_VSIG = NF;
// individual timesteps: slot NF+1 the largest ibin_old of the SPH neighbours
// (force.F90:1346-1353, the Saitoh-Makino limiter's input)
constexpr int FSLOT_NBIN = NF + 1;

// finish_cell_and_store_results (force.F90:2773-3328): one thread per particle
// (tree position ip) from its pair sums; timestep minima per warp, then one
// atomic per warp.
// individual timesteps in the finish: the particles' bins (caller order) and
// the step's counters; ibin null with global timesteps
struct IndFin {
  const unsigned char *actf_t;  // active flag per tree position
  int8_t *ibin;
  int *counters;                // [0] max new bin, [1] particles binned, [2] dt too small
  int nbinmax, istepfrac, allow_decrease;
};

// get_newbin (utils_indtimesteps.f90:230-287): the bin of a particle's new
// timestep; a shorter step moves it up at once, a longer one down by one bin
// and only where the lower bin's step ends on this substep
__device__ __forceinline__ int get_newbin(double dti, double dtmax, int ibini, const IndFin &ind, int &too_small) {
  const double dlog2 = 1.4426950408889634;
  int ibin_new;
  if (dti > dtmax) ibin_new = 0;
  else if (dti < TINY_D) ibin_new = MAXBINS;
  else ibin_new = max((int)(log(2.0 * dtmax / dti) * dlog2 - EPS_D), 0);
  if (ibin_new > MAXBINS) too_small = 1;
  if (ibin_new > ibini) return ibin_new;
  if (ibin_new < ibini && ibini <= ind.nbinmax && ind.allow_decrease &&
      (long long)ind.istepfrac % (1ll << (ind.nbinmax - (ibini - 1))) == 0)
    return ibini - 1;
  return ibini;
}

// The precision form's finish (MIXED): the per-particle chain (density, the
// pdV factor, div v, the MHD stress and cleaning, the timestep estimates) in
// FP32 from the FP64 values rounded on the integer pipe, where the FP64 form's
// divisions and square roots would hold the FP64 pipe; the accelerations and
// the dissipation sums stay the FP64 values of the pair sums, and the gravity
// far field stays FP64.
template <bool MIXED>
__global__ void __launch_bounds__(256) k_force_finish(Params p, int nt, const double *psum, int64_t ps,
                                                      const int *perm, const double *th, const double *jrec,
                                                      const double *jmhd, const double *eos_t, FarField ff,
                                                      ForceOut out, IndFin ind, int *err) {
  const int ipr = blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = ipr < nt && (!ind.actf_t || ind.actf_t[ipr]);  // inactive particles keep their forces
  const int ip = valid ? ipr : 0;
  const double pm = p.massoftype;
  const bool adiab = !p.isothermal;
  double fs[NF];
  // the slots the pair kernels wrote (3: potential, 7..11: MHD)
  for (int k = 0; k < NF; ++k)
    fs[k] = (k == 3 ? p.gravity : (k < 7 || p.mhd)) ? psum[k * ps + ip] : 0.0;
  const double vsm = psum[FSLOT_VSIG * ps + ip];
  const int pid = perm[ip];
  const double h = th[ip];
  const double pr = eos_t[2 * (size_t)ip], cs = eos_t[2 * (size_t)ip + 1];
  const double *rr = jrec + JREC * (size_t)ip;
  if (p.gravity) {
    // self-potential and far field (force.F90 finish_cell_and_store_results,
    // kdtree.F90:1799-1840); kernel_softening(0) potential = -7/5
    double epoti = 0.5 * pm * (fs[3] + pm * (-1.4) * (1.0 / h));
    const int l = ff.leaf_of[ip];
    const Node nl = ff.nodes[ff.leaves[l]];
    double fxi, fyi, fzi, poti;
    expand_taylor(ff.gleaf + LENFG * (size_t)l, ff.tx[ip] - nl.x, ff.ty[ip] - nl.y, ff.tz[ip] - nl.z, fxi, fyi, fzi,
                  poti);
    fs[0] += fxi; fs[1] += fyi; fs[2] += fzi;
    epoti += 0.5 * pm * poti;
    if (valid) out.poten[pid] = (float)epoti;
  }
  double *fo = out.fxyzu + 4 * (size_t)pid;
  double dtc = p.dtmax, dtf = BIGNUMBER, dtclean = BIGNUMBER;
  if constexpr (MIXED) {
    const float pmf = d2f_rn(pm), hf = d2f_rn(h), h1f = 1.0f / hf;
    const float t3 = d2f_rn(p.hfact) * (1.0f / fabsf(hf));
    const float rhof = pmf * (t3 * t3 * t3), rho1f = 1.0f / rhof;
    const float prf = d2f_rn(pr), csf = d2f_rn(cs);  // FP32 values held in FP64: exact
    float vwavef = csf, psif = 0.0f;
    if (p.mhd) {
      // B = rho B/rho, v_wave = sqrt(c_s^2 + |B/rho|^2 rho) (get_stress,
      // force.F90:2068-2168); the div B subtraction from the FP64 sums
      const double *m = jmhd + JMHD * (size_t)ip;
      const float brx = d2f_rn(m[10]), bry = d2f_rn(m[11]), brz = d2f_rn(m[12]);
      psif = d2f_rn(m[3]);
      const float bxf = brx * rhof, byf = bry * rhof, bzf = brz * rhof;
      vwavef = sqrtf(csf * csf + (brx * brx + bry * bry + brz * brz) * rhof);
      const float b2f = bxf * bxf + byf * byf + bzf * bzf;
      float frac = 0.0f;
      if (b2f > 0.0f) {
        const float betai = 2.0f * prf / b2f;
        frac = (betai < 2.0f) ? 1.0f : ((betai < 10.0f) ? (10.0f - betai) * 0.125f : 0.0f);
      }
      const double divBsymmi = fs[7];
      fs[0] -= (double)(bxf * frac) * divBsymmi;
      fs[1] -= (double)(byf * frac) * divBsymmi;
      fs[2] -= (double)(bzf * frac) * divBsymmi;
      if (valid) out.divBsymm[pid] = rhof * d2f_rn(divBsymmi);
    }
    if (valid) { fo[0] = fs[0]; fo[1] = fs[1]; fo[2] = fs[2]; }
    const float fxf = d2f_rn(fs[0]), fyf = d2f_rn(fs[1]), fzf = d2f_rn(fs[2]);
    const float f2f = fxf * fxf + fyf * fyf + fzf * fzf;
    const float drhodtf = pmf * d2f_rn(fs[4]);
    const float divvf = -drhodtf * rho1f;
    if (valid) out.divcurlv[pid] = divvf;
    double fxyz4 = 0.0;
    if (adiab) {
      if (p.ipdv_heating > 0) fxyz4 += (double)(prf * rho1f * rho1f * drhodtf);
      if (p.ishock_heating > 0) fxyz4 += fs[5];
      fxyz4 += fs[6];
    }
    if (p.mhd) {
      double *db = out.dBevol + 4 * (size_t)pid;
      if (valid) { db[0] = fs[8]; db[1] = fs[9]; db[2] = fs[10]; }
      if (p.psidecayfac > 0.0) {
        const float vclean = d2f_rn(p.overcleanfac) * vwavef;
        const float dtau = d2f_rn(p.psidecayfac) * vclean * h1f;
        if (valid) db[3] = (double)(-vclean * d2f_rn(fs[11]) * rho1f - psif * dtau - 0.5f * psif * divvf);
        dtclean = (double)(d2f_rn(p.C_cour) * hf / (vclean + TINY_F));
      }
    }
    const float vsigdtc = fmaxf(d2f_rn(vsm), vwavef);
    if (vsigdtc > TINY_F) dtc = (double)(d2f_rn(p.C_cour) * hf / (vsigdtc * fmaxf(d2f_rn(p.alpha), 1.0f)));
    if (adiab) {
      const double eni_ = rr[11];
      if (eni_ + dtc * fxyz4 < EPS_D && eni_ > EPS_D) fxyz4 = fxyz4 / (1.0 - dtc * fxyz4 / eni_);
      if (valid) fo[3] = fxyz4;
    }
    if (fabsf(f2f) > (float)EPS_D) dtf = (double)(d2f_rn(p.C_force) * sqrtf(hf / sqrtf(f2f)));
  } else {
    const double h1 = 1.0 / h;
    const double t3b = p.hfact * (1.0 / fabs(h));
    const double rho = pm * (t3b * t3b * t3b), rho1 = 1.0 / rho;
    double vwave = cs, bx = 0, by = 0, bz = 0, b2 = 0, psi = 0;
    if (p.mhd) {
      const double *m = jmhd + JMHD * (size_t)ip;
      bx = m[10] * rho; by = m[11] * rho; bz = m[12] * rho;
      psi = m[3];
      double pro2;
      get_stress(p, pr, cs, rho, rho1, bx, by, bz, pro2, vwave);
      b2 = bx * bx + by * by + bz * bz;
      const double divBsymmi = fs[7];
      double frac = 0.0;
      if (b2 > 0.0) {
        const double betai = 2.0 * pr / b2;
        frac = (betai < 2.0) ? 1.0 : ((betai < 10.0) ? (10.0 - betai) * 0.125 : 0.0);
      }
      fs[0] -= bx * divBsymmi * frac; fs[1] -= by * divBsymmi * frac; fs[2] -= bz * divBsymmi * frac;
      if (valid) out.divBsymm[pid] = (float)(rho * divBsymmi);
    }
    const double f2i = fs[0] * fs[0] + fs[1] * fs[1] + fs[2] * fs[2];
    if (valid) { fo[0] = fs[0]; fo[1] = fs[1]; fo[2] = fs[2]; }
    const double drhodti = pm * fs[4];
    const double divvi = -drhodti * rho1;
    if (valid) out.divcurlv[pid] = (float)divvi;
    double fxyz4 = 0.0;
    if (adiab) {
      if (p.ipdv_heating > 0) fxyz4 += pr * rho1 * rho1 * drhodti;
      if (p.ishock_heating > 0) fxyz4 += fs[5];
      fxyz4 += fs[6];
    }
    if (p.mhd) {
      double *db = out.dBevol + 4 * (size_t)pid;
      if (valid) { db[0] = fs[8]; db[1] = fs[9]; db[2] = fs[10]; }
      if (p.psidecayfac > 0.0) {
        const double vclean = p.overcleanfac * vwave;
        const double dtau = p.psidecayfac * vclean * h1;
        if (valid) db[3] = -vclean * fs[11] * rho1 - psi * dtau - 0.5 * psi * divvi;
        dtclean = p.C_cour * h / (vclean + TINY_D);
      }
    }
    const double vsigdtc = fmax(vsm, vwave);
    if (vsigdtc > TINY_D) dtc = p.C_cour * h / (vsigdtc * fmax(p.alpha, 1.0));
    if (adiab) {
      const double eni_ = rr[11];
      if (eni_ + dtc * fxyz4 < EPS_D && eni_ > EPS_D) fxyz4 = fxyz4 / (1.0 - dtc * fxyz4 / eni_);
      if (valid) fo[3] = fxyz4;
    }
    if (fabs(f2i) > EPS_D) dtf = p.C_force * sqrt(h / sqrt(f2i));
  }
  if (valid && (dtc < TINY_D || dtc > HUGE_D)) set_error(err, PH_ERR_DT);
  // warp minima on the bit patterns: for the positive timesteps the unsigned
  // order is the numeric order (as the atomic), and no FP64 instruction runs
  unsigned long long a = (unsigned long long)__double_as_longlong(valid ? dtc : HUGE_D);
  unsigned long long b = (unsigned long long)__double_as_longlong(valid ? fmin(dtf, dtclean) : HUGE_D);
  for (int o = 16; o > 0; o >>= 1) {
    a = min(a, __shfl_xor_sync(0xffffffffu, a, o));
    b = min(b, __shfl_xor_sync(0xffffffffu, b, o));
  }
  // an atomic only where it would lower the value read (which can only be
  // lower by then): 885k particles 96 -> 74 us
  if (lane_id() == 0) {
    unsigned long long *d = reinterpret_cast<unsigned long long *>(out.dtmin);
    if (a < *(volatile unsigned long long *)&d[0]) atomicMin(&d[0], a);
    if (b < *(volatile unsigned long long *)&d[1]) atomicMin(&d[1], b);
  }
  if (ind.ibin) {
    // force.F90:3273-3310: the particle's bin from min(dtc, dtf, dtclean), then
    // the Saitoh-Makino limiter (no more than one bin below any neighbour)
    int nb = 0, cnt = 0, small = 0;
    if (valid) {
      double dti = dtc;
      const double dtitmp = fmin(dtf, dtclean);
      if (dtitmp < dti + TINY_D && dtitmp < p.dtmax) dti = dtitmp;
      int bi = get_newbin(dti, p.dtmax, (int)ind.ibin[pid], ind, small);
      bi = max(bi, (int)psum[FSLOT_NBIN * ps + ip] - 1);
      // a bin above MAXBINS is reported (dt too small, the step stops before
      // its corrector); the stored bin stays within the bin tables
      bi = min(bi, MAXBINS);
      ind.ibin[pid] = (int8_t)bi;
      nb = bi; cnt = 1;
    }
    for (int o = 16; o > 0; o >>= 1) {
      nb = max(nb, __shfl_xor_sync(0xffffffffu, nb, o));
      cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
      small |= __shfl_xor_sync(0xffffffffu, small, o);
    }
    if (lane_id() == 0 && cnt) {
      atomicMax(&ind.counters[0], nb);
      atomicAdd(&ind.counters[1], cnt);
      if (small) atomicOr(&ind.counters[2], 1);
    }
  }
}

// wake the neighbours found by the active particles' force sums
// (force.F90:1346-1353): ibin_wake = max(ibin_wake, ibinnow - 1)
__global__ void k_wake_apply(int nt, const int *perm, const unsigned char *wakemark, int8_t *ibin_wake, int level) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nt || !wakemark[k]) return;
  const int pid = perm[k];
  if ((int)ibin_wake[pid] < level) ibin_wake[pid] = (int8_t)level;
}

// the stripes of each particle summed in stripe order through shared memory
// (the staged window's memory, no longer needed), written to psum by lanes < np
// (pm: the particle mass, left out of the pair terms, applied to every sum but
// d(rho)/dt's, which the finish multiplies)
template <bool IND, class Get>
__device__ __forceinline__ void store_pair_sums(PairSmem &sm, int lane, int np, int S, int s0, unsigned am,
                                                double *psum, int64_t ps, double pm, Get get) {
  constexpr int RW = IND ? NF + 2 : NF + 1;
  double *red = reinterpret_cast<double *>(&sm.st);
  __syncwarp();
  for (int k = 0; k < RW; ++k) red[lane * RW + k] = get(k);
  __syncwarp();
  if (lane < np) {
    double fs[NF];
    for (int k = 0; k < NF; ++k) fs[k] = 0.0;
    double vsm = 0.0, nb = 0.0;
    for (int q = 0; q < S; ++q) {
      const double *src = red + (lane * S + q) * RW;
      for (int k = 0; k < NF; ++k) fs[k] += src[k];
      vsm = fmax(vsm, src[NF]);
      if (IND) nb = fmax(nb, src[NF + 1]);
    }
    const size_t ip = (size_t)(s0 + (IND ? cell_pos(am, lane) : lane));
    for (int k = 0; k < NF; ++k) psum[k * ps + ip] = k != 4 ? pm * fs[k] : fs[k];
    psum[FSLOT_VSIG * ps + ip] = vsm;
    if (IND) psum[FSLOT_NBIN * ps + ip] = nb;
  }
}

// ------------------------------------------------------------------ FP64 pair terms
// The FP64 pair loops are bound by the FP64 pipe (2 lanes per SM and clock), so
// their cost is the number of FP64 instructions per pair. Each particle's own
// factors come from its record, no division or library square root is left
// (rsqrt_fast), the kernel needs no branch on q (kern_w), comparisons and
// maxima run on the integer pipe, and the particle mass is applied to the sums.
// i-side quantities (start_cell force.F90:2270-2340, compute_cell :2606-2629)
// of tree position i.
struct IFp64 {
  double h1, rho, c, pro2, vw, P, au, K, vx, vy, vz, u, gs, ab, avw, r21;
  double bx, by, bz, cl;
  double x, y, z;
};

template <bool MHD, bool GRAV>
__device__ __forceinline__ IFp64 ifp64_init(const Params &p, int i, const double *tx, const double *ty,
                                            const double *tz, const double *jrec, const double *jmhd) {
  IFp64 I;
  const double *r = jrec + JREC * (size_t)i;
  I.h1 = fabs(r[JR_H1]); I.rho = r[JR_RHO]; I.c = r[JR_C]; I.pro2 = r[JR_PRO2]; I.vw = r[JR_VW]; I.P = r[JR_P];
  I.au = r[JR_AU]; I.K = r[JR_K]; I.vx = r[JR_VX]; I.vy = r[JR_VY]; I.vz = r[JR_VZ]; I.u = r[JR_U];
  I.gs = GRAV ? r[JR_GS] : 0.0;
  I.ab = r[JR_AB]; I.avw = r[JR_AVW]; I.r21 = r[JR_R21];
  // start_cell takes 1/Omega = 1 where the stored value is not positive
  if (!(I.K < 0.0)) { const double h21 = I.h1 * I.h1; I.K = -0.75 * CNORMK * (h21 * h21); }
  I.bx = I.by = I.bz = I.cl = 0.0;
  if (MHD) {
    const double *m = jmhd + JMHD * (size_t)i;
    I.bx = m[JM_BX]; I.by = m[JM_BY]; I.bz = m[JM_BZ]; I.cl = m[JM_CL];
  }
  I.x = tx[i]; I.y = ty[i]; I.z = tz[i];
  return I;
}

// largest of two signal speeds as bit patterns (the first non-negative; a
// negative second one, whose clamp to zero changes no maximum, orders below)
__device__ __forceinline__ long long vmax_bits(long long a, double b) { return max(a, __double_as_longlong(b)); }

// softened self-gravity of one side (kernel_softening, kernel_cubic.f90:
// 101-120), u = 2 - q inside the kernel: fs/h^2 and, with POT, pot/h. For
// q >= 1 the reference's polynomials are expanded about q = 2,
//   q^2 fs = 1 - u^4 (1 - 4/5 u + u^2/6),  q pot = -1 + u^5 (1/10 - u/30).
template <bool POT>
__device__ __forceinline__ double softened(double u, double r, double y, double h1, double &pot) {
  if (__double2hiint(u) >= 0x3ff00000) {  // u >= 1: q <= 1
    const double q = r * h1, q2 = q * q;
    if (POT) pot = h1 * fma(q2, fma(q2, fma(0.1, q, -0.3), 2.0 / 3.0), -1.4);
    return h1 * h1 * q * fma(q2, fma(0.5, q, -1.2), 4.0 / 3.0);
  }
  const double u2 = u * u, u4 = u2 * u2;
  if (POT) pot = y * fma(u4 * u, fma(-1.0 / 30.0, u, 0.1), -1.0);
  return y * y * fma(-u4, fma(u, fma(1.0 / 6.0, u, -0.8), 1.0), 1.0);
}

// j-side pair sums of the symmetric evaluation: the force components, d(rho)/dt
// (f[4]), du/dt dissipation (f[5]) and conductivity (f[6]), then with MHD the
// divBsymm, dB/dt and div B diffusion terms, and the signal speed (last)
template <bool MHD>
struct NJS { static constexpr int n = MHD ? 12 : 7; };
// the psum slot of each j-side value
__device__ __forceinline__ int njs_slot(int v, bool mhd) {
  const int last = mhd ? 11 : 6;
  if (v == last) return NF;  // FSLOT_VSIG
  return v < 3 ? v : v + 1;  // 0,1,2 -> 0,1,2; 3.. -> 4..
}

// The plain 1/r^2 of a trial pair outside both kernels (force.F90:1991-2053).
__device__ __forceinline__ void far_pair_fp64(double dx, double dy, double dz, double y, double (&f)[NF]) {
  const double y3 = y * y * y;
  f[0] = fma(-dx, y3, f[0]); f[1] = fma(-dy, y3, f[1]); f[2] = fma(-dz, y3, f[2]);
  f[3] -= y;
}

// One trial pair (i, j) of compute_forces (force.F90:914-2060) in FP64 with the
// reference's neighbour test and cached-position rule (code, as separation_fp64
// takes it). The i-side sums (without the particle mass) go to f,
// vsigmax / nbi. With SYM the pair's contribution to j's own sums (j's force
// loop over i, the same pair term seen from j) is returned in jv; it is only
// requested for pairs without gravity and with global timesteps.
template <bool MHD, bool GRAV, bool IND, bool SYM>
__device__ __forceinline__ void force_pair_fp64(const Params &p, const IFp64 &I, int j, int code,
                                                const double *tx, const double *ty, const double *tz,
                                                const double *jrec, const double *jmhd,
                                                const int8_t *ibin_old_t, unsigned char *wakemark,
                                                double (&f)[NF], long long &vsigmax, int &nbi,
                                                double (&jv)[NJS<MHD>::n]) {
  const bool adiab = !p.isothermal;
  double dx, dy, dz;
  separation_fp64(p, I.x, I.y, I.z, j, code, tx, ty, tz, dx, dy, dz);
  const double *rj = jrec + JREC * (size_t)j;
  const double hj1 = rj[JR_H1];
  // With self-gravity the direction of a neighbour pair keeps the reference's
  // rounding (r^2 without contraction, the library's rsqrt): in solid-body
  // rotation, where such clouds start, dv . n is zero but for rounding, and
  // its sign switches the viscosity. The neighbours are a few per cent of the
  // trial list there, the other pairs are far_pair_fp64's.
  double r2, y;
  if (GRAV) {
    r2 = r2_exact(dx, dy, dz);
    y = r2 > TINY_D ? rsqrt(r2) : 0.0;
  } else {
    r2 = fma(dz, dz, fma(dy, dy, dx * dx));
    y = rsqrt_fast(r2);
  }
  const double r = r2 * y;
  double ui = fma(-r, I.h1, 2.0), uj = fma(-r, hj1, 2.0);
  bool qi_in = u_inside(ui), qj_in = u_inside(uj);
  if (u_near_edge(ui) || u_near_edge(uj)) {  // the reference's q^2 < 4
    qi_in = inside_exact(dx, dy, dz, I.h1);
    qj_in = inside_exact(dx, dy, dz, hj1);
  }
  if (!(qi_in || qj_in)) {
    if (GRAV) far_pair_fp64(dx, dy, dz, y, f);
    if (SYM) for (int v = 0; v < NJS<MHD>::n; ++v) jv[v] = 0.0;
    return;
  }
  if (IND) {  // force.F90:1346-1353: j is woken for the next step; the limiter's neighbour bin
    wakemark[j] = 1;
    nbi = max(nbi, (int)ibin_old_t[j]);
  }
  ui = qi_in ? ui : 0.0; uj = qj_in ? uj : 0.0;
  const double wi = kern_w(ui), wj = kern_w(uj);
  const double gi = I.K * fma(-wi, wi, ui * ui), gj = rj[JR_K] * fma(-wj, wj, uj * uj);
  double fgrav = 0.0;
  if (GRAV) {
    const double y2 = y * y;
    double phii = -y, none, fgi = y2, fgj = y2;
    if (qi_in) fgi = fma(I.gs, gi, softened<true>(ui, r, y, I.h1, phii));
    if (qj_in) fgj = fma(rj[JR_GS], gj, softened<false>(uj, r, y, hj1, none));
    fgrav = fgi + fgj;
    f[3] += phii;
  }
  // j's terms enter i's sums when q_j < 2, or always with MHD or an energy
  // equation (force.F90 usej); seen from j likewise
  const bool both = MHD || (adiab && !GRAV);
  const bool usej = both || qj_in, usei = both || qi_in;
  const double dvx = I.vx - rj[JR_VX], dvy = I.vy - rj[JR_VY], dvz = I.vz - rj[JR_VZ];
  double pv;  // dv . n
  if (GRAV) {
    const double nx = dx * y, ny = dy * y, nz = dz * y;
    pv = dvx * nx + dvy * ny + dvz * nz;
  } else {
    pv = y * fma(dvz, dz, fma(dvy, dy, dvx * dx));
  }
  const double vwj = rj[JR_VW];
  const double vsi = fma(-p.beta, pv, I.vw), vsj = fma(-p.beta, pv, vwj);
  vsigmax = vmax_bits(vsigmax, vsi);
  if (usej) vsigmax = vmax_bits(vsigmax, vsj);
  const double pgi = pv * gi;
  f[4] += pgi;
  double qi = 0.0, qj = 0.0;
  if (__double2hiint(pv) < 0) {  // approaching: artificial viscosity
    double vai = fma(-p.beta, pv, I.avw), vaj = fma(-p.beta, pv, rj[JR_AVW]);
    vai = __double2hiint(vai) < 0 ? 0.0 : vai; vaj = __double2hiint(vaj) < 0 ? 0.0 : vaj;
    qi = I.c * pv * vai;
    qj = rj[JR_C] * pv * vaj;
    if (adiab) f[5] = fma(qi, pgi, f[5]);
  }
  double gp = fma(rj[JR_PRO2] + qj, gj, (I.pro2 + qi) * gi);
  if (GRAV) gp = fma(0.5, fgrav, gp);
  double dendiss = 0.0;
  if (adiab && p.alphau != 0.0) {
    // conductivity: |dv . n| with self-gravity, else sqrt(2 |dP| / (rho_i + rho_j))
    // as sqrt(2) |dP| (|dP| (rho_i + rho_j))^(-1/2)
    double vsu;
    if (GRAV) vsu = fabs(pv);
    else { const double dP = fabs(I.P - rj[JR_P]); vsu = dP * rsqrt_fast(dP * (I.rho + rj[JR_RHO])); }
    dendiss = vsu * (I.u - rj[JR_U]) * fma(I.au, gi, rj[JR_AU] * gj);
    f[6] += dendiss;
  }
  if (SYM) {
    jv[3] = pv * gj;
    jv[4] = adiab ? qj * jv[3] : 0.0;
    jv[5] = -dendiss;
    long long b = vmax_bits(0, vsj);
    if (usei) b = vmax_bits(b, vsi);
    jv[NJS<MHD>::n - 1] = __longlong_as_double(b);
  }
  if constexpr (!MHD) {
    const double gpy = gp * y;
    f[0] = fma(-dx, gpy, f[0]); f[1] = fma(-dy, gpy, f[1]); f[2] = fma(-dz, gpy, f[2]);
    if (SYM) { jv[0] = dx * gpy; jv[1] = dy * gpy; jv[2] = dz * gpy; }
  } else {
    const double nx = dx * y, ny = dy * y, nz = dz * y;
    const double *mj = jmhd + JMHD * (size_t)j;
    const double bxj = mj[JM_BX], byj = mj[JM_BY], bzj = mj[JM_BZ];
    const double dBx = I.bx - bxj, dBy = I.by - byj, dBz = I.bz - bzj;
    const double projBj = fma(bzj, nz, fma(byj, ny, bxj * nx));
    const double projdB = fma(dBz, nz, fma(dBy, ny, dBx * nx));
    const double projBi = projBj + projdB;
    f[11] = fma(-projdB, gi, f[11]);  // div B diffusion
    const double tx_ = fma(-pv, nx, dvx), ty_ = fma(-pv, ny, dvy), tz_ = fma(-pv, nz, dvz);
    const double vsigB = sqrt_fast(fma(tz_, tz_, fma(ty_, ty_, tx_ * tx_)));
    const double dBdiss = vsigB * fma(I.ab, gi, rj[JR_AB] * gj);
    const double pmi = I.r21 * gi, pmj = rj[JR_R21] * gj;
    const double ti = pmi * projBi, tj = pmj * projBj;
    const double f7 = ti + tj;
    f[7] += f7;  // div B (symmetric)
    const double dpsi = fma(pmi, I.cl, pmj * mj[JM_CL]);
    f[8] = fma(-ti, dvx, fma(dBdiss, dBx, fma(-dpsi, nx, f[8])));
    f[9] = fma(-ti, dvy, fma(dBdiss, dBy, fma(-dpsi, ny, f[9])));
    f[10] = fma(-ti, dvz, fma(dBdiss, dBz, fma(-dpsi, nz, f[10])));
    double res = 0.0;
    if (p.iresistive_heating > 0 && adiab) {
      res = -0.5 * fma(dBz, dBz, fma(dBy, dBy, dBx * dBx)) * dBdiss;
      f[5] += res;
    }
    // anisotropic stress: -(S_i.n gi + S_j.n gj) with S = -(B/rho)(B/rho), i.e.
    // ti B_i + tj B_j
    if (SYM) {
      const double fx = fma(ti, I.bx, fma(tj, bxj, -nx * gp)), fy = fma(ti, I.by, fma(tj, byj, -ny * gp)),
                   fz = fma(ti, I.bz, fma(tj, bzj, -nz * gp));
      f[0] += fx; f[1] += fy; f[2] += fz;
      jv[0] = -fx; jv[1] = -fy; jv[2] = -fz;
      jv[4] += res;
      // from j: r -> -r, dv -> -dv, dB -> -dB; its own term -tj dv
      jv[6] = -f7;
      jv[7] = fma(-tj, dvx, fma(-dBdiss, dBx, dpsi * nx));
      jv[8] = fma(-tj, dvy, fma(-dBdiss, dBy, dpsi * ny));
      jv[9] = fma(-tj, dvz, fma(-dBdiss, dBz, dpsi * nz));
      jv[10] = -projdB * gj;
    } else {
      f[0] = fma(ti, I.bx, fma(tj, bxj, fma(-nx, gp, f[0])));
      f[1] = fma(ti, I.by, fma(tj, byj, fma(-ny, gp, f[1])));
      f[2] = fma(ti, I.bz, fma(tj, bzj, fma(-nz, gp, f[2])));
    }
  }
}

// Start of the per-side pair kernels: the cell of a warp, its active particles
// (IND: individual timesteps, inactive ones keep their forces) and the trial
// statistics. Returns false where the warp has nothing to do.
struct PairCell {
  int cell, s0, np, off, nleaf;
  unsigned am;
  float4 cc;  // centre, size
};
template <bool IND>
__device__ __forceinline__ bool pair_cell(PairCell &c, const Node *nodes, const int *leaves, int ncell,
                                          const int *cells, const int *cell_off, const int *cell_nleaf,
                                          const unsigned char *actf, const ForceOut &out, int *err) {
  const int a = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = lane_id();
  if (a >= ncell) return false;
  c.cell = cells ? cells[a] : a;
  const Node nd = nodes[leaves[c.cell]];
  c.np = nd.count; c.s0 = nd.start; c.am = 0u;
  if (c.np < 1 || c.np > MAXCELL) { if (lane == 0) set_error(err, PH_ERR_TREE); return false; }
  if (IND) c.am = cell_active_mask(actf, c.s0, nd.count, c.np);
  if (c.np == 0) return false;
  c.off = cell_off[c.cell]; c.nleaf = cell_nleaf[c.cell];
  c.cc = make_float4((float)nd.x, (float)nd.y, (float)nd.z, (float)nd.size);
  if (lane == 0) {
    atomicAdd(&out.stats[8], (unsigned long long)out.cell_ntrial[c.cell]);
    atomicAdd(&out.stats[10], (unsigned long long)c.np * (unsigned long long)out.cell_ntrial[c.cell]);
  }
  return true;
}

// totals of a cell -> psum: value k of particle il at idx = k np + il; the
// particle mass, left out of the pair terms, applied to every sum but
// d(rho)/dt's (which the finish multiplies) and the maxima
template <bool MHD, int NR, class S>
__device__ __forceinline__ void store_totals(const S &sm, int nv, int np, double pm, const double (&tot)[NR],
                                             double *psum, int64_t ps) {
  for (int r = 0; r < NR; ++r) {
    const int idx = lane_id() + 32 * r;
    if (idx < nv * np) {
      const int k = idx / np, slot = k < NJS<MHD>::n ? njs_slot(k, MHD) : FSLOT_NBIN;
      psum[slot * ps + sm.ipos[idx - k * np]] = slot == 4 || slot >= NF ? tot[r] : pm * tot[r];
    }
  }
}

// FP64 pairs from each side, without self-gravity: individual timesteps, and
// global ones when the symmetric loop is switched off
template <bool MHD, bool IND>
__global__ void __launch_bounds__(32 * MAX_WARPS) k_force(
    Params p, const Node *nodes, const int *leaves, int ncell, const LeafEntry *pool, const int *cell_off,
    const int *cell_nleaf, const double *tx, const double *ty, const double *tz, const double *th, const float4 *txf,
    const double *jrec, const double *jmhd, ForceOut out, double *psum, int64_t ps, double pf_hmin, const int *cells,
    const unsigned char *actf, const int8_t *ibin_old_t, unsigned char *wakemark, int *err) {
  constexpr int NV = NJS<MHD>::n + (IND ? 1 : 0), NR = (NV * MAXCELL + 31) / 32, VS = NJS<MHD>::n - 1;
  PairCell c;
  if (!pair_cell<IND>(c, nodes, leaves, ncell, cells, cell_off, cell_nleaf, actf, out, err)) return;
  extern __shared__ __align__(16) unsigned char dsm[];
  ListSmem &sm = reinterpret_cast<ListSmem *>(dsm)[threadIdx.x >> 5];
  const int lane = lane_id(), np = c.np;
  const float q2lim = 4.0f * 1.001f, INF = __int_as_float(0x7f800000);
  const float pf_hf = __double2float_ru(pf_hmin);
  auto accept = [&](float h) { return h > pf_hf ? q2lim * (h * h) : INF; };
  if (lane < np) {
    const int ip = c.s0 + (IND ? cell_pos(c.am, lane) : lane);
    float4 x = txf[ip];
    x.w = accept(d2f_rn(th[ip]));
    sm.xi[lane] = x;
    sm.ipos[lane] = ip;
  }
  const int qstride = LQ / np;
  double tot[NR];
  for (int r = 0; r < NR; ++r) tot[r] = 0.0;
  ListPos pos;
  __syncwarp();
  bool more = true;
  while (more) {
    int myc;
    more = SWEEP_END != sweep_list<false>(p, c.cc, np, pool, c.off, c.nleaf, txf, sm, qstride, pos, myc,
                                              [&](float h1) { return accept(__frcp_rn(h1)); });
    const QueueLanes ql = balance_queues(np, myc, sm);
    const int il = max(ql.il, 0);
    const IFp64 I = ifp64_init<MHD, false>(p, sm.ipos[il], tx, ty, tz, jrec, jmhd);
    double f[NF];
    for (int k = 0; k < NF; ++k) f[k] = 0.0;
    long long vsigmax = 0;  // largest signal speed (bit pattern)
    int nbi = 0;            // largest ibin_old of the SPH neighbours (individual timesteps)
    double jv[NJS<MHD>::n];
    for (int m = ql.m0; m < ql.c; m += ql.step)
      force_pair_fp64<MHD, false, IND, false>(p, I, sm.qj[il * qstride + m], sm.qc[il * qstride + m], tx, ty, tz, jrec,
                                              jmhd, ibin_old_t, wakemark, f, vsigmax, nbi, jv);
    static_assert(32 * NV <= LQ / 2, "lane sums staged in the queues' space");
    flush_lanes<NV>(np, sm, sm.red, tot,
        [&](int k) -> double {
          return k < VS ? f[njs_slot(k, MHD)] : (k == VS ? __longlong_as_double(vsigmax) : (double)nbi);
        },
        [](int k, double s, double v) -> double { return k < VS ? s + v : fmax_pos(s, v); });
  }
  store_totals<MHD>(sm, NV, np, p.massoftype, tot, psum, ps);
}

// FP64 pairs with self-gravity. The trial lists are long (thousands of
// particles at theta 0.5) and nearly all of it is far pairs, evaluated where
// they are tested: a lane per (particle, stripe) keeps their sums in registers.
template <bool MHD, bool IND>
__global__ void __launch_bounds__(32 * MAX_WARPS) k_force_grav(
    Params p, const Node *nodes, const int *leaves, int ncell, const LeafEntry *pool, const int *cell_off,
    const int *cell_nleaf, const double *tx, const double *ty, const double *tz, const double *th, const float4 *txf,
    const double *jrec, const double *jmhd, ForceOut out, double *psum, int64_t ps, double pf_hmin, const int *cells,
    const unsigned char *actf, const int8_t *ibin_old_t, unsigned char *wakemark, int *err) {
  const int w = threadIdx.x >> 5, lane = lane_id();
  const int a = blockIdx.x * (blockDim.x >> 5) + w;
  if (a >= ncell) return;
  const int cell = cells ? cells[a] : a;  // individual timesteps: the cells holding active particles
  const Node nd = nodes[leaves[cell]];
  const int np_all = nd.count, s0 = nd.start;
  if (np_all < 1 || np_all > MAXCELL) { if (lane == 0) set_error(err, PH_ERR_TREE); return; }
  // individual timesteps (IND): the cell's active particles take the lanes;
  // inactive ones keep their forces
  int np = np_all;
  unsigned am = 0u;
  if (IND) am = cell_active_mask(actf, s0, np_all, np);
  if (np == 0) return;
  const int S = 32 / np;
  const bool act = lane < np * S;
  const int il = act ? lane / S : 0, stripe = act ? lane % S : 0;
  const int i = s0 + (IND ? cell_pos(am, il) : il);
  const IFp64 I = ifp64_init<MHD, true>(p, i, tx, ty, tz, jrec, jmhd);
  const float4 xif = txf[i];
  const float hi21f = xif.w * xif.w;
  const bool pf_i = th[i] > pf_hmin;
  const float q2lim = 4.0f * 1.001f;
  const float pf_h1max = (float)(1.0 / pf_hmin);
  double f[NF];
  for (int k = 0; k < NF; ++k) f[k] = 0.0;
  long long vsigmax = 0;  // largest signal speed (bit pattern)
  int nbi = 0;  // largest ibin_old of the SPH neighbours (individual timesteps)
  const int off = cell_off[cell], nleaf = cell_nleaf[cell];
  if (lane == 0) {
    atomicAdd(&out.stats[8], (unsigned long long)out.cell_ntrial[cell]);
    atomicAdd(&out.stats[10], (unsigned long long)np * (unsigned long long)out.cell_ntrial[cell]);
  }
  const int ntrial = out.cell_ntrial[cell];
  extern __shared__ __align__(16) unsigned char dsm[];
  PairSmem &sm = reinterpret_cast<PairSmem *>(dsm)[w];
  Stage &stg = sm.st;
  for (int base = 0; base < ntrial; base += STAGE) {
    const int cnt = stage_window(p, pool, off, nleaf, ntrial, base, txf, stg);
    auto test = [&](int k) -> bool {
      if (stg.jidx[k] == i) return false;
      if (!pf_i) return true;
      const float4 xj = stg.pos[k];  // x, y, z (+ offset), 1/h
      if (xj.w >= pf_h1max) return true;
      float dxf = xif.x - xj.x, dyf = xif.y - xj.y, dzf = xif.z - xj.z;
      if (p.periodic) {
        if (fabsf(dxf) > 0.5f * p.dxboundf) dxf -= copysignf(p.dxboundf, dxf);
        if (fabsf(dyf) > 0.5f * p.dyboundf) dyf -= copysignf(p.dyboundf, dyf);
        if (fabsf(dzf) > 0.5f * p.dzboundf) dzf -= copysignf(p.dzboundf, dzf);
      }
      const float r2f = dxf * dxf + dyf * dyf + dzf * dzf;
      const bool near = r2f * fminf(hi21f, xj.w * xj.w) < q2lim;
      if (near) return true;
      // self-gravity: a trial pair provably outside both kernels (most of the
      // list) takes its 1/r^2 term here, in the dense test sweep, without being
      // queued with its record
      double dx, dy, dz;
      separation_fp64(p, I.x, I.y, I.z, stg.jidx[k], stg.code[k] | (base + k < CELLCACHE ? QC_CACHED : 0), tx, ty, tz,
                      dx, dy, dz);
      far_pair_fp64(dx, dy, dz, rsqrt_fast(fma(dz, dz, fma(dy, dy, dx * dx))), f);
      return false;
    };
    auto body = [&](int k) {
      double jv[NJS<MHD>::n];
      force_pair_fp64<MHD, true, IND, false>(p, I, stg.jidx[k], stg.code[k] | (base + k < CELLCACHE ? QC_CACHED : 0), tx,
                                             ty, tz, jrec, jmhd, ibin_old_t, wakemark, f, vsigmax, nbi, jv);
    };
    queue_window(cnt, S, act, il, stripe, sm.q, test, body);
  }
  store_pair_sums<IND>(sm, lane, np, S, s0, am, psum, ps, p.massoftype, [&](int q) -> double {
    return q < NF ? f[q] : (q == NF ? __longlong_as_double(vsigmax) : (double)nbi);
  });
}

// ------------------------------------------------------------------ symmetric FP64 pair loop
// Each unordered neighbour pair evaluated once (FP64, hydro and ideal MHD
// without self-gravity, global timesteps). A pair (i, j) of leaf cells A, B is
// evaluated by the cell whose leaf starts first in tree order: A takes the
// entries of its trial list whose first particle is at or after its own,
// which is a prefix of the list (the list is in decreasing order of first
// particle, the reference's stack order), and within its own leaf the pairs
// j > i. Every neighbour pair (q_i < 2 or q_j < 2) lies in both cells' trial
// lists (the walk opens every node within 2 max(h_i, h_j) of a cell), so it is
// evaluated exactly once; an entry present in one list only holds no
// neighbour pair and contributes nothing.
//
// The i-side sums are kept per lane as in k_force. The pair's contribution to
// j's sums is the same pair term seen from j (the reference evaluates it again
// in j's loop): it is added, in a fixed order, into a per-window array of the
// warp (lanes holding the same j are combined in lane order first), and each
// window's array is written to jbuf at j's flattened trial index of A's list.
// k_force_gather then adds, for every particle, the contributions that the
// cells before it left for it, in its own list's order. Pair terms and
// neighbour tests are those of force_pair_fp64 (the reference's rounding and
// cached-position rule from the evaluating cell's list); seen from j they differ
// from the reference's own evaluation by rounding only.
// (Work decomposition: sym_pairs in ph_walk.cuh. Per launch at 64^3 1.73 ms,
// against 2.45 for a lane per particle and stripe.)
template <bool MHD>
__global__ void __launch_bounds__(32) k_force_sym(
    Params p, const Node *nodes, const int *leaves, int ncell, const LeafEntry *pool, const int *cell_off,
    const int *cell_nleaf, const double *tx, const double *ty, const double *tz, const double *th,
    const float4 *txf, const double *jrec, const double *jmhd, ForceOut out, double *psum, int64_t ps, double pf_hmin,
    const int *toff, double *jbuf, int64_t jstride, int *err) {
  constexpr int NJ = NJS<MHD>::n, NR = (NJ * MAXCELL + 31) / 32;
  const int lane = lane_id(), cell = blockIdx.x;
  if (cell >= ncell) return;
  const Node nd = nodes[leaves[cell]];
  const int np = nd.count, s0 = nd.start;
  if (np < 1 || np > MAXCELL || np > p.minpart) { if (lane == 0) set_error(err, PH_ERR_TREE); return; }
  extern __shared__ __align__(16) unsigned char dsm[];
  ListSmemK &sm = *reinterpret_cast<ListSmemK *>(dsm);
  const float q2lim = 4.0f * 1.001f, INF = __int_as_float(0x7f800000);
  const float pf_hf = __double2float_ru(pf_hmin);
  auto accept = [&](float h) { return h > pf_hf ? q2lim * (h * h) : INF; };
  if (lane < np) {
    float4 x = txf[s0 + lane];
    x.w = accept(d2f_rn(th[s0 + lane]));
    sm.xi[lane] = x;
    sm.ipos[lane] = s0 + lane;
  }
  const int off = cell_off[cell];
  int nown, town;
  owned_prefix(pool, off, cell_nleaf[cell], s0, nown, town);
  if (lane == 0) {
    atomicAdd(&out.stats[8], (unsigned long long)out.cell_ntrial[cell]);
    atomicAdd(&out.stats[10], (unsigned long long)np * (unsigned long long)town);
  }
  const float4 cc = make_float4((float)nd.x, (float)nd.y, (float)nd.z, (float)nd.size);
  double tot[NR];
  for (int r = 0; r < NR; ++r) tot[r] = 0.0;
  IFp64 I;
  double f[NF];
  long long vsigmax = 0;  // largest signal speed (bit pattern)
  int nbi = 0;
  sym_pairs<NJ, true>(p, cc, np, pool, off, nown, txf, sm, (int64_t)toff[off], jbuf, jstride, tot,
      [&](float h1) { return accept(__frcp_rn(h1)); },
      [&](int il) {
        I = ifp64_init<MHD, false>(p, s0 + il, tx, ty, tz, jrec, jmhd);
        for (int k = 0; k < NF; ++k) f[k] = 0.0;
        vsigmax = 0;
      },
      [&](int j, int code, double (&jv)[NJ]) {
        force_pair_fp64<MHD, false, false, true>(p, I, j, code, tx, ty, tz, jrec, jmhd, nullptr, nullptr, f, vsigmax,
                                                 nbi, jv);
      },
      [&](int k) -> double { return k == NJ - 1 ? __longlong_as_double(vsigmax) : f[njs_slot(k, MHD)]; });
  store_totals<MHD>(sm, NJ, np, p.massoftype, tot, psum, ps);
}

// Per leaf cell B: add to its particles' pair sums the j-side contributions
// that k_force_sym left in jbuf: its own leaf's (the self entry) and those of
// every cell A before it in tree order whose list holds B (found by a binary
// search of A's list, which is in decreasing order of first particle), in the
// order of B's own trial list.
template <bool MHD>
__global__ void k_force_gather(const Node *nodes, const int *leaves, int ncell, const LeafEntry *pool,
                               const int *cell_off, const int *cell_nleaf, const int *cell_at, const int *toff,
                               const double *jbuf, int64_t jstride, double pm, double *psum, int64_t ps,
                               int *err) {
  constexpr int NJ = NJS<MHD>::n;
  const unsigned FULL = 0xffffffffu;
  const int w = threadIdx.x >> 5, lane = lane_id();
  const int cell = blockIdx.x * (blockDim.x >> 5) + w;
  if (cell >= ncell) return;
  const Node nd = nodes[leaves[cell]];
  const int np = nd.count, s0 = nd.start;
  if (np < 1 || np > MAXCELL) return;
  const int off = cell_off[cell], nleaf = cell_nleaf[cell];
  // per lane: the sums of (value v, particle t) pairs c = lane, lane + 32, ...
  constexpr int NC = (NJ * MAXCELL + 31) / 32;
  double acc[NC];
  for (int r = 0; r < NC; ++r) acc[r] = 0.0;
  // incoming entries: the suffix of B's list starting at or before s0
  for (int e0 = nleaf - 1; e0 >= 0; e0 -= 32) {
    // lanes take entries e0, e0-1, ... (descending index = ascending start),
    // then the warp walks them back in list order
    const int e = e0 - lane;
    int slot = -1;
    bool in = false;
    if (e >= 0) {
      const LeafEntry le = pool[off + e];
      in = le.start <= s0;
      if (le.start == s0) {
        slot = toff[off + e];
      } else if (in) {
        const int A = cell_at[le.start];
        const int aoff = cell_off[A];
        int lo = 0, hi = cell_nleaf[A] - 1;
        while (lo <= hi) {  // A's list: starts in decreasing order
          const int mid = (lo + hi) >> 1;
          const int st = pool[aoff + mid].start;
          if (st == s0) { slot = toff[aoff + mid]; break; }
          if (st > s0) lo = mid + 1; else hi = mid - 1;
        }
      }
    }
    const unsigned inb = __ballot_sync(FULL, in);
    const int nin = __popc(inb);  // a prefix of the lanes (suffix of the list)
    for (int q = nin - 1; q >= 0; --q) {  // in list order (lane nin-1 holds the first incoming entry)
      const int sl = __shfl_sync(FULL, slot, q);
      if (sl < 0) continue;
      for (int r = 0; r < NC; ++r) {
        const int c = lane + 32 * r;
        const int v = c / MAXCELL, t = c % MAXCELL;
        if (v < NJ && t < np) {
          const double y = jbuf[(int64_t)v * jstride + sl + t];
          acc[r] = (v == NJ - 1) ? fmax_pos(acc[r], y) : acc[r] + y;
        }
      }
    }
    if (nin < 32) break;  // the rest of the list starts after s0
  }
  for (int r = 0; r < NC; ++r) {
    const int c = lane + 32 * r;
    const int v = c / MAXCELL, t = c % MAXCELL;
    if (v < NJ && t < np) {
      double *dst = psum + (int64_t)njs_slot(v, MHD) * ps + s0 + t;
      // v == 3: d(rho)/dt, without the particle mass
      *dst = (v == NJ - 1) ? fmax_pos(*dst, acc[r]) : (v == 3 ? *dst + acc[r] : fma(pm, acc[r], *dst));
    }
  }
}

// trial entries each cell evaluates in the symmetric loop: those of its list
// entries starting at or after its own first particle
__global__ void k_owned_trials(const Node *nodes, const int *leaves, int ncell, const LeafEntry *pool,
                               const int *cell_off, const int *cell_nleaf, int *town) {
  const int w = threadIdx.x >> 5, lane = lane_id();
  const int cell = blockIdx.x * (blockDim.x >> 5) + w;
  if (cell >= ncell) return;
  const int s0 = nodes[leaves[cell]].start;
  const int off = cell_off[cell], nleaf = cell_nleaf[cell];
  int t = 0;
  for (int e = lane; e < nleaf; e += 32) {
    const LeafEntry le = pool[off + e];
    if (le.start >= s0) t += le.cc & 255;
  }
  t = warp_sum_int(t);
  if (lane == 0) town[cell] = t;
}

// flattened trial index of every pool entry: the cell's base (scan of the
// cells' trial counts) plus the counts of the entries before it in its list
__global__ void k_entry_offsets(int ncell, const int *cell_off, const int *cell_nleaf, const int *cell_tbase,
                                const LeafEntry *pool, int *toff) {
  const int w = threadIdx.x >> 5, lane = lane_id();
  const int cell = blockIdx.x * (blockDim.x >> 5) + w;
  if (cell >= ncell) return;
  const int off = cell_off[cell], nleaf = cell_nleaf[cell];
  int acc = cell_tbase[cell];
  for (int e0 = 0; e0 < nleaf; e0 += 32) {
    const int e = e0 + lane;
    const int cnt = e < nleaf ? (pool[off + e].cc & 255) : 0;
    int x = cnt;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (e < nleaf) toff[off + e] = acc + x - cnt;
    acc += __shfl_sync(0xffffffffu, x, 31);
  }
}

// cell index of every leaf, at the tree position of its first particle
__global__ void k_cell_at(const Node *nodes, const int *leaves, int ncell, int *cell_at) {
  const int cell = blockIdx.x * blockDim.x + threadIdx.x;
  if (cell < ncell) cell_at[nodes[leaves[cell]].start] = cell;
}

// ------------------------------------------------------------------ mixed precision
// Precision form: positions stay FP64, and a pair's separation is their
// difference rounded to FP32, formed from high and low FP32 parts (separation_2f;
// in FP64 for the closest pairs and those across a periodic image); W, grad W and
// every pair term are evaluated in FP32 and accumulated per particle in FP32 with
// compensated (Kahan) summation.

__device__ __forceinline__ float grkernf(float q) {
  if (q < 1.0f) return q * (2.25f * q - 3.0f);
  if (q < 2.0f) { float t = q - 2.0f; return -0.75f * (t * t); }
  return 0.0f;
}
// kernel_softening in FP32. For 1 <= q < 2 the reference's polynomials
// cancel to a few digits near q = 2 (numerators ~30 out of terms ~1000), so
// they are evaluated in t = 2 - q, where they read
//   30 q^2 fs = 30 - 30 t^4 + 24 t^5 - 5 t^6,  30 q pot = -30 + 3 t^5 - t^6
// (the same polynomials, expanded about q = 2).
__device__ __forceinline__ void kernel_softeningf(float q2, float q, float &pot, float &fs) {
  if (q < 1.0f) {
    float q4 = q2 * q2;
    pot = q4 * q * 0.1f - 0.3f * q4 + (2.0f / 3.0f) * q2 - 1.4f;
    fs = q * (15.0f * q2 * q - 36.0f * q2 + 40.0f) * (1.0f / 30.0f);
  } else if (q < 2.0f) {
    const float t = 2.0f - q, t4 = (t * t) * (t * t);
    const float q1 = 1.0f / q;
    pot = (-1.0f + t4 * t * (0.1f - t * (1.0f / 30.0f))) * q1;
    fs = (1.0f - t4 * (1.0f - t * (0.8f - t * (1.0f / 6.0f)))) * (q1 * q1);
  } else {
    pot = -1.0f / q;
    fs = 1.0f / q2;
  }
}


// The i-side quantities of the mixed pair loop for tree position i (its FP32
// record, positions as two floats).
template <bool MHD>
struct IMix {
  float h1, rho, c, pro2, vw, P, au, K, vx, vy, vz, u, gs, ab, avw, r21;
  float bx, by, bz, cl;
  Sep2 s;
};
template <bool MHD>
__device__ __forceinline__ IMix<MHD> imix_init(int i, const float4 *txf, const float4 *txl, const float *jrecf,
                                               const float *jmhdf) {
  IMix<MHD> I;
  const float4 *r4 = reinterpret_cast<const float4 *>(jrecf + JRECF * (size_t)i);
  const float4 a = r4[0], b = r4[1], c = r4[2], d = r4[3];
  I.h1 = a.x; I.rho = a.y; I.c = a.z; I.pro2 = a.w; I.vw = b.x; I.P = b.y; I.au = b.z; I.K = b.w;
  I.vx = c.x; I.vy = c.y; I.vz = c.z; I.u = c.w; I.gs = d.x; I.ab = d.y; I.avw = d.z; I.r21 = d.w;
  // start_cell takes 1/Omega = 1 where the stored value is not positive
  if (!(I.K > 0.0f)) I.K = (I.h1 * I.h1) * (I.h1 * I.h1) * (float)CNORMK;
  I.bx = I.by = I.bz = I.cl = 0.0f;
  if (MHD) {
    const float *m = jmhdf + JMHDF * (size_t)i;
    I.bx = m[JM_BX]; I.by = m[JM_BY]; I.bz = m[JM_BZ]; I.cl = m[JM_CL];
  }
  I.s = sep2_init(txf, txl, i);
  return I;
}

// the plain 1/r^2 of a trial pair outside both kernels (force.F90:1991-2053)
__device__ __forceinline__ void far_pair_mixed(float dx, float dy, float dz, float r2, Kahan (&f)[NF]) {
  const float y = rsqrt_nr(r2), y3 = y * y * y;
  f[0].add(-dx * y3); f[1].add(-dy * y3); f[2].add(-dz * y3);
  f[3].add(-y);
}

// The trial particle's FP32 record. Loaded after the separation, whose
// registers are free by then (cloud of 2M particles 91.6 -> 90.1 ms); with MHD
// before it, to have the longer pair's operands under way (force of 128^3
// particles 4.54 -> 4.52 ms).
struct MixRec {
  float4 a, b, c, d;
  __device__ __forceinline__ void load(const float *jrecf, int j) {
    const float4 *r4 = reinterpret_cast<const float4 *>(jrecf + JRECF * (size_t)j);
    a = r4[0]; b = r4[1]; c = r4[2]; d = r4[3];
  }
};

// One trial pair of compute_forces (force.F90:914-2060) in FP32 (sums without
// the particle mass)
template <bool MHD, bool GRAV, bool IND>
__device__ __forceinline__ void force_pair_mixed(const Params &p, const IMix<MHD> &I, int j, float dx, float dy,
                                                 float dz, float rij2, const MixRec &jr, const float *jmhdf,
                                                 const int8_t *ibin_old_t,
                                                 unsigned char *wakemark, Kahan (&f)[NF], float &vsigmax, int &nbi) {
  const bool adiab = !p.isothermal;
  const float beta = (float)p.beta;
  const float4 ra = jr.a, rb = jr.b, rc = jr.c, rd = jr.d;
  const float hj1 = ra.x;
  const float q2i = rij2 * (I.h1 * I.h1), q2j = rij2 * (hj1 * hj1);
  const bool qi_in = q2i < 4.0f, qj_in = q2j < 4.0f;
  if (!(qi_in || qj_in)) {
    if (GRAV) far_pair_mixed(dx, dy, dz, rij2, f);
    return;
  }
  if (IND) {  // force.F90:1346-1353: j is woken for the next step; the limiter's neighbour bin
    wakemark[j] = 1;
    nbi = max(nbi, (int)ibin_old_t[j]);
  }
  // coincident particles: no direction, rij1 = 0 (force.F90:1293-1298)
  const float rij1 = rij2 > TINY_F ? rsqrt_nr(rij2) : 0.0f;
  const float rij = rij2 * rij1;
  const float qi = rij * I.h1, qj = rij * hj1;
  const float gi = qi_in ? grkernf(qi) * I.K : 0.0f, gj = qj_in ? grkernf(qj) * rb.w : 0.0f;
  float fgrav = 0.0f;
  if (GRAV) {
    const float y2 = rij1 * rij1;
    float phii = -rij1, fgi = y2, fgj = y2;
    if (qi_in) {
      float fmi;
      kernel_softeningf(q2i, qi, phii, fmi);
      phii *= I.h1;
      fgi = fmi * (I.h1 * I.h1) + I.gs * gi;
    }
    if (qj_in) {
      float phij, fmj;
      kernel_softeningf(q2j, qj, phij, fmj);
      fgj = fmj * (hj1 * hj1) + rd.x * gj;
    }
    fgrav = 0.5f * (fgi + fgj);
    f[3].add(phii);
  }
  const float nx = dx * rij1, ny = dy * rij1, nz = dz * rij1;
  // j's terms enter when q_j < 2, or always with MHD or an energy equation
  const bool usej = MHD || (adiab && !GRAV) || qj_in;
  const float dvx = I.vx - rc.x, dvy = I.vy - rc.y, dvz = I.vz - rc.z;
  const float pv = dvx * nx + dvy * ny + dvz * nz;
  vsigmax = fmaxf(vsigmax, I.vw - beta * pv);  // starts at 0
  if (usej) vsigmax = fmaxf(vsigmax, rb.x - beta * pv);
  float qri = 0.0f, qrj = 0.0f;
  if (pv < 0.0f) {
    qri = I.c * fmaxf(I.avw - beta * pv, 0.0f) * pv;
    if (usej) qrj = ra.z * fmaxf(rd.z - beta * pv, 0.0f) * pv;
    if (adiab) f[5].add(qri * pv * gi);
  }
  const float gradp = (I.pro2 + qri) * gi + (usej ? (ra.w + qrj) * gj : 0.0f) + fgrav;
  if (adiab) {
    const float vsigu = GRAV ? fabsf(pv) : sqrt_nr(fabsf(I.P - rb.y) * __fdividef(2.0f, I.rho + ra.y));
    f[6].add(vsigu * (I.u - rc.w) * (I.au * gi + (usej ? rb.z * gj : 0.0f)));
  }
  float sx = 0.0f, sy = 0.0f, sz = 0.0f;
  if (MHD) {
    const float4 mj = *reinterpret_cast<const float4 *>(jmhdf + JMHDF * (size_t)j);
    const float clj = jmhdf[JMHDF * (size_t)j + JM_CL];
    const float dBx = I.bx - mj.x, dBy = I.by - mj.y, dBz = I.bz - mj.z;
    const float projBi = I.bx * nx + I.by * ny + I.bz * nz;
    const float projBj = mj.x * nx + mj.y * ny + mj.z * nz;
    const float projdB = dBx * nx + dBy * ny + dBz * nz;
    f[11].add(-projdB * gi);
    const float tx_ = dvx - pv * nx, ty_ = dvy - pv * ny, tz_ = dvz - pv * nz;
    const float vsigB = sqrt_nr(tx_ * tx_ + ty_ * ty_ + tz_ * tz_);
    const float dBdiss = (I.ab * gi + rd.y * gj) * vsigB;
    if (p.iresistive_heating > 0 && adiab) f[5].add(-0.5f * (dBx * dBx + dBy * dBy + dBz * dBz) * dBdiss);
    const float pmi = I.r21 * gi, pmj = rd.w * gj;
    const float ti = pmi * projBi, tj = pmj * projBj;
    f[7].add(ti + tj);
    const float dpsi = pmi * I.cl + pmj * clj;
    f[8].add(-ti * dvx + dBdiss * dBx - dpsi * nx);
    f[9].add(-ti * dvy + dBdiss * dBy - dpsi * ny);
    f[10].add(-ti * dvz + dBdiss * dBz - dpsi * nz);
    // anisotropic stress: -(S_i.n gi + S_j.n gj) with S = -(B/rho)(B/rho)
    sx = ti * I.bx + tj * mj.x; sy = ti * I.by + tj * mj.y; sz = ti * I.bz + tj * mj.z;
  }
  f[0].add(MHD ? sx - nx * gradp : -nx * gradp);
  f[1].add(MHD ? sy - ny * gradp : -ny * gradp);
  f[2].add(MHD ? sz - nz * gradp : -nz * gradp);
  f[4].add(pv * gi);
}

// 24 warps per SM (MHD 20) hide the pair's dependency chain best: at 64^3 the
// register allocation left alone (108 registers, 16 warps) takes 0.513 ms (MHD
// 0.75), this bound 0.47 (0.62), one more block 0.49 (0.70); self-gravity at
// 300001 particles 2.77 -> 2.39 ms.
//
// A velocity iteration evaluates the force again with the same positions and
// smoothing lengths, so its pairs, their separations and their lanes are those
// of the evaluation before. With REC the kernel writes each drain's pairs as the
// lanes take them: a row with every lane's particle, the number of pair rows and
// the cell's next drain, then rows of 32 (separation, trial particle; -1: idle
// lane). The rows are counted on past the buffer's end; the host then takes no
// part of the record.
struct PairRec {
  float4 *rows;    // rows of 32
  int *cell;       // first row of every cell
  int cap, *top;   // rows there are, rows taken
};
template <bool MHD, bool IND, bool REC>
__global__ void __launch_bounds__(32 * MAX_WARPS, MHD ? 5 : 6) k_force_mixed(
    Params p, const Node *nodes, const int *leaves, int ncell, const LeafEntry *pool, const int *cell_off,
    const int *cell_nleaf, const double *tx, const double *ty, const double *tz, const float4 *txf, const float4 *txl,
    const float *jrecf, const float *jmhdf, ForceOut out, double *psum, int64_t ps, const int *cells,
    const unsigned char *actf, const int8_t *ibin_old_t, unsigned char *wakemark, PairRec rec,
    int *err) {
  constexpr int NV = NJS<MHD>::n + (IND ? 1 : 0), NR = (NV * MAXCELL + 31) / 32, VS = NJS<MHD>::n - 1;
  PairCell c;
  if (!pair_cell<IND>(c, nodes, leaves, ncell, cells, cell_off, cell_nleaf, actf, out, err)) return;
  extern __shared__ __align__(16) unsigned char dsm[];
  ListSmem &sm = reinterpret_cast<ListSmem *>(dsm)[threadIdx.x >> 5];
  const int lane = lane_id(), np = c.np;
  const float q2lim = 4.0f * 1.001f;
  if (lane < np) {
    const int ip = c.s0 + (IND ? cell_pos(c.am, lane) : lane);
    float4 x = txf[ip];
    x.w = __fdividef(q2lim, x.w * x.w);
    sm.xi[lane] = x;
    sm.ipos[lane] = ip;
  }
  const int qstride = LQ / np;
  double tot[NR];
  for (int r = 0; r < NR; ++r) tot[r] = 0.0;
  ListPos pos;
  __syncwarp();
  bool more = true;
  int prev = -1;
  while (more) {
    int myc;
    more = SWEEP_END != sweep_list<false>(p, c.cc, np, pool, c.off, c.nleaf, txf, sm, qstride, pos, myc,
                                              [&](float h1) { return __fdividef(q2lim, h1 * h1); });
    const QueueLanes ql = balance_queues(np, myc, sm);
    const int il = max(ql.il, 0);
    float4 *rd = nullptr;  // the lane's next record slot
    int nit = 0;
    if constexpr (REC) {
      const int nst = ql.c > ql.m0 ? (ql.c - ql.m0 + ql.step - 1) / ql.step : 0;
      nit = (int)__reduce_max_sync(0xffffffffu, (unsigned)nst);
      int row = 0;
      if (lane == 0) row = atomicAdd(rec.top, 1 + nit);
      row = __shfl_sync(0xffffffffu, row, 0);
      if (row >= 0 && row <= rec.cap - (1 + nit)) {
        rd = rec.rows + 32 * (size_t)row + lane;
        *rd = make_float4(__int_as_float(ql.il), __int_as_float(nit), __int_as_float(-1), 0.0f);
        __syncwarp();
        if (lane == 0 && prev < 0) rec.cell[c.cell] = row;
        if (prev >= 0) rec.rows[32 * (size_t)prev + lane].z = __int_as_float(row);
        prev = row;
        rd += 32;
      }
    }
    const IMix<MHD> I = imix_init<MHD>(sm.ipos[il], txf, txl, jrecf, jmhdf);
    Kahan f[NF];
    float vsigmax = 0.0f;
    int nbi = 0;
    for (int m = ql.m0; m < ql.c; m += ql.step) {
      const int j = sm.qj[il * qstride + m];
      MixRec jr;
      if (MHD) jr.load(jrecf, j);
      float dx, dy, dz, r2;
      separation_2f(p, I.s, j, sm.qc[il * qstride + m] & 63, txf[j], txl[j], tx, ty, tz, dx, dy, dz, r2);
      if (!MHD) jr.load(jrecf, j);
      if (REC && rd) { *rd = make_float4(dx, dy, dz, __int_as_float(j)); rd += 32; --nit; }
      force_pair_mixed<MHD, false, IND>(p, I, j, dx, dy, dz, r2, jr, jmhdf, ibin_old_t, wakemark, f, vsigmax, nbi);
    }
    if (REC && rd)
      for (; nit > 0; --nit, rd += 32) *rd = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(-1));
    static_assert(32 * NV <= LQ / 2, "lane sums staged in the queues' space");
    flush_lanes<NV>(np, sm, sm.red, tot,
        [&](int k) -> double { return k < VS ? f[njs_slot(k, MHD)].value() : (k == VS ? (double)vsigmax : (double)nbi); },
        [](int k, double s, double v) -> double { return k < VS ? s + v : fmax_pos(s, v); });
  }
  store_totals<MHD>(sm, NV, np, p.massoftype, tot, psum, ps);
}

// The evaluations after a recorded one: same pairs, same lanes, same sums in the
// same order (bit-identical results) without the sweep, half of the kernel above
// (189 of 395 us at 64^3), and without the separations and their two gathers
// per pair; what remains waits for the trial particles' records. Three Sedov
// steps of 128^3 particles, five evaluations each: swept 99.5, with only the
// trial particles recorded 88.1 ms; and, the tree faster since, 82.7 against
// 77.7 ms with separations. With the Cullen-Dehnen switch at 96^3: 58.3, 47.2
// and 45.1 ms. 24 warps per SM: 20 or 28 make the Sedov steps 2 % longer, 32
// 14 %.
template <int NV>
struct ReplaySmem {
  double red[32 * NV];
  int ipos[MAXCELL];
  unsigned char first[MAXCELL], lanes[MAXCELL];
};
template <bool MHD>
__global__ void __launch_bounds__(32 * MAX_WARPS, MHD ? 5 : 6) k_force_replay(
    Params p, const Node *nodes, const int *leaves, int ncell, const int *cell_off, const int *cell_nleaf,
    const float4 *txf, const float4 *txl, const float *jrecf, const float *jmhdf, ForceOut out, double *psum, int64_t ps,
    PairRec rec, int *err) {
  constexpr int NV = NJS<MHD>::n, NR = (NV * MAXCELL + 31) / 32, VS = NV - 1;
  __shared__ ReplaySmem<NV> smem[MAX_WARPS];
  ReplaySmem<NV> &sm = smem[threadIdx.x >> 5];
  PairCell c;
  if (!pair_cell<false>(c, nodes, leaves, ncell, nullptr, cell_off, cell_nleaf, nullptr, out, err)) return;
  const int lane = lane_id(), np = c.np;
  if (lane < np) { sm.ipos[lane] = c.s0 + lane; sm.lanes[lane] = 0; sm.first[lane] = 0; }
  double tot[NR];
  for (int r = 0; r < NR; ++r) tot[r] = 0.0;
  __syncwarp();
  for (int row = rec.cell[c.cell], last = -1; row >= 0;) {
    // a cell's drains took their rows one after the other, each inside the
    // buffer: anything else is not a record, and following it need not end
    if (row <= last || row >= rec.cap) { if (lane == 0) set_error(err, PH_ERR_LIST); break; }
    const float4 *d = rec.rows + 32 * (size_t)row + lane;
    const float4 head = d[0];
    const int own = __float_as_int(head.x), il = max(own, 0);
    const int nit = min(__shfl_sync(0xffffffffu, __float_as_int(head.y), 0), rec.cap - 1 - row);
    last = row;
    row = __shfl_sync(0xffffffffu, __float_as_int(head.z), 0);
    const unsigned g = __match_any_sync(0xffffffffu, own);
    if (lane < np) sm.lanes[lane] = 0;
    __syncwarp();
    if (own >= 0 && lane == __ffs(g) - 1) { sm.first[il] = (unsigned char)lane; sm.lanes[il] = (unsigned char)__popc(g); }
    const IMix<MHD> I = imix_init<MHD>(sm.ipos[il], txf, txl, jrecf, jmhdf);
    Kahan f[NF];
    float vsigmax = 0.0f;
    int nbi = 0;
    const float4 none = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(-1));
    d += 32;
    float4 next = nit > 0 ? d[0] : none;
    for (int t = 0; t < nit; ++t) {
      const float4 a = next;
      d += 32;
      next = t + 1 < nit ? d[0] : none;
      const int j = __float_as_int(a.w);
      if (j >= 0) {
        MixRec jr;
        jr.load(jrecf, j);
        force_pair_mixed<MHD, false, false>(p, I, j, a.x, a.y, a.z, a.x * a.x + a.y * a.y + a.z * a.z, jr, jmhdf,
                                            nullptr, nullptr, f, vsigmax, nbi);
      }
    }
    flush_lanes<NV>(np, sm, sm.red, tot,
        [&](int k) -> double { return k < VS ? f[njs_slot(k, MHD)].value() : (double)vsigmax; },
        [](int k, double s, double v) -> double { return k < VS ? s + v : fmax_pos(s, v); });
  }
  store_totals<MHD>(sm, NV, np, p.massoftype, tot, psum, ps);
}

// Self-gravity: as k_force_grav, far pairs evaluated where they are tested.
template <bool MHD, bool IND>
__global__ void __launch_bounds__(32 * MAX_WARPS, MHD ? 5 : 6) k_force_mixed_grav(
    Params p, const Node *nodes, const int *leaves, int ncell, const LeafEntry *pool, const int *cell_off,
    const int *cell_nleaf, const double *tx, const double *ty, const double *tz, const float4 *txf, const float4 *txl,
    const float *jrecf, const float *jmhdf, ForceOut out, double *psum, int64_t ps, const int *cells,
    const unsigned char *actf, const int8_t *ibin_old_t, unsigned char *wakemark, int *err) {
  PairCell c;
  if (!pair_cell<IND>(c, nodes, leaves, ncell, cells, cell_off, cell_nleaf, actf, out, err)) return;
  const int lane = lane_id(), np = c.np;
  const int S = 32 / np;
  const bool act = lane < np * S;
  const int il = act ? lane / S : 0, stripe = act ? lane % S : 0;
  const int i = c.s0 + (IND ? cell_pos(c.am, il) : il);
  const IMix<MHD> I = imix_init<MHD>(i, txf, txl, jrecf, jmhdf);
  const float hi21f = I.h1 * I.h1;
  const float q2lim = 4.0f * 1.001f;
  const float hLx = 0.5f * p.dxboundf, hLy = 0.5f * p.dyboundf, hLz = 0.5f * p.dzboundf;
  Kahan f[NF];
  float vsigmax = 0.0f;
  int nbi = 0;
  const int ntrial = out.cell_ntrial[c.cell];
  extern __shared__ __align__(16) unsigned char dsm[];
  PairSmem &sm = reinterpret_cast<PairSmem *>(dsm)[threadIdx.x >> 5];
  Stage &stg = sm.st;
  for (int base = 0; base < ntrial; base += STAGE) {
    const int cnt = stage_window(p, pool, c.off, c.nleaf, ntrial, base, txf, stg);
    auto test = [&](int k) -> bool {
      const int j = stg.jidx[k];
      if (j == i) return false;
      const float4 xj = stg.pos[k];  // x, y, z (+ offset), 1/h
      float dxf = I.s.h.x - xj.x, dyf = I.s.h.y - xj.y, dzf = I.s.h.z - xj.z;
      if (p.periodic) {
        if (fabsf(dxf) > hLx) dxf -= copysignf(p.dxboundf, dxf);
        if (fabsf(dyf) > hLy) dyf -= copysignf(p.dyboundf, dyf);
        if (fabsf(dzf) > hLz) dzf -= copysignf(p.dzboundf, dzf);
      }
      const float r2f = dxf * dxf + dyf * dyf + dzf * dzf;
      if (r2f * fminf(hi21f, xj.w * xj.w) < q2lim) return true;
      const int code = stg.code[k];
      float dx, dy, dz, r2;
      separation_2f(p, I.s, j, code, code == 0 ? xj : txf[j], txl[j], tx, ty, tz, dx, dy, dz, r2);
      far_pair_mixed(dx, dy, dz, r2, f);
      return false;
    };
    queue_window(cnt, S, act, il, stripe, sm.q, test, [&](int k) {
      const int j = stg.jidx[k];
      MixRec jr;
      if (MHD) jr.load(jrecf, j);
      float dx, dy, dz, r2;
      separation_2f(p, I.s, j, stg.code[k], txf[j], txl[j], tx, ty, tz, dx, dy, dz, r2);
      if (!MHD) jr.load(jrecf, j);
      force_pair_mixed<MHD, true, IND>(p, I, j, dx, dy, dz, r2, jr, jmhdf, ibin_old_t, wakemark, f, vsigmax, nbi);
    });
  }
  store_pair_sums<IND>(sm, lane, np, S, c.s0, c.am, psum, ps, p.massoftype, [&](int q) -> double {
    return q < NF ? f[q].value() : (q == NF ? (double)vsigmax : (double)nbi);
  });
}

// whether force evaluations of this context can be recorded and replayed
bool pairs_recordable(const ph_ctx *c) {
  const Params &p = c->dp;
  return p.precision == PH_PREC_MIXED && !p.gravity && !p.ind && !c->keep_order;
}

static inline int nblk(int64_t n, int b) { return (int)((n + b - 1) / b); }

// whether this context's force evaluation takes the symmetric FP64 pair loop
static bool use_sym(const ph_ctx *c) {
  const Params &p = c->dp;
  return c->force_sym && p.precision != PH_PREC_MIXED && !p.gravity && !(p.ind && c->ibin);
}

// The flattened trial offsets of the owned entries of the force lists and the
// j-side buffer of the symmetric pair loop (after every list build).
static int prepare_sym(ph_ctx *c) {
  cudaStream_t st = c->stream;
  const int ncell = c->nleaves;
  const int nj = c->dp.mhd ? NJS<true>::n : NJS<false>::n;
  if (alloc_sym(c, 0, nj) != 0) return PH_ERR_CUDA;
  k_cell_at<<<nblk(ncell, 256), 256, 0, st>>>(c->nodes, c->leaves, ncell, c->cell_at);
  k_owned_trials<<<nblk(ncell, 4), 128, 0, st>>>(c->nodes, c->leaves, ncell, c->pool, c->cell_off, c->cell_nleaf,
                                                  c->cell_tbase);
  scan_int(c, c->cell_tbase, c->cell_tbase, ncell, c->cell_tbase + ncell);
  k_entry_offsets<<<nblk(ncell, 4), 128, 0, st>>>(ncell, c->cell_off, c->cell_nleaf, c->cell_tbase, c->pool,
                                                   c->toff);
  count_launch(c, 3);
  int total = 0;
  cudaMemcpyAsync(&total, c->cell_tbase + ncell, sizeof(int), cudaMemcpyDeviceToHost, st);
  if (cudaStreamSynchronize(st) != cudaSuccess) return PH_ERR_CUDA;
  if (total < 0) return PH_ERR_LIST;
  c->sym_total = total;
  return alloc_sym(c, (int64_t)total, nj) != 0 ? PH_ERR_CUDA : 0;
}

// Force trial lists (getneigh with the j-side hmax, or getneigh_dual with
// self-gravity, whose far-field coefficients are computed with them). They
// depend only on the tree and the node hmax values, so a force-only
// re-evaluation (velocity iterations, derivs icall=2) reuses the lists of the
// previous walk: the reference re-walks and gets the same lists.
int force_lists(ph_ctx *c) {
  cudaStream_t st = c->stream;
  const int ncell = c->nleaves;
  const Params p = c->dp;
  if (p.gravity && alloc_gravity(c) != 0) return PH_ERR_CUDA;
  bool levels_ok = false;
  for (int attempt = 0; !c->have_force_lists; ++attempt) {
    cudaMemsetAsync(c->pool_top, 0, sizeof(unsigned long long), st);
    cudaEventRecord(c->evk[4], st);
    if (p.gravity) {
      // getneigh_dual: the far field and the trial lists level by level, or
      // by the walks from the root when a level buffer overflowed
      const int fr = far_levels(c);
      if (fr > 0) return fr;
      levels_ok = fr == 0;
      if (!levels_ok) {
        cudaMemsetAsync(c->pool_top, 0, sizeof(unsigned long long), st);
        dual_walk(c);
      }
    } else {
      // individual timesteps: the cells holding active particles
      const bool ind = p.ind && c->ibin;
      const int nw = ind ? c->ncell_act : ncell;
      if (nw > 0) {
        launch_walk<true>(c->walk_warps, nw, st,
            p, c->nodes, c->nodesf, c->top_nodes, c->leaves, ind ? c->cell_act : nullptr, nw, nullptr, nullptr, c->pool,
            c->pool_cap, c->pool_top, c->cell_off, c->cell_nleaf, c->cell_ntrial, c->d_err);
        count_launch(c, 1);
      }
    }
    cudaEventRecord(c->evk[5], st);
    int herr = 0;
    cudaMemcpyAsync(&herr, c->d_err, sizeof(int), cudaMemcpyDeviceToHost, st);
    cudaStreamSynchronize(st);
    add_elapsed(c, 6, c->evk[4], c->evk[5]);
    if (herr == PH_ERR_LIST && attempt < 4) {
      cudaMemsetAsync(c->d_err, 0, sizeof(int), st);
      if (grow_pool(c) != 0) return PH_ERR_LIST;
      continue;
    }
    if (herr) return herr;
    if (use_sym(c)) {
      const int r = prepare_sym(c);
      if (r) return r;
    }
    c->have_force_lists = true;
    // the far field depends on the same tree, positions and node hmax
    if (p.gravity) {
      if (levels_ok) gravity_down(c);
      else gravity_far(c);
    }
  }
  return 0;
}

// cons2prim + force driver on the device-resident state; vel/Bv are the
// velocity and magnetic arrays the forces are evaluated with (vxyzu/Bevol or
// the step's predicted vpred/Bpred).
int force_dev(ph_ctx *c, const double *vel, const double *Bv) {
  if (!c->have_density) return PH_ERR_STATE;
  cudaStream_t st = c->stream;
  const int nt = (int)c->ntree, ncell = c->nleaves;
  const Params p = c->dp;
  double *eos_t = c->eos;  // tree order
  double *jmhd = c->jrec + JREC * (size_t)c->cap;
  const bool mixed = p.precision == PH_PREC_MIXED;
  float *jmhdf = c->jrecf + JRECF * (size_t)c->cap;
  if (mixed) low_words(c);
  if (c->keep_order)
    ro_force_prologue(c, vel);
  else if (mixed)
    k_force_prologue_mixed<<<nblk(nt, 256), 256, 0, st>>>(p, nt, c->perm, c->th, vel, Bv,
                                                          p.ind ? c->gradh : c->gradh_t, eos_t, c->jrec, jmhd,
                                                          c->jrecf, jmhdf, c->txf, c->alpha1, c->ddivvdt_c,
                                                          c->dvdx_c, c->alphaloc_t, c->d_err);
  else
    k_force_prologue<<<nblk(nt, 256), 256, 0, st>>>(p, nt, c->perm, c->th, vel, Bv,
                                                    p.ind ? c->gradh : c->gradh_t, eos_t, c->jrec, jmhd, c->txf,
                                                    c->alpha1, c->ddivvdt_c, c->dvdx_c,
                                                    c->alphaloc_t, c->d_err);
  count_launch(c, 1);
  const int lr = force_lists(c);
  if (lr) return lr;
  const double init[2] = {BIGNUMBER, BIGNUMBER};
  cudaMemcpyAsync(c->red, init, 2 * sizeof(double), cudaMemcpyHostToDevice, st);
  ForceOut out{c->fxyzu, c->dBevol, c->divcurlv, c->divBsymm, c->poten, c->red, c->stats, c->cell_ntrial};
  if (!(c->attr_done & 2u)) {
    const int lb = MAX_WARPS * (int)sizeof(ListSmem), pb = MAX_WARPS * (int)sizeof(PairSmem);
#define PH_FORCE_ATTR(M, I)                                                                                  \
  cudaFuncSetAttribute(k_force_mixed<M, I, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, lb);         \
  cudaFuncSetAttribute(k_force<M, I>, cudaFuncAttributeMaxDynamicSharedMemorySize, lb);                      \
  cudaFuncSetAttribute(k_force_mixed_grav<M, I>, cudaFuncAttributeMaxDynamicSharedMemorySize, pb);           \
  cudaFuncSetAttribute(k_force_grav<M, I>, cudaFuncAttributeMaxDynamicSharedMemorySize, pb)
    PH_FORCE_ATTR(false, false); PH_FORCE_ATTR(true, false); PH_FORCE_ATTR(false, true); PH_FORCE_ATTR(true, true);
#undef PH_FORCE_ATTR
    cudaFuncSetAttribute(k_force_mixed<false, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, lb);
    cudaFuncSetAttribute(k_force_mixed<true, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, lb);
    cudaFuncSetAttribute(k_force_sym<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         sym_smem_bytes<NJS<false>::n>(MAXCELL));
    cudaFuncSetAttribute(k_force_sym<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         sym_smem_bytes<NJS<true>::n>(MAXCELL));
    c->attr_done |= 2u;
  }
  const int fw = c->force_warps;
  // individual timesteps: only the cells holding active particles
  const bool ind = p.ind && c->ibin;
  const int *cells = ind ? c->cell_act : nullptr;
  const int nfc = ind ? c->ncell_act : ncell;
  const unsigned char *actf = ind ? c->actf_t : nullptr;
  const int8_t *ibo = ind ? c->ibin_old_t : nullptr;
  unsigned char *wake = ind ? c->wakemark : nullptr;
  IndFin indf{nullptr, nullptr, nullptr, 0, 0, 0};
  if (ind) {
    indf = IndFin{c->actf_t, c->ibin, c->d_ind, c->nbinmax, c->istepfrac, c->ind_icall < 2 ? 1 : 0};
    cudaMemsetAsync(c->d_ind, 0, 3 * sizeof(int), st);
  }
  if (nfc == 0) {
    cudaEventRecord(c->evk[0], st);
  } else if (c->keep_order) {
    cudaEventRecord(c->evk[0], st);
    ro_force(c);
  } else if (mixed) {
    cudaEventRecord(c->evk[0], st);
    const int mode = pairs_recordable(c) ? c->rec_mode : PAIRS_SWEEP;
    const PairRec rec{c->rec_rows, c->rec_cell, (int)c->rec_cap, c->counters + REC_ROWS};
    if (mode == PAIRS_RECORD) cudaMemsetAsync(c->counters + REC_ROWS, 0, sizeof(int), st);
#define PH_FORCE_ARGS                                                                                          \
  p, c->nodes, c->leaves, nfc, c->pool, c->cell_off, c->cell_nleaf, c->tx, c->ty, c->tz, c->txf, c->txl,       \
      c->jrecf, jmhdf, out, c->psum, c->cap, cells, actf, ibo, wake
#define PH_FORCE_MIXED(M, I, R)                                                                                \
  k_force_mixed<M, I, R><<<nblk(nfc, fw), 32 * fw, fw * sizeof(ListSmem), st>>>(PH_FORCE_ARGS, rec, c->d_err)
#define PH_FORCE_GRAV(M, I)                                                                                    \
  k_force_mixed_grav<M, I><<<nblk(nfc, fw), 32 * fw, fw * sizeof(PairSmem), st>>>(PH_FORCE_ARGS, c->d_err)
#define PH_FORCE_REPLAY(M)                                                                                     \
  k_force_replay<M><<<nblk(nfc, fw), 32 * fw, 0, st>>>(p, c->nodes, c->leaves, nfc, c->cell_off, c->cell_nleaf, \
                                                       c->txf, c->txl, c->jrecf, jmhdf,                        \
                                                       out, c->psum, c->cap, rec, c->d_err)
    if (p.gravity) {
      if (p.mhd) { if (ind) PH_FORCE_GRAV(true, true); else PH_FORCE_GRAV(true, false); }
      else { if (ind) PH_FORCE_GRAV(false, true); else PH_FORCE_GRAV(false, false); }
    } else if (mode == PAIRS_REPLAY) {
      if (p.mhd) PH_FORCE_REPLAY(true); else PH_FORCE_REPLAY(false);
    } else if (mode == PAIRS_RECORD) {
      if (p.mhd) PH_FORCE_MIXED(true, false, true); else PH_FORCE_MIXED(false, false, true);
    } else {
      if (p.mhd) { if (ind) PH_FORCE_MIXED(true, true, false); else PH_FORCE_MIXED(true, false, false); }
      else { if (ind) PH_FORCE_MIXED(false, true, false); else PH_FORCE_MIXED(false, false, false); }
    }
#undef PH_FORCE_ARGS
#undef PH_FORCE_GRAV
#undef PH_FORCE_REPLAY
#undef PH_FORCE_MIXED
  } else if (use_sym(c)) {
    cudaEventRecord(c->evk[0], st);
    if (p.mhd) {
      k_force_sym<true><<<nfc, 32, sym_smem_bytes<NJS<true>::n>(p.minpart), st>>>(
          p, c->nodes, c->leaves, nfc, c->pool, c->cell_off, c->cell_nleaf, c->tx, c->ty, c->tz, c->th, c->txf,
          c->jrec, jmhd, out, c->psum, c->cap, c->pf_hmin, c->toff, c->jbuf, c->jbuf_stride, c->d_err);
      k_force_gather<true><<<nblk(nfc, 4), 128, 0, st>>>(c->nodes, c->leaves, nfc, c->pool, c->cell_off,
                                                         c->cell_nleaf, c->cell_at, c->toff, c->jbuf,
                                                         c->jbuf_stride, p.massoftype, c->psum, c->cap, c->d_err);
    } else {
      k_force_sym<false><<<nfc, 32, sym_smem_bytes<NJS<false>::n>(p.minpart), st>>>(
          p, c->nodes, c->leaves, nfc, c->pool, c->cell_off, c->cell_nleaf, c->tx, c->ty, c->tz, c->th, c->txf,
          c->jrec, jmhd, out, c->psum, c->cap, c->pf_hmin, c->toff, c->jbuf, c->jbuf_stride, c->d_err);
      k_force_gather<false><<<nblk(nfc, 4), 128, 0, st>>>(c->nodes, c->leaves, nfc, c->pool, c->cell_off,
                                                          c->cell_nleaf, c->cell_at, c->toff, c->jbuf,
                                                          c->jbuf_stride, p.massoftype, c->psum, c->cap, c->d_err);
    }
    count_launch(c, 1);
  } else {
    cudaEventRecord(c->evk[0], st);
#define PH_FORCE_FP64_I(K, M, I, SM)                                                                           \
  K<M, I><<<nblk(nfc, fw), 32 * fw, fw * sizeof(SM), st>>>(                                                    \
      p, c->nodes, c->leaves, nfc, c->pool, c->cell_off, c->cell_nleaf, c->tx, c->ty, c->tz, c->th, c->txf,    \
      c->jrec, jmhd, out, c->psum, c->cap, c->pf_hmin, cells, actf, ibo, wake, c->d_err)
#define PH_FORCE_FP64(K, M, SM) do { if (ind) PH_FORCE_FP64_I(K, M, true, SM); else PH_FORCE_FP64_I(K, M, false, SM); } while (0)
    if (p.gravity) {
      if (p.mhd) PH_FORCE_FP64(k_force_grav, true, PairSmem);
      else PH_FORCE_FP64(k_force_grav, false, PairSmem);
    } else {
      if (p.mhd) PH_FORCE_FP64(k_force, true, ListSmem);
      else PH_FORCE_FP64(k_force, false, ListSmem);
    }
#undef PH_FORCE_FP64
#undef PH_FORCE_FP64_I
  }
  const FarField ff{c->gleaf, c->leaf_of, c->leaves, c->nodes, c->tx, c->ty, c->tz};
  if (mixed)
    k_force_finish<true><<<nblk(nt, 256), 256, 0, st>>>(p, nt, c->psum, c->cap, c->perm, c->th, c->jrec, jmhd,
                                                        eos_t, ff, out, indf, c->d_err);
  else
    k_force_finish<false><<<nblk(nt, 256), 256, 0, st>>>(p, nt, c->psum, c->cap, c->perm, c->th, c->jrec, jmhd,
                                                         eos_t, ff, out, indf, c->d_err);
  if (ind) {
    k_wake_apply<<<nblk(nt, 256), 256, 0, st>>>(nt, c->perm, c->wakemark, c->ibin_wake, c->ibinnow - 1);
    count_launch(c, 1);
  }
  cudaEventRecord(c->evk[1], st);
  count_launch(c, 2);
  c->have_force = true;
  return 0;
}

}  // namespace ph
