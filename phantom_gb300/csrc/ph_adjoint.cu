// Adjoint of density + force (differentiation form): gradients of
//   L = sum_i sum_k w(k,i) fxyzu(k,i)
// (accelerations and du/dt of one derivs evaluation, force.F90:914-3330 on
// the density solve of dens.F90:117-1681) with respect to the positions,
// velocities and thermal energies, for hydrodynamics (adiabatic or
// isothermal equation of state, artificial viscosity and conductivity, the
// viscosity parameter constant or per particle (Cullen & Dehnen switch:
// alphaind(1) is an input of one derivs, held fixed) and, for the
// accelerations, ideal MHD (magnetic pressure and
// anisotropic stress, the signal speed sqrt(c_s^2 + v_A^2) in the viscosity,
// the div B subtraction force.F90:2873-2890), also with respect to B/rho,
// and self-gravity: the softened near field of the trial pairs with its
// gradsoft term (force.F90:1303-1340) and the plain 1/r^2 pairs outside both
// kernels (force.F90:1991-2053), gradsoft = dh/drho h^-2 sum_j m dphi/dh
// (dens.F90, get_kernel_grav1) differentiated through the h-rho solve like
// 1/Omega, and the far field (kdtree.F90:1702-1840; its reverse is in the
// gravity source).
//
// Model differentiated: the converged h-rho solve, i.e. h_i the root of
// rho(h_i) = sum_j m W(r_ij, h_i), with Omega_i = 1 - (dh/drho)_i dRho_i/dh
// (gradh = 1/Omega) kept in FP64 (the reference stores it in float32; its
// rounding has no derivative). Implicit differentiation gives
//   dh_i/dx = (dh/drho)_i / Omega_i * d rho_i/dx  at fixed h_i.
//
// Work decomposition (nothing is stored between the forward and the adjoint
// beyond per-particle values; pair terms are recomputed):
//  1. k_adj_pairs: one warp per leaf cell over the force trial lists. Every
//     unordered pair {i,j} contributes c_ij + c_ji to L (c_ab: what a receives
//     from b, weighted by a's cotangents). Particle i evaluates the reverse
//     of both terms and keeps the derivatives with respect to its own
//     variables (explicit x_i, v_i and the per-particle primitives h, 1/Omega,
//     1/rho, P/rho^2, c_s, P, rho, u), so every pair is gathered on both sides
//     without atomics. It also sums d^2 rho_i/dh^2.
//  2. k_adj_coef: per particle, the chain rule to h and u and the coefficients
//     A_i (on d rho_i/dx) and B_i (on d(d rho_i/dh)/dx) of the implicit solve.
//  3. k_adj_dens: one warp per leaf cell, the gather of
//     m [A_k dW(r,h_k)/dr + B_k d2W(r,h_k)/dhdr + A_j dW(r,h_j)/dr + B_j d2W(r,h_j)/dhdr] r_kj/r
//     (with self-gravity also C_k dphi_h(r,h_k)/dr + C_j dphi_h(r,h_j)/dr,
//     C the coefficient on the gradsoft sum).
//  4. With self-gravity, the far field's reverse (gravity_adjoint_far).
#include <type_traits>

#include "ph_internal.h"
#include "ph_walk.cuh"

namespace ph {

constexpr int ADJ_WARPS = 4;
constexpr int NADJ = 24;  // pass-1 accumulators per particle

// adjoint record slots (tree order, ADJREC doubles per particle)
// (AR_CS holds the signal speed v_wave the viscosity uses: c_s, or
// sqrt(c_s^2 + v_A^2) with MHD; AR_CS0 the sound speed)
enum {
  AR_H = 0, AR_H1, AR_G, AR_RHO, AR_RHO1, AR_PRO2, AR_CS, AR_P, AR_U, AR_VX, AR_VY, AR_VZ,
  AR_WX, AR_WY, AR_WZ, AR_S, AR_A, AR_B, AR_GX, AR_GY, AR_GZ, AR_GVX, AR_GVY, AR_GVZ, AR_GU,
  AR_BX, AR_BY, AR_BZ, AR_KAP, AR_CS0, AR_GBX, AR_GBY, AR_GBZ, AR_ALPHA, AR_GS, AR_C,
  // MHD: psi, the cotangents of d(B/rho)/dt (OX..OZ) and dpsi/dt (ZETA), the
  // weights of the div B diffusion and drho/dt sums in dpsi/dt, and psi's
  // gradient
  AR_PSI, AR_OX, AR_OY, AR_OZ, AR_ZETA, AR_K11, AR_K4, AR_GPSI, AR_NSLOTS
};
static_assert(AR_NSLOTS <= ADJREC, "adjoint record slots");
// pass-1 accumulator slots (psum)
// (PA_GS: cotangent of gradsoft; PA_SG: sum m q dphi_h/dq over the kernel;
// PA_PSI: cotangent of psi; PA_FS4, PA_FS11: the forward drho/dt and div B
// diffusion sums of the receiver)
enum { PA_X = 0, PA_Y, PA_Z, PA_VX, PA_VY, PA_VZ, PA_H, PA_G, PA_RHO1, PA_PRO2, PA_CS, PA_P, PA_RHO, PA_U, PA_D2,
       PA_BX, PA_BY, PA_BZ, PA_DIVB, PA_GS, PA_SG, PA_PSI, PA_FS4, PA_FS11, PA_NSLOTS };
static_assert(PA_NSLOTS == NADJ && NADJ <= PSUM, "pass-1 slots");
static_assert(32 * NADJ * sizeof(double) <= sizeof(PairSmem), "pass-1 lane sums staged in the pair smem");

// per-lane accumulator of the adjoint pair sums: FP64 sums for the plain
// form, FP32 compensated (Kahan) sums for the precision form
template <typename T>
struct Acc;
template <>
struct Acc<double> {
  double s = 0.0;
  __device__ __forceinline__ void operator+=(double x) { s += x; }
  __device__ __forceinline__ void operator-=(double x) { s -= x; }
  __device__ __forceinline__ double value() const { return s; }
};
template <>
struct Acc<float> {
  Kahan k;
  __device__ __forceinline__ void operator+=(float x) { k.add(x); }
  __device__ __forceinline__ void operator-=(float x) { k.add(-x); }
  __device__ __forceinline__ double value() const { return k.value(); }
};

// M4 kernel shape w(q) (cnormk h^-3 separate) and its first two derivatives
template <typename T>
__device__ __forceinline__ void wshape(T q, T &w, T &w1, T &w2) {
  if (q < T(1.0)) {
    w = T(1.0) - T(1.5) * q * q + T(0.75) * q * q * q;
    w1 = q * (T(2.25) * q - T(3.0));
    w2 = T(4.5) * q - T(3.0);
  } else if (q < T(2.0)) {
    const T t = T(2.0) - q;
    w = T(0.25) * t * t * t;
    w1 = -T(0.75) * t * t;
    w2 = T(1.5) * t;
  } else {
    w = w1 = w2 = T(0.0);
  }
}

// kernel_softening's force term fsoft(q) (kernel_cubic.f90:101-120) and
// its derivative: q (15 q^3 - 36 q^2 + 40) / 30 inside q < 1,
// (-5 q^6 + 36 q^5 - 90 q^4 + 80 q^3 - 2) / (30 q^2) for 1 <= q < 2, 1/q^2
// outside
template <typename T>
__device__ __forceinline__ void softening(T q, T &fs, T &dfs) {
  if (q < T(1.0)) {
    const T q2 = q * q;
    fs = q * (T(0.5) * q2 * q - T(1.2) * q2 + T(4.0 / 3.0));
    dfs = T(2.0) * q2 * q - T(3.6) * q2 + T(4.0 / 3.0);
  } else if (q < T(2.0)) {
    const T q2 = q * q, q1 = T(1.0) / q;
    fs = q * (-T(1.0 / 6.0) * q2 * q + T(1.2) * q2 - T(3.0) * q + T(8.0 / 3.0)) - T(1.0 / 15.0) * q1 * q1;
    dfs = -T(2.0 / 3.0) * q2 * q + T(3.6) * q2 - T(6.0) * q + T(8.0 / 3.0) + T(2.0 / 15.0) * q1 * q1 * q1;
  } else {
    const T q1 = T(1.0) / q;
    fs = q1 * q1;
    dfs = -T(2.0) * q1 * q1 * q1;
  }
}

// d/dq of get_kernel_grav1's dphidh (kernel_cubic.f90:78-99):
// -3 q^4 + 6 q^3 - 4 q inside q < 1, q (q - 2)^3 for 1 <= q < 2
template <typename T>
__device__ __forceinline__ T dphidh_dq(T q) {
  if (q < T(1.0)) return q * (q * q * (T(6.0) - T(3.0) * q) - T(4.0));
  if (q < T(2.0)) { const T t = q - T(2.0); return q * t * t * t; }
  return T(0.0);
}

template <typename T>
struct AdjConst {
  T m, alpha, beta, alphau, cn;
  T alphaB, oc;  // artificial resistivity, overcleaning factor (MHD)
  bool adiab, pdv, shock, mhd, grav;
  bool induct;   // MHD: the dB/dt and dpsi/dt terms carry cotangents (or resistive heating is on)
  bool resist;   // resistive heating in du/dt (eos.f90:1898, adiabatic)
};

template <typename T>
struct Side {
  T h1, G, rho1, pro2, cs, P, rho, u, alpha;  // alpha: alphaind(1) (force.F90:1478, 2430-2433)
  T bx, by, bz;  // B/rho (MHD)
  T psi;         // Bevol(4) (MHD)
  T gs;          // gradsoft (self-gravity)
};

// 1/r of a pair, 0 for coincident particles as the forward (force.F90:1293-
// 1298): their terms have no direction and contribute no cotangents
template <typename T>
__device__ __forceinline__ T inv_sep(T r2, T r) {
  return r2 > (sizeof(T) == 8 ? T(TINY_D) : T(TINY_F)) ? T(1.0) / r : T(0.0);
}

// a receiver's cotangents: w of its acceleration, s of du/dt, kap of its div
// B sum (the div B subtraction), o of d(B/rho)/dt, k11 and k4 of its div B
// diffusion and drho/dt sums (through dpsi/dt)
template <typename T>
struct Wt {
  T wx, wy, wz, s, kap, ox, oy, oz, k11, k4;
};

// cotangents of one side's variables (divB, fs4, fs11: the forward div B,
// drho/dt and div B diffusion sums of a receiver, accumulated alongside)
template <typename T>
struct Bar {
  Acc<T> h, G, rho1, pro2, cs, P, rho, u, vx, vy, vz, bx, by, bz, divB, gs, psi, fs4, fs11;
};

// Reverse of the ordered pair term c = w . da_a + s . du_a + kap . divB_a
// (what receiver a gets from sender b, force.F90:1428-1990), d = x_a - x_b,
// dv = v_a - v_b. With MHD, da_a also holds the anisotropic stress
// -(S_a n gk_a + S_b n gk_b), S = -m (B/rho)(B/rho)^T, and divB_a gets
// m (gk_a (B_a/rho_a).n / rho_a ... ) as divBsymm (force.F90:1800-1830);
// kap is the receiver's cotangent of its divB sum (from the div B
// subtraction in the finish); c also holds o . d(B_a/rho_a)/dt, the div B
// diffusion and drho/dt sums weighted by k11 and k4, and the resistive
// heating. Accumulates the cotangents of side a (KEEP_A) or side b into g and
// returns dc/dd in (gdx, gdy, gdz).
template <typename T, bool KEEP_A, bool IND>
__device__ __forceinline__ void pair_rev(const AdjConst<T> &k, T dx, T dy, T dz, T dvx, T dvy,
                                         T dvz, const Side<T> &a, const Side<T> &b, const Wt<T> &wt,
                                         Bar<T> &g, T &gdx, T &gdy, T &gdz) {
  const T wx = wt.wx, wy = wt.wy, wz = wt.wz, s = wt.s, kap = wt.kap;
  const T r2 = dx * dx + dy * dy + dz * dz;
  const T r = sqrt(r2), rinv = inv_sep(r2, r);
  const T nx = dx * rinv, ny = dy * rinv, nz = dz * rinv;
  const T qa = r * a.h1, qb = r * b.h1;
  T wa, wpa, wppa, wb, wpb, wppb;
  wshape(qa, wa, wpa, wppa);
  wshape(qb, wb, wpb, wppb);
  const T hfa = k.cn * (a.h1 * a.h1) * (a.h1 * a.h1), hfb = k.cn * (b.h1 * b.h1) * (b.h1 * b.h1);
  const T gka = wpa * hfa * a.G, gkb = wpb * hfb * b.G;
  const T pv = dvx * nx + dvy * ny + dvz * nz;
  const T vsa_raw = a.alpha * a.cs - k.beta * pv, vsb_raw = b.alpha * b.cs - k.beta * pv;
  const T vsa = fmax(vsa_raw, T(0.0)), vsb = fmax(vsb_raw, T(0.0));
  const bool neg = pv < T(0.0);
  const T q2a = neg ? -T(0.5) * a.rho1 * vsa * pv : T(0.0), q2b = neg ? -T(0.5) * b.rho1 * vsb * pv : T(0.0);
  const T gpa = k.m * (a.pro2 + q2a) * gka, gpb = k.m * (b.pro2 + q2b) * gkb;
  // self-gravity: fg = m/2 (fg_a + fg_b), fg_a = fsoft(q_a)/h_a^2 + gradsoft_a gk_a
  // inside a's kernel, 1/r^2 outside (force.F90:1303-1340, 1991-2053)
  T fsa = T(0.0), dfsa = T(0.0), fsb = T(0.0), dfsb = T(0.0), fg = T(0.0);
  if (k.grav) {
    softening(qa, fsa, dfsa);
    softening(qb, fsb, dfsb);
    const T fga = qa < T(2.0) ? fsa * a.h1 * a.h1 + a.gs * gka : rinv * rinv;
    const T fgb = qb < T(2.0) ? fsb * b.h1 * b.h1 + b.gs * gkb : rinv * rinv;
    fg = T(0.5) * k.m * (fga + fgb);
  }
  // da_a = -n (gpa + gpb + fg)
  const T wn = wx * nx + wy * ny + wz * nz;
  const T gpt = k.grav ? (gpa + gpb) + fg : gpa + gpb;
  T nbx = -gpt * wx, nby = -gpt * wy, nbz = -gpt * wz;
  const T gp_bar = -wn;
  T gka_b = T(0.0), gkb_b = T(0.0), pv_b = T(0.0), q2a_b = T(0.0), q2b_b = T(0.0);
  T pro2a_b = T(0.0), pro2b_b = T(0.0), rho1a_b = T(0.0), rho1b_b = T(0.0), csa_b = T(0.0), csb_b = T(0.0);
  T Pa_b = T(0.0), Pb_b = T(0.0), rhoa_b = T(0.0), rhob_b = T(0.0), ua_b = T(0.0), ub_b = T(0.0);
  if (k.adiab && s != T(0.0)) {
    // du_a = [pdv] m P_a/rho_a^2 (pv gka) + [shock] m q2a pv gka + vsigu (u_a - u_b)(au_a gka + au_b gkb);
    // the pdV work uses the gas pressure (P_a rho_a^-2: without the magnetic
    // part that P/rho^2 of the stress carries with MHD)
    if (k.pdv) {
      if (k.mhd) {
        const T r2 = a.rho1 * a.rho1, c = s * k.m * pv * gka, pg = a.P * r2;
        Pa_b += c * r2;
        rho1a_b += c * T(2.0) * a.P * a.rho1;
        pv_b += s * k.m * pg * gka;
        gka_b += s * k.m * pg * pv;
      } else {  // P/rho^2 of the record is the gas value
        pro2a_b += s * k.m * pv * gka;
        const T t4b = s * k.m * a.pro2;
        pv_b += t4b * gka;
        gka_b += t4b * pv;
      }
    }
    if (k.shock) { q2a_b += s * k.m * pv * gka; pv_b += s * k.m * q2a * gka; gka_b += s * k.m * q2a * pv; }
    // conductivity signal speed: sqrt(2 |P_a - P_b| / (rho_a + rho_b)), or
    // |v_ab . n| with self-gravity (force.F90:1605-1621)
    const T dP = a.P - b.P, rs = a.rho + b.rho;
    const T X = fabs(dP) * T(2.0) / rs;
    const T vsigu = k.grav ? fabs(pv) : sqrt(X);
    const T den = a.u - b.u;
    const T aua = T(0.5) * k.m * k.alphau * a.rho1, aub = T(0.5) * k.m * k.alphau * b.rho1;
    const T E = aua * gka + aub * gkb;
    const T vsigu_b = s * den * E, den_b = s * vsigu * E;
    const T aua_b = s * vsigu * den * gka, aub_b = s * vsigu * den * gkb;
    gka_b += s * vsigu * den * aua;
    gkb_b += s * vsigu * den * aub;
    ua_b += den_b; ub_b -= den_b;
    rho1a_b += aua_b * T(0.5) * k.m * k.alphau;
    rho1b_b += aub_b * T(0.5) * k.m * k.alphau;
    if (k.grav) {
      if (pv != T(0.0)) pv_b += pv > T(0.0) ? vsigu_b : -vsigu_b;
    } else if (X > T(0.0)) {
      const T X_b = vsigu_b / (T(2.0) * vsigu);
      const T sg = dP > T(0.0) ? T(1.0) : -T(1.0);
      Pa_b += X_b * sg * T(2.0) / rs; Pb_b -= X_b * sg * T(2.0) / rs;
      rhoa_b -= X_b * X / rs; rhob_b -= X_b * X / rs;
    }
  }
  T bxa_b = T(0.0), bya_b = T(0.0), bza_b = T(0.0), bxb_b = T(0.0), byb_b = T(0.0), bzb_b = T(0.0), divb = T(0.0);
  if (k.mhd) {
    // stress: -w . (S_a n gka + S_b n gkb) = m [(w.B_a)(B_a.n) gka + (w.B_b)(B_b.n) gkb]
    const T wBa = wx * a.bx + wy * a.by + wz * a.bz, wBb = wx * b.bx + wy * b.by + wz * b.bz;
    const T Ban = a.bx * nx + a.by * ny + a.bz * nz, Bbn = b.bx * nx + b.by * ny + b.bz * nz;
    gka_b += k.m * wBa * Ban; gkb_b += k.m * wBb * Bbn;
    nbx += k.m * (wBa * gka * a.bx + wBb * gkb * b.bx);
    nby += k.m * (wBa * gka * a.by + wBb * gkb * b.by);
    nbz += k.m * (wBa * gka * a.bz + wBb * gkb * b.bz);
    bxa_b += k.m * gka * (wx * Ban + wBa * nx); bya_b += k.m * gka * (wy * Ban + wBa * ny);
    bza_b += k.m * gka * (wz * Ban + wBa * nz);
    bxb_b += k.m * gkb * (wx * Bbn + wBb * nx); byb_b += k.m * gkb * (wy * Bbn + wBb * ny);
    bzb_b += k.m * gkb * (wz * Bbn + wBb * nz);
    // divB_a += m (gka rho1a (B_a.n) + gkb rho1b (B_b.n)), weighted by kap
    divb = k.m * (gka * a.rho1 * Ban + gkb * b.rho1 * Bbn);
    if (kap != T(0.0)) {
      gka_b += kap * k.m * a.rho1 * Ban; gkb_b += kap * k.m * b.rho1 * Bbn;
      rho1a_b += kap * k.m * gka * Ban; rho1b_b += kap * k.m * gkb * Bbn;
      const T ca = kap * k.m * gka * a.rho1, cb = kap * k.m * gkb * b.rho1;
      bxa_b += ca * nx; bya_b += ca * ny; bza_b += ca * nz;
      bxb_b += cb * nx; byb_b += cb * ny; bzb_b += cb * nz;
      nbx += ca * a.bx + cb * b.bx; nby += ca * a.by + cb * b.by; nbz += ca * a.bz + cb * b.bz;
    }
  }
  T psia_b = T(0.0), psib_b = T(0.0), dvbx = T(0.0), dvby = T(0.0), dvbz = T(0.0), fs4 = T(0.0), fs11 = T(0.0);
  if (IND && k.mhd && k.induct) {
    // d(B_a/rho_a)/dt += -m rho_a^-2 gk_a (B_a.n) dv + dBdiss dB - dpsi n, with
    // dBdiss = (A_a gk_a + A_b gk_b) |dv - (dv.n) n|, A = m alphaB rho^-2 / 2,
    // dpsi = oc m (rho_a^-2 gk_a psi_a vw_a + rho_b^-2 gk_b psi_b vw_b);
    // fs11_a += -m (dB.n) gk_a; fs4_a += (dv.n) gk_a; du_a/dt += -|dB|^2 dBdiss / 2
    // (force.F90:1630-1671), B = (B/rho) rho
    const T Bax = a.bx * a.rho, Bay = a.by * a.rho, Baz = a.bz * a.rho;
    const T dBx = Bax - b.bx * b.rho, dBy = Bay - b.by * b.rho, dBz = Baz - b.bz * b.rho;
    const T r2a = a.rho1 * a.rho1, r2b = b.rho1 * b.rho1;
    const T pma = k.m * r2a * gka, pmb = k.m * r2b * gkb;
    const T projBa = Bax * nx + Bay * ny + Baz * nz;
    const T projdB = dBx * nx + dBy * ny + dBz * nz;
    const T tX = dvx - pv * nx, tY = dvy - pv * ny, tZ = dvz - pv * nz;
    const T vsigB = sqrt(tX * tX + tY * tY + tZ * tZ);
    const T hab = T(0.5) * k.m * k.alphaB;
    const T Aa = hab * r2a, Ab = hab * r2b;
    const T E = Aa * gka + Ab * gkb;
    const T dpsi = k.oc * (pma * a.psi * a.cs + pmb * b.psi * b.cs);
    fs4 = pv * gka;
    fs11 = -k.m * projdB * gka;
    const T odv = wt.ox * dvx + wt.oy * dvy + wt.oz * dvz;
    const T odB = wt.ox * dBx + wt.oy * dBy + wt.oz * dBz;
    const T on = wt.ox * nx + wt.oy * ny + wt.oz * nz;
    T Bbx = T(0.0), Bby = T(0.0), Bbz = T(0.0);  // cotangent of B_a
    T dBbx = E * vsigB * wt.ox, dBby = E * vsigB * wt.oy, dBbz = E * vsigB * wt.oz;  // of dB
    T E_b = vsigB * odB, vsB_b = E * odB;
    T pma_b = -projBa * odv, pmb_b = T(0.0);
    const T projBa_b = -pma * odv;
    Bbx += projBa_b * nx; Bby += projBa_b * ny; Bbz += projBa_b * nz;
    nbx += projBa_b * Bax - dpsi * wt.ox; nby += projBa_b * Bay - dpsi * wt.oy; nbz += projBa_b * Baz - dpsi * wt.oz;
    dvbx -= pma * projBa * wt.ox; dvby -= pma * projBa * wt.oy; dvbz -= pma * projBa * wt.oz;
    const T cl_b = -k.oc * on;
    pma_b += cl_b * a.psi * a.cs; psia_b += cl_b * pma * a.cs; csa_b += cl_b * pma * a.psi;
    pmb_b += cl_b * b.psi * b.cs; psib_b += cl_b * pmb * b.cs; csb_b += cl_b * pmb * b.psi;
    if (wt.k11 != T(0.0)) {
      const T c11 = -wt.k11 * k.m;
      dBbx += c11 * gka * nx; dBby += c11 * gka * ny; dBbz += c11 * gka * nz;
      nbx += c11 * gka * dBx; nby += c11 * gka * dBy; nbz += c11 * gka * dBz;
      gka_b += c11 * projdB;
    }
    if (wt.k4 != T(0.0)) { pv_b += wt.k4 * gka; gka_b += wt.k4 * pv; }
    if (k.resist && s != T(0.0)) {
      const T dB2 = dBx * dBx + dBy * dBy + dBz * dBz;
      dBbx -= s * E * vsigB * dBx; dBby -= s * E * vsigB * dBy; dBbz -= s * E * vsigB * dBz;
      E_b -= T(0.5) * s * dB2 * vsigB;
      vsB_b -= T(0.5) * s * dB2 * E;
    }
    gka_b += E_b * Aa + pma_b * k.m * r2a;
    gkb_b += E_b * Ab + pmb_b * k.m * r2b;
    const T r2a_b = E_b * gka * hab + pma_b * k.m * gka, r2b_b = E_b * gkb * hab + pmb_b * k.m * gkb;
    rho1a_b += T(2.0) * a.rho1 * r2a_b;
    rho1b_b += T(2.0) * b.rho1 * r2b_b;
    if (vsigB > T(0.0)) {
      const T c = vsB_b / vsigB;
      const T tbx = c * tX, tby = c * tY, tbz = c * tZ;
      const T ntb = nx * tbx + ny * tby + nz * tbz;
      dvbx += tbx - ntb * nx; dvby += tby - ntb * ny; dvbz += tbz - ntb * nz;
      nbx -= pv * tbx + ntb * dvx; nby -= pv * tby + ntb * dvy; nbz -= pv * tbz + ntb * dvz;
    }
    Bbx += dBbx; Bby += dBby; Bbz += dBbz;
    bxa_b += Bbx * a.rho; bya_b += Bby * a.rho; bza_b += Bbz * a.rho;
    rhoa_b += Bbx * a.bx + Bby * a.by + Bbz * a.bz;
    bxb_b -= dBbx * b.rho; byb_b -= dBby * b.rho; bzb_b -= dBbz * b.rho;
    rhob_b -= dBbx * b.bx + dBby * b.by + dBbz * b.bz;
  }
  pro2a_b += gp_bar * k.m * gka; q2a_b += gp_bar * k.m * gka; gka_b += gp_bar * k.m * (a.pro2 + q2a);
  pro2b_b += gp_bar * k.m * gkb; q2b_b += gp_bar * k.m * gkb; gkb_b += gp_bar * k.m * (b.pro2 + q2b);
  // self-gravity: fsoft(r/h)/h^2 has d/dr = fsoft' h^-3, d/dh = -h^-3 (q fsoft' + 2 fsoft)
  T rg_b = T(0.0), hag_b = T(0.0), hbg_b = T(0.0), gsa_b = T(0.0), gsb_b = T(0.0);
  if (k.grav) {
    const T fg_b = T(0.5) * k.m * gp_bar;
    if (qa < T(2.0)) {
      const T h3 = a.h1 * a.h1 * a.h1;
      rg_b += fg_b * dfsa * h3;
      hag_b -= fg_b * h3 * (qa * dfsa + T(2.0) * fsa);
      gsa_b += fg_b * gka;
      gka_b += fg_b * a.gs;
    } else {
      rg_b -= fg_b * T(2.0) * rinv * rinv * rinv;
    }
    if (qb < T(2.0)) {
      const T h3 = b.h1 * b.h1 * b.h1;
      rg_b += fg_b * dfsb * h3;
      hbg_b -= fg_b * h3 * (qb * dfsb + T(2.0) * fsb);
      gsb_b += fg_b * gkb;
      gkb_b += fg_b * b.gs;
    } else {
      rg_b -= fg_b * T(2.0) * rinv * rinv * rinv;
    }
  }
  T vsa_b = T(0.0), vsb_b = T(0.0);
  if (neg) {
    rho1a_b += q2a_b * (-T(0.5) * vsa * pv); vsa_b = q2a_b * (-T(0.5) * a.rho1 * pv); pv_b += q2a_b * (-T(0.5) * a.rho1 * vsa);
    rho1b_b += q2b_b * (-T(0.5) * vsb * pv); vsb_b = q2b_b * (-T(0.5) * b.rho1 * pv); pv_b += q2b_b * (-T(0.5) * b.rho1 * vsb);
  }
  if (vsa_raw > T(0.0)) { csa_b += vsa_b * a.alpha; pv_b -= vsa_b * k.beta; }
  if (vsb_raw > T(0.0)) { csb_b += vsb_b * b.alpha; pv_b -= vsb_b * k.beta; }
  // pv = dv . n
  nbx += pv_b * dvx; nby += pv_b * dvy; nbz += pv_b * dvz;
  // gk = w'(q) cn h^-4 G, q = r / h
  T r_b = rg_b, ha_b = hag_b, hb_b = hbg_b, Ga_b = T(0.0), Gb_b = T(0.0);
  if (qa < T(2.0)) {
    Ga_b = gka_b * wpa * hfa;
    const T qa_b = gka_b * wppa * hfa * a.G;
    ha_b += gka_b * (-T(4.0) * gka * a.h1) - qa_b * qa * a.h1;
    r_b += qa_b * a.h1;
  }
  if (qb < T(2.0)) {
    Gb_b = gkb_b * wpb * hfb;
    const T qb_b = gkb_b * wppb * hfb * b.G;
    hb_b += gkb_b * (-T(4.0) * gkb * b.h1) - qb_b * qb * b.h1;
    r_b += qb_b * b.h1;
  }
  // n = d / r, r = |d|
  const T nn = nbx * nx + nby * ny + nbz * nz;
  gdx = (nbx - nn * nx) * rinv + r_b * nx;
  gdy = (nby - nn * ny) * rinv + r_b * ny;
  gdz = (nbz - nn * nz) * rinv + r_b * nz;
  // (accumulators of physics that is off stay untouched: x + 0 costs an FP64
  // add, which IEEE arithmetic does not let the compiler drop)
  auto add_a = [&](Bar<T> &ga) {
    ga.h += ha_b; ga.G += Ga_b; ga.rho1 += rho1a_b; ga.pro2 += pro2a_b; ga.cs += csa_b; ga.P += Pa_b;
    ga.rho += rhoa_b; ga.u += ua_b;
    if (IND) { ga.vx += pv_b * nx + dvbx; ga.vy += pv_b * ny + dvby; ga.vz += pv_b * nz + dvbz; }
    else { ga.vx += pv_b * nx; ga.vy += pv_b * ny; ga.vz += pv_b * nz; }
    if (k.mhd) { ga.bx += bxa_b; ga.by += bya_b; ga.bz += bza_b; ga.divB += divb; }
    if (k.grav) ga.gs += gsa_b;
    if (IND) { ga.psi += psia_b; ga.fs4 += fs4; ga.fs11 += fs11; }
  };
  auto add_b = [&](Bar<T> &gbb) {
    gbb.h += hb_b; gbb.G += Gb_b; gbb.rho1 += rho1b_b; gbb.pro2 += pro2b_b; gbb.cs += csb_b; gbb.P += Pb_b;
    gbb.rho += rhob_b; gbb.u += ub_b;
    if (IND) { gbb.vx -= pv_b * nx + dvbx; gbb.vy -= pv_b * ny + dvby; gbb.vz -= pv_b * nz + dvbz; }
    else { gbb.vx -= pv_b * nx; gbb.vy -= pv_b * ny; gbb.vz -= pv_b * nz; }
    if (k.mhd) { gbb.bx += bxb_b; gbb.by += byb_b; gbb.bz += bzb_b; }
    if (k.grav) gbb.gs += gsb_b;
    if (IND) gbb.psi += psib_b;
  };
  if (KEEP_A) add_a(g);
  else add_b(g);
}

template <typename T>
__device__ __forceinline__ Side<T> load_side(const T *rec) {
  Side<T> sd;
  sd.h1 = rec[AR_H1]; sd.G = rec[AR_G]; sd.rho1 = rec[AR_RHO1]; sd.pro2 = rec[AR_PRO2]; sd.cs = rec[AR_CS];
  sd.P = rec[AR_P]; sd.rho = rec[AR_RHO]; sd.u = rec[AR_U]; sd.alpha = rec[AR_ALPHA];
  sd.bx = rec[AR_BX]; sd.by = rec[AR_BY]; sd.bz = rec[AR_BZ];
  sd.psi = rec[AR_PSI];
  sd.gs = rec[AR_GS];
  return sd;
}

template <typename T>
__device__ __forceinline__ Wt<T> load_wt(const T *rec) {
  Wt<T> w;
  w.wx = rec[AR_WX]; w.wy = rec[AR_WY]; w.wz = rec[AR_WZ]; w.s = rec[AR_S]; w.kap = rec[AR_KAP];
  w.ox = rec[AR_OX]; w.oy = rec[AR_OY]; w.oz = rec[AR_OZ]; w.k11 = rec[AR_K11]; w.k4 = rec[AR_K4];
  return w;
}

// fraction of the div B term subtracted from the force (force.F90:2873-2890)
// as a function of beta = 2 P / B^2, and its derivative
__device__ __forceinline__ void divb_frac(double beta, double &f, double &df) {
  if (beta < 2.0) { f = 1.0; df = 0.0; }
  else if (beta < 10.0) { f = (10.0 - beta) * 0.125; df = -0.125; }
  else { f = 0.0; df = 0.0; }
}

// the pair separation in the pass's arithmetic type: FP64 as formed, or
// rounded to FP32 (on the integer pipe) for the precision form
template <typename T>
__device__ __forceinline__ T sep_t(double d);
template <>
__device__ __forceinline__ double sep_t<double>(double d) { return d; }
template <>
__device__ __forceinline__ float sep_t<float>(double d) { return d2f_rn(d); }

template <typename T>
__device__ __forceinline__ void hydro_record(const Params &p, const double *r, T *o);
constexpr int HREC = 32;  // values per particle of the hydro record (hydro passes below)

// per-particle record: primitives of the force (cons2prim, eos.f90:184-237,
// rho = rhoh(h)), the velocities the force was evaluated with, and the
// cotangents w (accelerations) and s (du/dt) gathered to tree order
__global__ void k_adj_prologue(Params p, int n, const int *perm, const double *th, const double *gradh64,
                               const double *gsoft64, const double *vel, const double *Bevol, const double *w4,
                               const double *wB4, const float *alpha1, double *adj, float *adjf, double *hrec, float *hrecf,
                               float4 *txf) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int pid = perm[i];
  const double pm = p.massoftype;
  const double h = th[i];
  double *r = adj + ADJREC * (size_t)i;
  const double rho = rhoh(h, pm, p.hfact);
  const double *v = vel + 4 * (size_t)pid;
  double P, cs, u = 0.0;
  if (p.ieos == 1) { P = p.polyk * rho; cs = sqrt(p.polyk); }
  else {
    u = v[3];
    const double ponrho = (p.gamma > 1.0001) ? (p.gamma - 1.0) * u : 2.0 / 3.0 * u;
    P = ponrho * rho;
    cs = sqrt(p.gamma * ponrho);
  }
  r[AR_H] = h; r[AR_H1] = 1.0 / h; r[AR_G] = gradh64[i]; r[AR_RHO] = rho; r[AR_RHO1] = 1.0 / rho;
  r[AR_PRO2] = P / (rho * rho); r[AR_CS] = cs; r[AR_CS0] = cs; r[AR_P] = P; r[AR_U] = u;
  r[AR_VX] = v[0]; r[AR_VY] = v[1]; r[AR_VZ] = v[2];
  const double *w = w4 + 4 * (size_t)pid;
  r[AR_WX] = w[0]; r[AR_WY] = w[1]; r[AR_WZ] = w[2]; r[AR_S] = p.isothermal ? 0.0 : w[3];
  r[AR_BX] = r[AR_BY] = r[AR_BZ] = 0.0; r[AR_KAP] = 0.0;
  // the viscosity parameter of the evaluation: a fixed input of one derivs
  // (alphaind(1) evolves in the step, not in derivs)
  r[AR_ALPHA] = p.nalpha > 0 ? (double)alpha1[pid] : p.alpha;
  r[AR_GS] = p.gravity ? gsoft64[i] : 0.0;
  r[AR_C] = 0.0;
  r[AR_PSI] = r[AR_OX] = r[AR_OY] = r[AR_OZ] = r[AR_ZETA] = r[AR_K11] = r[AR_K4] = r[AR_GPSI] = 0.0;
  if (p.mhd) {
    // get_stress (force.F90:2068-2168): P/rho^2 + |B/rho|^2 / 2, v_wave^2 = c_s^2 + |B/rho|^2 rho;
    // div B subtraction weight kap = -(w . B) frac(beta), B = (B/rho) rho
    const double *b = Bevol + 4 * (size_t)pid;
    const double b2r = b[0] * b[0] + b[1] * b[1] + b[2] * b[2];
    r[AR_BX] = b[0]; r[AR_BY] = b[1]; r[AR_BZ] = b[2];
    r[AR_PRO2] += 0.5 * b2r;
    r[AR_CS] = sqrt(cs * cs + b2r * rho);
    const double B2 = b2r * rho * rho;
    double f = 0.0, df;
    if (B2 > 0.0) divb_frac(2.0 * P / B2, f, df);
    r[AR_KAP] = -(w[0] * b[0] + w[1] * b[1] + w[2] * b[2]) * rho * f;
    r[AR_PSI] = b[3];
    if (wB4) {
      // cotangents o of d(B/rho)/dt and zeta of dpsi/dt; dpsi/dt =
      // -vclean fs11 / rho - psi vclean psidecayfac / h + psi m fs4 / (2 rho)
      // (force.F90:3107-3123, vclean = overcleanfac v_wave; written only with
      // psidecayfac > 0) weights the div B diffusion sum fs11 by
      // k11 = -zeta vclean / rho and the drho/dt sum fs4 by k4 = zeta psi m / (2 rho)
      const double *wb = wB4 + 4 * (size_t)pid;
      r[AR_OX] = wb[0]; r[AR_OY] = wb[1]; r[AR_OZ] = wb[2];
      if (p.psidecayfac > 0.0) {
        const double vclean = p.overcleanfac * r[AR_CS];
        r[AR_ZETA] = wb[3];
        r[AR_K11] = -wb[3] * vclean / rho;
        r[AR_K4] = 0.5 * wb[3] * b[3] * pm / rho;
      }
    }
  }
  txf[i].w = (float)(1.0 / h);
  if (hrec) hydro_record(p, r, hrec + HREC * (size_t)i);
  if (hrecf) hydro_record(p, r, hrecf + HREC * (size_t)i);
  if (adjf) {  // FP32 copy of the record for the precision form's pair passes
    float *q = adjf + ADJREC * (size_t)i;
    for (int k = 0; k < AR_NSLOTS; ++k) q[k] = (float)r[k];
  }
}

// pass 1: pair reverse terms gathered per particle
// T = double: the plain form (FP64 pair terms); T = float: the precision
// form (pair separation formed in FP64 and rounded to FP32, pair terms in
// FP32 from the FP32 record copy, per-lane sums Kahan-compensated).
// IND: with the MHD induction, resistivity and cleaning terms (cotangents of
// dBevol, or resistive heating)
template <typename T, bool IND>
__global__ void __launch_bounds__(32 * ADJ_WARPS) k_adj_pairs(Params p, AdjConst<T> kc, const Node *nodes,
                                                              const int *leaves, int ncell, const LeafEntry *pool,
                                                              const int *cell_off, const int *cell_nleaf,
                                                              const int *cell_ntrial, const double *tx,
                                                              const double *ty, const double *tz, const float4 *txf,
                                                              const T *adj, double *psum, int64_t ps,
                                                              double pf_hmin, int *err) {
  const int w = threadIdx.x >> 5, lane = lane_id();
  const int cell = blockIdx.x * ADJ_WARPS + w;
  if (cell >= ncell) return;
  const Node nd = nodes[leaves[cell]];
  const int np = nd.count, s0 = nd.start;
  if (np < 1 || np > MAXCELL) { if (lane == 0) set_error(err, PH_ERR_TREE); return; }
  const int S = 32 / np;
  const bool act = lane < np * S;
  const int il = act ? lane / S : 0, stripe = act ? lane % S : 0;
  const int i = s0 + il;
  const T *ri = adj + ADJREC * (size_t)i;
  const Side<T> si = load_side(ri);
  const double xi = tx[i], yi = ty[i], zi = tz[i];
  const T vxi = ri[AR_VX], vyi = ri[AR_VY], vzi = ri[AR_VZ];
  const Wt<T> wti = load_wt(ri);
  const double hi = ri[AR_H];
  const float4 xif = txf[i];
  const float hi21f = xif.w * xif.w;
  // with self-gravity every trial pair has a term (no distance pre-filter)
  const bool pf_i = hi > pf_hmin && !p.gravity;
  const float pf_h1max = (float)(1.0 / pf_hmin);
  const float q2lim = 4.0f * 1.001f;
  Acc<T> gx, gy, gz, d2, sg;
  Bar<T> gi;
  const int off = cell_off[cell], nleaf = cell_nleaf[cell], ntrial = cell_ntrial[cell];
  const T h51 = si.h1 * si.h1 * si.h1 * si.h1 * si.h1;
  extern __shared__ __align__(16) unsigned char dsm[];
  PairSmem &sm = reinterpret_cast<PairSmem *>(dsm)[w];
  Stage &stg = sm.st;
  for (int base = 0; base < ntrial; base += STAGE) {
    const int cnt = stage_window(p, pool, off, nleaf, ntrial, base, txf, stg);
    auto test = [&](int k) -> bool {
      if (stg.jidx[k] == i) return false;
      if (!pf_i) return true;
      const float4 xj = stg.pos[k];
      if (xj.w >= pf_h1max) return true;
      float dxf = xif.x - xj.x, dyf = xif.y - xj.y, dzf = xif.z - xj.z;
      if (p.periodic) {
        if (fabsf(dxf) > 0.5f * p.dxboundf) dxf -= copysignf(p.dxboundf, dxf);
        if (fabsf(dyf) > 0.5f * p.dyboundf) dyf -= copysignf(p.dyboundf, dyf);
        if (fabsf(dzf) > 0.5f * p.dzboundf) dzf -= copysignf(p.dzboundf, dzf);
      }
      const float r2f = dxf * dxf + dyf * dyf + dzf * dzf;
      return r2f * fminf(hi21f, xj.w * xj.w) < q2lim;
    };
    auto body = [&](int k) {
      const int j = stg.jidx[k];
      const int code = stg.code[k];
      double dx = xi - (tx[j] + offset_of(code, 0, p.dxbound));
      double dy = yi - (ty[j] + offset_of(code, 1, p.dybound));
      double dz = zi - (tz[j] + offset_of(code, 2, p.dzbound));
      dx = wrap(dx, p.dxbound, p.hdlx, p.periodic); dy = wrap(dy, p.dybound, p.hdly, p.periodic);
      dz = wrap(dz, p.dzbound, p.hdlz, p.periodic);
      const T dxt = sep_t<T>(dx), dyt = sep_t<T>(dy), dzt = sep_t<T>(dz);
      const T *rj = adj + ADJREC * (size_t)j;
      const Side<T> sj = load_side(rj);
      const T dvx = vxi - rj[AR_VX], dvy = vyi - rj[AR_VY], dvz = vzi - rj[AR_VZ];
      T ax, ay, az;
      // i receives from j (weights of i) ...
      pair_rev<T, true, IND>(kc, dxt, dyt, dzt, dvx, dvy, dvz, si, sj, wti, gi, ax, ay, az);
      gx += ax; gy += ay; gz += az;
      // ... and j receives from i (weights of j); d -> -d
      pair_rev<T, false, IND>(kc, -dxt, -dyt, -dzt, -dvx, -dvy, -dvz, sj, si, load_wt(rj), gi, ax, ay, az);
      gx -= ax; gy -= ay; gz -= az;
      // d^2 rho_i / dh_i^2 = sum m cn h^-5 (12 w + 8 q w' + q^2 w'')
      const T q = sqrt(dxt * dxt + dyt * dyt + dzt * dzt) * si.h1;
      if (q < T(2.0)) {
        T w0, w1, w2;
        wshape(q, w0, w1, w2);
        d2 += kc.m * kc.cn * h51 * (T(12.0) * w0 + T(8.0) * q * w1 + q * q * w2);
        if (kc.grav) sg += kc.m * q * dphidh_dq(q);
      }
    };
    queue_window(cnt, S, act, il, stripe, sm.q, test, body);
  }
  // stripes of each particle summed in order through shared memory
  const double acc[NADJ] = {gx.value(),    gy.value(),   gz.value(),    gi.vx.value(),  gi.vy.value(),
                            gi.vz.value(), gi.h.value(), gi.G.value(),  gi.rho1.value(), gi.pro2.value(),
                            gi.cs.value(), gi.P.value(), gi.rho.value(), gi.u.value(),   d2.value(),
                            gi.bx.value(), gi.by.value(), gi.bz.value(), gi.divB.value(), gi.gs.value(),
                            sg.value(),    gi.psi.value(), gi.fs4.value(), gi.fs11.value()};
  double *red = reinterpret_cast<double *>(&sm.st);
  __syncwarp();
  for (int k = 0; k < NADJ; ++k) red[lane * NADJ + k] = acc[k];
  __syncwarp();
  if (lane < np) {
    double t[NADJ];
    for (int k = 0; k < NADJ; ++k) t[k] = 0.0;
    for (int q = 0; q < S; ++q)
      for (int k = 0; k < NADJ; ++k) t[k] += red[(lane * S + q) * NADJ + k];
    const size_t ip = (size_t)(s0 + lane);
    for (int k = 0; k < NADJ; ++k) psum[k * ps + ip] = t[k];
  }
}

// ------------------------------------------------------------------ hydro passes
// Hydro contexts (no MHD, no self-gravity) take a joint reverse of a pair: its
// whole contribution to L, C = c_ij + c_ji, is one scalar,
//   C / m = A G + pv (T_i g_i + T_j g_j) + (s_i - s_j) vsu (u_i - u_j) E,
//   A = -(w_i - w_j) . n,   G = X_i g_i + X_j g_j,   X = P/rho^2 + q,
//   T = s ([pdV] P/rho^2 + [shock] q),   E = au_i g_i + au_j g_j,
// (g the kernel gradient with 1/Omega, q the viscosity, pv = dv . n, vsu the
// conductivity's signal speed), so one reverse with the difference of the
// cotangents replaces the two of pair_rev, and the derivatives with respect to
// a particle's rho, P, P/rho^2 and c_s are folded into its h and u with
// factors from its record. Per unordered pair that is about 175 FP64
// instructions where the two reverses took 700 (with a dozen divisions and
// square roots); the passes are bound by the FP64 pipe.
// A particle's 10 values: position gradient (3), velocity gradient (3), h, 1/Omega
// (times 1/Omega), u, and the bracket of d^2 rho/dh^2, all without the
// particle mass; k_adj_gather or the store of the precision form scales them.
constexpr int NJA = 10;
enum {
  HR_H1 = 0, HR_KG, HR_KW, HR_RHO, HR_PRO2, HR_AVW, HR_C, HR_P, HR_U, HR_AU, HR_S, HR_WX, HR_WY, HR_WZ, HR_VX, HR_VY,
  HR_VZ, HR_KRP, HR_KUP, HR_KRPP, HR_KUPP, HR_KRC, HR_KRA, HR_KUC, HR_KH, HR_A3, HR_B1, HR_N
};
static_assert(HR_N <= HREC, "hydro record slots");

// kernel shape factors: HR_KG multiplies hs1 to g, HR_KW hs2 to dg/dr. FP64: hs1
// = s of kern_w (HR_KG with -3/4); FP32: dW/dq (s would cancel at small q)
template <typename T>
__host__ __device__ constexpr T hs1_fac() { return sizeof(T) == 8 ? T(-0.75) : T(1.0); }

struct HConst {
  double beta;
  bool cond, pdv, shock;
};

// the record of tree position i from its adjoint record. The HR_KR* are
// derivatives with respect to rho times drho/dh = -3 rho/h (HR_KH), which leaves
// no power of 1/rho above the first: u/rho^2 would leave the FP32 range with the
// pair's own factors from rho = 1e-17 down
template <typename T>
__device__ __forceinline__ void hydro_record(const Params &p, const double *r, T *o) {
  const double h1 = r[AR_H1], rho = r[AR_RHO], rho1 = r[AR_RHO1], cs = r[AR_CS0], u = r[AR_U];
  const double h4 = CNORMK * (h1 * h1) * (h1 * h1);
  const double gm1 = p.ieos == 1 ? 0.0 : ((p.gamma > 1.0001) ? p.gamma - 1.0 : 2.0 / 3.0);
  const double pon = p.ieos == 1 ? p.polyk : gm1 * u;
  const double au = 0.5 * p.alphau * rho1;
  const double v[HR_A3] = {h1, (double)hs1_fac<T>() * h4 * r[AR_G], 1.5 * h4 * h1 * r[AR_G], rho, r[AR_PRO2],
                           r[AR_ALPHA] * cs, -0.5 * rho1, r[AR_P], u, au, r[AR_S], r[AR_WX], r[AR_WY], r[AR_WZ],
                           r[AR_VX], r[AR_VY], r[AR_VZ], 3.0 * r[AR_PRO2] * h1, gm1 * rho1, -3.0 * pon * rho * h1,
                           gm1 * rho, -1.5 * rho1 * h1, 3.0 * au * h1,
                           cs > 0.0 ? r[AR_ALPHA] * p.gamma * gm1 / (2.0 * cs) : 0.0, -3.0 * rho * h1};
  for (int k = 0; k < HR_A3; ++k) o[k] = (T)v[k];
  if (p.ieos == 1) o[HR_KUC] = T(0.0);
}

__device__ __forceinline__ double inv_r(double r2) { return rsqrt_fast(r2); }
__device__ __forceinline__ float inv_r(float r2) { return r2 > TINY_F ? rsqrt_nr(r2) : 0.0f; }

// kernel shape at r h1: q, hs1, hs2 = w''/1.5 and the bracket 12 w + 8 q w' + q^2 w''
__device__ __forceinline__ void hshape(double r, double h1, double &q, double &hs1, double &hs2, double &d2) {
  double u = fma(-r, h1, 2.0);
  u = u_inside(u) ? u : 0.0;
  const double w = kern_w(u);
  q = 2.0 - u;
  hs1 = fma(-w, w, u * u);
  hs2 = fma(-2.0, w, u);
  // u (6 + u (10.5 u - 18)) - w/2 (6 + w (10.5 w - 18))
  d2 = fma(u, fma(u, fma(10.5, u, -18.0), 6.0), -0.5 * w * fma(w, fma(10.5, w, -18.0), 6.0));
}
__device__ __forceinline__ void hshape(float r, float h1, float &q, float &hs1, float &hs2, float &d2) {
  q = r * h1;
  if (q < 1.0f) {
    hs1 = q * (2.25f * q - 3.0f);
    hs2 = 3.0f * q - 2.0f;
    d2 = 12.0f + q * q * (31.5f * q - 45.0f);
  } else {
    const float t = fmaxf(2.0f - q, 0.0f);
    hs1 = -0.75f * t * t;
    hs2 = t;
    d2 = t * (6.0f + t * (10.5f * t - 18.0f));
  }
}

// The conductivity's signal speed vsu = sqrt(2 |dP| / rs), rs = rho_i + rho_j, and
// the share of its cotangent vsb in h (Ra, Rb) and u (Ua, Ub) of both sides. FP64:
// from y = (|dP| rs)^(-1/2). FP32: from the quotient, since y^2 with the pair's
// own factors leaves the range from rho = 1e-12 down (and |dP| rs itself at
// 1e-17), and each factor 1/rs meets a rho before anything else.
struct CondD { double y, t; };
struct CondF { float y, i; };
__device__ __forceinline__ double cond_speed(double dP, double rs, CondD &c) {
  const double dPa = fabs(dP);
  c.y = rsqrt_fast(dPa * rs);
  c.t = dPa * c.y;
  return 1.4142135623730951 * c.t;
}
__device__ __forceinline__ void cond_rev(const CondD &c, double dP, double vsu, double vsb, const double *a,
                                         const double *b, double &Ra, double &Rb, double &Ua, double &Ub) {
  const double w = 0.70710678118654752 * (vsb * c.y), rX = -w * (c.t * c.t);  // vsb dvsu/d|dP|, vsb dvsu/drs
  const double P = dP > 0.0 ? w : -w;
  Ra = fma(P, a[HR_KRPP], fma(rX, a[HR_KH], Ra)); Rb = fma(-P, b[HR_KRPP], fma(rX, b[HR_KH], Rb));
  Ua = fma(P, a[HR_KUPP], Ua); Ub = fma(-P, b[HR_KUPP], Ub);
}
__device__ __forceinline__ float cond_speed(float dP, float rs, CondF &c) {
  c.i = 1.0f / rs;
  const float t = 2.0f * fabsf(dP) * c.i;
  c.y = t >= TINY_F ? rsqrt_nr(t) : 0.0f;
  return t * c.y;
}
__device__ __forceinline__ void cond_rev(const CondF &c, float dP, float vsu, float vsb, const float *a, const float *b,
                                         float &Ra, float &Rb, float &Ua, float &Ub) {
  const float P = vsb * (dP > 0.0f ? c.y : -c.y), rX = -0.5f * vsb * vsu;  // each times rs
  Ra += P * (a[HR_KRPP] * c.i) + rX * (a[HR_KH] * c.i); Rb += rX * (b[HR_KH] * c.i) - P * (b[HR_KRPP] * c.i);
  Ua += P * (a[HR_KUPP] * c.i); Ub -= P * (b[HR_KUPP] * c.i);
}

// Reverse of C: the gradient gd with respect to d = x_i - x_j and gv to dv =
// v_i - v_j, and (h, 1/Omega, u, bracket) of both sides. a, b: hydro records.
template <typename T>
__device__ __forceinline__ void hydro_pair_rev(const HConst &k, T dx, T dy, T dz, T r2, const T *a, const T *b, T (&gd)[3],
                                               T (&gv)[3], T (&oa)[4], T (&ob)[4]) {
  const T beta = (T)k.beta;
  const T y = inv_r(r2), r = r2 * y;
  T qa_, s1a, s2a, d2a, qb_, s1b, s2b, d2b;
  hshape(r, a[HR_H1], qa_, s1a, s2a, d2a);
  hshape(r, b[HR_H1], qb_, s1b, s2b, d2b);
  const T ga = a[HR_KG] * s1a, gb = b[HR_KG] * s1b;
  const T dvx = a[HR_VX] - b[HR_VX], dvy = a[HR_VY] - b[HR_VY], dvz = a[HR_VZ] - b[HR_VZ];
  const T pv = y * (dvx * dx + dvy * dy + dvz * dz);
  const T wx = a[HR_WX] - b[HR_WX], wy = a[HR_WY] - b[HR_WY], wz = a[HR_WZ] - b[HR_WZ];
  const T A = -y * (wx * dx + wy * dy + wz * dz);
  const T sa = a[HR_S], sb = b[HR_S];
  const bool neg = pv < T(0.0);
  T va = T(0.0), vb = T(0.0), cpa = T(0.0), cpb = T(0.0), qa = T(0.0), qb = T(0.0);
  if (neg) {
    const T bp = beta * pv;
    va = a[HR_AVW] - bp; vb = b[HR_AVW] - bp;
    va = va > T(0.0) ? va : T(0.0); vb = vb > T(0.0) ? vb : T(0.0);
    cpa = a[HR_C] * pv; cpb = b[HR_C] * pv;
    qa = cpa * va; qb = cpb * vb;
  }
  const T Xa = a[HR_PRO2] + qa, Xb = b[HR_PRO2] + qb;
  const T Ta = sa * (k.pdv ? (k.shock ? Xa : a[HR_PRO2]) : (k.shock ? qa : T(0.0)));
  const T Tb = sb * (k.pdv ? (k.shock ? Xb : b[HR_PRO2]) : (k.shock ? qb : T(0.0)));
  T pvb = Ta * ga + Tb * gb;
  T gab = A * Xa + pv * Ta, gbb = A * Xb + pv * Tb;
  const T Asa = A + sa * pv, Asb = A + sb * pv;
  const T pa = ga * (k.pdv ? Asa : A), pb = gb * (k.pdv ? Asb : A);
  T Ra = pa * a[HR_KRP], Rb = pb * b[HR_KRP], Ua = pa * a[HR_KUP], Ub = pb * b[HR_KUP];
  if (neg) {
    const T ea = k.shock == k.pdv ? pa : ga * (k.shock ? Asa : A), eb = k.shock == k.pdv ? pb : gb * (k.shock ? Asb : A);
    const T vab = va > T(0.0) ? ea * cpa : T(0.0), vbb = vb > T(0.0) ? eb * cpb : T(0.0);
    const T fa = ea * va, fb = eb * vb;
    pvb += fa * a[HR_C] + fb * b[HR_C] - beta * (vab + vbb);
    Ra += (fa * pv) * a[HR_KRC]; Rb += (fb * pv) * b[HR_KRC];
    Ua += vab * a[HR_KUC]; Ub += vbb * b[HR_KUC];
  }
  if (k.cond) {
    const T dP = a[HR_P] - b[HR_P], rs = a[HR_RHO] + b[HR_RHO];
    typename std::conditional<sizeof(T) == 8, CondD, CondF>::type cd;
    const T vsu = cond_speed(dP, rs, cd);
    const T Sd = sa - sb, Du = a[HR_U] - b[HR_U];
    const T SD = Sd * Du, cu = SD * vsu;
    const T E = a[HR_AU] * ga + b[HR_AU] * gb;
    gab += cu * a[HR_AU]; gbb += cu * b[HR_AU];
    const T du = Sd * vsu * E;
    const T vsb = SD * E;
    Ra += (cu * ga) * a[HR_KRA];
    Rb += (cu * gb) * b[HR_KRA];
    Ua += du;
    Ub -= du;
    cond_rev(cd, dP, vsu, vsb, a, b, Ra, Rb, Ua, Ub);
  }
  const T Gs = Xa * ga + Xb * gb;
  const T nbx = pvb * dvx - Gs * wx, nby = pvb * dvy - Gs * wy, nbz = pvb * dvz - Gs * wz;
  const T nn = y * (nbx * dx + nby * dy + nbz * dz);
  const T za = gab * a[HR_KW] * s2a, zb = gbb * b[HR_KW] * s2b;
  const T c = y * ((za + zb) - nn * y);
  gd[0] = nbx * y + dx * c; gd[1] = nby * y + dy * c; gd[2] = nbz * y + dz * c;
  const T pvy = pvb * y;
  gv[0] = pvy * dx; gv[1] = pvy * dy; gv[2] = pvy * dz;
  oa[1] = gab * ga; ob[1] = gbb * gb;
  oa[0] = Ra - (za * qa_ + T(4.0) * a[HR_H1] * oa[1]);
  ob[0] = Rb - (zb * qb_ + T(4.0) * b[HR_H1] * ob[1]);
  oa[2] = Ua; ob[2] = Ub;
  oa[3] = d2a; ob[3] = d2b;
}

__host__ __device__ __forceinline__ int nja_slot(int v) {
  return v < 3 ? PA_X + v : (v < 6 ? PA_VX + (v - 3) : (v == 6 ? PA_H : (v == 7 ? PA_G : (v == 8 ? PA_U : PA_D2))));
}
// a summed value in the units of the pass-1 slots
__device__ __forceinline__ double nja_scaled(int v, double s, double m, double h1, double G) {
  if (v == 7) return m * s / G;
  if (v == 9) return m * CNORMK * (h1 * h1) * (h1 * h1) * h1 * s;
  return m * s;
}
// the pass-1 slots the hydro record has folded into h and u
__device__ __forceinline__ void nja_zero(double *psum, int64_t ps, size_t ip) {
  psum[PA_RHO1 * ps + ip] = 0.0; psum[PA_PRO2 * ps + ip] = 0.0; psum[PA_CS * ps + ip] = 0.0;
  psum[PA_P * ps + ip] = 0.0; psum[PA_RHO * ps + ip] = 0.0;
}

// acceptance and cell set-up of the hydro passes (txf.w = 1/h)
struct AdjCell { int np, s0, off, nleaf; float4 cc; };
__device__ __forceinline__ bool adj_cell(AdjCell &c, int cell, int ncell, const Node *nodes, const int *leaves,
                                         const int *cell_off, const int *cell_nleaf, const float4 *txf, float pf_hf,
                                         ListBase &sm, int *err) {
  if (cell >= ncell) return false;
  const Node nd = nodes[leaves[cell]];
  c.np = nd.count; c.s0 = nd.start;
  if (c.np < 1 || c.np > MAXCELL) { if (lane_id() == 0) set_error(err, PH_ERR_TREE); return false; }
  c.off = cell_off[cell]; c.nleaf = cell_nleaf[cell];
  c.cc = make_float4((float)nd.x, (float)nd.y, (float)nd.z, (float)nd.size);
  if (lane_id() < c.np) {
    float4 x = txf[c.s0 + lane_id()];
    const float h = __frcp_rn(x.w);
    x.w = h > pf_hf ? 4.0f * 1.001f * (h * h) : __int_as_float(0x7f800000);
    sm.xi[lane_id()] = x;
    sm.ipos[lane_id()] = c.s0 + lane_id();
  }
  return true;
}
__device__ __forceinline__ float adj_accept(float h1, float pf_hf) {
  const float h = __frcp_rn(h1);
  return h > pf_hf ? 4.0f * 1.001f * (h * h) : __int_as_float(0x7f800000);
}

// Pass 1, FP64: every unordered pair once (sym_pairs); j's values go through
// jbuf and k_adj_gather.
__global__ void __launch_bounds__(32) k_adj_pairs_sym(
    Params p, HConst kc, const Node *nodes, const int *leaves, int ncell, const LeafEntry *pool, const int *cell_off,
    const int *cell_nleaf, const double *tx, const double *ty, const double *tz, const float4 *txf, const double *hrec,
    double *psum, int64_t ps, double pf_hmin, const int *toff, double *jbuf, int64_t jstride, int *err) {
  extern __shared__ __align__(16) unsigned char dsm[];
  ListSmemK &sm = *reinterpret_cast<ListSmemK *>(dsm);
  const float pf_hf = __double2float_ru(pf_hmin);
  AdjCell c;
  if (!adj_cell(c, blockIdx.x, ncell, nodes, leaves, cell_off, cell_nleaf, txf, pf_hf, sm, err)) return;
  if (c.np > p.minpart) { if (lane_id() == 0) set_error(err, PH_ERR_TREE); return; }
  int nown, town;
  owned_prefix(pool, c.off, c.nleaf, c.s0, nown, town);
  constexpr int NR = (NJA * MAXCELL + 31) / 32;
  double tot[NR];
  for (int r = 0; r < NR; ++r) tot[r] = 0.0;
  double a[HR_A3], xi = 0.0, yi = 0.0, zi = 0.0, f[NJA];
  sym_pairs<NJA, false>(p, c.cc, c.np, pool, c.off, nown, txf, sm, (int64_t)toff[c.off], jbuf, jstride, tot,
      [&](float h1) { return adj_accept(h1, pf_hf); },
      [&](int il) {
        const int i = c.s0 + il;
        for (int k = 0; k < HR_A3; ++k) a[k] = hrec[HREC * (size_t)i + k];
        xi = tx[i]; yi = ty[i]; zi = tz[i];
        for (int k = 0; k < NJA; ++k) f[k] = 0.0;
      },
      [&](int j, int code, double (&jv)[NJA]) {
        double dx, dy, dz, gd[3], gv[3], oa[4], ob[4];
        separation_fp64(p, xi, yi, zi, j, code, tx, ty, tz, dx, dy, dz);
        hydro_pair_rev<double>(kc, dx, dy, dz, fma(dz, dz, fma(dy, dy, dx * dx)), a, hrec + HREC * (size_t)j, gd, gv, oa,
                               ob);
        for (int k = 0; k < 3; ++k) { f[k] += gd[k]; f[3 + k] += gv[k]; jv[k] = -gd[k]; jv[3 + k] = -gv[k]; }
        for (int k = 0; k < 4; ++k) { f[6 + k] += oa[k]; jv[6 + k] = ob[k]; }
      },
      [&](int k) -> double { return f[k]; });
  for (int r = 0; r < NR; ++r) {
    const int idx = lane_id() + 32 * r;
    if (idx < NJA * c.np) { const int k = idx / c.np; psum[nja_slot(k) * ps + c.s0 + (idx - k * c.np)] = tot[r]; }
  }
}

// Pass 1, precision form: each pair from both sides, i's values kept (FP32
// terms, compensated sums).
__global__ void __launch_bounds__(32 * ADJ_WARPS, 4) k_adj_pairs_hydro(
    Params p, HConst kc, const Node *nodes, const int *leaves, int ncell, const LeafEntry *pool, const int *cell_off,
    const int *cell_nleaf, const double *tx, const double *ty, const double *tz, const float4 *txf, const float4 *txl,
    const float *hrec, const double *adj, double *psum, int64_t ps, double pf_hmin, int *err) {
  extern __shared__ __align__(16) unsigned char dsm[];
  const int w = threadIdx.x >> 5;
  ListSmem &sm = reinterpret_cast<ListSmem *>(dsm)[w];
  const float pf_hf = __double2float_ru(pf_hmin);
  AdjCell c;
  if (!adj_cell(c, blockIdx.x * ADJ_WARPS + w, ncell, nodes, leaves, cell_off, cell_nleaf, txf, pf_hf, sm, err)) return;
  constexpr int NR = (NJA * MAXCELL + 31) / 32;
  double tot[NR];
  for (int r = 0; r < NR; ++r) tot[r] = 0.0;
  const int qstride = LQ / c.np;
  ListPos pos;
  __syncwarp();
  bool more = true;
  while (more) {
    int myc;
    more = SWEEP_END != sweep_list<false>(p, c.cc, c.np, pool, c.off, c.nleaf, txf, sm, qstride, pos, myc,
                                          [&](float h1) { return adj_accept(h1, pf_hf); });
    const QueueLanes ql = balance_queues(c.np, myc, sm);
    const int il = max(ql.il, 0), i = c.s0 + il;
    float a[HR_A3];
    for (int k = 0; k < HR_A3; ++k) a[k] = hrec[HREC * (size_t)i + k];
    const Sep2 I = sep2_init(txf, txl, i);
    Kahan f[NJA];
    for (int m = ql.m0; m < ql.c; m += ql.step) {
      const int j = sm.qj[il * qstride + m];
      float dx, dy, dz, r2, gd[3], gv[3], oa[4], ob[4], b[HR_A3];
      separation_2f(p, I, j, sm.qc[il * qstride + m] & 63, txf[j], txl[j], tx, ty, tz, dx, dy, dz, r2);
      const float4 *b4 = reinterpret_cast<const float4 *>(hrec + HREC * (size_t)j);
#pragma unroll
      for (int k = 0; k < (HR_A3 + 3) / 4; ++k) {
        const float4 v = b4[k];
        b[4 * k] = v.x;
        if (4 * k + 1 < HR_A3) b[4 * k + 1] = v.y;
        if (4 * k + 2 < HR_A3) b[4 * k + 2] = v.z;
        if (4 * k + 3 < HR_A3) b[4 * k + 3] = v.w;
      }
      hydro_pair_rev<float>(kc, dx, dy, dz, r2, a, b, gd, gv, oa, ob);
      for (int k = 0; k < 3; ++k) { f[k].add(gd[k]); f[3 + k].add(gv[k]); }
      for (int k = 0; k < 4; ++k) f[6 + k].add(oa[k]);
    }
    flush_lanes<NJA>(c.np, sm, sm.red, tot, [&](int k) -> double { return f[k].value(); },
                     [](int, double s, double v) -> double { return s + v; });
  }
  for (int r = 0; r < NR; ++r) {
    const int idx = lane_id() + 32 * r;
    if (idx < NJA * c.np) {
      const int k = idx / c.np;
      const size_t ip = (size_t)(c.s0 + (idx - k * c.np));
      const double *rec = adj + ADJREC * ip;
      psum[nja_slot(k) * ps + ip] = nja_scaled(k, tot[r], p.massoftype, rec[AR_H1], rec[AR_G]);
      if (k == 0) nja_zero(psum, ps, ip);
    }
  }
}

// Pass 2 of hydro contexts: the pair coefficient
//   m/r [A_i dW(r,h_i)/dr + B_i d2W(r,h_i)/dhdr + A_j dW(r,h_j)/dr + B_j d2W(r,h_j)/dhdr]
// is symmetric in i and j. With A3 and B1 of the record it is hs1 A3 + q hs2 B1
// of both sides over r.
template <typename T>
__device__ __forceinline__ T hydro_dens_coef(T r2, const T *a, const T *b) {
  const T y = inv_r(r2), r = r2 * y;
  T qa, s1a, s2a, qb, s1b, s2b, d2;
  hshape(r, a[0], qa, s1a, s2a, d2);
  hshape(r, b[0], qb, s1b, s2b, d2);
  return y * ((s1a * a[1] + (qa * s2a) * a[2]) + (s1b * b[1] + (qb * s2b) * b[2]));
}

__global__ void __launch_bounds__(32) k_adj_dens_sym(
    Params p, const Node *nodes, const int *leaves, int ncell, const LeafEntry *pool, const int *cell_off,
    const int *cell_nleaf, const double *tx, const double *ty, const double *tz, const float4 *txf, const double *hrec,
    double *psum, int64_t ps, double pf_hmin, const int *toff, double *jbuf, int64_t jstride, int *err) {
  extern __shared__ __align__(16) unsigned char dsm[];
  ListSmemK &sm = *reinterpret_cast<ListSmemK *>(dsm);
  const float pf_hf = __double2float_ru(pf_hmin);
  AdjCell c;
  if (!adj_cell(c, blockIdx.x, ncell, nodes, leaves, cell_off, cell_nleaf, txf, pf_hf, sm, err)) return;
  if (c.np > p.minpart) { if (lane_id() == 0) set_error(err, PH_ERR_TREE); return; }
  int nown, town;
  owned_prefix(pool, c.off, c.nleaf, c.s0, nown, town);
  constexpr int NR = (3 * MAXCELL + 31) / 32;
  double tot[NR];
  for (int r = 0; r < NR; ++r) tot[r] = 0.0;
  double a[3], xi = 0.0, yi = 0.0, zi = 0.0, f[3];
  auto load = [&](int i, double (&o)[3]) {
    const double *r = hrec + HREC * (size_t)i;
    o[0] = r[HR_H1]; o[1] = r[HR_A3]; o[2] = r[HR_B1];
  };
  sym_pairs<3, false>(p, c.cc, c.np, pool, c.off, nown, txf, sm, (int64_t)toff[c.off], jbuf, jstride, tot,
      [&](float h1) { return adj_accept(h1, pf_hf); },
      [&](int il) {
        const int i = c.s0 + il;
        load(i, a);
        xi = tx[i]; yi = ty[i]; zi = tz[i];
        for (int k = 0; k < 3; ++k) f[k] = 0.0;
      },
      [&](int j, int code, double (&jv)[3]) {
        double dx, dy, dz, b[3];
        load(j, b);
        separation_fp64(p, xi, yi, zi, j, code, tx, ty, tz, dx, dy, dz);
        const double co = hydro_dens_coef<double>(fma(dz, dz, fma(dy, dy, dx * dx)), a, b);
        f[0] = fma(co, dx, f[0]); f[1] = fma(co, dy, f[1]); f[2] = fma(co, dz, f[2]);
        jv[0] = -co * dx; jv[1] = -co * dy; jv[2] = -co * dz;
      },
      [&](int k) -> double { return f[k]; });
  for (int r = 0; r < NR; ++r) {
    const int idx = lane_id() + 32 * r;
    if (idx < 3 * c.np) { const int k = idx / c.np; psum[k * ps + c.s0 + (idx - k * c.np)] = tot[r]; }
  }
}

__global__ void __launch_bounds__(32 * ADJ_WARPS, 6) k_adj_dens_hydro(
    Params p, const Node *nodes, const int *leaves, int ncell, const LeafEntry *pool, const int *cell_off,
    const int *cell_nleaf, const double *tx, const double *ty, const double *tz, const float4 *txf, const float4 *txl,
    const float *hrec, double *psum, int64_t ps, double pf_hmin, int *err) {
  extern __shared__ __align__(16) unsigned char dsm[];
  const int w = threadIdx.x >> 5;
  ListSmem &sm = reinterpret_cast<ListSmem *>(dsm)[w];
  const float pf_hf = __double2float_ru(pf_hmin);
  AdjCell c;
  if (!adj_cell(c, blockIdx.x * ADJ_WARPS + w, ncell, nodes, leaves, cell_off, cell_nleaf, txf, pf_hf, sm, err)) return;
  constexpr int NR = (3 * MAXCELL + 31) / 32;
  double tot[NR];
  for (int r = 0; r < NR; ++r) tot[r] = 0.0;
  const int qstride = LQ / c.np;
  ListPos pos;
  __syncwarp();
  bool more = true;
  while (more) {
    int myc;
    more = SWEEP_END != sweep_list<false>(p, c.cc, c.np, pool, c.off, c.nleaf, txf, sm, qstride, pos, myc,
                                          [&](float h1) { return adj_accept(h1, pf_hf); });
    const QueueLanes ql = balance_queues(c.np, myc, sm);
    const int il = max(ql.il, 0), i = c.s0 + il;
    auto load = [&](int n, float (&o)[3]) {
      const float *r = hrec + HREC * (size_t)n;
      o[0] = r[HR_H1]; o[1] = r[HR_A3]; o[2] = r[HR_B1];
    };
    float a[3];
    load(i, a);
    const Sep2 I = sep2_init(txf, txl, i);
    Kahan f[3];
    for (int m = ql.m0; m < ql.c; m += ql.step) {
      const int j = sm.qj[il * qstride + m];
      float dx, dy, dz, r2, b[3];
      load(j, b);
      separation_2f(p, I, j, sm.qc[il * qstride + m] & 63, txf[j], txl[j], tx, ty, tz, dx, dy, dz, r2);
      const float co = hydro_dens_coef<float>(r2, a, b);
      f[0].add(co * dx); f[1].add(co * dy); f[2].add(co * dz);
    }
    flush_lanes<3>(c.np, sm, sm.red, tot, [&](int k) -> double { return f[k].value(); },
                   [](int, double s, double v) -> double { return s + v; });
  }
  for (int r = 0; r < NR; ++r) {
    const int idx = lane_id() + 32 * r;
    if (idx < 3 * c.np) { const int k = idx / c.np; psum[k * ps + c.s0 + (idx - k * c.np)] = tot[r]; }
  }
}

// Per leaf cell B: add to its particles' pass-1 (NJ = NJA) or pass-2 (NJ = 3)
// sums the j-side values that k_adj_pairs_sym or k_adj_dens_sym left in jbuf (its own leaf's entry and those of the cells
// before it whose lists hold B, found by a binary search), in the order of
// B's own list (as k_force_gather)
template <int NJ>
__global__ void k_adj_gather(const Node *nodes, const int *leaves, int ncell, const LeafEntry *pool,
                             const int *cell_off, const int *cell_nleaf, const int *cell_at, const int *toff,
                             const double *jbuf, int64_t jstride, const double *adj, double pm, double *psum,
                             int64_t ps) {
  const unsigned FULL = 0xffffffffu;
  const int w = threadIdx.x >> 5, lane = lane_id();
  const int cell = blockIdx.x * (blockDim.x >> 5) + w;
  if (cell >= ncell) return;
  const Node nd = nodes[leaves[cell]];
  const int np = nd.count, s0 = nd.start;
  if (np < 1 || np > MAXCELL) return;
  const int off = cell_off[cell], nleaf = cell_nleaf[cell];
  constexpr int NC = (NJ * MAXCELL + 31) / 32;
  double acc[NC];
  for (int r = 0; r < NC; ++r) acc[r] = 0.0;
  for (int e0 = nleaf - 1; e0 >= 0; e0 -= 32) {
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
    const int nin = __popc(inb);
    for (int q = nin - 1; q >= 0; --q) {
      const int sl = __shfl_sync(FULL, slot, q);
      if (sl < 0) continue;
      for (int r = 0; r < NC; ++r) {
        const int c = lane + 32 * r;
        const int v = c / MAXCELL, t = c % MAXCELL;
        if (v < NJ && t < np) acc[r] += jbuf[(int64_t)v * jstride + sl + t];
      }
    }
    if (nin < 32) break;
  }
  for (int r = 0; r < NC; ++r) {
    const int c = lane + 32 * r;
    const int v = c / MAXCELL, t = c % MAXCELL;
    if (v < NJ && t < np) {
      const size_t ip = (size_t)(s0 + t);
      double *dst = psum + (int64_t)(NJ == NJA ? nja_slot(v) : v) * ps + ip;
      if (NJ == NJA) {
        const double *rec = adj + ADJREC * ip;
        *dst = nja_scaled(v, *dst + acc[r], pm, rec[AR_H1], rec[AR_G]);
        if (v == 0) nja_zero(psum, ps, ip);
      } else {
        *dst += acc[r];
      }
    }
  }
}

// chain rule per particle and the implicit-solve coefficients
__global__ void k_adj_coef(Params p, int n, const double *psum, int64_t ps, double *adj, float *adjf, double *hrec,
                           float *hrecf) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double *r = adj + ADJREC * (size_t)i;
  const double pm = p.massoftype;
  const double h = r[AR_H], rho = r[AR_RHO], rho1 = r[AR_RHO1], G = r[AR_G], u = r[AR_U], cs = r[AR_CS0];
  auto ps_ = [&](int k) { return psum[k * ps + i]; };
  double P_b = ps_(PA_P), rho_b = ps_(PA_RHO) - ps_(PA_RHO1) * rho1 * rho1, cs_b = ps_(PA_CS);
  double bx_b = 0.0, by_b = 0.0, bz_b = 0.0, psi_b = 0.0, h_fin = 0.0;
  if (p.mhd) {
    psi_b = ps_(PA_PSI);
    const double zeta = r[AR_ZETA];
    if (zeta != 0.0) {
      // dpsi/dt = -vclean fs11 rho1 - psi dtau + psi m fs4 rho1 / 2, vclean =
      // overcleanfac v_wave, dtau = psidecayfac vclean / h (force.F90:3107-3123)
      const double psi = r[AR_PSI], fs4 = ps_(PA_FS4), fs11 = ps_(PA_FS11);
      const double vclean = p.overcleanfac * r[AR_CS], dtau = p.psidecayfac * vclean / h;
      psi_b += zeta * (-dtau + 0.5 * pm * fs4 * rho1);
      cs_b += zeta * p.overcleanfac * (-fs11 * rho1 - psi * p.psidecayfac / h);  // v_wave
      rho_b -= zeta * (-vclean * fs11 + 0.5 * psi * pm * fs4) * rho1 * rho1;
      h_fin = zeta * psi * dtau / h;
    }
    const double bx = r[AR_BX], by = r[AR_BY], bz = r[AR_BZ], b2r = bx * bx + by * by + bz * bz;
    bx_b = ps_(PA_BX); by_b = ps_(PA_BY); bz_b = ps_(PA_BZ);
    // P/rho^2 + |B/rho|^2/2: the magnetic part
    const double pro2_b = ps_(PA_PRO2);
    bx_b += pro2_b * bx; by_b += pro2_b * by; bz_b += pro2_b * bz;
    // v_wave = sqrt(c_s^2 + |B/rho|^2 rho)
    const double vw = r[AR_CS], vw_b = cs_b;
    cs_b = vw > 0.0 ? vw_b * cs / vw : 0.0;
    if (vw > 0.0) {
      bx_b += vw_b * rho * bx / vw; by_b += vw_b * rho * by / vw; bz_b += vw_b * rho * bz / vw;
      rho_b += vw_b * b2r / (2.0 * vw);
    }
    // div B subtraction: kap = -(w . B/rho) rho frac(beta), beta = 2 P / (|B/rho|^2 rho^2), times the sum
    const double D = ps_(PA_DIVB), P = r[AR_P];
    const double B2 = b2r * rho * rho;
    if (B2 > 0.0 && D != 0.0) {
      const double beta = 2.0 * P / B2;
      double f, df;
      divb_frac(beta, f, df);
      const double wb = r[AR_WX] * bx + r[AR_WY] * by + r[AR_WZ] * bz;
      bx_b += D * (-r[AR_WX] * rho * f + wb * rho * df * 2.0 * beta * bx / b2r);
      by_b += D * (-r[AR_WY] * rho * f + wb * rho * df * 2.0 * beta * by / b2r);
      bz_b += D * (-r[AR_WZ] * rho * f + wb * rho * df * 2.0 * beta * bz / b2r);
      rho_b += D * (-wb * f + wb * rho * df * 2.0 * beta / rho);
      P_b += D * (-wb * rho * df * beta / P);
    }
  }
  // rho-dependence of 1/rho, P/rho^2, P (eos); then h through rho = m (hfact/h)^3
  double u_b = ps_(PA_U);
  if (p.ieos == 1) {
    rho_b += P_b * p.polyk - ps_(PA_PRO2) * p.polyk * rho1 * rho1;
  } else {
    const double gm1 = (p.gamma > 1.0001) ? (p.gamma - 1.0) : 2.0 / 3.0;
    rho_b += P_b * gm1 * u - ps_(PA_PRO2) * gm1 * u * rho1 * rho1;
    u_b += P_b * gm1 * rho + ps_(PA_PRO2) * gm1 * rho1;
    if (cs > 0.0) u_b += cs_b * p.gamma * gm1 / (2.0 * cs);  // c_s = sqrt(gamma gm1 u)
  }
  double h_b = ps_(PA_H) + rho_b * (-3.0 * rho / h) + h_fin;
  // self-gravity: gradsoft = -K (S_phi + 1.4 m), K = h^2 / (3 m hfact^3),
  // S_phi = sum_j m dphi_h(r_ij/h): d/dh at fixed x = 2 gradsoft/h + K SG/h
  // (SG = sum m q dphi_h/dq), and the coefficient C = -K gradsoft_bar on
  // dS_phi/dx for pass 2
  double C = 0.0;
  if (p.gravity) {
    const double K = h * h / (3.0 * pm * p.hfact * p.hfact * p.hfact);
    const double GS_b = ps_(PA_GS);
    h_b += GS_b * (2.0 * r[AR_GS] + K * ps_(PA_SG)) / h;
    C = -GS_b * K;
  }
  r[AR_C] = C;
  const double G_b = ps_(PA_G);
  // implicit solve: Omega = 1 - dhdrho S, S = d rho / dh (at fixed x)
  const double dhdrho = -h / (3.0 * rho);
  const double Om = 1.0 / G;
  const double S = (1.0 - Om) / dhdrho;
  // d2 rho/dh2 including the self term m cn h^-5 * 12
  const double h1 = 1.0 / h;
  const double d2 = ps_(PA_D2) + pm * CNORMK * 12.0 * h1 * h1 * h1 * h1 * h1;
  const double dOm_dh = -(4.0 * dhdrho * h1) * S - dhdrho * d2;
  const double dG_dh = -G * G * dOm_dh;
  const double H = h_b + G_b * dG_dh;
  r[AR_A] = H * dhdrho * G;
  r[AR_B] = G_b * G * G * dhdrho;
  // pass 2 of hydro contexts: A h^-4 w' + B h^-5 (-4 w' - q w'') on hs1 and q hs2
  const double h4 = pm * CNORMK * (h1 * h1) * (h1 * h1), b5 = r[AR_B] * h4 * h1, a4 = r[AR_A] * h4 - 4.0 * b5;
  if (hrec) { double *o = hrec + HREC * (size_t)i; o[HR_A3] = hs1_fac<double>() * a4; o[HR_B1] = -1.5 * b5; }
  if (hrecf) { float *o = hrecf + HREC * (size_t)i; o[HR_A3] = (float)a4; o[HR_B1] = (float)(-1.5 * b5); }
  if (adjf) {
    float *q = adjf + ADJREC * (size_t)i;
    q[AR_A] = (float)r[AR_A]; q[AR_B] = (float)r[AR_B]; q[AR_C] = (float)C;
  }
  r[AR_GX] = ps_(PA_X); r[AR_GY] = ps_(PA_Y); r[AR_GZ] = ps_(PA_Z);
  r[AR_GVX] = ps_(PA_VX); r[AR_GVY] = ps_(PA_VY); r[AR_GVZ] = ps_(PA_VZ);
  r[AR_GU] = u_b;
  r[AR_GBX] = bx_b; r[AR_GBY] = by_b; r[AR_GBZ] = bz_b; r[AR_GPSI] = psi_b;
}

// pass 2: positions through the density sums
template <typename T>
__global__ void __launch_bounds__(32 * ADJ_WARPS) k_adj_dens(Params p, const Node *nodes, const int *leaves,
                                                             int ncell, const LeafEntry *pool, const int *cell_off,
                                                             const int *cell_nleaf, const int *cell_ntrial,
                                                             const double *tx, const double *ty, const double *tz,
                                                             const float4 *txf, const T *adj, double *psum,
                                                             int64_t ps, double pf_hmin, int *err) {
  const int w = threadIdx.x >> 5, lane = lane_id();
  const int cell = blockIdx.x * ADJ_WARPS + w;
  if (cell >= ncell) return;
  const Node nd = nodes[leaves[cell]];
  const int np = nd.count, s0 = nd.start;
  if (np < 1 || np > MAXCELL) { if (lane == 0) set_error(err, PH_ERR_TREE); return; }
  const int S = 32 / np;
  const bool act = lane < np * S;
  const int il = act ? lane / S : 0, stripe = act ? lane % S : 0;
  const int i = s0 + il;
  const T *ri = adj + ADJREC * (size_t)i;
  const T pm = (T)p.massoftype;
  const double xi = tx[i], yi = ty[i], zi = tz[i];
  const T h1i = ri[AR_H1], Ai = ri[AR_A], Bi = ri[AR_B], Ci = ri[AR_C];
  const bool grav = p.gravity != 0;
  const double hi = ri[AR_H];
  const T h4i = T(CNORMK) * h1i * h1i * h1i * h1i, h5i = h4i * h1i;
  const float4 xif = txf[i];
  const float hi21f = xif.w * xif.w;
  const bool pf_i = hi > pf_hmin;
  const float pf_h1max = (float)(1.0 / pf_hmin);
  const float q2lim = 4.0f * 1.001f;
  Acc<T> gx, gy, gz;
  const int off = cell_off[cell], nleaf = cell_nleaf[cell], ntrial = cell_ntrial[cell];
  extern __shared__ __align__(16) unsigned char dsm[];
  PairSmem &sm = reinterpret_cast<PairSmem *>(dsm)[w];
  Stage &stg = sm.st;
  for (int base = 0; base < ntrial; base += STAGE) {
    const int cnt = stage_window(p, pool, off, nleaf, ntrial, base, txf, stg);
    auto test = [&](int k) -> bool {
      if (stg.jidx[k] == i) return false;
      if (!pf_i) return true;
      const float4 xj = stg.pos[k];
      if (xj.w >= pf_h1max) return true;
      float dxf = xif.x - xj.x, dyf = xif.y - xj.y, dzf = xif.z - xj.z;
      if (p.periodic) {
        if (fabsf(dxf) > 0.5f * p.dxboundf) dxf -= copysignf(p.dxboundf, dxf);
        if (fabsf(dyf) > 0.5f * p.dyboundf) dyf -= copysignf(p.dyboundf, dyf);
        if (fabsf(dzf) > 0.5f * p.dzboundf) dzf -= copysignf(p.dzboundf, dzf);
      }
      const float r2f = dxf * dxf + dyf * dyf + dzf * dzf;
      return r2f * fminf(hi21f, xj.w * xj.w) < q2lim;
    };
    auto body = [&](int k) {
      const int j = stg.jidx[k];
      const int code = stg.code[k];
      double dx = xi - (tx[j] + offset_of(code, 0, p.dxbound));
      double dy = yi - (ty[j] + offset_of(code, 1, p.dybound));
      double dz = zi - (tz[j] + offset_of(code, 2, p.dzbound));
      dx = wrap(dx, p.dxbound, p.hdlx, p.periodic); dy = wrap(dy, p.dybound, p.hdly, p.periodic);
      dz = wrap(dz, p.dzbound, p.hdlz, p.periodic);
      const T dxt = sep_t<T>(dx), dyt = sep_t<T>(dy), dzt = sep_t<T>(dz);
      const T r2 = dxt * dxt + dyt * dyt + dzt * dzt, r = sqrt(r2), rinv = inv_sep(r2, r);
      const T *rj = adj + ADJREC * (size_t)j;
      T coef = T(0.0), w0, w1, w2;
      const T qi = r * h1i;
      if (qi < T(2.0)) {  // dW/dr = cn h^-4 w', d2W/dhdr = cn h^-5 (-4 w' - q w'')
        wshape(qi, w0, w1, w2);
        coef += Ai * h4i * w1 + Bi * h5i * (T(-4.0) * w1 - qi * w2);
        if (grav) coef += Ci * h1i * dphidh_dq(qi);
      }
      const T h1j = rj[AR_H1];
      const T qj = r * h1j;
      if (qj < T(2.0)) {
        wshape(qj, w0, w1, w2);
        const T h4j = T(CNORMK) * h1j * h1j * h1j * h1j;
        coef += rj[AR_A] * h4j * w1 + rj[AR_B] * h4j * h1j * (T(-4.0) * w1 - qj * w2);
        if (grav) coef += rj[AR_C] * h1j * dphidh_dq(qj);
      }
      coef *= pm * rinv;
      gx += coef * dxt; gy += coef * dyt; gz += coef * dzt;
    };
    queue_window(cnt, S, act, il, stripe, sm.q, test, body);
  }
  double *red = reinterpret_cast<double *>(&sm.st);
  __syncwarp();
  red[lane * 3] = gx.value(); red[lane * 3 + 1] = gy.value(); red[lane * 3 + 2] = gz.value();
  __syncwarp();
  if (lane < np) {
    double t0 = 0, t1 = 0, t2 = 0;
    for (int q = 0; q < S; ++q) {
      const double *src = red + (lane * S + q) * 3;
      t0 += src[0]; t1 += src[1]; t2 += src[2];
    }
    const size_t ip = (size_t)(s0 + lane);
    psum[ip] = t0; psum[ps + ip] = t1; psum[2 * ps + ip] = t2;
  }
}

// results in the caller's order: gradients with respect to xyzh (h slot 0:
// h is not an independent input), vxyzu and, with MHD, Bevol (B/rho and psi)
__global__ void k_adj_out(int n, const int *perm, const double *adj, const double *psum, int64_t ps, int grav,
                          double *gxyzh, double *gvxyzu, double *gBevol) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int pid = perm[i];
  const double *r = adj + ADJREC * (size_t)i;
  double *gx = gxyzh + 4 * (size_t)pid, *gv = gvxyzu + 4 * (size_t)pid;
  gx[0] = r[AR_GX] + psum[i]; gx[1] = r[AR_GY] + psum[ps + i]; gx[2] = r[AR_GZ] + psum[2 * ps + i]; gx[3] = 0.0;
  if (grav) {  // the far field's share (slots 3..5)
    gx[0] += psum[3 * ps + i]; gx[1] += psum[4 * ps + i]; gx[2] += psum[5 * ps + i];
  }
  gv[0] = r[AR_GVX]; gv[1] = r[AR_GVY]; gv[2] = r[AR_GVZ]; gv[3] = r[AR_GU];
  if (gBevol) {
    double *gb = gBevol + 4 * (size_t)pid;
    gb[0] = r[AR_GBX]; gb[1] = r[AR_GBY]; gb[2] = r[AR_GBZ]; gb[3] = r[AR_GPSI];
  }
}

static inline int nblk(int64_t n, int b) { return (int)((n + b - 1) / b); }

}  // namespace ph

using namespace ph;

namespace ph {

// The adjoint on the device-resident state: cotangents w of fxyzu and, with
// MHD, wB of dBevol (caller order, 4 rows per particle, device; wB may be
// null) -> gradients gx, gv (and gb with MHD), caller order, device. The tree, density and force lists are recomputed unless the
// state flags say they are current. Records ev[0..2] around the recompute and
// the adjoint passes and evk[0..1] around the pair passes.
int adjoint_dev(ph_ctx *c, const double *w_dev, const double *wB_dev, double *gx_d, double *gv_d, double *gb_d) {
  const Params p = c->dp;
  if (alloc_adjoint(c) != 0) return PH_ERR_CUDA;
  cudaStream_t st = c->stream;
  cudaEventRecord(c->ev[0], st);
  // forward state at the uploaded positions: tree, density, force lists
  int r = 0;
  if (!c->have_tree || (p.gravity && !c->tree_grav)) { r = build_tree(c); if (r) return r; }
  if (!c->have_density) { r = density(c, 1); if (r) return r; }
  r = force_lists(c);
  if (r) return r;
  cudaEventRecord(c->ev[1], st);
  const int nt = (int)c->ntree, ncell = c->nleaves;
  // cotangents staged in the pair-sum buffer (caller order, 4 per particle)
  const size_t n4 = 4 * (size_t)c->n;
  const bool wB = p.mhd && wB_dev;
  cudaMemcpyAsync(c->psum, w_dev, sizeof(double) * n4, cudaMemcpyDeviceToDevice, st);
  if (wB) cudaMemcpyAsync(c->psum + n4, wB_dev, sizeof(double) * n4, cudaMemcpyDeviceToDevice, st);
  const bool mixed = p.precision == PH_PREC_MIXED;
  // hydro contexts: the joint pair reverse, from its own records (in the force
  // records' space, which the next force call rebuilds); FP64 on the symmetric
  // force lists, each pair once
  const bool hydro = !p.mhd && !p.gravity && !c->keep_order;
  if (hydro && mixed) low_words(c);
  const bool sym = hydro && !mixed && c->force_sym && c->toff && c->sym_total > 0;
  double *hrec = sym ? c->jrec : nullptr;
  float *hrecf = hydro && mixed ? c->jrecf : nullptr;
  k_adj_prologue<<<nblk(nt, 256), 256, 0, st>>>(p, nt, c->perm, c->th, c->gradh64, c->gsoft64, c->vxyzu, c->Bevol,
                                                c->psum, wB ? c->psum + n4 : nullptr, c->alpha1, c->adj,
                                                mixed && !hydro ? c->adjf : nullptr, hrec, hrecf, c->txf);
  const int smem = ADJ_WARPS * (int)sizeof(PairSmem), lsmem = ADJ_WARPS * (int)sizeof(ListSmem);
  if (!(c->attr_done & 4u)) {
    const auto at = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaFuncSetAttribute(k_adj_pairs<double, false>, at, smem);
    cudaFuncSetAttribute(k_adj_pairs<double, true>, at, smem);
    cudaFuncSetAttribute(k_adj_dens<double>, at, smem);
    cudaFuncSetAttribute(k_adj_pairs<float, false>, at, smem);
    cudaFuncSetAttribute(k_adj_pairs<float, true>, at, smem);
    cudaFuncSetAttribute(k_adj_dens<float>, at, smem);
    cudaFuncSetAttribute(k_adj_pairs_sym, at, sym_smem_bytes<NJA>(MAXCELL));
    cudaFuncSetAttribute(k_adj_dens_sym, at, sym_smem_bytes<3>(MAXCELL));
    cudaFuncSetAttribute(k_adj_pairs_hydro, at, lsmem);
    cudaFuncSetAttribute(k_adj_dens_hydro, at, lsmem);
    c->attr_done |= 4u;
  }
  cudaEventRecord(c->evk[0], st);
  const HConst hc{p.beta, !p.isothermal && p.alphau != 0.0, p.ipdv_heating > 0, p.ishock_heating > 0};
  if (hydro && mixed) {
    k_adj_pairs_hydro<<<nblk(ncell, ADJ_WARPS), 32 * ADJ_WARPS, lsmem, st>>>(
        p, hc, c->nodes, c->leaves, ncell, c->pool, c->cell_off, c->cell_nleaf, c->tx, c->ty, c->tz, c->txf, c->txl,
        hrecf, c->adj, c->psum, c->cap, c->pf_hmin, c->d_err);
    k_adj_coef<<<nblk(nt, 256), 256, 0, st>>>(p, nt, c->psum, c->cap, c->adj, nullptr, nullptr, hrecf);
    k_adj_dens_hydro<<<nblk(ncell, ADJ_WARPS), 32 * ADJ_WARPS, lsmem, st>>>(
        p, c->nodes, c->leaves, ncell, c->pool, c->cell_off, c->cell_nleaf, c->tx, c->ty, c->tz, c->txf, c->txl, hrecf,
        c->psum, c->cap, c->pf_hmin, c->d_err);
  } else if (sym) {
    if (alloc_sym(c, c->sym_total, NJA) != 0) return PH_ERR_CUDA;
    k_adj_pairs_sym<<<ncell, 32, sym_smem_bytes<NJA>(p.minpart), st>>>(
        p, hc, c->nodes, c->leaves, ncell, c->pool, c->cell_off, c->cell_nleaf, c->tx, c->ty, c->tz, c->txf, hrec,
        c->psum, c->cap, c->pf_hmin, c->toff, c->jbuf, c->jbuf_stride, c->d_err);
    k_adj_gather<NJA><<<nblk(ncell, 4), 128, 0, st>>>(c->nodes, c->leaves, ncell, c->pool, c->cell_off,
                                                      c->cell_nleaf, c->cell_at, c->toff, c->jbuf, c->jbuf_stride,
                                                      c->adj, p.massoftype, c->psum, c->cap);
    k_adj_coef<<<nblk(nt, 256), 256, 0, st>>>(p, nt, c->psum, c->cap, c->adj, nullptr, hrec, nullptr);
    k_adj_dens_sym<<<ncell, 32, sym_smem_bytes<3>(p.minpart), st>>>(
        p, c->nodes, c->leaves, ncell, c->pool, c->cell_off, c->cell_nleaf, c->tx, c->ty, c->tz, c->txf, hrec, c->psum,
        c->cap, c->pf_hmin, c->toff, c->jbuf, c->jbuf_stride, c->d_err);
    k_adj_gather<3><<<nblk(ncell, 4), 128, 0, st>>>(c->nodes, c->leaves, ncell, c->pool, c->cell_off, c->cell_nleaf,
                                                    c->cell_at, c->toff, c->jbuf, c->jbuf_stride, c->adj,
                                                    p.massoftype, c->psum, c->cap);
    count_launch(c, 2);
  } else {
    auto consts = [&](auto &kc) {
      using T = decltype(kc.m);
      kc.m = (T)p.massoftype; kc.alpha = (T)p.alpha; kc.beta = (T)p.beta; kc.alphau = (T)p.alphau; kc.cn = (T)CNORMK;
      kc.adiab = !p.isothermal; kc.pdv = p.ipdv_heating > 0; kc.shock = p.ishock_heating > 0; kc.mhd = p.mhd != 0;
      kc.grav = p.gravity != 0;
      kc.alphaB = (T)p.alphaB; kc.oc = (T)p.overcleanfac;
      kc.resist = p.mhd && p.iresistive_heating > 0 && !p.isothermal;
      kc.induct = p.mhd && (wB || kc.resist);
    };
    const int nb = nblk(ncell, ADJ_WARPS), nthr = 32 * ADJ_WARPS;
#define PH_ADJ(T, REC, RECF)                                                                                      \
  do {                                                                                                            \
    AdjConst<T> kc;                                                                                               \
    consts(kc);                                                                                                   \
    (kc.induct ? k_adj_pairs<T, true> : k_adj_pairs<T, false>)<<<nb, nthr, smem, st>>>(                           \
        p, kc, c->nodes, c->leaves, ncell, c->pool, c->cell_off, c->cell_nleaf, c->cell_ntrial, c->tx, c->ty,     \
        c->tz, c->txf, REC, c->psum, c->cap, c->pf_hmin, c->d_err);                                               \
    k_adj_coef<<<nblk(nt, 256), 256, 0, st>>>(p, nt, c->psum, c->cap, c->adj, RECF, nullptr, nullptr);            \
    k_adj_dens<T><<<nb, nthr, smem, st>>>(p, c->nodes, c->leaves, ncell, c->pool, c->cell_off, c->cell_nleaf,     \
                                          c->cell_ntrial, c->tx, c->ty, c->tz, c->txf, REC, c->psum, c->cap,      \
                                          c->pf_hmin, c->d_err);                                                  \
  } while (0)
    if (mixed) PH_ADJ(float, c->adjf, c->adjf);
    else PH_ADJ(double, c->adj, nullptr);
#undef PH_ADJ
  }
  // self-gravity: the far field's share of the position gradients (slots 3..5)
  if (p.gravity) gravity_adjoint_far(c, c->adj + AR_WX, ADJREC, c->psum + 3 * c->cap, c->cap);
  cudaEventRecord(c->evk[1], st);
  k_adj_out<<<nblk(nt, 256), 256, 0, st>>>(nt, c->perm, c->adj, c->psum, c->cap, p.gravity ? 1 : 0, gx_d, gv_d,
                                           gb_d);
  count_launch(c, 5);
  cudaEventRecord(c->ev[2], st);
  return 0;
}

}  // namespace ph

extern "C" {

int ph_adjoint_full(ph_ctx *c, const double *w_fxyzu, const double *w_dBevol, double *g_xyzh, double *g_vxyzu,
                    double *g_Bevol) {
  if (!c || !w_fxyzu || !g_xyzh || !g_vxyzu) return PH_ERR_ARG;
  if (c->n <= 0) return PH_ERR_NOPART;
  const Params p = c->dp;
  // individual timesteps: an evaluation re-computes the active particles'
  // forces only (the inactive ones keep theirs), and its lists cover the
  // active cells only; its adjoint is not built
  if (p.ind) return PH_ERR_NOT_BUILT;
  if (p.mhd && !g_Bevol) return PH_ERR_ARG;
  if (alloc_adjoint(c) != 0) return PH_ERR_CUDA;
  cudaStream_t st = c->stream;
  reset_timers(c);
  const size_t n = (size_t)c->n;
  const bool wB = p.mhd && w_dBevol;
  // cotangents in caller order, staged where the recompute of the tree and
  // density (whose pair sums use psum, whose velocity-derivative pass uses
  // jrec) cannot overwrite them
  if (alloc_rollout(c, 8 * n) != 0) return PH_ERR_CUDA;
  copy_vrows_h2d(c, c->ro_buf, w_fxyzu, (size_t)n);
  if (wB) cudaMemcpyAsync(c->ro_buf + 4 * n, w_dBevol, sizeof(double) * 4 * n, cudaMemcpyHostToDevice, st);
  double *gx_d = c->jrec, *gv_d = c->jrec + 4 * n, *gb_d = p.mhd ? c->jrec + 8 * n : nullptr;
  int r = adjoint_dev(c, c->ro_buf, wB ? c->ro_buf + 4 * n : nullptr, gx_d, gv_d, gb_d);
  if (r) return r;
  cudaMemcpyAsync(g_xyzh, gx_d, sizeof(double) * 4 * n, cudaMemcpyDeviceToHost, st);
  copy_vrows_d2h(c, g_vxyzu, gv_d, (size_t)n);
  if (p.mhd) cudaMemcpyAsync(g_Bevol, gb_d, sizeof(double) * 4 * n, cudaMemcpyDeviceToHost, st);
  if (cudaStreamSynchronize(st) != cudaSuccess) return PH_ERR_CUDA;
  int herr = 0;
  cudaMemcpy(&herr, c->d_err, sizeof(int), cudaMemcpyDeviceToHost);
  if (herr) return herr;
  float ms;
  // device time: [0] forward recompute (tree, density, lists), [2] adjoint
  // passes, [4] the pair passes, [7] total (cotangent upload included,
  // gradient download excluded)
  cudaEventElapsedTime(&ms, c->ev[0], c->ev[1]); c->last_ms[0] = ms;
  cudaEventElapsedTime(&ms, c->ev[1], c->ev[2]); c->last_ms[2] = ms;
  add_elapsed(c, 4, c->evk[0], c->evk[1]);
  cudaEventElapsedTime(&ms, c->ev[0], c->ev[2]); c->last_ms[7] = ms;
  return check_launch(c) == cudaSuccess ? 0 : PH_ERR_CUDA;
}

int ph_adjoint(ph_ctx *c, const double *w_fxyzu, double *g_xyzh, double *g_vxyzu, double *g_Bevol) {
  return ph_adjoint_full(c, w_fxyzu, nullptr, g_xyzh, g_vxyzu, g_Bevol);
}

}  // extern "C"
