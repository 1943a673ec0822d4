// Hydro evaluations of the precision form's rollouts (ph_rollout_adjoint).
//
// A rollout's gradient runs through the square root of |P_i - P_j| in the
// conductivity's signal speed and through the viscosity's switch at v.r = 0 at
// every step, so FP32 pair sums leave single components of it undetermined. On
// hydro lattices (viscosity and conductivity on), against the FP64 rollout of the
// same steps: median relative error 2e-6, 99 % of the components within 2e-3, but
// the largest error, over the largest component, 0.04 after 2 steps of 40^3
// particles, 0.25 after 8; and the pair sums of ph_step's kernels, of the same
// accuracy in another order, give a gradient that differs as much (0.03 and
// 1.4; in norm 1.6e-4 and 5e-3). A program that follows a rollout's gradient from
// one version to the next would see those components jump, so rollouts keep
// the pair order (a lane per particle and stripe, windows of STAGE entries) and the
// arithmetic (FP64 separations rounded to FP32) their results have had; adjoint_dev
// likewise keeps the reverse of both ordered terms for them. Their trajectory is
// therefore not ph_step's bit for bit.
#include "ph_internal.h"
#include "ph_walk.cuh"

namespace ph {

constexpr int RO_NN = 13;             // density: neighbour count slot (bit pattern)
constexpr int RO_NF = 12;             // force: sums 0..6 in use, then the signal speed
constexpr int RO_JREC = 16, RO_JF = 16;  // record strides (doubles, floats)

// get_density_sums (dens.F90:578-857) of the active cells
__global__ void __launch_bounds__(32 * MAX_WARPS) k_ro_density(
    Params p, const Node *nodes, const int *leaves, const int *act, int nact, const LeafEntry *pool,
    const int *cell_off, const int *cell_nleaf, const int *cell_ntrial, const double *tx, const double *ty,
    const double *tz, const float4 *txf, const double *hcur, double *psum, int64_t ps, unsigned long long *stats,
    int *err) {
  extern __shared__ __align__(16) unsigned char dsm[];
  const int w = threadIdx.x >> 5, lane = lane_id();
  const int a = blockIdx.x * (blockDim.x >> 5) + w;
  if (a >= nact) return;
  const int cell = act[a];
  const Node nd = nodes[leaves[cell]];
  const int np = nd.count, s0 = nd.start;
  if (np < 1 || np > MAXCELL) {
    if (lane == 0) set_error(err, PH_ERR_TREE);
    return;
  }
  const int S = 32 / np;
  const bool active_lane = lane < np * S;
  const int il = active_lane ? lane / S : 0, stripe = active_lane ? lane % S : 0;
  const int i = s0 + il;
  const double pm = p.massoftype;
  const double xi = tx[i], yi = ty[i], zi = tz[i];
  const double hi = hcur[i], hi1 = ddiv(1.0, hi), hi21 = dmul(hi1, hi1);
  const float4 xif = txf[i];
  const float hi21f = (float)hi21;
  const float q2lim = 4.0f * 1.001f;
  Kahan kacc[2];
  const float hi1f = (float)hi1, pmf = (float)pm;
  int nn = 0;
  const int off = cell_off[cell], nleaf = cell_nleaf[cell];
  const int ntrial = cell_ntrial[cell];
  if (lane == 0) {
    atomicAdd(&stats[9], (unsigned long long)ntrial);
    atomicAdd(&stats[11], (unsigned long long)np * (unsigned long long)ntrial);
  }
  PairSmem &sm = reinterpret_cast<PairSmem *>(dsm)[w];
  for (int base = 0; base < ntrial; base += STAGE) {
    const int cnt = stage_window(p, pool, off, nleaf, ntrial, base, txf, sm.st);
    auto test = [&](int k) -> bool {
      if (sm.st.jidx[k] == i) return false;  // ignoreself (dens.F90:650)
      const float4 xj = sm.st.pos[k];
      float dxf = xif.x - xj.x, dyf = xif.y - xj.y, dzf = xif.z - xj.z;
      if (p.periodic) {
        if (fabsf(dxf) > 0.5f * p.dxboundf) dxf -= copysignf(p.dxboundf, dxf);
        if (fabsf(dyf) > 0.5f * p.dyboundf) dyf -= copysignf(p.dyboundf, dyf);
        if (fabsf(dzf) > 0.5f * p.dzboundf) dzf -= copysignf(p.dzboundf, dzf);
      }
      const float r2f = dxf * dxf + dyf * dyf + dzf * dzf;
      return r2f * hi21f < q2lim;
    };
    // the pair's operands, then its body
    struct PF { int code; float4 xj; double x, y, z; };
    auto load = [&](int k) -> PF {
      PF f;
      const int j = sm.st.jidx[k];
      f.code = sm.st.code[k]; f.xj = sm.st.pos[k];
      f.x = tx[j]; f.y = ty[j]; f.z = tz[j];
      return f;
    };
    auto body_m = [&](const PF &pf) {
      {
        // separation formed in FP64 (the periodic image chosen on the FP32
        // copy), rounded to FP32; W, dW/dh and the sums in FP32 (Kahan)
        const float4 xj = pf.xj;
        float dx, dy, dz;
        separation_mixed(p, xi, yi, zi, pf.x, pf.y, pf.z, pf.code, xif.x - xj.x, xif.y - xj.y, xif.z - xj.z, dx,
                         dy, dz);
        const float r2 = dx * dx + dy * dy + dz * dz;
        const float q2 = r2 * hi21f;
        if (q2 < 4.0f) {
          const float rij = sqrtf(r2), q = rij * hi1f;
          float wab, grk;
          if (q < 1.0f) { wab = 0.75f * q2 * q - 1.5f * q2 + 1.0f; grk = q * (2.25f * q - 3.0f); }
          else { const float t2 = q - 2.0f; wab = -0.25f * t2 * t2 * t2; grk = -0.75f * t2 * t2; }
          kacc[0].add(wab * pmf);
          kacc[1].add((-q * grk - 3.0f * wab) * pmf);
          ++nn;
        }
      }
    };
    queue_window(cnt, S, active_lane, il, stripe, sm.q, test, [&](int k) { body_m(load(k)); });
  }
  // the stripes of each particle in stripe order (in the staged window's space)
  constexpr int RW = 3;
  double *red = reinterpret_cast<double *>(&sm.st);
  __syncwarp();
  for (int k = 0; k < 2; ++k) red[lane * RW + k] = kacc[k].value();
  red[lane * RW + 2] = __longlong_as_double((long long)nn);
  __syncwarp();
  if (lane < np) {
    double r[2] = {0.0, 0.0};
    long long nni = 0;
    for (int q = 0; q < S; ++q) {
      const double *src = red + (lane * S + q) * RW;
      for (int k = 0; k < 2; ++k) r[k] = dadd(r[k], src[k]);
      nni += __double_as_longlong(src[2]);
    }
    const size_t ip = (size_t)(s0 + lane);
    for (int k = 0; k < 2; ++k) psum[k * ps + ip] = r[k];
    psum[RO_NN * ps + ip] = __longlong_as_double(nni);
  }
}

// cons2prim (cons2prim.f90:326-456) and the FP32 particle records of k_ro_force
__global__ void k_ro_prologue(Params p, int n, const int *perm, const double *th, const double *vel,
                              const float *gradh, double *eos_t, double *jrec, float *jrecf, float4 *txf, int *err) {
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
  const float pro2 = P * rho1 * rho1, vwave = cs;
  const size_t g = (size_t)j;
  const float mrho5 = 0.5f * pmf * rho1;
  float *o = jrecf + RO_JF * (size_t)j;
  o[0] = h1; o[1] = rho; o[2] = rho1; o[3] = pro2; o[4] = vwave; o[5] = P;
  o[6] = mrho5 * d2f_rn(p.alphau); o[7] = gradh[2 * g];
  o[8] = d2f_rn(v[0]); o[9] = d2f_rn(v[1]); o[10] = d2f_rn(v[2]); o[11] = u;
  o[12] = gradh[2 * g + 1];
  o[13] = mrho5 * d2f_rn(p.alphaB) * rho1;
  o[14] = d2f_rn(p.alpha);
  o[15] = rho1 * rho1;
  jrec[RO_JREC * (size_t)j + 11] = p.isothermal ? 0.0 : v[3];  // the finish's u
  txf[j].w = h1;
}

// M4 dW/dq (kernel_cubic.f90:56-66)
__device__ __forceinline__ float ro_grkern(float q) {
  if (q < 1.0f) return q * (2.25f * q - 3.0f);
  if (q < 2.0f) { float t = q - 2.0f; return -0.75f * (t * t); }
  return 0.0f;
}

// compute_forces (force.F90:914-2060), hydro
__global__ void __launch_bounds__(32 * MAX_WARPS) k_ro_force(
    Params p, const Node *nodes, const int *leaves, int ncell, const LeafEntry *pool, const int *cell_off,
    const int *cell_nleaf, const int *cell_ntrial, const double *tx, const double *ty, const double *tz,
    const float4 *txf, const float *jrecf, unsigned long long *stats, double *psum, int64_t ps, int *err) {
  const int w = threadIdx.x >> 5, lane = lane_id();
  const int a = blockIdx.x * (blockDim.x >> 5) + w;
  if (a >= ncell) return;
  const int cell = a;
  const Node nd = nodes[leaves[cell]];
  const int np = nd.count, s0 = nd.start;
  if (np < 1 || np > MAXCELL) { if (lane == 0) set_error(err, PH_ERR_TREE); return; }
  const int S = 32 / np;
  const bool act = lane < np * S;
  const int il = act ? lane / S : 0, stripe = act ? lane % S : 0;
  const int i = s0 + il;
  const float pmf = (float)p.massoftype;
  const bool adiab = !p.isothermal;
  // i-side from the FP32 particle record (its density is rhoh(1/(1/h)) rather
  // than rhoanddhdrho's m (hfact/h)^3: a last-ulp difference in FP64, nil in FP32)
  const float *ri = jrecf + RO_JF * (size_t)i;
  const float hi1f = ri[0], hi21f = hi1f * hi1f;
  const float gradhi = (ri[7] > 0.0f) ? ri[7] : 1.0f;
  const float hfacgrkern = hi21f * hi21f * (float)CNORMK * gradhi;
  const float rhoif = ri[1], rho1if = ri[2], pro2if = ri[3], vwaveif = ri[4], prif = ri[5];
  const float auterm = ri[6];
  const float alphai = ri[14], beta = (float)p.beta;
  const float vxi = ri[8], vyi = ri[9], vzi = ri[10], eni = ri[11];
  const double xi = tx[i], yi = ty[i], zi = tz[i];
  const float4 xif = txf[i];
  const float q2lim = 4.0f * 1.001f;
  const float hLx = 0.5f * p.dxboundf, hLy = 0.5f * p.dyboundf, hLz = 0.5f * p.dzboundf;
  Kahan f[7];
  float vsigmax = 0.0f;
  const int off = cell_off[cell], nleaf = cell_nleaf[cell];
  if (lane == 0) {
    atomicAdd(&stats[8], (unsigned long long)cell_ntrial[cell]);
    atomicAdd(&stats[10], (unsigned long long)np * (unsigned long long)cell_ntrial[cell]);
  }
  const int ntrial = cell_ntrial[cell];
  extern __shared__ __align__(16) unsigned char dsm[];
  PairSmem &sm = reinterpret_cast<PairSmem *>(dsm)[w];
  Stage &stg = sm.st;
  for (int base = 0; base < ntrial; base += STAGE) {
    const int cnt = stage_window(p, pool, off, nleaf, ntrial, base, txf, stg);
    auto test = [&](int k) -> bool {
      if (stg.jidx[k] == i) return false;
      const float4 xj = stg.pos[k];  // x, y, z (+ offset), 1/h
      const float ux = xif.x - xj.x, uy = xif.y - xj.y, uz = xif.z - xj.z;
      float dxf = ux, dyf = uy, dzf = uz;
      if (p.periodic) {
        if (fabsf(dxf) > hLx) dxf -= copysignf(p.dxboundf, dxf);
        if (fabsf(dyf) > hLy) dyf -= copysignf(p.dyboundf, dyf);
        if (fabsf(dzf) > hLz) dzf -= copysignf(p.dzboundf, dzf);
      }
      const float r2f = dxf * dxf + dyf * dyf + dzf * dzf;
      return r2f * fminf(hi21f, xj.w * xj.w) < q2lim;
    };
    struct PF { int code; float4 xj; double x, y, z; float4 r0, r1, r2, r3; };
    auto load = [&](int k) -> PF {
      PF f;
      const int j = stg.jidx[k];
      f.code = stg.code[k]; f.xj = stg.pos[k];
      f.x = tx[j]; f.y = ty[j]; f.z = tz[j];
      const float4 *r4 = reinterpret_cast<const float4 *>(jrecf + RO_JF * (size_t)j);
      f.r0 = r4[0]; f.r1 = r4[1]; f.r2 = r4[2]; f.r3 = r4[3];
      return f;
    };
    auto body = [&](const PF &pf) {
      const float4 xj = pf.xj;
      float dx, dy, dz;
      separation_mixed(p, xi, yi, zi, pf.x, pf.y, pf.z, pf.code, xif.x - xj.x, xif.y - xj.y, xif.z - xj.z, dx,
                       dy, dz);
      const float rij2 = dx * dx + dy * dy + dz * dz;
      const float rj[RO_JF] = {pf.r0.x, pf.r0.y, pf.r0.z, pf.r0.w, pf.r1.x, pf.r1.y, pf.r1.z, pf.r1.w,
                               pf.r2.x, pf.r2.y, pf.r2.z, pf.r2.w, pf.r3.x, pf.r3.y, pf.r3.z, pf.r3.w};
      const float hj1 = rj[0];
      const float hj21 = hj1 * hj1;
      const float q2i = rij2 * hi21f, q2j = rij2 * hj21;
      const bool qi_in = q2i < 4.0f, qj_in = q2j < 4.0f;
      if (qi_in || qj_in) {
        // coincident particles: no direction, rij1 = 0 (force.F90:1293-1298)
        const float rij1 = rij2 > TINY_F ? rsqrt_nr(rij2) : 0.0f;
        const float rij = rij2 * rij1;
        const float qi = rij * hi1f;
        float grkerni = 0.0f;
        if (qi_in) grkerni = ro_grkern(qi) * hfacgrkern;
        const float runix = dx * rij1, runiy = dy * rij1, runiz = dz * rij1;
        float grkernj = 0.0f;
        bool usej = false;
        if (qj_in) {
          const float qj = rij * hj1;
          grkernj = ro_grkern(qj) * (hj21 * hj21 * (float)CNORMK) * rj[7];
          usej = true;
        }
        if (adiab) usej = true;
        const float dvx = vxi - rj[8], dvy = vyi - rj[9], dvz = vzi - rj[10];
        const float projv = dvx * runix + dvy * runiy + dvz * runiz;
        const float denij = adiab ? eni - rj[11] : 0.0f;
        vsigmax = fmaxf(vsigmax, fmaxf(vwaveif - beta * projv, 0.0f));
        const float vsigavi = fmaxf(alphai * vwaveif - beta * projv, 0.0f);
        float rho1j = 0, pro2j = 0, vwavej = 0, autermj = 0, vsigavj = 0, prj = 0;
        const float rhoj = rj[1];
        if (usej) {
          rho1j = rj[2]; pro2j = rj[3]; vwavej = rj[4]; prj = rj[5];
          autermj = rj[6];
          vsigmax = fmaxf(vsigmax, fmaxf(vwavej - beta * projv, 0.0f));
          vsigavj = fmaxf(rj[14] * vwavej - beta * projv, 0.0f);  // alphaj = alphaind(1,j)
        }
        float qrho2i = 0.0f, qrho2j = 0.0f;
        if (projv < 0.0f) {
          qrho2i = -0.5f * rho1if * vsigavi * projv;
          if (usej) qrho2j = -0.5f * rho1j * vsigavj * projv;
        }
        const float gradpi = pmf * (pro2if + qrho2i) * grkerni;
        const float gradpj = usej ? pmf * (pro2j + qrho2j) * grkernj : 0.0f;
        if (adiab) {
          const float vsigu = sqrtf(fabsf(prif - prj) * __fdividef(2.0f, rhoif + rhoj));
          f[5].add(pmf * qrho2i * projv * grkerni);
          f[6].add(vsigu * denij * (auterm * grkerni + autermj * grkernj));
        }
        const float gradp = gradpi + gradpj;
        f[0].add(-runix * gradp);
        f[1].add(-runiy * gradp);
        f[2].add(-runiz * gradp);
        f[4].add(projv * grkerni);
      }
    };
    queue_window(cnt, S, act, il, stripe, sm.q, test, [&](int k) { body(load(k)); });
  }
  // the stripes of each particle in stripe order (in the staged window's space)
  constexpr int RW = 8;
  double *red = reinterpret_cast<double *>(&sm.st);
  __syncwarp();
  for (int k = 0; k < RW; ++k) red[lane * RW + k] = k < 7 ? f[k].value() : (double)vsigmax;
  __syncwarp();
  if (lane < np) {
    double fs[7];
    for (int k = 0; k < 7; ++k) fs[k] = 0.0;
    double vsm = 0.0;
    for (int q = 0; q < S; ++q) {
      const double *src = red + (lane * S + q) * RW;
      for (int k = 0; k < 7; ++k) fs[k] += src[k];
      vsm = fmax(vsm, src[7]);
    }
    const size_t ip = (size_t)(s0 + lane);
    for (int k = 0; k < 7; ++k) psum[k * ps + ip] = fs[k];
    psum[RO_NF * ps + ip] = vsm;
  }
}

static inline int ro_blocks(int64_t n, int b) { return (int)((n + b - 1) / b); }
constexpr int RO_WARPS = 4;

static void ro_attributes(ph_ctx *c) {
  if (c->attr_done & 8u) return;
  const int bytes = RO_WARPS * (int)sizeof(PairSmem);
  cudaFuncSetAttribute(k_ro_density, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  cudaFuncSetAttribute(k_ro_force, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  c->attr_done |= 8u;
}

// one pass of the density pair sums over the active cells
void ro_density(ph_ctx *c, const int *act, int nact) {
  ro_attributes(c);
  k_ro_density<<<ro_blocks(nact, RO_WARPS), 32 * RO_WARPS, RO_WARPS * sizeof(PairSmem), c->stream>>>(
      c->dp, c->nodes, c->leaves, act, nact, c->pool, c->cell_off, c->cell_nleaf, c->cell_ntrial, c->tx, c->ty, c->tz,
      c->txf, c->hcur, c->psum, c->cap, c->stats, c->d_err);
}

void ro_force_prologue(ph_ctx *c, const double *vel) {
  const int nt = (int)c->ntree;
  k_ro_prologue<<<ro_blocks(nt, 256), 256, 0, c->stream>>>(c->dp, nt, c->perm, c->th, vel, c->gradh_t, c->eos, c->jrec,
                                                           c->jrecf, c->txf, c->d_err);
}

void ro_force(ph_ctx *c) {
  ro_attributes(c);
  k_ro_force<<<ro_blocks(c->nleaves, RO_WARPS), 32 * RO_WARPS, RO_WARPS * sizeof(PairSmem), c->stream>>>(
      c->dp, c->nodes, c->leaves, c->nleaves, c->pool, c->cell_off, c->cell_nleaf, c->cell_ntrial, c->tx, c->ty, c->tz,
      c->txf, c->jrecf, c->stats, c->psum, c->cap, c->d_err);
}

}  // namespace ph
