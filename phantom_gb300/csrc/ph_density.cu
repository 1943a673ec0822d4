// Density h-rho Newton-Raphson solve (K4): densityiterate (dens.F90:117-568)
// with get_density_sums (dens.F90:578-857), finish_cell (dens.F90:1382-1466),
// compute_hmax (dens.F90:1275-1289) and store_results (dens.F90:1511-1681).
//
// Work decomposition: k_density_pairs takes one warp per active leaf cell. The
// warp sweeps the cell's trial list with one trial particle per lane, queues
// for each of the cell's particles the ones that pass the distance pre-filter,
// and sums the queued pairs with its lanes dealt out by queue length (list
// sweep and balanced drain). The sums of each particle go to a per-particle
// array, and k_density_finish (16 lanes per cell) takes the Newton-Raphson
// update, the cell-wide convergence test, the neighbour-list redo decision and
// store_results. Cells iterate in device-wide passes; a cell whose hmax grew is
// re-walked before its next pass, as the reference does per cell.
//
// Neighbour decisions are exact: an FP32 pre-filter with a 1e-3 margin in q^2
// only discards pairs that are provably outside the kernel, and every other
// pair is tested in FP64 with the reference's rounding (no FMA contraction,
// cached positions x_j + offset for the first 1000 trial entries).
#include <type_traits>

#include "ph_internal.h"
#include "ph_walk.cuh"

namespace ph {

constexpr int NACC = 13;  // rho, gradh, gradsoft, divB + 9 dB/dx sums

// get_kernel_grav1 (kernel_cubic.f90:78-99) dphidh term in FP32 (mixed form).
// For 1 <= q < 2 the reference's polynomial vanishes at q = 2 out of terms ~30; in t = 2 - q it is exactly
// t^4 (1/2 - t/5), evaluated that way.
__device__ __forceinline__ float dphidh_f(float q2, float q) {
  if (q < 1.0f) {
    const float q4 = q2 * q2;
    return -0.6f * q4 * q + 1.5f * q4 - 2.0f * q2 + 1.4f;
  } else if (q < 2.0f) {
    const float t = 2.0f - q, t2 = t * t;
    return t2 * t2 * (0.5f - 0.2f * t);
  }
  return 0.0f;
}

// B_j rho_j per tree position for the MHD sums (FP64 rows of 4, or FP32 for
// the mixed form), rho_j from h_j at entry of the density call (the value the
// divcurlB sums read)
__global__ void k_dens_bprep(Params p, int n, const int *perm, const double *Bevol, const double *hj_entry,
                             double *bj, float4 *bjf) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double rho = rhoh(hj_entry[i], p.massoftype, p.hfact);
  const double *b = Bevol + 4 * (size_t)perm[i];
  const double bx = dmul(b[0], rho), by = dmul(b[1], rho), bz = dmul(b[2], rho);
  if (bjf) {
    bjf[i] = make_float4((float)bx, (float)by, (float)bz, 0.0f);
  } else {
    double *o = bj + 4 * (size_t)i;
    o[0] = bx; o[1] = by; o[2] = bz;
  }
}

// the low parts of position i
__device__ __forceinline__ float4 low_parts(const double *tx, const double *ty, const double *tz, const float4 *txf,
                                            int i) {
  const float4 f = txf[i];
  return make_float4(d2f_rn(tx[i] - (double)f.x), d2f_rn(ty[i] - (double)f.y), d2f_rn(tz[i] - (double)f.z), 0.0f);
}
__global__ void k_low_words(int n, const double *tx, const double *ty, const double *tz, const float4 *txf,
                            float4 *txl) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) txl[i] = low_parts(tx, ty, tz, txf, i);
}

// gather per-particle tree-order inputs: h, and for the mixed form the low
// parts of the positions (txf holds the high parts, set by the tree build)
__global__ void k_dens_gather(int n, const int *perm, const double *xyzh, const double *tx, const double *ty,
                              const double *tz, double *hcur, double *hold, const float4 *txf, float4 *txl) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double h = xyzh[4 * (size_t)perm[i] + 3];
  hcur[i] = h; hold[i] = h;
  if (txl) txl[i] = low_parts(tx, ty, tz, txf, i);
}

__global__ void k_dens_init_cells(int ncell, const int *leaves, const Node *nodes, double *cell_hmax,
                                  int *cell_nits, int *act) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncell) return;
  cell_hmax[c] = nodes[leaves[c]].hmax;
  cell_nits[c] = 0;
  act[c] = c;
}

// per-particle pair sums written by k_density_pairs (tree order, slot-major
// with stride ps): slots 0..NACC-1 the sums, then the neighbour count and the
// neighbour-set hash (bit patterns) of each particle, self excluded
constexpr int DSLOT_NN = NACC, DSLOT_HASH = NACC + 1;

struct DensOut {
  double *xyzh;
  float *gradh, *divcurlv, *divcurlB;
  int32_t *nneigh;
  uint64_t *nhash;
  double *th;            // treecache h update (dens.F90:1596)
  double *gradh64;       // 1/Omega in FP64 per tree position (read by the adjoint)
  double *gsoft64;       // gradsoft in FP64 per tree position (self-gravity; read by the adjoint)
  float *gradh_t;        // gradh(2,:) per tree position (read by the force)
  int diag;              // write the caller-order gradh, divcurlv, divcurlB, nneigh, nhash
  double *dvterm;        // cnormk gradh / (rho h^4) per tree position for the dv pass (or null)
  double *rhomax;
  unsigned long long *stats;  // nneightry, nneighact, maxneightry, maxneighact, ncalc, np, ncalls
};

// get_density_sums (dens.F90:578-857) for the active cells: one warp per cell,
// the trial list swept into per-particle queues and drained with the lanes
// dealt out by queue length (list sweep). The neighbour test is the
// reference's: FP32 with a 1e-3 margin in r^2 rejects pairs provably outside
// the kernel (bypassed when h is small against the coordinates), the rest is
// decided in FP64. 28 warps per SM (the dB sums aside): Sedov 100^3, mixed, the
// passes 7.9 -> 7.0 ms against the unbounded allocation's 24.
template <bool MIXED, bool MHD, bool GRAV>
__global__ void __launch_bounds__(32 * MAX_WARPS, MHD ? 4 : 7) k_density_pairs(
    Params p, const Node *nodes, const int *leaves, const int *act, int nact, const LeafEntry *pool,
    const int *cell_off, const int *cell_nleaf, const int *cell_ntrial, const int *perm, const double *tx,
    const double *ty, const double *tz, const float4 *txf, const float4 *txl, const double *hcur, const double *Bevol,
    const double *bj64, const float4 *bjf, double *psum, int64_t ps, unsigned long long *stats, double pf_hmin, const unsigned char *actf,
    int want_hash, int *err) {
  extern __shared__ __align__(16) unsigned char dsm[];
  const int w = threadIdx.x >> 5, lane = lane_id();
  const int a = blockIdx.x * (blockDim.x >> 5) + w;
  if (a >= nact) return;
  const int cell = act[a];
  const Node nd = nodes[leaves[cell]];
  const int np_all = nd.count, s0 = nd.start;
  if (np_all < 1 || np_all > MAXCELL) {
    if (lane == 0) set_error(err, PH_ERR_TREE);
    return;
  }
  int np = np_all;
  unsigned am = 0u;  // active particles (individual timesteps)
  if (actf) am = cell_active_mask(actf, s0, np_all, np);
  if (np == 0) return;
  ListSmem &sm = reinterpret_cast<ListSmem *>(dsm)[w];
  const double pm = p.massoftype;
  const float pmf = d2f_rn(pm);
  double h1own = 0.0;  // lane il: 1/h of particle il
  if (lane < np) {
    const int ip = s0 + (actf ? cell_pos(am, lane) : lane);
    const double h = hcur[ip];
    h1own = ddiv(1.0, h);
    const float hf = d2f_rn(h);
    float4 x = txf[ip];
    x.w = MIXED || h > pf_hmin ? 4.0f * 1.001f * (hf * hf) : __int_as_float(0x7f800000);
    sm.xi[lane] = x;
    sm.ipos[lane] = ip;
  }
  const int off = cell_off[cell], nleaf = cell_nleaf[cell];
  if (lane == 0) {
    const int ntrial = cell_ntrial[cell];
    atomicAdd(&stats[9], (unsigned long long)ntrial);
    atomicAdd(&stats[11], (unsigned long long)np * (unsigned long long)ntrial);
  }
  const float4 cc = make_float4((float)nd.x, (float)nd.y, (float)nd.z, (float)nd.size);
  const int qstride = LQ / np;
  // sum slots: sum W m, sum (-q dW/dq - 3 W) m, sum phi m, with MHD the dB sums
  // (3 div B, 4..12 dB_a/dx_b, whose diagonal no output reads), the neighbour
  // count and the neighbour-set hash (bit patterns)
  constexpr int NA = MHD ? NACC : 3, RW = NA + 2, NR = (RW * MAXCELL + 31) / 32, PHI = 3;
  double tot[NR];
  for (int r = 0; r < NR; ++r) tot[r] = 0.0;
  ListPos pos;
  __syncwarp();
  static_assert(32 * RW <= LQ / 2, "lane sums staged in the queues' space");
  bool more = true;
  while (more) {
    int myc;
    more = SWEEP_END != sweep_list<false>(p, cc, np, pool, off, nleaf, txf, sm, qstride, pos, myc, [](float) { return 0.0f; });
    const QueueLanes ql = balance_queues(np, myc, sm);
    const int il = max(ql.il, 0), i = sm.ipos[il];
    const double hi1 = __shfl_sync(0xffffffffu, h1own, il);
    const int *qj = sm.qj + il * qstride;
    const unsigned char *qc = sm.qc + il * qstride;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    double accb[MHD ? 9 : 1] = {};
    Kahan kacc[MIXED ? NA : 1];
    int nn = 0;
    unsigned long long hh = 0;
    // B_i rho_i with the h of this pass (B_j with h at entry of the call)
    double bxi = 0.0, byi = 0.0, bzi = 0.0;
    if (MHD) {
      const double *b = Bevol + 4 * (size_t)perm[i];
      const double rho = rhoh(hcur[i], pm, p.hfact);
      bxi = dmul(b[0], rho); byi = dmul(b[1], rho); bzi = dmul(b[2], rho);
    }
    if constexpr (MIXED) {
      const Sep2 I = sep2_init(txf, txl, i);
      const float hi1f = d2f_rn(hi1), hi21f = d2f_rn(dmul(hi1, hi1));
      float4 bi = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (MHD) bi = make_float4((float)bxi, (float)byi, (float)bzi, 0.0f);
      for (int m = ql.m0; m < ql.c; m += ql.step) {
        // separation to FP32 precision of the FP64 positions; W, dW/dh and the
        // sums in FP32 (Kahan)
        const int j = qj[m];
        float dx, dy, dz, r2;
        separation_2f(p, I, j, qc[m] & 63, txf[j], txl[j], tx, ty, tz, dx, dy, dz, r2);
        const float q2 = r2 * hi21f;
        if (q2 < 4.0f) {
          const float rij = sqrtf(r2), q = rij * hi1f;
          float wab, grk;
          if (q < 1.0f) { wab = 0.75f * q2 * q - 1.5f * q2 + 1.0f; grk = q * (2.25f * q - 3.0f); }
          else { const float t2 = q - 2.0f; wab = -0.25f * t2 * t2 * t2; grk = -0.75f * t2 * t2; }
          kacc[0].add(wab * pmf);
          kacc[1].add((-q * grk - 3.0f * wab) * pmf);
          if (GRAV) kacc[2].add(dphidh_f(q2, q) * pmf);
          ++nn;
          if (want_hash) hh += mix64((unsigned long long)perm[j] + 1ull);
          if constexpr (MHD) {
            const float r1g = grk / (rij + 1.0e-30f);
            const float rux = dx * r1g * pmf, ruy = dy * r1g * pmf, ruz = dz * r1g * pmf;
            const float4 bj = bjf[j];
            const float dBx = bi.x - bj.x, dBy = bi.y - bj.y, dBz = bi.z - bj.z;
            kacc[3].add(dBx * rux + dBy * ruy + dBz * ruz);
            kacc[4].add(dBx * rux); kacc[5].add(dBx * ruy); kacc[6].add(dBx * ruz);
            kacc[7].add(dBy * rux); kacc[8].add(dBy * ruy); kacc[9].add(dBy * ruz);
            kacc[10].add(dBz * rux); kacc[11].add(dBz * ruy); kacc[12].add(dBz * ruz);
          }
        }
      }
    } else {
      const double xi = tx[i], yi = ty[i], zi = tz[i];
      for (int m = ql.m0; m < ql.c; m += ql.step) {
        // separation and r^2 (6 FP64 instructions), r (5), the kernel sums (7).
        // acc[0] = sum u s, acc[1] = sum w^2, acc[2] = sum s (combined after the
        // loop), acc[PHI] the softening sum
        const int j = qj[m];
        double dx, dy, dz;
        separation_fp64(p, xi, yi, zi, j, qc[m], tx, ty, tz, dx, dy, dz);
        const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
        const double y = rsqrt_seed(r2), t = r2 * y;
        const double e = fma(-t, y, 1.0), pe = fma(0.375, e, 0.5) * e;
        const double u = fma(-fma(t, pe, t), hi1, 2.0);
        // the reference's test where the sign of u does not decide it
        bool in = u_inside(u);
        if (u_near_edge(u)) in = inside_exact(dx, dy, dz, hi1);
        if (in) {
          const double w = kern_w(u), u2 = u * u, s = fma(-w, w, u2);
          acc[0] = fma(u, s, acc[0]);
          acc[1] = fma(w, w, acc[1]);
          acc[2] += s;
          if (GRAV) {
            // get_kernel_grav1 (kernel_cubic.f90:78-99): u^4 (1/2 - u/5) - w^4 (1 - 2w/5) / 16
            const double w2 = w * w;
            acc[PHI] = fma(u2 * u2, fma(-0.2, u, 0.5), acc[PHI]);
            acc[PHI] = fma(w2 * w2, fma(0.025, w, -0.0625), acc[PHI]);
          }
          ++nn;
          if (want_hash) hh += mix64((unsigned long long)perm[j] + 1ull);
          if constexpr (MHD) {  // dens.F90:745-829 (getdB): dW/dq / r = -3/4 s / r
            const double r1g = -0.75 * s * fma(y, pe, y);
            const double rux = dx * r1g, ruy = dy * r1g, ruz = dz * r1g;
            const double *bj = bj64 + 4 * (size_t)j;
            const double dBx = bxi - bj[0], dBy = byi - bj[1], dBz = bzi - bj[2];
            accb[0] = fma(dBx, rux, fma(dBy, ruy, fma(dBz, ruz, accb[0])));
            accb[2] = fma(dBx, ruy, accb[2]); accb[3] = fma(dBx, ruz, accb[3]);
            accb[4] = fma(dBy, rux, accb[4]); accb[6] = fma(dBy, ruz, accb[6]);
            accb[7] = fma(dBz, rux, accb[7]); accb[8] = fma(dBz, ruy, accb[8]);
          }
        }
      }
    }
    flush_lanes<RW>(np, sm, sm.red, tot,
        [&](int k) -> double {
          if (k == NA) return __longlong_as_double((long long)nn);
          if (k == NA + 1) return __longlong_as_double((long long)hh);
          if constexpr (MIXED) return kacc[k].value();
          else {
            if (k == 0) return 0.25 * pm * (acc[0] + acc[1]);
            if (k == 1) return 0.75 * pm * (2.0 * (acc[2] - acc[0]) - acc[1]);
            if (k == 2) return GRAV ? pm * acc[PHI] : 0.0;
            return MHD && k != 4 && k != 8 && k != 12 ? pm * accb[k == 3 ? 0 : k - 3] : 0.0;
          }
        },
        [](int k, double s, double v) -> double {
          if (k >= NA) return __longlong_as_double(__double_as_longlong(s) + __double_as_longlong(v));
          return dadd(s, v);
        });
  }
  for (int r = 0; r < NR; ++r) {
    const int idx = lane + 32 * r;
    if (idx < RW * np) {
      const int k = idx / np;
      const int slot = k < NA ? k : (k == NA ? DSLOT_NN : DSLOT_HASH);
      psum[slot * ps + sm.ipos[idx - k * np]] = tot[r];
    }
  }
}

// ------------------------------------------------------------------ velocity derivatives
// Sums for the Cullen & Dehnen switch (getdv, dens.F90:745-802): div v, the
// velocity and acceleration gradients and the R matrix, over each cell's
// final trial list with the h of its converged iteration (the reference
// stores the sums of that iteration, dens.F90:1630-1663), in one pass after
// the h-rho solve. Then, per particle, the exact-linear gradients
// (dens.F90:866-1101): div v, dvdx(9) and d(div v)/dt. vf holds the pass's
// velocities and accelerations (vx, vy, vz, ax, ay, az) in tree order, vff
// an FP32 copy (mixed form).
constexpr int NDV = 25;  // div v, dv_a/dx_b (9), da_a/dx_b (9), R (6)

__global__ void k_dv_gather(int n, const int *perm, const double *vel, const double *fxyzu, double *vf, float *vff) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const size_t pid = (size_t)perm[j];
  double *o = vf + 6 * (size_t)j;
  for (int k = 0; k < 3; ++k) { o[k] = vel[4 * pid + k]; o[3 + k] = fxyzu[4 * pid + k]; }
  if (vff) for (int k = 0; k < 6; ++k) vff[6 * (size_t)j + k] = d2f_rn(o[k]);
}

// dens.F90:866-891, 899-989, 997-1055, 1086-1101 (reference rounding)
__device__ __forceinline__ void exactlinear3(double ax, double ay, double az, const double *rm, double ddenom,
                                             double &gx, double &gy, double &gz) {
  gx = dmul(dadd(dadd(dmul(ax, rm[0]), dmul(ay, rm[1])), dmul(az, rm[2])), ddenom);
  gy = dmul(dadd(dadd(dmul(ax, rm[1]), dmul(ay, rm[3])), dmul(az, rm[4])), ddenom);
  gz = dmul(dadd(dadd(dmul(ax, rm[2]), dmul(ay, rm[4])), dmul(az, rm[5])), ddenom);
}
__device__ void dv_from_sums(const double *rs, double term, double &divv, double &ddivvdt, double *dv) {
  // rs[0]: div v; rs[1..9]: dv_a/dx_b; rs[10..18]: da_a/dx_b; rs[19..24]: rxx rxy rxz ryy ryz rzz
  const double rxx = rs[19], rxy = rs[20], rxz = rs[21], ryy = rs[22], ryz = rs[23], rzz = rs[24];
  const double denom = dsub(dsub(dsub(dadd(dmul(dmul(rxx, ryy), rzz), dmul(dmul(dmul(2.0, rxy), rxz), ryz)),
                                      dmul(dmul(rxx, ryz), ryz)),
                                 dmul(dmul(ryy, rxz), rxz)),
                            dmul(dmul(rzz, rxy), rxy));
  double rm[6];
  rm[0] = dsub(dmul(ryy, rzz), dmul(ryz, ryz)); rm[1] = dsub(dmul(rxz, ryz), dmul(rzz, rxy));
  rm[2] = dsub(dmul(rxy, ryz), dmul(rxz, ryy)); rm[3] = dsub(dmul(rzz, rxx), dmul(rxz, rxz));
  rm[4] = dsub(dmul(rxy, rxz), dmul(rxx, ryz)); rm[5] = dsub(dmul(rxx, ryy), dmul(rxy, rxy));
  divv = dmul(-rs[0], term);
  double div_a;
  if (fabs(denom) > TINY_D) {
    const double ddenom = ddiv(1.0, denom);
    double g0, g1, g2, gax, gay, gaz;
    exactlinear3(rs[10], rs[11], rs[12], rm, ddenom, gax, g1, g2);
    exactlinear3(rs[13], rs[14], rs[15], rm, ddenom, g0, gay, g2);
    exactlinear3(rs[16], rs[17], rs[18], rm, ddenom, g0, g1, gaz);
    div_a = -dadd(dadd(gax, gay), gaz);
    for (int a = 0; a < 3; ++a) {
      double gx, gy, gz;
      exactlinear3(rs[1 + 3 * a], rs[2 + 3 * a], rs[3 + 3 * a], rm, ddenom, gx, gy, gz);
      dv[3 * a] = -gx; dv[3 * a + 1] = -gy; dv[3 * a + 2] = -gz;
    }
  } else {
    div_a = dmul(-term, dadd(dadd(rs[10], rs[14]), rs[18]));
    for (int q = 0; q < 9; ++q) dv[q] = dmul(-rs[1 + q], term);
  }
  const double sq = dadd(dadd(dmul(dv[0], dv[0]), dmul(dv[4], dv[4])), dmul(dv[8], dv[8]));
  const double cr = dadd(dadd(dmul(dv[1], dv[3]), dmul(dv[2], dv[6])), dmul(dv[5], dv[7]));
  ddivvdt = dsub(div_a, dadd(sq, dmul(2.0, cr)));
}

template <bool MIXED>
__global__ void __launch_bounds__(32 * MAX_WARPS, 4) k_density_dv(
    Params p, const Node *nodes, const int *leaves, int ncell, const LeafEntry *pool, const int *cell_off,
    const int *cell_nleaf, const double *tx, const double *ty, const double *tz, const float4 *txf, const float4 *txl,
    const double *hcur, const double *vf, const float *vff, double *dvsum, int64_t ps, double pf_hmin,
    const int *cells, const unsigned char *actf) {
  extern __shared__ __align__(16) unsigned char dsm[];
  const int w = threadIdx.x >> 5, lane = lane_id();
  const int a = blockIdx.x * (blockDim.x >> 5) + w;
  if (a >= ncell) return;
  const int cell = cells ? cells[a] : a;
  const Node nd = nodes[leaves[cell]];
  const int np_all = nd.count, s0 = nd.start;
  if (np_all < 1 || np_all > MAXCELL) return;  // reported by k_density_pairs
  int np = np_all;
  unsigned am = 0u;
  if (actf) am = cell_active_mask(actf, s0, np_all, np);
  if (np == 0) return;
  ListSmem &sm = reinterpret_cast<ListSmem *>(dsm)[w];
  const double pm = p.massoftype;
  const float pmf = d2f_rn(pm);
  double h1own = 0.0;  // lane il: 1/h of particle il
  if (lane < np) {
    const int ip = s0 + (actf ? cell_pos(am, lane) : lane);
    const double h = hcur[ip];
    h1own = rcp_fast(h);
    const float hf = d2f_rn(h);
    float4 x = txf[ip];
    x.w = MIXED || h > pf_hmin ? 4.0f * 1.001f * (hf * hf) : __int_as_float(0x7f800000);
    sm.xi[lane] = x;
    sm.ipos[lane] = ip;
  }
  const float4 cc = make_float4((float)nd.x, (float)nd.y, (float)nd.z, (float)nd.size);
  const int off = cell_off[cell], nleaf = cell_nleaf[cell], qstride = LQ / np;
  // totals per (sum, particle): FP32 in the mixed form (each lane's compensated
  // sum read out, the lanes added in FP32), FP64 in two halves otherwise
  using T = typename std::conditional<MIXED, float, double>::type;
  constexpr int RA = MIXED ? NDV : 13, RB = MIXED ? 1 : NDV - RA;
  constexpr int NRA = (RA * MAXCELL + 31) / 32, NRB = (RB * MAXCELL + 31) / 32;
  static_assert(32 * RA * sizeof(T) <= sizeof(sm.qj), "lane sums staged in the queues' space");
  T ta[NRA], tb[NRB];
  for (int r = 0; r < NRA; ++r) ta[r] = T(0.0);
  for (int r = 0; r < NRB; ++r) tb[r] = T(0.0);
  ListPos pos;
  __syncwarp();
  bool more = true;
  while (more) {
    int myc;
    more = SWEEP_END != sweep_list<false>(p, cc, np, pool, off, nleaf, txf, sm, qstride, pos, myc,
                                          [](float) { return 0.0f; });
    const QueueLanes ql = balance_queues(np, myc, sm);
    const int il = max(ql.il, 0), i = sm.ipos[il];
    const double hi1 = __shfl_sync(0xffffffffu, h1own, il);
    const int *qj = sm.qj + il * qstride;
    const unsigned char *qc = sm.qc + il * qstride;
    const auto sum = [](int, T s, T v) -> T { return s + v; };
    if constexpr (MIXED) {
      const Sep2 I = sep2_init(txf, txl, i);
      const float hi1f = d2f_rn(hi1), hi21f = d2f_rn(hi1 * hi1);
      float vi[6];
      for (int k = 0; k < 6; ++k) vi[k] = vff[6 * (size_t)i + k];
      Kahan kacc[NDV];
      for (int m = ql.m0; m < ql.c; m += ql.step) {
        const int j = qj[m];
        float dx, dy, dz, r2;
        separation_2f(p, I, j, qc[m] & 63, txf[j], txl[j], tx, ty, tz, dx, dy, dz, r2);
        if (r2 * hi21f < 4.0f) {
          const float rij = sqrt_nr(r2), q = rij * hi1f;
          const float grk = q < 1.0f ? q * (2.25f * q - 3.0f) : -0.75f * (q - 2.0f) * (q - 2.0f);
          const float r1g = grk / (rij + 1.0e-30f);
          const float rux = dx * r1g * pmf, ruy = dy * r1g * pmf, ruz = dz * r1g * pmf;
          const float2 *v2 = reinterpret_cast<const float2 *>(vff + 6 * (size_t)j);
          const float2 va = v2[0], vb = v2[1], vc = v2[2];
          const float dvx = vi[0] - va.x, dvy = vi[1] - va.y, dvz = vi[2] - vb.x;
          const float dax = vi[3] - vb.y, day = vi[4] - vc.x, daz = vi[5] - vc.y;
          kacc[0].add(dvx * rux + dvy * ruy + dvz * ruz);
          kacc[1].add(dvx * rux); kacc[2].add(dvx * ruy); kacc[3].add(dvx * ruz);
          kacc[4].add(dvy * rux); kacc[5].add(dvy * ruy); kacc[6].add(dvy * ruz);
          kacc[7].add(dvz * rux); kacc[8].add(dvz * ruy); kacc[9].add(dvz * ruz);
          kacc[10].add(dax * rux); kacc[11].add(dax * ruy); kacc[12].add(dax * ruz);
          kacc[13].add(day * rux); kacc[14].add(day * ruy); kacc[15].add(day * ruz);
          kacc[16].add(daz * rux); kacc[17].add(daz * ruy); kacc[18].add(daz * ruz);
          kacc[19].add(-dx * rux); kacc[20].add(-dx * ruy); kacc[21].add(-dx * ruz);
          kacc[22].add(-dy * ruy); kacc[23].add(-dy * ruz); kacc[24].add(-dz * ruz);
        }
      }
      flush_lanes<RA>(np, sm, reinterpret_cast<float *>(sm.qj), ta,
                      [&](int k) -> float { return __fsub_rn(kacc[k].s, kacc[k].c); }, sum);
    } else {
      const double xi = tx[i], yi = ty[i], zi = tz[i];
      const double *vfi = vf + 6 * (size_t)i;
      double acc[NDV];
      for (int k = 0; k < NDV; ++k) acc[k] = 0.0;
      for (int m = ql.m0; m < ql.c; m += ql.step) {
        const int j = qj[m];
        double dx, dy, dz;
        separation_fp64(p, xi, yi, zi, j, qc[m], tx, ty, tz, dx, dy, dz);
        const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
        const double y = rsqrt_seed(r2), t = r2 * y;
        const double e = fma(-t, y, 1.0), pe = fma(0.375, e, 0.5) * e;
        const double u = fma(-fma(t, pe, t), hi1, 2.0);
        bool in = u_inside(u);
        if (u_near_edge(u)) in = inside_exact(dx, dy, dz, hi1);
        if (in) {
          const double w = kern_w(u), s = fma(-w, w, u * u);
          const double r1g = -0.75 * pm * s * fma(y, pe, y);
          const double ru[3] = {dx * r1g, dy * r1g, dz * r1g};
          const double *vj = vf + 6 * (size_t)j;
          double d[6];
#pragma unroll
          for (int k = 0; k < 6; ++k) d[k] = vfi[k] - vj[k];
          acc[0] = fma(d[0], ru[0], fma(d[1], ru[1], fma(d[2], ru[2], acc[0])));
#pragma unroll
          for (int k = 0; k < 6; ++k)
            for (int b = 0; b < 3; ++b) acc[1 + 3 * k + b] = fma(d[k], ru[b], acc[1 + 3 * k + b]);
          acc[19] = fma(-dx, ru[0], acc[19]); acc[20] = fma(-dx, ru[1], acc[20]); acc[21] = fma(-dx, ru[2], acc[21]);
          acc[22] = fma(-dy, ru[1], acc[22]); acc[23] = fma(-dy, ru[2], acc[23]); acc[24] = fma(-dz, ru[2], acc[24]);
        }
      }
      flush_lanes<RA>(np, sm, sm.red, ta, [&](int k) -> double { return acc[k]; }, sum);
      flush_lanes<RB>(np, sm, sm.red, tb, [&](int k) -> double { return acc[RA + k]; }, sum);
    }
  }
  for (int r = 0; r < NRA; ++r) {
    const int idx = lane + 32 * r;
    if (idx < RA * np) { const int k = idx / np; dvsum[k * ps + sm.ipos[idx - k * np]] = (double)ta[r]; }
  }
  if constexpr (!MIXED) {
    for (int r = 0; r < NRB; ++r) {
      const int idx = lane + 32 * r;
      if (idx < RB * np) { const int k = idx / np; dvsum[(RA + k) * ps + sm.ipos[idx - k * np]] = tb[r]; }
    }
  }
}

// per particle: the exact-linear gradients from the sums (dense lanes: the
// FP64 pipe costs the same per warp instruction whatever its active lanes)
__global__ void k_dv_finish(int n, const double *dvsum, int64_t ps, const double *dvterm, const int *perm,
                            float *ddivvdt_c, float *dvdx_c, float *divcurlv, float *curl3, int diag,
                            const unsigned char *actf) {
  const int ip = blockIdx.x * blockDim.x + threadIdx.x;
  if (ip >= n || (actf && !actf[ip])) return;
  double rs[NDV];
  for (int k = 0; k < NDV; ++k) rs[k] = dvsum[k * ps + ip];
  double divv, ddivvdt, dv[9];
  dv_from_sums(rs, dvterm[ip], divv, ddivvdt, dv);
  // caller order: with individual timesteps inactive particles keep theirs
  // across tree builds
  const size_t pid = (size_t)perm[ip];
  ddivvdt_c[pid] = (float)ddivvdt;
  for (int q = 0; q < 9; ++q) dvdx_c[9 * pid + q] = (float)dv[q];
  if (diag) divcurlv[pid] = (float)divv;
  if (curl3) {  // curl v (dens.F90:919-923): sums 1..9 are dv_a r_b (a, b = x, y, z)
    const double t = dvterm[ip];
    curl3[3 * pid] = (float)(-(rs[8] - rs[6]) * t);
    curl3[3 * pid + 1] = (float)(-(rs[3] - rs[7]) * t);
    curl3[3 * pid + 2] = (float)(-(rs[4] - rs[2]) * t);
  }
}

// Newton-Raphson update of one particle from its sums (finish_rhosum
// dens.F90:1486-1500, finish_cell dens.F90:1425-1462). FP64 throughout, without
// its divisions: 1/h by rcp_fast, rho(h) = m (hfact/h)^3, dh/drho = -h^4 /
// (3 m hfact^3), the convergence test multiplied out. The FP64 pipe bounds the
// finish; per pass over 2M particles 0.97 -> 0.45 ms. The results are as close
// to the exact values as with the reference's divisions and pow, though not
// the same bits (400k updates, h from 0.003 to 0.6, largest and rms error in
// 2^-53: rho 5.5 and 1.54 here, 5.8 and 1.51 there; 1/Omega 6.4 and 0.92, 6.6 and
// 0.94; the final h 5.3 and 1.28, 6.1 and 2.07; the next h 2.8 and 0.64, 4.7 and
// 0.89), so a particle whose update falls on the edge of tolh to a few 2^-53 may
// stop one iteration apart from the reference.
struct DensNR {
  double rhoi, dhdrhoi, omega1, hmine;  // omega1 = 1/Omega
  bool conv;
};
__device__ __forceinline__ DensNR dens_nr(const Params &p, double r0, double r1, double hme, double h_old) {
  const double pm = p.massoftype;
  DensNR o;
  const double h1 = rcp_fast(hme), h21 = h1 * h1, ch21 = CNORMK * h21;
  o.rhoi = (r0 + pm) * (ch21 * h1);
  const double gradhi = fma(-3.0, pm, r1) * (ch21 * h21);
  const double h2 = hme * hme, mh3 = pm * (p.hfact * p.hfact * p.hfact);
  o.dhdrhoi = -(h2 * h2) * p.dhdrho1;
  const double omegai = fma(-o.dhdrhoi, gradhi, 1.0);
  const double func = fma(mh3, h21 * h1, -o.rhoi);  // rho(h) - rho
  o.omega1 = rcp_fast(omegai);
  const double dfdh1 = o.dhdrhoi * (omegai > TINY_D ? o.omega1 : rcp_fast(fabs(omegai + EPS_D)));
  double hnew = fma(-func, dfdh1, hme);
  if (hnew > 1.2 * hme) hnew = 1.2 * hme;
  else if (hnew < 0.8 * hme) hnew = 0.8 * hme;
  o.conv = fabs(hnew - hme) < p.tolh * h_old && omegai > 0.0 && hme > 0.0;
  o.hmine = o.conv ? hme : hnew;
  return o;
}

// finish_cell + compute_hmax (dens.F90:1275-1289) + the redo decision and,
// for converged cells, store_results (dens.F90:1561-1677). A cell takes a
// 16-lane segment of a warp for its decisions: lane q holds its particle q, the
// cell-wide convergence test and hmax are segment shuffles, and lane 0 acts for
// the cell. The particles' FP64 work, which bounds the kernel, is done between
// by threads packed over the block's particles: in the segments half of the
// lanes would be idle and an FP64 instruction takes as long for one lane as
// for 32 (885k particles, the last pass 220 -> 119 us, passes that mostly raise
// hmax 220 -> 183). Global maxima and statistics are reduced per block before one atomic
// each (a per-particle atomic on rhomax would serialise 2M updates on one
// address).
constexpr int FIN_SEG = 16;  // lanes per cell, >= MAXCELL
constexpr int FIN_THREADS = 256;
static_assert(MAXCELL <= FIN_SEG, "a finish segment holds a whole cell");

__global__ void __launch_bounds__(FIN_THREADS) k_density_finish(
    Params p, int icall, const Node *nodes, Node *nodes_w, const int *leaves, const int *act, int nact,
    const double *psum, int64_t ps, const int *cell_ntrial, const int *perm, double *hcur, const double *hold,
    double *cell_hmax, int *cell_nits, int *need_walk, int *next_act, int *nnext, DensOut out, NodeF *nodesf,
    const unsigned char *actf, int *err) {
  __shared__ unsigned long long bst[8];  // stats 0..6, rhomax bits
  constexpr int CELLS = FIN_THREADS / FIN_SEG;
  __shared__ double pnh[FIN_THREADS];    // per packed particle: new h, tree position, cell, converged
  __shared__ int pi[FIN_THREADS];
  __shared__ unsigned char pc[FIN_THREADS], pconv[FIN_THREADS];
  __shared__ int cnp[CELLS], cnits[CELLS], ctry[CELLS];  // per cell; iterations 0: not converged
  if (threadIdx.x < 8) bst[threadIdx.x] = 0ull;
  const unsigned FULL = 0xffffffffu;
  const int lane = lane_id(), q = lane & (FIN_SEG - 1), seg = threadIdx.x / FIN_SEG;
  const long long a = ((long long)blockIdx.x * FIN_THREADS + threadIdx.x) / FIN_SEG;
  bool cell_ok = a < nact;
  int cell = 0, leaf = 0, np = 0, s0 = 0;
  if (cell_ok) {
    cell = act[a];
    leaf = leaves[cell];
    np = nodes[leaf].count;
    s0 = nodes[leaf].start;
    cell_ok = np >= 1 && np <= MAXCELL;  // else reported by k_density_pairs
  }
  // the cell's active particles (individual timesteps): this segment's bits of the ballot
  const unsigned bal = __ballot_sync(FULL, cell_ok && q < np && (!actf || actf[s0 + q]));
  const unsigned segm = (bal >> (lane & ~(FIN_SEG - 1))) & ((1u << FIN_SEG) - 1u);
  np = __popc(segm);
  const bool mine = cell_ok && q < np;
  const size_t ip = (size_t)(s0 + (mine ? (int)__fns(segm, 0, q + 1) : q));
  const double pm = p.massoftype;
  if (q == 0) { cnp[seg] = cell_ok ? np : 0; cnits[seg] = 0; }
  __syncthreads();
  int first_p = 0, total = 0;
  for (int k = 0; k < CELLS; ++k) {
    first_p += k < seg ? cnp[k] : 0;
    total += cnp[k];
  }
  if (mine) { pi[first_p + q] = (int)ip; pc[first_p + q] = (unsigned char)seg; }
  __syncthreads();
  const bool packed = (int)threadIdx.x < total;
  const size_t jp = packed ? (size_t)pi[threadIdx.x] : 0;
  DensNR o{};
  if (packed) {
    o = dens_nr(p, psum[jp], psum[ps + jp], hcur[jp], hold[jp]);
    pnh[threadIdx.x] = o.hmine;
    pconv[threadIdx.x] = o.conv ? 1 : 0;
  }
  __syncthreads();
  int conv = !mine || pconv[first_p + q] ? 1 : 0;
  const double hmine = mine ? pnh[first_p + q] : 0.0;
  double hm = hmine;
  for (int m = 1; m < FIN_SEG; m <<= 1) {
    conv &= __shfl_xor_sync(FULL, conv, m);
    hm = fmax_pos(hm, __shfl_xor_sync(FULL, hm, m));
  }
  if (icall == 0) conv = 1;
  const double hmax_new = dmul(1.01, hm);
  const int nits = cell_ok ? cell_nits[cell] + 1 : 0;
  const bool lead = cell_ok && q == 0;
  bool append = false, redo = false;
  if (cell_ok && !conv) {
    if (nits >= MAXDENSITS) {
      if (lead) set_error(err, PH_ERR_DENS_NOCONV);
    } else {
      if (mine) hcur[ip] = hmine;
      if (lead) {
        redo = hmax_new > cell_hmax[cell];
        cell_nits[cell] = nits;
        cell_hmax[cell] = hmax_new;
        if (redo) {
          // set_hmaxcell neigh_kdtree.f90:115-131
          nodes_w[leaf].hmax = hmax_new;
          const float hf = (float)hmax_new;
          nodesf[leaf].hmax = hf;
          int pa = nodes[leaf].parent;
          // an ancestor that holds as much already was, or is being, raised
          // with all of its own ancestors: the climb ends there. (Climbing to
          // the root each time, the growing cells queued for its one address:
          // 885k particles, a pass 589 -> 223 us.)
          while (pa >= 0 && *(volatile double *)&nodes_w[pa].hmax < hmax_new) {
            atomic_max_pos(&nodes_w[pa].hmax, hmax_new);
            atomicMax(reinterpret_cast<int *>(&nodesf[pa].hmax), __float_as_int(hf));
            pa = nodes[pa].parent;
          }
        }
        need_walk[cell] = redo ? 1 : 0;
        append = true;
      }
    }
  }
  // cells for the next pass: one atomic per warp
  const unsigned ba = __ballot_sync(FULL, append);
  if (ba) {
    const int first = __ffs(ba) - 1;
    int base = 0;
    if (lane == first) base = atomicAdd(nnext, __popc(ba));
    base = __shfl_sync(FULL, base, first);
    if (append) next_act[base + __popc(ba & ((1u << lane) - 1))] = cell;
  }
  unsigned long long sv[5] = {0ull, 0ull, 0ull, 0ull, 0ull}, mx[2] = {0ull, 0ull};
  double rhoi_max = 0.0;
  if (lead && conv) {
    cell_hmax[cell] = hmax_new; cell_nits[cell] = nits; need_walk[cell] = 0;
    cnits[seg] = nits;
    ctry[seg] = cell_ntrial[cell];
  }
  __syncthreads();
  if (packed && cnits[pc[threadIdx.x]] > 0) {
    const size_t ip = jp;
    const int nits = cnits[pc[threadIdx.x]], ntry = ctry[pc[threadIdx.x]];
    const double hme = hcur[ip];
    if (hme < 0.0) set_error(err, PH_ERR_NEG_H);
    if (hme >= 0.0) {
      const int pid = perm[ip];
      const double grad = o.omega1;
      const double hfin = p.hfact * cbrt_fast(pm * rcp_fast(o.rhoi));  // hrho (part.F90:845-850)
      out.xyzh[4 * (size_t)pid + 3] = hfin;
      out.th[ip] = hfin;
      if (hfin < 0.0) set_error(err, PH_ERR_NEG_H);
      const float gradf = (float)grad;
      out.gradh64[ip] = grad;
      float gsf = 0.0f;
      if (p.gravity) {
        const double h1 = rcp_fast(hme);
        const double gs = fma(DPHIDH0, pm, psum[2 * ps + ip]) * (h1 * h1) * o.dhdrhoi;
        gsf = (float)gs;
        out.gsoft64[ip] = gs;
      }
      out.gradh_t[2 * ip] = gradf;
      out.gradh_t[2 * ip + 1] = gsf;
      if (out.diag || p.ind) {  // individual timesteps: the force reads gradh in caller order
        out.gradh[2 * (size_t)pid] = gradf;
        if (p.gravity || p.ind) out.gradh[2 * (size_t)pid + 1] = gsf;
      }
      rhoi_max = o.rhoi;
      double term = 0.0;
      if (out.dvterm || out.diag) {
        const double h1 = ddiv(1.0, hme), h21 = dmul(h1, h1), h41 = dmul(h21, h21);
        term = dmul(dmul(dmul(CNORMK, (double)gradf), ddiv(1.0, o.rhoi)), h41);
      }
      if (out.dvterm) out.dvterm[ip] = term;
      // getdv is .false. under CONST_AV (dens.F90:1638-1640)
      if (out.diag) out.divcurlv[pid] = -(float)(0.0 * term);
      if (p.mhd && out.diag) {
        const double r3 = psum[3 * ps + ip], r5 = psum[5 * ps + ip], r6 = psum[6 * ps + ip],
                     r7 = psum[7 * ps + ip], r9 = psum[9 * ps + ip], r10 = psum[10 * ps + ip],
                     r11 = psum[11 * ps + ip];
        float *db = out.divcurlB + 4 * (size_t)pid;
        db[0] = (float)(dmul(-r3, term));
        db[1] = (float)(dmul(-dsub(r11, r9), term));
        db[2] = (float)(dmul(-dsub(r6, r10), term));
        db[3] = (float)(dmul(-dsub(r7, r5), term));
      }
      const int nni = (int)__double_as_longlong(psum[DSLOT_NN * ps + ip]) + 1;  // + self
      if (out.diag) {
        out.nneigh[pid] = nni;
        out.nhash[pid] = (uint64_t)__double_as_longlong(psum[DSLOT_HASH * ps + ip]);
      }
      // nneightry, nneighact, ncalc, np summed; maxneightry, maxneighact
      sv[0] = (unsigned long long)ntry; sv[1] = (unsigned long long)nni; sv[2] = (unsigned long long)nits;
      sv[3] = 1ull;
      mx[0] = (unsigned long long)ntry; mx[1] = (unsigned long long)nni;
    }
  }
  sv[4] = (lead && redo) ? 1ull : 0ull;
  for (int m = 16; m > 0; m >>= 1) {
    for (int k = 0; k < 5; ++k) sv[k] += __shfl_xor_sync(FULL, sv[k], m);
    for (int k = 0; k < 2; ++k) mx[k] = max(mx[k], __shfl_xor_sync(FULL, mx[k], m));
  }
  for (int m = 16; m > 0; m >>= 1) rhoi_max = fmax_pos(rhoi_max, __shfl_xor_sync(FULL, rhoi_max, m));
  if (lane == 0) {
    if (sv[3]) {
      atomicAdd(&bst[0], sv[0]); atomicAdd(&bst[1], sv[1]); atomicMax(&bst[2], mx[0]);
      atomicMax(&bst[3], mx[1]); atomicAdd(&bst[4], sv[2]); atomicAdd(&bst[5], sv[3]);
      atomicMax(&bst[7], (unsigned long long)__double_as_longlong(rhoi_max));
    }
    if (sv[4]) atomicAdd(&bst[6], sv[4]);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (bst[5]) {
      atomicAdd(&out.stats[0], bst[0]); atomicAdd(&out.stats[1], bst[1]); atomicMax(&out.stats[2], bst[2]);
      atomicMax(&out.stats[3], bst[3]); atomicAdd(&out.stats[4], bst[4]); atomicAdd(&out.stats[5], bst[5]);
      atomic_max_pos(out.rhomax, __longlong_as_double((long long)bst[7]));
    }
    if (bst[6]) atomicAdd(&out.stats[6], bst[6]);
  }
}

static inline int nblk(int64_t n, int b) { return (int)((n + b - 1) / b); }

// The low parts for the precision form's force and adjoint, where the density
// before them was the plain form's (else its gather has written them)
void low_words(ph_ctx *c) {
  if (c->have_low) return;
  const int nt = (int)c->ntree;
  k_low_words<<<nblk(nt, 256), 256, 0, c->stream>>>(nt, c->tx, c->ty, c->tz, c->txf, c->txl);
  count_launch(c, 1);
  c->have_low = true;
}

// densityiterate driver
int density(ph_ctx *c, int icall) {
  if (!c->have_tree || (c->dp.gravity && !c->tree_grav)) return PH_ERR_STATE;
  c->have_force_lists = false;  // the density walks reuse the list pool
  cudaStream_t st = c->stream;
  const int nt = (int)c->ntree, ncell = c->nleaves;
  const Params p = c->dp;
  k_dens_gather<<<nblk(nt, 256), 256, 0, st>>>(nt, c->perm, c->xyzh, c->tx, c->ty, c->tz, c->hcur, c->hold, c->txf,
                                              p.precision == PH_PREC_MIXED ? c->txl : nullptr);
  c->have_low = c->have_low || p.precision == PH_PREC_MIXED;
  k_dens_init_cells<<<nblk(ncell, 256), 256, 0, st>>>(ncell, c->leaves, c->nodes, c->cell_hmax, c->cell_nits, c->act_a);
  cudaMemsetAsync(c->stats, 0, 8 * sizeof(unsigned long long), st);
  cudaMemsetAsync(c->red, 0, 8 * sizeof(double), st);
  count_launch(c, 2);
  // h_j used by the divcurlB sums: the value at entry of the pass (race-free
  // form of the reference's fast_divcurlB read of xyzh(4,j), dens.F90:811)
  const double *hj_entry = c->hold;
  // the Bevol of the evaluation (Bpred in a step: derivs passes its Bevol
  // argument on to densityiterate, deriv.f90:135)
  const double *Bd = c->dens_B ? c->dens_B : c->Bevol;
  // the div B and curl B sums feed divcurlB only, which only a ph_density call
  // returns (ideal MHD forces do not read it): the evaluations of derivs and
  // the step take the density sums alone
  const bool dB = p.mhd && c->want_diag;
  if (dB) {
    k_dens_bprep<<<nblk(nt, 256), 256, 0, st>>>(p, nt, c->perm, Bd, hj_entry, c->jrec,
                                                p.precision == PH_PREC_MIXED ? c->bjf : nullptr);
    count_launch(c, 1);
  }
  int nact = ncell;
  const unsigned char *actf = p.ind ? c->actf_t : nullptr;
  if (p.ind) {  // individual timesteps: leaf cells holding an active particle only
    cudaMemcpyAsync(c->act_a, c->cell_act, sizeof(int) * (size_t)c->ncell_act, cudaMemcpyDeviceToDevice, st);
    nact = c->ncell_act;
  }
  int *act = c->act_a, *nxt = c->act_b;
  int *need = c->cell_state;  // redo flags
  fill_int(c, need, ncell, 1);
  cudaMemsetAsync(c->pool_top, 0, sizeof(unsigned long long), st);
  // dens.F90:202-203: velocity derivatives for the viscosity switch
  // velocity derivatives for the Cullen & Dehnen switch or curl v (dens.F90:202-203)
  const bool getdv = (p.nalpha >= 2 || p.curlv) && (icall <= 1 || icall == 3);
  DensOut out{c->xyzh, c->gradh, c->divcurlv, c->divcurlB, c->nneigh, c->nhash, c->th, c->gradh64, c->gsoft64,
              c->gradh_t,
              c->want_diag ? 1 : 0, getdv ? c->dvterm_t : nullptr, c->red + 2, c->stats};
  double pf_hmin = c->pf_hmin;
  const int dw = c->dens_warps, ww = c->walk_warps;
  const int smem = dw * (int)sizeof(ListSmem);
  if (!(c->attr_done & 1u)) {
    const int smax = MAX_WARPS * (int)sizeof(ListSmem);
    cudaFuncSetAttribute(k_density_pairs<true, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smax);
    cudaFuncSetAttribute(k_density_pairs<true, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smax);
    cudaFuncSetAttribute(k_density_pairs<true, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smax);
    cudaFuncSetAttribute(k_density_pairs<true, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smax);
    cudaFuncSetAttribute(k_density_pairs<false, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smax);
    cudaFuncSetAttribute(k_density_pairs<false, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smax);
    cudaFuncSetAttribute(k_density_pairs<false, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smax);
    cudaFuncSetAttribute(k_density_pairs<false, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smax);
    c->attr_done |= 1u;
  }
  for (int pass = 0; nact > 0; ++pass) {
    if (pass > MAXDENSITS + 2) return PH_ERR_DENS_NOCONV;
    for (int attempt = 0;; ++attempt) {
      cudaEventRecord(c->evk[4], st);
      launch_walk<false>(ww, nact, st,
          p, c->nodes, c->nodesf, c->top_nodes, c->leaves, act, nact, need, c->cell_hmax, c->pool, c->pool_cap, c->pool_top,
          c->cell_off, c->cell_nleaf, c->cell_ntrial, c->d_err);
      cudaEventRecord(c->evk[5], st);
      count_launch(c, 1);
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
      break;
    }
    cudaMemsetAsync(c->counters + 8, 0, sizeof(int), st);
    cudaEventRecord(c->evk[2], st);
#define PH_DENS(X, M, G)                                                                                         \
  k_density_pairs<X, M, G><<<nblk(nact, dw), 32 * dw, smem, st>>>(                                    \
      p, c->nodes, c->leaves, act, nact, c->pool, c->cell_off, c->cell_nleaf, c->cell_ntrial, c->perm, c->tx, c->ty,  \
      c->tz, c->txf, c->txl, c->hcur, Bd, c->jrec, c->bjf, c->psum, c->cap, c->stats, pf_hmin, actf,             \
      c->want_diag ? 1 : 0, c->d_err)
    if (c->keep_order) {
      ro_density(c, act, nact);
    } else if (p.precision == PH_PREC_MIXED) {
      if (dB) { if (p.gravity) PH_DENS(true, true, true); else PH_DENS(true, true, false); }
      else { if (p.gravity) PH_DENS(true, false, true); else PH_DENS(true, false, false); }
    } else {
      if (dB) { if (p.gravity) PH_DENS(false, true, true); else PH_DENS(false, true, false); }
      else { if (p.gravity) PH_DENS(false, false, true); else PH_DENS(false, false, false); }
    }
#undef PH_DENS
    k_density_finish<<<nblk((int64_t)nact * FIN_SEG, FIN_THREADS), FIN_THREADS, 0, st>>>(p, icall, c->nodes, c->nodes, c->leaves, act, nact, c->psum,
                                                      c->cap, c->cell_ntrial, c->perm, c->hcur, c->hold,
                                                      c->cell_hmax, c->cell_nits, need, nxt, c->counters + 8, out,
                                                      c->nodesf, actf, c->d_err);
    cudaEventRecord(c->evk[3], st);
    count_launch(c, 2);
    int hv[2];
    cudaMemcpyAsync(&hv[0], c->counters + 8, sizeof(int), cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(&hv[1], c->d_err, sizeof(int), cudaMemcpyDeviceToHost, st);
    cudaStreamSynchronize(st);
    add_elapsed(c, 5, c->evk[2], c->evk[3]);
    if (hv[1]) return hv[1];
    nact = hv[0];
    std::swap(act, nxt);
  }
  if (getdv) {  // velocity derivatives on the final lists (Cullen & Dehnen switch)
    const double *vel = c->dens_vel ? c->dens_vel : c->vxyzu;
    const bool mixed = p.precision == PH_PREC_MIXED;
    k_dv_gather<<<nblk(nt, 256), 256, 0, st>>>(nt, c->perm, vel, c->fxyzu, c->jrec, mixed ? c->jrecf : nullptr);
    if (!c->dvsum && alloc_dvsum(c) != 0) return PH_ERR_CUDA;
    const int dw = c->dens_warps;
    const int smem = dw * (int)sizeof(ListSmem);
    const int *dv_cells = p.ind ? c->cell_act : nullptr;
    const int ndv = p.ind ? c->ncell_act : ncell;
    if (mixed)
      k_density_dv<true><<<nblk(ndv, dw), 32 * dw, smem, st>>>(
          p, c->nodes, c->leaves, ndv, c->pool, c->cell_off, c->cell_nleaf, c->tx, c->ty, c->tz, c->txf, c->txl, c->hcur,
          c->jrec, c->jrecf, c->dvsum, c->cap, pf_hmin, dv_cells, actf);
    else
      k_density_dv<false><<<nblk(ndv, dw), 32 * dw, smem, st>>>(
          p, c->nodes, c->leaves, ndv, c->pool, c->cell_off, c->cell_nleaf, c->tx, c->ty, c->tz, c->txf, c->txl, c->hcur,
          c->jrec, nullptr, c->dvsum, c->cap, pf_hmin, dv_cells, actf);
    if (p.curlv && alloc_curlv(c) != 0) return PH_ERR_CUDA;
    k_dv_finish<<<nblk(nt, 256), 256, 0, st>>>(nt, c->dvsum, c->cap, c->dvterm_t, c->perm, c->ddivvdt_c, c->dvdx_c,
                                                c->divcurlv, p.curlv ? c->curl3 : nullptr, c->want_diag ? 1 : 0,
                                                actf);
    count_launch(c, 3);
  }
  if (check_launch(c) != cudaSuccess) return PH_ERR_CUDA;
  c->have_density = true;
  return 0;
}

}  // namespace ph
