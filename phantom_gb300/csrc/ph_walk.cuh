// Leaf-cell neighbour walk (K3): getneigh (kdtree.F90:1221-1347) with
// cache_neighbours (kdtree.F90:1175-1213), one warp per leaf cell.
//
// The warp expands up to 32 stack entries at a time. The reference walk pops
// the right child first, so its trial list is the opened leaves in decreasing
// order of their first particle; each emitted leaf is written to the slot of
// its rank in that order, which reproduces the reference trial list exactly
// (including which entries fall inside the 1000-entry position cache).
#pragma once
#include "ph_common.cuh"

namespace ph {

constexpr int WALK_STK = 512;
constexpr int WALK_EM = 1024;

// 8 KB per walking warp (28 warps per SM): an emitted leaf keeps its first
// particle and, in 16 bits, its count (at most MAXCELL) and offset code
struct WalkShared {
  int stk[WALK_STK];
  int start[WALK_EM];
  unsigned short cc[WALK_EM];
  __device__ __forceinline__ void put(int e, int first, int count, int code) {
    start[e] = first;
    cc[e] = (unsigned short)(count | (code << 5));
  }
  __device__ __forceinline__ int count(int e) const { return cc[e] & 31; }
};
static_assert(MAXCELL < 32, "a leaf's count in five bits");

// Writes the nem emitted leaves of a warp to pool[off ...] in the reference
// walk's order (descending first particle; first particles are distinct).
__device__ __forceinline__ void write_ranked(const LeafEntry *em, int nem, LeafEntry *__restrict__ pool,
                                             unsigned long long off) {
  for (int e = lane_id(); e < nem; e += 32) {
    const LeafEntry me = em[e];
    int rank = 0;
    for (int q = 0; q < nem; ++q) rank += (em[q].start > me.start) ? 1 : 0;
    pool[off + rank] = me;
  }
}
__device__ __forceinline__ void write_ranked(const WalkShared &sh, int nem, LeafEntry *__restrict__ pool,
                                             unsigned long long off) {
  for (int e = lane_id(); e < nem; e += 32) {
    const int me = sh.start[e];
    int rank = 0;
    for (int q = 0; q < nem; ++q) rank += sh.start[q] > me ? 1 : 0;
    LeafEntry le;
    le.start = me;
    le.cc = sh.count(e) | ((sh.cc[e] >> 5) << 8);
    pool[off + rank] = le;
  }
}

// ------------------------------------------------------------------ staging
// The trial list of a cell is a list of whole leaves. For the pair loops it is
// expanded, window by window, into a flat per-warp array in shared memory:
// the tree index of each trial particle, its periodic offset code and its FP32
// position with the offset applied (w = the caller's 4th component of txf).
// Entry k of window `base` is trial-list position n = base + k, which decides
// whether the reference would use its cached position (n < 1000).
constexpr int STAGE = 256;

template <int W>
struct StageN {
  float4 pos[W];
  int jidx[W];
  unsigned char code[W];
};
using Stage = StageN<STAGE>;

template <int W>
__device__ __forceinline__ int stage_window_n(const Params &p, const LeafEntry *__restrict__ pool, int off,
                                              int nleaf, int ntrial, int base, const float4 *__restrict__ txf,
                                              StageN<W> &st) {
  const int lane = lane_id();
  const int end = min(ntrial, base + W);
  int acc = 0;
  for (int e0 = 0; e0 < nleaf && acc < end; e0 += 32) {
    const int e = e0 + lane;
    LeafEntry le{0, 0};
    if (e < nleaf) le = pool[off + e];
    const int jc = le.cc & 255;
    int x = jc;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    const int n_first = acc + x - jc;
    if (jc > 0 && n_first < end && n_first + jc > base) {
      const int code = le.cc >> 8;
      const float ox = offset_of_f(code, 0, p.dxboundf), oy = offset_of_f(code, 1, p.dyboundf),
                  oz = offset_of_f(code, 2, p.dzboundf);
      for (int t = 0; t < jc; ++t) {
        const int n = n_first + t;
        if (n >= base && n < end) {
          const int k = n - base;
          float4 q = txf[le.start + t];
          q.x += ox; q.y += oy; q.z += oz;
          st.pos[k] = q;
          st.jidx[k] = le.start + t;
          st.code[k] = (unsigned char)code;
        }
      }
    }
    acc += __shfl_sync(0xffffffffu, x, 31);
  }
  __syncwarp();
  return end - base;
}

__device__ __forceinline__ int stage_window(const Params &p, const LeafEntry *__restrict__ pool, int off,
                                            int nleaf, int ntrial, int base, const float4 *__restrict__ txf,
                                            Stage &st) {
  return stage_window_n<STAGE>(p, pool, off, nleaf, ntrial, base, txf, st);
}

// ------------------------------------------------------------------ mixed-form separation
// Pair separation of the mixed form: formed in FP64 from the FP64 positions,
// rounded to FP32. The periodic image is the staged leaf's offset (code) plus
// the wrap decided on the FP32 separation of the staged copy (dxf, dyf, dzf);
// per axis the two add up to a shift of m box lengths, |m| <= 2. Unshifted
// pairs (nearly all) cost three FP64 subtractions. Shifted ones take their
// own branch: an FP64 warp instruction holds the FP64 pipe for the same time
// whether or not its lanes are predicated on, so the shift must not be issued
// for warps that have none.
__device__ __forceinline__ int image_shift(int code, int axis, bool wrap, float d) {
  const int c = (code >> (2 * axis)) & 3;
  return (c == 1 ? 1 : (c == 2 ? -1 : 0)) + (wrap ? (d > 0.0f ? 1 : -1) : 0);
}
__device__ __forceinline__ double shift_len(int m, double L) {
  return m == 0 ? 0.0 : (m == 1 ? L : (m == -1 ? -L : (double)m * L));
}
__device__ __forceinline__ void separation_mixed(const Params &p, double xi, double yi, double zi, double xj,
                                                 double yj, double zj, int code, float dxf, float dyf, float dzf,
                                                 float &dx, float &dy, float &dz) {
  bool wx = false, wy = false, wz = false;
  if (p.periodic) {
    wx = fabsf(dxf) > 0.5f * p.dxboundf; wy = fabsf(dyf) > 0.5f * p.dyboundf; wz = fabsf(dzf) > 0.5f * p.dzboundf;
  }
  const int mx = image_shift(code, 0, wx, dxf), my = image_shift(code, 1, wy, dyf),
            mz = image_shift(code, 2, wz, dzf);
  if ((mx | my | mz) == 0) {
    dx = d2f_rn(xi - xj); dy = d2f_rn(yi - yj); dz = d2f_rn(zi - zj);
  } else {
    dx = d2f_rn((xi - xj) - shift_len(mx, p.dxbound));
    dy = d2f_rn((yi - yj) - shift_len(my, p.dybound));
    dz = d2f_rn((zi - zj) - shift_len(mz, p.dzbound));
  }
}

// ------------------------------------------------------------------ FP64 separation
// Pair separation with the reference's rounding: cached positions x_j + offset
// for the first 1000 trial entries (dens.F90:660-669, force.F90:1258-1269),
// else x_i - x_j and the wrap into the half box. Inside the box (nearly every
// pair) that is three FP64 subtractions: the wrap test compares bit patterns,
// and the offset and shift adds sit in branches of their own, since an FP64
// instruction holds the pipe for a whole warp when one lane needs it.
// code: the leaf's periodic offset, with QC_CACHED where the reference uses its
// cached position
constexpr int QC_CACHED = 64;
__device__ __forceinline__ void separation_fp64(const Params &p, double xi, double yi, double zi, int j, int code,
                                                const double *tx, const double *ty, const double *tz,
                                                double &dx, double &dy, double &dz) {
  double xj = tx[j], yj = ty[j], zj = tz[j];
  if (code > QC_CACHED) {
    xj = dadd(xj, offset_of(code, 0, p.dxbound)); yj = dadd(yj, offset_of(code, 1, p.dybound));
    zj = dadd(zj, offset_of(code, 2, p.dzbound));
  }
  dx = dsub(xi, xj); dy = dsub(yi, yj); dz = dsub(zi, zj);
  if (p.periodic && (abs_gt(dx, p.hdlx) || abs_gt(dy, p.hdly) || abs_gt(dz, p.hdlz))) {
    dx = wrap(dx, p.dxbound, p.hdlx, true); dy = wrap(dy, p.dybound, p.hdly, true);
    dz = wrap(dz, p.dzbound, p.hdlz, true);
  }
}

// the reference's neighbour test r^2 h^-2 < 4 with its rounding. Out of line:
// inlined, the compiler evaluates its six FP64 instructions for every pair
// instead of branching around them
static __device__ __noinline__ bool inside_exact(double dx, double dy, double dz, double h1) {
  return dmul(r2_exact(dx, dy, dz), dmul(h1, h1)) < RADKERN2;
}

// The same separation without the FP64 pipe: each coordinate is kept as two
// floats, x = hi + lo to 2^-49 of |x| (txf, txl), and hi_i - hi_j with its exact
// rounding error (Knuth's two-sum) plus lo_i - lo_j gives x_i - x_j rounded to
// FP32. That costs eight FP32 additions per axis, where the FP64 subtraction
// held the FP64 pipe (45-49 % of the mixed pair kernels' time) and its rounding
// to FP32 took ten integer instructions. What the two floats leave out is about
// 2^-48 |x|. Against the exact separation, over 2M pairs per octave of r/|x|, the
// error is that of the rounded FP64 subtraction down to r = 2^-15 |x| (largest
// 5.94e-8 r both, rms 2.537e-8 r, equal to five digits; at 2^-19 it is 6.04e-8
// against 5.92e-8), so closer pairs, and pairs across a periodic image, take the
// FP64 separation (out of line). Neighbour pairs of the benchmark's sets lie above
// 2^-11 |x|.
struct Sep2 {
  float4 h, l;   // particle i
  float guard;   // smallest r^2 the two floats serve
  int i;
};
__device__ __forceinline__ Sep2 sep2_init(const float4 *__restrict__ txf, const float4 *__restrict__ txl, int i) {
  Sep2 s;
  s.h = txf[i]; s.l = txl[i]; s.i = i;
  const float m = 3.0517578125e-05f * fmaxf(fmaxf(fabsf(s.h.x), fabsf(s.h.y)), fabsf(s.h.z));
  s.guard = m * m;
  return s;
}
__device__ __forceinline__ float diff2(float ah, float al, float bh, float bl) {
  const float s = __fsub_rn(ah, bh), t = __fsub_rn(s, ah);
  const float e = __fsub_rn(__fsub_rn(ah, __fsub_rn(s, t)), __fadd_rn(bh, t));
  return __fadd_rn(s, __fadd_rn(e, __fsub_rn(al, bl)));
}
// FP64 separation with the pair's periodic image (the leaf's offset code, then
// the wrap of what is left), rounded to FP32; u: the unshifted FP32 separation
static __device__ __noinline__ float3 separation_image(const double *tx, const double *ty, const double *tz, int i,
                                                       int j, int code, float ux, float uy, float uz, double Lx,
                                                       double Ly, double Lz) {
  const float fx = (float)Lx, fy = (float)Ly, fz = (float)Lz;
  ux -= offset_of_f(code, 0, fx); uy -= offset_of_f(code, 1, fy); uz -= offset_of_f(code, 2, fz);
  const int mx = image_shift(code, 0, fabsf(ux) > 0.5f * fx, ux), my = image_shift(code, 1, fabsf(uy) > 0.5f * fy, uy),
            mz = image_shift(code, 2, fabsf(uz) > 0.5f * fz, uz);
  return make_float3(d2f_rn((tx[i] - tx[j]) - shift_len(mx, Lx)), d2f_rn((ty[i] - ty[j]) - shift_len(my, Ly)),
                     d2f_rn((tz[i] - tz[j]) - shift_len(mz, Lz)));
}
__device__ __forceinline__ void separation_2f(const Params &p, const Sep2 &I, int j, int code, const float4 &jh,
                                              const float4 &jl, const double *tx, const double *ty, const double *tz,
                                              float &dx, float &dy, float &dz, float &r2) {
  dx = diff2(I.h.x, I.l.x, jh.x, jl.x);
  dy = diff2(I.h.y, I.l.y, jh.y, jl.y);
  dz = diff2(I.h.z, I.l.z, jh.z, jl.z);
  r2 = dx * dx + dy * dy + dz * dz;
  bool rare = r2 < I.guard;
  if (p.periodic)
    rare = rare || code != 0 || fabsf(dx) > 0.5f * p.dxboundf || fabsf(dy) > 0.5f * p.dyboundf ||
           fabsf(dz) > 0.5f * p.dzboundf;
  if (rare) {
    const bool per = p.periodic != 0;
    const double Lx = per ? p.dxbound : 1.0e300, Ly = per ? p.dybound : 1.0e300, Lz = per ? p.dzbound : 1.0e300;
    const float3 d = separation_image(tx, ty, tz, I.i, j, code, dx, dy, dz, Lx, Ly, Lz);
    dx = d.x; dy = d.y; dz = d.z;
    r2 = dx * dx + dy * dy + dz * dz;
  }
}

// ------------------------------------------------------------------ active particles of a cell
// With individual timesteps a cell's pair loops run over its active
// particles only (dens.F90:1293-1378, force.F90 start_cell skip inactive
// ones). The warp takes the ballot of the cell's activity flags (tree
// order; null when every particle is active): np becomes the active count
// and slot k of the cell maps to tree position s0 + cell_pos(m, k).
__device__ __forceinline__ unsigned cell_active_mask(const unsigned char *actf, int s0, int np_all, int &np) {
  const int lane = lane_id();
  const unsigned m = __ballot_sync(0xffffffffu, lane < np_all && (!actf || actf[s0 + lane]));
  np = __popc(m);
  return m;
}
__device__ __forceinline__ int cell_pos(unsigned m, int k) { return (int)__fns(m, 0, k + 1); }

// ------------------------------------------------------------------ pair queues
// Most staged trial entries fail the cheap distance test (about 1 in 8 is a
// neighbour), so a pair body run directly inside the test loop executes with
// a few lanes of the warp active. Instead, lane (il, stripe) tests entries
// stripe, stripe + S, ... of the window for particle il and appends the
// accepted window indices to il's queue, in window order; a queue that may
// overflow in the next round, and every queue at the end of the window, is
// drained by the S lanes of its particle (queue entry m by lane m % S). The
// bodies then run with nearly every lane active.
constexpr int QCAP = 64;

struct PairQ {
  unsigned short k[MAXCELL][QCAP];
};

// per-warp dynamic shared memory of the pair kernels
struct PairSmem {
  Stage st;
  PairQ q;
};

template <class Test, class Body>
__device__ __forceinline__ void queue_window(int cnt, int S, bool act, int il, int stripe, PairQ &q, Test &&test,
                                             Body &&body) {
  const unsigned FULL = 0xffffffffu;
  const int lane = lane_id();
  const unsigned gmask = !act ? 0u : (S >= 32 ? FULL : (((1u << S) - 1u) << (il * S)));
  const unsigned lt = (1u << lane) - 1u;
  const int nr = (cnt + S - 1) / S;
  int qn = 0;
  for (int r = 0; r < nr; ++r) {
    const int k = r * S + stripe;
    const bool ok = act && k < cnt && test(k);
    const unsigned b = __ballot_sync(FULL, ok);
    if (ok) q.k[il][qn + __popc(b & gmask & lt)] = (unsigned short)k;
    qn += __popc(b & gmask);
    // qn <= QCAP - S before this round's appends, so no queue overflows
    if (r == nr - 1 || (int)__reduce_max_sync(FULL, (unsigned)qn) > QCAP - S) {
      __syncwarp();
      for (int m = stripe; act && m < qn; m += S) body((int)q.k[il][m]);
      __syncwarp();
      qn = 0;
    }
  }
}

// ------------------------------------------------------------------ list sweep
// Trial list -> per-particle pair queues -> balanced drain, by one warp.
//
// The sweep: batches of BATCH leaf entries are expanded into shared memory (tree
// index and offset code per trial particle); each lane then takes one trial
// particle (its FP32 position in registers, loaded one chunk ahead) and the
// warp tests it against the cell's particles one after the other, their FP32
// positions broadcast from shared memory. One ballot per particle gives the
// accepted lanes their queue slots. Per 32 tests that is about 17 instructions,
// where testing with a lane per (particle, stripe) took about 45 (a shared
// position load, the periodic wrap, two ballots and queue bounds each).
// Whether a chunk needs the periodic wrap at all is decided once per chunk.
//
// The drain: queues are emptied when one is nearly full or the list ends,
// normally once per cell. The lanes are dealt out so that the particle with
// most pairs per lane has as few as possible (balance_queues); with a fixed
// 32/np lanes per particle the longest queue set the pace and a fifth (density)
// to two fifths (symmetric force) of the lane slots were idle.
constexpr int BATCH = 24;             // leaf entries of a batch
constexpr int LW = BATCH * MAXCELL;   // trial particles of a batch
constexpr int LQ = 1024;              // queue slots per warp, dealt out evenly to the cell's particles

struct __align__(16) ListBase {
  float4 xi[MAXCELL];     // cell particles: x, y, z, acceptance r^2
  int ipos[MAXCELL];      // their tree positions
  int j[LW];              // the batch
  unsigned char code[LW];
  unsigned char own[32];  // drain: lane -> particle
  unsigned char first[MAXCELL], lanes[MAXCELL];
};
struct ListSmem : ListBase {
  union {
    int qj[LQ];           // accepted trial particle
    double red[LQ / 2];   // lane sums of the flush
  };
  unsigned char qc[LQ];   // its offset code, QC_CACHED where the reference uses its cached position
};
// queue of batch indices (code[] then holds the flagged codes)
struct ListSmemK : ListBase {
  union {
    unsigned short qj[LQ];
    double red[32 * 12];
  };
};

struct ListPos {  // the sweep's place in the list
  int e0 = 0, nbase = 0, cnt = 0, k0 = 0;
  bool open = false;
};
enum { SWEEP_END = 0, SWEEP_FULL = 1, SWEEP_BATCH = 2 };

// expand the BATCH leaf entries from e0 on; returns the number of trial particles
__device__ __forceinline__ int expand_batch(const LeafEntry *__restrict__ pool, int off, int nleaf, int e0,
                                            ListBase &sm) {
  const int e = e0 + lane_id();
  LeafEntry le{0, 0};
  if (lane_id() < BATCH && e < nleaf) le = pool[off + e];
  const int jc = le.cc & 255, code = le.cc >> 8;
  int x = jc;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane_id() >= o) x += y;
  }
  const int k = x - jc;
  for (int t = 0; t < jc; ++t) { sm.j[k + t] = le.start + t; sm.code[k + t] = (unsigned char)code; }
  return __shfl_sync(0xffffffffu, x, 31);
}

// Sweep on from `pos` until the list ends (SWEEP_END) or a queue is nearly full
// (SWEEP_FULL: drain, then call again). sm.xi / sm.ipos describe the np cell
// particles; ew(w) is the acceptance r^2 of a trial particle with txf.w = w;
// myc receives lane il's count for particle il. With AFTER only trial
// particles after the cell particle in tree order are accepted, the queue
// holds batch indices, and the sweep also returns at the end of every batch
// (SWEEP_BATCH: drain; trial particles [nbase, nbase + cnt) of the list are
// done); SWEEP_END then leaves nothing to drain.
template <bool AFTER, class Smem, class EW>
__device__ __forceinline__ int sweep_list(const Params &p, float4 cc, int np, const LeafEntry *__restrict__ pool,
                                          int off, int nleaf, const float4 *__restrict__ txf, Smem &sm, int qstride,
                                          ListPos &pos, int &myc, EW ew) {
  const unsigned FULL = 0xffffffffu;
  const int lane = lane_id();
  const unsigned lt = (1u << lane) - 1u;
  const float hx = 0.4995f * p.dxboundf - cc.w, hy = 0.4995f * p.dyboundf - cc.w, hz = 0.4995f * p.dzboundf - cc.w;
  int qn[MAXCELL];  // next free slot of each particle's queue
#pragma unroll
  for (int il = 0; il < MAXCELL; ++il) qn[il] = il * qstride;
  const int ipf = sm.ipos[0], ipl = sm.ipos[np - 1];  // ascending
  myc = 0;
  int j = -1;
  float4 e = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  bool fresh = true;  // the chunk at k0 is not loaded yet
  int state;
  while (true) {
    if (pos.k0 >= pos.cnt) {
      if (AFTER && pos.open) { pos.open = false; state = SWEEP_BATCH; break; }
      pos.nbase += pos.cnt;
      if (pos.e0 >= nleaf) { pos.k0 = pos.cnt = 0; state = SWEEP_END; break; }
      __syncwarp();
      pos.cnt = expand_batch(pool, off, nleaf, pos.e0, sm);
      pos.e0 += BATCH;
      pos.k0 = 0;
      pos.open = true;
      fresh = true;
      __syncwarp();
    }
    const int k = pos.k0 + lane;
    if (fresh) {
      j = k < pos.cnt ? sm.j[k] : -1;
      if (j >= 0) e = txf[j];
      fresh = false;
    }
    const int jc = j;
    float4 x = e;
    const int code = jc >= 0 ? sm.code[k] : 0;
    j = k + 32 < pos.cnt ? sm.j[k + 32] : -1;
    if (j >= 0) e = txf[j];
    bool wr = false;
    if (p.periodic) {
      if (code != 0) {
        x.x += offset_of_f(code, 0, p.dxboundf); x.y += offset_of_f(code, 1, p.dyboundf);
        x.z += offset_of_f(code, 2, p.dzboundf);
      }
      wr = __any_sync(FULL, jc >= 0 && (fabsf(cc.x - x.x) > hx || fabsf(cc.y - x.y) > hy || fabsf(cc.z - x.z) > hz));
    }
    const float w = ew(x.w);
    if (jc < 0) x.x = __int_as_float(0x7f800000);  // past the end: r^2 infinite, never accepted
    // chunks that hold the cell's own particles: no pair with itself (AFTER: or
    // with an earlier one)
    const bool own = __any_sync(FULL, jc >= ipf && jc <= ipl);
    const unsigned char flag =
        (unsigned char)(code != 0 ? code | (pos.nbase + k < CELLCACHE ? QC_CACHED : 0) : 0);
    if (AFTER && jc >= 0) sm.code[k] = flag;
    int left = qstride;
#pragma unroll
    for (int il = 0; il < MAXCELL; ++il) {
      if (il >= np) break;
      const float4 xi = sm.xi[il];
      float dx = xi.x - x.x, dy = xi.y - x.y, dz = xi.z - x.z;
      if (wr) {
        if (fabsf(dx) > 0.5f * p.dxboundf) dx -= copysignf(p.dxboundf, dx);
        if (fabsf(dy) > 0.5f * p.dyboundf) dy -= copysignf(p.dyboundf, dy);
        if (fabsf(dz) > 0.5f * p.dzboundf) dz -= copysignf(p.dzboundf, dz);
      }
      bool ok = dx * dx + dy * dy + dz * dz < fmaxf(xi.w, w);
      if (own) {
        const int ip = sm.ipos[il];
        ok = ok && (AFTER ? jc > ip : jc != ip);
      }
      const unsigned b = __ballot_sync(FULL, ok);
      if (ok) {
        const int q = qn[il] + __popc(b & lt);
        if constexpr (AFTER) { sm.qj[q] = (unsigned short)k; }
        else { sm.qj[q] = jc; sm.qc[q] = flag; }
      }
      qn[il] += __popc(b);
      left = min(left, (il + 1) * qstride - qn[il]);
    }
    pos.k0 += 32;
    if (left < 32) { state = SWEEP_FULL; break; }
  }
#pragma unroll
  for (int il = 0; il < MAXCELL; ++il)
    if (lane == il) myc = qn[il] - il * qstride;
  if (lane >= np) myc = 0;
  return state;
}

// Deal the 32 lanes out to the particles' queues (lane il < np holds its
// count c): the smallest number s of pairs per lane for which sum ceil(c/s)
// fits, from 32 s >= sum c up. Each lane gets its particle (il, -1: none), its
// first queue entry, the step and the count.
struct QueueLanes { int il, m0, step, c; };
__device__ __forceinline__ QueueLanes balance_queues(int np, int c, ListBase &sm) {
  const unsigned FULL = 0xffffffffu;
  const int lane = lane_id();
  if (lane >= np) c = 0;
  int s = max(1, (warp_sum_int(c) + 31) >> 5), need, tot;
  while (true) {
    need = (c + s - 1) / s;
    tot = warp_sum_int(need);
    if (tot <= 32) break;
    ++s;
  }
  int x = need;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(FULL, x, o);
    if (lane >= o) x += y;
  }
  x -= need;
  for (int t = 0; t < need; ++t) sm.own[x + t] = (unsigned char)lane;
  if (lane < np) { sm.first[lane] = (unsigned char)x; sm.lanes[lane] = (unsigned char)need; }
  __syncwarp();
  QueueLanes a;
  a.il = lane < tot ? (int)sm.own[lane] : -1;
  const int src = max(a.il, 0);
  a.m0 = lane - __shfl_sync(FULL, x, src);
  a.step = __shfl_sync(FULL, need, src);
  a.c = a.il >= 0 ? __shfl_sync(FULL, c, src) : (__shfl_sync(FULL, c, src), 0);
  return a;
}

// Sum RW values of every lane into per-(value, particle) totals: total idx =
// value * np + particle lives in tot[idx / 32] of lane idx % 32. The lane
// values pass through shared memory at red (32 RW doubles, free when every lane
// is done with the queues) and are added in lane order, so totals are
// deterministic.
template <int RW, int NR, class S, class T, class Get, class Add>
__device__ __forceinline__ void flush_lanes(int np, const S &sm, T *red, T (&tot)[NR], Get get, Add add) {
  static_assert(RW * MAXCELL <= 32 * NR, "totals per lane");
  const int lane = lane_id();
  __syncwarp();
#pragma unroll
  for (int k = 0; k < RW; ++k) red[lane * RW + k] = get(k);
  __syncwarp();
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const int idx = lane + 32 * r;
    if (idx < RW * np) {
      const int k = idx / np, il = idx - k * np;
      const T *src = red + (int)sm.first[il] * RW + k;
      const int nl = sm.lanes[il];
      for (int q = 0; q < nl; ++q) tot[r] = add(k, tot[r], src[q * RW]);
    }
  }
  __syncwarp();
}

// ------------------------------------------------------------------ symmetric pair passes
// Skeleton of the passes that evaluate every unordered neighbour pair once
// (force, adjoint). Cell A owns the entries of its trial list that start at or
// after its own leaf (a prefix: the list is in decreasing order of first
// particle) and, in its own leaf, the pairs j > i. Each owned batch is swept
// and drained; a pair's NJ values for j go to a per-batch array in shared
// memory and from there to jbuf at j's flattened trial index, its values for i
// stay in the lane (begin/body/get) until the drain's end.
//
// The j-side array of a batch (NJ values of up to BATCH leaves) bounds the warps
// per SM: 24 entries hold the owned half of most lists (37 entries at hfact
// 1.2) in one batch and leave room for 11 warps of the force pass at the
// reference's leaf size. One warp per block: the SM's shared memory then fills
// in the smallest steps (force per launch at 64^3, hydro / MHD: 1, 2, 4 warps
// per block 1.88 / 3.66, 1.95 / 3.98, 2.20 / 5.48 ms; batches of 16 entries 1.96
// / 3.72 ms at one warp).
template <int NJ>
__host__ __device__ constexpr int sym_smem_bytes(int minpart) {
  return (int)sizeof(ListSmemK) + 8 * NJ * BATCH * minpart;
}
// max of two non-negative doubles on the integer pipe (signal speeds: the
// FP64 max would occupy the scarce FP64 pipe)
__device__ __forceinline__ double fmax_pos(double a, double b) {
  return __longlong_as_double(max(__double_as_longlong(a), __double_as_longlong(b)));
}

// the owned prefix of a cell's list: entries and trial particles
__device__ __forceinline__ void owned_prefix(const LeafEntry *__restrict__ pool, int off, int nleaf, int s0, int &nown,
                                             int &town) {
  const unsigned FULL = 0xffffffffu;
  nown = 0; town = 0;
  for (int e0 = 0; e0 < nleaf; e0 += 32) {
    const int e = e0 + lane_id();
    LeafEntry le{0, 0};
    if (e < nleaf) le = pool[off + e];
    const bool own = e < nleaf && le.start >= s0;
    nown += __popc(__ballot_sync(FULL, own));
    town += warp_sum_int(own ? (le.cc & 255) : 0);
    if (!__all_sync(FULL, e >= nleaf || own)) break;
  }
}

// VMAX: value NJ-1 is a maximum (of non-negative doubles), the others sums.
// begin(il): the lane's particle; body(j, code, jv): one pair; get(v): the
// lane's i-side value; tot: totals per (value, particle) as flush_lanes.
template <int NJ, bool VMAX, int NR, class EW, class Begin, class Body, class Get>
__device__ __forceinline__ void sym_pairs(const Params &p, float4 cc, int np, const LeafEntry *__restrict__ pool,
                                          int off, int nown, const float4 *__restrict__ txf, ListSmemK &sm, int64_t tb,
                                          double *jbuf, int64_t jstride, double (&tot)[NR], EW ew, Begin begin,
                                          Body body, Get get) {
  const unsigned FULL = 0xffffffffu;
  const int lane = lane_id();
  const unsigned lt = (1u << lane) - 1u;
  double *js = reinterpret_cast<double *>(&sm + 1);
  const int jw = BATCH * p.minpart, qstride = LQ / np;
  for (int q = lane; q < NJ * jw; q += 32) js[q] = 0.0;
  ListPos pos;
  while (true) {
    __syncwarp();
    int myc;
    const int st = sweep_list<true>(p, cc, np, pool, off, nown, txf, sm, qstride, pos, myc, ew);
    if (st == SWEEP_END) break;
    const QueueLanes ql = balance_queues(np, myc, sm);
    const int il = max(ql.il, 0);
    begin(il);
    const unsigned short *qj = sm.qj + il * qstride;
    const int nst = ql.c > ql.m0 ? (ql.c - ql.m0 + ql.step - 1) / ql.step : 0;
    const int nstmax = (int)__reduce_max_sync(FULL, (unsigned)nst);
    // the particles of a cell accept nearly the same j in nearly the same
    // order, so aligned queues would put the same j in many lanes at once;
    // each particle starts at its own rotation of its queue instead
    const int rot = ql.c > 0 ? (il * ql.c) / np : 0;
    for (int t = 0; t < nstmax; ++t) {
      const bool valid = t < nst;
      int m = ql.m0 + t * ql.step + rot;
      if (m >= ql.c) m -= ql.c;
      const int kk = valid ? (int)qj[m] : -1;
      double jv[NJ];
      for (int v = 0; v < NJ; ++v) jv[v] = 0.0;
      if (valid) body(sm.j[kk], (int)sm.code[kk], jv);
      // lanes holding the same j: the lowest adds the others' values in
      // lane order, then adds the group's sum to j's batch slot
      const unsigned g = __match_any_sync(FULL, valid ? kk : -1 - lane);
      const int gs = __popc(g);
      const int gmax = (int)__reduce_max_sync(FULL, (unsigned)gs);
      const bool lead = valid && (g & lt) == 0u;
      for (int u = 1; u < gmax; ++u) {
        const int src = u < gs ? (int)__fns(g, 0, u + 1) : lane;
        for (int v = 0; v < NJ; ++v) {
          const double y = __shfl_sync(FULL, jv[v], src);
          if (lead && u < gs) jv[v] = VMAX && v == NJ - 1 ? fmax_pos(jv[v], y) : jv[v] + y;
        }
      }
      if (lead)
        for (int v = 0; v < NJ; ++v)
          js[v * jw + kk] = VMAX && v == NJ - 1 ? fmax_pos(js[v * jw + kk], jv[v]) : js[v * jw + kk] + jv[v];
      __syncwarp();
    }
    // j-side sums of a finished batch -> jbuf (value-major, flattened trial index)
    if (st == SWEEP_BATCH) {
      for (int v = 0; v < NJ; ++v)
        for (int k = lane; k < pos.cnt; k += 32) {
          jbuf[(int64_t)v * jstride + tb + pos.nbase + k] = js[v * jw + k];
          js[v * jw + k] = 0.0;
        }
    }
    static_assert(NJ <= 12, "lane sums staged in the queues' space");
    flush_lanes<NJ>(np, sm, sm.red, tot, get,
        [](int k, double s, double v) -> double { return VMAX && k == NJ - 1 ? fmax_pos(s, v) : s + v; });
  }
}

// The walking cell: position, size and search radius (exact and FP32).
struct WalkCell {
  double xp, yp, zp, xsizei, rcuti;
  float xpf, ypf, zpf, xsf, rcf;
};

// Node test of getneigh (kdtree.F90:1251-1290, get_sep :1468-1501) in the
// reference's FP64 rounding. Returns whether the node is opened; code gets
// the periodic offset code (2 bits per axis, 1: +L, 2: -L).
template <bool GET_HJ>
__device__ __forceinline__ bool node_open_exact(const Params &p, const Node &n, const WalkCell &w, double tree_acc2,
                                                int &code) {
  double dx = dsub(w.xp, n.x), dy = dsub(w.yp, n.y), dz = dsub(w.zp, n.z);
  code = 0;
  if (p.periodic) {
    if (fabs(dx) > p.hdlx) { double o = dmul(p.dxbound, sign1(dx)); dx = dsub(dx, o); code |= (o > 0 ? 1 : 2); }
    if (fabs(dy) > p.hdly) { double o = dmul(p.dybound, sign1(dy)); dy = dsub(dy, o); code |= (o > 0 ? 1 : 2) << 2; }
    if (fabs(dz) > p.hdlz) { double o = dmul(p.dzbound, sign1(dz)); dz = dsub(dz, o); code |= (o > 0 ? 1 : 2) << 4; }
  }
  const double r2 = r2_exact(dx, dy, dz);
  double rcut = w.rcuti;
  if (GET_HJ) { double rcutj = dmul(RADKERN, n.hmax); rcut = fmax(w.rcuti, rcutj); }
  const double t = dadd(dadd(w.xsizei, n.size), rcut);
  bool open = r2 < dmul(t, t);
  if (p.gravity) {
    const double s2 = dadd(w.xsizei, n.size);
    open = open || (dmul(tree_acc2, r2) < dmul(s2, s2));
  }
  return open;
}

// The same test decided in FP32 on the node mirror: each FP32 separation d'
// is within E = 2^-22 (|x'_cell| + |x'_node|) of the FP64 one (+ 2^-22 L
// after a periodic shift), which brackets r^2 and the wrap decisions; the
// thresholds carry a 1e-5 relative margin for their FP32 rounding. A test
// the bounds cannot decide is repeated exactly on the FP64 node record, so
// the outcome is always the reference's.
template <bool GET_HJ>
__device__ __forceinline__ bool node_open(const Params &p, const NodeF &nf, const Node *__restrict__ nodes, int nd,
                                          const WalkCell &w, double tree_acc2, float tacc2f, int &code) {
  const float E0 = 2.384185791015625e-07f;  // 2^-22
  float dx = w.xpf - nf.x, dy = w.ypf - nf.y, dz = w.zpf - nf.z;
  float ex = E0 * (fabsf(w.xpf) + fabsf(nf.x)), ey = E0 * (fabsf(w.ypf) + fabsf(nf.y)),
        ez = E0 * (fabsf(w.zpf) + fabsf(nf.z));
  code = 0;
  bool amb = false;
  if (p.periodic) {
    const float hx = 0.5f * p.dxboundf, hy = 0.5f * p.dyboundf, hz = 0.5f * p.dzboundf;
    const float bx = ex + E0 * hx, by = ey + E0 * hy, bz = ez + E0 * hz;
    if (fabsf(dx) > hx + bx) {
      const float o = copysignf(p.dxboundf, dx); dx -= o; code |= (o > 0.0f ? 1 : 2); ex += E0 * p.dxboundf;
    } else if (fabsf(dx) >= hx - bx) amb = true;
    if (fabsf(dy) > hy + by) {
      const float o = copysignf(p.dyboundf, dy); dy -= o; code |= (o > 0.0f ? 1 : 2) << 2; ey += E0 * p.dyboundf;
    } else if (fabsf(dy) >= hy - by) amb = true;
    if (fabsf(dz) > hz + bz) {
      const float o = copysignf(p.dzboundf, dz); dz -= o; code |= (o > 0.0f ? 1 : 2) << 4; ez += E0 * p.dzboundf;
    } else if (fabsf(dz) >= hz - bz) amb = true;
  }
  if (!amb) {
    const float lx = fmaxf(fabsf(dx) - ex, 0.0f), ly = fmaxf(fabsf(dy) - ey, 0.0f), lz = fmaxf(fabsf(dz) - ez, 0.0f);
    const float ux = fabsf(dx) + ex, uy = fabsf(dy) + ey, uz = fabsf(dz) + ez;
    const float lb = (lx * lx + ly * ly + lz * lz) * (1.0f - 1.0e-5f);
    const float ub = (ux * ux + uy * uy + uz * uz) * (1.0f + 1.0e-5f);
    const float rc = GET_HJ ? fmaxf(w.rcf, 2.0f * nf.hmax) : w.rcf;
    const float t = w.xsf + nf.size + rc;
    const float tlo = t * (1.0f - 1.0e-5f), thi = t * (1.0f + 1.0e-5f);
    int st = (ub < tlo * tlo) ? 1 : ((lb > thi * thi) ? 0 : 2);
    if (p.gravity && st != 1) {
      const float s2 = w.xsf + nf.size;
      const float slo = s2 * (1.0f - 1.0e-5f), shi = s2 * (1.0f + 1.0e-5f);
      const int g = (tacc2f * ub < slo * slo) ? 1 : ((tacc2f * lb > shi * shi) ? 0 : 2);
      st = (g == 1) ? 1 : ((st == 0 && g == 0) ? 0 : 2);
    }
    if (st != 2) return st == 1;
  }
  const Node n = nodes[nd];
  return node_open_exact<GET_HJ>(p, n, w, tree_acc2, code);
}

// Walk of one cell by a warp. Returns the number of emitted leaves (in walk
// order, in sh) or -1 on overflow. All 32 lanes must call it. The first five
// levels (top, by heap index) are tested in one round, lane = node: a node is
// reached if its ancestors' bits are all set in the ballot of the tests. Level
// by level they took six rounds of mostly idle lanes out of about seventeen.
// A round waits for its node loads, so rounds are what the walk costs: whole
// density calls of a 7^3 ball 1508 -> 1417 us, rollouts of 40^3 particles
// 56.9 -> 53.2 ms (walks of 64^3: 135 us a pass).
template <bool GET_HJ>
__device__ int walk_cell(const Params &p, const Node *__restrict__ nodes, const NodeF *__restrict__ nodesf,
                         const int *__restrict__ topn, const WalkCell &wc, WalkShared &sh) {
  const unsigned FULL = 0xffffffffu;
  const int lane = lane_id();
  const double tree_acc2 = p.tree_accuracy * p.tree_accuracy;
  const float tacc2f = (float)tree_acc2;
  int top = 0, nem = 0;
  bool overflow = false, first = true;
  while (first || top > 0) {
    const int k = min(32, top);
    const int nd = first ? topn[lane] : ((lane < k) ? sh.stk[top - k + lane] : -1);
    top -= k;
    __syncwarp();
    bool open = false, leaf = false;
    int code = 0, il = -1, ir = -1, count = 0;
    if (nd >= 0) {
      const NodeF nf = nodesf[nd];
      open = node_open<GET_HJ>(p, nf, nodes, nd, wc, tree_acc2, tacc2f, code);
      leaf = nf.left < 0;
      il = nf.left; ir = nf.right; count = nf.count;
    }
    bool push = open && !leaf;
    if (first) {
      const unsigned O = __ballot_sync(FULL, open);
      for (int a = lane >> 1; a >= 1; a >>= 1) open = open && ((O >> a) & 1u);
      push = open && !leaf && lane >= 16;  // the others' children are in this round
      first = false;
    }
    const bool emit = open && leaf;
    unsigned be = __ballot_sync(FULL, emit);
    if (emit) {
      int pos = nem + __popc(be & ((1u << lane) - 1));
      if (pos < WALK_EM) sh.put(pos, ir, count, code);
    }
    nem += __popc(be);
    unsigned bp = __ballot_sync(FULL, push);
    if (push) {
      int pos = top + 2 * __popc(bp & ((1u << lane) - 1));
      if (pos + 1 < WALK_STK) { sh.stk[pos] = il; sh.stk[pos + 1] = ir; }
    }
    top += 2 * __popc(bp);
    if (top >= WALK_STK || nem > WALK_EM) { overflow = true; break; }
    __syncwarp();
  }
  __syncwarp();
  if (overflow) return -1;
  return nem;
}

// K3 for the density: walk the cells of `act` whose redo flag is set
// W warps (cells) per block, W in {1, 2, 4} (static shared memory, <= 40 KB)
template <bool GET_HJ, int W>
__global__ void __launch_bounds__(32 * W) k_walk(Params p, const Node *nodes, const NodeF *nodesf, const int *topn,
                                                          const int *leaves,
                                                          const int *act, int nact, const int *need,
                                                          const double *cell_hmax, LeafEntry *pool,
                                                          long long pool_cap, unsigned long long *pool_top,
                                                          int *cell_off, int *cell_nleaf, int *cell_ntrial,
                                                          int *err) {
  __shared__ WalkShared sh[W];
  const int w = threadIdx.x >> 5, lane = lane_id();
  const int a = blockIdx.x * W + w;
  if (a >= nact) return;
  const int cell = act ? act[a] : a;
  if (need && !need[cell]) return;
  const Node nd = nodes[leaves[cell]];
  WalkCell wc;
  wc.xp = nd.x; wc.yp = nd.y; wc.zp = nd.z; wc.xsizei = nd.size;
  wc.rcuti = dmul(RADKERN, cell_hmax ? cell_hmax[cell] : nd.hmax);
  wc.xpf = (float)wc.xp; wc.ypf = (float)wc.yp; wc.zpf = (float)wc.zp; wc.xsf = (float)wc.xsizei;
  wc.rcf = (float)wc.rcuti;
  int nem = walk_cell<GET_HJ>(p, nodes, nodesf, topn, wc, sh[w]);
  if (nem < 0) {
    if (lane == 0) set_error(err, PH_ERR_STACK);
    return;
  }
  int tot = 0;
  for (int e = lane; e < nem; e += 32) tot += sh[w].count(e);
  tot = warp_sum_int(tot);
  unsigned long long off = 0;
  if (lane == 0) off = atomicAdd(pool_top, (unsigned long long)nem);
  off = __shfl_sync(0xffffffffu, off, 0);
  if ((long long)(off + nem) > pool_cap) {
    if (lane == 0) set_error(err, PH_ERR_LIST);
    return;
  }
  write_ranked(sh[w], nem, pool, off);
  if (lane == 0) { cell_off[cell] = (int)off; cell_nleaf[cell] = nem; cell_ntrial[cell] = tot; }
}

// k_walk with the context's warps per block (1, 2 or 4)
template <bool GET_HJ, class... A>
inline void launch_walk(int warps, int ncells, cudaStream_t st, A... args) {
  if (warps >= 4) k_walk<GET_HJ, 4><<<(ncells + 3) / 4, 128, 0, st>>>(args...);
  else if (warps == 2) k_walk<GET_HJ, 2><<<(ncells + 1) / 2, 64, 0, st>>>(args...);
  else k_walk<GET_HJ, 1><<<ncells, 32, 0, st>>>(args...);
}

}  // namespace ph
