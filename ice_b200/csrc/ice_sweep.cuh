// ice_sweep.cuh -- a stage as two kernels of independent threads, without shared memory or barriers:
//
//  k_flux   the fluxes of the x, y and z faces and of every boundary record, each into its own array (one
//           launch, a range of CTAs per kind: they do not depend on one another);
//  k_cells  the cells' update: a cell's boundary records in face order, its two faces per direction in the
//           odd-then-even order of tile_sweep (Mod_Fluxes.f90:470-506), the source k_source
//           wrote, R = (R/vol + S) dt (Lib_Residual.f90:147-156) and the RK stage
//           in conservative variables with the reference's floors (Lib_Newstate.f90:198-219).
//
// Every cell's limited slope along a direction is computed once and serves both of its faces: along x by
// the thread of the cell, handed to the thread of the cell below by a warp shuffle; along y and z by a
// march, which keeps the slope and the difference quotient of the last cell in registers. The slope is
// the value state_reconstruction computes for either face (Lib_Reconstruction.f90:17-78: the same operands
// and operations), so the plain form keeps its bits.
//
// What bounds it and why this split. One kernel with the planes of a tile staged in shared memory, its faces
// dealt out to the threads and the update behind a barrier moved 24 nc bytes per cell and stage, but took the
// registers and shared memory of all its phases at once: one CTA of 6 to 8 warps per SM in FP64 (20 % of the
// issue slots, dependent FP64 chains), two in FP32 (49 %), DRAM at 5 and 16 % of peak. Here the faces need
// 72 to 128 registers (168 for AG in FP64) and no barrier, every direction is in flight at once, and the fluxes cost
// 6 nc words per cell of bandwidth that stood idle. FP64: the two divisions of every limited slope
// run branchless and side by side (ice_div.h), where a compiled division's branch ordered them one after the
// other. The one kernel (+ records; CUDA events) / k_flux + k_cells (the profiler's launch times), one B200: FP64 IG
// 96 x 95 x 97 967 / 215 + 63 us, AG 64 x 61 x 67 693 + 161 / 142 + 39 us; FP32 form IG 128 x 126 x 129
// 516 + 28 / 168 + 136 us, AG 96^3 387 + 30 / 146 + 98 us.
#pragma once
#include "ice_kernels.cuh"

namespace ice {

constexpr int SW_NT = 128;                      // threads per CTA
constexpr int SW_XC = SW_NT / 32 * 31;          // cells whose upper x face one CTA computes

// The CTAs per SM the flux and the cell kernel are held to, and which loads of the cell kernel wait.
// Flux: 6 against 5 in the FP32-flux form 192 / 214 us (IG, 128 x 126 x 129; AG at 6 spills, 209 / 164 us on
// 96^3), 3 against 2 for FP64 AG 152 / 160 us (64 x 61 x 67), 4 against 3 and 5 for FP64 IG 225 / 248 / 246 us
// (96 x 95 x 97).
// Cells: a warp holds a register for every load in flight, so a cell's six fluxes and its state at once cost
// warps. late 1 asks for the state only when the x and y fluxes are summed, 2 for the z fluxes too. AG FP64:
// 56.5 us with all at once at 2 CTAs, 56.0 / 57.3 at late 1 and 2, 48.3 - 50.1 at late 2 and 3 CTAs (all at
// once and 3 CTAs: 69, it spills). AG FP32 (4 CTAs): 126.8 us all at once, 104.7 at late 1, 109.0 at late 2. IG FP64 (4):
// 77.3 / 73.7 / 81.3 us at late 0, 1, 2. IG FP32: 138.9 us all at once at 5 CTAs, 136.8
// at late 1 and 6 (145.4 and 144.5 with one of the two). MK FP32: flux 7 against 6 and cells 6 against 5, all at
// once, with IG's: three families on 8 blocks, 1.7 M cells, 29.3 -> 28.6 ms of 8 steps, flux 202 -> 199 us and
// cells 138 -> 134 (means of the families).
template <int CL, typename R> struct SweepOcc {
  static constexpr int flux = sizeof(R) == 8 ? (CL == AG ? 3 : 4) : CL == AG ? 4 : CL == IG ? 6 : 7;
  static constexpr int cells = sizeof(R) == 8 ? (CL == AG ? 3 : 4) : CL == AG ? 4 : 6;
  static constexpr int late = sizeof(R) == 8 ? (CL == AG ? 2 : 1) : CL == MK ? 0 : 1;
};

// Limited slope of one cell from its two difference quotients.
template <int CL, int LIM, typename R>
__device__ __forceinline__ void slope_of(int lim, const R* sf, const R* sb, R dlf, R dlb, R dlc, bool first, bool fast,
                                         R* s) {
  R cx, cy;
  limiter_bounds<R>(dlf, dlb, dlc, cx, cy);
  limited<NC<CL>::v, LIM, R>(lim, sf, sb, cx, cy, first, fast, s);
}

// The two states of a face from its cells' limited slopes, with state_reconstruction's fallback:
// the weight halves until both states are physical, and the first-order states are taken below
// 1e-18 (Lib_Reconstruction.f90:40-76). Returns true when the first-order states are unphysical.
template <int CL, typename R, typename QL, typename QR>
__device__ __forceinline__ bool states_from_slopes(const QL& ql, const R* sl, R dll, bool fl,
                                                   const QR& qr, const R* sr, R dlr, bool fr, R beta,
                                                   R* pl, R* pr) {
  constexpr int nc = NC<CL>::v;
  R limval = beta;
  bool st_l = false, st_r = false;
  for (int pass = 0; (!st_l || !st_r) && pass < 256; ++pass) {
    if (pass == 255) limval = (R)0;
    // a first-order side has zero slopes; its zero weight keeps a non-finite sensor out of it
    const R wl = fl ? (R)0 : limval, wr = fr ? (R)0 : limval;
#pragma unroll
    for (int v = 0; v < nc; ++v) {
      pl[v] = ql[v] + (sl[v]*wl)*dll;
      pr[v] = qr[v] - (sr[v]*wr)*dlr;
    }
    st_l = fl || check_prim<CL>(pl);
    st_r = fr || check_prim<CL>(pr);
    limval = (R)0.5*limval;
    if (limval < (R)1e-18 && !(st_l && st_r)) {
#pragma unroll
      for (int v = 0; v < nc; ++v) { pl[v] = ql[v]; pr[v] = qr[v]; }
      if (!(check_prim<CL>(pl) && check_prim<CL>(pr))) return true;
      break;
    }
  }
  return false;
}

// One face from its two cells and their slopes.
template <int CL, int RS, typename R>
__device__ __forceinline__ bool face_of(const Geo& G, const FamDev& F, int d, long long fi, const R* ql, const R* sl,
                                        R dll, bool fl, const R* qr, const R* sr, R dlr, bool fr, R bf, R* out) {
  constexpr int nc = NC<CL>::v;
  R nrm[3], area, pl[nc], pr[nc], f[nc];
  face_geometry<R>(G, d, fi, nrm, area);
  const bool bad = states_from_slopes<CL, R>(ql, sl, dll, fl, qr, sr, dlr, fr, bf, pl, pr);
  riemann<CL, RS, R>(pl, pr, nrm, f, (R)F.mat.cp);
#pragma unroll
  for (int v = 0; v < nc; ++v) out[v] = f[v] * area;
  return bad;
}

template <typename R> __device__ __forceinline__ R beta_at(const FamDev& F, long long q) {
  return F.sd ? ((const R*)F.betaR)[q] : (R)1;
}

// March up one column along direction D (1: y, 2: z) from cell (i, j, k): the faces above it and the next n - 1
// cells. One code for both directions: its size is what the instruction cache feels.
template <int CL, int RS, int LIM, typename R>
__device__ __forceinline__ bool march(const Geo& G, const FamDev& F, const DBlock& B, int D, int i, int j, int k, int n) {
  constexpr int nc = NC<CL>::v;
  R* out = (R*)F.Ff[D];
  const int N = D == 1 ? B.nj : B.nk;
  int c = D == 1 ? j : k;
  const int end = c + n;
  const long long gs = gstride(B, D);
  const long long rs = D == 1 ? (long long)(B.ni + 2) : (long long)(B.ni + 2) * (B.nj + 2);
  const long long qs = D == 1 ? (long long)B.ni : (long long)B.ni * B.nj;
  long long g = gidx(B, i, j, k), r = ridx(B, i, j, k), q = iidx(B, i, j, k);
  long long fi = fidx(B, D, i, j, k, c + 1);
  const R re = (R)kRhoEmpty;
  bool bad = false;
  R a[nc], b[nc], d[nc], sl[nc];
  R lc = cell_length<R>(G, D, r), ln = cell_length<R>(G, D, r + rs), dlc;
  bool ea, eb, first, kd;
  {
    R m[nc], sb[nc];
#pragma unroll
    for (int v = 0; v < nc; ++v) {
      const double* P = F.Up + (long long)v * G.NG + g;
      m[v] = (R)P[-gs]; a[v] = (R)P[0]; b[v] = (R)P[gs];
    }
    R lm = cell_length<R>(G, D, r - rs);
    if (c == 0 && F.inj[g - gs]) lm = (R)0;
    const R dlb = (R)0.5*(lm + lc), dlf = (R)0.5*(lc + ln);
    dlc = (R)0.5*lc;
    ea = a[0] <= re; eb = b[0] <= re;
    first = m[0] <= re || ea || eb;
    const bool k0 = quotients<nc, R>(m, a, dlb, sb);
    kd = quotients<nc, R>(a, b, dlf, d);
    slope_of<CL, LIM, R>(F.limiter, d, sb, dlf, dlb, dlc, first, k0 && kd, sl);
  }
  R ba = beta_at<R>(F, q);
  for (; c < end; ++c) {
    R f[nc], x[nc], df[nc], sr[nc];
#pragma unroll
    for (int v = 0; v < nc; ++v) x[v] = (R)F.Up[(long long)v * G.NG + g + 2 * gs];
    const R lx = cell_length<R>(G, D, r + 2 * rs);
    const bool ex = x[0] <= re;
    const R lp = (c + 1 == N - 1 && F.inj[g + 2 * gs]) ? (R)0 : lx;
    const R dlb = (R)0.5*(lc + ln), dlf = (R)0.5*(ln + lp), dln = (R)0.5*ln;
    const bool fn = ea || eb || ex;
    const bool kf = quotients<nc, R>(b, x, dlf, df);
    slope_of<CL, LIM, R>(F.limiter, df, d, dlf, dlb, dln, fn, kd && kf, sr);
    const R bb = beta_at<R>(F, q + qs);
    bad |= face_of<CL, RS, R>(G, F, D, fi, a, sl, dlc, first, b, sr, dln, fn, mn(ba, bb), f);
#pragma unroll
    for (int v = 0; v < nc; ++v) out[(long long)v * G.NF[D] + fi] = f[v];
#pragma unroll
    for (int v = 0; v < nc; ++v) { a[v] = b[v]; b[v] = x[v]; d[v] = df[v]; sl[v] = sr[v]; }
    lc = ln; ln = lx; dlc = dln; first = fn; kd = kf; ea = eb; eb = ex; ba = bb;
    g += gs; r += rs; q += qs; fi += qs;
  }
  return bad;
}

// The x faces of SW_XC consecutive cells (flat over the block, i fastest): lane t of a warp takes the slope
// of its cell, and the face above it with the slope of lane t + 1; 31 faces a warp, lane 31 being the next
// warp's first.
template <int CL, int RS, int LIM, typename R>
__device__ __forceinline__ bool x_faces(const Geo& G, const FamDev& F, const DBlock& B, int base) {
  constexpr int nc = NC<CL>::v;
  const int lane = threadIdx.x & 31, wrp = threadIdx.x >> 5;
  const long long ncell = (long long)B.ni * B.nj * B.nk;
  long long l = (long long)base + wrp * 31 + lane;
  const bool in = l < ncell;
  if (!in) l = ncell - 1;
  const unsigned u = (unsigned)l, ni = (unsigned)B.ni, nj = (unsigned)B.nj;
  const unsigned jk = u / ni;
  const int i = (int)(u % ni), j = (int)(jk % nj), k = (int)(jk / nj);
  const long long g = gidx(B, i, j, k), r = ridx(B, i, j, k);
  R m[nc], a[nc], b[nc];
#pragma unroll
  for (int v = 0; v < nc; ++v) {
    const double* P = F.Up + (long long)v * G.NG + g;
    m[v] = (R)P[-1]; a[v] = (R)P[0]; b[v] = (R)P[1];
  }
  R lm = cell_length<R>(G, 0, r - 1), lc = cell_length<R>(G, 0, r), lp = cell_length<R>(G, 0, r + 1);
  if (i == 0 && F.inj[g - 1]) lm = (R)0;
  if (i == B.ni - 1 && F.inj[g + 1]) lp = (R)0;
  const R re = (R)kRhoEmpty;
  const bool first = m[0] <= re || a[0] <= re || b[0] <= re;
  const R dlb = (R)0.5*(lm + lc), dlf = (R)0.5*(lc + lp), dlc = (R)0.5*lc;
  R s[nc], sr[nc];
  {
    R sf[nc], sb[nc];
    const bool k0 = quotients<nc, R>(m, a, dlb, sb);
    const bool k1 = quotients<nc, R>(a, b, dlf, sf);
    slope_of<CL, LIM, R>(F.limiter, sf, sb, dlf, dlb, dlc, first, k0 && k1, s);
  }
#pragma unroll
  for (int v = 0; v < nc; ++v) sr[v] = __shfl_down_sync(0xffffffffu, s[v], 1);
  const R dlr = __shfl_down_sync(0xffffffffu, dlc, 1);
  const bool fr = __shfl_down_sync(0xffffffffu, (int)first, 1) != 0;
  const long long q = B.ioff + l;
  R bf = beta_at<R>(F, q);
  if (F.sd) bf = mn(bf, __shfl_down_sync(0xffffffffu, bf, 1));
  if (!in || lane == 31 || i >= B.ni - 1) return false;
  R f[nc];
  const long long fi = fidx(B, 0, i, j, k, i + 1);
  const bool bad = face_of<CL, RS, R>(G, F, 0, fi, a, s, dlc, first, b, sr, dlr, fr, bf, f);
  R* out = (R*)F.Ff[0] + fi;
#pragma unroll
  for (int v = 0; v < nc; ++v) out[(long long)v * G.NF[0]] = f[v];
  return bad;
}

// r -+ the cell's two faces along one direction in tile_sweep's odd-then-even order: c the 1-based index,
// n the cells of the direction, lo and hi the fluxes of the faces below and above (the block's boundary
// faces are in the sum already).
template <int nc, typename R>
__device__ __forceinline__ void add_faces(R* r, int c, int n, const R* lo, const R* hi) {
  if (c % 2 == 1) {
    if (c < n) {
#pragma unroll
      for (int v = 0; v < nc; ++v) r[v] = r[v] - hi[v];
    }
    if (c > 1) {
#pragma unroll
      for (int v = 0; v < nc; ++v) r[v] = r[v] + lo[v];
    }
  } else {
#pragma unroll
    for (int v = 0; v < nc; ++v) r[v] = r[v] + lo[v];
    if (c < n) {
#pragma unroll
      for (int v = 0; v < nc; ++v) r[v] = r[v] - hi[v];
    }
  }
}

// The update of cell q (at g in the pools) from its summed residual r (see the head of this file) and its
// FP64 state p.
template <int CL, typename R>
__device__ __forceinline__ void cell_update(const Geo& G, const FamDev& F, long long q, long long g, const R* r,
                                            const double* p, int write_r, Status* st) {
  constexpr int nc = NC<CL>::v;
  double s[nc];
#pragma unroll
  for (int v = 0; v < nc; ++v) s[v] = 0.0;
  if (F.coupled && (sizeof(R) == 8 || F.src_ready)) {   // the source kernel ran first
#pragma unroll
    for (int v = 0; v < nc; ++v) s[v] = F.Sf ? (double)F.Sf[(long long)v * G.NI + q] : F.S[(long long)v * G.NI + q];
  } else if (sizeof(R) == 4 && F.coupled) {             // compute_source_ on the stage's state
    R pr[nc], gr[9], sr[nc];
#pragma unroll
    for (int v = 0; v < nc; ++v) pr[v] = (R)p[v];
#pragma unroll
    for (int v = 0; v < 9; ++v) gr[v] = (R)G.gasf[(long long)v * G.NI + q];
    R tau = cell_source<CL, R>(pr, gr, gr[5], gr[6], gr[7], gr[8], F.mat, F.drag, F.heat, F.blow, sr);
#pragma unroll
    for (int v = 0; v < nc; ++v) s[v] = (F.frozen_mask & (1u << v)) ? 0.0 : (double)sr[v];
    if (F.write_tau) F.tau[q] = (double)tau;
  }
  if (F.xstep) accumulate_source<CL>(F.xstep, G.NI, q, s, F.xfirst, F.rk);
  const double dt = F.dt ? F.dt[q] : *F.dtg;
  const double vol = G.vol[q];
  double rd[nc];
  if constexpr (sizeof(R) == 4) {
    const double ivol = 1.0 / vol;
#pragma unroll
    for (int v = 0; v < nc; ++v) rd[v] = ((double)r[v]*ivol + s[v]) * dt;
  } else {
    const double y = ice_div_recip(vol);
    bool ok = ice_div_by(vol);
#pragma unroll
    for (int v = 0; v < nc; ++v) { ok = ok && dividend((double)r[v]); rd[v] = ice_div_quot((double)r[v], vol, y); }
    if (!ok) {
#pragma unroll
      for (int v = 0; v < nc; ++v) rd[v] = quot_any((double)r[v], vol);
    }
  }
  if constexpr (sizeof(R) == 8) {
#pragma unroll
    for (int v = 0; v < nc; ++v) rd[v] = (rd[v] + s[v]) * dt;
  }
  if (F.imports) {                          // add_births (Lib_Residual.f90:164-210): the coupler's rates
#pragma unroll
    for (int v = 0; v < nc; ++v) rd[v] = rd[v] + F.imports[(long long)v * G.NI + q] * dt;
  }
#pragma unroll
  for (int v = 0; v < nc; ++v) if (F.frozen_mask & (1u << v)) rd[v] = 0.0;
  if (write_r) {
#pragma unroll
    for (int v = 0; v < nc; ++v) F.resid[(long long)v * G.NI + q] = rd[v];
    return;
  }
  double po[nc], co[nc], cn[nc];
  const bool u0p = F.U0 == F.Up;            // the first RK stage: U_0 is the stencil state itself
#pragma unroll
  for (int v = 0; v < nc; ++v) po[v] = u0p ? p[v] : F.U0[(long long)v * G.NG + g];
  if constexpr (sizeof(R) == 4) {
    prim2cons_fma<CL>(po, co, F.mat.cp);
    prim2cons_fma<CL>(p, cn, F.mat.cp);
  } else {
    prim2cons<CL, double>(po, co, F.mat.cp);
    prim2cons<CL, double>(p, cn, F.mat.cp);
  }
#pragma unroll
  for (int v = 0; v < nc; ++v) { double rr = (cn[v] - co[v] + rd[v]) * F.rk; cn[v] = co[v] + rr; }
  if (cn[0] < 0.0) atomicAdd(&st->nfloored, 1ULL);
  double pn[nc];
  cons2prim<CL, sizeof(R) == 4>(cn, pn, F.mat.cp);
  if constexpr (sizeof(R) == 4) {
    if (F.realize && realize<CL>(pn)) atomicAdd(&st->nrealized, 1ULL);
  }
  if (!check_prim<CL, double>(pn)) atomicOr(&st->flags, (unsigned)ICE_GPU_ST_NAN_STATE);
#pragma unroll
  for (int v = 0; v < nc; ++v) F.Uo[(long long)v * G.NG + g] = pn[v];
}

// The first nrb CTAs take the boundary records (long chains: they start first), the others a job each.
template <int CL, int RS, int LIM, typename R>
__global__ void __launch_bounds__(SW_NT, SweepOcc<CL, R>::flux)
k_flux(Geo G, FamDev F, const SweepJob* __restrict__ jobs, const DRec* recs, const int* frec, int nfrec, int nrb, Status* st) {
  bool bad = false;
  if ((int)blockIdx.x < nrb) {
    bad = rec_thread<CL, RS, LIM, R>(G, F, recs, frec, nfrec, blockIdx.x * SW_NT + threadIdx.x);
    if (bad) atomicOr(&st->flags, (unsigned)ICE_GPU_ST_BAD_RECON);
    return;
  }
  const SweepJob t = jobs[blockIdx.x - nrb];
  const DBlock B = G.blk[t.b];
  if (t.kind == SW_X) {
    for (int m = 0; m < t.n; ++m) bad |= x_faces<CL, RS, LIM, R>(G, F, B, t.base + m * SW_XC);
  } else {
    const int col = t.base + threadIdx.x;
    const bool y = t.kind == SW_Y;
    const int i = col % B.ni, o = col / B.ni;    // the column: (i, k) along y, (i, j) along z
    if (o < (y ? B.nk : B.nj)) bad = march<CL, RS, LIM, R>(G, F, B, t.kind, i, y ? t.c0 : o, y ? o : t.c0, t.n);
  }
  if (bad) atomicOr(&st->flags, (unsigned)ICE_GPU_ST_BAD_RECON);
}

// The update of every cell. write_r: store R instead of updating (IRS runs).
template <int CL, typename R>
__global__ void __launch_bounds__(SW_NT, SweepOcc<CL, R>::cells) k_cells(Geo G, FamDev F, int write_r, Status* st) {
  constexpr int nc = NC<CL>::v;
  const long long q = (long long)blockIdx.x * SW_NT + threadIdx.x;
  if (q >= G.NI) return;
  const int b = find_block(G.blk, G.nb, q);
  if (!stepped(G, b)) return;
  const DBlock B = G.blk[b];
  const unsigned l = (unsigned)(q - B.ioff), ni = (unsigned)B.ni, nj = (unsigned)B.nj;   // < 2^31 cells a block
  const unsigned jk = l / ni;
  const int i = (int)(l % ni), j = (int)(jk % nj), k = (int)(jk / nj);
  const long long g = gidx(B, i, j, k);
  constexpr int LATE = SweepOcc<CL, R>::late;
  double p[nc];
  R x0[nc], x1[nc], y0[nc], y1[nc], z0[nc], z1[nc];
  const R* z = (const R*)F.Ff[2] + fidx(B, 2, i, j, k, k);
  const long long up = (long long)B.ni * B.nj;
  {                                              // on their way before the first use
    const R* x = (const R*)F.Ff[0] + fidx(B, 0, i, j, k, i);
    const R* y = (const R*)F.Ff[1] + fidx(B, 1, i, j, k, j);
#pragma unroll
    for (int v = 0; v < nc; ++v) {
      x0[v] = x[v * G.NF[0]]; x1[v] = x[v * G.NF[0] + 1];
      y0[v] = y[v * G.NF[1]]; y1[v] = y[v * G.NF[1] + B.ni];
      if (LATE < 2) { z0[v] = z[v * G.NF[2]]; z1[v] = z[v * G.NF[2] + up]; }
      if (LATE < 1) p[v] = F.Up[(long long)v * G.NG + g];
    }
  }
  R r[nc];
#pragma unroll
  for (int v = 0; v < nc; ++v) r[v] = (R)0;
  if (i == 0 || i == B.ni - 1 || j == 0 || j == B.nj - 1 || k == 0 || k == B.nk - 1) {
    double acc[nc];
    edge_sum<nc>(B, i, j, k, acc, [&](int d, int v) { return d == 0 ? x0[v] : d == 1 ? y0[v] : LATE < 2 ? z0[v] : z[v * G.NF[2]]; },
                 [&](int d, int v) { return d == 0 ? x1[v] : d == 1 ? y1[v] : LATE < 2 ? z1[v] : z[v * G.NF[2] + up]; });
#pragma unroll
    for (int v = 0; v < nc; ++v) r[v] = (R)acc[v];
  }
  if (B.ni >= 2) add_faces<nc>(r, i + 1, B.ni, x0, x1);
  if (B.nj >= 2) add_faces<nc>(r, j + 1, B.nj, y0, y1);
  if constexpr (LATE > 0) {
    asm volatile("" ::: "memory");               // keeps these loads behind the sums above
#pragma unroll
    for (int v = 0; v < nc; ++v) {
      if (LATE > 1) { z0[v] = z[v * G.NF[2]]; z1[v] = z[v * G.NF[2] + up]; }
      p[v] = F.Up[(long long)v * G.NG + g];
    }
  }
  if (B.nk >= 2) add_faces<nc>(r, k + 1, B.nk, z0, z1);
  cell_update<CL, R>(G, F, q, g, r, p, write_r, st);
}

}  // namespace ice
