// ice_kernels.cuh -- the kernels of the solve stage that depend on the closure (and the Riemann
// solver), but for the flux and cell kernels (ice_sweep.cuh): per-cell dt, the ghost fill of both layers, the
// boundary records' fluxes, the source, the FP32-flux form's 1-D stage kernel and the separate update of the
// IRS path. Included by the per-closure units
// (ice_fam_*.cu) and by ice_gpu.cu, each instantiating what it launches.
#pragma once
#include "ice_layout.cuh"

namespace ice {
namespace {

// ------------------------------------------------------------------ stencil functor
template <typename R, int NC_> struct RegStencil {   // q(s, v): cell s = 0..3 of the stencil, variable v
  R v[4][NC_];
  __device__ __forceinline__ R operator()(int s, int q) const { return v[s][q]; }
};

// One interior face along d between the 0-based cells (i,j,k) and its upper neighbour:
// face_flux + compute_flux_ (Mod_Fluxes.f90:599-685). Returns true on an unphysical
// first-order face. The stencil is converted once into registers.
template <int CL, int RS, int LIM, typename R>
__device__ __forceinline__ bool face_flux(const Geo& G, const FamDev& F, const DBlock& B, int d, int i, int j, int k,
                                         R* flux) {
  constexpr int nc = NC<CL>::v;
  const int c = d == 0 ? i : d == 1 ? j : k;
  const int n = d == 0 ? B.ni : d == 1 ? B.nj : B.nk;
  const int o0 = d == 0, o1 = d == 1, o2 = d == 2;
  R bf = (R)1;
  if (F.beta) bf = (R)mn(F.beta[iidx(B, i, j, k)], F.beta[iidx(B, i + o0, j + o1, k + o2)]);
  const double* dl = G.dl + (long long)d * G.NR;
  const long long r0 = ridx(B, i, j, k);
  const long long rs = d == 0 ? 1LL : d == 1 ? (long long)(B.ni + 2) : (long long)(B.ni + 2) * (B.nj + 2);
  R l0 = (R)dl[r0 - rs], l1 = (R)dl[r0], l2 = (R)dl[r0 + rs], l3 = (R)dl[r0 + 2 * rs];
  const long long st = gstride(B, d);
  const long long g0 = gidx(B, i, j, k) - st;
  if (c == 0 && F.inj[g0]) l0 = (R)0;
  if (c == n - 2 && F.inj[g0 + 3 * st]) l3 = (R)0;
  R dl0 = (R)0.5*(l0 + l1), dl1 = (R)0.5*(l1 + l2), dl2 = (R)0.5*(l2 + l3);
  R dll = (R)0.5*l1, dlr = (R)0.5*l2;
  R pl[nc], pr[nc], fl[nc];
  bool bad;
  RegStencil<R, nc> q;
#pragma unroll
  for (int s2 = 0; s2 < 4; ++s2)
#pragma unroll
    for (int v = 0; v < nc; ++v) q.v[s2][v] = (R)__ldg(F.Up + (long long)v * G.NG + g0 + s2 * st);
  bad = reconstruct<CL, LIM, R>(F.limiter, q, dl0, dl1, dl2, dll, dlr, pl, pr, bf);
  const long long fi = fidx(B, d, i, j, k, c + 1);
  const long long NF = G.NF[d];
  const double* fc = G.face[d];
  R nrm[3] = {(R)fc[fi], (R)fc[NF + fi], (R)fc[2 * NF + fi]};
  R area = (R)fc[3 * NF + fi];
  riemann<CL, RS, R>(pl, pr, nrm, fl, (R)F.mat.cp);
#pragma unroll
  for (int v = 0; v < nc; ++v) flux[v] = fl[v] * area;
  return bad;
}

// Normal and area of face fi along d: the FP64 arrays in the plain form, the packed single-precision
// copy (one 16-byte load, the same roundings) in the FP32-flux form.
template <typename R>
__device__ __forceinline__ void face_geometry(const Geo& G, int d, long long fi, R* nrm, R& area) {
  if constexpr (sizeof(R) == 4) {
    const float4 f = G.ff[d][fi];
    nrm[0] = f.x; nrm[1] = f.y; nrm[2] = f.z; area = f.w;
  } else {
    const long long NF = G.NF[d];
    const double* fc = G.face[d];
    nrm[0] = fc[fi]; nrm[1] = fc[NF + fi]; nrm[2] = fc[2 * NF + fi]; area = fc[3 * NF + fi];
  }
}

// The length along d of the cell at ring index r, in the precision of R (the same rounding either way).
template <typename R>
__device__ __forceinline__ R cell_length(const Geo& G, int d, long long r) {
  if constexpr (sizeof(R) == 4) return G.dlf[(long long)d * G.NR + r];
  else return G.dl[(long long)d * G.NR + r];
}

// The Jameson weight of cell (i,j,k) of block B from the stage's density in global memory (the
// boundary kernels; compute_beta, Mod_Fluxes.f90:366-389).
template <typename R>
__device__ __forceinline__ R beta_cell(const FamDev& F, const DBlock& B, int i, int j, int k) {
  const double* P = F.Up;
  return sd_rho<R>((R)P[gidx(B, i, j, k)], (R)P[gidx(B, i - 1, j, k)], (R)P[gidx(B, i + 1, j, k)],
                   (R)P[gidx(B, i, j - 1, k)], (R)P[gidx(B, i, j + 1, k)],
                   (R)P[gidx(B, i, j, k - 1)], (R)P[gidx(B, i, j, k + 1)]);
}

// record_flux (Mod_BC_Fluxes.f90:180-272): the flux through a record's face into its cell. R is the
// reconstruction and Riemann type (double in the plain form, float in the FP32-flux form); LIM the
// limiter the kernel is specialised for (the same formulas as the run-time switch in double).
// The four stencil cells are read into registers before the reconstruction, so that their loads
// are in flight together (the reconstruction's branches would otherwise order them).
template <int CL, int RS, int LIM, typename R>
__device__ bool record_flux(const Geo& G, const FamDev& F, const DRec& r, double* flux, const double* beta_face) {
  constexpr int nc = NC<CL>::v;
  const DBlock& B = G.blk[r.b];
  int f = r.f, i = r.i, j = r.j, k = r.k;
  int g0 = (f == 1) - (f == 2), g1 = (f == 3) - (f == 4), g2 = (f == 5) - (f == 6);  // guide(f,:)
  int ig = i - g0, jg = j - g1, kg = k - g2;
  int ig2 = i - 2 * g0, jg2 = j - 2 * g1, kg2 = k - 2 * g2;
  int ip = i + g0, jp = j + g1, kp = k + g2;
  int dir = (f + 1) / 2 - 1;
  R bv = beta_face ? (R)*beta_face : (F.sd ? beta_cell<R>(F, B, i, j, k) : (R)1);
  R dl_g1 = cell_length<R>(G, dir, ridx(B, ig, jg, kg));
  R dl_m = cell_length<R>(G, dir, ridx(B, i, j, k));
  R dl_4 = cell_length<R>(G, dir, ridx(B, ip, jp, kp));
  // the stencil in the order of the direction: ghost 2, ghost 1, the cell, its inner neighbour below a face of
  // odd number, the other way round above one of even number (one code for both: the records of a run's two
  // ends share warps)
  const bool odd = f % 2 == 1;
  const bool ig_inj = F.inj[gidx(B, ig, jg, kg)], ip_inj = F.inj[gidx(B, ip, jp, kp)];
  const R dl_out = dl_g1;                                               // ghost 2 to ghost 1
  const R dl_face = ig_inj ? (R)0.5*dl_m : odd ? (R)0.5*(dl_g1 + dl_m) : (R)0.5*(dl_m + dl_g1);
  const R dl_in = ip_inj ? (R)0.5*dl_m : odd ? (R)0.5*(dl_m + dl_4) : (R)0.5*(dl_4 + dl_m);
  const R half_g = ig_inj ? (R)0 : (R)0.5*dl_g1, half_m = (R)0.5*dl_m;
  const R dl0 = odd ? dl_out : dl_in, dl1 = dl_face, dl2 = odd ? dl_in : dl_out;
  const R dll = odd ? half_g : half_m, dlr = odd ? half_m : half_g;
  const long long step = odd ? gidx(B, ip, jp, kp) - gidx(B, i, j, k) : gidx(B, ig, jg, kg) - gidx(B, i, j, k);
  const long long a0 = odd ? gidx(B, ig2, jg2, kg2) : gidx(B, ip, jp, kp);
  const int c = dir == 0 ? i : dir == 1 ? j : k;
  const long long fi = fidx(B, dir, i, j, k, odd ? c : c + 1);         // the face below the cell, or above it
  R nrm[3], area;
  face_geometry<R>(G, dir, fi, nrm, area);
  const double* P = F.Up;
  R stn[4][nc], pl[nc], pr[nc], fl[nc];
#pragma unroll
  for (int s4 = 0; s4 < 4; ++s4)
#pragma unroll
    for (int v = 0; v < nc; ++v) stn[s4][v] = (R)P[(long long)v * G.NG + a0 + s4 * step];
  auto q = [&](int s, int v) { return stn[s][v]; };
  const bool bad = reconstruct<CL, LIM, R>(F.limiter, q, dl0, dl1, dl2, dll, dlr, pl, pr, bv);
  riemann<CL, RS, R>(pl, pr, nrm, fl, (R)F.mat.cp);
#pragma unroll
  for (int v = 0; v < nc; ++v) flux[v] = odd ? (double)(fl[v] * area) : (double)(-(fl[v] * area));
  return bad;
}

// ------------------------------------------------------------------ step control
// Locates the block of interior cell q (flat over every block) by binary search on ioff.
__device__ __forceinline__ int find_block(const DBlock* blk, int nb, long long q) {
  int lo = 0, hi = nb - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (blk[mid].ioff <= q) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// The indices of interior cell q of block B, by 32-bit arithmetic (a block has fewer than 2^31 cells; in 64 bits
// the divisions were half of the sensor kernel's instructions).
__device__ __forceinline__ void decode(const DBlock& B, long long q, int& i, int& j, int& k) {
  const unsigned l = (unsigned)(q - B.ioff), ni = (unsigned)B.ni, nj = (unsigned)B.nj, jk = l / ni;
  i = (int)(l % ni);
  j = (int)(jk % nj);
  k = (int)(jk / nj);
}

// compute_dt for every family in one pass (Mod_dt.f90:11-112, 256-275; Mod_Explicit.f90:46-61): each
// cell's metric rows are read once for all families; the cell's indices come from its block by 32-bit
// arithmetic (ice_gpu_create refuses a block of 2^31 cells or more). Per family the operations of
// compute_dt_ in its order; the global step is the smallest over every family and cell (an exact
// minimum, so the order of the families does not matter). Bound by its reads. The rows' unit vectors and
// moduli are formed once, when the metrics are set (k_rows: the scaled norm and the divisions were two
// thirds of the kernel's instructions), and the signal speeds' and the rate's quotients are branchless:
// A resident grid strides over the cells: one reduction and one atomic a CTA, not one per 256 cells, behind
// which the slot stood idle. IG, 128 x 126 x 129 cells: 122 us with the rows formed in the step, 89 with a CTA
// per 256 cells, 77 now.
// The minimum's start value, 1e+5 in single precision (Mod_Explicit.f90:40-44), as bits.
constexpr unsigned long long kDtStart = 0x40f86a0000000000ull;

struct DtFam {
  const double* Up;
  const double* tau;
  double* dt_out;   // the per-cell step (steady runs), or null
  int closure, coupled;
};
struct DtArgs {
  DtFam f[ICE_GPU_MAX_FAMILIES];
  int nf, ramp, ndir, time_accurate;
  double cfl, dt_max, tau_factor;
};

// The unit vector and the modulus of every metric row of the cells q0 .. q0 + n - 1, as compute_dt_ forms them.
__global__ void k_rows(const double* __restrict__ M, double* __restrict__ row, long long NI, long long q0, long long n) {
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const long long q = q0 + e;
    for (int d = 0; d < 3; ++d) {
      const double t0 = M[(long long)d * NI + q], t1 = M[(long long)(3 + d) * NI + q], t2 = M[(long long)(6 + d) * NI + q];
      const double g = norm2_3(t0, t1, t2);
      row[(long long)(4 * d) * NI + q] = t0 / g;
      row[(long long)(4 * d + 1) * NI + q] = t1 / g;
      row[(long long)(4 * d + 2) * NI + q] = t2 / g;
      row[(long long)(4 * d + 3) * NI + q] = g;
    }
  }
}

// The signal speeds of state p along the three rows (wavespeed of each).
template <int CL>
__device__ __forceinline__ void row_speeds(const double* p, const double (*vs)[4], double* ws) {
  if constexpr (CL == MK) {
    ws[0] = ws[1] = ws[2] = 0.0;
  } else if constexpr (CL == IG) {
    ws[0] = ws[1] = ws[2] = wavespeed<CL>(p, vs[0]);         // the same along every row
  } else {
    const double b = p[0] + epsv<double>(), y = ice_div_recip(b);
    bool ok = ice_div_by(b);
#pragma unroll
    for (int d = 0; d < 3; ++d) {                // (the rows beyond ndir are zero)
      const double* n = vs[d];
      const double pnn = n[0]*(p[4]*n[0] + p[5]*n[1] + p[6]*n[2]) +
                         n[1]*(p[5]*n[0] + p[7]*n[1] + p[8]*n[2]) +
                         n[2]*(p[6]*n[0] + p[8]*n[1] + p[9]*n[2]);
      const double a = 3.0*fmax(pnn, 0.0);
      ok = ok && dividend(a);
      ws[d] = sqrt(ice_div_quot(a, b, y));
    }
    if (!ok) {
#pragma unroll
      for (int d = 0; d < 3; ++d) ws[d] = wavespeed<CL>(p, vs[d]);
    }
  }
}

template <int CL>
__device__ __forceinline__ double family_dt(const Geo& G, const DtFam& f, const DtArgs& a, long long q, long long g,
                                            const double (*vs)[4], int it) {
  constexpr int nc = NC<CL>::v, used = CL == MK ? 4 : CL == IG ? 5 : 10;      // what a rate depends on
  double p[nc];
#pragma unroll
  for (int v = 0; v < used; ++v) p[v] = f.Up[(long long)v * G.NG + g];
  const bool bound = f.coupled && a.tau_factor > 0.0;
  const double tau = bound ? f.tau[q] : 0.0;     // with the state's loads, not after the rate
  double ws[3], rate = 0.0;
  row_speeds<CL>(p, vs, ws);
#pragma unroll
  for (int d = 0; d < 3; ++d)
    if (d < a.ndir) rate = rate + (fabs(p[1]*vs[d][0] + p[2]*vs[d][1] + p[3]*vs[d][2]) + ws[d]) * vs[d][3];
  double dt = (double)1e+5f;
  if (rate > 0.0) {
    bool ok = true;
    double r = quot(1.0, rate, ok);
    if (!ok) r = 1.0/rate;
    dt = mn(dt, r);
  }
  dt = dt * a.cfl;
  if (it <= a.ramp) dt = dt * (double)it / (double)a.ramp;
  dt = mn(dt, a.dt_max);
  if (bound && p[0] > kRhoEmpty && !not_finite(tau) && tau > 0.0) dt = mn(dt, a.tau_factor*tau);
  if (f.dt_out) f.dt_out[q] = dt;
  return dt;
}

// The end of the dt part of a step (Mod_Explicit.f90:40-44, 67-73): the step's dt, the time, the counters, and
// the minimum's start value for the next step.
__device__ __forceinline__ void finish_dt(Status* st, int time_accurate) {
  const double d = __longlong_as_double((long long)atomicAdd(&st->dtbits, 0ull));   // past L1: other CTAs' minima
  st->dtglobal = d;
  if (time_accurate) st->time = st->time + d;
  st->iter += 1;
  st->iter_from_call += 1;
  st->dtbits = kDtStart;
}

// finish: the last CTA to give its minimum ends the dt part (no bounds of imports or other ranks follow).
__global__ void __launch_bounds__(256, 4) k_dt_all(Geo G, DtArgs a, int finish, Status* st) {
  double dt = INFINITY;
  const int it = st->iter + 1;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < G.NI; q += (long long)gridDim.x * blockDim.x) {
    const int bq = find_block(G.blk, G.nb, q);
    if (!stepped(G, bq)) continue;
    const DBlock& B = G.blk[bq];
    int i, j, k;
    decode(B, q, i, j, k);
    const long long g = gidx(B, i, j, k);
    double vs[3][4];
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
      for (int m = 0; m < 4; ++m) vs[d][m] = d < a.ndir ? G.row[(long long)(4 * d + m) * G.NI + q] : 0.0;
    for (int p = 0; p < a.nf; ++p) {
      const DtFam& f = a.f[p];
      double d = f.closure == ICE_CLOSURE_MK ? family_dt<MK>(G, f, a, q, g, vs, it)
               : f.closure == ICE_CLOSURE_IG ? family_dt<IG>(G, f, a, q, g, vs, it)
                                             : family_dt<AG>(G, f, a, q, g, vs, it);
      dt = mn(dt, d);
    }
  }
  // warp and block min; a positive double orders as its bits
  unsigned long long bits = (unsigned long long)__double_as_longlong(dt);
  for (int o = 16; o > 0; o >>= 1) bits = min(bits, __shfl_xor_sync(0xffffffffu, bits, o));
  __shared__ unsigned long long wmin[8];
  if ((threadIdx.x & 31) == 0) wmin[threadIdx.x >> 5] = bits;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long m = wmin[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = min(m, wmin[w]);
    atomicMin(&st->dtbits, m);
    if (finish) {
      __threadfence();
      if (atomicAdd(&st->done, 1u) == gridDim.x - 1) {
        __threadfence();
        st->done = 0u;
        finish_dt(st, a.time_accurate);
      }
    }
  }
}

__global__ void k_time(Status* st, int time_accurate) {
  finish_dt(st, time_accurate);
}

// The rate of compute_dt_ (Mod_dt.f90:256-275): sum over the resolved directions of (|u . versor| +
// the closure's signal speed) times the modulus of the metric row, for the state p of cell q.
template <int CL>
__device__ __forceinline__ double dt_rate(const Geo& G, long long q, const double* p, int ndir) {
  double rate = 0.0;
  for (int d = 0; d < ndir; ++d) {
    double t0 = G.M[(long long)d * G.NI + q], t1 = G.M[(long long)(3 + d) * G.NI + q], t2 = G.M[(long long)(6 + d) * G.NI + q];
    double gn = norm2_3(t0, t1, t2);
    double vs[3] = {t0 / gn, t1 / gn, t2 / gn};
    rate = rate + (fabs(p[1]*vs[0] + p[2]*vs[1] + p[3]*vs[2]) + wavespeed<CL>(p, vs)) * gn;
  }
  return rate;
}

__global__ void k_empty_init(EmptyScan* e) {
  e->floor_bits = (unsigned long long)__double_as_longlong(1.79769313486231570e+308);
  e->src_bits = e->floor_bits;
  e->umax_bits[0] = e->umax_bits[1] = e->umax_bits[2] = 0ULL;
  e->filled = 0u;
}

// bound_empty_dt's first pass (Mod_dt.f90:134-196) over one family's cells, with the coupler's
// imports as the only source: an occupied cell (density above rho_empty) gives its step and speeds;
// an empty cell with a positive mass rate gives the speeds of what it receives (the rate's momentum
// over its mass) and the step of compute_dt_ at that speed, times cfl.
template <int CL>
__global__ void __launch_bounds__(256) k_empty_scan(Geo G, FamDev F, const double* dt_cell, double cfl, int ndir,
                                                    EmptyScan* e) {
  long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= G.NI) return;
  const DBlock& B = G.blk[find_block(G.blk, G.nb, q)];
  int i, j, k; decode(B, q, i, j, k);
  constexpr int nc = NC<CL>::v;
  const long long g = gidx(B, i, j, k);
  double p[nc];
#pragma unroll
  for (int v = 0; v < nc; ++v) p[v] = F.Up[(long long)v * G.NG + g];
  double s[4];
#pragma unroll
  for (int v = 0; v < 4; ++v) s[v] = F.imports[(long long)v * G.NI + q];
  if (s[0] > 0.0) atomicOr(&e->filled, 1u);
  if (p[0] > kRhoEmpty) {
    if (dt_cell) atomicMin(&e->floor_bits, (unsigned long long)__double_as_longlong(dt_cell[q]));
    for (int a = 0; a < 3; ++a) atomicMax(&e->umax_bits[a], (unsigned long long)__double_as_longlong(fabs(p[1 + a])));
    return;
  }
  if (!(s[0] > 0.0)) return;
  p[1] = s[1]/s[0]; p[2] = s[2]/s[0]; p[3] = s[3]/s[0];
  for (int a = 0; a < 3; ++a) atomicMax(&e->umax_bits[a], (unsigned long long)__double_as_longlong(fabs(p[1 + a])));
  double dts = (double)1e+5f;
  const double rate = dt_rate<CL>(G, q, p, ndir);
  if (rate > 0.0) dts = mn(dts, 1.0/rate);
  atomicMin(&e->src_bits, (unsigned long long)__double_as_longlong(dts*cfl));
}

// bound_empty_dt's second pass (Mod_dt.f90:197-214) and bound_removal_dt (Mod_dt.f90:220-242). Time-
// accurate: the global step lowered to the sources' step (when a source fills anything) and to each
// cell's removal step (its density over the rate the coupler takes out). Steady: each empty cell's
// step lowered to the smaller of the occupied cells' smallest step and the sources', and to cfl over
// its rate at the largest speeds; each cell's to its removal step. Only minima: the order of the two
// bounds does not change a bit.
template <int CL>
__global__ void __launch_bounds__(256) k_empty_apply(Geo G, FamDev F, double* dt_cell, double cfl, int ndir,
                                                     const EmptyScan* e, Status* st) {
  long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= G.NI) return;
  const DBlock& B = G.blk[find_block(G.blk, G.nb, q)];
  int i, j, k; decode(B, q, i, j, k);
  const double rho = F.Up[gidx(B, i, j, k)];
  const bool filled = e->filled != 0u;
  const double src_dt = __longlong_as_double((long long)e->src_bits);
  if (!dt_cell) {                                    // time-accurate
    if (q == 0 && filled) atomicMin(&st->dtbits, e->src_bits);
  } else if (filled && !(rho > kRhoEmpty)) {
    const double floor_dt = mn(__longlong_as_double((long long)e->floor_bits), src_dt);
    double umax[3];
    for (int a = 0; a < 3; ++a) umax[a] = __longlong_as_double((long long)e->umax_bits[a]);
    double rate = 0.0;
    for (int d = 0; d < ndir; ++d) {
      double sum = umax[0]*fabs(G.M[(long long)d * G.NI + q]);
      sum = sum + umax[1]*fabs(G.M[(long long)(3 + d) * G.NI + q]);
      sum = sum + umax[2]*fabs(G.M[(long long)(6 + d) * G.NI + q]);
      rate = rate + sum;
    }
    double dts = floor_dt;
    if (rate > 0.0) dts = mn(dts, cfl/rate);
    dt_cell[q] = mn(dt_cell[q], dts);
  }
  const double out = -F.imports[q];
  if (!(out > 0.0)) return;
  const double dts = rho/out;
  if (!dt_cell) atomicMin(&st->dtbits, (unsigned long long)__double_as_longlong(dts));
  else dt_cell[q] = mn(dt_cell[q], dts);
}

// ------------------------------------------------------------------ ghosts
__device__ __forceinline__ int ghost_rule(const DRec& r, double veln) {
  int rule = 0;  // copy
  if (r.type == 200) rule = 1;
  else if (r.type == 300 || r.type == 301) {
    if (veln*(double)(1 - 2*(r.f % 2)) <= 0.0 || r.f == 3) rule = 1;
  } else if (r.type >= 401 && r.type <= 403) {
    if (!(veln*(double)(1 - 2*(r.f % 2)) > 0.0)) {
      rule = 2;
      if (r.massflux == 0.0) rule = 1;
    }
  }
  return rule;
}

__device__ __forceinline__ void rec_normal(const Geo& G, const DBlock& B, const DRec& r, double* n, double* area) {
  int d = (r.f - 1) / 2;
  int F = (d == 0 ? r.i : d == 1 ? r.j : r.k) + 1 - (r.f % 2);   // im - mod(fm,2), 1-based
  long long fi = fidx(B, d, r.i, r.j, r.k, F);
  long long NF = G.NF[d];
  n[0] = G.face[d][fi]; n[1] = G.face[d][NF + fi]; n[2] = G.face[d][2 * NF + fi];
  if (area) *area = G.face[d][3 * NF + fi];
}

// ghost_chimera (Lib_Ghost.f90:439-466): ghost cell gg (layer 1 or 2) of a chimera record from its
// donors, the weighted sum of their conservative states in donor order, back to primitive with the
// closure's floors. The donors are interior cells, which no ghost fill writes.
template <int CL>
__device__ __forceinline__ void chimera_ghost(const Geo& G, const FamDev& F, const DRec& r, int layer, long long gg) {
  constexpr int nc = NC<CL>::v;
  const double* P = F.Ug;
  const long long NG = G.NG;
  const int d0 = r.cd0 + (layer == 1 ? 0 : r.cn1), d1 = d0 + (layer == 1 ? r.cn1 : r.cn2);
  double cs[nc];
#pragma unroll
  for (int v = 0; v < nc; ++v) cs[v] = 0.0;
  for (int d = d0; d < d1; ++d) {
    const int4 dn = F.cdon[d];
    const long long gd = gidx(G.blk[dn.x], dn.y, dn.z, dn.w);
    const double w = F.cw[d];
    double pd[nc], cd[nc];
#pragma unroll
    for (int v = 0; v < nc; ++v) pd[v] = P[v * NG + gd];
    prim2cons<CL, double>(pd, cd, F.mat.cp);
#pragma unroll
    for (int v = 0; v < nc; ++v) cs[v] = cs[v] + w*cd[v];
  }
  double pg[nc];
  cons2prim<CL>(cs, pg, F.mat.cp);
#pragma unroll
  for (int v = 0; v < nc; ++v) F.Ug[v * NG + gg] = pg[v];
}

// ghost_record (Lib_Ghost.f90:76-267)
template <int CL>
__device__ __forceinline__ void ghost1_rec(const Geo& G, const FamDev& F, const DRec& r) {
  constexpr int nc = NC<CL>::v;
  const DBlock& B = G.blk[r.b];
  int g0 = (r.f == 1) - (r.f == 2), g1 = (r.f == 3) - (r.f == 4), g2 = (r.f == 5) - (r.f == 6);
  long long gg = gidx(B, r.i - g0, r.j - g1, r.k - g2);
  long long gm = gidx(B, r.i, r.j, r.k);
  double* P = F.Ug;
  const long long NG = G.NG;
  switch (r.type) {
    case 101: case 201: {
      const DBlock& S = G.blk[r.bs];
      long long gs = gidx(S, r.is, r.js, r.ks);
#pragma unroll
      for (int v = 0; v < nc; ++v) P[v * NG + gg] = P[v * NG + gs];
      break;
    }
    case 200: case 300: case 301: {
      double nrm[3]; rec_normal(G, B, r, nrm, nullptr);
      double m[nc];
#pragma unroll
      for (int v = 0; v < nc; ++v) m[v] = P[v * NG + gm];
      double gv[nc];
#pragma unroll
      for (int v = 0; v < nc; ++v) gv[v] = m[v];
      double vel[3] = {m[1], m[2], m[3]};
      double veln = vel[0]*nrm[0] + vel[1]*nrm[1] + vel[2]*nrm[2];
      if (ghost_rule(r, veln) == 1) {
        for (int a = 0; a < 3; ++a) vel[a] = vel[a] - 2.0*veln*nrm[a];
        if constexpr (CL == AG) mirror_tensor(m + 4, nrm, gv + 4);
      }
      gv[1] = vel[0]; gv[2] = vel[1]; gv[3] = vel[2];
#pragma unroll
      for (int v = 0; v < nc; ++v) P[v * NG + gg] = gv[v];
      break;
    }
    case 0: case 400: {
#pragma unroll
      for (int v = 0; v < nc; ++v) P[v * NG + gg] = P[v * NG + gm];
      break;
    }
    case 401: case 402: case 403: {
      double nrm[3]; rec_normal(G, B, r, nrm, nullptr);
      double m[nc];
#pragma unroll
      for (int v = 0; v < nc; ++v) m[v] = P[v * NG + gm];
      double vel[3] = {m[1], m[2], m[3]};
      double veln = vel[0]*nrm[0] + vel[1]*nrm[1] + vel[2]*nrm[2];
      int rule = ghost_rule(r, veln);
      F.inj[gg] = (rule == 2);
      double gv[nc];
      if (rule == 0) {
#pragma unroll
        for (int v = 0; v < nc; ++v) gv[v] = m[v];
      } else if (rule == 1) {
#pragma unroll
        for (int v = 0; v < nc; ++v) gv[v] = m[v];
        for (int a = 0; a < 3; ++a) vel[a] = vel[a] - 2.0*veln*nrm[a];
        gv[1] = vel[0]; gv[2] = vel[1]; gv[3] = vel[2];
        if constexpr (CL == AG) mirror_tensor(m + 4, nrm, gv + 4);
      } else {
#pragma unroll
        for (int v = 0; v < nc; ++v) gv[v] = 0.0;
        double sgn = (double)(2*(r.f % 2) - 1);
        double inward[3] = {sgn*nrm[0], sgn*nrm[1], sgn*nrm[2]};
        long long q = iidx(B, r.i, r.j, r.k);
        const double* gas = G.gas;
        double v3[3], speed;
        auto injv = [&](double sp) {
          if (r.normal_dir) { v3[0] = sp*inward[0]; v3[1] = sp*inward[1]; v3[2] = sp*inward[2]; }
          else { v3[0] = sp*r.cb*r.ca; v3[1] = sp*r.cb*r.sa; v3[2] = sp*r.sb; }
        };
        if (r.type == 401) {
          double gu = gas[1 * G.NI + q], gvv = gas[2 * G.NI + q], gw = gas[3 * G.NI + q];
          double vn = gu*inward[0] + gvv*inward[1] + gw*inward[2];
          injv(r.velocity*vn);
          gv[1] = v3[0]; gv[2] = v3[1]; gv[3] = v3[2];
          gv[0] = r.massflux*gas[q]/r.velocity;
          vn = fabs(gv[1]*nrm[0] + gv[2]*nrm[1] + gv[3]*nrm[2]);
          if (r.gfixed > 0.0 && vn > 0.0) gv[0] = gv[0] + r.massflux*r.gfixed/vn;
          gv[nc - 2] = r.temperature*gas[4 * G.NI + q];
        } else if (r.type == 402) {
          injv(r.velocity);
          gv[1] = v3[0]; gv[2] = v3[1]; gv[3] = v3[2];
          double vn = gv[1]*nrm[0] + gv[2]*nrm[1] + gv[3]*nrm[2];
          gv[0] = r.massflux/fabs(vn);
          gv[nc - 2] = r.temperature;
        } else {
          speed = norm2_3(gas[1 * G.NI + q], gas[2 * G.NI + q], gas[3 * G.NI + q]);
          injv(r.velocity*speed);
          gv[1] = v3[0]; gv[2] = v3[1]; gv[3] = v3[2];
          double vn = gv[1]*nrm[0] + gv[2]*nrm[1] + gv[3]*nrm[2];
          gv[0] = r.massflux/fabs(vn);
          gv[nc - 2] = r.temperature;
        }
        gv[nc - 1] = gv[0]/F.mat.rho/r.vol_p;
        if constexpr (CL == IG) gv[4] = 1e-6;
        if constexpr (CL == AG) { gv[4] = 1e-6; gv[7] = 1e-6; gv[9] = 1e-6; }
      }
#pragma unroll
      for (int v = 0; v < nc; ++v) P[v * NG + gg] = gv[v];
      break;
    }
    case 102:
      chimera_ghost<CL>(G, F, r, 1, gg);
      break;
    default: break;
  }
}

// second_ghost_record (Lib_Ghost.f90:312-387)
template <int CL>
__device__ __forceinline__ void ghost2_rec(const Geo& G, const FamDev& F, const DRec& r) {
  constexpr int nc = NC<CL>::v;
  if (r.type == 0) return;
  const DBlock& B = G.blk[r.b];
  int g0 = (r.f == 1) - (r.f == 2), g1 = (r.f == 3) - (r.f == 4), g2 = (r.f == 5) - (r.f == 6);
  long long gg1 = gidx(B, r.i - g0, r.j - g1, r.k - g2);
  long long gg2 = gidx(B, r.i - 2 * g0, r.j - 2 * g1, r.k - 2 * g2);
  long long gm = gidx(B, r.i, r.j, r.k);
  long long gp = gidx(B, r.i + g0, r.j + g1, r.k + g2);
  double* P = F.Ug;
  const long long NG = G.NG;
  switch (r.type) {
    case 101: case 201: {
      const DBlock& S = G.blk[r.bs];
      int s0 = (r.fs == 1) - (r.fs == 2), s1 = (r.fs == 3) - (r.fs == 4), s2 = (r.fs == 5) - (r.fs == 6);
      long long gs = gidx(S, r.is + s0, r.js + s1, r.ks + s2);
#pragma unroll
      for (int v = 0; v < nc; ++v) P[v * NG + gg2] = P[v * NG + gs];
      break;
    }
    case 200: case 300: case 301: case 401: case 402: case 403: {
      double nrm[3]; rec_normal(G, B, r, nrm, nullptr);
      double m1 = P[1 * NG + gm], m2 = P[2 * NG + gm], m3 = P[3 * NG + gm];
      double veln = m1*nrm[0] + m2*nrm[1] + m3*nrm[2];
      int rule = ghost_rule(r, veln);
      double gv[nc];
      if (rule == 2) {
#pragma unroll
        for (int v = 0; v < nc; ++v) gv[v] = P[v * NG + gg1];
      } else {
        double mp[nc];
#pragma unroll
        for (int v = 0; v < nc; ++v) { mp[v] = P[v * NG + gp]; gv[v] = mp[v]; }
        if (rule == 1) {
          double d = mp[1]*nrm[0] + mp[2]*nrm[1] + mp[3]*nrm[2];
          for (int a = 0; a < 3; ++a) gv[1 + a] = mp[1 + a] - 2.0*d*nrm[a];
          if constexpr (CL == AG) mirror_tensor(mp + 4, nrm, gv + 4);
        }
      }
#pragma unroll
      for (int v = 0; v < nc; ++v) P[v * NG + gg2] = gv[v];
      break;
    }
    case 102:
      chimera_ghost<CL>(G, F, r, 2, gg2);
      break;
    default: {
#pragma unroll
      for (int v = 0; v < nc; ++v) P[v * NG + gg2] = 3.0*P[v * NG + gg1] - 3.0*P[v * NG + gm] + P[v * NG + gp];
      break;
    }
  }
}

// The ghost layers of every record, one thread per record; layers: 1 the first, 2 the second, 3 both.
// compute_ghost fills layer 1 of every record and then fill_second_ghost layer 2 (Lib_Ghost.f90:29-387).
// A record's layer 2 reads its own layer-1 cell and the cell one further inside (of its block, or of the
// source block of a connection). Where that block is two cells or more deep along the record's face
// direction the cell is interior, no other record writes it, and one thread does both layers in turn
// (layers = 3). Where it is one cell deep the cell is the opposite face's layer-1 ghost, which another
// record writes: then the host launches layer 1 of every record first and layer 2 after it.
// The copying records (layers = 3) come as GhostCopy: every load first, then every store, the values and
// operations of ghost1_rec followed by ghost2_rec (layer 2 of a 400 record, 3 g1 - 3 m + p, with g1 the layer-1
// value just copied from m). Bound by the records' and cells' bytes: on a 509 x 512 plane, whose 260,608 cells
// have two k faces each, reading the whole record cost 34 us a launch.
// An AG thread takes a third of a record's variables, so that more of them wait on memory at once: 45 / 35 us on
// 8 blocks of 1.7 M cells; MK and IG in two parts gained nothing there and lost 20 % on the plane.
template <int CL> struct GhostPart {
  static constexpr int n = CL == AG ? 3 : 1, nv = (NC<CL>::v + n - 1) / n;
};

template <int CL>
__device__ __forceinline__ void ghost_copy(double* P, long long NG, const GhostCopy& c, bool ext, int v0) {
  constexpr int nv = GhostPart<CL>::nv, nc = NC<CL>::v;
  double a[nv], b[nv];
  const bool two = c.g2 != kNoGhost;
  P += (long long)v0 * NG;
#pragma unroll
  for (int v = 0; v < nv; ++v) if (v0 + v < nc) a[v] = P[v * NG + c.m];
  if (two) {
#pragma unroll
    for (int v = 0; v < nv; ++v) if (v0 + v < nc) b[v] = P[v * NG + c.p];
  }
#pragma unroll
  for (int v = 0; v < nv; ++v) if (v0 + v < nc) P[v * NG + c.g1] = a[v];
  if (two) {
#pragma unroll
    for (int v = 0; v < nv; ++v) if (v0 + v < nc) P[v * NG + c.g2] = ext ? 3.0*a[v] - 3.0*a[v] + b[v] : b[v];
  }
}

// The first nrb CTAs take the records, the others the copies, part by part.
template <int CL>
__global__ void k_ghost(Geo G, FamDev F, const DRec* recs, int nrec, int nrb, int layers, const GhostCopy* copies, int ncopy,
                        int next) {
  if ((int)blockIdx.x >= nrb) {
    const int ncb = (gridDim.x - nrb) / GhostPart<CL>::n, cb = blockIdx.x - nrb;
    const int n = (cb % ncb) * blockDim.x + threadIdx.x;
    if (n < ncopy) ghost_copy<CL>(F.Ug, G.NG, copies[n], n < next, cb / ncb * GhostPart<CL>::nv);
    return;
  }
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= nrec) return;
  const int run = recs[n].run;                   // a face listed more than once: its records in table order
  if (!stepped(G, recs[n].b)) return;
  if (layers & 1) for (int m = 0; m < run; ++m) ghost1_rec<CL>(G, F, recs[n + m]);
  if (layers & 2) for (int m = 0; m < run; ++m) ghost2_rec<CL>(G, F, recs[n + m]);
}

// ------------------------------------------------------------------ boundary fluxes
// A split run's BETA exchange: the Jameson weight of each listed cell (0-based block, i, j, k), as the
// record kernel of the same precision and translation unit evaluates it (rec_face).
template <typename R>
__global__ void k_pack_beta(Geo G, FamDev F, const int4* __restrict__ e, int n, double* __restrict__ out) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const int4 x = e[q];
  out[q] = F.sd ? (double)beta_cell<R>(F, G.blk[x.x], x.y, x.z, x.w) : 1.0;
}

// The place of the face f of the 0-based cell (i, j, k) in its direction's flux array.
__device__ __forceinline__ long long face_place(const DBlock& B, int f, int i, int j, int k) {
  const int d = (f - 1) / 2, c = d == 0 ? i : d == 1 ? j : k;
  return fidx(B, d, i, j, k, f % 2 == 1 ? c : c + 1);
}

// The flux x into a cell through its face f, stored as the cells' update reads it: added from the face below
// the cell, taken off from the face above it.
template <int CL, typename R>
__device__ __forceinline__ void put_flux(const Geo& G, const FamDev& F, const DBlock& B, int f, int i, int j, int k,
                                         const double* x, double sign) {
  constexpr int nc = NC<CL>::v;
  const int d = (f - 1) / 2;
  R* out = (R*)F.Ff[d] + face_place(B, f, i, j, k);
  const double s = f % 2 == 1 ? sign : -sign;
#pragma unroll
  for (int v = 0; v < nc; ++v) out[(long long)v * G.NF[d]] = (R)(s * x[v]);
}

// The flux through one boundary record's face (Mod_BC_Fluxes.f90:105-170); a connection's is computed by the
// owner, with the smaller of the two cells' Jameson weights, for both cells.
template <int CL, int RS, int LIM, typename R>
__device__ __forceinline__ bool rec_face(const Geo& G, const FamDev& F, const DRec* recs, int rec) {
  constexpr int nc = NC<CL>::v;
  const DRec& r = recs[rec];
  if (!stepped(G, r.b)) return false;
  double fl[nc];
  double bf = 0.0;
  const bool conn = r.type == 101 || r.type == 201;
  if (conn) {
    R bo = (R)1, bq = (R)1;
    if (F.sd) {
      bo = beta_cell<R>(F, G.blk[r.b], r.i, r.j, r.k);
      // a partner in a block another rank steps: its weight, which that rank sent (ICE_GPU_HALO_BETA)
      bq = stepped(G, r.pb) ? beta_cell<R>(F, G.blk[r.pb], r.pi, r.pj, r.pk)
                            : (R)F.beta[iidx(G.blk[r.pb], r.pi, r.pj, r.pk)];
    }
    bf = (double)mn(bo, bq);
  }
  const bool bad = record_flux<CL, RS, LIM, R>(G, F, r, fl, conn ? &bf : nullptr);
  if (!r.summed) put_flux<CL, R>(G, F, G.blk[r.b], r.f, r.i, r.j, r.k, fl, 1.0);
  if (conn) {
    if (r.pf) put_flux<CL, R>(G, F, G.blk[r.pb], r.pf, r.pi, r.pj, r.pk, fl, -1.0);
    if (F.connF) {
#pragma unroll
      for (int v = 0; v < nc; ++v) F.connF[(long long)r.cf * nc + v] = fl[v];
    }
  }
  return bad;
}

// Thread n of the records' fluxes: record frec[n], or after them the faces that only another family's records
// give a flux (FamDev::zface).
template <int CL, int RS, int LIM, typename R>
__device__ __forceinline__ bool rec_thread(const Geo& G, const FamDev& F, const DRec* recs, const int* frec, int nfrec, int n) {
  if (n < nfrec) return rec_face<CL, RS, LIM, R>(G, F, recs, frec[n]);
  if (n - nfrec < F.nzface) {
    const ZeroFace z = F.zface[n - nfrec];
#pragma unroll
    for (int v = 0; v < NC<CL>::v; ++v) ((R*)F.Ff[z.d])[(long long)v * G.NF[z.d] + z.at] = (R)0;
  }
  return false;
}

// A split run: the fluxes of the connections whose owner another rank steps, as that rank sent them
// (ICE_GPU_HALO_FLUX).
template <int CL, typename R>
__global__ void k_conn_in(Geo G, FamDev F, const DRec* recs, int nrec) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= nrec) return;
  const DRec& r = recs[n];
  if ((r.type != 101 && r.type != 201) || r.owner || !stepped(G, r.b) || stepped(G, r.pb)) return;
  put_flux<CL, R>(G, F, G.blk[r.b], r.f, r.i, r.j, r.k, F.connF + (long long)r.cf * NC<CL>::v, -1.0);
}

template <int CL, int RS, int LIM, typename R>
__global__ void __launch_bounds__(128, 4) k_rec(Geo G, FamDev F, const DRec* recs, const int* frec, int nfrec, Status* st) {
  if (rec_thread<CL, RS, LIM, R>(G, F, recs, frec, nfrec, blockIdx.x * blockDim.x + threadIdx.x))
    atomicOr(&st->flags, (unsigned)ICE_GPU_ST_BAD_RECON);
}

// The cells of a table that lists one of their faces more than once, or a connection that is not one owner and its one
// partner: every record of the cell in the order of faces and table (bound_cell, Mod_BC_Fluxes.f90:105-144), connections from
// connF. Such a cell's boundary fluxes are wanted for their sum alone: it goes to the first of its boundary faces,
// zeros to the others. parts = 3: what a float leaves of it to the next two (the FP32-flux form's 1-D runs, whose cells sum in
// FP64 and have four faces or more there). Runs after the record and flux kernels and after a split run's exchange.
template <int CL, int RS, typename R>
__global__ void __launch_bounds__(128, 4) k_cell_sum(Geo G, FamDev F, const DRec* recs, const int* first, const int* list, int n,
                                                     int parts, Status* st) {
  constexpr int nc = NC<CL>::v;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  const DRec& o = recs[list[first[c]]];
  if (!stepped(G, o.b)) return;
  double acc[nc];
#pragma unroll
  for (int v = 0; v < nc; ++v) acc[v] = 0.0;
  bool bad = false;
  for (int m = first[c]; m < first[c + 1]; ++m) {
    const DRec& r = recs[list[m]];
    double fl[nc];
    if (r.type == 101 || r.type == 201) {
#pragma unroll
      for (int v = 0; v < nc; ++v) { const double x = F.connF[(long long)r.cf * nc + v]; fl[v] = r.owner ? x : -x; }
    } else {
      bad |= record_flux<CL, RS, LIM_ANY, R>(G, F, r, fl, nullptr);
    }
#pragma unroll
    for (int v = 0; v < nc; ++v) acc[v] = acc[v] + fl[v];
  }
  const DBlock& B = G.blk[o.b];
  for (int f = 1; f <= 6; ++f) {
    const int d = (f - 1) / 2, x = d == 0 ? o.i : d == 1 ? o.j : o.k, len = d == 0 ? B.ni : d == 1 ? B.nj : B.nk;
    if (x != (f % 2 == 1 ? 0 : len - 1)) continue;
    double part[nc];
#pragma unroll
    for (int v = 0; v < nc; ++v) {
      part[v] = parts > 0 ? (double)(R)acc[v] : 0.0;
      acc[v] = not_finite(part[v]) ? 0.0 : acc[v] - part[v];
    }
    put_flux<CL, R>(G, F, B, f, o.i, o.j, o.k, part, 1.0);
    --parts;
  }
  if (bad) atomicOr(&st->flags, (unsigned)ICE_GPU_ST_BAD_RECON);
}

// The sum of a cell's boundary fluxes in face order: lo(d, v), hi(d, v) the fluxes of the faces below and above
// it along d.
template <int nc, typename LoFn, typename HiFn>
__device__ __forceinline__ void edge_sum(const DBlock& B, int i, int j, int k, double* acc, const LoFn& lo, const HiFn& hi) {
#pragma unroll
  for (int v = 0; v < nc; ++v) {
    double a = 0.0;
    if (i == 0) a = a + (double)lo(0, v);
    if (i == B.ni - 1) a = a - (double)hi(0, v);
    if (j == 0) a = a + (double)lo(1, v);
    if (j == B.nj - 1) a = a - (double)hi(1, v);
    if (k == 0) a = a + (double)lo(2, v);
    if (k == B.nk - 1) a = a - (double)hi(2, v);
    acc[v] = a;
  }
}

// ------------------------------------------------------------------ the stage

// compute_source (Mod_Sources.f90:19-72): the source of every cell of one family, from the state
// at the start of the stage and the frozen gas; written to S (and tau, on the last stage), which
// the stage kernel adds to the residual. Its own kernel, so that the iterative closures do not
// share the stencil kernel's registers.
// Bound by its chains (four to six powers, the Langmuir-Knudsen iteration), so it wants warps: 64 registers
// (4 CTAs per SM) against 80 and 128 (3, 2) take 82 / 91 / 95 us in FP64 (evaporating AG, 64 x 61 x 67) although
// some spill (74 / 74 / 86 us for IG without evaporation, 96 x 95 x 97).
template <int CL, typename R>
__global__ void __launch_bounds__(256, 4) k_source(Geo G, FamDev F) {
  constexpr int nc = NC<CL>::v;
  long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= G.NI) return;
  const int bq = find_block(G.blk, G.nb, q);
  if (!stepped(G, bq)) return;
  const DBlock& B = G.blk[bq];
  const unsigned l = (unsigned)(q - B.ioff), ni = (unsigned)B.ni, nj = (unsigned)B.nj;   // < 2^31 cells a block
  const unsigned i = l % ni, jk = l / ni, j = jk % nj, k = jk / nj;
  const long long g = gidx(B, (int)i, (int)j, (int)k);
  R p[nc], gas[5], s[nc];
#pragma unroll
  for (int v = 0; v < nc; ++v) p[v] = (R)F.Up[(long long)v * G.NG + g];
  R gr[9];
#pragma unroll
  for (int v = 0; v < 9; ++v) gr[v] = sizeof(R) == 4 ? (R)G.gasf[(long long)v * G.NI + q] : (R)G.gas[(long long)v * G.NI + q];
#pragma unroll
  for (int v = 0; v < 5; ++v) gas[v] = gr[v];
  R tau = cell_source<CL, R>(p, gas, gr[5], gr[6], gr[7], gr[8], F.mat, F.drag, F.heat, F.blow, s);
  if constexpr (sizeof(R) == 4) {
#pragma unroll
    for (int v = 0; v < nc; ++v) F.Sf[(long long)v * G.NI + q] = (F.frozen_mask & (1u << v)) ? 0.f : s[v];
  } else {
#pragma unroll
    for (int v = 0; v < nc; ++v) F.S[(long long)v * G.NI + q] = (F.frozen_mask & (1u << v)) ? 0.0 : (double)s[v];
  }
  if (F.write_tau) F.tau[q] = (double)tau;
}

// The stage kernel of the FP32-flux form's 1-D runs, whose residual sums and divisions are FP64. One CTA of
// TX x TY threads (256) owns a column tile of one block and marches up a chunk of KZ planes. On each
// plane every thread computes exactly one x face (the face below
// its cell), one y face and one z face (the face above its cell; the one below comes from the
// plane before, or is computed once at the chunk's first plane) into shared memory, so the work is
// the same for every thread; then each cell of the tile's (TX-1) x (TY-1) interior takes its two
// faces per direction in the reference's odd-then-even order (Mod_Fluxes.f90:470-506), adds the
// source, forms R = (R/vol + S) dt, and applies the RK stage in conservative variables with the
// reference's floors and checks (Lib_Newstate.f90:198-219).
#ifndef ICE_STAGE_MINB
#define ICE_STAGE_MINB 1      // resident CTAs per SM the register allocation is held to
#endif
template <int CL, int RS, int LIM, typename R>
__global__ void __launch_bounds__(256, ICE_STAGE_MINB)
k_stage(Geo G, FamDev F, const Tile* tiles, int TX, int TY, int KZ, Status* st) {
  constexpr int nc = NC<CL>::v;
  extern __shared__ double smem[];
  const int NT = TX * TY;
  double* Fx = smem;                  // [nc][NT]
  double* Fy = smem + nc * NT;
  double* Fz0 = smem + 2 * nc * NT;
  double* Fz1 = smem + 3 * nc * NT;
  const Tile t = tiles[blockIdx.x];
  const DBlock& B = G.blk[t.b];
  const int tid = threadIdx.x;
  const int tx = tid % TX, ty = tid / TX;
  const int i = t.i0 + tx, j = t.j0 + ty;
  const bool ax = B.ni >= 2, ay = B.nj >= 2, az = B.nk >= 2;
  const bool col = i < B.ni && j < B.nj;
  const bool owner = col && (ax ? tx < TX - 1 : tx == 0) && (ay ? ty < TY - 1 : ty == 0);
  const int k1 = min(t.k0 + KZ, B.nk);
  bool bad = false;
  double* flo = Fz0;
  double* fhi = Fz1;
  if (az && col && t.k0 >= 1) {       // the face below the chunk's first plane
    R fl[nc];
    bad |= face_flux<CL, RS, LIM, R>(G, F, B, 2, i, j, t.k0 - 1, fl);
#pragma unroll
    for (int v = 0; v < nc; ++v) flo[v * NT + tid] = (double)fl[v];
  }
  for (int k = t.k0; k < k1; ++k) {
    if (ax && col && i >= 1) {        // x face below (i,j,k)
      R fl[nc];
      bad |= face_flux<CL, RS, LIM, R>(G, F, B, 0, i - 1, j, k, fl);
#pragma unroll
      for (int v = 0; v < nc; ++v) Fx[v * NT + tid] = (double)fl[v];
    }
    if (ay && col && j >= 1) {        // y face below (i,j,k)
      R fl[nc];
      bad |= face_flux<CL, RS, LIM, R>(G, F, B, 1, i, j - 1, k, fl);
#pragma unroll
      for (int v = 0; v < nc; ++v) Fy[v * NT + tid] = (double)fl[v];
    }
    if (az && col && k <= B.nk - 2) { // z face above (i,j,k)
      R fl[nc];
      bad |= face_flux<CL, RS, LIM, R>(G, F, B, 2, i, j, k, fl);
#pragma unroll
      for (int v = 0; v < nc; ++v) fhi[v * NT + tid] = (double)fl[v];
    }
    __syncthreads();
    if (owner) {
      const long long q = iidx(B, i, j, k);
      double r[nc];
      edge_sum<nc>(B, i, j, k, r, [&](int d, int v) {
        return ((const R*)F.Ff[d])[(long long)v * G.NF[d] + fidx(B, d, i, j, k, d == 0 ? i : d == 1 ? j : k)];
      }, [&](int d, int v) {
        return ((const R*)F.Ff[d])[(long long)v * G.NF[d] + fidx(B, d, i, j, k, (d == 0 ? i : d == 1 ? j : k) + 1)];
      });
      // direction 1: face tid+1 is the cell's upper face, face tid its lower one
      if (ax) {
        const int ci = i + 1, n = B.ni;
        if (ci % 2 == 1) {
          if (ci < n) {
#pragma unroll
            for (int v = 0; v < nc; ++v) r[v] = r[v] - Fx[v * NT + tid + 1];
          }
          if (ci > 1) {
#pragma unroll
            for (int v = 0; v < nc; ++v) r[v] = r[v] + Fx[v * NT + tid];
          }
        } else {
#pragma unroll
          for (int v = 0; v < nc; ++v) r[v] = r[v] + Fx[v * NT + tid];
          if (ci < n) {
#pragma unroll
            for (int v = 0; v < nc; ++v) r[v] = r[v] - Fx[v * NT + tid + 1];
          }
        }
      }
      if (ay) {
        const int cj = j + 1, n = B.nj;
        if (cj % 2 == 1) {
          if (cj < n) {
#pragma unroll
            for (int v = 0; v < nc; ++v) r[v] = r[v] - Fy[v * NT + tid + TX];
          }
          if (cj > 1) {
#pragma unroll
            for (int v = 0; v < nc; ++v) r[v] = r[v] + Fy[v * NT + tid];
          }
        } else {
#pragma unroll
          for (int v = 0; v < nc; ++v) r[v] = r[v] + Fy[v * NT + tid];
          if (cj < n) {
#pragma unroll
            for (int v = 0; v < nc; ++v) r[v] = r[v] - Fy[v * NT + tid + TX];
          }
        }
      }
      if (az) {
        const int ck = k + 1, n = B.nk;
        if (ck % 2 == 1) {
          if (ck < n) {
#pragma unroll
            for (int v = 0; v < nc; ++v) r[v] = r[v] - fhi[v * NT + tid];
          }
          if (ck > 1) {
#pragma unroll
            for (int v = 0; v < nc; ++v) r[v] = r[v] + flo[v * NT + tid];
          }
        } else {
#pragma unroll
          for (int v = 0; v < nc; ++v) r[v] = r[v] + flo[v * NT + tid];
          if (ck < n) {
#pragma unroll
            for (int v = 0; v < nc; ++v) r[v] = r[v] - fhi[v * NT + tid];
          }
        }
      }
      const long long g = gidx(B, i, j, k);
      double p[nc];
#pragma unroll
      for (int v = 0; v < nc; ++v) p[v] = F.Up[(long long)v * G.NG + g];
      double s[nc];
#pragma unroll
      for (int v = 0; v < nc; ++v)
        s[v] = F.coupled ? (double)F.Sf[(long long)v * G.NI + q] : 0.0;
      if (F.xstep) accumulate_source<CL>(F.xstep, G.NI, q, s, F.xfirst, F.rk);
      const double dt = F.dt ? F.dt[q] : *F.dtg;
      const double vol = G.vol[q];
#pragma unroll
      for (int v = 0; v < nc; ++v) r[v] = (r[v]/vol + s[v]) * dt;
      if (F.imports) {                          // add_births (Lib_Residual.f90:164-210): the coupler's rates
#pragma unroll
        for (int v = 0; v < nc; ++v) r[v] = r[v] + F.imports[(long long)v * G.NI + q] * dt;
      }
#pragma unroll
      for (int v = 0; v < nc; ++v) if (F.frozen_mask & (1u << v)) r[v] = 0.0;
      double po[nc], co[nc], cn[nc];
#pragma unroll
      for (int v = 0; v < nc; ++v) po[v] = F.U0[(long long)v * G.NG + g];
      prim2cons<CL, double>(po, co, F.mat.cp);
      prim2cons<CL, double>(p, cn, F.mat.cp);
#pragma unroll
      for (int v = 0; v < nc; ++v) { double rr = (cn[v] - co[v] + r[v]) * F.rk; cn[v] = co[v] + rr; }
      if (cn[0] < 0.0) atomicAdd(&st->nfloored, 1ULL);
      cons2prim<CL>(cn, p, F.mat.cp);
      if (F.realize && realize<CL>(p)) atomicAdd(&st->nrealized, 1ULL);
      if (!check_prim<CL, double>(p)) atomicOr(&st->flags, (unsigned)ICE_GPU_ST_NAN_STATE);
#pragma unroll
      for (int v = 0; v < nc; ++v) F.Uo[(long long)v * G.NG + g] = p[v];
    }
    __syncthreads();
    double* tmp = flo; flo = fhi; fhi = tmp;
  }
  if (bad) atomicOr(&st->flags, (unsigned)ICE_GPU_ST_BAD_RECON);
}

// ------------------------------------------------------------------ IRS and the separate update
template <int CL>
__global__ void k_update(Geo G, FamDev F, Status* st) {
  long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= G.NI) return;
  constexpr int nc = NC<CL>::v;
  const DBlock& B = G.blk[find_block(G.blk, G.nb, q)];
  int i, j, k; decode(B, q, i, j, k);
  long long g = gidx(B, i, j, k);
  double p[nc], po[nc], co[nc], cn[nc];
#pragma unroll
  for (int v = 0; v < nc; ++v) { p[v] = F.Up[(long long)v * G.NG + g]; po[v] = F.U0[(long long)v * G.NG + g]; }
  prim2cons<CL, double>(po, co, F.mat.cp);
  prim2cons<CL, double>(p, cn, F.mat.cp);
#pragma unroll
  for (int v = 0; v < nc; ++v) { double rr = (cn[v] - co[v] + F.resid[(long long)v * G.NI + q]) * F.rk; cn[v] = co[v] + rr; }
  if (cn[0] < 0.0) atomicAdd(&st->nfloored, 1ULL);
  cons2prim<CL>(cn, p, F.mat.cp);
  if (!check_prim<CL, double>(p)) atomicOr(&st->flags, (unsigned)ICE_GPU_ST_NAN_STATE);
#pragma unroll
  for (int v = 0; v < nc; ++v) F.Uo[(long long)v * G.NG + g] = p[v];
}


// ------------------------------------------------------------------ sensor
template <typename R> __global__ void k_beta(Geo G, FamDev F) {
  long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= G.NI) return;
  const DBlock& B = G.blk[find_block(G.blk, G.nb, q)];
  int i, j, k; decode(B, q, i, j, k);
  const double* P = F.Up;   // variable 0: density
  ((R*)F.betaR)[q] = sd_rho<R>((R)P[gidx(B, i, j, k)], (R)P[gidx(B, i - 1, j, k)], (R)P[gidx(B, i + 1, j, k)],
                      (R)P[gidx(B, i, j - 1, k)], (R)P[gidx(B, i, j + 1, k)],
                      (R)P[gidx(B, i, j, k - 1)], (R)P[gidx(B, i, j, k + 1)]);
}


// One Jacobi sweep of direction d (Lib_IRS.f90:278-293): out = (R + b (star_{-1} + star_{+1}))/(1+2b),
// with the ghost values of star fixed to the first and last cell of R (zero gradient).
__global__ void k_irs(Geo G, int nc, const double* R0, const double* star, double* out, int d, double beta) {
  long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= G.NI) return;
  const DBlock& B = G.blk[find_block(G.blk, G.nb, q)];
  int i, j, k; decode(B, q, i, j, k);
  int c = d == 0 ? i : d == 1 ? j : k;
  int n = d == 0 ? B.ni : d == 1 ? B.nj : B.nk;
  long long st = d == 0 ? 1 : d == 1 ? B.ni : (long long)B.ni * B.nj;
  long long qm = c > 0 ? q - st : q;         // ghost 0 = cell 1 of the original residual
  long long qp = c < n - 1 ? q + st : q;
  for (int v = 0; v < nc; ++v) {
    const double* S = (c > 0 ? star : R0) + (long long)v * G.NI;
    const double* Sp = (c < n - 1 ? star : R0) + (long long)v * G.NI;
    out[(long long)v * G.NI + q] = (R0[(long long)v * G.NI + q] + beta*(S[qm] + Sp[qp])) / (1.0 + 2.0*beta);
  }
}


// ------------------------------------------------------------------ residual norm
// residual_sq (Mod_Diagnostic.f90:106-130): per CTA, sums of (new - old)^2 of rho, u, v, w, T
// over a contiguous range of one block's cells, reduced in a fixed order.

__global__ void k_norm(Geo G, const double* Un, const double* Uo, int iT, const NormChunk* ch, double* part) {
  const NormChunk c = ch[blockIdx.x];
  const DBlock& B = G.blk[c.b];
  double acc[5] = {0, 0, 0, 0, 0};
  for (long long q = c.q0 + threadIdx.x; q < c.q1; q += blockDim.x) {
    int i, j, k; decode(B, q, i, j, k);
    long long g = gidx(B, i, j, k);
    int vs[5] = {0, 1, 2, 3, iT};
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      double d = fabs(Un[(long long)vs[m] * G.NG + g] - Uo[(long long)vs[m] * G.NG + g]);
      acc[m] = acc[m] + d*d;
    }
  }
  __shared__ double red[5][256];
#pragma unroll
  for (int m = 0; m < 5; ++m) red[m][threadIdx.x] = acc[m];
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) {
#pragma unroll
      for (int m = 0; m < 5; ++m) red[m][threadIdx.x] = red[m][threadIdx.x] + red[m][threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
#pragma unroll
    for (int m = 0; m < 5; ++m) part[(long long)blockIdx.x * 5 + m] = red[m][0];
  }
}


}  // namespace
}  // namespace ice
