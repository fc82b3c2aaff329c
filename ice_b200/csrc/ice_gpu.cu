// ice_gpu.cu -- the B200 (sm_100a) solve stage of ICE's Eulerian dispersed-phase time step,
// behind the C ABI of include/ice_gpu.h.
//
// One call of ice_gpu_step replaces `call Explicit_Step(grid)` (src/lib/driver/Wrap_Solve.f90:26;
// numerics/time/explicit/Mod_Explicit.f90:11-245). Every array is resident in HBM; a step is a
// CUDA graph of:
//   k_dt_all       per-cell CFL dt of every family + global min (FP64)  (Mod_dt.f90:11-112,256-275)
//   (k_empty_scan, k_empty_apply for a family with the coupler's imports: Mod_dt.f90:134-242)
//                  and the end of the dt part: dtglobal, time += dt, counters (Mod_Explicit.f90:40-73; k_time
//                  where the bounds of imports or of other ranks come after it)
//   per family, per RK stage:
//     k_source     the source (plain form; an evaporating family of the FP32-flux form; 1-D runs), or the
//                  surrogate's k_source_mlp                            (Mod_Sources.f90:465-622)
//     (in the FP32-flux form's 1-D runs k_rec and k_stage take the place of k_flux and k_cells)
//     k_ghost      both ghost layers from the record list (two launches, layer 1 then
//                  layer 2, where a block is one cell deep along a record's face), block
//                  connections as on-device copies in one HBM pool    (Lib_Ghost.f90:29-387)
//     k_beta       Jameson sensor (when on)                           (Mod_Fluxes.f90:366-389)
//     k_flux       the fluxes of the boundary records (Mod_BC_Fluxes.f90:105-170) and of the interior faces
//                  (Mod_Fluxes.f90:599-685); k_cell_sum where the table lists a face of a cell more than once
//     k_cells      the cells' update: a cell's boundary faces, then its interior faces in the odd-then-even
//                  order (Mod_Fluxes.f90:421-521), the source (in the FP32-flux form evaluated here for a family
//                  without evaporation: Mod_Sources.f90:465-622), the residual
//                  with the coupler's imports (Lib_Residual.f90:147-210) and the RK update with
//                  cons<->prim and the state checks (Lib_Newstate.f90:198-219)
//     (k_irs, k_update when implicit residual smoothing is on: Lib_IRS.f90:34-86)
//
// The state is stored structure-of-arrays, one contiguous array per variable over every block
// of a family (ghost layers included), in three buffers that rotate over the RK stages: the
// stage reads U_{k-1} (stencil) and U_0 (pointwise) and writes U_k, so no state copy
// (state_copy, Lib_Newstate.f90:65-106) and no zeroing of the residual (Lib_Residual.f90:13-41)
// remain: the residual lives in registers.
#include <cuda_runtime.h>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <cstdarg>
#include <cmath>
#include <vector>
#include <string>
#include <algorithm>
#include <memory>
#include "ice_kernels.cuh"
#include "ice_sweep.cuh"
#include "ice_mlp.cuh"
#include "ice_tune.h"
#include "../../include/ice_gpu.h"

using namespace ice;

namespace {

constexpr int kMaxF = ICE_GPU_MAX_FAMILIES;
constexpr int kMaxNC = 12;     // variables of the largest closure (AG)

// ------------------------------------------------------------------ host side
struct HRec {
  int b, i, j, k, f, type, p, bs, is, js, ks, fs, partner, owner, cf;
  double massflux, velocity, alpha, beta, temperature, radius, gfixed, normal_dir;
};

template <typename T> struct DevBuf {
  T* p = nullptr; size_t n = 0;
  bool on_host = false;                      // managed memory held on the host
  ~DevBuf() { if (p) cudaFree(p); }
  cudaError_t alloc(size_t count) {
    if (p) { cudaFree(p); p = nullptr; }
    n = 0; on_host = false;
    if (count == 0) return cudaSuccess;
    const cudaError_t e = cudaMalloc((void**)&p, count * sizeof(T));
    if (e == cudaSuccess) n = count;
    else { p = nullptr; cudaGetLastError(); }          // reported here, not by the next call's check
    return e;
  }
  // For what can lie on the host at a price: where the device has no room left, managed memory held there, which
  // the kernels read and write over the bus: 5 steps of AG on 261 k cells in FP64 took 62 ms so, 19 with room (pages
  // that move to the full device evict one another: 47 s).
  cudaError_t alloc_or_managed(size_t count) {
    cudaError_t e = alloc(count);
    if (e != cudaErrorMemoryAllocation) return e;
    e = cudaMallocManaged((void**)&p, count * sizeof(T));
    int dev = 0;
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaMemAdvise(p, count * sizeof(T), cudaMemAdviseSetPreferredLocation, cudaCpuDeviceId);
    if (e == cudaSuccess) e = cudaMemAdvise(p, count * sizeof(T), cudaMemAdviseSetAccessedBy, dev);
    if (e == cudaSuccess) { n = count; on_host = true; }
    else { if (p) cudaFree(p); p = nullptr; cudaGetLastError(); }
    return e;
  }
};

struct FamHost {
  int closure, riemann, nc;
  DevBuf<double> S[3];
  DevBuf<unsigned char> inj;
  DevBuf<double> dt, tau, beta;
  DevBuf<float> betaf;                       // the FP32-flux form's Jameson weights
  DevBuf<double> connF, resid, resid2, resid3, src;
  DevBuf<DRec> recs;
  DevBuf<DRec> grecs;                        // the ghost kernel's records, and its copies (upload_recs)
  DevBuf<GhostCopy> gcopy;
  int ngrec = 0, ncopy = 0, next = 0;
  bool ghost_split = false;                  // the ghost layers in two launches (upload_recs)
  DevBuf<int> frec;                          // the records whose flux is computed, in the record kernel's thread order
  int nfrec = 0;
  DevBuf<int> sfirst, slist;                 // the cells of k_cell_sum: their first records, their records
  int nsum = 0;
  DevBuf<ZeroFace> zface;                    // FamDev::zface
  int nzface = 0;
  DevBuf<SweepJob> fjobs;                    // the flux kernel's CTAs (ice_sweep.cuh)
  int nfjob = 0;
  // the evaporation surrogate (FP32-flux form): the network's BF16 image, its standardisation and
  // envelope, its FP32 parameters; on = the stage's source comes from the surrogate source kernel
  DevBuf<unsigned char> mlp_img;
  MlpNorm mlp_norm;
  std::vector<float> mlp_w;
  bool sur_on = false;
  int nrec = 0, nbc = 0, nown = 0, ncf = 0;
  std::vector<int> h_first, h_list, h_own;   // 0-based record numbers of the whole table
  std::vector<int> h_grp;                    // the family's records: their numbers in the table
  std::vector<DRec> h_recs;                  // the device records, kept to attach chimera donors
  DevBuf<int4> cdon;                         // chimera donors (0-based block, i, j, k) and weights
  DevBuf<double> cw;
  DevBuf<double> imp;                        // the coupler's imports [v][NI] (ice_gpu_set_imports)
  DevBuf<EmptyScan> escan;                   // bound_empty_dt's reductions
  bool have_imp = false;
  DevBuf<double> xstep;                      // the step's weighted source, slots 1-4 and energy [5][NI]
};


}  // namespace

struct ice_gpu_ctx {
  ice_gpu_params P;
  int nb = 0;
  int nsm = 148;            // the GPU's SMs
  std::vector<int> dims;
  std::vector<DBlock> hblk;
  long long NG = 0, NI = 0, NR = 0, NF[3] = {0, 0, 0};
  DevBuf<DBlock> blk;
  DevBuf<double> face[3], vol, dl, M, gas;
  DevBuf<double> row;       // Geo::row, formed from M before the first step after a block's metrics
  DevBuf<float4> facef[3];  // the FP32-flux form's geometry (Geo::ff, dlf), rounded from the FP64 arrays
  DevBuf<float> dlf;
  DevBuf<float> gasf;       // the FP32-flux form's copy of the gas (Geo::gasf)
  // the face fluxes of one family's stage (the families step one after the other), words of 4 or 8 bytes; zeroed
  // when they are allocated and after a new boundary table (flux_ok)
  DevBuf<unsigned char> flux;
  size_t flux_at[3] = {0, 0, 0};
  int flux_word = 0;
  bool flux_ok = false, rows_ok = false;
  bool geo32_ok = false;
  bool have_gas = false;
  std::vector<bool> have_block;
  std::vector<bool> gas_set;     // per block: ice_gpu_set_gas was called
  bool have_records = false;
  bool exchange = false;  // two-way coupling: the step's weighted source is kept for the gas
  int nchim = 0;          // 102 records of the table
  bool have_chimera = true;   // their donors are set (ice_gpu_set_chimera)
  FamHost fam[kMaxF];
  std::vector<HRec> recs;
  DevBuf<Tile> tiles;
  int ntile = 0, TX = 0, TY = 0, KZ = 0;
  DevBuf<NormChunk> chunks;
  DevBuf<double> npart;
  int nchunk = 0;
  std::vector<int> chunk_block;
  DevBuf<Status> st;
  cudaStream_t stream = nullptr;
  cudaGraphExec_t graph[3] = {nullptr, nullptr, nullptr};
  // ice_gpu_step_host: the step cut into its dt part and one graph per family (per buffer phase), two
  // copy streams, the caller's arrays staged in one device buffer, one event per family
  cudaGraphExec_t graph_pre[3] = {nullptr, nullptr, nullptr};
  cudaGraphExec_t graph_fam[3][kMaxF] = {};
  cudaStream_t s_up = nullptr, s_down = nullptr;
  // the step's second branch (capture_step), captured only
  cudaStream_t s_prep = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_prep[kMaxF] = {}, ev_done[kMaxF] = {}, ev_src[kMaxF] = {};
  cudaEvent_t ev_up = nullptr, ev_fam[kMaxF] = {};
  DevBuf<double> xall;
  int phase = 0;          // buffer holding the current state
  int prev_phase = -1;    // buffer holding the state before the last step
  double res_reference = 0.0;  // the first non-zero density residual of a steady run (0: none yet)
  bool res_end = false;        // the last step ended the run on res-threshold
  double last_norm[5] = {0, 0, 0, 0, 0};
  bool profiling = false;
  double kms[KC_N] = {0};
  // the block split (ice_gpu_set_partition, _set_halo, _set_exchange_hook): the blocks this rank steps
  // (empty: all), on the device too; per kind and family the entries sent and received (0-based int4:
  // block, i, j, k; or the connection face in x); the hook and its pinned host buffers
  std::vector<unsigned char> owned;
  DevBuf<unsigned char> owned_dev;
  std::vector<int4> hs[3][kMaxF], hr[3][kMaxF];
  DevBuf<int4> hs_dev[3][kMaxF], hr_dev[3][kMaxF];
  ice_gpu_exchange_fn hook = nullptr;
  void* hook_user = nullptr;
  DevBuf<double> xdev;
  double* xhost = nullptr;
  size_t xhost_n = 0;
  int xerr = 0;                  // the first failure of an exchange of the running call
  unsigned long long xbits = 0;  // the reduced dt on its way back to the device
  long long nlaunch = 0;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  cudaEvent_t t0 = nullptr, t1 = nullptr;   // around a call's steps
  Status* hst = nullptr;    // the status as the last call's steps left it (page-locked)
  DevBuf<double> xfer;    // one block of one family in the caller's layout (upload/download)
  long long ng_max = 0;
  std::string err;
};

static std::string g_create_err;

static bool sur_active(const ice_gpu_ctx* c, int p) {
  const FamHost& H = c->fam[p];
  return H.sur_on && H.mlp_img.p && c->P.coupled && c->P.precision == ICE_PREC_FP32FLUX && !c->P.irs;
}

// The caller's prim(nc, -1:ni+2, -1:nj+2, -1:nk+2) (variable fastest) <-> one block of the SoA pool,
// whose rows are px long (the row padding is never read).
__device__ __forceinline__ long long pool_of(long long q, int ni4, int nj4, int px) {
  long long x = q % ni4, r = q / ni4;
  return (r / nj4) * ((long long)px * nj4) + (r % nj4) * px + x;
}
__global__ void k_aos2soa(const double* __restrict__ a, double* __restrict__ s, long long NG, long long n, int nc,
                          int ni4, int nj4, int px) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
    long long d = pool_of(q, ni4, nj4, px);
    for (int v = 0; v < nc; ++v) s[(long long)v * NG + d] = a[(long long)nc * q + v];
  }
}
__global__ void k_soa2aos(const double* __restrict__ s, double* __restrict__ a, long long NG, long long n, int nc,
                          int ni4, int nj4, int px) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
    long long d = pool_of(q, ni4, nj4, px);
    for (int v = 0; v < nc; ++v) a[(long long)nc * q + v] = s[(long long)v * NG + d];
  }
}
__global__ void k_inj2pool(const unsigned char* __restrict__ a, unsigned char* __restrict__ s, long long n,
                           int ni4, int nj4, int px) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
    s[pool_of(q, ni4, nj4, px)] = a[q];
}
static unsigned grid_of(long long n) { return (unsigned)std::min<long long>((n + 255) / 256, 148LL * 16); }

static int fail(ice_gpu_ctx* c, int code, const char* fmt, ...) {
  char buf[1024];
  va_list ap; va_start(ap, fmt); vsnprintf(buf, sizeof buf, fmt, ap); va_end(ap);
  if (c) c->err = buf; else g_create_err = buf;
  return code;
}

#define CK(call) do { cudaError_t e_ = (call); if (e_ != cudaSuccess) \
  return fail(c, ICE_GPU_ECUDA, "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); } while (0)

static int nbase_of(int cl) { return cl == ICE_CLOSURE_MK ? 6 : cl == ICE_CLOSURE_IG ? 7 : 12; }

static void free_graphs(ice_gpu_ctx* c) {
  for (auto& g : c->graph) if (g) { cudaGraphExecDestroy(g); g = nullptr; }
  for (auto& g : c->graph_pre) if (g) { cudaGraphExecDestroy(g); g = nullptr; }
  for (auto& row : c->graph_fam) for (auto& g : row) if (g) { cudaGraphExecDestroy(g); g = nullptr; }
}

// Gives back the device memory of what a step makes again (ensure_flux): the metric rows, the face fluxes, the
// FP32-flux form's weights. Between calls only: the next step's ensure_flux places them anew. False: nothing lay on the device.
static bool yield_room(ice_gpu_ctx* c) {
  bool any = (c->row.p && !c->row.on_host) || (c->flux.p && !c->flux.on_host);
  for (int p = 0; p < c->P.nfam; ++p) any = any || (c->fam[p].betaf.p && !c->fam[p].betaf.on_host);
  if (!any || cudaStreamSynchronize(c->stream) != cudaSuccess) return false;
  free_graphs(c);
  c->row.alloc(0); c->flux.alloc(0);
  for (int p = 0; p < c->P.nfam; ++p) c->fam[p].betaf.alloc(0);
  c->rows_ok = c->flux_ok = false;
  c->flux_word = 0;
  return true;
}

// Device memory for what has no place on the host, after create: the step's own work memory makes room for it.
template <typename T> static cudaError_t with_room(ice_gpu_ctx* c, DevBuf<T>& b, size_t count) {
  const cudaError_t e = b.alloc(count);
  return e == cudaErrorMemoryAllocation && yield_room(c) ? b.alloc(count) : e;
}

// The surrogate source runs for family p: on, trained, a coupled run in the FP32-flux form.
static bool sur_active(const ice_gpu_ctx* c, int p);

// The stage runs in FP64: the plain form, and every IRS run.
static bool sweeps64(const ice_gpu_ctx* c) { return c->P.precision != ICE_PREC_FP32FLUX || c->P.irs; }
// The FP32-flux form's 1-D stage kernel runs (ice_kernels.cuh).
static bool plane(const ice_gpu_ctx* c) { return !sweeps64(c) && c->P.ndir == 1; }

// Family p's source has a kernel of its own.
static bool own_source(const ice_gpu_ctx* c, int p) {
  return c->P.coupled && (sweeps64(c) || plane(c) || sur_active(c, p) || c->P.fam[p].evap != 0);
}

// The buffer stage srk reads as its stencil (U_{k-1}) when the step starts from buffer `phase`.
static int stencil_buffer(const ice_gpu_ctx*, int srk, int phase) {
  return srk == 1 ? phase : srk == 2 ? (phase + 1) % 3 : (phase + 2) % 3;
}

static FamDev make_famdev(ice_gpu_ctx* c, int p, int srk, int phase) {
  FamHost& H = c->fam[p];
  const ice_gpu_family& pf = c->P.fam[p];
  FamDev F;
  memset(&F, 0, sizeof F);
  F.closure = H.closure; F.riemann = H.riemann; F.nc = H.nc;
  F.limiter = c->P.limiter; F.sd = c->P.shock_detector; F.coupled = c->P.coupled;
  F.realize = c->P.precision == ICE_PREC_FP32FLUX && !c->P.no_realize;
  F.drag = c->P.drag; F.heat = c->P.heat; F.blow = c->P.blow;
  F.frozen_mask = 0;
  for (int q = 0; q < pf.nfrozen; ++q) F.frozen_mask |= 1u << (pf.frozen[q] - 1);
  F.mat.rho = pf.rho_al; F.mat.cp = pf.cs_al; F.mat.lv = pf.lv_al; F.mat.emiss = pf.emiss;
  F.mat.evap = pf.evap; F.mat.intf = pf.intf;
  for (int q = 0; q < ICE_GPU_NEP; ++q) F.mat.ep[q] = pf.ep[q];
  // buffer roles (see the rotation in step_graph)
  int a = phase, b = (phase + 1) % 3;
  int up = stencil_buffer(c, srk, phase);
  int out = srk == 1 ? b : srk == 2 ? (phase + 2) % 3 : b;
  F.U0 = H.S[a].p; F.Up = H.S[up].p; F.Ug = H.S[up].p; F.Uo = H.S[out].p;
  F.inj = H.inj.p;
  F.beta = c->P.shock_detector ? H.beta.p : nullptr;
  F.betaw = H.beta.p;
  F.betaR = plane(c) || sweeps64(c) ? (void*)H.beta.p : (void*)H.betaf.p;
  F.dt = c->P.time_accurate ? nullptr : H.dt.p;
  F.dtg = &c->st.p->dtglobal;
  F.tau = H.tau.p;
  F.S = H.src.p;
  F.Sf = sweeps64(c) ? nullptr : (float*)H.src.p;      // an IRS run's stage, and so its source, is FP64 in both forms
  F.connF = c->owned.empty() && H.nsum == 0 ? nullptr : H.connF.p;
  for (int d = 0; d < 3; ++d) F.Ff[d] = c->flux.p + c->flux_at[d];
  F.zface = H.zface.p; F.nzface = H.nzface;
  F.cdon = H.cdon.p; F.cw = H.cw.p;
  F.imports = H.have_imp ? H.imp.p : nullptr;
  F.xstep = (c->exchange && c->P.coupled) ? H.xstep.p : nullptr;
  F.xfirst = srk == 1;
  F.resid = H.resid.p;
  static const double RKC[3][3] = {{1.0, 0.0, 0.0}, {1.0, 0.50, 0.0}, {1.0, 0.25, 2.0/3.0}};
  F.rk = RKC[c->P.nrk - 1][srk - 1];
  F.write_tau = srk == c->P.nrk;
  F.src_ready = (sur_active(c, p) || (c->P.coupled && pf.evap != 0)) ? 1 : 0;
  return F;
}

static Geo make_geo(ice_gpu_ctx* c) {
  Geo G;
  G.blk = c->blk.p; G.nb = c->nb;
  G.NG = c->NG; G.NI = c->NI; G.NR = c->NR;
  for (int d = 0; d < 3; ++d) { G.NF[d] = c->NF[d]; G.face[d] = c->face[d].p; }
  G.vol = c->vol.p; G.dl = c->dl.p; G.M = c->M.p; G.gas = c->gas.p; G.row = c->row.p;
  for (int d = 0; d < 3; ++d) G.ff[d] = c->facef[d].p;
  G.dlf = c->dlf.p;
  G.gasf = c->gasf.p;
  G.owned = c->owned.empty() ? nullptr : c->owned_dev.p;
  return G;
}

__global__ void k_face32(const double* f, long long NF, float4* out) {
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < NF; q += (long long)gridDim.x * blockDim.x)
    out[q] = make_float4((float)f[q], (float)f[NF + q], (float)f[2 * NF + q], (float)f[3 * NF + q]);
}

__global__ void k_dl32(const double* dl, long long n, float* out) {
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
    out[q] = (float)dl[q];
}

// The FP32-flux form's geometry: the face normals and areas packed per face and the cell lengths in
// single precision, rounded as the kernels rounded each value on reading (allocated once, so that
// captured graphs keep their pointers; converted again after any ice_gpu_set_block).
static int build_geo32(ice_gpu_ctx* c) {
  if (c->P.precision != ICE_PREC_FP32FLUX || c->geo32_ok) return 0;
  bool fresh = false;
  for (int d = 0; d < 3; ++d) {
    if (!c->facef[d].p && c->NF[d] > 0) { CK(with_room(c, c->facef[d], (size_t)c->NF[d])); fresh = true; }
    if (c->NF[d] > 0) {
      k_face32<<<grid_of(c->NF[d]), 256, 0, c->stream>>>(c->face[d].p, c->NF[d], c->facef[d].p);
      CK(cudaGetLastError());
    }
  }
  if (!c->dlf.p) { CK(with_room(c, c->dlf, (size_t)3 * c->NR)); fresh = true; }
  k_dl32<<<grid_of(3 * c->NR), 256, 0, c->stream>>>(c->dl.p, 3 * c->NR, c->dlf.p);
  CK(cudaGetLastError());
  if (c->P.coupled && c->gas.p) {
    if (!c->gasf.p) { CK(with_room(c, c->gasf, (size_t)9 * c->NI)); fresh = true; }
    k_dl32<<<grid_of(9 * c->NI), 256, 0, c->stream>>>(c->gas.p, 9 * c->NI, c->gasf.p);
    CK(cudaGetLastError());
  }
  CK(cudaStreamSynchronize(c->stream));
  if (fresh) free_graphs(c);          // graphs captured before the buffers existed hold null pointers
  c->geo32_ok = true;
  return 0;
}

// ---------------------------------------------------------------- kernel dispatch
#define GRID(n, t) ((unsigned)(((n) + (t) - 1) / (t)))

// ---------------------------------------------------------------- the block split's exchanges
// Pack and unpack of the exchange lists (0-based int4 entries: block, i, j, k; a connection face in x).
__global__ void k_pack_cells(Geo G, const double* __restrict__ U, int nc, const int4* __restrict__ e, int n,
                             double* __restrict__ out) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const int4 x = e[q];
  const long long g = gidx(G.blk[x.x], x.y, x.z, x.w);
  for (int v = 0; v < nc; ++v) out[(long long)q * nc + v] = U[(long long)v * G.NG + g];
}
__global__ void k_unpack_cells(Geo G, double* __restrict__ U, int nc, const int4* __restrict__ e, int n,
                               const double* __restrict__ in) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const int4 x = e[q];
  const long long g = gidx(G.blk[x.x], x.y, x.z, x.w);
  for (int v = 0; v < nc; ++v) U[(long long)v * G.NG + g] = in[(long long)q * nc + v];
}
__global__ void k_unpack_beta(Geo G, double* __restrict__ beta, const int4* __restrict__ e, int n,
                              const double* __restrict__ in) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const int4 x = e[q];
  beta[iidx(G.blk[x.x], x.y, x.z, x.w)] = in[q];
}
__global__ void k_pack_flux(const double* __restrict__ F, int nc, const int4* __restrict__ e, int n,
                            double* __restrict__ out) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  for (int v = 0; v < nc; ++v) out[(long long)q * nc + v] = F[(long long)e[q].x * nc + v];
}
__global__ void k_unpack_flux(double* __restrict__ F, int nc, const int4* __restrict__ e, int n,
                              const double* __restrict__ in) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  for (int v = 0; v < nc; ++v) F[(long long)e[q].x * nc + v] = in[(long long)q * nc + v];
}

static int ensure_xbuf(ice_gpu_ctx* c, size_t n, cudaStream_t s) {
  if (c->xdev.n >= n && c->xhost_n >= n) return 0;
  CK(cudaStreamSynchronize(s));                    // the last exchange's copy and unpack read the buffers
  if (c->xdev.n < n) CK(with_room(c, c->xdev, n));
  if (c->xhost_n < n) {
    if (c->xhost) cudaFreeHost(c->xhost);
    c->xhost = nullptr; c->xhost_n = 0;
    CK(cudaMallocHost((void**)&c->xhost, n * sizeof(double)));
    c->xhost_n = n;
  }
  return 0;
}

// The buffers for the largest exchange of a step, before the step's work memory takes its place.
static int ensure_xbufs(ice_gpu_ctx* c) {
  size_t n = 1;
  if (c->owned.empty()) return 0;
  for (int kind = 0; kind < 3; ++kind)
    for (int p = 0; p < c->P.nfam; ++p)
      n = std::max(n, (c->hs[kind][p].size() + c->hr[kind][p].size()) * (kind == ICE_GPU_HALO_BETA ? 1 : c->fam[p].nc) + 1);
  return ensure_xbuf(c, n, c->stream);
}

// One exchange of a split step (Mod_GhostExchange.f90:737-800 for the cells), at its point of the
// family's stage: pack on the device, copy to the host, the hook, copy back, unpack. The stream is
// drained before the hook, so the hook sees this stage's data and no kernel waits on another rank.
// The first failure is kept (xerr) and reported by the step; later exchanges of the call are skipped.
static void halo_xchg(const LaunchArgs& a, int kind) {
  ice_gpu_ctx* c = (ice_gpu_ctx*)a.tick_ctx;
  if (c->xerr) return;
  const int p = a.fam, nc = c->fam[p].nc, w = kind == ICE_GPU_HALO_BETA ? 1 : nc;
  const int ns = (int)c->hs[kind][p].size(), nr = (int)c->hr[kind][p].size();
  const size_t ls = (size_t)ns * w, lr = (size_t)nr * w;
  if (ensure_xbuf(c, ls + lr + 1, a.s)) { c->xerr = ICE_GPU_ECUDA; return; }
  double* ds = c->xdev.p; double* dr = c->xdev.p + ls;
  const int4* es = c->hs_dev[kind][p].p; const int4* er = c->hr_dev[kind][p].p;
  if (ns > 0) {
    if (kind == ICE_GPU_HALO_CELLS) k_pack_cells<<<GRID(ns, 128), 128, 0, a.s>>>(a.G, a.F.Up, nc, es, ns, ds);
    else if (kind == ICE_GPU_HALO_FLUX) k_pack_flux<<<GRID(ns, 128), 128, 0, a.s>>>(a.F.connF, nc, es, ns, ds);
    else {
      // in the translation unit of the closure's connection kernel, compiled as it is, for its bits
      const int cl = c->fam[p].closure;
      const bool f32 = a.precision == ICE_PREC_FP32FLUX;
      if (cl == ICE_CLOSURE_MK) (f32 ? launch_pack_beta_mk_f32 : launch_pack_beta_mk_f64)(a, es, ns, ds);
      else if (cl == ICE_CLOSURE_IG) (f32 ? launch_pack_beta_ig_f32 : launch_pack_beta_ig_f64)(a, es, ns, ds);
      else (f32 ? launch_pack_beta_ag_f32 : launch_pack_beta_ag_f64)(a, es, ns, ds);
    }
    cudaMemcpyAsync(c->xhost, ds, ls * sizeof(double), cudaMemcpyDeviceToHost, a.s);
  }
  if (cudaStreamSynchronize(a.s) != cudaSuccess || cudaGetLastError() != cudaSuccess) {
    c->xerr = ICE_GPU_ECUDA; fail(c, ICE_GPU_ECUDA, "split exchange: a CUDA error before the hook");
    return;
  }
  if (!c->hook) { c->xerr = ICE_GPU_ENOTREADY; fail(c, ICE_GPU_ENOTREADY, "a split run needs its exchange hook"); return; }
  if (c->hook(c->hook_user, kind, p + 1, (int64_t)ls, c->xhost, (int64_t)lr, c->xhost + ls) != 0) {
    c->xerr = ICE_GPU_EEXCH; fail(c, ICE_GPU_EEXCH, "the exchange hook failed (kind %d, family %d)", kind, p + 1);
    return;
  }
  if (nr > 0) {
    cudaMemcpyAsync(dr, c->xhost + ls, lr * sizeof(double), cudaMemcpyHostToDevice, a.s);
    if (kind == ICE_GPU_HALO_CELLS) k_unpack_cells<<<GRID(nr, 128), 128, 0, a.s>>>(a.G, a.F.Ug, nc, er, nr, dr);
    else if (kind == ICE_GPU_HALO_FLUX) k_unpack_flux<<<GRID(nr, 128), 128, 0, a.s>>>(a.F.connF, nc, er, nr, dr);
    else k_unpack_beta<<<GRID(nr, 128), 128, 0, a.s>>>(a.G, a.F.betaw, er, nr, dr);
  }
}

// The reductions of a split run: the minimum (DT) or the sum (NORM) over the ranks of n doubles.
static int halo_reduce(ice_gpu_ctx* c, int kind, double* x, long long n) {
  if (c->owned.empty()) return 0;
  if (!c->hook) return fail(c, ICE_GPU_ENOTREADY, "a split run needs its exchange hook (ice_gpu_set_exchange_hook)");
  std::vector<double> in(x, x + n);
  if (c->hook(c->hook_user, kind, 0, n, in.data(), n, x) != 0)
    return fail(c, ICE_GPU_EEXCH, "the exchange hook failed (kind %d)", kind);
  return 0;
}

static void launch_family(ice_gpu_ctx* c, int p, int srk, int phase, cudaStream_t s,
                          void (*tick)(void*, int, cudaStream_t), int part = PART_ALL) {
  FamHost& H = c->fam[p];
  LaunchArgs a;
  a.G = make_geo(c);
  a.F = make_famdev(c, p, srk, phase);
  a.recs = H.recs.p; a.nrec = H.nrec; a.ghost_split = H.ghost_split;
  a.grecs = H.grecs.p; a.ngrec = H.ngrec; a.gcopy = H.gcopy.p; a.ncopy = H.ncopy; a.next = H.next;
  a.frec = H.frec.p; a.nfrec = H.nfrec;
  a.fjobs = H.fjobs.p; a.nfjob = H.nfjob;
  a.sfirst = H.sfirst.p; a.slist = H.slist.p; a.nsum = H.nsum;
  a.tiles = c->tiles.p; a.ntile = c->ntile; a.TX = c->TX; a.TY = c->TY; a.KZ = c->KZ;
  a.plane = plane(c);
  a.part = part;
  a.mlp_img = sur_active(c, p) ? H.mlp_img.p : nullptr;
  a.own_source = own_source(c, p);
  a.mlp_norm = &H.mlp_norm;
  a.ndir = c->P.ndir; a.sd = c->P.shock_detector; a.irs = c->P.irs; a.precision = c->P.precision;
  a.irs_beta = c->P.irs_beta;
  a.resid = H.resid.p; a.resid2 = H.resid2.p; a.resid3 = H.resid3.p;
  a.st = c->st.p;
  a.s = s;
  a.tick = tick; a.tick_ctx = c;
  a.xchg = c->owned.empty() ? nullptr : halo_xchg;
  a.fam = p;
  if (H.closure == ICE_CLOSURE_MK) launch_family_mk(a);
  else if (H.closure == ICE_CLOSURE_IG) launch_family_ig(a);
  else launch_family_ag(a);
}

// A family the coupler feeds or drains: bound_empty_dt and bound_removal_dt (Mod_Explicit.f90:57-60),
// after every family's compute_dt (k_dt_all).
static void launch_dt_bounds(ice_gpu_ctx* c, int p, int phase, cudaStream_t s) {
  if (!c->fam[p].have_imp) return;
  Geo G = make_geo(c);
  FamDev F = make_famdev(c, p, 1, phase);
  double* dto = c->P.time_accurate ? nullptr : c->fam[p].dt.p;
  unsigned g = GRID(c->NI, 256);
  EmptyScan* e = c->fam[p].escan.p;
  k_empty_init<<<1, 1, 0, s>>>(e);
  switch (c->fam[p].closure) {
    case ICE_CLOSURE_MK:
      k_empty_scan<MK><<<g, 256, 0, s>>>(G, F, dto, c->P.cfl, c->P.ndir, e);
      k_empty_apply<MK><<<g, 256, 0, s>>>(G, F, dto, c->P.cfl, c->P.ndir, e, c->st.p);
      break;
    case ICE_CLOSURE_IG:
      k_empty_scan<IG><<<g, 256, 0, s>>>(G, F, dto, c->P.cfl, c->P.ndir, e);
      k_empty_apply<IG><<<g, 256, 0, s>>>(G, F, dto, c->P.cfl, c->P.ndir, e, c->st.p);
      break;
    default:
      k_empty_scan<AG><<<g, 256, 0, s>>>(G, F, dto, c->P.cfl, c->P.ndir, e);
      k_empty_apply<AG><<<g, 256, 0, s>>>(G, F, dto, c->P.cfl, c->P.ndir, e, c->st.p);
      break;
  }
}

static int next_phase(const ice_gpu_ctx* c, int phase) {
  return c->P.nrk == 2 ? (phase + 2) % 3 : (phase + 1) % 3;
}

// One Explicit_Step on stream s starting from buffer `phase`: the step's dt over every family, then
// each family's RK stages (the families are independent of one another within a step).
static void enqueue_step_dt(ice_gpu_ctx* c, int phase, cudaStream_t s, void (*tick)(void*, int, cudaStream_t)) {
  // the step kernel ends the dt part itself unless bounds of imports or other ranks follow it
  bool finish = c->owned.empty();
  for (int p = 0; p < c->P.nfam; ++p) finish = finish && !c->fam[p].have_imp;
  {
    DtArgs a;
    memset(&a, 0, sizeof a);
    a.nf = c->P.nfam; a.ramp = c->P.cfl_ramp_iter; a.ndir = c->P.ndir; a.time_accurate = c->P.time_accurate;
    a.cfl = c->P.cfl; a.dt_max = c->P.dt_max; a.tau_factor = c->P.tau_factor;
    for (int p = 0; p < c->P.nfam; ++p) {
      FamDev F = make_famdev(c, p, 1, phase);
      a.f[p].Up = F.Up; a.f[p].tau = F.tau; a.f[p].coupled = F.coupled; a.f[p].closure = c->fam[p].closure;
      a.f[p].dt_out = c->P.time_accurate ? nullptr : c->fam[p].dt.p;
    }
    k_dt_all<<<std::min(GRID(c->NI, 256), 4u * (unsigned)c->nsm), 256, 0, s>>>(make_geo(c), a, finish ? 1 : 0, c->st.p);
  }
  for (int p = 0; p < c->P.nfam; ++p) launch_dt_bounds(c, p, phase, s);
  if (!c->owned.empty() && !c->xerr) {
    // a split run: the step's dt is the smallest over every rank (Mod_Explicit.f90:67-73)
    unsigned long long bits = 0;
    if (cudaMemcpyAsync(&bits, &c->st.p->dtbits, sizeof bits, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess) {
      c->xerr = ICE_GPU_ECUDA; fail(c, ICE_GPU_ECUDA, "split exchange: reading the dt");
    } else {
      double d;
      memcpy(&d, &bits, sizeof d);
      if (halo_reduce(c, ICE_GPU_HALO_DT, &d, 1)) c->xerr = ICE_GPU_EEXCH;
      memcpy(&bits, &d, sizeof d);
      c->xbits = bits;
      cudaMemcpyAsync(&c->st.p->dtbits, &c->xbits, sizeof bits, cudaMemcpyHostToDevice, s);
      cudaStreamSynchronize(s);
    }
  }
  if (!finish) k_time<<<1, 1, 0, s>>>(c->st.p, c->P.time_accurate);
  if (tick) tick(c, KC_DT, s);
}

static void enqueue_step_family(ice_gpu_ctx* c, int p, int phase, cudaStream_t s,
                                void (*tick)(void*, int, cudaStream_t)) {
  for (int srk = 1; srk <= c->P.nrk; ++srk) launch_family(c, p, srk, phase, s, tick);
}

// The step: its dt over every family, then the families' RK stages one family after the other.
static void enqueue_step(ice_gpu_ctx* c, int phase, cudaStream_t s, void (*tick)(void*, int, cudaStream_t)) {
  enqueue_step_dt(c, phase, s, tick);
  for (int p = 0; p < c->P.nfam; ++p) enqueue_step_family(c, p, phase, s, tick);
}

// The step as a graph of two branches: the families' faces and updates on s, stage by stage, and on a second
// stream their ghosts and sensors, under the faces of the families before them, and their sources, which only
// the update reads, under their own faces too: kernels that wait on memory or on their own chains beside
// ones that leave half of the issue slots free. The families share the face fluxes, so their faces stay one
// after the other. Three families on 8 blocks of 1.7 M cells, 8 steps in the FP32-flux form: 32.8 ms in one
// branch, 31.4 in two; 4 blocks of 0.35 M cells, 5 steps in FP64: 12.3 and 11.5, 10.8 with the sources under the
// faces. One family takes the second branch while a cell a thread is less than four waves in FP64, one and a half in
// the FP32-flux form, whose faces leave less idle. ms of 6 steps in one branch and in two, by thousands of cells:
//   FP32, evaporating: AG 30 0.528 / 0.496, 79 0.842 / 0.810, 125 1.097 / 1.115, 175 1.468 / 1.510, 300 2.18 / 2.24; IG 125 0.745 / 0.717
//   FP64: AG evaporating 30 1.21 / 0.96, 262 5.02 / 4.91, 342 6.39 / 6.24, 884 14.55 / 14.40; IG inert 175 1.93 / 1.86, 342 3.05 / 3.03,
//   884 6.51 / 6.56, 1,727 12.07 / 12.14
static bool two_branches(const ice_gpu_ctx* c) {
  const long long wave = 4LL * SW_NT * c->nsm;
  return c->P.nfam > 1 || (own_source(c, 0) && 2 * c->NI < (sweeps64(c) ? 8 : 3) * wave);
}

static cudaError_t capture_step(ice_gpu_ctx* c, int phase, cudaStream_t s) {
  if (!two_branches(c)) { enqueue_step(c, phase, s, nullptr); return cudaSuccess; }
  cudaError_t e = cudaSuccess;
  auto ck = [&](cudaError_t x) { if (e == cudaSuccess) e = x; };
  enqueue_step_dt(c, phase, s, nullptr);
  ck(cudaEventRecord(c->ev_fork, s));
  ck(cudaStreamWaitEvent(c->s_prep, c->ev_fork, 0));
  for (int srk = 1; srk <= c->P.nrk; ++srk)
    for (int p = 0; p < c->P.nfam; ++p) {
      if (srk > 1) ck(cudaStreamWaitEvent(c->s_prep, c->ev_done[p], 0));
      launch_family(c, p, srk, phase, c->s_prep, nullptr, PART_GHOSTS);
      ck(cudaEventRecord(c->ev_prep[p], c->s_prep));
      launch_family(c, p, srk, phase, c->s_prep, nullptr, PART_SOURCE);
      ck(cudaEventRecord(c->ev_src[p], c->s_prep));
      ck(cudaStreamWaitEvent(s, c->ev_prep[p], 0));
      launch_family(c, p, srk, phase, s, nullptr, PART_FACES);
      ck(cudaStreamWaitEvent(s, c->ev_src[p], 0));
      launch_family(c, p, srk, phase, s, nullptr, PART_CELLS);
      ck(cudaEventRecord(c->ev_done[p], s));
    }
  return e;
}

// The step's graph from buffer `phase`.
static int step_graph(ice_gpu_ctx* c, int phase) {
  if (c->graph[phase]) return 0;
  if (two_branches(c) && !c->s_prep) {
    CK(cudaStreamCreateWithFlags(&c->s_prep, cudaStreamNonBlocking));
    CK(cudaEventCreateWithFlags(&c->ev_fork, cudaEventDisableTiming));
    for (int p = 0; p < c->P.nfam; ++p) {
      CK(cudaEventCreateWithFlags(&c->ev_prep[p], cudaEventDisableTiming));
      CK(cudaEventCreateWithFlags(&c->ev_done[p], cudaEventDisableTiming));
      CK(cudaEventCreateWithFlags(&c->ev_src[p], cudaEventDisableTiming));
    }
  }
  cudaGraph_t g;
  CK(cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
  const cudaError_t e = capture_step(c, phase, c->stream);
  CK(cudaStreamEndCapture(c->stream, &g));
  CK(e);
  CK(cudaGraphInstantiate(&c->graph[phase], g, 0));
  cudaGraphDestroy(g);
  return 0;
}

static void prof_tick(void* vc, int cls, cudaStream_t s) {
  ice_gpu_ctx* c = (ice_gpu_ctx*)vc;
  cudaEventRecord(c->ev1, s);
  cudaEventSynchronize(c->ev1);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, c->ev0, c->ev1);
  c->kms[cls] += ms;
  cudaEventRecord(c->ev0, s);
}

static long long launches_per_step(const ice_gpu_ctx* c) {
  bool finish = c->owned.empty();
  for (int p = 0; p < c->P.nfam; ++p) finish = finish && !c->fam[p].have_imp;
  long long n = finish ? 1 : 2;
  for (int p = 0; p < c->P.nfam; ++p) n += c->fam[p].have_imp ? 3 : 0;
  for (int p = 0; p < c->P.nfam; ++p) {
    const FamHost& H = c->fam[p];
    long long per = (H.ngrec + H.ncopy > 0 ? (H.ghost_split ? 2 : 1) : 0) + (c->P.shock_detector ? 1 : 0) + (own_source(c, p) ? 1 : 0) +
                    (H.nfrec + H.nzface > 0 || (!plane(c) && H.nfjob > 0)) + (H.nsum > 0);
    per += c->P.irs ? (2 + 2 * c->P.ndir) : 1;
    n += per * c->P.nrk;
  }
  return n;
}

// ---------------------------------------------------------------- set-up helpers
// The tiles of the FP32-flux form's 1-D stage kernel: TX cells of a row, the last being the next tile's first.
static void tile_shape(int& TX, int& TY, int& KZ) { TX = 256; TY = 1; KZ = 1; }

// The schedule of a closure: its row of the tuned table (ice_tune.h), or ICE_GPU_TUNE="kz,zpass,wcap".
static TuneRow tune_of(int closure) {
  TuneRow r = kTune[std::min(std::max(closure, 1), 3) - 1];
  if (const char* e = getenv("ICE_GPU_TUNE")) {
    int kz, zp, wc;
    if (sscanf(e, "%d,%d,%d", &kz, &zp, &wc) == 3 && kz >= 1 && kz <= 32 && zp >= 0 && wc >= 1) r = TuneRow{kz, zp, wc};
  }
  return r;
}

// The march length of the flux kernel along one direction, over the owned blocks: per candidate length the
// threads there are, in waves of the GPU's resident threads, times what a thread does (its faces and the
// extra slope a march starts with, tr.zpass thirds of a face). A run that fills the GPU marches far, a small
// one takes one face a thread.
static int choose_march(const ice_gpu_ctx* c, int d, double slots, const TuneRow& tr) {
  static const int cand[] = {1, 2, 3, 4, 6, 8, 12, 16, 24, 32};
  int best = 1;
  double best_t = 0.0;
  for (int len : cand) {
    if (len > tr.kz) break;
    double thr = 0.0, longest = 0.0;
    for (int b = 0; b < c->nb; ++b) {
      if (!c->owned.empty() && !c->owned[b]) continue;
      const int* n = &c->dims[3 * b];
      const int m = n[d], nch = (m + len - 1) / len;
      thr += (double)n[0] * n[1] * n[2] / m * nch;
      longest = std::max(longest, (double)((m + nch - 1) / nch));
    }
    const double t = std::max(1.0, thr / slots) * (longest + tr.zpass / 3.0);
    if (best_t == 0.0 || t < 0.99 * best_t) { best = len; best_t = t; }
  }
  return best;
}

// The flux kernel's CTAs (ice_sweep.cuh) over the owned blocks, by slabs of wcap planes: the x, y and z faces of
// a slab one after the other, so that the second and third read the state from L2.
static int build_sweeps(ice_gpu_ctx* c) {
  int dev = 0;
  CK(cudaGetDevice(&dev));
  CK(cudaDeviceGetAttribute(&c->nsm, cudaDevAttrMultiProcessorCount, dev));
  const bool f64 = sweeps64(c);
  for (int p = 0; p < c->P.nfam; ++p) {
    FamHost& H = c->fam[p];
    const TuneRow tr = tune_of(H.closure);
    const int occ = H.closure == ICE_CLOSURE_AG   ? (f64 ? SweepOcc<AG, double>::flux : SweepOcc<AG, float>::flux)
                    : H.closure == ICE_CLOSURE_IG ? (f64 ? SweepOcc<IG, double>::flux : SweepOcc<IG, float>::flux)
                                                  : (f64 ? SweepOcc<MK, double>::flux : SweepOcc<MK, float>::flux);
    const double slots = (double)c->nsm * occ * SW_NT;
    // groups of SW_XC cells an x CTA takes: the start of a CTA (its job, its block, their loads) is a chain of its
    // own, 183 / 172 us for one / four groups (FP32 IG, 128 x 126 x 129); one in a run too small for two waves
    const int cx = (int)std::min(4.0, std::max(1.0, (double)c->NI / (2.0 * slots)));
    const int cy = choose_march(c, 1, slots, tr), cz = choose_march(c, 2, slots, tr);
    std::vector<SweepJob> f;
    std::vector<int> slab;           // per job, its slab of the block
    for (int b = 0; b < c->nb; ++b) {
      if (!c->owned.empty() && !c->owned[b]) continue;       // a split run steps its own blocks
      const int ni = c->dims[3 * b], nj = c->dims[3 * b + 1], nk = c->dims[3 * b + 2];
      const long long ncell = (long long)ni * nj * nk;
      auto put = [&](int kind, long long base, int c0, int n, int k) {
        f.push_back(SweepJob{b, kind, (int)base, c0, n});
        slab.push_back(k / tr.wcap);
      };
      if (ni >= 2)
        for (long long q = 0; q < ncell; q += (long long)cx * SW_XC) put(SW_X, q, 0, cx, (int)(q / ((long long)ni * nj)));
      auto chunks = [&](int kind, int n, int len, long long cols) {
        const int nch = (n + len - 1) / len, base = n / nch, extra = n % nch;
        for (long long q = 0; q < cols; q += SW_NT)
          for (int ch = 0, k = 0; ch < nch; ++ch) {
            const int hz = base + (ch < extra ? 1 : 0);
            put(kind, q, k, hz, kind == SW_Y ? (int)(q / ni) : k);
            k += hz;
          }
      };
      if (nj >= 2) chunks(SW_Y, nj - 1, cy, (long long)ni * nk);
      if (nk >= 2) chunks(SW_Z, nk - 1, cz, (long long)ni * nj);
    }
    std::vector<int> ord(f.size());
    for (size_t q = 0; q < ord.size(); ++q) ord[q] = (int)q;
    std::stable_sort(ord.begin(), ord.end(), [&](int x, int y) {
      if (f[x].b != f[y].b) return f[x].b < f[y].b;
      return slab[x] < slab[y];
    });
    std::vector<SweepJob> g(f.size());
    for (size_t q = 0; q < ord.size(); ++q) g[q] = f[ord[q]];
    H.nfjob = (int)g.size();
    CK(with_room(c, H.fjobs, g.size()));
    if (!g.empty()) CK(cudaMemcpy(H.fjobs.p, g.data(), g.size() * sizeof(SweepJob), cudaMemcpyHostToDevice));
  }
  return 0;
}

// What a step keeps beyond its states and inputs: the metric rows (after a block's metrics), the face fluxes,
// the largest family's, in the word of the running form, and the FP32-flux form's weights; the faces no record gives a flux
// are zero and stay so (after a change of form, after a new boundary table). 96 + 12 nc (24 nc) bytes a cell
// in 3-D. Made when the blocks and the table are complete (setup_work), so that the first step does not pay for
// them; on a device that the rest fills, in managed memory: such a run is slower, not refused.
static int ensure_flux(ice_gpu_ctx* c) {
  if (!c->rows_ok) {
    if (!c->row.p) CK(c->row.alloc_or_managed((size_t)12 * c->NI));
    k_rows<<<grid_of(c->NI), 256, 0, c->stream>>>(c->M.p, c->row.p, c->NI, 0, c->NI);
    CK(cudaGetLastError());
    c->rows_ok = true;
  }
  const int word = sweeps64(c) ? 8 : 4;
  if (word == 4 && c->P.shock_detector && !plane(c))
    for (int p = 0; p < c->P.nfam; ++p)
      if (!c->fam[p].betaf.p) {
        CK(c->fam[p].betaf.alloc_or_managed(c->NI));
        free_graphs(c);
      }
  if (c->flux_ok && c->flux_word == word) return 0;
  size_t nc = 0;
  for (int p = 0; p < c->P.nfam; ++p) nc = std::max(nc, (size_t)c->fam[p].nc);
  CK(cudaStreamSynchronize(c->stream));
  if (c->flux_word != word) free_graphs(c);      // they hold the pointers and the form
  size_t n = 0;
  for (int d = 0; d < 3; ++d) {
    c->flux_at[d] = n;
    n += (nc * c->NF[d] * word + 255) & ~(size_t)255;
  }
  if (c->flux_word != word) {
    c->flux_word = 0;
    CK(c->flux.alloc_or_managed(n));
  }
  CK(cudaMemsetAsync(c->flux.p, 0, n, c->stream));
  c->flux_word = word;
  c->flux_ok = true;
  return 0;
}

// After a block's metrics or a boundary table: a step's work memory, once both are complete.
static int setup_work(ice_gpu_ctx* c) {
  if (!c->have_records || !std::all_of(c->have_block.begin(), c->have_block.end(), [](bool x) { return x; })) return 0;
  return ensure_flux(c);
}

static int build_tiles(ice_gpu_ctx* c) {
  tile_shape(c->TX, c->TY, c->KZ);
  std::vector<Tile> t;
  if (c->P.ndir == 1) {
    for (int b = 0; b < c->nb; ++b) {
      if (!c->owned.empty() && !c->owned[b]) continue;       // a split run steps its own blocks
      int ni = c->dims[3 * b], nj = c->dims[3 * b + 1], nk = c->dims[3 * b + 2];
      int sx = ni >= 2 ? c->TX - 1 : 1;
      for (int k = 0; k < nk; ++k)
        for (int j = 0; j < nj; ++j)
          for (int i = 0; i < ni; i += sx) t.push_back(Tile{b, i, j, k, 1});
    }
    c->ntile = (int)t.size();
    CK(with_room(c, c->tiles, t.size()));
    CK(cudaMemcpy(c->tiles.p, t.data(), t.size() * sizeof(Tile), cudaMemcpyHostToDevice));
  }
  if (int rc = build_sweeps(c)) return rc;
  // norm chunks: 2048 cells of one block each
  std::vector<NormChunk> ch;
  c->chunk_block.clear();
  for (int b = 0; b < c->nb; ++b) {
    long long n = (long long)c->dims[3 * b] * c->dims[3 * b + 1] * c->dims[3 * b + 2];
    for (long long q = 0; q < n; q += 2048) {
      ch.push_back(NormChunk{b, c->hblk[b].ioff + q, c->hblk[b].ioff + std::min(n, q + 2048)});
      c->chunk_block.push_back(b);
    }
  }
  c->nchunk = (int)ch.size();
  CK(with_room(c, c->chunks, ch.size()));
  CK(cudaMemcpy(c->chunks.p, ch.data(), ch.size() * sizeof(NormChunk), cudaMemcpyHostToDevice));
  CK(with_room(c, c->npart, (size_t)c->nchunk * 5));
  return 0;
}

extern "C" {

int ice_gpu_create(const ice_gpu_params* P, int32_t nblocks, const int32_t* dims, ice_gpu_ctx** out) {
  ice_gpu_ctx* c = nullptr;
  if (!P || !dims || !out || nblocks < 1) return fail(nullptr, ICE_GPU_EINVAL, "create: null argument or no block");
  if (P->nfam < 1 || P->nfam > kMaxF) return fail(nullptr, ICE_GPU_EINVAL, "create: nfam %d out of 1..%d", P->nfam, kMaxF);
  if (P->nrk < 1 || P->nrk > 3) return fail(nullptr, ICE_GPU_EINVAL, "create: nrk %d", P->nrk);
  if (P->ndir < 1 || P->ndir > 3) return fail(nullptr, ICE_GPU_EINVAL, "create: ndir %d", P->ndir);
  for (int p = 0; p < P->nfam; ++p) {
    const ice_gpu_family& f = P->fam[p];
    if (f.closure < 1 || f.closure > 3) return fail(nullptr, ICE_GPU_EINVAL, "family %d: closure %d", p + 1, f.closure);
    if (f.riemann == ICE_RIEMANN_SAUREL && f.closure != ICE_CLOSURE_MK)
      return fail(nullptr, ICE_GPU_EINVAL, "family %d: riemann-solver = Saurel is specific to the MK closure; use Rusanov or HLLE", p + 1);
    if (f.liq != 0 || f.boil != 0)
      return fail(nullptr, ICE_GPU_EINVAL, "family %d: liquid-conduction P2T and boiling ZGR are not supported", p + 1);
  }
  if (P->irs && P->time_accurate)
    return fail(nullptr, ICE_GPU_EINVAL, "irs = true needs time-accurate = false (Assign_Setup.f90:79-83)");
  std::unique_ptr<ice_gpu_ctx> u(new ice_gpu_ctx);
  c = u.get();
  c->P = *P;
  c->nb = nblocks;
  c->dims.assign(dims, dims + 3 * nblocks);
  c->have_block.assign(nblocks, false);
  c->gas_set.assign(nblocks, false);
  long long G = 0, I = 0, R = 0, F0 = 0, F1 = 0, F2 = 0;
  for (int b = 0; b < nblocks; ++b) {
    int ni = dims[3 * b], nj = dims[3 * b + 1], nk = dims[3 * b + 2];
    if (ni < 1 || nj < 1 || nk < 1) return fail(nullptr, ICE_GPU_EINVAL, "block %d: dims %d %d %d", b + 1, ni, nj, nk);
    if ((long long)ni * nj * nk >= (1LL << 31))
      return fail(nullptr, ICE_GPU_EINVAL, "block %d: %lld cells, at most 2^31 - 1 per block", b + 1, (long long)ni * nj * nk);
    DBlock B;
    B.ni = ni; B.nj = nj; B.nk = nk;
    B.px = (ni + 4 + 1) & ~1;
    B.pxy = (long long)B.px * (nj + 4);
    B.goff = G; B.ioff = I; B.roff = R; B.foff[0] = F0; B.foff[1] = F1; B.foff[2] = F2;
    G += B.pxy * (nk + 4);
    c->ng_max = std::max(c->ng_max, (long long)(ni + 4) * (nj + 4) * (nk + 4));
    I += (long long)ni * nj * nk;
    R += (long long)(ni + 2) * (nj + 2) * (nk + 2);
    F0 += (long long)(ni + 1) * nj * nk; F1 += (long long)ni * (nj + 1) * nk; F2 += (long long)ni * nj * (nk + 1);
    c->hblk.push_back(B);
  }
  c->NG = G; c->NI = I; c->NR = R; c->NF[0] = F0; c->NF[1] = F1; c->NF[2] = F2;
  cudaError_t e;
#define CKC(call) do { e = (call); if (e != cudaSuccess) return fail(nullptr, ICE_GPU_ECUDA, "%s: %s", #call, cudaGetErrorString(e)); } while (0)
  CKC(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
  CKC(c->blk.alloc(nblocks));
  CKC(cudaMemcpy(c->blk.p, c->hblk.data(), nblocks * sizeof(DBlock), cudaMemcpyHostToDevice));
  for (int d = 0; d < 3; ++d) CKC(c->face[d].alloc((size_t)4 * c->NF[d]));
  CKC(c->vol.alloc(I));
  CKC(c->dl.alloc((size_t)3 * R));
  CKC(c->M.alloc((size_t)9 * I));
  if (P->coupled) CKC(c->gas.alloc((size_t)9 * I));
  for (int p = 0; p < P->nfam; ++p) {
    FamHost& H = c->fam[p];
    H.closure = P->fam[p].closure; H.riemann = P->fam[p].riemann; H.nc = nbase_of(H.closure);
    for (int s = 0; s < 3; ++s) {
      CKC(H.S[s].alloc((size_t)H.nc * G));
      // poison: a ghost cell no record fills stays NaN, as Allocate_Block leaves it
      CKC(cudaMemset(H.S[s].p, 0xFF, sizeof(double) * H.nc * G));
    }
    CKC(H.inj.alloc(G)); CKC(cudaMemset(H.inj.p, 0, G));
    CKC(H.dt.alloc(I));
    CKC(H.tau.alloc(I));
    std::vector<double> inf(I, INFINITY);
    CKC(cudaMemcpy(H.tau.p, inf.data(), I * sizeof(double), cudaMemcpyHostToDevice));
    CKC(H.beta.alloc(I));
    std::vector<double> one(I, 1.0);
    CKC(cudaMemcpy(H.beta.p, one.data(), I * sizeof(double), cudaMemcpyHostToDevice));
    if (P->coupled) CKC(H.src.alloc((size_t)H.nc * I));
    if (P->irs) { CKC(H.resid.alloc((size_t)H.nc * I)); CKC(H.resid2.alloc((size_t)H.nc * I)); CKC(H.resid3.alloc((size_t)H.nc * I)); }
  }
  CKC(c->st.alloc(1));
  Status s0; memset(&s0, 0, sizeof s0);
  s0.dtbits = kDtStart;
  CKC(cudaMemcpy(c->st.p, &s0, sizeof s0, cudaMemcpyHostToDevice));
  CKC(cudaEventCreate(&c->ev0)); CKC(cudaEventCreate(&c->ev1));
  CKC(cudaEventCreate(&c->t0)); CKC(cudaEventCreate(&c->t1));
  CKC(cudaMallocHost((void**)&c->hst, sizeof(Status)));
#undef CKC
  if (build_tiles(c)) { g_create_err = c->err; return ICE_GPU_ECUDA; }
  *out = u.release();
  return 0;
}

int ice_gpu_destroy(ice_gpu_ctx* c) {
  if (!c) return 0;
  cudaStreamSynchronize(c->stream);
  free_graphs(c);
  if (c->ev0) cudaEventDestroy(c->ev0);
  if (c->ev1) cudaEventDestroy(c->ev1);
  if (c->t0) cudaEventDestroy(c->t0);
  if (c->t1) cudaEventDestroy(c->t1);
  if (c->hst) cudaFreeHost(c->hst);
  if (c->s_up) { cudaStreamSynchronize(c->s_up); cudaStreamDestroy(c->s_up); }
  if (c->s_down) { cudaStreamSynchronize(c->s_down); cudaStreamDestroy(c->s_down); }
  if (c->ev_up) cudaEventDestroy(c->ev_up);
  if (c->xhost) cudaFreeHost(c->xhost);
  for (auto& e : c->ev_fam) if (e) cudaEventDestroy(e);
  if (c->s_prep) cudaStreamDestroy(c->s_prep);
  if (c->ev_fork) cudaEventDestroy(c->ev_fork);
  for (auto& e : c->ev_prep) if (e) cudaEventDestroy(e);
  for (auto& e : c->ev_done) if (e) cudaEventDestroy(e);
  for (auto& e : c->ev_src) if (e) cudaEventDestroy(e);
  if (c->stream) cudaStreamDestroy(c->stream);
  delete c;
  return 0;
}

int ice_gpu_last_error(const ice_gpu_ctx* c, char* buf, int32_t n) {
  if (!buf || n <= 0) return ICE_GPU_EINVAL;
  const std::string& s = c ? c->err : g_create_err;
  strncpy(buf, s.c_str(), n - 1); buf[n - 1] = 0;
  return 0;
}

int ice_gpu_set_block(ice_gpu_ctx* c, int32_t b1, const double* f1, const double* f2, const double* f3,
                      const double* vol, const double* dl, const double* M) {
  if (!c) return ICE_GPU_EINVAL;
  if (b1 < 1 || b1 > c->nb) return fail(c, ICE_GPU_EINVAL, "set_block: block %d out of range", b1);
  if (!f1 || !f2 || !f3 || !vol || !dl || !M) return fail(c, ICE_GPU_EINVAL, "set_block: null array");
  const DBlock& B = c->hblk[b1 - 1];
  int ni = B.ni, nj = B.nj, nk = B.nk;
  const double* fs[3] = {f1, f2, f3};
  long long nf[3] = {(long long)(ni + 1) * nj * nk, (long long)ni * (nj + 1) * nk, (long long)ni * nj * (nk + 1)};
  std::vector<double> tmp;
  CK(cudaStreamSynchronize(c->stream));             // the rows of the metrics before these
  for (int d = 0; d < 3; ++d) {
    tmp.resize(nf[d]);
    for (int comp = 0; comp < 4; ++comp) {
      for (long long q = 0; q < nf[d]; ++q) tmp[q] = fs[d][4 * q + comp];
      CK(cudaMemcpy(c->face[d].p + (long long)comp * c->NF[d] + B.foff[d], tmp.data(), nf[d] * sizeof(double), cudaMemcpyHostToDevice));
    }
  }
  long long ncell = (long long)ni * nj * nk, nring = (long long)(ni + 2) * (nj + 2) * (nk + 2);
  CK(cudaMemcpy(c->vol.p + B.ioff, vol, ncell * sizeof(double), cudaMemcpyHostToDevice));
  tmp.resize(nring);
  for (int comp = 0; comp < 3; ++comp) {
    for (long long q = 0; q < nring; ++q) tmp[q] = dl[3 * q + comp];
    CK(cudaMemcpy(c->dl.p + (long long)comp * c->NR + B.roff, tmp.data(), nring * sizeof(double), cudaMemcpyHostToDevice));
  }
  // M on the interior cells only (compute_dt reads nothing else)
  tmp.resize(ncell);
  for (int comp = 0; comp < 9; ++comp) {
    for (int k = 0; k < nk; ++k) for (int j = 0; j < nj; ++j) for (int i = 0; i < ni; ++i) {
      long long r = ((long long)(k + 1) * (nj + 2) + (j + 1)) * (ni + 2) + (i + 1);
      tmp[((long long)k * nj + j) * ni + i] = M[9 * r + comp];
    }
    CK(cudaMemcpy(c->M.p + (long long)comp * c->NI + B.ioff, tmp.data(), ncell * sizeof(double), cudaMemcpyHostToDevice));
  }
  CK(cudaStreamSynchronize(cudaStreamLegacy));      // the copies, which the stream's kernels do not wait for
  c->have_block[b1 - 1] = true;
  c->geo32_ok = false;
  if (!c->rows_ok) return setup_work(c);
  k_rows<<<grid_of(ncell), 256, 0, c->stream>>>(c->M.p, c->row.p, c->NI, B.ioff, ncell);     // new metrics of one block
  CK(cudaGetLastError());
  return 0;
}

int ice_gpu_set_gas(ice_gpu_ctx* c, int32_t b1, const double* prim5, const double* R, const double* gam,
                    const double* k, const double* mu) {
  if (!c) return ICE_GPU_EINVAL;
  if (!c->P.coupled) return fail(c, ICE_GPU_EINVAL, "set_gas: the run is not coupled");
  if (b1 < 1 || b1 > c->nb) return fail(c, ICE_GPU_EINVAL, "set_gas: block %d out of range", b1);
  const DBlock& B = c->hblk[b1 - 1];
  long long n = (long long)B.ni * B.nj * B.nk;
  std::vector<double> tmp(n);
  for (int comp = 0; comp < 5; ++comp) {
    for (long long q = 0; q < n; ++q) tmp[q] = prim5[5 * q + comp];
    CK(cudaMemcpy(c->gas.p + (long long)comp * c->NI + B.ioff, tmp.data(), n * sizeof(double), cudaMemcpyHostToDevice));
  }
  const double* rest[4] = {R, gam, k, mu};
  for (int comp = 0; comp < 4; ++comp)
    CK(cudaMemcpy(c->gas.p + (long long)(5 + comp) * c->NI + B.ioff, rest[comp], n * sizeof(double), cudaMemcpyHostToDevice));
  c->gas_set[b1 - 1] = true;
  c->geo32_ok = false;                 // the FP32-flux form's copy of the gas is made again
  c->have_gas = std::all_of(c->gas_set.begin(), c->gas_set.end(), [](bool x) { return x; });
  return 0;
}

int ice_gpu_upload_state(ice_gpu_ctx* c, int32_t b1, int32_t p1, const double* prim, const uint8_t* inj) {
  if (!c) return ICE_GPU_EINVAL;
  if (b1 < 1 || b1 > c->nb || p1 < 1 || p1 > c->P.nfam) return fail(c, ICE_GPU_EINVAL, "upload_state: bad block/family");
  if (!prim) return fail(c, ICE_GPU_EINVAL, "upload_state: null prim");
  const DBlock& B = c->hblk[b1 - 1];
  FamHost& H = c->fam[p1 - 1];
  long long ng = (long long)(B.ni + 4) * (B.nj + 4) * (B.nk + 4);
  if (!c->xfer.p) CK(with_room(c, c->xfer, (size_t)c->ng_max * kMaxNC));
  CK(cudaStreamSynchronize(c->stream));
  CK(cudaMemcpyAsync(c->xfer.p, prim, (size_t)ng * H.nc * sizeof(double), cudaMemcpyHostToDevice, c->stream));
  k_aos2soa<<<grid_of(ng), 256, 0, c->stream>>>(c->xfer.p, H.S[c->phase].p + B.goff, c->NG, ng, H.nc,
                                                 B.ni + 4, B.nj + 4, B.px);
  CK(cudaGetLastError());
  if (inj) {
    CK(cudaStreamSynchronize(c->stream));
    CK(cudaMemcpyAsync(c->xfer.p, inj, ng, cudaMemcpyHostToDevice, c->stream));
    k_inj2pool<<<grid_of(ng), 256, 0, c->stream>>>((const unsigned char*)c->xfer.p, H.inj.p + B.goff, ng,
                                                   B.ni + 4, B.nj + 4, B.px);
    CK(cudaGetLastError());
  }
  CK(cudaStreamSynchronize(c->stream));
  c->prev_phase = -1;
  return 0;
}

int ice_gpu_download_state(ice_gpu_ctx* c, int32_t b1, int32_t p1, double* prim) {
  if (!c) return ICE_GPU_EINVAL;
  if (b1 < 1 || b1 > c->nb || p1 < 1 || p1 > c->P.nfam) return fail(c, ICE_GPU_EINVAL, "download_state: bad block/family");
  const DBlock& B = c->hblk[b1 - 1];
  FamHost& H = c->fam[p1 - 1];
  long long ng = (long long)(B.ni + 4) * (B.nj + 4) * (B.nk + 4);
  if (!prim) return fail(c, ICE_GPU_EINVAL, "download_state: null prim");
  if (!c->xfer.p) CK(with_room(c, c->xfer, (size_t)c->ng_max * kMaxNC));
  k_soa2aos<<<grid_of(ng), 256, 0, c->stream>>>(H.S[c->phase].p + B.goff, c->xfer.p, c->NG, ng, H.nc,
                                                 B.ni + 4, B.nj + 4, B.px);
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(prim, c->xfer.p, (size_t)ng * H.nc * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
  CK(cudaStreamSynchronize(c->stream));
  return 0;
}

int ice_gpu_set_time(ice_gpu_ctx* c, double time, int32_t iter, int32_t iter_from_call) {
  if (!c) return ICE_GPU_EINVAL;
  Status s;
  CK(cudaStreamSynchronize(c->stream));
  CK(cudaMemcpy(&s, c->st.p, sizeof s, cudaMemcpyDeviceToHost));
  s.time = time; s.iter = iter; s.iter_from_call = iter_from_call;
  CK(cudaMemcpy(c->st.p, &s, sizeof s, cudaMemcpyHostToDevice));
  return 0;
}

int ice_gpu_set_res_reference(ice_gpu_ctx* c, double ref) {
  if (!c) return ICE_GPU_EINVAL;
  c->res_reference = ref;
  return 0;
}

int ice_gpu_get_res_reference(ice_gpu_ctx* c, double* ref) {
  if (!c) return ICE_GPU_EINVAL;
  if (!ref) return fail(c, ICE_GPU_EINVAL, "get_res_reference: null pointer");
  *ref = c->res_reference;
  return 0;
}

int ice_gpu_update_params(ice_gpu_ctx* c, const ice_gpu_params* P) {
  if (!c || !P) return ICE_GPU_EINVAL;
  if (P->nfam != c->P.nfam || P->ndir != c->P.ndir) return fail(c, ICE_GPU_EINVAL, "update_params: nfam and ndir may not change");
  for (int p = 0; p < P->nfam; ++p) {
    if (P->fam[p].closure != c->P.fam[p].closure) return fail(c, ICE_GPU_EINVAL, "update_params: closures may not change");
    if (P->fam[p].riemann == ICE_RIEMANN_SAUREL && P->fam[p].closure != ICE_CLOSURE_MK)
      return fail(c, ICE_GPU_EINVAL, "update_params: Saurel is specific to MK");
  }
  if (P->irs && P->time_accurate) return fail(c, ICE_GPU_EINVAL, "update_params: irs needs a steady run");
  if (P->irs && !c->P.irs) {
    for (int p = 0; p < c->P.nfam; ++p) {
      FamHost& H = c->fam[p];
      CK(with_room(c, H.resid, (size_t)H.nc * c->NI)); CK(with_room(c, H.resid2, (size_t)H.nc * c->NI)); CK(with_room(c, H.resid3, (size_t)H.nc * c->NI));
    }
  }
  CK(cudaStreamSynchronize(c->stream));
  c->P = *P;
  for (int p = 0; p < c->P.nfam; ++p) c->fam[p].riemann = P->fam[p].riemann;
  free_graphs(c);
  return 0;
}

// The family's device records (table order, which the record kernel indexes), and what the ghost kernel
// reads, ordered by block, face and cell with the first index fastest, so that the threads of a warp fill
// neighbouring ghost cells of one face (a face's ghosts are its own, so the order of the fills does not
// change a value): the copying records of the stepped blocks as GhostCopy, the others as they are, and the records of a face
// listed more than once one after the other in table order, for one thread.
// ghost_split: some record's block (or, for a connection, its source block) is one cell deep along the
// record's face direction, so that record's second ghost layer reads the first layer of the opposite face's
// record; the ghost kernel then runs as two launches, every record as it is.
static int upload_recs(ice_gpu_ctx* c, FamHost& H) {
  const std::vector<DRec>& dr = H.h_recs;
  CK(with_room(c, H.recs, dr.size()));
  H.ghost_split = false;
  for (const DRec& r : dr) {
    if (r.type == 0 || r.type == 102) continue;
    if (c->dims[3 * r.b + (r.f - 1) / 2] == 1) H.ghost_split = true;
    if ((r.type == 101 || r.type == 201) && c->dims[3 * r.bs + (r.fs - 1) / 2] == 1) H.ghost_split = true;
  }
  H.ngrec = H.ncopy = H.next = 0;
  if (dr.empty()) return 0;
  CK(cudaMemcpy(H.recs.p, dr.data(), dr.size() * sizeof(DRec), cudaMemcpyHostToDevice));
  std::vector<int> ord(dr.size());
  for (size_t q = 0; q < ord.size(); ++q) ord[q] = (int)q;
  std::stable_sort(ord.begin(), ord.end(), [&](int x, int y) {
    const DRec& a = dr[x]; const DRec& b = dr[y];
    if (a.b != b.b) return a.b < b.b;
    if (a.f != b.f) return a.f < b.f;
    if (a.k != b.k) return a.k < b.k;
    if (a.j != b.j) return a.j < b.j;
    return a.i < b.i;
  });
  auto at = [&](int b, int i, int j, int k) {
    const DBlock& B = c->hblk[b];
    return (unsigned)(B.goff + (k + 2) * B.pxy + (long long)(j + 2) * B.px + (i + 2));
  };
  std::vector<DRec> g;
  std::vector<GhostCopy> ext, copy;
  auto same = [&](size_t x, size_t y) {
    const DRec& a = dr[ord[x]]; const DRec& b = dr[ord[y]];
    return a.b == b.b && a.f == b.f && a.k == b.k && a.j == b.j && a.i == b.i;
  };
  size_t end = 0;                                            // of the records of one face
  for (size_t n = 0; n < ord.size(); ++n) {
    const bool lead = n == end;
    if (lead) while (end < ord.size() && same(n, end)) ++end;
    DRec r = dr[ord[n]];
    r.run = lead ? (int)(end - n) : 0;
    const bool conn = r.type == 101 || r.type == 201;
    if (H.ghost_split || r.run != 1 || !(conn || r.type == 0 || r.type == 400)) { g.push_back(r); continue; }
    if (!c->owned.empty() && !c->owned[r.b]) continue;       // a split run fills its own blocks' ghosts
    const int g0 = (r.f == 1) - (r.f == 2), g1 = (r.f == 3) - (r.f == 4), g2 = (r.f == 5) - (r.f == 6);
    GhostCopy x;
    x.g1 = at(r.b, r.i - g0, r.j - g1, r.k - g2);
    x.g2 = r.type == 0 ? kNoGhost : at(r.b, r.i - 2 * g0, r.j - 2 * g1, r.k - 2 * g2);
    if (conn) {
      const int s0 = (r.fs == 1) - (r.fs == 2), s1 = (r.fs == 3) - (r.fs == 4), s2 = (r.fs == 5) - (r.fs == 6);
      x.m = at(r.bs, r.is, r.js, r.ks); x.p = at(r.bs, r.is + s0, r.js + s1, r.ks + s2);
    } else {
      x.m = at(r.b, r.i, r.j, r.k); x.p = at(r.b, r.i + g0, r.j + g1, r.k + g2);
    }
    (conn ? copy : ext).push_back(x);
  }
  H.next = (int)ext.size();
  ext.insert(ext.end(), copy.begin(), copy.end());
  H.ncopy = (int)ext.size();
  H.ngrec = (int)g.size();
  CK(with_room(c, H.grecs, g.size()));
  CK(with_room(c, H.gcopy, ext.size()));
  if (!g.empty()) CK(cudaMemcpy(H.grecs.p, g.data(), g.size() * sizeof(DRec), cudaMemcpyHostToDevice));
  if (!ext.empty()) CK(cudaMemcpy(H.gcopy.p, ext.data(), ext.size() * sizeof(GhostCopy), cudaMemcpyHostToDevice));
  return 0;
}

// build_local_bc_index + collect_boundary_cells + collect_owner_records
// (parallel/Mod_GhostExchange.f90:103-360) for a device that owns every block.
int ice_gpu_set_records(ice_gpu_ctx* c, int32_t nrec, const int32_t* ri, const double* rr) {
  if (!c) return ICE_GPU_EINVAL;
  if (nrec < 0 || (nrec > 0 && (!ri || !rr))) return fail(c, ICE_GPU_EINVAL, "set_records: bad arguments");
  c->recs.resize(nrec);
  for (int n = 0; n < nrec; ++n) {
    const int32_t* q = ri + (long long)n * ICE_GPU_REC_INTS;
    const double* x = rr + (long long)n * ICE_GPU_REC_REALS;
    HRec& r = c->recs[n];
    r.b = q[0]; r.i = q[1]; r.j = q[2]; r.k = q[3]; r.f = q[4]; r.type = q[5]; r.p = q[6];
    r.bs = q[7]; r.is = q[8]; r.js = q[9]; r.ks = q[10]; r.fs = q[11]; r.partner = q[12]; r.owner = q[13]; r.cf = q[14];
    r.massflux = x[0]; r.velocity = x[1]; r.alpha = x[2]; r.beta = x[3]; r.temperature = x[4]; r.radius = x[5];
    r.gfixed = x[6]; r.normal_dir = x[7];
    if (r.b < 1 || r.b > c->nb || r.p < 1 || r.p > c->P.nfam || r.f < 1 || r.f > 6)
      return fail(c, ICE_GPU_EINVAL, "record %d: bad block, family or face", n + 1);
    const int* d = &c->dims[3 * (r.b - 1)];
    if (r.i < 1 || r.i > d[0] || r.j < 1 || r.j > d[1] || r.k < 1 || r.k > d[2])
      return fail(c, ICE_GPU_EINVAL, "record %d: cell %d %d %d outside block %d", n + 1, r.i, r.j, r.k, r.b);
    {
      const int ijk[3] = {r.i, r.j, r.k};
      int dd = (r.f - 1) / 2;
      if (ijk[dd] != (r.f % 2 == 1 ? 1 : d[dd]))
        return fail(c, ICE_GPU_EINVAL, "record %d: cell %d %d %d is off its face %d", n + 1, r.i, r.j, r.k, r.f);
    }
    int t = r.type;
    bool known = t == 0 || t == 101 || t == 201 || t == 102 || t == 200 || t == 300 || t == 301 || t == 400 ||
                 (t >= 401 && t <= 403);
    if (!known) return fail(c, ICE_GPU_EINVAL, "record %d: boundary code %d is not supported on the device", n + 1, t);
    if (t == 101 || t == 201) {
      if (r.bs < 1 || r.bs > c->nb) return fail(c, ICE_GPU_EINVAL, "record %d: source block %d", n + 1, r.bs);
      if (r.fs < 1 || r.fs > 6) return fail(c, ICE_GPU_EINVAL, "record %d: source face %d", n + 1, r.fs);
      const int* ds = &c->dims[3 * (r.bs - 1)];
      int g0 = (r.fs == 1) - (r.fs == 2), g1 = (r.fs == 3) - (r.fs == 4), g2 = (r.fs == 5) - (r.fs == 6);
      int s1[3] = {r.is, r.js, r.ks}, s2[3] = {r.is + g0, r.js + g1, r.ks + g2};
      for (int a = 0; a < 3; ++a)
        if (s1[a] < 1 || s1[a] > ds[a] || s2[a] < 1 || s2[a] > ds[a])
          return fail(c, ICE_GPU_EINVAL, "record %d: the two source cells of its ghosts are not inside block %d", n + 1, r.bs);
      if (r.partner < 1 || r.partner > nrec || r.cf < 1) return fail(c, ICE_GPU_EINVAL, "record %d: connection not paired", n + 1);
    }
    // read_bc (io/IO_BC.f90:264-271): a 401 or 403 inlet that injects (non-zero mass flux) reads the gas
    // speed; a run without a gas phase refuses it while the table is read. A zero-flux inlet mirrors
    // (ghost_rule, Lib_Ghost.f90:409) and reads no gas.
    if ((t == 401 || t == 403) && r.massflux != 0.0 && !c->P.coupled)
      return fail(c, ICE_GPU_EINVAL, "record %d: inlet %d takes its speed from the gas, and the run has no gas", n + 1, t);
  }
  c->have_records = false;                                // until the table is on the device whole
  std::vector<std::vector<int>> sum_cells(c->P.nfam);     // per family, a record of each cell of k_cell_sum
  for (int p = 0; p < c->P.nfam; ++p) {
    FamHost& H = c->fam[p];
    // the family's records in table order
    std::vector<int> grp;
    for (int n = 0; n < nrec; ++n) if (c->recs[n].p == p + 1) grp.push_back(n);
    std::vector<int> pos(nrec, -1);
    for (size_t q = 0; q < grp.size(); ++q) pos[grp[q]] = (int)q;
    std::vector<DRec> dr(grp.size());
    int ncf = 0;
    for (size_t q = 0; q < grp.size(); ++q) {
      const HRec& r = c->recs[grp[q]];
      DRec& d = dr[q];
      d.b = r.b - 1; d.i = r.i - 1; d.j = r.j - 1; d.k = r.k - 1; d.f = r.f; d.type = r.type;
      d.bs = r.bs - 1; d.is = r.is - 1; d.js = r.js - 1; d.ks = r.ks - 1; d.fs = r.fs;
      d.owner = r.owner; d.cf = r.cf - 1;
      if (r.type == 101 || r.type == 201) {
        const HRec& q2 = c->recs[r.partner - 1];
        d.pb = q2.b - 1; d.pi = q2.i - 1; d.pj = q2.j - 1; d.pk = q2.k - 1; d.pf = q2.f;
        ncf = std::max(ncf, r.cf);
      } else { d.pb = d.pi = d.pj = d.pk = 0; d.pf = 1; }
      d.normal_dir = r.normal_dir != 0.0;
      d.massflux = r.massflux; d.velocity = r.velocity; d.alpha = r.alpha; d.beta = r.beta;
      d.temperature = r.temperature; d.radius = r.radius; d.gfixed = r.gfixed;
      d.ca = cos(r.alpha); d.sa = sin(r.alpha); d.cb = cos(r.beta); d.sb = sin(r.beta);
      d.vol_p = 4.0/3.0*kPi*pow(r.radius, 3.0);
      d.cd0 = d.cn1 = d.cn2 = 0;
      d.run = 1; d.summed = 0;
    }
    H.nrec = (int)grp.size();
    H.h_grp = grp;
    H.h_recs = dr;
    // boundary cells: block by block in cell order, the records of a cell by face (stable)
    H.h_first.clear(); H.h_list.clear();
    for (int b = 0; b < c->nb; ++b) {
      const DBlock& B = c->hblk[b];
      long long ncell = (long long)B.ni * B.nj * B.nk;
      std::vector<int> head(ncell, -1), tail(ncell, -1), next(nrec, -1);
      for (int n : grp) {
        const HRec& r = c->recs[n];
        if (r.b != b + 1 || r.type == 0) continue;
        long long q = ((long long)(r.k - 1) * B.nj + (r.j - 1)) * B.ni + (r.i - 1);
        if (head[q] < 0) head[q] = n; else next[tail[q]] = n;
        tail[q] = n;
      }
      for (long long q = 0; q < ncell; ++q) {
        if (head[q] < 0) continue;
        int s0 = (int)H.h_list.size();
        H.h_first.push_back(s0);
        for (int n = head[q]; n >= 0; n = next[n]) H.h_list.push_back(n);
        for (size_t m = s0 + 1; m < H.h_list.size(); ++m) {
          int n = H.h_list[m]; long long l = (long long)m - 1;
          while (l >= s0 && c->recs[H.h_list[l]].f > c->recs[n].f) { H.h_list[l + 1] = H.h_list[l]; --l; }
          H.h_list[l + 1] = n;
        }
      }
    }
    H.nbc = (int)H.h_first.size();
    H.h_first.push_back((int)H.h_list.size());
    // connection owners, table order
    H.h_own.clear();
    for (int n : grp) {
      const HRec& r = c->recs[n];
      if ((r.type == 101 || r.type == 201) && r.owner) H.h_own.push_back(n);
    }
    H.nown = (int)H.h_own.size();
    H.ncf = ncf;
    // the records whose flux is computed: connections by their owner (of several with one number the last, as
    // one after the other would leave it); the symmetry records (200) of an MK family carry none (Mod_BC_Fluxes.f90:128)
    auto has_flux = [&](const DRec& d) { return d.type != 0 && !(d.type == 200 && H.closure == ICE_CLOSURE_MK); };
    auto is_conn = [](const DRec& d) { return d.type == 101 || d.type == 201; };
    std::vector<int> giver(ncf, -1);
    for (size_t q = 0; q < grp.size(); ++q)
      if (is_conn(H.h_recs[q]) && H.h_recs[q].owner) giver[H.h_recs[q].cf] = (int)q;
    // the place of x's partner among the family's records where x's flux is the partner's too, or -1
    auto taker = [&](int x) {
      const int y = pos[c->recs[grp[x]].partner - 1];
      return y >= 0 && is_conn(H.h_recs[y]) && !H.h_recs[y].owner && H.h_recs[y].cf == H.h_recs[x].cf ? y : -1;
    };
    for (int x : giver) if (x >= 0 && taker(x) < 0) H.h_recs[x].pf = 0;
    // the cells whose fluxes k_cell_sum adds: a face listed more than once, a connection that takes its number's flux otherwise
    std::vector<int> fr, sfirst, slist;
    for (size_t q = 0; q + 1 < H.h_first.size(); ++q) {
      bool sum = false;
      int face = 0;
      const size_t at = slist.size(), fat = fr.size();
      for (int l = H.h_first[q]; l < H.h_first[q + 1]; ++l) {
        const int x = pos[H.h_list[l]];
        const DRec& d = H.h_recs[x];
        if (!has_flux(d)) continue;
        sum |= d.f == face;
        face = d.f;
        slist.push_back(x);
        if (!is_conn(d)) { fr.push_back(x); continue; }
        const int g = giver[d.cf];
        sum |= d.owner ? g != x : g < 0 || taker(g) != x;
        if (g == x) fr.push_back(x);
      }
      if (!sum) { slist.resize(at); continue; }
      sfirst.push_back((int)at);
      fr.resize(std::remove_if(fr.begin() + fat, fr.end(), [&](int x) { return !is_conn(H.h_recs[x]); }) - fr.begin());
    }
    H.nsum = (int)sfirst.size();
    for (int at : sfirst) sum_cells[p].push_back(slist[at]);
    for (int x : slist) H.h_recs[x].summed = 1;
    sfirst.push_back((int)slist.size());
    CK(with_room(c, H.sfirst, sfirst.size()));
    CK(with_room(c, H.slist, std::max<size_t>(slist.size(), 1)));
    CK(cudaMemcpy(H.sfirst.p, sfirst.data(), sfirst.size() * sizeof(int), cudaMemcpyHostToDevice));
    if (!slist.empty()) CK(cudaMemcpy(H.slist.p, slist.data(), slist.size() * sizeof(int), cudaMemcpyHostToDevice));
    // the record kernel's thread order: by block, face and whether it is a connection, then by cell, so that
    // the threads of a warp take the same branches and neighbouring cells
    std::stable_sort(fr.begin(), fr.end(), [&](int x, int y) {
      const DRec& a = H.h_recs[x]; const DRec& b = H.h_recs[y];
      if (a.b != b.b) return a.b < b.b;
      if (a.f != b.f) return a.f < b.f;
      const int ca = a.type == 101 || a.type == 201, cb = b.type == 101 || b.type == 201;
      if (ca != cb) return ca < cb;
      if (a.k != b.k) return a.k < b.k;
      if (a.j != b.j) return a.j < b.j;
      return a.i < b.i;
    });
    H.nfrec = (int)fr.size();
    CK(with_room(c, H.frec, std::max<size_t>(fr.size(), 1)));
    if (!fr.empty()) CK(cudaMemcpy(H.frec.p, fr.data(), fr.size() * sizeof(int), cudaMemcpyHostToDevice));
    CK(with_room(c, H.connF, (size_t)std::max(ncf, 1) * H.nc));
    CK(cudaMemset(H.connF.p, 0, (size_t)std::max(ncf, 1) * H.nc * sizeof(double)));
    if (int rc = upload_recs(c, H)) return rc;
  }
  // the boundary faces that a family leaves without a flux where another has one: its record kernel zeroes them
  bool alike = true;       // every family has the same codes face by face, none an MK family's 200 and no cell of k_cell_sum
  for (int p = 0; p < c->P.nfam && alike; ++p) {
    const std::vector<DRec>& x = c->fam[p].h_recs; const std::vector<DRec>& y = c->fam[0].h_recs;
    alike = x.size() == y.size() && c->fam[p].nsum == 0;
    for (size_t q = 0; q < x.size() && alike; ++q)
      alike = x[q].type == y[q].type && x[q].b == y[q].b && x[q].f == y[q].f && x[q].i == y[q].i && x[q].j == y[q].j &&
              x[q].k == y[q].k && x[q].type != 200;
  }
  for (int p = 0; p < c->P.nfam; ++p) c->fam[p].nzface = 0;
  if (!alike) {
    std::vector<std::vector<long long>> has(c->P.nfam);      // (place of the face) * 4 + direction
    auto place = [&](const DRec& d, int f) {
      const DBlock& B = c->hblk[d.b];
      const int dir = (f - 1) / 2;
      const long long i = d.i + (dir == 0 && f % 2 == 0), j = d.j + (dir == 1 && f % 2 == 0),
                      k = d.k + (dir == 2 && f % 2 == 0);
      const long long ni = B.ni + (dir == 0), nj = B.nj + (dir == 1);
      return (B.foff[dir] + (k * nj + j) * ni + i) * 4 + dir;
    };
    std::vector<long long> all;
    for (int p = 0; p < c->P.nfam; ++p) {
      for (const DRec& d : c->fam[p].h_recs)
        if (d.type != 0 && !(d.type == 200 && c->fam[p].closure == ICE_CLOSURE_MK)) has[p].push_back(place(d, d.f));
      for (int x : sum_cells[p]) {               // k_cell_sum writes all of their boundary faces
        const DRec& d = c->fam[p].h_recs[x];
        const int* n = &c->dims[3 * d.b];
        const int at[3] = {d.i, d.j, d.k};
        for (int f = 1; f <= 6; ++f)
          if (at[(f - 1) / 2] == (f % 2 == 1 ? 0 : n[(f - 1) / 2] - 1)) has[p].push_back(place(d, f));
      }
      std::sort(has[p].begin(), has[p].end());
      has[p].erase(std::unique(has[p].begin(), has[p].end()), has[p].end());
      all.insert(all.end(), has[p].begin(), has[p].end());
    }
    std::sort(all.begin(), all.end());
    all.erase(std::unique(all.begin(), all.end()), all.end());
    for (int p = 0; p < c->P.nfam; ++p) {
      std::vector<ZeroFace> z;
      for (long long x : all)
        if (!std::binary_search(has[p].begin(), has[p].end(), x)) z.push_back(ZeroFace{x / 4, (int)(x % 4)});
      FamHost& H = c->fam[p];
      H.nzface = (int)z.size();
      CK(with_room(c, H.zface, z.size()));
      if (!z.empty()) CK(cudaMemcpy(H.zface.p, z.data(), z.size() * sizeof(ZeroFace), cudaMemcpyHostToDevice));
    }
  }
  c->flux_ok = false;                  // the new table's faces without a flux are zeroed again
  c->nchim = 0;
  for (const HRec& r : c->recs) c->nchim += r.type == 102;
  c->have_chimera = c->nchim == 0;
  c->have_records = true;
  free_graphs(c);
  return setup_work(c);
}

// The donors of the table's chimera records (ICE_bc_type%ni, donorID, volume_fraction,
// base/Advanced_Types_m.f90:29-31, as read_bc reads them, io/IO_BC.f90:209-236), attached to the
// family record lists that ice_gpu_set_records built.
int ice_gpu_set_chimera(ice_gpu_ctx* c, int32_t nrec, const int32_t* nchi, const int32_t* donor, const double* weight) {
  if (!c) return ICE_GPU_EINVAL;
  if (!c->have_records) return fail(c, ICE_GPU_ENOTREADY, "set_chimera: set the boundary table first");
  if (nrec != (int32_t)c->recs.size() || (nrec > 0 && !nchi))
    return fail(c, ICE_GPU_EINVAL, "set_chimera: %d records given, the table has %d", nrec, (int)c->recs.size());
  std::vector<long long> off(nrec + 1, 0);
  for (int n = 0; n < nrec; ++n) {
    const int n1 = nchi[2 * n], n2 = nchi[2 * n + 1];
    if (n1 < 0 || n2 < 0) return fail(c, ICE_GPU_EINVAL, "record %d: negative donor count", n + 1);
    if (c->recs[n].type != 102 && (n1 || n2))
      return fail(c, ICE_GPU_EINVAL, "record %d: donors given to a record of code %d", n + 1, c->recs[n].type);
    if (c->recs[n].type == 102 && (n1 < 1 || n2 < 1))
      return fail(c, ICE_GPU_EINVAL, "record %d: a chimera record needs donors for both ghost layers", n + 1);
    off[n + 1] = off[n] + n1 + n2;
  }
  if (off[nrec] > 0 && (!donor || !weight)) return fail(c, ICE_GPU_EINVAL, "set_chimera: null donor arrays");
  if (off[nrec] > (1LL << 30)) return fail(c, ICE_GPU_EINVAL, "set_chimera: %lld donors", off[nrec]);
  for (long long s = 0; s < off[nrec]; ++s) {
    const int32_t* d = donor + 4 * s;
    if (d[0] < 1 || d[0] > c->nb) return fail(c, ICE_GPU_EINVAL, "donor %lld: block %d", s + 1, d[0]);
    const int* dm = &c->dims[3 * (d[0] - 1)];
    if (d[1] < 1 || d[1] > dm[0] || d[2] < 1 || d[2] > dm[1] || d[3] < 1 || d[3] > dm[2])
      return fail(c, ICE_GPU_EINVAL, "donor %lld: cell %d %d %d is not an interior cell of block %d", s + 1, d[1], d[2],
                  d[3], d[0]);
    if (!std::isfinite(weight[s])) return fail(c, ICE_GPU_EINVAL, "donor %lld: weight is not finite", s + 1);
  }
  c->have_chimera = false;                                // until the donors are on the device whole
  for (int p = 0; p < c->P.nfam; ++p) {
    FamHost& H = c->fam[p];
    std::vector<int4> dn;
    std::vector<double> dw;
    for (size_t q = 0; q < H.h_grp.size(); ++q) {
      const int n = H.h_grp[q];
      DRec& d = H.h_recs[q];
      d.cd0 = (int)dn.size(); d.cn1 = nchi[2 * n]; d.cn2 = nchi[2 * n + 1];
      for (long long s = off[n]; s < off[n + 1]; ++s) {
        const int32_t* x = donor + 4 * s;
        dn.push_back(make_int4(x[0] - 1, x[1] - 1, x[2] - 1, x[3] - 1));
        dw.push_back(weight[s]);
      }
    }
    if (int rc = upload_recs(c, H)) return rc;
    CK(with_room(c, H.cdon, std::max<size_t>(dn.size(), 1)));
    CK(with_room(c, H.cw, std::max<size_t>(dw.size(), 1)));
    if (!dn.empty()) {
      CK(cudaMemcpy(H.cdon.p, dn.data(), dn.size() * sizeof(int4), cudaMemcpyHostToDevice));
      CK(cudaMemcpy(H.cw.p, dw.data(), dw.size() * sizeof(double), cudaMemcpyHostToDevice));
    }
  }
  c->have_chimera = true;
  free_graphs(c);
  return 0;
}

// The coupler's imports into family p of block b (ICE_cond_phase_type%imports, which the coupler's
// add_birth_rate, add_absorption_rate and add_removal_rate accumulate: coupling/Mod_Exchange.f90:270-390),
// (ncond, ni, nj, nk) in the driver's layout; NULL sets the block's to zero. The first call for a family
// allocates them (zero elsewhere), and from then on the family's steps add them to the residual and
// bound its steps as bound_empty_dt and bound_removal_dt do.
int ice_gpu_set_imports(ice_gpu_ctx* c, int32_t b1, int32_t p1, const double* imports) {
  if (!c) return ICE_GPU_EINVAL;
  if (b1 < 1 || b1 > c->nb || p1 < 1 || p1 > c->P.nfam) return fail(c, ICE_GPU_EINVAL, "set_imports: bad block/family");
  FamHost& H = c->fam[p1 - 1];
  const DBlock& B = c->hblk[b1 - 1];
  const long long n = (long long)B.ni * B.nj * B.nk;
  if (imports)
    for (long long q = 0; q < n * H.nc; ++q)
      if (!std::isfinite(imports[q])) return fail(c, ICE_GPU_EINVAL, "set_imports: a rate is not finite");
  CK(cudaStreamSynchronize(c->stream));
  if (!H.have_imp) {
    CK(with_room(c, H.imp, (size_t)c->NI * H.nc));
    CK(cudaMemset(H.imp.p, 0, (size_t)c->NI * H.nc * sizeof(double)));
    CK(with_room(c, H.escan, 1));
    H.have_imp = true;
    free_graphs(c);
  }
  std::vector<double> col((size_t)n);
  for (int v = 0; v < H.nc; ++v) {
    for (long long q = 0; q < n; ++q) col[(size_t)q] = imports ? imports[q * H.nc + v] : 0.0;
    CK(cudaMemcpy(H.imp.p + (long long)v * c->NI + B.ioff, col.data(), (size_t)n * sizeof(double), cudaMemcpyHostToDevice));
  }
  return 0;
}

// Two-way coupling (twcoupled): every stage adds its source to the step's running sum
// (add_stage_source, Mod_Explicit.f90:257-280), which the gas reads after the step as exchange_rate.
int ice_gpu_set_exchange(ice_gpu_ctx* c, int32_t on) {
  if (!c) return ICE_GPU_EINVAL;
  if (on && !c->P.coupled) return fail(c, ICE_GPU_EINVAL, "set_exchange: the run is not coupled to a gas");
  CK(cudaStreamSynchronize(c->stream));
  if (on && !c->exchange)
    for (int p = 0; p < c->P.nfam; ++p) {
      FamHost& H = c->fam[p];
      CK(with_room(c, H.xstep, (size_t)5 * c->NI));
      CK(cudaMemset(H.xstep.p, 0, (size_t)5 * c->NI * sizeof(double)));
    }
  c->exchange = on != 0;
  free_graphs(c);
  return 0;
}

// exchange_rate (coupling/Mod_Exchange.f90:60-78) of every cell of family p in block b over the last step,
// (5, ni, nj, nk): the mass, momentum and energy the gas receives per unit volume and time, the
// negated step source of the family (no burning family: nothing generated, no heat of reaction).
int ice_gpu_exchange_rate(ice_gpu_ctx* c, int32_t b1, int32_t p1, double* x) {
  if (!c) return ICE_GPU_EINVAL;
  if (b1 < 1 || b1 > c->nb || p1 < 1 || p1 > c->P.nfam || !x) return fail(c, ICE_GPU_EINVAL, "exchange_rate: bad arguments");
  if (!c->exchange) return fail(c, ICE_GPU_ENOTREADY, "exchange_rate: exchange is off (ice_gpu_set_exchange)");
  const DBlock& B = c->hblk[b1 - 1];
  const long long n = (long long)B.ni * B.nj * B.nk;
  std::vector<double> col((size_t)n);
  CK(cudaStreamSynchronize(c->stream));
  for (int m = 0; m < 5; ++m) {
    CK(cudaMemcpy(col.data(), c->fam[p1 - 1].xstep.p + (long long)m * c->NI + B.ioff, (size_t)n * sizeof(double),
                  cudaMemcpyDeviceToHost));
    for (long long q = 0; q < n; ++q) x[q * 5 + m] = -col[(size_t)q];
  }
  return 0;
}

int ice_gpu_index_maps(const ice_gpu_ctx* c, int32_t p1, int32_t* nbcell, int32_t* first, int32_t* nrecs,
                       int32_t* recs, int32_t* nown, int32_t* own) {
  if (!c || p1 < 1 || p1 > c->P.nfam || !nbcell || !nrecs || !nown) return ICE_GPU_EINVAL;
  const FamHost& H = c->fam[p1 - 1];
  *nbcell = H.nbc; *nrecs = (int)H.h_list.size(); *nown = H.nown;
  if (first) for (size_t q = 0; q < H.h_first.size(); ++q) first[q] = H.h_first[q] + 1;
  if (recs) for (size_t q = 0; q < H.h_list.size(); ++q) recs[q] = H.h_list[q] + 1;
  if (own) for (size_t q = 0; q < H.h_own.size(); ++q) own[q] = H.h_own[q] + 1;
  return 0;
}

static int check_ready(ice_gpu_ctx* c) {
  for (int b = 0; b < c->nb; ++b) if (!c->have_block[b]) return fail(c, ICE_GPU_ENOTREADY, "block %d has no metrics", b + 1);
  if (!c->have_records) return fail(c, ICE_GPU_ENOTREADY, "no boundary table");
  if (!c->have_chimera)
    return fail(c, ICE_GPU_ENOTREADY, "%d chimera records have no donors (ice_gpu_set_chimera)", c->nchim);
  // the sources of a coupled run and the ghosts of its 401 and 403 inlets read the gas of their block:
  // refused here, before any launch, where a block has none (an uncoupled run's injecting 401 or 403
  // inlets were refused by ice_gpu_set_records)
  if (c->P.coupled && !c->have_gas) return fail(c, ICE_GPU_ENOTREADY, "a coupled run needs the gas of every block");
  return 0;
}

static int finish_step(ice_gpu_ctx* c, ice_gpu_step_out* out);

int ice_gpu_step(ice_gpu_ctx* c, int32_t nsteps, ice_gpu_step_out* out) {
  if (!c) return ICE_GPU_EINVAL;
  if (int rc = check_ready(c)) return rc;
  if (int rc = build_geo32(c)) return rc;
  if (int rc = ensure_xbufs(c)) return rc;
  if (int rc = ensure_flux(c)) return rc;
  if (nsteps < 0) return fail(c, ICE_GPU_EINVAL, "step: nsteps %d", nsteps);
  cudaStream_t s = c->stream;
  if (c->profiling) {
    for (double& x : c->kms) x = 0.0;
    c->nlaunch = 0;
  }
  // res-threshold ends a steady run once its density residual has fallen by res_threshold from the
  // first non-zero one (Mod_Explicit.f90:193-240): such a run takes the norm after every step and the
  // call ends at the step that meets it
  const bool res_stop = !c->P.time_accurate && c->P.res_threshold > 0.0;
  c->res_end = false;
  CK(cudaEventRecord(c->t0, s));
  for (int n = 0; n < nsteps && !c->res_end; ++n) {
    int ph = c->phase;
    if (c->profiling) {
      CK(cudaEventRecord(c->ev0, s));
      enqueue_step(c, ph, s, prof_tick);
      c->nlaunch += launches_per_step(c);
    } else if (!c->owned.empty()) {
      // a split run: launched as it goes, the stream drained at each exchange for the hook
      c->xerr = 0;
      enqueue_step(c, ph, s, nullptr);
      if (c->xerr) {
        cudaStreamSynchronize(s);
        return c->xerr;
      }
    } else {
      if (int rc = step_graph(c, ph)) return rc;
      CK(cudaGraphLaunch(c->graph[ph], s));
    }
    c->prev_phase = ph;
    c->phase = next_phase(c, ph);
    if (res_stop) {
      if (int rc = ice_gpu_residual_norm(c, c->last_norm, nullptr)) return rc;
      if (c->res_reference == 0.0) c->res_reference = c->last_norm[0];
      c->res_end = c->res_reference > 0.0 && c->last_norm[0] <= c->P.res_threshold * c->res_reference;
    }
  }
  CK(cudaEventRecord(c->t1, s));
  CK(cudaMemcpyAsync(c->hst, c->st.p, sizeof(Status), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  return finish_step(c, out);
}

// The step's report from the status the call copied after its steps (the stream has drained).
static int finish_step(ice_gpu_ctx* c, ice_gpu_step_out* out) {
  CK(cudaGetLastError());
  const Status& h = *c->hst;
  float dms = 0.f;
  CK(cudaEventElapsedTime(&dms, c->t0, c->t1));
  int rc = 0;
  if (out) {
    out->dtglobal = h.dtglobal; out->time = h.time; out->iter = h.iter; out->status = (int)h.flags;
    const bool res_stop = !c->P.time_accurate && c->P.res_threshold > 0.0;
    out->nfloored = (int64_t)h.nfloored; out->have_norm = res_stop ? 1 : 0;
    out->nrealized = (int64_t)h.nrealized;
    bool endsim = h.iter_from_call >= c->P.itermax || c->res_end || h.time >= c->P.time_threshold;
    bool iosim = c->P.sol_diter > 0 && h.iter % c->P.sol_diter == 0;
    out->todo = endsim ? 3 : iosim ? 2 : 1;
    for (int m = 0; m < 5; ++m) out->residual[m] = res_stop ? c->last_norm[m] : 0.0;
    out->device_ms = dms;
  }
  if (h.flags & (ICE_GPU_ST_NAN_STATE | ICE_GPU_ST_BAD_RECON)) {
    rc = fail(c, ICE_GPU_ESTATE, "%s", (h.flags & ICE_GPU_ST_NAN_STATE) ?
              "invalid state after the update (NaN or infinity)" : "unphysical state at first order on a face");
  }
  return rc;
}

// ice_gpu_step with the state on the host: upload every block and family, nsteps steps, download.
// The uploads run on their own stream into one staging buffer (converted to the pools as each
// block lands); the step waits for them (its dt is a minimum over every family); the last step runs
// one graph per family, converts each family's new state as soon as its own stages end, and its
// download runs on a third stream under the next family's stages. The largest families step first,
// so that the download left after the last stage is the smallest.
int ice_gpu_step_host(ice_gpu_ctx* c, int32_t nsteps, const double* const* prim_in, double* const* prim_out,
                      ice_gpu_step_out* out) {
  if (!c) return ICE_GPU_EINVAL;
  if (int rc = check_ready(c)) return rc;
  if (int rc = build_geo32(c)) return rc;
  if (nsteps < 1) return fail(c, ICE_GPU_EINVAL, "step_host: nsteps %d", nsteps);
  if (!prim_in || !prim_out) return fail(c, ICE_GPU_EINVAL, "step_host: null array list");
  if (!c->owned.empty()) return fail(c, ICE_GPU_EINVAL, "step_host: a split run steps through ice_gpu_step");
  const int nf = c->P.nfam;
  for (int q = 0; q < c->nb * nf; ++q)
    if (!prim_in[q] || !prim_out[q]) return fail(c, ICE_GPU_EINVAL, "step_host: null array for block %d family %d",
                                                 q / nf + 1, q % nf + 1);
  if (c->profiling || (!c->P.time_accurate && c->P.res_threshold > 0.0)) {
    // per-class timing, or a steady run that may end on res-threshold inside the call: the plain
    // calls, one after another
    for (int b = 0; b < c->nb; ++b)
      for (int p = 0; p < nf; ++p)
        if (int rc = ice_gpu_upload_state(c, b + 1, p + 1, prim_in[b * nf + p], nullptr)) return rc;
    if (int rc = ice_gpu_step(c, nsteps, out)) return rc;
    for (int b = 0; b < c->nb; ++b)
      for (int p = 0; p < nf; ++p)
        if (int rc = ice_gpu_download_state(c, b + 1, p + 1, prim_out[b * nf + p])) return rc;
    return 0;
  }
  // staging offsets: block-major, family within
  std::vector<long long> off((size_t)c->nb * nf + 1, 0);
  for (int b = 0; b < c->nb; ++b) {
    const DBlock& B = c->hblk[b];
    const long long ng = (long long)(B.ni + 4) * (B.nj + 4) * (B.nk + 4);
    for (int p = 0; p < nf; ++p) off[(size_t)b * nf + p + 1] = off[(size_t)b * nf + p] + ng * c->fam[p].nc;
  }
  if (c->xall.n < (size_t)off.back()) CK(with_room(c, c->xall, (size_t)off.back()));
  if (int rc = ensure_flux(c)) return rc;        // after xall: the fluxes can do without device memory
  if (!c->s_up) CK(cudaStreamCreateWithFlags(&c->s_up, cudaStreamNonBlocking));
  if (!c->s_down) CK(cudaStreamCreateWithFlags(&c->s_down, cudaStreamNonBlocking));
  if (!c->ev_up) CK(cudaEventCreateWithFlags(&c->ev_up, cudaEventDisableTiming));
  for (int p = 0; p < nf; ++p) if (!c->ev_fam[p]) CK(cudaEventCreateWithFlags(&c->ev_fam[p], cudaEventDisableTiming));
  cudaStream_t s = c->stream;
  CK(cudaStreamSynchronize(s));
  // families by size, largest first (their order within a step does not change any result)
  std::vector<int> order(nf);
  for (int p = 0; p < nf; ++p) order[p] = p;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return c->fam[a].nc > c->fam[b].nc; });
  CK(cudaEventRecord(c->t0, c->s_up));
  const int ph0 = c->phase;
  for (int p : order)
    for (int b = 0; b < c->nb; ++b) {
      const DBlock& B = c->hblk[b];
      const FamHost& H = c->fam[p];
      const long long ng = (long long)(B.ni + 4) * (B.nj + 4) * (B.nk + 4);
      double* x = c->xall.p + off[(size_t)b * nf + p];
      CK(cudaMemcpyAsync(x, prim_in[b * nf + p], (size_t)ng * H.nc * sizeof(double), cudaMemcpyHostToDevice, c->s_up));
      k_aos2soa<<<grid_of(ng), 256, 0, c->s_up>>>(x, H.S[ph0].p + B.goff, c->NG, ng, H.nc, B.ni + 4, B.nj + 4, B.px);
      CK(cudaGetLastError());
    }
  CK(cudaEventRecord(c->ev_up, c->s_up));
  CK(cudaStreamWaitEvent(s, c->ev_up, 0));
  for (int n = 0; n < nsteps; ++n) {
    const int ph = c->phase;
    if (n + 1 < nsteps) {              // the last step alone is cut by families, for their downloads
      if (int rc = step_graph(c, ph)) return rc;
      CK(cudaGraphLaunch(c->graph[ph], s));
      c->prev_phase = ph;
      c->phase = next_phase(c, ph);
      continue;
    }
    if (!c->graph_pre[ph]) {
      cudaGraph_t g;
      CK(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
      enqueue_step_dt(c, ph, s, nullptr);
      CK(cudaStreamEndCapture(s, &g));
      CK(cudaGraphInstantiate(&c->graph_pre[ph], g, 0));
      cudaGraphDestroy(g);
    }
    CK(cudaGraphLaunch(c->graph_pre[ph], s));
    const int phn = next_phase(c, ph);
    for (int p : order) {
      if (!c->graph_fam[ph][p]) {
        cudaGraph_t g;
        CK(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        enqueue_step_family(c, p, ph, s, nullptr);
        CK(cudaStreamEndCapture(s, &g));
        CK(cudaGraphInstantiate(&c->graph_fam[ph][p], g, 0));
        cudaGraphDestroy(g);
      }
      CK(cudaGraphLaunch(c->graph_fam[ph][p], s));
      // the family's new state is final: converted to the caller's layout in order on the step's stream
      // (a conversion kernel beside the stage kernels would wait for SM room), then downloaded on the
      // copy stream beside the next family's stages
      const FamHost& H = c->fam[p];
      for (int b = 0; b < c->nb; ++b) {
        const DBlock& B = c->hblk[b];
        const long long ng = (long long)(B.ni + 4) * (B.nj + 4) * (B.nk + 4);
        double* x = c->xall.p + off[(size_t)b * nf + p];
        k_soa2aos<<<grid_of(ng), 256, 0, s>>>(H.S[phn].p + B.goff, x, c->NG, ng, H.nc, B.ni + 4, B.nj + 4, B.px);
        CK(cudaGetLastError());
      }
      CK(cudaEventRecord(c->ev_fam[p], s));
      CK(cudaStreamWaitEvent(c->s_down, c->ev_fam[p], 0));
      for (int b = 0; b < c->nb; ++b) {
        const DBlock& B = c->hblk[b];
        const long long ng = (long long)(B.ni + 4) * (B.nj + 4) * (B.nk + 4);
        CK(cudaMemcpyAsync(prim_out[b * nf + p], c->xall.p + off[(size_t)b * nf + p],
                           (size_t)ng * H.nc * sizeof(double), cudaMemcpyDeviceToHost, c->s_down));
      }
    }
    c->prev_phase = ph;
    c->phase = phn;
  }
  CK(cudaMemcpyAsync(c->hst, c->st.p, sizeof(Status), cudaMemcpyDeviceToHost, s));
  CK(cudaEventRecord(c->t1, c->s_down));
  CK(cudaStreamSynchronize(c->s_down));
  CK(cudaStreamSynchronize(s));
  return finish_step(c, out);
}

int ice_gpu_residual_norm(ice_gpu_ctx* c, double* total, double* fam) {
  if (!c || !total) return ICE_GPU_EINVAL;
  if (c->prev_phase < 0) return fail(c, ICE_GPU_ENOTREADY, "residual_norm: no step taken since the state was set");
  Geo G = make_geo(c);
  int nf = c->P.nfam;
  std::vector<double> part((size_t)c->nb * nf * 5, 0.0);
  std::vector<double> h((size_t)c->nchunk * 5);
  for (int p = 0; p < nf; ++p) {
    FamHost& H = c->fam[p];
    k_norm<<<c->nchunk, 256, 0, c->stream>>>(G, H.S[c->phase].p, H.S[c->prev_phase].p, nbase_of(H.closure) - 2,
                                             c->chunks.p, c->npart.p);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(h.data(), c->npart.p, h.size() * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    CK(cudaStreamSynchronize(c->stream));
    for (int q = 0; q < c->nchunk; ++q) {
      if (!c->owned.empty() && !c->owned[c->chunk_block[q]]) continue;    // another rank's block
      double* a = &part[((size_t)c->chunk_block[q] * nf + p) * 5];
      for (int m = 0; m < 5; ++m) a[m] = a[m] + h[(size_t)q * 5 + m];
    }
  }
  // a split run: every block's partial sums come from the one rank that steps it (the others add
  // zeros), so the sums below keep the block order of an unsplit run
  if (int rc = halo_reduce(c, ICE_GPU_HALO_NORM, part.data(), (long long)part.size())) return rc;
  double tot[5] = {0, 0, 0, 0, 0};
  for (int b = 0; b < c->nb; ++b) for (int p = 0; p < nf; ++p) for (int m = 0; m < 5; ++m) tot[m] = tot[m] + part[((size_t)b * nf + p) * 5 + m];
  for (int m = 0; m < 5; ++m) total[m] = sqrt(tot[m]);
  if (fam) {
    for (int p = 0; p < nf; ++p) {
      double f[5] = {0, 0, 0, 0, 0};
      for (int b = 0; b < c->nb; ++b) for (int m = 0; m < 5; ++m) f[m] = f[m] + part[((size_t)b * nf + p) * 5 + m];
      for (int m = 0; m < 5; ++m) fam[p * 5 + m] = sqrt(f[m]);
    }
  }
  return 0;
}

// ---------------------------------------------------------------- the block split
int ice_gpu_set_partition(ice_gpu_ctx* c, const int32_t* owned) {
  if (!c) return ICE_GPU_EINVAL;
  if (!owned) {
    c->owned.clear();
  } else {
    if (c->P.irs) return fail(c, ICE_GPU_EINVAL, "set_partition: IRS is not supported in a split run");
    if (c->nchim > 0) return fail(c, ICE_GPU_EINVAL, "set_partition: chimera records are not supported in a split run");
    for (int p = 0; p < c->P.nfam; ++p)
      if (c->fam[p].have_imp) return fail(c, ICE_GPU_EINVAL, "set_partition: imports are not supported in a split run");
    std::vector<unsigned char> o(c->nb);
    int n = 0;
    for (int b = 0; b < c->nb; ++b) { o[b] = owned[b] != 0; n += o[b]; }
    if (n == 0) return fail(c, ICE_GPU_EINVAL, "set_partition: this rank steps no block");
    c->owned = o;
    CK(with_room(c, c->owned_dev, c->nb));
    CK(cudaMemcpy(c->owned_dev.p, o.data(), c->nb, cudaMemcpyHostToDevice));
  }
  CK(cudaStreamSynchronize(c->stream));
  free_graphs(c);
  const bool had = c->have_records;
  c->have_records = false;                                   // until the tables are on the device again
  for (int p = 0; p < c->P.nfam; ++p)
    if (int rc = upload_recs(c, c->fam[p])) return rc;       // the ghost copies are of the stepped blocks
  if (build_tiles(c)) return ICE_GPU_ECUDA;
  c->have_records = had;
  return 0;
}

int ice_gpu_set_halo(ice_gpu_ctx* c, int32_t kind, int32_t p1, int32_t nsend, const int32_t* send, int32_t nrecv,
                     const int32_t* recv) {
  if (!c) return ICE_GPU_EINVAL;
  if (kind < 0 || kind > 2 || p1 < 1 || p1 > c->P.nfam || nsend < 0 || nrecv < 0 || (nsend > 0 && !send) ||
      (nrecv > 0 && !recv))
    return fail(c, ICE_GPU_EINVAL, "set_halo: bad arguments");
  const int p = p1 - 1;
  std::vector<int4> lists[2];
  for (int side = 0; side < 2; ++side) {
    const int n = side ? nrecv : nsend;
    const int32_t* e = side ? recv : send;
    for (int q = 0; q < n; ++q) {
      const int32_t* x = e + 4 * q;
      if (kind == ICE_GPU_HALO_FLUX) {
        if (x[0] < 1 || x[0] > c->fam[p].ncf) return fail(c, ICE_GPU_EINVAL, "set_halo: connection face %d", x[0]);
        lists[side].push_back(make_int4(x[0] - 1, 0, 0, 0));
        continue;
      }
      if (x[0] < 1 || x[0] > c->nb) return fail(c, ICE_GPU_EINVAL, "set_halo: block %d", x[0]);
      const int* d = &c->dims[3 * (x[0] - 1)];
      if (x[1] < 1 || x[1] > d[0] || x[2] < 1 || x[2] > d[1] || x[3] < 1 || x[3] > d[2])
        return fail(c, ICE_GPU_EINVAL, "set_halo: cell %d %d %d outside block %d", x[1], x[2], x[3], x[0]);
      lists[side].push_back(make_int4(x[0] - 1, x[1] - 1, x[2] - 1, x[3] - 1));
    }
  }
  c->hs[kind][p] = lists[0];
  c->hr[kind][p] = lists[1];
  CK(with_room(c, c->hs_dev[kind][p], lists[0].size()));
  CK(with_room(c, c->hr_dev[kind][p], lists[1].size()));
  if (!lists[0].empty())
    CK(cudaMemcpy(c->hs_dev[kind][p].p, lists[0].data(), lists[0].size() * sizeof(int4), cudaMemcpyHostToDevice));
  if (!lists[1].empty())
    CK(cudaMemcpy(c->hr_dev[kind][p].p, lists[1].data(), lists[1].size() * sizeof(int4), cudaMemcpyHostToDevice));
  return 0;
}

int ice_gpu_set_exchange_hook(ice_gpu_ctx* c, ice_gpu_exchange_fn fn, void* user) {
  if (!c) return ICE_GPU_EINVAL;
  c->hook = fn; c->hook_user = user;
  return 0;
}

int ice_gpu_set_profiling(ice_gpu_ctx* c, int32_t on) {
  if (!c) return ICE_GPU_EINVAL;
  c->profiling = on != 0;
  return 0;
}

int ice_gpu_kernel_times(const ice_gpu_ctx* c, double* ms, int32_t nclass, int64_t* nlaunch) {
  if (!c) return ICE_GPU_EINVAL;
  for (int q = 0; q < nclass && q < KC_N; ++q) ms[q] = c->kms[q];
  if (nlaunch) *nlaunch = c->profiling ? c->nlaunch : 0;
  return 0;
}

// ---------------------------------------------------------------- the evaporation surrogate
int ice_gpu_surrogate_train(ice_gpu_ctx* c, int32_t p1, const ice_gpu_surrogate_opts* o, ice_gpu_surrogate_report* rep) {
  if (!c || !o) return ICE_GPU_EINVAL;
  if (p1 < 1 || p1 > c->P.nfam) return fail(c, ICE_GPU_EINVAL, "surrogate_train: family %d out of range", p1);
  if (int rc = check_ready(c)) return rc;
  if (!c->P.coupled) return fail(c, ICE_GPU_EINVAL, "surrogate_train: the run is not coupled (no source to replace)");
  const ice_gpu_family& pf = c->P.fam[p1 - 1];
  if (pf.evap == 0) return fail(c, ICE_GPU_EINVAL, "surrogate_train: family %d has no evaporation", p1);
  if (o->nsamples < 1024 || o->nsamples > (1LL << 26) || o->epochs < 1 || o->batch < 64 || o->batch > 65536 ||
      !(o->lr > 0) || !(o->val_frac > 0 && o->val_frac < 0.5))
    return fail(c, ICE_GPU_EINVAL, "surrogate_train: options out of range");
  FamHost& H = c->fam[p1 - 1];
  DevBuf<float> X, T;
  CK(with_room(c, X, (size_t)o->nsamples * MLP_IN));
  CK(with_room(c, T, (size_t)o->nsamples * 2));
  FamDev F = make_famdev(c, p1 - 1, 1, c->phase);
  if (mlp_make_samples(H.closure, make_geo(c), F, c->P.drag, c->P.heat, c->P.blow, o->nsamples, o->seed, o->jitter,
                       X.p, T.p, c->stream))
    return fail(c, ICE_GPU_ECUDA, "surrogate_train: sample kernel: %s", cudaGetErrorString(cudaGetLastError()));
  MlpTrainOpts to{o->nsamples, o->epochs, o->batch, o->lr, o->jitter, o->seed, o->val_frac};
  MlpTrainReport tr{};
  std::string err;
  for (int again = 0;; ++again) {
    if (!mlp_train(X.p, T.p, o->nsamples, to, H.mlp_w, H.mlp_norm, tr, c->stream, err)) break;
    const cudaError_t e = cudaGetLastError();
    if (again == 0 && e == cudaErrorMemoryAllocation && yield_room(c)) continue;
    return fail(c, ICE_GPU_ECUDA, "%s: %s", err.c_str(), cudaGetErrorString(e));
  }
  std::vector<unsigned char> img;
  mlp_image(H.mlp_w.data(), img);
  CK(with_room(c, H.mlp_img, img.size()));
  CK(cudaMemcpy(H.mlp_img.p, img.data(), img.size(), cudaMemcpyHostToDevice));
  H.sur_on = true;
  free_graphs(c);
  if (rep) {
    rep->train_loss = tr.train_loss; rep->val_loss = tr.val_loss;
    rep->mdot_rel_median = tr.mdot_rel_median; rep->mdot_rel_p99 = tr.mdot_rel_p99;
    rep->q_rel_median = tr.q_rel_median; rep->q_rel_p99 = tr.q_rel_p99;
    rep->seconds = tr.seconds; rep->nsamples = tr.nsamples; rep->steps = tr.steps;
    for (int a = 0; a < MLP_IN; ++a) { rep->env_lo[a] = H.mlp_norm.env_lo[a]; rep->env_hi[a] = H.mlp_norm.env_hi[a]; }
  }
  return 0;
}

int ice_gpu_surrogate_enable(ice_gpu_ctx* c, int32_t p1, int32_t on) {
  if (!c) return ICE_GPU_EINVAL;
  if (p1 < 1 || p1 > c->P.nfam) return fail(c, ICE_GPU_EINVAL, "surrogate_enable: family %d out of range", p1);
  FamHost& H = c->fam[p1 - 1];
  if (on && !H.mlp_img.p) return fail(c, ICE_GPU_ENOTREADY, "surrogate_enable: family %d has no trained network", p1);
  CK(cudaStreamSynchronize(c->stream));
  H.sur_on = on != 0;
  free_graphs(c);
  return 0;
}

int ice_gpu_surrogate_stats(const ice_gpu_ctx* c, int64_t* counts) {
  if (!c || !counts) return ICE_GPU_EINVAL;
  Status h;
  if (cudaStreamSynchronize(c->stream) != cudaSuccess ||
      cudaMemcpy(&h, c->st.p, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return ICE_GPU_ECUDA;
  counts[0] = (int64_t)h.sur_cells; counts[1] = (int64_t)h.sur_env; counts[2] = (int64_t)h.sur_res;
  return 0;
}

int ice_gpu_mlp_grad(const float* w, const float* x, const float* t, int32_t n, float* grad, float* loss) {
  if (!w || !x || !t || !grad || !loss || n < 1 || n > 65536) return fail(nullptr, ICE_GPU_EINVAL, "mlp_grad: bad arguments");
  std::string err;
  if (mlp_grad_host(w, x, t, n, grad, loss, err)) return fail(nullptr, ICE_GPU_ECUDA, "%s", err.c_str());
  return 0;
}

int ice_gpu_mlp_infer(const float* w, const float* x, int32_t n, float* y) {
  if (!w || !x || !y || n < 1) return fail(nullptr, ICE_GPU_EINVAL, "mlp_infer: bad arguments");
  std::string err;
  if (mlp_infer_host(w, x, n, y, err)) return fail(nullptr, ICE_GPU_ECUDA, "%s", err.c_str());
  return 0;
}

// Pair_Connections (io/IO_BC.f90:360-510)
int ice_gpu_pair_connections(int32_t nb, const int32_t* dims, int32_t ngroups, int32_t nrec, int32_t* rec,
                             char* err, int32_t errlen) {
  auto R = [&](int n, int f) -> int32_t& { return rec[(long long)n * ICE_GPU_REC_INTS + f]; };
  enum { Fb, Fi, Fj, Fk, Ff, Ftype, Fp, Fbs, Fis, Fjs, Fks, Ffs, Fpartner, Fowner, Fcf };
  auto tang = [](int f, int i, int j, int k, int* t) {
    if (f <= 2) { t[0] = j; t[1] = k; } else if (f <= 4) { t[0] = i; t[1] = k; } else { t[0] = i; t[1] = j; }
  };
  auto msg = [&](const char* fmt, int a, int b2) {
    if (err && errlen > 0) snprintf(err, errlen, fmt, a, b2);
    return ICE_GPU_EINVAL;
  };
  if (nb < 1 || ngroups < 1 || nrec < 0 || !dims || (nrec > 0 && !rec)) return msg("bad arguments (%d %d)", nb, ngroups);
  for (int n = 0; n < nrec; ++n)
    if (R(n, Ftype) == 101 || R(n, Ftype) == 201) { R(n, Fpartner) = 0; R(n, Fowner) = 0; R(n, Fcf) = 0; }
  for (int p = 1; p <= ngroups; ++p) {
    std::vector<std::vector<int>> map((size_t)nb * 6);
    std::vector<int> mdim((size_t)nb * 12, 0);
    for (int n = p - 1; n < nrec; n += ngroups) {
      int ty = R(n, Ftype);
      if (ty != 101 && ty != 201) continue;
      int b = R(n, Fb), f = R(n, Ff), t[2], nt[2];
      if (b < 1 || b > nb || f < 1 || f > 6) return msg("record %d: bad block or face %d", n + 1, f);
      size_t key = (size_t)(b - 1) * 6 + (f - 1);
      if (map[key].empty()) {
        tang(f, dims[3 * (b - 1)], dims[3 * (b - 1) + 1], dims[3 * (b - 1) + 2], nt);
        map[key].assign((size_t)nt[0] * nt[1], 0);
        mdim[2 * key] = nt[0]; mdim[2 * key + 1] = nt[1];
      }
      tang(f, R(n, Fi), R(n, Fj), R(n, Fk), t);
      if (t[0] < 1 || t[1] < 1 || t[0] > mdim[2 * key] || t[1] > mdim[2 * key + 1]) return msg("record %d: cell off its face %d", n + 1, f);
      map[key][(size_t)(t[1] - 1) * mdim[2 * key] + (t[0] - 1)] = n + 1;
    }
    for (int n = p - 1; n < nrec; n += ngroups) {
      int ty = R(n, Ftype);
      if (ty != 101 && ty != 201) continue;
      int b = R(n, Fbs), f = R(n, Ffs), q = 0, t[2];
      if (b >= 1 && b <= nb && f >= 1 && f <= 6) {
        size_t key = (size_t)(b - 1) * 6 + (f - 1);
        if (!map[key].empty()) {
          tang(f, R(n, Fis), R(n, Fjs), R(n, Fks), t);
          if (t[0] >= 1 && t[1] >= 1 && t[0] <= mdim[2 * key] && t[1] <= mdim[2 * key + 1])
            q = map[key][(size_t)(t[1] - 1) * mdim[2 * key] + (t[0] - 1)];
        }
      }
      if (q) {
        int qq = q - 1;
        if (R(qq, Fi) != R(n, Fis) || R(qq, Fj) != R(n, Fjs) || R(qq, Fk) != R(n, Fks)) q = 0;
      }
      if (!q) return msg("record %d points at no connection record of its family (face %d)", n + 1, f);
      if (q == n + 1) return msg("record %d points at its own cell and face %d", n + 1, f);
      int qq = q - 1;
      if (R(qq, Ftype) != ty || R(qq, Fbs) != R(n, Fb) || R(qq, Ffs) != R(n, Ff) || R(qq, Fis) != R(n, Fi) ||
          R(qq, Fjs) != R(n, Fj) || R(qq, Fks) != R(n, Fk))
        return msg("records %d and %d do not point at each other", n + 1, q);
      int across = dims[3 * (b - 1) + (f + 1) / 2 - 1];
      if (across < 2) return msg("record %d: the block across has %d cell across its face", n + 1, across);
      R(n, Fpartner) = q;
      int fn = R(n, Ff), fq = R(qq, Ff);
      if (fn % 2 == 0 && fq % 2 == 1) R(n, Fowner) = 1;
      else if (fn % 2 == 1 && fq % 2 == 0) R(n, Fowner) = 0;
      else {
        int k1[5] = {R(n, Fb), R(n, Ff), R(n, Fk), R(n, Fj), R(n, Fi)};
        int k2[5] = {R(qq, Fb), R(qq, Ff), R(qq, Fk), R(qq, Fj), R(qq, Fi)};
        int less = 0;
        for (int m = 0; m < 5; ++m) if (k1[m] != k2[m]) { less = k1[m] < k2[m]; break; }
        R(n, Fowner) = less;
      }
    }
    int nf = 0;
    for (int n = p - 1; n < nrec; n += ngroups) {
      int ty = R(n, Ftype);
      if ((ty != 101 && ty != 201) || !R(n, Fowner)) continue;
      ++nf;
      R(n, Fcf) = nf;
      R(R(n, Fpartner) - 1, Fcf) = nf;
    }
  }
  return 0;
}

}  // extern "C"
