// ice_layout.cuh -- the device layout of the solve stage: blocks, geometry, records, status,
// the per-family view the kernels read, and the launch interface of the per-closure units.
#pragma once
#include <cuda_runtime.h>
#include "ice_physics.cuh"

namespace ice {


// ------------------------------------------------------------------ device layout
struct DBlock {
  int ni, nj, nk;
  int px;             // row pitch of the ghost-cell pools: ni + 4 rounded up to even, so that every row,
                      // plane and block starts on a 16-byte boundary
  long long pxy;      // plane pitch, px * (nj + 4)
  long long goff;     // ghost-cell pools (1-gc:n+gc)^3
  long long ioff;     // interior pools
  long long roff;     // ring pools (0:n+1)^3
  long long foff[3];  // face pools of each direction
};

struct Geo {                 // geometry shared by the families
  const DBlock* blk;
  int nb;
  long long NG, NI, NR, NF[3];
  const double* face[3];     // 4 SoA components (nx, ny, nz, A) of NF[d] each
  const double* vol;         // NI
  const double* dl;          // 3 SoA components of NR
  const double* M;           // 9 SoA components of NI (column-major c(3,3))
  const double* row;         // per direction the metric row's unit vector and modulus, 4 SoA components of NI each
  const double* gas;         // 9 SoA components of NI: rho u v w T R gam k mu
  // the FP32-flux form's copies of the face geometry (nx, ny, nz, A of a face in one 16-byte word) and
  // of the cell lengths, rounded once from the FP64 arrays above (null in the plain form)
  const float4* ff[3];
  const float* dlf;
  const float* gasf;         // the FP32-flux form's copy of the frozen gas (coupled runs), rounded once
  // a split run (ice_gpu_set_partition): per block, whether this rank steps it; null when it steps all
  const unsigned char* owned;
};
__device__ __forceinline__ bool stepped(const Geo& G, int b) { return !G.owned || G.owned[b]; }


struct DRec {                // one boundary record, 0-based cells
  int b, i, j, k, f, type;
  int bs, is, js, ks, fs;
  int owner, cf;             // cf 0-based (-1 when none)
  int run;                   // among the ghost kernel's records: this one and those of the same face after it; 0 after the first
  int pb, pi, pj, pk, pf;    // the partner's cell and its own face (connections; fs says where the ghosts come from), pf 0
                             // where the owner's flux is not the partner's (k_cell_sum)
  int normal_dir;
  double massflux, velocity, alpha, beta, temperature, radius, gfixed;
  // host-computed once per record (the platform libm of the driver's host, as the
  // reference's ghost_record evaluates them): cos/sin of the inlet angles and 4/3 pi r^3
  double ca, sa, cb, sb, vol_p;
  // chimera (102): donors cd0 .. cd0 + cn1 - 1 of ghost layer 1, then cn2 of layer 2, in the family's
  // donor arrays (FamDev::cdon, cw)
  int cd0, cn1, cn2;
  int summed;                // k_cell_sum gives the cell's boundary faces
};

// The two ghost cells of a record that copies cells (0, 400, 101, 201), as places in a variable's pool: the first
// layer g1 takes m, the second g2 takes p (a 400 record 3 g1 - 3 m + p); code 0 has no second (g2 = kNoGhost).
// Sixteen bytes in place of a record's 192. A pool has fewer than 2^32 places: three buffers of six
// doubles for each are more than the GPU holds.
struct GhostCopy { unsigned m, p, g1, g2; };
constexpr unsigned kNoGhost = 0xffffffffu;

struct Status {
  unsigned int flags;
  unsigned int done;          // CTAs of the step kernel that have given their minimum (k_dt_all)
  unsigned long long nfloored;
  unsigned long long dtbits;  // running min of dt as the bits of a positive double
  double dtglobal;
  double time;
  int iter;
  int iter_from_call;
  unsigned long long sur_cells, sur_env, sur_res;   // surrogate: cells, envelope and check fallbacks
  unsigned long long nrealized;  // cells the chosen form's realizability correction changed
};

__device__ __forceinline__ long long gidx(const DBlock& B, int i, int j, int k) {
  return B.goff + (long long)(k + 2) * B.pxy + (long long)(j + 2) * B.px + (i + 2);
}
__device__ __forceinline__ long long iidx(const DBlock& B, int i, int j, int k) {
  return B.ioff + ((long long)k * B.nj + j) * B.ni + i;
}
__device__ __forceinline__ long long ridx(const DBlock& B, int i, int j, int k) {
  return B.roff + ((long long)(k + 1) * (B.nj + 2) + (j + 1)) * (B.ni + 2) + (i + 1);
}
// face d with Fortran index F (the 1-based index of the cell below it along d), other indices 0-based
__device__ __forceinline__ long long fidx(const DBlock& B, int d, int i, int j, int k, int F) {
  if (d == 0) return B.foff[0] + ((long long)k * B.nj + j) * (B.ni + 1) + F;
  if (d == 1) return B.foff[1] + ((long long)k * (B.nj + 1) + F) * B.ni + i;
  return B.foff[2] + ((long long)F * B.nj + j) * B.ni + i;
}
__device__ __forceinline__ long long gstride(const DBlock& B, int d) {
  return d == 0 ? 1LL : d == 1 ? (long long)B.px : B.pxy;
}

struct ZeroFace { long long at; int d; };    // a face: its place in direction d's flux array

struct FamDev {              // what the kernels of one family read
  int closure, riemann, nc, limiter, sd, coupled, drag, heat, blow;
  unsigned int frozen_mask;  // bit v: slot v+1 frozen
  Mat mat;
  const double* U0;          // pointwise U_0
  const double* Up;          // stencil U_{k-1}
  double* Uo;                // U_k
  double* Ug;                // buffer whose ghosts the ghost kernels fill (== Up)
  unsigned char* inj;
  const double* beta;        // NI, or null (1)
  double* betaw;
  void* betaR;               // NI: the Jameson weights of a stage in the form's precision (ice_sweep.cuh)
  const double* dt;          // NI (steady) or null
  const double* dtg;         // &status->dtglobal (time-accurate)
  double* tau;               // NI
  double* S;                 // [v][NI]: the stage's source (coupled runs)
  float* Sf;                 // the FP32-flux form's source, [v][NI] floats in the same buffer (else null)
  double* connF;             // [ncf][nc]: a split run's connection fluxes on their way to and from other ranks, and those
                             // k_cell_sum reads (else null)
  void* Ff[3];               // the face fluxes of a stage [v][NF] per direction, in the form's precision; a face
                             // of the block's boundary holds its record's flux, zero where no record has one
  const ZeroFace* zface;     // the boundary faces without a flux that another family's stage gave one
  int nzface;
  const int4* cdon;          // chimera donors: 0-based block, i, j, k
  const double* cw;          // chimera donor weights
  const double* imports;     // [v][NI]: the coupler's rates into the cells, or null
  double* xstep;             // [5][NI]: the step's weighted source in slots 1-4 and the energy slot, or null
  int xfirst;                // this stage starts the running sum (stage 1)
  double* resid;             // IRS: [v][NI]
  double rk;
  int write_tau;
  int src_ready;             // S holds this stage's source already (its own kernel or the surrogate's ran)
  int realize;               // the FP32-flux form's realizability correction is on
};

// bound_empty_dt's reductions over one family's cells, as the bits of non-negative doubles (which
// order as their bits): the smallest step of an occupied cell, the smallest step of a source, the
// largest speed per axis, and whether a source fills anything.
struct EmptyScan {
  unsigned long long floor_bits, src_bits, umax_bits[3];
  unsigned int filled, pad;
};

// A tile of the 1-D stage kernel.
struct Tile { int b, i0, j0, k0, nkz; };
struct MlpNorm;

// One CTA's share of the flux kernel (ice_sweep.cuh): the x faces above n groups of SW_XC cells from base of block
// b (flat over the block), or the y or z faces above the cells c0 .. c0 + n - 1 of the columns base.. (flat over the plane
// across them).
enum { SW_X = 0, SW_Y = 1, SW_Z = 2 };
struct SweepJob { int b, kind, base, c0, n; };
struct NormChunk { int b; long long q0, q1; };

// The parts of a family's stage: its source's own kernel, its ghosts and sensor, its faces, its cells' update.
enum { PART_SOURCE = 1, PART_GHOSTS = 2, PART_FACES = 4, PART_CELLS = 8, PART_ALL = 15 };

// Everything one family's stage needs, for the launcher of its closure's translation unit.
struct LaunchArgs {
  Geo G;
  FamDev F;
  const DRec* recs; int nrec;
  const GhostCopy* gcopy; int ncopy, next;           // the ghosts that copy cells, the extrapolating ones first
  const DRec* grecs; int ngrec;                      // the other records, in the ghost kernel's order
  int ghost_split;                                   // a record's second layer reads another's first
  const int* frec; int nfrec;                        // the records whose flux is computed, in thread order
  const SweepJob* fjobs; int nfjob;                  // the flux kernel's CTAs
  const int* sfirst; const int* slist; int nsum;     // the cells of k_cell_sum and their records
  const Tile* tiles; int ntile; int TX, TY, KZ;     // the 1-D stage kernel's tiles
  bool own_source;                                   // the source has a kernel of its own
  const unsigned char* mlp_img;                      // the family's surrogate network (null: the plain closure)
  const MlpNorm* mlp_norm;
  int ndir, sd, irs, precision;
  int part;                                          // PART_* bits
  int plane;                                         // the FP32-flux form's 1-D stage kernel runs (ice_kernels.cuh)
  double irs_beta;
  double* resid; double* resid2; double* resid3;
  Status* st;
  cudaStream_t s;
  void (*tick)(void*, int, cudaStream_t);
  void* tick_ctx;
  // a split run: the exchange of one kind (ICE_GPU_HALO_CELLS, BETA, FLUX) of this family at its point
  // of the stage, called on every rank whatever its local work (null when every block is stepped here)
  void (*xchg)(const struct LaunchArgs&, int kind);
  int fam;                                           // 0-based family
};

enum { KC_DT = 0, KC_GHOST, KC_BETA, KC_BOUND, KC_STAGE, KC_IRS, KC_NORM, KC_SOURCE, KC_N };

// the boundary and ghost kernels of a family's stage (ice_fam_<closure>.cu), which call the stage
// kernel of its closure and precision (ice_stage_<closure>_<f64|f32>.cu)
void launch_family_mk(const LaunchArgs& a);
void launch_family_ig(const LaunchArgs& a);
void launch_family_ag(const LaunchArgs& a);
void launch_source_mk_f64(const LaunchArgs& a);
void launch_source_mk_f32(const LaunchArgs& a);
void launch_source_ig_f64(const LaunchArgs& a);
void launch_source_ig_f32(const LaunchArgs& a);
void launch_source_ag_f64(const LaunchArgs& a);
void launch_source_ag_f32(const LaunchArgs& a);
void launch_flux_mk_f64(const LaunchArgs& a);
void launch_beta_mk_f64(const LaunchArgs& a);
void launch_flux_mk_f32(const LaunchArgs& a);
void launch_beta_mk_f32(const LaunchArgs& a);
void launch_flux_ig_f64(const LaunchArgs& a);
void launch_beta_ig_f64(const LaunchArgs& a);
void launch_flux_ig_f32(const LaunchArgs& a);
void launch_beta_ig_f32(const LaunchArgs& a);
void launch_flux_ag_f64(const LaunchArgs& a);
void launch_beta_ag_f64(const LaunchArgs& a);
void launch_flux_ag_f32(const LaunchArgs& a);
void launch_beta_ag_f32(const LaunchArgs& a);
void launch_pack_beta_mk_f64(const LaunchArgs& a, const int4* e, int n, double* out);
void launch_pack_beta_mk_f32(const LaunchArgs& a, const int4* e, int n, double* out);
void launch_pack_beta_ig_f64(const LaunchArgs& a, const int4* e, int n, double* out);
void launch_pack_beta_ig_f32(const LaunchArgs& a, const int4* e, int n, double* out);
void launch_pack_beta_ag_f64(const LaunchArgs& a, const int4* e, int n, double* out);
void launch_pack_beta_ag_f32(const LaunchArgs& a, const int4* e, int n, double* out);
void launch_stage_mk_f64(const LaunchArgs& a, bool write_r);
void launch_stage_mk_f32(const LaunchArgs& a, bool write_r);
void launch_stage_ig_f64(const LaunchArgs& a, bool write_r);
void launch_stage_ig_f32(const LaunchArgs& a, bool write_r);
void launch_stage_ag_f64(const LaunchArgs& a, bool write_r);
void launch_stage_ag_f32(const LaunchArgs& a, bool write_r);

}  // namespace ice
