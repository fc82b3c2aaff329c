// ice_fam.cuh -- the launcher of one family's RK stage, templated on its closure and Riemann
// solver: ghost layers, sensor, fluxes of the boundary records (in the plain form of every face),
// then the stage kernel of the closure and precision (ice_stage.cuh), and the IRS sweeps when they are on.
#pragma once
#include "ice_kernels.cuh"
#include "ice_mlp.cuh"

namespace ice {

template <int CL> inline void launch_stage_of(const LaunchArgs& a, bool write_r) {
  const bool f32 = a.precision == ICE_PREC_FP32FLUX && !write_r;
  if constexpr (CL == MK) { if (f32) launch_stage_mk_f32(a, write_r); else launch_stage_mk_f64(a, write_r); }
  else if constexpr (CL == IG) { if (f32) launch_stage_ig_f32(a, write_r); else launch_stage_ig_f64(a, write_r); }
  else { if (f32) launch_stage_ag_f32(a, write_r); else launch_stage_ag_f64(a, write_r); }
}

template <int CL> inline void launch_flux_of(const LaunchArgs& a) {
  const bool f32 = a.precision == ICE_PREC_FP32FLUX && !a.irs;
  if constexpr (CL == MK) { if (f32) launch_flux_mk_f32(a); else launch_flux_mk_f64(a); }
  else if constexpr (CL == IG) { if (f32) launch_flux_ig_f32(a); else launch_flux_ig_f64(a); }
  else { if (f32) launch_flux_ag_f32(a); else launch_flux_ag_f64(a); }
}

template <int CL> inline void launch_beta_of(const LaunchArgs& a) {
  const bool f32 = a.precision == ICE_PREC_FP32FLUX && !a.irs;
  if constexpr (CL == MK) { if (f32) launch_beta_mk_f32(a); else launch_beta_mk_f64(a); }
  else if constexpr (CL == IG) { if (f32) launch_beta_ig_f32(a); else launch_beta_ig_f64(a); }
  else { if (f32) launch_beta_ag_f32(a); else launch_beta_ag_f64(a); }
}

template <int CL> inline void launch_source_of(const LaunchArgs& a) {
  const bool f32 = a.precision == ICE_PREC_FP32FLUX && !a.irs;
  if constexpr (CL == MK) { if (f32) launch_source_mk_f32(a); else launch_source_mk_f64(a); }
  else if constexpr (CL == IG) { if (f32) launch_source_ig_f32(a); else launch_source_ig_f64(a); }
  else { if (f32) launch_source_ag_f32(a); else launch_source_ag_f64(a); }
}

template <int CL, int RS>
void launch_family_t(const LaunchArgs& a) {
  constexpr int nc = NC<CL>::v;
  cudaStream_t s = a.s;
  auto tick = [&](int cls) { if (a.tick) a.tick(a.tick_ctx, cls, s); };
  auto grid = [](long long n, int t) { return (unsigned)((n + t - 1) / t); };
  // compute_source comes first in the stage (Mod_Explicit.f90:111-117). In the FP32-flux form the cells'
  // kernel evaluates the source of a family without evaporation itself; an evaporating family's source
  // (iterative, with lane-divergent trip counts) runs in its own kernel at full occupancy, or in the
  // surrogate's source kernel, and the stage reads it (FamDev::src_ready). So does every FP64 source, whose
  // deterministic elementary functions would take the cells' kernel's registers, and the plane kernel's.
  if ((a.part & PART_SOURCE) && a.own_source) {
    if (a.mlp_img) launch_source_mlp(CL, a, a.mlp_img, *a.mlp_norm);
    else launch_source_of<CL>(a);
    tick(KC_SOURCE);
  }
  if (a.part & PART_GHOSTS) {
    if (a.xchg) a.xchg(a, ICE_GPU_HALO_CELLS);   // the remote source cells of the ghost layers
    if (a.ngrec + a.ncopy > 0) {
      const unsigned nrb = grid(a.ngrec, 128), g = nrb + GhostPart<CL>::n * grid(a.ncopy, 128);
      if (a.ghost_split) {
        k_ghost<CL><<<g, 128, 0, s>>>(a.G, a.F, a.grecs, a.ngrec, nrb, 1, nullptr, 0, 0);
        k_ghost<CL><<<g, 128, 0, s>>>(a.G, a.F, a.grecs, a.ngrec, nrb, 2, nullptr, 0, 0);
      } else {
        k_ghost<CL><<<g, 128, 0, s>>>(a.G, a.F, a.grecs, a.ngrec, nrb, 3, a.gcopy, a.ncopy, a.next);
      }
      tick(KC_GHOST);
    }
    if (a.sd) {                                  // the Jameson sensor
      launch_beta_of<CL>(a);
      tick(KC_BETA);
    }
    if (a.xchg) a.xchg(a, ICE_GPU_HALO_BETA);    // the weights of partner cells another rank steps
  }
  if (a.part & PART_FACES) {
    launch_flux_of<CL>(a);
    tick(a.plane ? KC_BOUND : KC_STAGE);         // (else the interior faces come with the records)
  }
  if (!(a.part & PART_CELLS)) return;
  if (!a.irs) {
    launch_stage_of<CL>(a, false);
    tick(KC_STAGE);
    return;
  }
  launch_stage_of<CL>(a, true);
  tick(KC_STAGE);
  // two Jacobi sweeps per direction; each direction smooths the residual the last one left
  const long long NI = a.G.NI;
  for (int d = 0; d < a.ndir; ++d) {
    k_irs<<<grid(NI, 256), 256, 0, s>>>(a.G, nc, a.resid, a.resid, a.resid2, d, a.irs_beta);
    k_irs<<<grid(NI, 256), 256, 0, s>>>(a.G, nc, a.resid, a.resid2, a.resid3, d, a.irs_beta);
    cudaMemcpyAsync(a.resid, a.resid3, sizeof(double) * nc * NI, cudaMemcpyDeviceToDevice, s);
  }
  tick(KC_IRS);
  k_update<CL><<<grid(NI, 256), 256, 0, s>>>(a.G, a.F, a.st);
  tick(KC_STAGE);
}

}  // namespace ice
