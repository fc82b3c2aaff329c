// ice_stage.cuh -- the launchers of the stage's kernels of one closure and precision: the Riemann
// solver and the limiter are compile-time parameters of the kernel (van Leer and minmod
// specialised, every other limiter through the run-time switch).
#pragma once
#include "ice_kernels.cuh"
#include "ice_sweep.cuh"

namespace ice {

// The cells' update (ice_sweep.cuh); in 1-D runs of the FP32-flux form the plane kernel of ice_kernels.cuh, whose
// residual sums and divisions are FP64 (one tile of 256 cells per CTA).
template <int CL, int RS, int LIM, typename R>
void launch_stage_k(const LaunchArgs& a, bool write_r) {
  constexpr int nc = NC<CL>::v;
  if constexpr (sizeof(R) == 4) {
    if (a.plane) {
      const size_t sh = sizeof(double) * 4 * nc * (size_t)a.TX * a.TY;
      static bool attr = false;
      if (!attr) {
        cudaFuncSetAttribute(k_stage<CL, RS, LIM_ANY, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, 98304);
        attr = true;
      }
      k_stage<CL, RS, LIM_ANY, R><<<a.ntile, a.TX * a.TY, sh, a.s>>>(a.G, a.F, a.tiles, a.TX, a.TY, a.KZ, a.st);
      return;
    }
  }
  k_cells<CL, R><<<(unsigned)((a.G.NI + SW_NT - 1) / SW_NT), SW_NT, 0, a.s>>>(a.G, a.F, write_r ? 1 : 0, a.st);
}

template <int CL, int RS, typename R>
void launch_stage_l(const LaunchArgs& a, bool write_r) {
  if (a.F.limiter == ICE_LIM_VANLEER) launch_stage_k<CL, RS, ICE_LIM_VANLEER, R>(a, write_r);
  else if (a.F.limiter == ICE_LIM_MINMOD) launch_stage_k<CL, RS, ICE_LIM_MINMOD, R>(a, write_r);
  else launch_stage_k<CL, RS, LIM_ANY, R>(a, write_r);
}

// The fluxes of the boundary records and the interior faces (of the records alone before the plane kernel).
template <int CL, int RS, int LIM, typename R>
void launch_flux_k(const LaunchArgs& a) {
  const int nrb = (a.nfrec + a.F.nzface + SW_NT - 1) / SW_NT;
  if (a.plane) {
    if constexpr (sizeof(R) == 4) {
      if (nrb > 0) k_rec<CL, RS, LIM, R><<<nrb, SW_NT, 0, a.s>>>(a.G, a.F, a.recs, a.frec, a.nfrec, a.st);
    }
  } else if (nrb + a.nfjob > 0) {
    k_flux<CL, RS, LIM, R><<<nrb + a.nfjob, SW_NT, 0, a.s>>>(a.G, a.F, a.fjobs, a.recs, a.frec, a.nfrec, nrb, a.st);
  }
  if (a.xchg) {                                  // connection fluxes to the partners another rank steps
    a.xchg(a, ICE_GPU_HALO_FLUX);
    if (a.nrec > 0) k_conn_in<CL, R><<<(a.nrec + 127) / 128, 128, 0, a.s>>>(a.G, a.F, a.recs, a.nrec);
  }
  if (a.nsum > 0)
    k_cell_sum<CL, RS, R><<<(a.nsum + 127) / 128, 128, 0, a.s>>>(a.G, a.F, a.recs, a.sfirst, a.slist, a.nsum, a.plane ? 3 : 1, a.st);
}

// The Jameson weights as the faces read them: in the precision of the fluxes, in FP64 for the plane kernel.
template <typename R>
void launch_beta_t(const LaunchArgs& a) {
  const unsigned g = (unsigned)((a.G.NI + 255) / 256);
  if (a.plane) k_beta<double><<<g, 256, 0, a.s>>>(a.G, a.F);
  else k_beta<R><<<g, 256, 0, a.s>>>(a.G, a.F);
}

template <int CL, int RS, typename R>
void launch_flux_l(const LaunchArgs& a) {
  if (a.F.limiter == ICE_LIM_VANLEER) launch_flux_k<CL, RS, ICE_LIM_VANLEER, R>(a);
  else if (a.F.limiter == ICE_LIM_MINMOD) launch_flux_k<CL, RS, ICE_LIM_MINMOD, R>(a);
  else launch_flux_k<CL, RS, LIM_ANY, R>(a);
}

template <int CL, typename R>
void launch_flux_t(const LaunchArgs& a) {
  if constexpr (CL == MK) {
    if (a.F.riemann == ICE_RIEMANN_SAUREL) { launch_flux_l<CL, ICE_RIEMANN_SAUREL, R>(a); return; }
  }
  if (a.F.riemann == ICE_RIEMANN_HLLE) launch_flux_l<CL, ICE_RIEMANN_HLLE, R>(a);
  else launch_flux_l<CL, ICE_RIEMANN_RUSANOV, R>(a);
}

template <typename R>
void launch_pack_beta_t(const LaunchArgs& a, const int4* e, int n, double* out) {
  k_pack_beta<R><<<(unsigned)((n + 127) / 128), 128, 0, a.s>>>(a.G, a.F, e, n, out);
}

template <int CL, typename R>
void launch_source_t(const LaunchArgs& a) {
  k_source<CL, R><<<(unsigned)((a.G.NI + 255) / 256), 256, 0, a.s>>>(a.G, a.F);
}

template <int CL, typename R>
void launch_stage_t(const LaunchArgs& a, bool write_r) {
  if constexpr (CL == MK) {
    if (a.F.riemann == ICE_RIEMANN_SAUREL) { launch_stage_l<CL, ICE_RIEMANN_SAUREL, R>(a, write_r); return; }
  }
  if (a.F.riemann == ICE_RIEMANN_HLLE) launch_stage_l<CL, ICE_RIEMANN_HLLE, R>(a, write_r);
  else launch_stage_l<CL, ICE_RIEMANN_RUSANOV, R>(a, write_r);
}

}  // namespace ice
