// Launch sequence of one tracer-advection step for a batch of tracers
// (do_oce_adv_tra, lib/oce_adv_tra_driver.F90:23-294, plus the caller's
// tendency update). Included by one translation unit per precision.
#pragma once
#include <cuda_runtime.h>

#include <string>

#include "fesom_tracer_gb300.h"
#include "fgb_internal.hpp"
#include "fgb_kernels.cuh"
#include "fgb_vimpl.cuh"

namespace fgb {
#if FGB_FAST64
inline namespace fast64 {
#else
inline namespace exact64 {
#endif

template <typename R, int HOR, bool FCT>
void launch_hflux_as(const DMesh& m, const StepPtrs<R>& a, bool vf, const double2* grad, cudaStream_t s) {
  const int grid = (m.E + kEdgeTile - 1) / kEdgeTile;
  if (HOR != 0 && grad) {
    if (vf) k_hflux<R, HOR, FCT, true, HOR != 0><<<grid, kEdgeThreads, 0, s>>>(m, a, grad);
    else k_hflux<R, HOR, FCT, false, HOR != 0><<<grid, kEdgeThreads, 0, s>>>(m, a, grad);
  } else {
    if (vf) k_hflux<R, HOR, FCT, true, false><<<grid, kEdgeThreads, 0, s>>>(m, a, nullptr);
    else k_hflux<R, HOR, FCT, false, false><<<grid, kEdgeThreads, 0, s>>>(m, a, nullptr);
  }
}
template <typename R, int HOR>
void launch_hflux(const DMesh& m, const StepPtrs<R>& a, bool fct, bool vf, const double2* grad, cudaStream_t s) {
  if (fct) launch_hflux_as<R, HOR, true>(m, a, vf, grad, s);
  else launch_hflux_as<R, HOR, false>(m, a, vf, grad, s);
}

// Dynamic shared memory above the 48 KB default needs an opt-in per kernel.
template <typename F>
void allow_smem(F* kernel, size_t bytes) {
  if (bytes > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// Launches a node kernel. Tracers per chunk: the requested 1, 2 or 4 if it
// divides K, else at most 4 and as many as leave room for the kernel's blocks
// in an SM's shared memory (with room for six where the registers allow seven,
// the QR4C LO stage of 200^2x64 took 702 us against 668, four tracers, and 1533
// against 1394 with 90 layers, six tracers and T_AB apart), fewer where that
// takes a warp fewer rounds: the lanes share a chunk's (tracer, layer) pairs,
// and chunks of three 48-layer tracers leave half a round idle (eight tracers,
// T_AB apart, fast form: chunks of three 1097 us, of two 1017). Columns too
// deep for nw of them in a block's shared memory take fewer. bytes(kc): shared
// memory of one warp.
template <typename F, typename R, typename B>
void launch_nodes(F* kernel, int blocks, const DMesh& m, const StepPtrs<R>& a, int nw, int want, B bytes,
                  cudaStream_t s) {
  int kc = a.K < 4 ? a.K : 4;
  if ((want == 1 || want == 2 || want == 4) && a.K % want == 0) {
    kc = want;
  } else {
    while (kc > 1 && blocks * kNodeWarps * bytes(kc) > (size_t)220 * 1024) --kc;
    auto rounds = [&](int c) {  // of a warp over a full column's pairs
      auto of = [&](int t) { return (t * m.nz + kWarp - 1) / kWarp; };
      return a.K / c * of(c) + of(a.K % c);
    };
    for (int c = kc - 1; c >= 1; --c)
      if (rounds(c) < rounds(kc)) kc = c;
  }
  while (nw > 1 && nw * bytes(kc) > (size_t)227 * 1024) nw /= 2;
  const size_t sm = nw * bytes(kc);
  allow_smem(kernel, sm);
  kernel<<<(m.N + nw - 1) / nw, nw * kWarp, sm, s>>>(m, a, kc);
}

template <typename R, int VER>
void launch_lo(const DMesh& m, const StepPtrs<R>& a, int nw, int want, cudaStream_t s) {
  launch_nodes(k_fct_lo<R, VER>, lo_blocks(VER), m, a, nw, want,
               [&](int kc) { return warp_smem<R>(lo_slices(VER, kc, a.TA != a.T), m.LW, 0); }, s);
}

template <typename R>
void launch_ratio(const DMesh& m, const StepPtrs<R>& a, int nw, int want, cudaStream_t s) {
  launch_nodes(k_fct_ratio<R>, kRatioBlocks, m, a, nw, want,
               [&](int kc) { return warp_smem<R>(ratio_slices(kc), m.LW, kClBytes); }, s);
}

template <typename R>
void launch_update(const DMesh& m, const StepPtrs<R>& a, int nw, int want, cudaStream_t s) {
  launch_nodes(k_fct_update<R>, kUpdateBlocks, m, a, nw, want,
               [&](int kc) { return warp_smem<R>(upd_slices(kc), m.LW, 0); }, s);
}

template <typename R, int VER>
void launch_nofct(const DMesh& m, const StepPtrs<R>& a, int nw, int want, cudaStream_t s) {
  launch_nodes(k_nofct_update<R, VER>, kNofctBlocks, m, a, nw, want,
               [&](int kc) { return warp_smem<R>(nofct_slices(VER, kc), m.LW, 0); }, s);
}

template <typename R>
void launch_lo_ver(const DMesh& m, const StepPtrs<R>& a, int ver, int nw, int want, cudaStream_t s) {
  switch (ver) {
    case FGB_VER_QR4C: launch_lo<R, 1>(m, a, nw, want, s); break;
    case FGB_VER_CDIFF: launch_lo<R, 2>(m, a, nw, want, s); break;
    case FGB_VER_PPM: launch_lo<R, 3>(m, a, nw, want, s); break;
    default: launch_lo<R, 0>(m, a, nw, want, s); break;
  }
}

template <typename R>
void launch_nofct_ver(const DMesh& m, const StepPtrs<R>& a, int ver, int nw, int want, cudaStream_t s) {
  switch (ver) {
    case FGB_VER_QR4C: launch_nofct<R, 1>(m, a, nw, want, s); break;
    case FGB_VER_CDIFF: launch_nofct<R, 2>(m, a, nw, want, s); break;
    case FGB_VER_PPM: launch_nofct<R, 3>(m, a, nw, want, s); break;
    default: launch_nofct<R, 0>(m, a, nw, want, s); break;
  }
}

template <typename R>
int launch_stages(const DMesh& m, const fgb_step_desc& d, int mask, cudaStream_t s, int* nlaunch,
                  std::string* err) {
  const int K = d.ntracers;
  if (K < 1 || K > 65535) { *err = "ntracers must be in 1..65535"; return -1; }
  if (d.tracer_vec > 1) { *err = "tracer groups (tracer_vec > 1) are a layout of the FP32 form"; return -1; }
  if (d.hor < 0 || d.hor > 2 || d.ver < 0 || d.ver > 3 || d.lim < 0 || d.lim > 1) {
    *err = "unknown advection scheme";
    return -1;
  }
  if (!d.T || !d.vel || !d.w || !d.we || !d.workspace) { *err = "null device pointer"; return -1; }
  if (d.ab_order < 0 || d.ab_order > 2) { *err = "ab_order must be 0, 1 or 2"; return -1; }
  const WorkspaceLayout wl = workspace_layout<R>(m, K);
  if (d.workspace_bytes < wl.total) { *err = "workspace too small"; return -1; }
  if ((d.ver == FGB_VER_QR4C || d.ver == FGB_VER_PPM) && m.min_layers < 2) {
    *err = "QR4C/PPM need at least two layers in every column";
    return -1;
  }
  const bool fct = d.lim == FGB_LIM_FCT;
  const bool wsplit = fct && d.wi;
  if (wsplit) {
    if (const char* why = vert_impl_check(m)) { *err = why; return -1; }
  }
  char* ws = static_cast<char*>(d.workspace);
  StepPtrs<R> a;
  a.T = static_cast<R*>(d.T);
  a.TA = d.TA ? static_cast<const R*>(d.TA) : a.T;
  a.TAout = static_cast<R*>(d.TAout);
  a.vel = static_cast<const R*>(d.vel);
  a.w = static_cast<const R*>(d.w);
  a.we = static_cast<const R*>(d.we);
  a.wi = wsplit ? static_cast<const R*>(d.wi) : nullptr;
  a.vf = reinterpret_cast<R*>(ws + wl.off[0]);
  a.adfh = reinterpret_cast<R*>(ws + wl.off[2]);
  a.lo = reinterpret_cast<R*>(ws + wl.off[3]);
  a.adfv = reinterpret_cast<R*>(ws + wl.off[4]);
  a.rpm = reinterpret_cast<R*>(ws + wl.off[5]);
  a.del = static_cast<R*>(d.del);
  a.sT = d.strideT;
  a.sTA = d.TA ? d.strideTA : d.strideT;
  a.sE = (long long)m.E * m.LZ;
  a.sN = (long long)m.N * m.LZ;
  a.sW = (long long)m.N * m.LW;
  a.dt = (R)d.dt;
  a.ph = (R)d.ph;
  a.pv = (R)d.pv;
  a.K = K;
  a.ab2 = d.ab_order == 2;
  a.ab_old = (R)(-(0.5 + d.ab_eps));
  a.ab_new = (R)(1.5 + d.ab_eps);
  auto pick_w = [](int want, int a, int b, int c, int def) {
    return (want == a || want == b || want == c) ? want : def;
  };
  const int nw_lo = pick_w(d.cfg[1], 1, 2, 4, kNodeWarps);
  const int nw_ratio = pick_w(d.cfg[2], 1, 2, 4, kNodeWarps);
  const int nw_upd = pick_w(d.cfg[3], 1, 2, 4, kNodeWarps);
  int launches = 0;
  const bool hflux = mask & FGB_STAGE_HFLUX, vflux = mask & FGB_STAGE_VFLUX;
  if (vflux && !hflux) {
    k_vflux<R><<<(m.E + kEdgeTile - 1) / kEdgeTile, kEdgeThreads, 0, s>>>(m, a.vel, a.vf);
    ++launches;
  }
  if (hflux) {
    // The element gradients of MUSCL and MFCT use the space of the LO, vertical
    // flux and limiting-factor arrays (consecutive in the workspace), when this
    // call writes those afterwards or no stage reads them, and they fit (two
    // elements per node at most, as in any triangulation of the plane or torus).
    // They hold wet layers only: level tables with windows below a triangle (a
    // restart record may have some) take each edge's gradients from its values.
    const long long room = wl.total - wl.off[3], need = (long long)K * m.M * m.LZ * 2 * (long long)sizeof(R);
    const int later = FGB_STAGE_LO | FGB_STAGE_RATIO;
    double2* grad = nullptr;
    if (d.hor != FGB_HOR_UPW1 && m.windows_wet && need <= room && (!fct || (mask & later) == later)) {
      grad = reinterpret_cast<double2*>(ws + wl.off[3]);
      k_elem_grad<R><<<(m.M + kElemTile - 1) / kElemTile, kEdgeThreads, 0, s>>>(m, a, grad);
      ++launches;
    }
    if (d.hor == FGB_HOR_UPW1) launch_hflux<R, 0>(m, a, fct, vflux, grad, s);
    else if (d.hor == FGB_HOR_MUSCL) launch_hflux<R, 1>(m, a, fct, vflux, grad, s);
    else launch_hflux<R, 2>(m, a, fct, vflux, grad, s);
    ++launches;
  }
  if (fct) {
    if (mask & FGB_STAGE_LO) {
      launch_lo_ver<R>(m, a, d.ver, nw_lo, d.cfg[4], s);
      ++launches;
      if (wsplit) {
        launch_vert_impl<R>(m, a.lo, a.wi, K, a.sN, a.dt, s);
        ++launches;
      }
    }
    if (mask & FGB_STAGE_RATIO) {
      launch_ratio<R>(m, a, nw_ratio, d.cfg[5], s);
      ++launches;
    }
    if (mask & FGB_STAGE_UPDATE) {
      launch_update<R>(m, a, nw_upd, d.cfg[6], s);
      ++launches;
    }
  } else if (mask & FGB_STAGE_UPDATE) {
    launch_nofct_ver<R>(m, a, d.ver, nw_upd, d.cfg[6], s);
    ++launches;
  }
  *nlaunch = launches;
  cudaError_t ce = cudaGetLastError();
  if (ce != cudaSuccess) {
    *err = std::string("kernel launch failed: ") + cudaGetErrorString(ce);
    return -1;
  }
  return 0;
}

}  // inline namespace
}  // namespace fgb
