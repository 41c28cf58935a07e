// FP32 form of the step: argument checks and dispatch to the kernels of the
// tracer-group width (fgb_fast.cuh).
#include <algorithm>
#include <cstdint>

#include "fgb_internal.hpp"

namespace fgb {
namespace fast {
int launch_fast_kv1(const DMesh& m, const FastPtrs& a, const LaunchArgs& L, cudaStream_t s);
int launch_fast_kv2(const DMesh& m, const FastPtrs& a, const LaunchArgs& L, cudaStream_t s);
int launch_fast_kv4(const DMesh& m, const FastPtrs& a, const LaunchArgs& L, cudaStream_t s);
}  // namespace fast

WorkspaceLayout workspace_layout_f32(const DMesh& m, int K) { return workspace_layout<float>(m, K); }

// UPW1 edge fluxes: whether the per-edge kernel is the faster one. It takes two
// layers per lane, 64 at a time; groups of two and four tracers fill its loads
// on larger meshes. Its time over the tiled kernel's, 24^2 to 724^2 columns of
// 20 to 64 layers: with a T_AB of its own (two rows to stage per node), four
// tracers 3.1 .. 1.0 up to 300,000 node-layers and 0.66 to 0.97 from 590,000 on,
// eight 1.1 at 590,000 to 770,000, 0.66 to 1.06 from 1.0 million on, two 1.2 at
// 590,000, 0.76 to 0.95 from 1.0 million on (20 to 32 and 75 layers, which leave
// more than a quarter of its lanes idle, 0.96 to 1.4), six 1.1 to 1.3 at 1.0 to
// 1.3 million, 0.73 to 1.0 above 2 million; no limiter, T_AB shared, four and eight
// tracers 1.0 to 1.2 up to 2 million, 0.80 to 1.09 above; with the limiter (and
// for six tracers without) 0.88 to 0.96 at 16.8 million and 64 layers, 1.0 to 1.4
// with fewer layers or columns; two tracers 0.97 to 2.8 with T_AB shared, one
// 1.04 to 3.4 everywhere.
bool upw1_per_edge(const DMesh& m, int KV, int groups, bool fct, bool own_ta) {
  const long long cells = (long long)m.N * m.LZ;
  if (KV == 1) return false;
  const int passes = (m.LZ + 63) / 64 * 64;  // layers its lanes could hold
  if (fct && own_ta) return cells > (1LL << 19) * (4 / KV) * std::min(groups, 2) && (KV == 4 || 4 * m.LZ >= 3 * passes);
  if (!fct && KV == 4) return cells > 1LL << 21;
  return (KV == 4 || groups > 1) && cells >= 1LL << 24 && 4 * m.LZ > 3 * passes;
}

int launch_stages_f32(const DMesh& m, const fgb_step_desc& d, int mask, cudaStream_t s, int* nlaunch,
                      std::string* err) {
  using namespace fast;
  *nlaunch = 0;
  const int K = d.ntracers;
  const int KV = d.tracer_vec <= 1 ? 1 : d.tracer_vec;
  if (K < 1 || K > 65535) { *err = "ntracers must be in 1..65535"; return -1; }
  if (KV != 1 && KV != 2 && KV != 4) { *err = "tracer_vec must be 0, 1, 2 or 4"; return -1; }
  if (K % KV) { *err = "tracer_vec must divide ntracers"; return -1; }
  if (d.hor < 0 || d.hor > 2 || d.ver < 0 || d.ver > 3 || d.lim < 0 || d.lim > 1) {
    *err = "unknown advection scheme";
    return -1;
  }
  if (!d.T || !d.vel || !d.w || !d.we || !d.workspace) { *err = "null device pointer"; return -1; }
  if (d.ab_order < 0 || d.ab_order > 2) { *err = "ab_order must be 0, 1 or 2"; return -1; }
  const WorkspaceLayout wl = workspace_layout<float>(m, K);
  if (d.workspace_bytes < wl.total) { *err = "workspace too small"; return -1; }
  if ((d.ver == FGB_VER_QR4C || d.ver == FGB_VER_PPM) && m.min_layers < 2) {
    *err = "QR4C/PPM need at least two layers in every column";
    return -1;
  }
  if (d.hor != FGB_HOR_UPW1 && !m.fast_tri_ok) {
    *err = "FP32 MUSCL/MFCT: an upwind triangle does not hold its edge node";
    return -1;
  }
  // Offsets inside a group are 32-bit (units of KV floats).
  const long long lim = 1LL << 32;
  if ((long long)m.E * m.LZ >= lim || 2LL * m.N * m.LZ >= lim || (long long)m.N * m.LW >= lim ||
      (long long)m.M * m.LZ >= lim) {
    *err = "mesh too large for the FP32 form (edges x padded layers must stay below 2^32)";
    return -1;
  }
  const uintptr_t al = 4u * KV;
  auto misaligned = [&](const void* p) { return p && (reinterpret_cast<uintptr_t>(p) % al) != 0; };
  if (misaligned(d.T) || misaligned(d.TA) || misaligned(d.TAout) || misaligned(d.del) || misaligned(d.Tlo) ||
      reinterpret_cast<uintptr_t>(d.vel) % 8 != 0 || d.strideT % KV != 0 || (d.TA && d.strideTA % KV != 0)) {
    *err = "FP32 tracer arrays must be aligned to their group (4 * tracer_vec bytes, strides multiples of tracer_vec)";
    return -1;
  }
  // the workspace's arrays start at multiples of 256 bytes from its base; the
  // pairs of limiting factors are read and written 32 bytes at a time
  if (reinterpret_cast<uintptr_t>(d.workspace) % 32 != 0) {
    *err = "the FP32 form's workspace must be 32-byte aligned (cudaMalloc gives 256)";
    return -1;
  }
  const bool wsplit = d.lim == FGB_LIM_FCT && d.wi;
  if (wsplit) {
    if (m.min_layers < 2) { *err = "w_split needs at least two layers in every column"; return -1; }
    if (vimpl_block_bytes(m.LZ, KV) > 227 * 1024) { *err = "w_split: too many layers for one block"; return -1; }
    if (reinterpret_cast<uintptr_t>(d.wi) % 4 != 0) { *err = "wi must be 4-byte aligned"; return -1; }
  }
  char* ws = static_cast<char*>(d.workspace);
  FastPtrs a;
  a.T = static_cast<float*>(d.T);
  a.TA = d.TA ? static_cast<const float*>(d.TA) : a.T;
  a.TAout = static_cast<float*>(d.TAout);
  a.vel = static_cast<const float*>(d.vel);
  a.w = static_cast<const float*>(d.w);
  a.we = static_cast<const float*>(d.we);
  a.wi = wsplit ? static_cast<const float*>(d.wi) : nullptr;
  a.vf = reinterpret_cast<float*>(ws + wl.off[0]);
  a.adfh = reinterpret_cast<float*>(ws + wl.off[2]);
  a.lo = reinterpret_cast<float*>(ws + wl.off[3]);
  a.adfv = reinterpret_cast<float*>(ws + wl.off[4]);
  a.rpm = reinterpret_cast<float*>(ws + wl.off[5]);
  a.del = static_cast<float*>(d.del);
  a.gT = d.strideT;
  a.gTA = d.TA ? d.strideTA : d.strideT;
  a.gE = (long long)m.E * m.LZ * KV;
  a.gN = (long long)m.N * m.LZ * KV;
  a.gW = (long long)m.N * m.LW * KV;
  a.G = K / KV;
  a.dt = (float)d.dt;
  a.ph = (float)d.ph;
  a.pv = (float)d.pv;
  a.wsplit_fused = 0;  // set per launch of the LO kernel
  a.comp = ~d.fp32_plain_sums & 7;
  a.Tlo = d.del ? nullptr : static_cast<float*>(d.Tlo);
  a.ab2 = d.ab_order == 2;
  a.ab_old = (float)(-(0.5 + d.ab_eps));
  a.ab_new = (float)(1.5 + d.ab_eps);
  auto pick = [](int want, int x, int y, int z, int def) { return (want == x || want == y || want == z) ? want : def; };
  LaunchArgs L;
  L.mask = mask;
  L.edge_warps = pick(d.cfg[0], 2, 4, 8, 8);
  L.nw_lo = pick(d.cfg[1], 1, 2, 4, 4);
  L.nw_ratio = pick(d.cfg[2], 1, 2, 4, 4);
  L.nw_upd = pick(d.cfg[3], 1, 2, 4, 4);
  auto ns = [](int want, int def) { return (want == 1 || want == 2) ? want : def; };
  L.ns_h = ns(d.cfg[7], 2);
  // LO: 3 (the default where it applies) the whole-column kernel for columns of
  // at most 64 layers; 1 or 2 layers per lane per pass. Under w_split the
  // whole-column kernel leaves the implicit step to a second kernel
  // (kf_vert_pcr), the two-layer one solves it in the same pass. What the whole
  // column saves is the scheme's work, most for PPM, and its tables, which
  // several groups share; the second kernel costs a pass over the LO field,
  // groups of four tracers most. Two-layer kernel's time over the two kernels',
  // 48^2 to 400^2 columns of 20 to 64 layers: PPM 1.04 to 1.4; several groups of
  // one or two tracers 1.0 to 1.3; QR4C one tracer 1.0 to 1.1, eight 1.0 to 1.2,
  // two 0.87 to 1.07, four 0.95 to 1.2 (0.95 to 0.99 at 220^2); UPW1 with one
  // tracer and plain sums 1.0 to 1.13, otherwise UPW1 and CDIFF 0.85 to 1.07 for
  // one and two tracers, 0.8 to 1.05 for four and eight. Below
  // a wave of columns the second launch costs more than either saves.
  const int groups = K / KV;
  const bool whole_pays = d.ver == FGB_VER_PPM || (d.ver == FGB_VER_QR4C && (KV == 1 || groups > 1)) ||
                          (KV <= 2 && groups > 1) || (d.ver == FGB_VER_UPW1 && KV == 1 && !(a.comp & 1));
  const bool whole = m.LZ <= 64 && (!wsplit || (m.N > kWaveColumns && whole_pays) || d.cfg[4] == 3);
  L.ns_lo = (d.cfg[4] == 1 || d.cfg[4] == 2) ? d.cfg[4] : (whole ? 3 : 2);
  // ratio: 1 or 2 layers per lane with shared-memory staging, or 3 (the default)
  // the whole column per warp without shared memory
  L.ns_ratio = (d.cfg[5] >= 1 && d.cfg[5] <= 4) ? d.cfg[5] : 0;
  L.ns_upd = ns(d.cfg[6], 1);
  L.vimpl_thomas = d.cfg[8] == 1;
  // Edge fluxes: the tiled kernel unless cfg[0] or cfg[7] asks for a shape of
  // the per-edge one. A block of the tiled kernel holds at most 32 edges, so a
  // small mesh still fills the GPU, and layers outside their triangles' window
  // go to a kernel of their own. Edge stage, per-edge kernel against tiled:
  // 48x40x30, 3 tracers, 103 against 20 us; closed 513^2x64, 2 tracers, 930 /
  // 370 us; pi refined to 188,661 nodes, 47 layers, 4 tracers, 670 / 305 us;
  // 250x230x47, 2 tracers, 149 / 85 us; 256^2x64, 4 tracers, 162 / 121 us; no
  // size was slower with MUSCL or MFCT. UPW1 reads an edge's two nodes only, so
  // staging rows gains less: see upw1_per_edge.
  // The tiled kernel stages rows with 16-byte asynchronous copies; fields on
  // other addresses take the per-edge kernel.
  auto al16 = [](const void* p) { return p == nullptr || reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  const bool tile = d.cfg[9] == 1 || (d.cfg[0] == 0 && d.cfg[7] == 0 &&
                                      !(d.hor == FGB_HOR_UPW1 && upw1_per_edge(m, KV, groups, d.lim == FGB_LIM_FCT,
                                                                               a.TA != a.T)));
  L.hflux_tile = tile && al16(d.T) && al16(d.TA) && al16(d.workspace) && (d.strideT * 4) % 16 == 0 &&
                 (!d.TA || (d.strideTA * 4) % 16 == 0);
  L.hor = d.hor;
  L.ver = d.ver;
  L.fct = d.lim == FGB_LIM_FCT;
  int n = 0;
  if (KV == 4) n = launch_fast_kv4(m, a, L, s);
  else if (KV == 2) n = launch_fast_kv2(m, a, L, s);
  else n = launch_fast_kv1(m, a, L, s);
  *nlaunch = n;
  cudaError_t ce = cudaGetLastError();
  if (ce != cudaSuccess) {
    *err = std::string("kernel launch failed: ") + cudaGetErrorString(ce);
    return -1;
  }
  return 0;
}
}  // namespace fgb
