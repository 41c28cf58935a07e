// Device kernels of the FP64 forms of the FESOM2 tracer-advection step
// (do_oce_adv_tra, lib/oce_adv_tra_driver.F90:23-294) for GB300 (sm_103a).
//
// Layout: level index fastest, columns padded to LZ layers / LW interfaces.
// Node kernels run one warp per column and deal its (tracer, layer) pairs to
// the lanes; edge kernels deal the (edge, layer) pairs of a tile of edges to a
// block. The reference's edge scatters (atomics / OpenMP locks) are replaced by
// gathers over each node's incident edges in ascending edge order, which
// reproduces the reference's per-node summation order exactly.
//
// R is the storage and arithmetic type. Every expression keeps the
// reference's evaluation order; the FP64 translation unit is compiled without
// fused multiply-add so the device result equals the CPU restatement bit for bit.
#pragma once
#include <cstdint>

#include "fgb_bits.cuh"
#include "fgb_device.hpp"
#include "fgb_intdiv.cuh"

#ifndef FGB_FAST64
#define FGB_FAST64 0
#endif

namespace fgb {
// Two compilations of these kernels live side by side, kept apart by their
// inline namespace: the bit-exact FP64 form (no fused multiply-add, every
// division as the reference writes it) and, with FGB_FAST64, the fast FP64
// form (fused multiply-add; divisions by constants become products with the
// reciprocal constant, and dt / areasvol and 1 / hnode_new are formed once
// per layer and shared by the tracers and edges of a node).
#if FGB_FAST64
inline namespace fast64 {
#else
inline namespace exact64 {
#endif

constexpr int kWarp = 32;

template <typename R>
struct GeoSel;
template <>
struct GeoSel<double> {
  __host__ __device__ static const GeoPtrs<double>& get(const DMesh& m) { return m.g64; }
};
template <>
struct GeoSel<float> {
  __host__ __device__ static const GeoPtrs<float>& get(const DMesh& m) { return m.g32; }
};

// a < b ? a : b and a > b ? a : b, compared on the integer pipe.
template <typename R>
__device__ __forceinline__ R rmin(R a, R b) { return bits64::lesser(a, b); }
template <typename R>
__device__ __forceinline__ R rmax(R a, R b) { return bits64::greater(a, b); }
template <typename R>
__device__ __forceinline__ R rabs(R a) { return bits64::magnitude(a); }

// Division: correctly rounded (bit parity with the CPU restatement), on the
// integer pipe.
template <typename R>
__device__ __forceinline__ R fdiv(R a, R b) { return intdiv::divide(a, b); }
// a * b on the integer pipe in the exact form, where a kernel keeps the FP64
// pipe busy and the integer pipe idle (the update kernel, with more integer
// work per FP64 instruction, slowed down: 1.85 against 1.61 ms); the fast form
// fuses it with an addition.
__device__ __forceinline__ double imul(double a, double b) {
  if constexpr (FGB_FAST64) return a * b;
  else return intdiv::multiply(a, b);
}
// A divisor shared by several quotients: prepared once in the exact form (the
// fast form multiplies with reciprocals instead).
struct LayerDivisor {
  intdiv::Divisor d;
  __device__ __forceinline__ explicit LayerDivisor(double b) {
    if constexpr (!FGB_FAST64) d = intdiv::prepare(b);
  }
};
// a / 3 and a / 6: the reference's division, or (fast form) the product with
// the reciprocal constant.
__device__ __forceinline__ double third(double a) {
  if constexpr (FGB_FAST64) return a * (1.0 / 3.0);
  else return intdiv::divide(a, intdiv::three());
}
__device__ __forceinline__ double sixth(double a) {
  if constexpr (FGB_FAST64) return a * (1.0 / 6.0);
  else return intdiv::divide(a, intdiv::six());
}
// (x dt) / areasvol: the reference's order with the layer's prepared
// areasvol, or (fast form) x times the layer's dt / areasvol, formed once.
template <typename R>
__device__ __forceinline__ R dt_per_vol(R x, R dt, const LayerDivisor& av, R rdt_av) {
  if constexpr (FGB_FAST64) return x * rdt_av;
  else return intdiv::divide(x * dt, av.d);
}
template <typename R>
__device__ __forceinline__ R rdt_vol(R dt, R av) {
  if constexpr (FGB_FAST64) return fdiv(dt, av);
  else return R(0);  // unused by the exact form
}

// ---------------------------------------------------------------------------
// Edges. A block of the edge kernels takes kEdgeTile edges of the visit order
// (the three edge families interleaved by node, for cache locality); their
// tables are staged once, then each thread takes one (edge, layer) pair at a
// time, so that warps are full whatever the number of layers: these kernels
// are bound by the FP64 pipe, which a warp instruction with idle lanes
// occupies as long as a full one (one edge per warp, two layers per lane,
// left a quarter of the lanes idle at 48 layers).
// ---------------------------------------------------------------------------
constexpr int kEdgeTile = 16;
constexpr int kEdgeThreads = 256;

struct EdgeTab {
  int e, n1, n2, el1, el2, nl1, nl2;  // ulevels = 1: element 1 contributes at layers 1..nl1, element 2 at 1..nl2
  int up, dn, gm0, gm1, nb1, nb2;
  double dX1, dY1, dX2, dY2, ex, ey;
};

template <int HOR>
__device__ __forceinline__ EdgeTab load_edge(const DMesh& m, int w) {
  EdgeTab q{};
  const int e = m.edge_order ? m.edge_order[w] : w;
  q.e = e;
  q.n1 = m.edge_nodes[2 * e];
  q.n2 = m.edge_nodes[2 * e + 1];
  q.el1 = m.edge_tri[2 * e];
  q.el2 = m.edge_tri[2 * e + 1];
  q.nl1 = m.edge_lev[4 * e + 1];
  q.nl2 = q.el2 >= 0 ? m.edge_lev[4 * e + 3] : 0;
  const double* cr = m.g64.edge_cross + 4 * (size_t)e;
  q.dX1 = cr[0];
  q.dY1 = cr[1];
  q.dX2 = cr[2];
  q.dY2 = cr[3];
  q.gm0 = -1;
  if (HOR != 0) {
    q.gm0 = m.edge_gm[2 * e];
    q.gm1 = m.edge_gm[2 * e + 1];
    q.up = m.edge_updn[2 * e];
    q.dn = m.edge_updn[2 * e + 1];
    q.ex = m.g64.edge_dxa[2 * e];
    q.ey = m.g64.edge_dxa[2 * e + 1];
    q.nb1 = m.nbl[q.n1];
    q.nb2 = m.nbl[q.n2];
  }
  return q;
}

// Volume flux through the edge's segments at layer k (vflux of
// lib/oce_adv_tra_hor.F90:174,194,215-216).
__device__ __forceinline__ double edge_vflux(const DMesh& m, const EdgeTab& q, const double* __restrict__ vel, int k) {
  const bool s1 = k < q.nl1, s2 = k < q.nl2;
  double v1 = 0.0, v2 = 0.0;
  if (s1) {
    const size_t i = (size_t)q.el1 * m.LZ + k;
    const double u = vel[2 * i], w = vel[2 * i + 1];
    v1 = imul(-(w * q.dX1) + imul(u, q.dY1), m.g64.helem[i]);
  }
  if (s2) {
    const size_t i = (size_t)q.el2 * m.LZ + k;
    const double u = vel[2 * i], w = vel[2 * i + 1];
    v2 = imul(w * q.dX2 - imul(u, q.dY2), m.g64.helem[i]);
  }
  return s1 && s2 ? v1 + v2 : (s1 ? v1 : v2);
}

// ---------------------------------------------------------------------------
// Volume flux through each edge segment (shared by all tracers of a step),
// for calls of single stages; a whole step forms it in the edge-flux kernel.
// ---------------------------------------------------------------------------
template <typename R>
__global__ void __launch_bounds__(kEdgeThreads) k_vflux(DMesh m, const R* __restrict__ vel, R* __restrict__ vf) {
  __shared__ EdgeTab tab[kEdgeTile];
  const int w0 = blockIdx.x * kEdgeTile, ne = min(kEdgeTile, m.E - w0);
  if ((int)threadIdx.x < ne) tab[threadIdx.x] = load_edge<0>(m, w0 + threadIdx.x);
  __syncthreads();
  for (unsigned i = threadIdx.x; i < (unsigned)(ne * m.LZ); i += kEdgeThreads) {
    const unsigned j = i / (unsigned)m.LZ, k = i - j * (unsigned)m.LZ;
    vf[(size_t)tab[j].e * m.LZ + k] = edge_vflux(m, tab[j], vel, (int)k);
  }
}

// Elemental gradient of T at layer k (tr_xy, coefficients gradient_sca of
// lib/oce_mesh.F90:2512-2534).
template <typename R>
__device__ __forceinline__ void elem_grad(const DMesh& m, const GeoPtrs<R>& g, const R* __restrict__ T, int el,
                                          size_t k, R& gx, R& gy) {
  const size_t LZ = m.LZ;
  const int a = m.elem_nodes[3 * el], b = m.elem_nodes[3 * el + 1], c = m.elem_nodes[3 * el + 2];
  const R ta = T[a * LZ + k], tb = T[b * LZ + k], tc = T[c * LZ + k];
  const R* gs = g.grad_sca + 6 * (size_t)el;
  gx = gs[0] * ta + gs[1] * tb + gs[2] * tc;
  gy = gs[3] * ta + gs[4] * tb + gs[5] * tc;
}

// The elemental gradients of every wet layer and tracer, (K, M, LZ) pairs: each
// triangle is the up- or downwind one of three edges on average, which would
// form its gradient again (ten FP64 instructions of each edge's 25 per side).
constexpr int kElemTile = 16;
template <typename R>
__global__ void __launch_bounds__(kEdgeThreads) k_elem_grad(DMesh m, StepPtrs<R> a, double2* __restrict__ out) {
  const int w0 = blockIdx.x * kElemTile, ne = min(kElemTile, m.M - w0);
  const size_t LZ = m.LZ;
  for (unsigned i = threadIdx.x; i < (unsigned)(ne * m.LZ); i += kEdgeThreads) {
    const unsigned j = i / (unsigned)m.LZ, k = i - j * (unsigned)m.LZ;
    const int el = w0 + (int)j;
    if ((int)k >= m.elem_nlev[el] - 1) continue;
    const int na = m.elem_nodes[3 * el], nb = m.elem_nodes[3 * el + 1], nc = m.elem_nodes[3 * el + 2];
    const R* gs = m.g64.grad_sca + 6 * (size_t)el;
    const R x0 = gs[0], x1 = gs[1], x2 = gs[2], y0 = gs[3], y1 = gs[4], y2 = gs[5];
    for (int t = 0; t < a.K; ++t) {
      const R* __restrict__ T = a.TA + t * a.sTA + k;
      const R ta = T[na * LZ], tb = T[nb * LZ], tc = T[nc * LZ];
      out[((size_t)t * m.M + el) * LZ + k] = make_double2(x0 * ta + imul(x1, tb) + imul(x2, tc), y0 * ta + imul(y1, tb) + imul(y2, tc));
    }
  }
}

// Element gradients of one tracer: from k_elem_grad's array, or formed here.
template <bool GRAD>
__device__ __forceinline__ void grad_at(const DMesh& m, const double* __restrict__ T, const double2* __restrict__ G,
                                        int el, int k, double& gx, double& gy) {
  if constexpr (GRAD) {
    const double2 v = G[(size_t)el * m.LZ + k];
    gx = v.x;
    gy = v.y;
  } else {
    elem_grad(m, m.g64, T, el, (size_t)k, gx, gy);
  }
}

// Area-weighted mean of the element gradients around a node at layer z
// (lib/oce_muscl_adv.F90:393-410).
template <bool GRAD>
__device__ __forceinline__ void node_mean_grad(const DMesh& m, const double* __restrict__ T,
                                               const double2* __restrict__ G, int n, int k, double& gx, double& gy) {
  double tvol = 0.0, tx = 0.0, ty = 0.0;
  const int z = k + 1;
  for (int j = m.nie_ptr[n]; j < m.nie_ptr[n + 1]; ++j) {
    const int el = m.nie_idx[j];
    if (m.elem_nlev[el] - 1 < z) continue;
    double ex, ey;
    grad_at<GRAD>(m, T, G, el, k, ex, ey);
    const double ar = m.g64.elem_area[el];
    tvol = tvol + ar;
    tx = tx + ex * ar;
    ty = ty + ey * ar;
  }
  const intdiv::Divisor d = intdiv::prepare(tvol);
  gx = intdiv::divide(tx, d);
  gy = intdiv::divide(ty, d);
}

// ---------------------------------------------------------------------------
// Horizontal edge fluxes of all K tracers. FCT: the antidiffusive flux
// HO(T_AB) - LO(T) (adv_tra_hor_* with o_init_zero=.false. after
// adv_tra_hor_upw1, lib/oce_adv_tra_driver.F90:95,244-255); otherwise the HO
// flux. HOR: 0 UPW1 (lib/oce_adv_tra_hor.F90:218-220), 1 MUSCL (:454-497, with
// the nboundary_lay mask c_lo), 2 MFCT (:748-790). VF: the volume fluxes are
// formed and stored here (else read). GRAD: element gradients from
// k_elem_grad's array. Results are stored at the edge's own index.
// Bound by the FP64 pipe: 15 FP64 instructions per layer and tracer (MUSCL,
// ph = 1; 87 in the form it replaced) and two divisions by six on the integer
// pipe. 512^2 x 48, 2 tracers: volume fluxes, gradients and edge fluxes 4.4 ms
// together against 10.9 (2.9 with the products that have moved since).
// ---------------------------------------------------------------------------
// The flux for any ph and for very large, infinite and NaN values.
static __device__ __noinline__ double hor_flux_any(double v, double Tm1, double Tm2, double ph) {
  return intdiv::behind_branch<double>([&] {
    const double cHO = (v + fabs(v)) * Tm1 + (v - fabs(v)) * Tm2;
    return -((0.5 * (1.0 - ph)) * cHO) - ((v * ph) * 0.5) * (Tm1 + Tm2);
  });
}

// The flux of edge q at layer k, all tracers. MEAN: outside the triangles' window (or without
// triangles), the mean gradients around both nodes.
template <int HOR, bool FCT, bool VF, bool GRAD, bool MEAN>
__device__ __forceinline__ void hor_flux(const DMesh& m, const StepPtrs<double>& a, const double2* __restrict__ grad,
                                         const EdgeTab& q, int k) {
  const size_t LZ = m.LZ, ek = (size_t)q.e * LZ + k;
  const bool ta_sep = a.TA != a.T, ph1 = a.ph == 1.0;
  double v;
  if (VF) {
    v = edge_vflux(m, q, a.vel, k);
    a.vf[ek] = v;
  } else {
    v = a.vf[ek];
  }
  const double B = bits64::half(ph1 ? v : intdiv::hw_mul(v, a.ph));
  const bool c1 = HOR == 2 || q.nb1 > k, c2 = HOR == 2 || q.nb2 > k;
  const size_t i1 = q.n1 * LZ + k, i2 = q.n2 * LZ + k;
  for (int t = 0; t < a.K; ++t) {
    const double* __restrict__ T = a.T + t * a.sT;
    const double* __restrict__ TA = ta_sep ? a.TA + t * a.sTA : T;
    const double s1 = TA[i1], s2 = TA[i2];
    double lo = 0.0;  // minus the low-order flux
    if (FCT) lo = ta_sep ? bits64::upwind(v, T[i1], T[i2]) : bits64::upwind(v, s1, s2);
    double h;
    if (HOR == 0) {
      h = -(FCT && !ta_sep ? lo : bits64::upwind(v, s1, s2));
    } else {
      const double2* __restrict__ G = GRAD ? grad + (size_t)t * m.M * LZ : nullptr;
      double g1, g2, g3, g4;
      if (MEAN) {
        node_mean_grad<GRAD>(m, TA, G, q.n1, k, g1, g3);
        node_mean_grad<GRAD>(m, TA, G, q.n2, k, g2, g4);
      } else {
        grad_at<GRAD>(m, TA, G, q.up, k, g1, g3);
        grad_at<GRAD>(m, TA, G, q.dn, k, g2, g4);
      }
      const double d2 = bits64::twice(s2 - s1);
      double r1 = sixth(d2 + imul(q.ex, g1) + imul(q.ey, g3)), r2 = sixth(d2 + imul(q.ex, g2) + imul(q.ey, g4));
      if (HOR == 1 && !(c1 && c2)) {
        if (bits64::finite(r1, r2)) {
          r1 = c1 ? r1 : 0.0;
          r2 = c2 ? r2 : 0.0;
        } else {
          r1 = intdiv::hw_mul(r1, c1 ? 1.0 : 0.0);
          r2 = intdiv::hw_mul(r2, c2 ? 1.0 : 0.0);
        }
      }
      const double Tm1 = s1 + r1, Tm2 = s2 - r2;
      // ph = 1: the upwind part is an exact zero (unless its products overflow)
      if (ph1 && bits64::moderate(Tm1, Tm2) && bits64::moderate(v)) h = -(B * (Tm1 + Tm2));
      else h = hor_flux_any(v, Tm1, Tm2, a.ph);
    }
    a.adfh[t * a.sE + ek] = FCT ? h + lo : h;
  }
}

// A tile's layers in three lists, each dealt to the threads by itself: those in the triangles'
// window, those with mean gradients (some eight times the work: mixed into the first list, a
// single one held its whole warp), and those below the edge, which are zero.
template <typename R, int HOR, bool FCT, bool VF, bool GRAD>
__global__ void __launch_bounds__(kEdgeThreads, 4) k_hflux(DMesh m, StepPtrs<R> a, const double2* __restrict__ grad) {
  __shared__ EdgeTab tab[kEdgeTile];
  __shared__ int win[kEdgeTile][2];         // the window's layers [first, end) per edge (0-based)
  __shared__ int ptr[3][kEdgeTile + 1];     // starts of the edges' parts of the three lists
  const int w0 = blockIdx.x * kEdgeTile, ne = min(kEdgeTile, m.E - w0), tid = threadIdx.x;
  if (tid < kWarp) {
    int cnt[3] = {0, 0, 0};
    if (tid < ne) {
      const EdgeTab q = load_edge<HOR>(m, w0 + tid);
      tab[tid] = q;
      const int hi = max(q.nl1, q.nl2);
      const TriangleWindow w = HOR != 0 ? triangle_window(q.gm0, q.gm1, hi) : TriangleWindow{0, hi};
      win[tid][0] = w.first;
      win[tid][1] = w.end;
      cnt[0] = w.end - w.first;
      cnt[1] = hi - cnt[0];
      cnt[2] = m.LZ - hi;
    }
#pragma unroll
    for (int l = 0; l < 3; ++l) {
#pragma unroll
      for (int d = 1; d < kEdgeTile; d *= 2) {
        const int x = __shfl_up_sync(0xffffffffu, cnt[l], d);
        if (tid >= d) cnt[l] += x;
      }
      if (tid < kEdgeTile) ptr[l][tid + 1] = cnt[l];
      if (tid == 0) ptr[l][0] = 0;
    }
  }
  __syncthreads();
  auto edge_of = [&](int l, int i) {  // the edge of a list's item i
    int j = 0;
#pragma unroll
    for (int d = kEdgeTile / 2; d > 0; d /= 2)
      if (i >= ptr[l][j + d]) j += d;
    return j;
  };
  for (int i = tid; i < ptr[0][kEdgeTile]; i += kEdgeThreads) {
    const int j = edge_of(0, i);
    hor_flux<HOR, FCT, VF, GRAD, false>(m, a, grad, tab[j], win[j][0] + i - ptr[0][j]);
  }
  if (HOR != 0)
    for (int i = tid; i < ptr[1][kEdgeTile]; i += kEdgeThreads) {
      const int j = edge_of(1, i);
      int k = i - ptr[1][j];
      if (k >= win[j][0]) k += win[j][1] - win[j][0];
      hor_flux<HOR, FCT, VF, GRAD, true>(m, a, grad, tab[j], k);
    }
  for (int i = tid; i < ptr[2][kEdgeTile]; i += kEdgeThreads) {
    const int j = edge_of(2, i);
    const size_t ek = (size_t)tab[j].e * m.LZ + max(tab[j].nl1, tab[j].nl2) + i - ptr[2][j];
    if (VF) a.vf[ek] = R(0);
    for (int t = 0; t < a.K; ++t) a.adfh[t * a.sE + ek] = R(0);
  }
}

// ---------------------------------------------------------------------------
// Node-column kernels. One warp per node. The node's incident edges (ascending
// edge index, the reference's scatter order) and its FCT cluster are staged
// once in shared memory. The column's (tracer, layer) pairs of a chunk of up to
// kc tracers are dealt to the lanes one at a time, down to the column's bottom:
// warps are full whatever the number of layers (the kernels are bound by the
// FP64 pipe, which a warp instruction with idle lanes occupies as long as a
// full one), a lane holds one layer of one tracer (few registers, more warps),
// and its chain of dependent operations is short. Per (tracer, layer) the
// summation order is the reference's. 512^2 x 48, 2 tracers, side by side with
// two layers per lane and a compile-time tracer chunk: LO 1.95 / 3.34 ms, ratio
// 1.50 / 2.07, update 1.62 / 2.64 (with what came after 1.63, 1.51, 1.55);
// closed 321^2 x 64, fast form: 2.17 / 2.43, 0.68 / 0.76, 0.65 / 1.11 (1.76,
// 0.69, 0.66); 361 columns of 9 layers, no limiter: 10 / 18 us.
// ---------------------------------------------------------------------------
struct Nbr {
  int e, role, other, lo, hi;
};
constexpr int kMaxDeg = 16;  // incident edges staged per node; more are read from global memory
constexpr int kMaxCl = 24;   // cluster nodes staged per node

__device__ __forceinline__ Nbr nbr_global(const DMesh& m, int j) {
  const int code = m.ne_code[j];
  return Nbr{code >> 1, code & 1, m.ne_other[j], m.ne_lo[j], m.ne_hi[j]};
}

struct NbrList {
  const Nbr* s;
  int j0, deg;
  __device__ __forceinline__ Nbr get(const DMesh& m, int j) const {
    return deg <= kMaxDeg ? s[j] : nbr_global(m, j0 + j);
  }
};

__device__ __forceinline__ NbrList stage_nbrs(const DMesh& m, int n, Nbr* s, int lane) {
  NbrList L{s, m.ne_ptr[n], m.ne_ptr[n + 1] - m.ne_ptr[n]};
  if (L.deg <= kMaxDeg)
    for (int j = lane; j < L.deg; j += kWarp) s[j] = nbr_global(m, L.j0 + j);
  return L;
}

// Shared memory of one warp: `slices` columns of LW values, the edge list and
// `extra_bytes` more.
template <typename R>
__host__ __device__ constexpr size_t warp_smem(int slices, int LW, int extra_bytes) {
  return ((size_t)slices * LW * sizeof(R) + kMaxDeg * sizeof(Nbr) + extra_bytes + 15) / 16 * 16;
}
// Columns of the vertical schemes' geometry and of one tracer's work (QR4C
// slopes; PPM slopes and edge values).
__host__ __device__ constexpr int ver_geo_slices(int ver) { return ver == 3 ? 10 : (ver == 1 ? 4 : 0); }
__host__ __device__ constexpr int ver_work_slices(int ver) { return ver == 3 ? 2 : (ver == 1 ? 1 : 0); }
__host__ __device__ constexpr int lo_slices(int ver, int kc, bool ta_sep) {
  return ver_geo_slices(ver) + kc * (2 + (ta_sep ? 1 : 0) + ver_work_slices(ver));
}
__host__ __device__ constexpr int ratio_slices(int kc) { return 2 * kc; }
__host__ __device__ constexpr int upd_slices(int kc) { return kc; }
__host__ __device__ constexpr int nofct_slices(int ver, int kc) {
  return ver_geo_slices(ver) + kc * (2 + ver_work_slices(ver));
}
constexpr int kClBytes = kMaxCl * 2 * (int)sizeof(int);
// Blocks of kNodeWarps columns per SM that the node kernels' registers are held to (reasons at the kernels).
constexpr int kNodeWarps = 4;
__host__ __device__ constexpr int lo_blocks(int ver) { return ver == 1 ? 7 : 6; }
constexpr int kRatioBlocks = 6, kUpdateBlocks = 7, kNofctBlocks = 6;

// The column of one node: interfaces nzmin..nzmax (1-based), layers k0..k0+nlay-1 (0-based).
struct Column {
  int n, nzmin, nzmax, k0;
  unsigned nlay;
  size_t iz, iw;  // first layer / interface of the node in (N,LZ) / (N,LW) arrays
  __device__ __forceinline__ Column(const DMesh& m, int n_)
      : n(n_), nzmin(m.ulev[n_]), nzmax(m.nlev[n_]), k0(nzmin - 1), nlay((unsigned)(nzmax - nzmin)),
        iz((size_t)n_ * m.LZ), iw((size_t)n_ * m.LW) {}
};

// ---------------------------------------------------------------------------
// Vertical high-order fluxes (lib/oce_adv_tra_ver.F90:248-712).
// VER: 0 UPW1, 1 QR4C, 2 CDIFF, 3 PPM.
// ---------------------------------------------------------------------------
// The expressions of very large, infinite and NaN values and of any num_ord, out of line.
static __device__ __noinline__ double qr4c_any(double W, double tm1, double tm2, double num_ord, double A) {
  return intdiv::behind_branch<double>([&] {
    const double tm = (W + fabs(W)) * tm1 + (W - fabs(W)) * tm2;
    return (-((0.5 * (1.0 - num_ord)) * tm) - (num_ord * (0.5 * (tm1 + tm2))) * W) * A;
  });
}
static __device__ __noinline__ double hw_ppm_bottom(double Tu, double Tl, double W) {
  return intdiv::behind_branch<double>([&] {
    const double s = copysign(1.0, W);
    return -(Tu * (s < 0.0 ? s : 0.0)) + Tl * (s > 0.0 ? s : 0.0);
  });
}

// What a vertical scheme needs of a column's geometry, for all its tracers.
// PPM: the quotients of layer thicknesses, which the reference forms per tracer
// and twice per layer (a layer's deltaj at one interface and deltajp1 at the
// next are the same expression of the same operands), by layer (ga, gb, gc)
// and by interface (gh..gl), and x / 2 and 1 - 2/3 x of the upwind layer.
// QR4C: zbar - Z of both layers and the prepared divisor Z(z-1) - Z(z) (fast
// form: its reciprocal).
template <int VER>
struct VerGeo {
  double* s;
  int LW;
  __device__ __forceinline__ double& at(int slice, int k) const { return s[slice * LW + k]; }
  enum { GA, GB, GC, GH, GI, GJ, GK, GL, HX, CX };  // PPM
  enum { A1, A2, DZ, DX };                             // QR4C

  __device__ __forceinline__ void form(const DMesh& m, const Column& c, const double* __restrict__ w, double dt,
                                       int lane) const {
    using bits64::twice;
    const GeoPtrs<double>& g = m.g64;
    if constexpr (VER == 1) {
      const double* Z = g.Z3 + c.iz;
      for (int i = c.nzmin + lane; i <= c.nzmax - 2; i += kWarp) {
        const double zb = g.zbar3[c.iw + i], Z0 = Z[i], Zu = Z[i - 1];
        at(A1, i) = zb - Z0;
        at(A2, i) = zb - Zu;
        const intdiv::Divisor d = intdiv::prepare(Zu - Z0);
        at(DZ, i) = FGB_FAST64 ? intdiv::divide(1.0, d) : d.b;
        at(DX, i) = bits64::from_bits(d.x);
      }
    }
    if constexpr (VER == 3) {
      const double* h = g.hnode_new + c.iz;
      for (int j = c.nzmin + lane; j <= c.nzmax - 3; j += kWarp) {  // layers (0-based) with both neighbours
        const double hm = h[j - 1], h0 = h[j], hp = h[j + 1], sm = hm + h0;
        at(GA, j) = fdiv(h0, sm + hp);
        at(GB, j) = fdiv(twice(hm) + h0, hp + h0);
        at(GC, j) = fdiv(h0 + twice(hp), sm);
      }
      for (int i = c.nzmin + 1 + lane; i <= c.nzmax - 3; i += kWarp) {  // interfaces (0-based) of the four-point formula
        const double hm = h[i - 2], h0 = h[i - 1], hp = h[i], hpp = h[i + 1], su = hm + h0, sl = hpp + hp;
        const intdiv::Divisor ds = intdiv::prepare(h0 + hp), du = intdiv::prepare(twice(h0) + hp),
                              dl = intdiv::prepare(twice(hp) + h0);
        at(GH, i) = intdiv::divide(twice(hp) * h0, ds) * (intdiv::divide(su, du) - intdiv::divide(sl, dl));
        at(GI, i) = intdiv::divide(h0 * su, du);
        at(GJ, i) = intdiv::divide(hp * sl, dl);
        at(GK, i) = intdiv::divide(h0, ds);
        at(GL, i) = fdiv(1.0, su + hp + hpp);
      }
      for (int i = c.nzmin + lane; i <= c.nzmax - 2; i += kWarp) {
        const double W = w[c.iw + i];  // x = min(W dt / h, 1) of the layer below (W > 0) or min(-(W dt / h), 1) above
        const bool up = bits64::sign_clear(W);
        const double q = fdiv(W * dt, g.hnode[c.iz + (up ? i : i - 1)]);
        const double x = rmin(up ? q : -q, 1.0);
        at(HX, i) = bits64::half(x);
        at(CX, i) = 1.0 - (2.0 / 3.0) * x;
      }
    }
  }
};

// Tracer work of a scheme before its fluxes: T, and the scheme's columns S
// (and, for PPM, TV) of kc tracers, LW apart. Ends synchronised.
template <int VER>
__device__ __forceinline__ void ver_prepare(const VerGeo<VER>& g, const Column& c, const double* T, double* S,
                                            double* TV, const double* __restrict__ w, unsigned kc, int lane) {
  const int LW = g.LW;
  if constexpr (VER == 1) {
    // slopes (T(z-1) - T(z)) / (Z(z-1) - Z(z)) by interface: an interface uses its own and both neighbours'
    const unsigned cnt = c.nlay - 1;
    for (unsigned it = lane; it < kc * cnt; it += kWarp) {
      const unsigned t = it / cnt;
      const int i = c.nzmin + (int)(it - t * cnt);
      const double* Ti = T + t * LW;
      const double d = Ti[i - 1] - Ti[i];
      if constexpr (FGB_FAST64) {
        S[t * LW + i] = d * g.at(g.DZ, i);
      } else {
        S[t * LW + i] = intdiv::divide(d, intdiv::prepared(g.at(g.DZ, i), bits64::to_bits(g.at(g.DX, i))));
      }
    }
    __syncwarp();
  }
  if constexpr (VER == 3) {
    const int cnt = c.nzmax - 2 - c.nzmin;  // layers (0-based) nzmin..nzmax-3
    for (int it = lane; cnt > 0 && it < (int)kc * cnt; it += kWarp) {
      const int t = it / cnt, j = c.nzmin + it - t * cnt;
      const double* Ti = T + t * LW;
      const double d1 = Ti[j + 1] - Ti[j], d0 = Ti[j] - Ti[j - 1];
      const double del = g.at(g.GA, j) * (g.at(g.GB, j) * d1 + g.at(g.GC, j) * d0);
      double r = 0.0;
      if (bits64::product_positive(d1, d0))
        r = copysign(rmin(rmin(rabs(del), rabs(bits64::twice(d1))), rabs(bits64::twice(d0))), del);
      S[t * LW + j] = r;
    }
    __syncwarp();
    // edge values tv (:510-594); the later assignment wins where the special cases coincide
    const unsigned ni = c.nlay + 1;
    for (unsigned it = lane; it < kc * ni; it += kWarp) {
      const unsigned t = it / ni;
      const int i = c.k0 + (int)(it - t * ni), z = i + 1;
      const double* Ti = T + t * LW;
      double e;
      if (z >= c.nzmin + 2 && z <= c.nzmax - 2) {
        const double T0 = Ti[i - 1], d = Ti[i] - T0;
        e = (T0 + g.at(g.GK, i) * d) +
            g.at(g.GL, i) * (g.at(g.GH, i) * d - g.at(g.GI, i) * S[t * LW + i] + g.at(g.GJ, i) * S[t * LW + i - 1]);
      } else if (z == c.nzmax) {
        e = Ti[c.nzmax - 2];
      } else if (z == c.nzmax - 1) {
        const double Tu = Ti[c.nzmax - 3], Tl = Ti[c.nzmax - 2], W = w[c.iw + c.nzmax - 2];
        e = bits64::finite(Tu, Tl) ? (bits64::sign_clear(W) ? Tl : Tu) : hw_ppm_bottom(Tu, Tl, W);
      } else if (z == c.nzmin + 1) {
        e = bits64::half(Ti[i - 1] + Ti[i]);
      } else {
        e = Ti[i];
      }
      TV[t * LW + i] = e;
    }
    __syncwarp();
  }
}

// First-order upwind flux through interface i (0-based, above layer i).
__device__ __forceinline__ double ver_upw1(const double* T, int i, int k0, double W, double A) {
  const double T0 = T[i], Tu = i == k0 ? T0 : T[i - 1];
  return -imul(bits64::upwind(W, T0, Tu, i == k0), A);
}

// The flux of a layer's parabola through one of its interfaces (:598-632) for
// hx = x / 2 and cx = 1 - 2/3 x, x = min(|W| dt / h, 1).
__device__ __forceinline__ double ppm_layer(double aL, double aR, double T0, double hx, double cx, bool upper, double A,
                                            double W) {
  if (!bits64::product_positive(aR - T0, T0 - aL) &&
      ((bits64::finite(aR, aL) && bits64::finite(T0)) || intdiv::hw_mul(aR - T0, T0 - aL) <= 0.0)) {
    aL = T0;
    aR = T0;
  }
  double d = aR - aL, c = T0 - bits64::half(aL + aR), dc = d * c, dd = sixth(d * d);
  if (bits64::exceeds(dc, dd)) {
    aL = 3.0 * T0 - bits64::twice(aR);
    d = aR - aL;
    c = T0 - bits64::half(aR + aL);
    dc = d * c;
    dd = sixth(d * d);
  }
  if (bits64::exceeds(-dd, dc)) {
    aR = 3.0 * T0 - bits64::twice(aL);
    d = aR - aL;
    c = T0 - bits64::half(aL + aR);
  }
  const double aj = 6.0 * c;
  const double tv = upper ? -aL - hx * (d + cx * aj) : -aR + hx * (d - cx * aj);
  return (tv * A) * W;
}

// High-order flux through interface i (0-based, above layer i of the column)
// minus f0 ("X - flux"). The boundary interfaces differ in their operands only,
// so that the lanes holding them do not make the warp run each case in turn.
template <int VER>
__device__ __forceinline__ double ver_flux(const VerGeo<VER>& g, const Column& c, const double* T, const double* S,
                                           const double* TV, int i, double W, double A, double num_ord, double f0) {
  const int z = i + 1;
  if constexpr (VER == 0) return ver_upw1(T, i, c.k0, W, A) - f0;
  if constexpr (VER == 1) {
    const double T0 = T[i], Tu = i == c.k0 ? T0 : T[i - 1];
    const bool mid = z >= c.nzmin + 2 && z <= c.nzmax - 2;
    double x = Tu, y = T0;
    if (mid) {
      const double q2 = bits64::twice(S[i]);
      y = T0 + third(imul(q2 + S[i + 1], g.at(g.A1, i)));
      x = Tu + third(imul(q2 + S[i - 1], g.at(g.A2, i)));
    }
    const double mean = i == c.k0 ? T0 : bits64::half(x + y);
    double ho = -imul(mean * W, A);
    // num_ord = 1: the upwind part is an exact zero (unless its products overflow)
    if (mid && !(num_ord == 1.0 && bits64::moderate(x, y) && bits64::moderate(W))) ho = qr4c_any(W, y, x, num_ord, A);
    const double f = ho - f0;
    return z == c.nzmin + 1 && z == c.nzmax - 1 ? ho - f : f;  // written twice (:405-411)
  }
  if constexpr (VER == 2) {
    const double T0 = T[i];
    return -(((i == c.k0 ? T0 : bits64::half(T[i == c.k0 ? i : i - 1] + T0)) * W) * A) - f0;
  }
  // PPM
  if (i == c.k0) return -((TV[i] * W) * A) - f0;
  // neither W > 0 nor W < 0 (:598-632): zero, and NaN, the bits above infinity's
  if ((bits64::to_bits(W) << 1) - 1 >= 0xffe0000000000000ull) return 0.0 - f0;
  const bool up = bits64::sign_clear(W);
  const int L = up ? i : i - 1;  // the layer whose parabola crosses the interface
  return ppm_layer(TV[L], TV[L + 1], T[L], g.at(g.HX, i), g.at(g.CX, i), up, A, W) - f0;
}

// ---------------------------------------------------------------------------
// FCT stage 1: low-order solution fct_LO (lib/oce_adv_tra_driver.F90:91-235)
// and the vertical antidiffusive flux HO(T_AB, w) - LO(T, w_e). The low-order
// horizontal edge fluxes are formed here from T and the edge volume fluxes,
// with the expression adv_tra_hor_upw1 uses (lib/oce_adv_tra_hor.F90:218-220).
// kc: tracers per chunk.
// Blocks per SM: QR4C keeps its values in 72 registers without a spill and the
// seventh block covers gather latency (512^2x48, 2 tracers, whole step 7694 ->
// 7603 us). The others' registers leave room for seven as they are (PPM 72,
// UPW1 66, CDIFF 64); compiled for seven, PPM takes 68 and was slower all the
// same (321^2 basin, fast form, step 4530 -> 4555 us), so their bound is six.
// ---------------------------------------------------------------------------
template <typename R, int VER>
__global__ void __launch_bounds__(kNodeWarps * kWarp, lo_blocks(VER)) k_fct_lo(DMesh m, StepPtrs<R> a, int kc_max) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & (kWarp - 1), wib = threadIdx.x / kWarp;
  const int vi = blockIdx.x * (blockDim.x / kWarp) + wib;
  if (vi >= m.N) return;
  const Column c(m, visit_node(m, vi));
  const GeoPtrs<R>& g = m.g64;
  const size_t LZ = m.LZ, LW = m.LW;
  const bool ta_sep = a.TA != a.T;
  const int slices = lo_slices(VER, kc_max, ta_sep);
  unsigned char* base = smem_raw + (size_t)wib * warp_smem<R>(slices, m.LW, 0);
  const VerGeo<VER> geo{reinterpret_cast<R*>(base), m.LW};
  R* sT = geo.s + ver_geo_slices(VER) * LW;
  R* sF = sT + kc_max * LW;  // low-order vertical fluxes
  R* sTA = ta_sep ? sF + kc_max * LW : sT;
  R* sS = (ta_sep ? sTA : sF) + kc_max * LW;
  R* sTV = sS + kc_max * LW;
  const NbrList nb = stage_nbrs(m, c.n, reinterpret_cast<Nbr*>(base + slices * LW * sizeof(R)), lane);
  geo.form(m, c, a.w, a.dt, lane);
  const R dt = a.dt;
  for (int t0 = 0; t0 < a.K; t0 += kc_max) {
    const unsigned kc = min(kc_max, a.K - t0), items = kc * c.nlay;
    __syncwarp();
    for (unsigned it = lane; it < items; it += kWarp) {
      const unsigned t = it / c.nlay;
      const int k = c.k0 + (int)(it - t * c.nlay);
      sT[t * LW + k] = a.T[(t0 + t) * a.sT + c.iz + k];
      if (ta_sep) sTA[t * LW + k] = a.TA[(t0 + t) * a.sTA + c.iz + k];
    }
    __syncwarp();
    // LO vertical flux: adv_tra_ver_upw1(we, ttf) with init zero
    for (unsigned it = lane; it < items; it += kWarp) {
      const unsigned t = it / c.nlay;
      const int i = c.k0 + (int)(it - t * c.nlay);
      sF[t * LW + i] = ver_upw1(sT + t * LW, i, c.k0, a.we[c.iw + i], g.area[c.iw + i]);
    }
    if (lane < (int)kc) sF[lane * LW + c.nzmax - 1] = R(0);
    __syncwarp();
    for (unsigned it = lane; it < items; it += kWarp) {
      const unsigned t = it / c.nlay;
      const int k = c.k0 + (int)(it - t * c.nlay), z = k + 1;
      const R* __restrict__ T = a.T + (t0 + t) * a.sT + k;
      const R tn = sT[t * LW + k];
      const R hn = g.hnode[c.iz + k], hnn = g.hnode_new[c.iz + k], av = g.areasvol[c.iz + k];
      R acc = R(0);
#pragma unroll 2
      for (int j = 0; j < nb.deg; ++j) {
        const Nbr q = nb.get(m, j);
        if (z < q.lo || z > q.hi) continue;
        const R v = a.vf[(size_t)q.e * LZ + k], to = T[(size_t)q.other * LZ];
        // the second node gains what the first one loses
        const R x = bits64::upwind(v, q.role ? to : tn, q.role ? tn : to);
        acc = acc + bits64::negate_if(x, !q.role);
      }
      const R dF = sF[t * LW + k] - sF[t * LW + k + 1];
      R l;
      if constexpr (FGB_FAST64) {
        l = (tn * hn + (acc + dF) * rdt_vol(dt, av)) * fdiv(R(1), hnn);
      } else {
        l = fdiv(imul(tn, hn) + fdiv(imul(acc + dF, dt), av), hnn);
      }
      a.lo[(t0 + t) * a.sN + c.iz + k] = l;
    }
    for (unsigned t = 0; t < kc; ++t)  // below the bottom
      for (int k = c.nzmax - 1 + lane; k < (int)LZ; k += kWarp) a.lo[(t0 + t) * a.sN + c.iz + k] = R(0);
    if (a.wi) {
      // w_split: the antidiffusive flux takes the upwind flux of the full w
      // (lib/oce_adv_tra_driver.F90:221-231)
      __syncwarp();  // every lane has read the LO fluxes before they are overwritten
      for (unsigned it = lane; it < items; it += kWarp) {
        const unsigned t = it / c.nlay;
        const int i = c.k0 + (int)(it - t * c.nlay);
        sF[t * LW + i] = ver_upw1(sT + t * LW, i, c.k0, a.w[c.iw + i], g.area[c.iw + i]);
      }
    }
    // HO vertical flux on T_AB with w; adf_v = HO - LO ("X - flux")
    ver_prepare<VER>(geo, c, sTA, sS, sTV, a.w, kc, lane);
    for (unsigned it = lane; it < items; it += kWarp) {
      const unsigned t = it / c.nlay;
      const int i = c.k0 + (int)(it - t * c.nlay);
      a.adfv[(t0 + t) * a.sW + c.iw + i] = ver_flux<VER>(geo, c, sTA + t * LW, sS + t * LW, sTV + t * LW, i, a.w[c.iw + i],
                                                         g.area[c.iw + i], a.pv, sF[t * LW + i]);
    }
    for (unsigned t = 0; t < kc; ++t)  // from the bottom interface on
      for (int i = c.nzmax - 1 + lane; i < (int)LW; i += kWarp) a.adfv[(t0 + t) * a.sW + c.iw + i] = R(0);
  }
}

// The larger of lo and t joins the upper bound, the smaller the lower one (integer keys).
__device__ __forceinline__ void join_bounds(double lo, double t, long long& mx, long long& mn) {
  const long long a = bits64::key(lo), b = bits64::key(t);
  const bool gt = a > b;
  mx = max(mx, gt ? a : b);
  mn = min(mn, gt ? b : a);
}
// The sums of the positive and of the negative terms: a term joins one of them
// (the other would add an exact zero), so each costs one FP64 addition.
__device__ __forceinline__ void add_part(double f, double& pos, double& neg) {
  const bool p = bits64::sign_clear(f);
  const double t = (p ? pos : neg) + f;
  pos = p ? t : pos;
  neg = p ? neg : t;
}
// Their first two terms x and -y: max(0, x) + max(0, -y) and min(0, x) + min(0, -y).
__device__ __forceinline__ void first_parts(double x, double y, double& pos, double& neg) {
  const bool px = bits64::sign_clear(x), py = !bits64::sign_clear(y);
  const double t = x - y, u = bits64::negate_if(y, true);
  pos = px ? (py ? t : x) : (py ? u : 0.0);
  neg = px ? (py ? 0.0 : u) : (py ? x : t);
}
// A NaN term belongs to both sums.
__device__ __forceinline__ void spread_nan(double& pos, double& neg) {
  if (bits64::finite(pos, neg)) return;
  if (isnan(pos)) neg = pos;
  else if (isnan(neg)) pos = neg;
}

// ---------------------------------------------------------------------------
// FCT stage 2: bounds a1-a3, antidiffusive sums b1 and the limiting factors
// b2 (lib/oce_adv_tra_fct.F90:98-374). The cluster bound is the maximum over
// the cluster's elements of the maximum over their nodes; max is exact, so
// the distinct nodes with the deepest layer reaching them give the same value.
// ---------------------------------------------------------------------------
template <typename R>
__global__ void __launch_bounds__(kNodeWarps * kWarp, kRatioBlocks) k_fct_ratio(DMesh m, StepPtrs<R> a, int kc_max) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & (kWarp - 1), wib = threadIdx.x / kWarp;
  const int vi = blockIdx.x * (blockDim.x / kWarp) + wib;
  if (vi >= m.N) return;
  const Column c(m, visit_node(m, vi));
  const GeoPtrs<R>& g = m.g64;
  const size_t LZ = m.LZ, LW = m.LW;
  unsigned char* base = smem_raw + (size_t)wib * warp_smem<R>(ratio_slices(kc_max), m.LW, kClBytes);
  R* smax = reinterpret_cast<R*>(base);
  R* smin = smax + kc_max * LW;
  const NbrList nb = stage_nbrs(m, c.n, reinterpret_cast<Nbr*>(base + ratio_slices(kc_max) * LW * sizeof(R)), lane);
  int* scl = reinterpret_cast<int*>(base + ratio_slices(kc_max) * LW * sizeof(R) + kMaxDeg * sizeof(Nbr));
  const int c0 = m.cl_ptr[c.n], ncl = m.cl_ptr[c.n + 1] - c0, minlev = m.cl_minlev[c.n];
  const bool cl_staged = ncl <= kMaxCl;
  if (cl_staged)
    for (int j = lane; j < ncl; j += kWarp) {
      scl[2 * j] = m.cl_node[c0 + j];
      scl[2 * j + 1] = m.cl_lev[c0 + j];
    }
  const R dt = a.dt;
  for (int t0 = 0; t0 < a.K; t0 += kc_max) {
    const unsigned kc = min(kc_max, a.K - t0), items = kc * c.nlay;
    __syncwarp();
    for (unsigned it = lane; it < items; it += kWarp) {
      const unsigned t = it / c.nlay;
      const int k = c.k0 + (int)(it - t * c.nlay), z = k + 1;
      const R* __restrict__ lo = a.lo + (t0 + t) * a.sN + k;
      const R* __restrict__ T = a.T + (t0 + t) * a.sT + k;
      // AUX = -/+1e3 of elements without the layer joins the bound (lib/oce_adv_tra_fct.F90:139-145)
      const R first = z > minlev ? R(-1e3) : R(-INFINITY);
      // the bounds as integer keys (bits64::key), which order as the values do
      long long mx = bits64::key(first), mn = bits64::key(-first);
#pragma unroll 2
      for (int j = 0; j < ncl; ++j) {
        const int node = cl_staged ? scl[2 * j] : m.cl_node[c0 + j];
        const int lev = cl_staged ? scl[2 * j + 1] : m.cl_lev[c0 + j];
        if (z <= lev) join_bounds(lo[(size_t)node * LZ], T[(size_t)node * LZ], mx, mn);
      }
      R x = bits64::unkey(mx), y = bits64::unkey(mn);
      // A NaN is the largest or the smallest key of all, so it is still there:
      // the bounds again with the floating-point comparisons, whose outcome
      // with NaNs depends on the order.
      if (mx > bits64::kKeyInf || mn < -bits64::kKeyInf - 1) {
        x = first;
        y = -first;
        for (int j = 0; j < ncl; ++j) {
          if (z > m.cl_lev[c0 + j]) continue;
          const size_t v = (size_t)m.cl_node[c0 + j] * LZ;
          x = rmax(x, rmax(lo[v], T[v]));
          y = rmin(y, rmin(lo[v], T[v]));
        }
      }
      smax[t * LW + k] = x;
      smin[t * LW + k] = y;
    }
    __syncwarp();
    for (unsigned it = lane; it < items; it += kWarp) {
      const unsigned t = it / c.nlay;
      const int k = c.k0 + (int)(it - t * c.nlay), z = k + 1;
      const R* __restrict__ adfv = a.adfv + (t0 + t) * a.sW + c.iw + k;
      const R* __restrict__ adfh = a.adfh + (t0 + t) * a.sE + k;
      R pl, mi;
      first_parts(adfv[0], adfv[1], pl, mi);
#pragma unroll 2
      for (int j = 0; j < nb.deg; ++j) {
        const Nbr q = nb.get(m, j);
        if (z >= q.lo && z <= q.hi) add_part(bits64::negate_if(adfh[(size_t)q.e * LZ], q.role), pl, mi);
      }
      spread_nan(pl, mi);
      const R lo = a.lo[(t0 + t) * a.sN + c.iz + k];
      const R* mxs = smax + t * LW + k;
      const R* mns = smin + t * LW + k;
      R x = mxs[0], y = mns[0];
      if (z != c.nzmax - 1 && z != c.nzmin) {
        x = rmax(rmax(mxs[-1], x), mxs[1]);
        y = rmin(rmin(mns[-1], y), mns[1]);
      }
      const R av = g.areasvol[c.iz + k];
      const LayerDivisor dv(av);
      const R rd = rdt_vol(dt, av);
      const R rp = rmin(R(1), fdiv(x - lo, dt_per_vol(pl, dt, dv, rd) + R(1e-16)));
      const R rm = rmin(R(1), fdiv(y - lo, dt_per_vol(mi, dt, dv, rd) - R(1e-16)));
      reinterpret_cast<double2*>(a.rpm)[(t0 + t) * a.sN + c.iz + k] = make_double2(rp, rm);
    }
    for (unsigned t = 0; t < kc; ++t)  // below the bottom
      for (int k = c.nzmax - 1 + lane; k < (int)LZ; k += kWarp)
        reinterpret_cast<double2*>(a.rpm)[(t0 + t) * a.sN + c.iz + k] = make_double2(0.0, 0.0);
  }
}

// New value and its AB level of one layer, from the layer's tendency e.
template <typename R>
__device__ __forceinline__ void store_new(const StepPtrs<R>& a, int t, size_t i, R Tn, R e, R hnn) {
  const R nv = FGB_FAST64 ? Tn + e * fdiv(R(1), hnn) : Tn + fdiv(e, hnn);
  a.T[t * a.sT + i] = nv;
  if (a.del) a.del[t * a.sN + i] = e;
  if (a.TAout) a.TAout[t * a.sTA + i] = a.ab2 ? a.ab_old * Tn + a.ab_new * nv : nv;
}
// The AB level of the layers below a column's bottom, whose values stay.
template <typename R>
__device__ __forceinline__ void store_ab_below(const DMesh& m, const StepPtrs<R>& a, const Column& c, int lane) {
  if (!a.TAout) return;
  for (int t = 0; t < a.K; ++t)
    for (int k = c.nzmax - 1 + lane; k < m.LZ; k += kWarp) {
      const R Tn = a.T[t * a.sT + c.iz + k];
      a.TAout[t * a.sTA + c.iz + k] = a.ab2 ? a.ab_old * Tn + a.ab_new * Tn : Tn;
    }
}

// ---------------------------------------------------------------------------
// FCT stage 3: limiting b3 (lib/oce_adv_tra_fct.F90:396-471), flux divergence
// (oce_tra_adv_flux2dtracer with use_lo, lib/oce_adv_tra_driver.F90:298-450)
// and the caller's tendency update (src/fesom_analytic.F90:419-437 or, with a
// persistent del_ttf, lib/tracer_c_interface.F90:194-214). The limiting
// factors are at most 1 (or NaN), so the reference's min(1, a, b) is min(a, b).
// Seven blocks per SM: 72 registers (77 with six blocks, 36 % of the warps in
// flight, gathers as long a wait as the FP64 pipe) still hold everything; the
// 512^2x48 step with 2 tracers 7785 -> 7694 us. Eight (64) would spill.
// ---------------------------------------------------------------------------
template <typename R>
__global__ void __launch_bounds__(kNodeWarps * kWarp, kUpdateBlocks) k_fct_update(DMesh m, StepPtrs<R> a, int kc_max) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & (kWarp - 1), wib = threadIdx.x / kWarp;
  const int vi = blockIdx.x * (blockDim.x / kWarp) + wib;
  if (vi >= m.N) return;
  const Column c(m, visit_node(m, vi));
  const GeoPtrs<R>& g = m.g64;
  const size_t LZ = m.LZ, LW = m.LW;
  unsigned char* base = smem_raw + (size_t)wib * warp_smem<R>(upd_slices(kc_max), m.LW, 0);
  R* sF = reinterpret_cast<R*>(base);  // limited vertical fluxes
  const NbrList nb = stage_nbrs(m, c.n, reinterpret_cast<Nbr*>(base + upd_slices(kc_max) * LW * sizeof(R)), lane);
  const R dt = a.dt;
  for (int t0 = 0; t0 < a.K; t0 += kc_max) {
    const unsigned kc = min(kc_max, a.K - t0), items = kc * c.nlay;
    __syncwarp();
    for (unsigned it = lane; it < items; it += kWarp) {
      const unsigned t = it / c.nlay;
      const int i = c.k0 + (int)(it - t * c.nlay);
      const double2* __restrict__ Rn = reinterpret_cast<const double2*>(a.rpm) + (t0 + t) * a.sN + c.iz + i;
      const R f = a.adfv[(t0 + t) * a.sW + c.iw + i];
      const bool pos = bits64::sign_clear(f);
      const double2 own = Rn[0];
      R ae = pos ? own.x : own.y;
      if (i > c.k0) {
        const double2 above = Rn[-1];
        ae = rmin(pos ? above.y : above.x, ae);
      }
      sF[t * LW + i] = ae * f;
    }
    if (lane < (int)kc) sF[lane * LW + c.nzmax - 1] = a.adfv[(t0 + lane) * a.sW + c.iw + c.nzmax - 1];
    __syncwarp();
    for (unsigned it = lane; it < items; it += kWarp) {
      const unsigned t = it / c.nlay;
      const int k = c.k0 + (int)(it - t * c.nlay), z = k + 1;
      const R* __restrict__ adfh = a.adfh + (t0 + t) * a.sE + k;
      const double2* __restrict__ Rg = reinterpret_cast<const double2*>(a.rpm) + (t0 + t) * a.sN + k;
      const double2 own = Rg[c.iz];
      const R av = g.areasvol[c.iz + k], hn = g.hnode[c.iz + k], hnn = g.hnode_new[c.iz + k];
      const R lo = a.lo[(t0 + t) * a.sN + c.iz + k], Tn = a.T[(t0 + t) * a.sT + c.iz + k];
      const LayerDivisor dv(av);        // exact form only
      const R rd = rdt_vol(dt, av);     // fast form only
      R dh = R(0);
#pragma unroll 2
      for (int j = 0; j < nb.deg; ++j) {
        const Nbr q = nb.get(m, j);
        if (z < q.lo || z > q.hi) continue;
        const R f = adfh[(size_t)q.e * LZ];
        const double2 o = Rg[(size_t)q.other * LZ];
        // this node's factor and the other one's, for the flux's sign; the reference takes the
        // first node's against the second node's
        const bool up = bits64::sign_clear(f) != (bool)q.role;
        const R mine = up ? own.x : own.y, oth = up ? o.y : o.x;
        const R x = dt_per_vol((q.role ? rmin(oth, mine) : rmin(mine, oth)) * f, dt, dv, rd);
        dh = dh + bits64::negate_if(x, q.role);
      }
      // the reference's (0 - T hnode) + LO hnode_new, then the vertical flux divergence
      R e = lo * hnn - Tn * hn;
      e = e + dt_per_vol(sF[t * LW + k] - sF[t * LW + k + 1], dt, dv, rd);
      if (a.del) dh = a.del[(t0 + t) * a.sN + c.iz + k] + dh;
      store_new(a, t0 + (int)t, c.iz + k, Tn, dh + e, hnn);
    }
  }
  store_ab_below(m, a, c, lane);
}

// ---------------------------------------------------------------------------
// Without a limiter: vertical HO flux on T_AB with w_e, flux divergence
// (oce_tra_adv_flux2dtracer) and the tendency update in one pass.
// ---------------------------------------------------------------------------
template <typename R, int VER>
__global__ void __launch_bounds__(kNodeWarps * kWarp, kNofctBlocks) k_nofct_update(DMesh m, StepPtrs<R> a, int kc_max) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & (kWarp - 1), wib = threadIdx.x / kWarp;
  const int vi = blockIdx.x * (blockDim.x / kWarp) + wib;
  if (vi >= m.N) return;
  const Column c(m, visit_node(m, vi));
  const GeoPtrs<R>& g = m.g64;
  const size_t LZ = m.LZ, LW = m.LW;
  const int slices = nofct_slices(VER, kc_max);
  unsigned char* base = smem_raw + (size_t)wib * warp_smem<R>(slices, m.LW, 0);
  const VerGeo<VER> geo{reinterpret_cast<R*>(base), m.LW};
  R* sTA = geo.s + ver_geo_slices(VER) * LW;
  R* sF = sTA + kc_max * LW;
  R* sS = sF + kc_max * LW;
  R* sTV = sS + kc_max * LW;
  const NbrList nb = stage_nbrs(m, c.n, reinterpret_cast<Nbr*>(base + slices * LW * sizeof(R)), lane);
  geo.form(m, c, a.we, a.dt, lane);
  const R dt = a.dt;
  for (int t0 = 0; t0 < a.K; t0 += kc_max) {
    const unsigned kc = min(kc_max, a.K - t0), items = kc * c.nlay;
    __syncwarp();
    for (unsigned it = lane; it < items; it += kWarp) {
      const unsigned t = it / c.nlay;
      const int k = c.k0 + (int)(it - t * c.nlay);
      sTA[t * LW + k] = a.TA[(t0 + t) * a.sTA + c.iz + k];
    }
    __syncwarp();
    ver_prepare<VER>(geo, c, sTA, sS, sTV, a.we, kc, lane);
    for (unsigned it = lane; it < items; it += kWarp) {
      const unsigned t = it / c.nlay;
      const int i = c.k0 + (int)(it - t * c.nlay);
      sF[t * LW + i] = ver_flux<VER>(geo, c, sTA + t * LW, sS + t * LW, sTV + t * LW, i, a.we[c.iw + i], g.area[c.iw + i],
                                     a.pv, R(0));
    }
    if (lane < (int)kc) sF[lane * LW + c.nzmax - 1] = R(0);
    __syncwarp();
    for (unsigned it = lane; it < items; it += kWarp) {
      const unsigned t = it / c.nlay;
      const int k = c.k0 + (int)(it - t * c.nlay), z = k + 1;
      const R* __restrict__ flux = a.adfh + (t0 + t) * a.sE + k;
      const R av = g.areasvol[c.iz + k], hnn = g.hnode_new[c.iz + k], Tn = a.T[(t0 + t) * a.sT + c.iz + k];
      const LayerDivisor dv(av);     // exact form only
      const R rd = rdt_vol(dt, av);  // fast form only
      R dh = R(0);
#pragma unroll 2
      for (int j = 0; j < nb.deg; ++j) {
        const Nbr q = nb.get(m, j);
        if (z < q.lo || z > q.hi) continue;
        dh = dh + bits64::negate_if(dt_per_vol(flux[(size_t)q.e * LZ], dt, dv, rd), q.role);
      }
      const R e = dt_per_vol(sF[t * LW + k] - sF[t * LW + k + 1], dt, dv, rd);
      if (a.del) dh = a.del[(t0 + t) * a.sN + c.iz + k] + dh;
      store_new(a, t0 + (int)t, c.iz + k, Tn, dh + e, hnn);
    }
  }
  store_ab_below(m, a, c, lane);
}

}  // inline namespace
}  // namespace fgb
