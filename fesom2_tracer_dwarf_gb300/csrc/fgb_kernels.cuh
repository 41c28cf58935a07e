// Device kernels of the FESOM2 tracer-advection step (do_oce_adv_tra,
// lib/oce_adv_tra_driver.F90:23-294) for GB300 (sm_103a).
//
// Layout: level index fastest, columns padded to LZ layers / LW interfaces.
// Node-column kernels run one warp per node with the column staged in shared
// memory; edge kernels run one warp per edge, lanes over layers (coalesced
// rows) with two consecutive layers per lane. Node kernels loop over the
// tracers of a launch KC at a time, so the mesh tables, geometry and edge
// volume fluxes they load serve all tracers. The reference's edge scatters (atomics / OpenMP locks) are
// replaced by gathers over each node's incident edges in ascending edge order,
// which reproduces the reference's per-node summation order exactly.
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
    v1 = (-(w * q.dX1) + u * q.dY1) * m.g64.helem[i];
  }
  if (s2) {
    const size_t i = (size_t)q.el2 * m.LZ + k;
    const double u = vel[2 * i], w = vel[2 * i + 1];
    v2 = (w * q.dX2 - u * q.dY2) * m.g64.helem[i];
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
      out[((size_t)t * m.M + el) * LZ + k] = make_double2(x0 * ta + x1 * tb + x2 * tc, y0 * ta + y1 * tb + y2 * tc);
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

// Two consecutive layers per lane: vector loads and stores of R pairs.
template <typename R>
struct V2T;
template <>
struct V2T<float> {
  using T = float2;
};
template <>
struct V2T<double> {
  using T = double2;
};
template <typename R>
using vec2 = typename V2T<R>::T;
template <typename R>
__device__ __forceinline__ vec2<R> ld2(const R* p) {
  return *reinterpret_cast<const vec2<R>*>(p);
}
template <typename R>
__device__ __forceinline__ void st2(R* p, R a, R b) {
  vec2<R> v;
  v.x = a;
  v.y = b;
  *reinterpret_cast<vec2<R>*>(p) = v;
}

// Four values per lane (two layers of an interleaved pair array).
template <typename R>
struct Q4 {
  R a, b, c, d;
};
__device__ __forceinline__ Q4<float> ld4(const float* p) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  return Q4<float>{v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ Q4<double> ld4(const double* p) {
  const double2 u = *reinterpret_cast<const double2*>(p), v = *reinterpret_cast<const double2*>(p + 2);
  return Q4<double>{u.x, u.y, v.x, v.y};
}
__device__ __forceinline__ void st4(float* p, float a, float b, float c, float d) {
  *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}
__device__ __forceinline__ void st4(double* p, double a, double b, double c, double d) {
  *reinterpret_cast<double2*>(p) = make_double2(a, b);
  *reinterpret_cast<double2*>(p + 2) = make_double2(c, d);
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
// together against 10.9.
// ---------------------------------------------------------------------------
// The slow forms behind it, out of line (see bits64): the reconstruction's mask as a
// product where a value is infinite or NaN, and the flux for any ph.
static __device__ __noinline__ double hw_product(double a, double b) { return a * b; }
static __device__ __noinline__ double hor_flux_any(double v, double Tm1, double Tm2, double ph) {
  const double cHO = (v + fabs(v)) * Tm1 + (v - fabs(v)) * Tm2;
  return -((0.5 * (1.0 - ph)) * cHO) - ((v * ph) * 0.5) * (Tm1 + Tm2);
}

template <typename R, int HOR, bool FCT, bool VF, bool GRAD>
__global__ void __launch_bounds__(kEdgeThreads, 3) k_hflux(DMesh m, StepPtrs<R> a, const double2* __restrict__ grad) {
  __shared__ EdgeTab tab[kEdgeTile];
  const int w0 = blockIdx.x * kEdgeTile, ne = min(kEdgeTile, m.E - w0);
  if ((int)threadIdx.x < ne) tab[threadIdx.x] = load_edge<HOR>(m, w0 + threadIdx.x);
  __syncthreads();
  const size_t LZ = m.LZ;
  const bool ta_sep = a.TA != a.T;
  const bool ph1 = a.ph == R(1);
  for (unsigned i = threadIdx.x; i < (unsigned)(ne * m.LZ); i += kEdgeThreads) {
    const unsigned j = i / (unsigned)m.LZ;
    const int k = (int)(i - j * (unsigned)m.LZ), z = k + 1;
    const EdgeTab& q = tab[j];
    const size_t ek = (size_t)q.e * LZ + k;
    R v;
    if (VF) {
      v = edge_vflux(m, q, a.vel, k);
      a.vf[ek] = v;
    }
    if (z > max(q.nl1, q.nl2)) {
      for (int t = 0; t < a.K; ++t) a.adfh[t * a.sE + ek] = R(0);
      continue;
    }
    if (!VF) v = a.vf[ek];
    const R B = bits64::half(ph1 ? v : v * a.ph);
    const bool tri = q.gm0 >= 0 && z >= q.gm0 && z <= q.gm1 - 1;
    const bool c1 = HOR == 2 || q.nb1 - z >= 0, c2 = HOR == 2 || q.nb2 - z >= 0;
    const size_t i1 = q.n1 * LZ + k, i2 = q.n2 * LZ + k;
    for (int t = 0; t < a.K; ++t) {
      const R* __restrict__ T = a.T + t * a.sT;
      const R* __restrict__ TA = ta_sep ? a.TA + t * a.sTA : T;
      const R s1 = TA[i1], s2 = TA[i2];
      R lo = R(0);  // minus the low-order flux
      if (FCT) lo = ta_sep ? bits64::upwind(v, T[i1], T[i2]) : bits64::upwind(v, s1, s2);
      R h;
      if (HOR == 0) {
        h = -(FCT && !ta_sep ? lo : bits64::upwind(v, s1, s2));
      } else {
        const double2* __restrict__ G = GRAD ? grad + (size_t)t * m.M * LZ : nullptr;
        R g1, g2, g3, g4;
        if (tri) {
          grad_at<GRAD>(m, TA, G, q.up, k, g1, g3);
          grad_at<GRAD>(m, TA, G, q.dn, k, g2, g4);
        } else {
          node_mean_grad<GRAD>(m, TA, G, q.n1, k, g1, g3);
          node_mean_grad<GRAD>(m, TA, G, q.n2, k, g2, g4);
        }
        const R d2 = bits64::twice(s2 - s1);
        R r1 = sixth(d2 + q.ex * g1 + q.ey * g3), r2 = sixth(d2 + q.ex * g2 + q.ey * g4);
        if (HOR == 1 && !(c1 && c2)) {
          if (bits64::finite(r1, r2)) {
            r1 = c1 ? r1 : R(0);
            r2 = c2 ? r2 : R(0);
          } else {
            r1 = hw_product(r1, c1 ? R(1) : R(0));
            r2 = hw_product(r2, c2 ? R(1) : R(0));
          }
        }
        const R Tm1 = s1 + r1, Tm2 = s2 - r2;
        // ph = 1: the upwind part is an exact zero (of finite values)
        if (ph1 && bits64::finite(Tm1, Tm2) && bits64::finite(v)) h = -(B * (Tm1 + Tm2));
        else h = hor_flux_any(v, Tm1, Tm2, a.ph);
      }
      a.adfh[t * a.sE + ek] = FCT ? h + lo : h;
    }
  }
}

// ---------------------------------------------------------------------------
// Vertical fluxes of one column at interface z (1-based), given the staged
// column. flux_old is the value the reference subtracts ("X - flux").
// VER: 0 UPW1, 1 QR4C, 2 CDIFF, 3 PPM (lib/oce_adv_tra_ver.F90:248-712).
// Staged arrays are 0-based by layer/interface.
// ---------------------------------------------------------------------------
template <typename R>
struct Col {
  const R* T;     // tracer at layers
  const R* W;     // vertical velocity at interfaces
  const R* area;  // at interfaces
  const R* hn;    // hnode at layers (PPM)
  const R* hnn;   // hnode_new at layers (PPM)
  const R* Z;     // Z_3d_n at layers (QR4C)
  const R* zb;    // zbar_3d_n at interfaces (QR4C)
  const R* tv;    // PPM edge values at interfaces
};

template <typename R>
__device__ __forceinline__ R ver_upw1(const Col<R>& c, int z, int nzmin, int nzmax, R fold) {
  if (z == nzmin) return -((c.W[z - 1] * c.T[z - 1]) * c.area[z - 1]) - fold;
  if (z == nzmax) return R(0) - fold;
  return -(bits64::upwind(c.W[z - 1], c.T[z - 1], c.T[z - 2]) * c.area[z - 1]) - fold;
}

// QR4C: the layer-to-layer slopes (T(z-1) - T(z)) / (Z(z-1) - Z(z)) are staged in c.tv by
// interface (qr4c_slopes): an interface uses its own and both neighbours'.
template <typename R>
__device__ __forceinline__ R ver_qr4c(const Col<R>& c, int z, int nzmin, int nzmax, R num_ord, R fold) {
  const R W = c.W[z - 1];
  if (z == nzmin) return -((c.T[z - 1] * W) * c.area[z - 1]) - fold;
  if (z == nzmax) return R(0) - fold;
  if (z == nzmin + 1 || z == nzmax - 1) {
    const R x = -((bits64::half(c.T[z - 2] + c.T[z - 1]) * W) * c.area[z - 1]);
    R f = x - fold;
    if (nzmin + 1 == nzmax - 1) f = x - f;  // written twice (lib/oce_adv_tra_ver.F90:405-411)
    return f;
  }
  const R T0 = c.T[z - 1], Tm1 = c.T[z - 2];
  const R q2 = bits64::twice(c.tv[z - 1]), qu = c.tv[z], qd = c.tv[z - 2];
  const R zb = c.zb[z - 1];
  const R tm1 = T0 + third((q2 + qu) * (zb - c.Z[z - 1]));
  const R tm2 = Tm1 + third((q2 + qd) * (zb - c.Z[z - 2]));
  const R mean = (num_ord * bits64::half(tm1 + tm2)) * W;
  // num_ord = 1: the upwind part is an exact zero (of finite values)
  if (num_ord == R(1) && bits64::finite(tm1, tm2) && bits64::finite(W)) return -mean * c.area[z - 1] - fold;
  const R tm = (W + rabs(W)) * tm1 + (W - rabs(W)) * tm2;
  return (-((R(0.5) * (R(1) - num_ord)) * tm) - mean) * c.area[z - 1] - fold;
}

// The slopes of KC tracer columns (T, q: LW apart), the divisor of an interface prepared once.
template <typename R, int KC>
__device__ __forceinline__ void qr4c_slopes(const R* T, const R* Z, R* q, int LW, int nzmin, int nzmax, int lane) {
  for (int iz = nzmin + lane; iz < nzmax - 1; iz += kWarp) {
    const intdiv::Divisor dz = intdiv::prepare(Z[iz - 1] - Z[iz]);
    const R rz = FGB_FAST64 ? intdiv::divide(R(1), dz) : R(0);
#pragma unroll
    for (int i = 0; i < KC; ++i) {
      const R d = T[i * LW + iz - 1] - T[i * LW + iz];
      q[i * LW + iz] = FGB_FAST64 ? d * rz : intdiv::divide(d, dz);
    }
  }
}

template <typename R>
__device__ __forceinline__ R ver_cdiff(const Col<R>& c, int z, int nzmin, int nlev, R fold) {
  const int nzmax = nlev - 1;  // lib/oce_adv_tra_ver.F90:689
  if (z == nzmin) return -((c.W[z - 1] * c.T[z - 1]) * c.area[z - 1]) - fold;
  if (z <= nzmax) {
    const R tv = bits64::half(c.T[z - 2] + c.T[z - 1]);
    return -((tv * c.W[z - 1]) * c.area[z - 1]) - fold;
  }
  return fold;  // the bottom interface is left untouched
}

// PPM edge value tv(z) of lib/oce_adv_tra_ver.F90:510-594 outside its
// four-point range (column_ppm has that); the later assignment wins where the
// special cases coincide.
template <typename R>
__device__ __forceinline__ R ppm_tv_end(const R* T, const R* W, int z, int nzmin, int nzmax) {
  if (z == nzmax) return T[nzmax - 2];
  if (z == nzmax - 1) {
    const R Tu = T[nzmax - 3], Tl = T[nzmax - 2];
    if (bits64::finite(Tu, Tl)) return bits64::sign_clear(W[nzmax - 2]) ? Tl : Tu;
    const R s = copysign(R(1), W[nzmax - 2]);
    return -(Tu * rmin(s, R(0))) + Tl * rmax(s, R(0));
  }
  if (z == nzmin + 1) return bits64::half(T[nzmin - 1] + T[nzmin]);
  return T[nzmin - 1];
}

// The flux of a layer's parabola through one of its interfaces
// (lib/oce_adv_tra_ver.F90:598-632) for x = min(|W| dt / h, 1), hx = x / 2 and
// cx = 1 - 2/3 x of the layer.
template <typename R>
__device__ __forceinline__ R ppm_layer_x(R aL, R aR, R T0, R hx, R cx, bool upper, R area, R W) {
  if (!bits64::product_positive(aR - T0, T0 - aL)) {
    // (a NaN product is not <= 0)
    if (bits64::finite(aR, aL) && bits64::finite(T0)) {
      aL = T0;
      aR = T0;
    } else if ((aR - T0) * (T0 - aL) <= R(0)) {
      aL = T0;
      aR = T0;
    }
  }
  R d = aR - aL, c = T0 - bits64::half(aL + aR), dc = d * c, dd = sixth(d * d);
  if (bits64::exceeds(dc, dd)) {
    aL = R(3) * T0 - bits64::twice(aR);
    d = aR - aL;
    c = T0 - bits64::half(aR + aL);
    dc = d * c;
    dd = sixth(d * d);
  }
  if (bits64::exceeds(-dd, dc)) {
    aR = R(3) * T0 - bits64::twice(aL);
    d = aR - aL;
    c = T0 - bits64::half(aL + aR);
  }
  const R aj = R(6) * c;
  const R tv = upper ? -aL - hx * (d + cx * aj) : -aR + hx * (d - cx * aj);
  return (tv * area) * W;
}

// x of ppm_layer: upper side min(W dt / h, 1), lower side min(-(W dt / h), 1).
template <typename R>
__device__ __forceinline__ R ppm_x(R W, R dt, R dzj, bool upper) {
  return upper ? rmin(fdiv(W * dt, dzj), R(1)) : rmin(-fdiv(W * dt, dzj), R(1));
}

template <typename R, int VER>  // not PPM: column_ppm
__device__ __forceinline__ R ver_flux(const Col<R>& c, int z, int nzmin, int nzmax, R num_ord, R dt, R fold) {
  if (VER == 1) return ver_qr4c(c, z, nzmin, nzmax, num_ord, fold);
  if (VER == 2) return ver_cdiff(c, z, nzmin, nzmax, fold);
  return ver_upw1(c, z, nzmin, nzmax, fold);
}

// Shared-memory slices of one warp's column.
template <typename R>
struct ColSmem {
  R* s;
  int LW;
  __device__ R* slice(int i) const { return s + (size_t)i * LW; }
};

template <typename R>
__device__ __forceinline__ void stage(R* dst, const R* __restrict__ src, int n, int lane) {
  for (int k = lane; k < n; k += kWarp) dst[k] = src[k];
}

// Vertical flux of the column into out[iz] (interfaces) by a scheme other
// than PPM; QR4C needs its slopes in c.tv. fold[iz] holds the value subtracted.
template <typename R, int VER>
__device__ __forceinline__ void column_ver_flux(const Col<R>& c, const R* fold, R* out, int nl, int nzmin, int nzmax,
                                                R num_ord, R dt, int lane) {
  for (int iz = lane; iz < nl; iz += kWarp) {
    const int z = iz + 1;
    const R f0 = fold ? fold[iz] : R(0);
    out[iz] = (z >= nzmin && z <= nzmax) ? ver_flux<R, VER>(c, z, nzmin, nzmax, num_ord, dt, f0) : f0;
  }
  __syncwarp();
}

// PPM vertical fluxes of KC tracer columns of one node (adv_tra_vert_ppm,
// lib/oce_adv_tra_ver.F90:448-644). What the reference forms per interface is
// formed once: the limited slope of a layer (its deltaj at one interface and
// deltajp1 at the next are the same expression of the same operands) and, for
// all tracers, the quotients of layer thicknesses, whose divisors repeat. T,
// tv, fold and out hold KC columns LW apart; fold == out is allowed. tv holds
// the slopes by layer first and is overwritten with the edge values from the
// bottom up, each pass after the slopes it reads.
template <typename R, int KC>
__device__ __forceinline__ void column_ppm_multi(const Col<R>& g, const R* T, R* tv, const R* fold, R* out, int LW,
                                                 int nl, int nzmin, int nzmax, R dt, int lane) {
  const R* hnn = g.hnn;
  for (int j = nzmin + lane; j <= nzmax - 3; j += kWarp) {  // layers (0-based) with both neighbours
    const R dzm = hnn[j - 1], dz = hnn[j], dzp = hnn[j + 1];
    const R sm = dzm + dz;
    const R ga = fdiv(dz, sm + dzp);
    const R gb = fdiv(bits64::twice(dzm) + dz, dzp + dz), gc = fdiv(dz + bits64::twice(dzp), sm);
#pragma unroll
    for (int i = 0; i < KC; ++i) {
      const R* Ti = T + i * LW;
      const R d1 = Ti[j + 1] - Ti[j], d0 = Ti[j] - Ti[j - 1];
      const R del = ga * (gb * d1 + gc * d0);
      R r = R(0);
      if (bits64::product_positive(d1, d0))
        r = copysign(rmin(rmin(rabs(del), rabs(bits64::twice(d1))), rabs(bits64::twice(d0))), del);
      tv[i * LW + j] = r;
    }
  }
  __syncwarp();
  for (int base = (nl - 1) / kWarp * kWarp; base >= 0; base -= kWarp) {
    const int iz = base + lane, z = iz + 1;
    R e[KC];
    if (z >= nzmin + 2 && z <= nzmax - 2) {
      const R dzjm1 = hnn[iz - 2], dzj = hnn[iz - 1], dzjp1 = hnn[iz], dzjp2 = hnn[iz + 1];
      const R su = dzjm1 + dzj, sl = dzjp2 + dzjp1;
      const intdiv::Divisor ds = intdiv::prepare(dzj + dzjp1), du = intdiv::prepare(bits64::twice(dzj) + dzjp1),
                            dl = intdiv::prepare(bits64::twice(dzjp1) + dzj);
      const R gh = intdiv::divide(bits64::twice(dzjp1) * dzj, ds) * (intdiv::divide(su, du) - intdiv::divide(sl, dl));
      const R gi = intdiv::divide(dzj * su, du), gj = intdiv::divide(dzjp1 * sl, dl);
      const R gk = intdiv::divide(dzj, ds), gl = fdiv(R(1), su + dzjp1 + dzjp2);
#pragma unroll
      for (int i = 0; i < KC; ++i) {
        const R T0 = T[i * LW + iz - 1], d = T[i * LW + iz] - T0;
        e[i] = (T0 + gk * d) + gl * (gh * d - gi * tv[i * LW + iz] + gj * tv[i * LW + iz - 1]);
      }
    } else {
#pragma unroll
      for (int i = 0; i < KC; ++i) e[i] = (z < nzmin || z > nzmax) ? R(0) : ppm_tv_end(T + i * LW, g.W, z, nzmin, nzmax);
    }
    __syncwarp();
    if (iz < nl) {
#pragma unroll
      for (int i = 0; i < KC; ++i) tv[i * LW + iz] = e[i];
    }
  }
  __syncwarp();
  for (int iz = lane; iz < nl; iz += kWarp) {
    const int z = iz + 1;
    R f0[KC];
#pragma unroll
    for (int i = 0; i < KC; ++i) f0[i] = fold ? fold[i * LW + iz] : R(0);
    if (z < nzmin || z > nzmax) {
#pragma unroll
      for (int i = 0; i < KC; ++i) out[i * LW + iz] = f0[i];
      continue;
    }
    if (z == nzmin) {
#pragma unroll
      for (int i = 0; i < KC; ++i)
        out[i * LW + iz] = -((tv[i * LW + nzmin - 1] * g.W[nzmin - 1]) * g.area[nzmin - 1]) - f0[i];
      continue;
    }
    const R W = g.W[z - 1];
    if (z < nzmax && W != R(0)) {
      const bool up = W > R(0);
      const int L = up ? z : z - 1;  // the layer whose parabola crosses the interface
      const R x = ppm_x(W, dt, g.hn[L - 1], up);
      const R hx = bits64::half(x), cx = R(1) - R(2.0 / 3.0) * x;
#pragma unroll
      for (int i = 0; i < KC; ++i)
        out[i * LW + iz] =
            ppm_layer_x(tv[i * LW + L - 1], tv[i * LW + L], T[i * LW + L - 1], hx, cx, up, g.area[z - 1], W) - f0[i];
    } else {
#pragma unroll
      for (int i = 0; i < KC; ++i) out[i * LW + iz] = R(0) - f0[i];
    }
  }
  __syncwarp();
}

// ---------------------------------------------------------------------------
// Node-column kernels. One warp per node, two layers per lane; tracers are
// processed KC at a time. The node's incident edges (ascending edge index,
// the reference's scatter order) and its FCT cluster are staged once in
// shared memory; gathers run edge-outer, tracer-inner, so every edge's
// metadata is read once and the loads of all KC tracers are in flight
// together. Per-(tracer, layer) summation order is the reference's.
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
__host__ __device__ constexpr int lo_slices(int KC) { return 7 + 4 * KC; }
__host__ __device__ constexpr int ratio_slices(int KC) { return 3 * KC; }
__host__ __device__ constexpr int upd_slices(int KC) { return 3 * KC; }
__host__ __device__ constexpr int nofct_slices(int KC) { return 7 + 3 * KC; }
constexpr int kClBytes = kMaxCl * 2 * (int)sizeof(int);

// ---------------------------------------------------------------------------
// FCT stage 1: low-order solution fct_LO (lib/oce_adv_tra_driver.F90:91-235)
// and the vertical antidiffusive flux HO(T_AB, w) - LO(T, w_e). The low-order
// horizontal edge fluxes are formed here from T and the edge volume fluxes,
// with the expression adv_tra_hor_upw1 uses (lib/oce_adv_tra_hor.F90:218-220).
// ---------------------------------------------------------------------------
template <typename R, int VER, int KC>
__global__ void __launch_bounds__(128, (sizeof(R) == 4 ? 8 : 4)) k_fct_lo(DMesh m, StepPtrs<R> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & (kWarp - 1), wib = threadIdx.x / kWarp;
  const int vi = blockIdx.x * (blockDim.x / kWarp) + wib;
  if (vi >= m.N) return;
  const int n = visit_node(m, vi);
  const GeoPtrs<R>& g = GeoSel<R>::get(m);
  const size_t LZ = m.LZ, LW = m.LW;
  const int nl = m.nl, nz = m.nz;
  unsigned char* base = smem_raw + (size_t)wib * warp_smem<R>(lo_slices(KC), m.LW, 0);
  R* sl = reinterpret_cast<R*>(base);
  R *sW = sl, *sWE = sl + LW, *sA = sl + 2 * LW, *sHn = sl + 3 * LW, *sHnn = sl + 4 * LW, *sX = sl + 5 * LW;
  R* sZ = sl + 6 * LW;
  R* sT = sl + 7 * LW;                 // KC columns
  R* sTA = sT + (size_t)KC * LW;       // KC columns (T_AB when it is a separate field)
  R* sFv = sTA + (size_t)KC * LW;      // KC columns of vertical fluxes
  R* sTv = sFv + (size_t)KC * LW;      // KC columns of PPM edge values
  const NbrList nb = stage_nbrs(m, n, reinterpret_cast<Nbr*>(base + lo_slices(KC) * LW * sizeof(R)), lane);
  stage(sW, a.w + n * LW, nl, lane);
  stage(sWE, a.we + n * LW, nl, lane);
  stage(sA, g.area + n * LW, nl, lane);
  if (VER == 3) {
    stage(sHn, g.hnode + n * LZ, nz, lane);
    stage(sHnn, g.hnode_new + n * LZ, nz, lane);
  }
  if (VER == 1) {
    stage(sZ, g.Z3 + n * LZ, nz, lane);
    stage(sX, g.zbar3 + n * LW, nl, lane);
  }
  const int nzmin = m.ulev[n], nzmax = m.nlev[n];
  const bool ta_sep = a.TA != a.T;
  const R dt = a.dt;
  for (int t0 = 0; t0 < a.K; t0 += KC) {
#pragma unroll
    for (int i = 0; i < KC; ++i) {
      stage(sT + i * LW, a.T + (t0 + i) * a.sT + n * LZ, nz, lane);
      if (ta_sep) stage(sTA + i * LW, a.TA + (t0 + i) * a.sTA + n * LZ, nz, lane);
    }
    __syncwarp();
    // LO vertical flux: adv_tra_ver_upw1(we, ttf) with init zero.
    for (int i = 0; i < KC; ++i) {
      Col<R> clo{sT + i * LW, sWE, sA, sHn, sHnn, sZ, sX, nullptr};
      column_ver_flux<R, 0>(clo, nullptr, sFv + i * LW, nl, nzmin, nzmax, R(1), dt, lane);
    }
    for (int p = lane; 2 * p < m.LZ; p += kWarp) {
      const int k0 = 2 * p, z0 = k0 + 1, z1 = k0 + 2;
      R acc0[KC], acc1[KC];
#pragma unroll
      for (int i = 0; i < KC; ++i) acc0[i] = acc1[i] = R(0);
#pragma unroll 2
      for (int j = 0; j < nb.deg; ++j) {
        const Nbr q = nb.get(m, j);
        const bool a0 = z0 >= q.lo && z0 <= q.hi, a1 = z1 >= q.lo && z1 <= q.hi;
        const vec2<R> vv = ld2(a.vf + (size_t)q.e * LZ + k0);
#pragma unroll
        for (int i = 0; i < KC; ++i) {
          const vec2<R> to = ld2(a.T + (t0 + i) * a.sT + (size_t)q.other * LZ + k0);
          const R tn0 = sT[i * LW + k0], tn1 = sT[i * LW + k0 + 1];
          if (q.role) {  // this node is the edge's second node
            if (a0) acc0[i] = acc0[i] + bits64::upwind(vv.x, to.x, tn0);
            if (a1) acc1[i] = acc1[i] + bits64::upwind(vv.y, to.y, tn1);
          } else {
            if (a0) acc0[i] = acc0[i] - bits64::upwind(vv.x, tn0, to.x);
            if (a1) acc1[i] = acc1[i] - bits64::upwind(vv.y, tn1, to.y);
          }
        }
      }
      const vec2<R> hn = ld2(g.hnode + n * LZ + k0), hnn = ld2(g.hnode_new + n * LZ + k0);
      const vec2<R> av = ld2(g.areasvol + n * LZ + k0);
      const bool w0 = z0 >= nzmin && z0 <= nzmax - 1, w1 = z1 >= nzmin && z1 <= nzmax - 1;
      // fast form: dt / areasvol and 1 / hnode_new of the two layers, once
      const vec2<R> rd{rdt_vol(dt, av.x), rdt_vol(dt, av.y)};
      const vec2<R> rh{FGB_FAST64 ? fdiv(R(1), hnn.x) : R(0), FGB_FAST64 ? fdiv(R(1), hnn.y) : R(0)};
      const LayerDivisor vd0(av.x), vd1(av.y), hd0(hnn.x), hd1(hnn.y);  // exact form only
#pragma unroll
      for (int i = 0; i < KC; ++i) {
        const R* Ti = sT + i * LW;
        const R* Fi = sFv + i * LW;
        R l0 = acc0[i], l1 = acc1[i];
        if constexpr (FGB_FAST64) {
          if (w0) l0 = (Ti[k0] * hn.x + (acc0[i] + (Fi[k0] - Fi[k0 + 1])) * rd.x) * rh.x;
          if (w1) l1 = (Ti[k0 + 1] * hn.y + (acc1[i] + (Fi[k0 + 1] - Fi[k0 + 2])) * rd.y) * rh.y;
        } else {
          if (w0) {
            const R x = dt_per_vol(acc0[i] + (Fi[k0] - Fi[k0 + 1]), dt, vd0, R(0));
            l0 = intdiv::divide(Ti[k0] * hn.x + x, hd0.d);
          }
          if (w1) {
            const R x = dt_per_vol(acc1[i] + (Fi[k0 + 1] - Fi[k0 + 2]), dt, vd1, R(0));
            l1 = intdiv::divide(Ti[k0 + 1] * hn.y + x, hd1.d);
          }
        }
        st2(a.lo + (t0 + i) * a.sN + n * LZ + k0, l0, l1);
      }
    }
    __syncwarp();  // every lane has read the LO fluxes before they are overwritten
    if (a.wi) {
      // w_split: the antidiffusive flux takes the upwind flux of the full w
      // (lib/oce_adv_tra_driver.F90:221-231)
      for (int i = 0; i < KC; ++i) {
        Col<R> clw{sT + i * LW, sW, sA, sHn, sHnn, sZ, sX, nullptr};
        column_ver_flux<R, 0>(clw, nullptr, sFv + i * LW, nl, nzmin, nzmax, R(1), dt, lane);
      }
    }
    // HO vertical flux on T_AB with w; adf_v = HO - LO ("X - flux").
    if constexpr (VER == 3) {
      const Col<R> g{nullptr, sW, sA, sHn, sHnn, sZ, sX, nullptr};
      column_ppm_multi<R, KC>(g, ta_sep ? sTA : sT, sTv, sFv, sFv, (int)LW, nl, nzmin, nzmax, dt, lane);
    }
    if constexpr (VER == 1) {
      qr4c_slopes<R, KC>(ta_sep ? sTA : sT, sZ, sTv, (int)LW, nzmin, nzmax, lane);
      __syncwarp();
    }
    for (int i = 0; i < KC; ++i) {
      if constexpr (VER != 3) {
        const Col<R> cho{(ta_sep ? sTA : sT) + i * LW, sW, sA, sHn, sHnn, sZ, sX, sTv + i * LW};
        column_ver_flux<R, VER>(cho, sFv + i * LW, sFv + i * LW, nl, nzmin, nzmax, a.pv, dt, lane);
      }
      R* __restrict__ adfv = a.adfv + (t0 + i) * a.sW + n * LW;
      for (int iz = lane; iz < (int)LW; iz += kWarp) adfv[iz] = iz < nl ? sFv[i * LW + iz] : R(0);
    }
    __syncwarp();
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
template <typename R, int KC>
__global__ void __launch_bounds__(128, (sizeof(R) == 4 ? 8 : 4)) k_fct_ratio(DMesh m, StepPtrs<R> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & (kWarp - 1), wib = threadIdx.x / kWarp;
  const int vi = blockIdx.x * (blockDim.x / kWarp) + wib;
  if (vi >= m.N) return;
  const int n = visit_node(m, vi);
  const GeoPtrs<R>& g = GeoSel<R>::get(m);
  const size_t LZ = m.LZ, LW = m.LW;
  unsigned char* base = smem_raw + (size_t)wib * warp_smem<R>(ratio_slices(KC), m.LW, kClBytes);
  R* smax = reinterpret_cast<R*>(base);
  R* smin = smax + (size_t)KC * LW;
  R* sadv = smin + (size_t)KC * LW;
  const NbrList nb = stage_nbrs(m, n, reinterpret_cast<Nbr*>(base + ratio_slices(KC) * LW * sizeof(R)), lane);
  int* scl = reinterpret_cast<int*>(base + ratio_slices(KC) * LW * sizeof(R) + kMaxDeg * sizeof(Nbr));
  const int c0 = m.cl_ptr[n], ncl = m.cl_ptr[n + 1] - c0, minlev = m.cl_minlev[n];
  const bool cl_staged = ncl <= kMaxCl;
  if (cl_staged)
    for (int j = lane; j < ncl; j += kWarp) {
      scl[2 * j] = m.cl_node[c0 + j];
      scl[2 * j + 1] = m.cl_lev[c0 + j];
    }
  const int nzmin = m.ulev[n], nzmax = m.nlev[n];
  const R big = R(1e3), dt = a.dt;
  const R inf = R(INFINITY);
  for (int t0 = 0; t0 < a.K; t0 += KC) {
#pragma unroll
    for (int i = 0; i < KC; ++i) stage(sadv + i * LW, a.adfv + (t0 + i) * a.sW + n * LW, m.nl, lane);
    __syncwarp();
    for (int p = lane; 2 * p < m.LZ; p += kWarp) {
      const int k0 = 2 * p, z0 = k0 + 1, z1 = k0 + 2;
      // AUX = -/+1e3 of elements without the layer joins the bound (lib/oce_adv_tra_fct.F90:139-145)
      const R mx0i = z0 > minlev ? -big : -inf, mx1i = z1 > minlev ? -big : -inf;
      // the bounds as integer keys (bits64::key), which order as the values do
      long long mx0[KC], mx1[KC], mn0[KC], mn1[KC];
#pragma unroll
      for (int i = 0; i < KC; ++i) {
        mx0[i] = bits64::key(mx0i);
        mx1[i] = bits64::key(mx1i);
        mn0[i] = bits64::key(-mx0i);
        mn1[i] = bits64::key(-mx1i);
      }
#pragma unroll 2
      for (int j = 0; j < ncl; ++j) {
        const int node = cl_staged ? scl[2 * j] : m.cl_node[c0 + j];
        const int lev = cl_staged ? scl[2 * j + 1] : m.cl_lev[c0 + j];
        const bool a0 = z0 <= lev, a1 = z1 <= lev;
#pragma unroll
        for (int i = 0; i < KC; ++i) {
          const size_t v = (size_t)node * LZ + k0;
          const vec2<R> lv = ld2(a.lo + (t0 + i) * a.sN + v), tv = ld2(a.T + (t0 + i) * a.sT + v);
          if (a0) join_bounds(lv.x, tv.x, mx0[i], mn0[i]);
          if (a1) join_bounds(lv.y, tv.y, mx1[i], mn1[i]);
        }
      }
      // A NaN is the largest or the smallest key of all, so it is still there:
      // the column's bounds again with the floating-point comparisons, whose
      // outcome with NaNs depends on the order.
      bool nan = false;
#pragma unroll
      for (int i = 0; i < KC; ++i)
        nan |= max(mx0[i], mx1[i]) > bits64::kKeyInf || min(mn0[i], mn1[i]) < -bits64::kKeyInf - 1;
      if (nan) {
        for (int i = 0; i < KC; ++i) {
          R x0 = mx0i, x1 = mx1i, y0 = -mx0i, y1 = -mx1i;
          for (int j = 0; j < ncl; ++j) {
            const int lev = m.cl_lev[c0 + j];
            const size_t v = (size_t)m.cl_node[c0 + j] * LZ + k0;
            const vec2<R> lv = ld2(a.lo + (t0 + i) * a.sN + v), tv = ld2(a.T + (t0 + i) * a.sT + v);
            if (z0 <= lev) {
              x0 = rmax(x0, rmax(lv.x, tv.x));
              y0 = rmin(y0, rmin(lv.x, tv.x));
            }
            if (z1 <= lev) {
              x1 = rmax(x1, rmax(lv.y, tv.y));
              y1 = rmin(y1, rmin(lv.y, tv.y));
            }
          }
          smax[i * LW + k0] = x0;
          smax[i * LW + k0 + 1] = x1;
          smin[i * LW + k0] = y0;
          smin[i * LW + k0 + 1] = y1;
        }
        continue;
      }
#pragma unroll
      for (int i = 0; i < KC; ++i) {
        smax[i * LW + k0] = bits64::unkey(mx0[i]);
        smax[i * LW + k0 + 1] = bits64::unkey(mx1[i]);
        smin[i * LW + k0] = bits64::unkey(mn0[i]);
        smin[i * LW + k0 + 1] = bits64::unkey(mn1[i]);
      }
    }
    __syncwarp();
    for (int p = lane; 2 * p < m.LZ; p += kWarp) {
      const int k0 = 2 * p;
      R pl0[KC], pl1[KC], mi0[KC], mi1[KC];
#pragma unroll
      for (int i = 0; i < KC; ++i) {
        const R* ad = sadv + i * LW;
        first_parts(ad[k0], ad[k0 + 1], pl0[i], mi0[i]);
        first_parts(ad[k0 + 1], ad[k0 + 2], pl1[i], mi1[i]);
      }
      const int z0 = k0 + 1, z1 = k0 + 2;
#pragma unroll 2
      for (int j = 0; j < nb.deg; ++j) {
        const Nbr q = nb.get(m, j);
        const bool a0 = z0 >= q.lo && z0 <= q.hi, a1 = z1 >= q.lo && z1 <= q.hi;
#pragma unroll
        for (int i = 0; i < KC; ++i) {
          const vec2<R> f = ld2(a.adfh + (t0 + i) * a.sE + (size_t)q.e * LZ + k0);
          if (a0) add_part(bits64::negate_if(f.x, q.role), pl0[i], mi0[i]);
          if (a1) add_part(bits64::negate_if(f.y, q.role), pl1[i], mi1[i]);
        }
      }
      const vec2<R> av = ld2(g.areasvol + n * LZ + k0);
      const LayerDivisor dv[2] = {LayerDivisor(av.x), LayerDivisor(av.y)};
#pragma unroll
      for (int i = 0; i < KC; ++i) {
        const R* mxs = smax + i * LW;
        const R* mns = smin + i * LW;
        const vec2<R> lo = ld2(a.lo + (t0 + i) * a.sN + n * LZ + k0);
        R out_p[2] = {R(0), R(0)}, out_m[2] = {R(0), R(0)};
#pragma unroll
        for (int l = 0; l < 2; ++l) {
          const int k = k0 + l, z = k + 1;
          if (z < nzmin || z > nzmax - 1) continue;
          const R lov = l ? lo.y : lo.x;
          R bmax, bmin;
          if (z == nzmax - 1 || z == nzmin) {
            bmax = mxs[k] - lov;
            bmin = mns[k] - lov;
          } else {
            bmax = rmax(rmax(mxs[k - 1], mxs[k]), mxs[k + 1]) - lov;
            bmin = rmin(rmin(mns[k - 1], mns[k]), mns[k + 1]) - lov;
          }
          const R avk = l ? av.y : av.x;
          const R rdk = rdt_vol(dt, avk);
          R pl = l ? pl1[i] : pl0[i], mi = l ? mi1[i] : mi0[i];
          spread_nan(pl, mi);
          R flux = dt_per_vol(pl, dt, dv[l], rdk) + R(1e-16);
          out_p[l] = rmin(R(1), fdiv(bmax, flux));
          flux = dt_per_vol(mi, dt, dv[l], rdk) - R(1e-16);
          out_m[l] = rmin(R(1), fdiv(bmin, flux));
        }
        st4(a.rpm + 2 * ((t0 + i) * a.sN + n * LZ + k0), out_p[0], out_m[0], out_p[1], out_m[1]);
      }
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// FCT stage 3: limiting b3 (lib/oce_adv_tra_fct.F90:396-471), flux divergence
// (oce_tra_adv_flux2dtracer with use_lo, lib/oce_adv_tra_driver.F90:298-450)
// and the caller's tendency update (src/fesom_analytic.F90:419-437 or, with a
// persistent del_ttf, lib/tracer_c_interface.F90:194-214).
// ---------------------------------------------------------------------------
template <typename R, int KC>
__global__ void __launch_bounds__(128, (sizeof(R) == 4 ? 8 : 4)) k_fct_update(DMesh m, StepPtrs<R> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & (kWarp - 1), wib = threadIdx.x / kWarp;
  const int vi = blockIdx.x * (blockDim.x / kWarp) + wib;
  if (vi >= m.N) return;
  const int n = visit_node(m, vi);
  const GeoPtrs<R>& g = GeoSel<R>::get(m);
  const size_t LZ = m.LZ, LW = m.LW;
  const int nz = m.nz, nl = m.nl;
  unsigned char* base = smem_raw + (size_t)wib * warp_smem<R>(upd_slices(KC), m.LW, 0);
  R* sLv = reinterpret_cast<R*>(base);
  R* sRp = sLv + (size_t)KC * LW;
  R* sRm = sRp + (size_t)KC * LW;
  const NbrList nb = stage_nbrs(m, n, reinterpret_cast<Nbr*>(base + upd_slices(KC) * LW * sizeof(R)), lane);
  const int nzmin = m.ulev[n], nzmax = m.nlev[n];
  const R dt = a.dt;
  for (int t0 = 0; t0 < a.K; t0 += KC) {
#pragma unroll
    for (int i = 0; i < KC; ++i) {
      const R* src = a.rpm + 2 * ((t0 + i) * a.sN + n * LZ);
      for (int k = lane; k < nz; k += kWarp) {
        sRp[i * LW + k] = src[2 * k];
        sRm[i * LW + k] = src[2 * k + 1];
      }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < KC; ++i) {
      const R* __restrict__ adfv = a.adfv + (t0 + i) * a.sW + n * LW;
      const R* Rp = sRp + i * LW;
      const R* Rm = sRm + i * LW;
      for (int iz = lane; iz < nl; iz += kWarp) {
        const int z = iz + 1;
        R f = adfv[iz];
        const bool pos = bits64::sign_clear(f);
        if (z == nzmin) f = (pos ? Rp[iz] : Rm[iz]) * f;
        else if (z > nzmin && z <= nzmax - 1)
          f = rmin(pos ? Rm[iz - 1] : Rp[iz - 1], pos ? Rp[iz] : Rm[iz]) * f;
        sLv[i * LW + iz] = f;
      }
    }
    __syncwarp();
    for (int p = lane; 2 * p < m.LZ; p += kWarp) {
      const int k0 = 2 * p, z0 = k0 + 1, z1 = k0 + 2;
      const vec2<R> av = ld2(g.areasvol + n * LZ + k0);
      const vec2<R> rd{rdt_vol(dt, av.x), rdt_vol(dt, av.y)};  // fast form only
      const LayerDivisor vd0(av.x), vd1(av.y);                   // exact form only
      R dh0[KC], dh1[KC];
#pragma unroll
      for (int i = 0; i < KC; ++i) dh0[i] = dh1[i] = R(0);
#pragma unroll 2
      for (int j = 0; j < nb.deg; ++j) {
        const Nbr q = nb.get(m, j);
        const bool a0 = z0 >= q.lo && z0 <= q.hi, a1 = z1 >= q.lo && z1 <= q.hi;
        const size_t o = (size_t)q.other * LZ + k0;
#pragma unroll
        for (int i = 0; i < KC; ++i) {
          const vec2<R> f = ld2(a.adfh + (t0 + i) * a.sE + (size_t)q.e * LZ + k0);
          const Q4<R> ro = ld4(a.rpm + 2 * ((t0 + i) * a.sN + o));
          const vec2<R> rpo{ro.a, ro.c}, rmo{ro.b, ro.d};
          const R rpn0 = sRp[i * LW + k0], rpn1 = sRp[i * LW + k0 + 1];
          const R rmn0 = sRm[i * LW + k0], rmn1 = sRm[i * LW + k0 + 1];
          // this node's factor and the other one's, for the flux's sign; the reference takes the
          // first node's against the second node's
          if (a0) {
            const bool up = bits64::sign_clear(f.x) != (bool)q.role;
            const R own = up ? rpn0 : rmn0, oth = up ? rmo.x : rpo.x;
            const R x = dt_per_vol((q.role ? rmin(oth, own) : rmin(own, oth)) * f.x, dt, vd0, rd.x);
            dh0[i] = q.role ? dh0[i] - x : dh0[i] + x;
          }
          if (a1) {
            const bool up = bits64::sign_clear(f.y) != (bool)q.role;
            const R own = up ? rpn1 : rmn1, oth = up ? rmo.y : rpo.y;
            const R x = dt_per_vol((q.role ? rmin(oth, own) : rmin(own, oth)) * f.y, dt, vd1, rd.y);
            dh1[i] = q.role ? dh1[i] - x : dh1[i] + x;
          }
        }
      }
      const vec2<R> hn = ld2(g.hnode + n * LZ + k0), hnn = ld2(g.hnode_new + n * LZ + k0);
      const bool w0 = z0 >= nzmin && z0 <= nzmax - 1, w1 = z1 >= nzmin && z1 <= nzmax - 1;
      const vec2<R> rh{FGB_FAST64 ? fdiv(R(1), hnn.x) : R(0), FGB_FAST64 ? fdiv(R(1), hnn.y) : R(0)};
      const LayerDivisor hd0(hnn.x), hd1(hnn.y);
#pragma unroll
      for (int i = 0; i < KC; ++i) {
        R* __restrict__ T = a.T + (t0 + i) * a.sT + n * LZ + k0;
        const vec2<R> Tn = ld2(T);
        const vec2<R> lo = ld2(a.lo + (t0 + i) * a.sN + n * LZ + k0);
        const R* Lv = sLv + i * LW;
        R* del = a.del ? a.del + (t0 + i) * a.sN + n * LZ + k0 : nullptr;
        const vec2<R> d0 = del ? ld2(del) : vec2<R>{R(0), R(0)};
        R dv0 = lo.x * hnn.x - Tn.x * hn.x;  // the reference's (0 - T hnode) + LO hnode_new
        dv0 = dv0 + dt_per_vol(Lv[k0] - Lv[k0 + 1], dt, vd0, rd.x);
        R dv1 = lo.y * hnn.y - Tn.y * hn.y;
        dv1 = dv1 + dt_per_vol(Lv[k0 + 1] - Lv[k0 + 2], dt, vd1, rd.y);
        const R e0 = (del ? d0.x + dh0[i] : dh0[i]) + dv0, e1 = (del ? d0.y + dh1[i] : dh1[i]) + dv1;
        R n0 = Tn.x, n1v = Tn.y;
        if constexpr (FGB_FAST64) {
          if (w0) n0 = Tn.x + e0 * rh.x;
          if (w1) n1v = Tn.y + e1 * rh.y;
        } else {
          if (w0) n0 = Tn.x + intdiv::divide(e0, hd0.d);
          if (w1) n1v = Tn.y + intdiv::divide(e1, hd1.d);
        }
        st2(T, n0, n1v);
        if (del) st2(del, w0 ? e0 : d0.x, w1 ? e1 : d0.y);
        if (a.TAout) {
          R* ta = a.TAout + (t0 + i) * a.sTA + n * LZ + k0;
          if (a.ab2) st2(ta, a.ab_old * Tn.x + a.ab_new * n0, a.ab_old * Tn.y + a.ab_new * n1v);
          else st2(ta, n0, n1v);
        }
      }
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// Without a limiter: vertical HO flux on T_AB with w_e, flux divergence
// (oce_tra_adv_flux2dtracer) and the tendency update in one pass.
// ---------------------------------------------------------------------------
template <typename R, int VER, int KC>
__global__ void __launch_bounds__(128, (sizeof(R) == 4 ? 8 : 4)) k_nofct_update(DMesh m, StepPtrs<R> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & (kWarp - 1), wib = threadIdx.x / kWarp;
  const int vi = blockIdx.x * (blockDim.x / kWarp) + wib;
  if (vi >= m.N) return;
  const int n = visit_node(m, vi);
  const GeoPtrs<R>& g = GeoSel<R>::get(m);
  const size_t LZ = m.LZ, LW = m.LW;
  const int nl = m.nl, nz = m.nz;
  unsigned char* base = smem_raw + (size_t)wib * warp_smem<R>(nofct_slices(KC), m.LW, 0);
  R* sl = reinterpret_cast<R*>(base);
  R *sW = sl, *sA = sl + LW, *sHn = sl + 2 * LW, *sHnn = sl + 3 * LW, *sX = sl + 4 * LW, *sZ = sl + 5 * LW;
  R* sTA = sl + 7 * LW;              // KC columns
  R* sF = sTA + (size_t)KC * LW;     // KC columns
  R* sTv = sF + (size_t)KC * LW;     // KC columns
  const NbrList nb = stage_nbrs(m, n, reinterpret_cast<Nbr*>(base + nofct_slices(KC) * LW * sizeof(R)), lane);
  stage(sW, a.we + n * LW, nl, lane);
  stage(sA, g.area + n * LW, nl, lane);
  if (VER == 3) {
    stage(sHn, g.hnode + n * LZ, nz, lane);
    stage(sHnn, g.hnode_new + n * LZ, nz, lane);
  }
  if (VER == 1) {
    stage(sZ, g.Z3 + n * LZ, nz, lane);
    stage(sX, g.zbar3 + n * LW, nl, lane);
  }
  const int nzmin = m.ulev[n], nzmax = m.nlev[n];
  const R dt = a.dt;
  for (int t0 = 0; t0 < a.K; t0 += KC) {
#pragma unroll
    for (int i = 0; i < KC; ++i) stage(sTA + i * LW, a.TA + (t0 + i) * a.sTA + n * LZ, nz, lane);
    __syncwarp();
    if constexpr (VER == 3) {
      const Col<R> gc{nullptr, sW, sA, sHn, sHnn, sZ, sX, nullptr};
      column_ppm_multi<R, KC>(gc, sTA, sTv, nullptr, sF, (int)LW, nl, nzmin, nzmax, dt, lane);
    } else {
      if constexpr (VER == 1) {
        qr4c_slopes<R, KC>(sTA, sZ, sTv, (int)LW, nzmin, nzmax, lane);
        __syncwarp();
      }
      for (int i = 0; i < KC; ++i) {
        const Col<R> c{sTA + i * LW, sW, sA, sHn, sHnn, sZ, sX, sTv + i * LW};
        column_ver_flux<R, VER>(c, nullptr, sF + i * LW, nl, nzmin, nzmax, a.pv, dt, lane);
      }
    }
    for (int p = lane; 2 * p < m.LZ; p += kWarp) {
      const int k0 = 2 * p, z0 = k0 + 1, z1 = k0 + 2;
      const vec2<R> av = ld2(g.areasvol + n * LZ + k0);
      const vec2<R> rd{rdt_vol(dt, av.x), rdt_vol(dt, av.y)};  // fast form only
      const LayerDivisor vd0(av.x), vd1(av.y);                   // exact form only
      R dh0[KC], dh1[KC];
#pragma unroll
      for (int i = 0; i < KC; ++i) dh0[i] = dh1[i] = R(0);
#pragma unroll 2
      for (int j = 0; j < nb.deg; ++j) {
        const Nbr q = nb.get(m, j);
        const bool a0 = z0 >= q.lo && z0 <= q.hi, a1 = z1 >= q.lo && z1 <= q.hi;
#pragma unroll
        for (int i = 0; i < KC; ++i) {
          const vec2<R> f = ld2(a.adfh + (t0 + i) * a.sE + (size_t)q.e * LZ + k0);
          if (q.role) {
            if (a0) dh0[i] = dh0[i] - dt_per_vol(f.x, dt, vd0, rd.x);
            if (a1) dh1[i] = dh1[i] - dt_per_vol(f.y, dt, vd1, rd.y);
          } else {
            if (a0) dh0[i] = dh0[i] + dt_per_vol(f.x, dt, vd0, rd.x);
            if (a1) dh1[i] = dh1[i] + dt_per_vol(f.y, dt, vd1, rd.y);
          }
        }
      }
      const vec2<R> hnn = ld2(g.hnode_new + n * LZ + k0);
      const bool w0 = z0 >= nzmin && z0 <= nzmax - 1, w1 = z1 >= nzmin && z1 <= nzmax - 1;
      const vec2<R> rh{FGB_FAST64 ? fdiv(R(1), hnn.x) : R(0), FGB_FAST64 ? fdiv(R(1), hnn.y) : R(0)};
      const LayerDivisor hd0(hnn.x), hd1(hnn.y);
#pragma unroll
      for (int i = 0; i < KC; ++i) {
        const R* F = sF + i * LW;
        R* __restrict__ T = a.T + (t0 + i) * a.sT + n * LZ + k0;
        const vec2<R> Tn = ld2(T);
        R* del = a.del ? a.del + (t0 + i) * a.sN + n * LZ + k0 : nullptr;
        const vec2<R> d0 = del ? ld2(del) : vec2<R>{R(0), R(0)};
        const R dv0 = dt_per_vol(F[k0] - F[k0 + 1], dt, vd0, rd.x);
        const R dv1 = dt_per_vol(F[k0 + 1] - F[k0 + 2], dt, vd1, rd.y);
        const R e0 = (del ? d0.x + dh0[i] : dh0[i]) + dv0, e1 = (del ? d0.y + dh1[i] : dh1[i]) + dv1;
        R n0 = Tn.x, n1v = Tn.y;
        if constexpr (FGB_FAST64) {
          if (w0) n0 = Tn.x + e0 * rh.x;
          if (w1) n1v = Tn.y + e1 * rh.y;
        } else {
          if (w0) n0 = Tn.x + intdiv::divide(e0, hd0.d);
          if (w1) n1v = Tn.y + intdiv::divide(e1, hd1.d);
        }
        st2(T, n0, n1v);
        if (del) st2(del, w0 ? e0 : d0.x, w1 ? e1 : d0.y);
        if (a.TAout) {
          R* ta = a.TAout + (t0 + i) * a.sTA + n * LZ + k0;
          if (a.ab2) st2(ta, a.ab_old * Tn.x + a.ab_new * n0, a.ab_old * Tn.y + a.ab_new * n1v);
          else st2(ta, n0, n1v);
        }
      }
    }
    __syncwarp();
  }
}

}  // inline namespace
}  // namespace fgb
