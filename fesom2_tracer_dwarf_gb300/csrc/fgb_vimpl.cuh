// Implicit vertical advection of the w_split option (adv_tra_vert_impl,
// lib/oce_adv_tra_ver.F90:90-244), applied in place to the FCT low-order
// solution between the LO and ratio kernels (lib/oce_adv_tra_driver.F90:
// 221-228). Per node column, the upwind scheme with the implicit vertical
// velocity wi is a tridiagonal system over the layers nzmin..nzmax-1, solved
// by the Thomas algorithm in the reference's operation order.
//
// One lane per (node, tracer): the sweeps are serial over the layers, so a warp
// that gives each lane a system of its own issues a thirty-second of the FP64
// instructions of one that solves its node's systems on a lane or two (131x117
// columns of 8..37 layers, 3 tracers: LO stage 1.77 -> 0.41 ms). Each lane forms its coefficients as
// it goes and keeps its ratios cp and solution terms tp in shared memory for
// the way back. FP64 form: bit-identical to the reference's arithmetic
// (including the solve for the increment); boundary rows take zero
// coefficients in the general expressions, which leaves the values the
// reference's special rows have. (The FP32 form has its own kernels.)
#pragma once
#include <cuda_runtime.h>

#include "fgb_device.hpp"
#include "fgb_kernels.cuh"

namespace fgb {
#if FGB_FAST64
inline namespace fast64 {
#else
inline namespace exact64 {
#endif

// Shared memory of a one-warp block: (tp, cp) of every layer and lane.
inline size_t vimpl_smem(int LZ) { return (size_t)LZ * kWarp * sizeof(double2); }

template <typename R>
__global__ void __launch_bounds__(kWarp) k_vert_impl(DMesh m, R* __restrict__ lo, const R* __restrict__ wi, int K,
                                                    long long sN, R dt) {
  extern __shared__ __align__(16) unsigned char vimpl_smem_raw[];
  double2* s = reinterpret_cast<double2*>(vimpl_smem_raw) + threadIdx.x;  // [layer][lane]
  const long long it = (long long)blockIdx.x * kWarp + threadIdx.x;
  if (it >= (long long)m.N * K) return;
  const int vi = (int)(it / K), t = (int)(it - (long long)vi * K);
  const Column c(m, visit_node(m, vi));
  const GeoPtrs<R>& g = m.g64;
  const int k0 = c.k0, k1 = c.nzmax - 2;  // first and last layer (0-based)
  R* __restrict__ col = lo + t * sN + c.iz;
  const R* __restrict__ wn = wi + c.iw;
  const R* __restrict__ an = g.area + c.iw;
  R W1 = wn[k0], ar1 = an[k0], Tm = R(0), Tk = col[k0], cp = R(0), tp = R(0);
  for (int k = k0; k <= k1; ++k) {
    const R W0 = W1, ar0 = ar1, hnn = g.hnode_new[c.iz + k];
    const bool last = k == k1;
    W1 = last ? R(0) : wn[k + 1];
    ar1 = last ? ar0 : an[k + 1];
    const R Tp = last ? R(0) : col[k + 1];
    const intdiv::Divisor av = intdiv::prepare(g.areasvol[c.iz + k]);
    const R v0 = intdiv::divide(dt * ar0, av), v1 = intdiv::divide(dt * ar1, av);
    const R w0p = k == k0 ? W0 : rmax(W0, R(0)), w0m = rmin(W0, R(0));
    const R a = k == k0 ? R(0) : w0m * v0;
    const R cc = -(rmax(W1, R(0)) * v1);
    const R b = (hnn + w0p * v0) - rmin(W1, R(0)) * v1;
    const R r = -(a * Tm) - (b - hnn) * Tk - cc * Tp;
    const intdiv::Divisor mm = intdiv::prepare(b - cp * a);
    tp = intdiv::divide(r - tp * a, mm);
    cp = intdiv::divide(cc, mm);
    s[k * kWarp] = make_double2(tp, cp);
    Tm = Tk;
    Tk = Tp;
  }
  R x = tp;
  col[k1] = Tm + x;
  for (int k = k1 - 1; k >= k0; --k) {
    const double2 q = s[k * kWarp];
    x = q.x - q.y * x;
    col[k] = col[k] + x;
  }
}

// Checks of a w_split launch: columns of at least two layers (with one, the
// reference's right-hand side reads the layer above the column) and at most
// the layers that the interface has always taken (345; the kernel's shared
// memory would hold more). Returns nullptr or the reason.
inline const char* vert_impl_check(const DMesh& m) {
  if (m.min_layers < 2) return "w_split needs at least two layers in every column";
  if (672 * (m.LZ | 1) > 227 * 1024) return "w_split: too many layers for one block";
  return nullptr;
}

// Launches k_vert_impl over all nodes and tracers (after vert_impl_check).
template <typename R>
inline void launch_vert_impl(const DMesh& m, R* lo, const R* wi, int K, long long sN, R dt, cudaStream_t s) {
  const size_t smem = vimpl_smem(m.LZ);
  if (smem > 48 * 1024)
    cudaFuncSetAttribute(k_vert_impl<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const long long items = (long long)m.N * K;
  k_vert_impl<R><<<(unsigned)((items + kWarp - 1) / kWarp), kWarp, smem, s>>>(m, lo, wi, K, sN, dt);
}

}  // inline namespace
}  // namespace fgb
