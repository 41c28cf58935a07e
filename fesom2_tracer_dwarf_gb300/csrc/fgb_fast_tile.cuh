// FP32 edge fluxes, tiled (same fluxes as kf_hflux: lib/oce_adv_tra_hor.F90
// UPW1 :218-220, MUSCL :454-497, MFCT :748-790; FCT: high-order minus
// low-order).
//
// The edges' tracer reads are gathers of node rows (layers fastest): the two
// nodes of the edge and the other vertices of its up- and downwind triangles.
// Neighbouring edges of the visit order share most of these nodes, so the
// visit order is cut into tiles (at mesh upload) of at most kTileEdges edges
// touching at most kTileNodes distinct nodes, and one block per tile stages
// each distinct node row once per pass of kTileChunk layers in shared memory
// with asynchronous 16-byte copies, then computes all edges of the tile from
// there, one edge per warp at a time.
#pragma once
#include <cuda_runtime.h>

#include "fgb_fast.cuh"

namespace fgb {
namespace fast {

constexpr int kTileThreads = 128;
constexpr int kTileChunk = 32;  // layers per pass: lane l handles layer k0 + l of one edge

// 16-byte asynchronous copy global -> shared (cp.async, L2 only), and the
// wait for all of this thread's copies.
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// Shared memory: edge records, the start of each edge's six node rows in the
// staged rows (16 bits each: slot x kTileChunk; 12 bytes per edge, which keeps
// seven blocks of the largest tiles on an SM), the node ids, the TA rows
// (+ T rows when T_AB is separate under FCT) of the mesh's largest tile (maxn
// nodes) and the volume-flux rows of one pass.
__host__ __device__ constexpr size_t tile_smem_bytes(int KV, bool tsep, int maxn) {
  return (size_t)kTileEdges * sizeof(EdgeRec) + (size_t)kTileEdges * 12 + (size_t)kTileNodes * 4 +
         (size_t)(tsep ? 2 : 1) * maxn * kTileChunk * KV * 4 + (size_t)kTileEdges * kTileChunk * 4;
}
static_assert(kTileNodes * kTileChunk < 65536, "row starts are 16-bit");

// One layer's flux of an edge from the values at its nodes (T_AB: s1, s2; T: q1, q2) and the
// MUSCL/MFCT increments p1, p2 of its nodes (c1, c2: the nboundary_lay mask).
template <int HOR, bool FCT, int KV>
__device__ __forceinline__ V<KV> tile_flux(const V<KV>& s1, const V<KV>& s2, const V<KV>& q1, const V<KV>& q2,
                                           const V<KV>& p1, const V<KV>& p2, float v, float ph, float c1, float c2) {
  const float vp = v + fabsf(v), vm = v - fabsf(v);
  V<KV> h;
  if (HOR == 0) {
    h = muls(fmas(s2, vm, muls(s1, vp)), -0.5f);
  } else {
    const V<KV> tm1 = fmas(p1, c1, s1), tm2 = fmas(p2, -c2, s2);
    const V<KV> cho = fmas(tm2, vm, muls(tm1, vp));
    h = fmas(add(tm1, tm2), -((v * ph) * 0.5f), muls(cho, -(0.5f * (1.f - ph))));
  }
  return FCT ? fmas(fmas(q2, vm, muls(q1, vp)), 0.5f, h) : h;
}

template <int HOR, bool FCT, int KV>
__device__ __forceinline__ void hflux_tile(const DMesh& m, const FastPtrs& a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  EdgeRec* recs = reinterpret_cast<EdgeRec*>(smem_raw);
  // row starts of n1 | n2 and of the upwind triangle's two other vertices (rsA), of
  // the downwind triangle's two others (rsD)
  uint2* rsA = reinterpret_cast<uint2*>(smem_raw + kTileEdges * sizeof(EdgeRec));
  unsigned* rsD = reinterpret_cast<unsigned*>(rsA + kTileEdges);
  int* nodes = reinterpret_cast<int*>(rsD + kTileEdges);
  const bool ta_sep = a.TA != a.T;
  const bool tsep = FCT && ta_sep;
  V<KV>* rowsA = reinterpret_cast<V<KV>*>(nodes + kTileNodes);  // [node slot][layer of the pass]
  V<KV>* rowsT = tsep ? rowsA + m.tile_max_nodes * kTileChunk : rowsA;
  float* rowsV = reinterpret_cast<float*>(rowsA + (tsep ? 2 : 1) * m.tile_max_nodes * kTileChunk);  // [edge][layer]
  const int tid = threadIdx.x, lane = tid & (kW - 1), warp = tid / kW;
  const int t = blockIdx.x;
  const int p0 = m.tile_ptr[t], ne = m.tile_ptr[t + 1] - p0;
  const int q0 = m.tile_nptr[t], nn = m.tile_nptr[t + 1] - q0;
  __shared__ int s_hi;  // the deepest layer of the tile's edges
  if (tid == 0) s_hi = 0;
  __syncthreads();
  for (int i = tid; i < ne; i += kTileThreads) {
    fill_edge<HOR>(m, p0 + i, recs[i]);
    const uint2 sl = *reinterpret_cast<const uint2*>(m.tile_slots + 8 * (size_t)(p0 + i));
    auto two = [](unsigned a, unsigned b) { return (a * kTileChunk) | ((b * kTileChunk) << 16); };
    rsA[i] = make_uint2(two(sl.x & 0xff, (sl.x >> 8) & 0xff), two((sl.x >> 16) & 0xff, sl.x >> 24));
    rsD[i] = two(sl.y & 0xff, (sl.y >> 8) & 0xff);
    atomicMax(&s_hi, recs[i].hi);
  }
  for (int i = tid; i < nn; i += kTileThreads) nodes[i] = m.tile_nodes[q0 + i];
  const unsigned LZ = m.LZ;
  for (unsigned k0 = 0; k0 < LZ; k0 += kTileChunk) {
    const int rows = (int)min((unsigned)kTileChunk, LZ - k0);
    for (int gi = 0; gi < a.G; ++gi) {
      const float* __restrict__ TAg = ta_sep ? a.TA + gi * a.gTA : a.T + gi * a.gT;
      const float* __restrict__ Tg = a.T + gi * a.gT;
      float* __restrict__ out = a.adfh + gi * a.gE;
      __syncthreads();  // the previous pass has read the rows (first pass: records filled)
      if ((int)k0 >= s_hi) {
        // below every edge of the tile: the fluxes are zero (the node kernels read them)
        if (lane < rows)
          for (int j = warp; j < ne; j += kTileThreads / kW) st<KV>(out, (unsigned)recs[j].e * LZ + k0 + lane, splat<KV>(0.f));
        continue;
      }
      // Stage the pass with 16-byte asynchronous copies: a node's rows of the
      // pass are rows * KV floats from (node * LZ + k0) * KV, a multiple of 16
      // bytes from a 16-byte boundary (LZ, k0 and rows are multiples of 4).
      {
        // each thread copies the same 16-byte unit u of every (kTileThreads / upr)-th row
        constexpr int upr = kTileChunk * KV / 4;  // 16-byte units per staged node row
        static_assert(kTileThreads % upr == 0, "whole rows per round");
        const int used = rows * KV / 4;
        const int u = tid % upr;
        if (u < used) {
          float* dA = reinterpret_cast<float*>(rowsA) + 4 * u;
          float* dT = reinterpret_cast<float*>(rowsT) + 4 * u;
          for (int j = tid / upr; j < nn; j += kTileThreads / upr) {
            const size_t off = ((size_t)nodes[j] * LZ + k0) * KV + 4 * u;
            cp_async16(dA + (size_t)j * kTileChunk * KV, TAg + off);
            if (tsep) cp_async16(dT + (size_t)j * kTileChunk * KV, Tg + off);
          }
        }
      }
      if (gi == 0) {
        constexpr int upv = kTileChunk / 4;
        static_assert(kTileThreads % upv == 0, "whole rows per round");
        const int uv = tid % upv;
        if (4 * uv < rows)
          for (int j = tid / upv; j < ne; j += kTileThreads / upv)
            cp_async16(rowsV + j * kTileChunk + 4 * uv, a.vf + (size_t)recs[j].e * LZ + k0 + 4 * uv);
      }
      cp_async_wait_all();
      __syncthreads();
      // The pass's layers on the lanes; a pass of at most 16, 8 or 4 layers gives a warp 2, 4 or 8
      // edges at a time.
      const int wid = rows > 16 ? 32 : (rows > 8 ? 16 : (rows > 4 ? 8 : 4));
      const int l = lane & (wid - 1);
      const int z = (int)k0 + l + 1;
      if (l < rows)
        for (int j = (warp * kW + lane) / wid; j < ne; j += kTileThreads / wid) {
          // the edge's record in vector reads (broadcast to its lanes)
          const int4* rv = reinterpret_cast<const int4*>(&recs[j]);
          const int4 r0 = rv[0], r1 = rv[1];  // e, n1, n2, hi | gm0, gm1, nb1, nb2
          const uint2 rs = rsA[j];
          const bool act = z <= r0.w;
          const bool tri_ok = HOR == 0 || (r1.x >= 0 && z >= r1.x && z <= r1.y - 1);
          if (act && !tri_ok) continue;  // kf_hflux_mean's
          V<KV> r = splat<KV>(0.f);
          if (act) {
            const float v = rowsV[j * kTileChunk + l];
            const V<KV> s1 = rowsA[(rs.x & 0xffff) + l];
            const V<KV> s2 = rowsA[(rs.x >> 16) + l];
            const V<KV> q1 = tsep ? rowsT[(rs.x & 0xffff) + l] : s1;
            const V<KV> q2 = tsep ? rowsT[(rs.x >> 16) + l] : s2;
            V<KV> p1 = s1, p2 = s2;
            if (HOR != 0) {
              const float4 wu = reinterpret_cast<const float4*>(&recs[j])[4];
              const float4 wd = reinterpret_cast<const float4*>(&recs[j])[5];
              const V<KV> dT3 = muls(sub(s2, s1), 1.f / 3.f);
              const unsigned rd = rsD[j];
              const V<KV> u1 = rowsA[(rs.y & 0xffff) + l];
              const V<KV> u2 = rowsA[(rs.y >> 16) + l];
              const V<KV> d1 = rowsA[(rd & 0xffff) + l];
              const V<KV> d2 = rowsA[(rd >> 16) + l];
              p1 = fmas(u2, wu.z, fmas(u1, wu.y, fmas(s1, wu.x, dT3)));
              p2 = fmas(d2, wd.z, fmas(d1, wd.y, fmas(s2, wd.x, dT3)));
            }
            const float c1 = (HOR == 2 || r1.z - z >= 0) ? 1.f : 0.f, c2 = (HOR == 2 || r1.w - z >= 0) ? 1.f : 0.f;
            r = tile_flux<HOR, FCT, KV>(s1, s2, q1, q2, p1, p2, v, a.ph, c1, c2);
          }
          st<KV>(out, (unsigned)r0.x * LZ + k0 + l, r);
        }
    }
  }
}
template <int HOR, bool FCT, int KV>
__global__ void __launch_bounds__(kTileThreads) kf_hflux_tile(DMesh m, FastPtrs a) {
  hflux_tile<HOR, FCT, KV>(m, a);
}
template <int HOR, bool FCT, int KV>
__global__ void __launch_bounds__(kTileThreads) kf_hflux_tile_g(DMesh m, FastPtrs a) {
  hflux_tile<HOR, FCT, KV>(m, group_of(a, blockIdx.y));
}


// The edges' layers outside their triangles' window (or of edges without
// triangles), after kf_hflux_tile: the mean gradients around both nodes. Such a
// layer has some fifteen times the loads of one in the window, and a warp of
// kf_hflux_tile with a single one waited for it; the mesh lists them in runs of
// up to kMeanRun layers (DMesh::mean_seg). Two threads share a layer, one per
// node; tracer groups over blockIdx.y: the chain of dependent gathers is what
// takes the time. Edge stage with this kernel against the same layers computed
// inside kf_hflux_tile (which falls from 72 to 48 registers): pi mesh of
// 188,661 nodes, 47 layers, 4 tracers 305 / 438 us; closed 513^2x64, 2 tracers
// 370 / 476; 48x40x30, 3 tracers (its seam) 20 / 35.
template <int HOR, bool FCT, int KV>
__global__ void __launch_bounds__(kTileThreads) kf_hflux_mean(DMesh m, FastPtrs a) {
  const MeanItem it = mean_item(blockIdx.x, kTileThreads, threadIdx.x);
  const int2 seg = it.run < m.nmean ? reinterpret_cast<const int2*>(m.mean_seg)[it.run] : make_int2(0, 0);
  const int l = it.layer, side = it.side;
  const bool act = l < (seg.y >> 16);
  const int e = seg.x, n1 = m.edge_nodes[2 * e], n2 = m.edge_nodes[2 * e + 1];
  const unsigned LZ = m.LZ, k = (unsigned)(seg.y & 0xffff) + (act ? l : 0);
  const float* __restrict__ Tg = a.T + blockIdx.y * a.gT;
  const float* __restrict__ TAg = a.TA != a.T ? a.TA + blockIdx.y * a.gTA : Tg;
  V<KV> gx = splat<KV>(0.f), gy = gx;
  if (act) node_grad<KV, 3>(m, TAg, side ? n2 : n1, k, gx, gy);
  const float ex = m.g32.edge_dxa[2 * e], ey = m.g32.edge_dxa[2 * e + 1];
  const V<KV> p = muls(fmas(gy, ey, muls(gx, ex)), 1.f / 6.f);
  const V<KV> o = shfl_v(p, threadIdx.x ^ 1);  // the other node's
  if (!act || side) return;
  const V<KV> s1 = ld<KV>(TAg, n1 * LZ + k), s2 = ld<KV>(TAg, n2 * LZ + k);
  V<KV> q1 = s1, q2 = s2;
  if (FCT && a.TA != a.T) {
    q1 = ld<KV>(Tg, n1 * LZ + k);
    q2 = ld<KV>(Tg, n2 * LZ + k);
  }
  const V<KV> dT3 = muls(sub(s2, s1), 1.f / 3.f);
  const float c1 = (HOR == 2 || m.nbl[n1] > (int)k) ? 1.f : 0.f, c2 = (HOR == 2 || m.nbl[n2] > (int)k) ? 1.f : 0.f;
  st<KV>(a.adfh + blockIdx.y * a.gE, (unsigned)e * LZ + k,
         tile_flux<HOR, FCT, KV>(s1, s2, q1, q2, add(p, dT3), add(o, dT3), a.vf[(unsigned)e * LZ + k], a.ph, c1, c2));
}

}  // namespace fast
}  // namespace fgb
