// More variants of the FP32 step's kernels, instantiated alone so that
// tests/test_kernel_variants.py can read ptxas's spill report for them.
#include "fgb_fast_launch.cuh"

namespace fgb {
namespace fast {

// per-edge edge fluxes (fields without 16-byte alignment, launch shapes asked for)
template __global__ void kf_hflux<1, true, 4, 1>(DMesh, FastPtrs);
template __global__ void kf_hflux<1, true, 4, 2>(DMesh, FastPtrs);
template __global__ void kf_hflux<2, true, 4, 1>(DMesh, FastPtrs);
template __global__ void kf_hflux<2, true, 4, 2>(DMesh, FastPtrs);
template __global__ void kf_hflux<1, true, 2, 1>(DMesh, FastPtrs);
// mean-gradient layers
template __global__ void kf_hflux_mean<1, true, 4>(DMesh, FastPtrs);
template __global__ void kf_hflux_mean<2, true, 2>(DMesh, FastPtrs);
// LO stage, QR4C and PPM, separate T_AB and w_e without w_split
template __global__ void kf_lo64<1, 4, true, true, false>(DMesh, FastPtrs);
template __global__ void kf_lo64<3, 4, true, true, false>(DMesh, FastPtrs);
template __global__ void kf_lo64<1, 2, false, true, false>(DMesh, FastPtrs);
// limiting factors and update with compensated sums, groups of one and two tracers
template __global__ void kf_ratio64<2, false, true>(DMesh, FastPtrs);
template __global__ void kf_ratio64<1, false, true>(DMesh, FastPtrs);
template __global__ void kf_update<1, 1, false, true, false>(DMesh, FastPtrs);
// update of two tracers with plain sums: three edges in flight cost 8 bytes and
// are faster all the same (250x230x47: 119 -> 107 us)
template __global__ void kf_update<2, 1, false, false, false>(DMesh, FastPtrs);

// volume fluxes, a thread per four layers
void* keep_vflux4() { return reinterpret_cast<void*>(&kf_vflux4); }

}  // namespace fast
}  // namespace fgb
