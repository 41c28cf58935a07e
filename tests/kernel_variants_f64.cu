// The exact FP64 form's kernels, instantiated alone for tests/test_kernel_variants.py's spill report.
#include "fgb_step.cuh"

namespace fgb {
inline namespace exact64 {

template __global__ void k_fct_lo<double, 1>(DMesh, StepPtrs<double>, int);
template __global__ void k_fct_lo<double, 3>(DMesh, StepPtrs<double>, int);
template __global__ void k_fct_ratio<double>(DMesh, StepPtrs<double>, int);
template __global__ void k_fct_update<double>(DMesh, StepPtrs<double>, int);
template __global__ void k_nofct_update<double, 3>(DMesh, StepPtrs<double>, int);
template __global__ void k_hflux<double, 1, true, true, true>(DMesh, StepPtrs<double>, const double2*);

}  // inline namespace
}  // namespace fgb
