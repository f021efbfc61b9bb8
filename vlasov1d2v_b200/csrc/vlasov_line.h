// Launches of the line-form stage kernel (vlasov_stage_line.cuh).  The instantiations per order,
// stage kind and background split live in vlasov_line64.cu and vlasov_line32.cu.
#pragma once

#include <cuda_runtime.h>

#include "vlasov_kernels.cuh"

namespace vl {

// the coefficients a context holds, from which a launch fills its tables
struct LineCoef {
    const double *up, *xi, *xw;   // [n n], [n 2], [n]
    double ju, jv;
};

// one stage of order n (1..10) over grid (G, nx); a.bg_rb selects the background-split form
template <typename T>
cudaError_t line_launch(int n, const StageArgs &a, const LineCoef &lc, dim3 grid, cudaStream_t s);
// resident CTAs per SM of a stage kind's kernels (the fewer of its background forms); sets their
// shared-memory limits
template <typename T>
int line_occupancy(int n, int kind);
// v elements per tile
int line_ept(int n);
// dynamic shared memory of a CTA (bytes)
template <typename T>
size_t line_smem(int n);

template <>
cudaError_t line_launch<double>(int n, const StageArgs &a, const LineCoef &lc, dim3 grid, cudaStream_t s);
template <>
cudaError_t line_launch<float>(int n, const StageArgs &a, const LineCoef &lc, dim3 grid, cudaStream_t s);
template <>
size_t line_smem<double>(int n);
template <>
size_t line_smem<float>(int n);
template <>
int line_occupancy<double>(int n, int kind);
template <>
int line_occupancy<float>(int n, int kind);

}  // namespace vl
