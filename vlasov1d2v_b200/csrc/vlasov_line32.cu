// FP32 instantiations of the line-form stage kernel (see vlasov_line.h).
#include "vlasov_line.cuh"

namespace vl {

template <>
cudaError_t line_launch<float>(int n, const StageArgs &a, const LineCoef &lc, dim3 grid, cudaStream_t s) {
    return lk::with_order(n, cudaErrorInvalidValue,
                          [&](auto nc) { return lk::launch<decltype(nc)::value, float>(a, lc, grid, s); });
}

template <>
size_t line_smem<float>(int n) {
    return lk::with_order(n, (size_t)0, [](auto nc) { return LineGeom<decltype(nc)::value, float>::smem_bytes(); });
}

template <>
int line_occupancy<float>(int n, int kind) {
    return lk::with_order(n, 1, [&](auto nc) { return lk::occupancy<decltype(nc)::value, float>(kind); });
}

}  // namespace vl
