// Instantiation machinery of the line-form stage kernel, shared by vlasov_line64.cu and
// vlasov_line32.cu.
#pragma once

#include <algorithm>
#include <type_traits>

#include "vlasov_line.h"
#include "vlasov_stage_line.cuh"

namespace vl {
namespace lk {

template <int N, typename T>
LineTables<N, T> tables(const LineCoef &lc) {
    LineTables<N, T> t;
    for (int i = 0; i < N; ++i) {
        for (int m = 0; m < N; ++m) t.up[i * N + m] = (T)lc.up[i * N + m];
        t.xl[i] = (T)lc.xi[2 * i];
        t.xr[i] = (T)(-lc.xi[2 * i + 1]);
        t.wu[i] = lc.xw[i] / lc.ju;
        t.wv[i] = lc.xw[i] / lc.jv;
    }
    return t;
}

template <int N, typename T>
cudaError_t launch(const StageArgs &a0, const LineCoef &lc, dim3 grid, cudaStream_t s) {
    using G = LineGeom<N, T>;
    StageArgs a = a0;
    a.never = -1;
    const LineTables<N, T> tb = tables<N, T>(lc);
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = stage_config(a, grid, G::THREADS, G::smem_bytes(), s, &attr);
    auto go = [&](auto kc) {
        constexpr int K = decltype(kc)::value;
        if constexpr (sizeof(T) == 4) {
            if (a.bg_rb != nullptr) {
                return cudaLaunchKernelEx(&cfg, &stage_line_kernel<N, T, K, 1>, a, tb);
            }
        }
        return cudaLaunchKernelEx(&cfg, &stage_line_kernel<N, T, K, 0>, a, tb);
    };
    if (a.kind == KIND_EULER) return go(std::integral_constant<int, KIND_EULER>{});
    if (a.kind == KIND_COMBINE) return go(std::integral_constant<int, KIND_COMBINE>{});
    return go(std::integral_constant<int, KIND_RHS>{});
}

template <int N, typename T>
int occupancy(int kind) {
    using G = LineGeom<N, T>;
    auto one = [&](auto *k) {
        int blocks = 0;
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::smem_bytes());
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k, G::THREADS, G::smem_bytes()) != cudaSuccess)
            return 1;
        return blocks > 0 ? blocks : 1;
    };
    auto both = [&](auto kc) {
        constexpr int K = decltype(kc)::value;
        int o = one(stage_line_kernel<N, T, K, 0>);
        if constexpr (sizeof(T) == 4) o = std::min(o, one(stage_line_kernel<N, T, K, 1>));
        return o;
    };
    if (kind == KIND_EULER) return both(std::integral_constant<int, KIND_EULER>{});
    if (kind == KIND_COMBINE) return both(std::integral_constant<int, KIND_COMBINE>{});
    return both(std::integral_constant<int, KIND_RHS>{});
}

// F is called with std::integral_constant<int, n>
template <typename F, typename R>
R with_order(int n, R other, F &&f) {
    switch (n) {
        case 1: return f(std::integral_constant<int, 1>{});
        case 2: return f(std::integral_constant<int, 2>{});
        case 3: return f(std::integral_constant<int, 3>{});
        case 4: return f(std::integral_constant<int, 4>{});
        case 5: return f(std::integral_constant<int, 5>{});
        case 6: return f(std::integral_constant<int, 6>{});
        case 7: return f(std::integral_constant<int, 7>{});
        case 8: return f(std::integral_constant<int, 8>{});
        case 9: return f(std::integral_constant<int, 9>{});
        case 10: return f(std::integral_constant<int, 10>{});
        default: return other;
    }
}

}  // namespace lk
}  // namespace vl
