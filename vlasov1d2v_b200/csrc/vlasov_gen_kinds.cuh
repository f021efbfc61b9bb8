// Instantiation machinery shared by vlasov_gen_kinds64.cu and vlasov_gen_kinds32.cu: one kernel
// per (order, form, stage kind, background split), dispatched from run-time values.
#pragma once

#include <cstring>

#include "vlasov_gen_kinds.h"

namespace vl {
namespace gk {

template <typename T, int N, bool PAIR, int K, int B, bool FUSE = false>
constexpr auto kernel() {
    if constexpr (PAIR)
        return &stage_gen_pair_kernel<N, T, K, B, FUSE>;
    else
        return &stage_gen_tma_kernel<N, T, K, B, FUSE>;
}

template <typename T, int N, bool PAIR, int K, int B, bool FUSE = false>
cudaError_t launch_one(dim3 grid, size_t smem, cudaStream_t s, const StageArgs &a, const StageTables<T> &tb,
                       const GenMaps &maps) {
    constexpr int THREADS = PAIR ? GenPairGeom<N, T>::THREADS : GenTmaGeom<N, T>::THREADS;
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = stage_config(a, grid, THREADS, smem, s, &attr);
    return cudaLaunchKernelEx(&cfg, kernel<T, N, PAIR, K, B, FUSE>(), a, tb, maps);
}

template <typename T, int N, bool PAIR>
cudaError_t launch_n(int kind, bool bg, dim3 grid, size_t smem, cudaStream_t s, const StageArgs &a,
                     const StageTables<T> &tb, const GenMaps &maps) {
    constexpr bool HAS_BG = sizeof(T) == 4;   // the background split is a form of FP32 states
    if constexpr (gen_fusable<T>(N, PAIR)) {
        if (a.ff.mode != FUSE_NONE) {
            if (HAS_BG && bg) {
                constexpr int B1 = HAS_BG ? 1 : 0;
                if (kind == KIND_EULER) return launch_one<T, N, PAIR, KIND_EULER, B1, true>(grid, smem, s, a, tb, maps);
                return launch_one<T, N, PAIR, KIND_COMBINE, B1, true>(grid, smem, s, a, tb, maps);
            }
            if (kind == KIND_EULER) return launch_one<T, N, PAIR, KIND_EULER, 0, true>(grid, smem, s, a, tb, maps);
            return launch_one<T, N, PAIR, KIND_COMBINE, 0, true>(grid, smem, s, a, tb, maps);
        }
    }
    if (kind == KIND_EULER) {
        if (HAS_BG && bg) return launch_one<T, N, PAIR, KIND_EULER, HAS_BG ? 1 : 0>(grid, smem, s, a, tb, maps);
        return launch_one<T, N, PAIR, KIND_EULER, 0>(grid, smem, s, a, tb, maps);
    }
    if (kind == KIND_COMBINE) {
        if (HAS_BG && bg) return launch_one<T, N, PAIR, KIND_COMBINE, HAS_BG ? 1 : 0>(grid, smem, s, a, tb, maps);
        return launch_one<T, N, PAIR, KIND_COMBINE, 0>(grid, smem, s, a, tb, maps);
    }
    if (HAS_BG && bg) return launch_one<T, N, PAIR, KIND_RHS, HAS_BG ? 1 : 0>(grid, smem, s, a, tb, maps);
    return launch_one<T, N, PAIR, KIND_RHS, 0>(grid, smem, s, a, tb, maps);
}

// shared-memory limits of every instantiation that launch_n launches, and the fewest CTAs of one that an SM
// keeps resident
template <typename T, int N, bool PAIR>
int prepare_n(size_t smem) {
    constexpr int THREADS = PAIR ? GenPairGeom<N, T>::THREADS : GenTmaGeom<N, T>::THREADS;
    int occ = 32;
    auto one = [&](auto *k) {
        int blocks = 0;
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k, THREADS, smem) != cudaSuccess || blocks < 1)
            blocks = 1;
        occ = blocks < occ ? blocks : occ;
    };
    auto kinds = [&](auto bc) {
        constexpr int B = decltype(bc)::value;
        one(kernel<T, N, PAIR, KIND_EULER, B>());
        one(kernel<T, N, PAIR, KIND_COMBINE, B>());
        one(kernel<T, N, PAIR, KIND_RHS, B>());
        if constexpr (gen_fusable<T>(N, PAIR)) {
            one(kernel<T, N, PAIR, KIND_EULER, B, true>());
            one(kernel<T, N, PAIR, KIND_COMBINE, B, true>());
        }
    };
    kinds(std::integral_constant<int, 0>{});
    if constexpr (sizeof(T) == 4) kinds(std::integral_constant<int, 1>{});
    return occ;
}

}  // namespace gk
}  // namespace vl
