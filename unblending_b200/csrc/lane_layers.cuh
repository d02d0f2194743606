// Lane kernels (one pixel per lane) of one layer count, UNB_SOLVER_LAYERS: first
// pass and refinement in FP64 and FP32, batched first pass in FP64. Included by lane_l<L>.cu,
// which are compiled with --fmad=false as the other solve kernels are.
#include <algorithm>

#include "solver_dispatch.hpp"
#include "lane_solver.cuh"

#ifndef UNB_SOLVER_LAYERS
#error "define UNB_SOLVER_LAYERS before including lane_layers.cuh"
#endif

namespace unb {

namespace {
constexpr int kL = UNB_SOLVER_LAYERS;

template <class T, bool R, bool BATCH>
cudaError_t lanes(const Models<T>& m, const SolverControls& c, const SolveArgs& a, int sms, cudaStream_t s) {
    auto k = solve_lanes<T, kL, R, BATCH>;
    if (!a.history) return cudaErrorInvalidValue;
    constexpr int smem = lane_smem_bytes(kL, sizeof(T) == 4);
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kLaneBlock, smem);
    if (e != cudaSuccess) return e;
    const int blocks = std::min(std::max(1, per_sm) * sms, a.history_lanes / kLaneBlock);
    if (blocks < 1) return cudaErrorInvalidValue;
    k<<<blocks, kLaneBlock, smem, s>>>(m, c, a);
    return cudaGetLastError();
}

}  // namespace

template <> cudaError_t solve_lanes_layers<kL>(bool refine, bool batch, const Models<double>& m, const SolverControls& c,
                                               const SolveArgs& a, int sms, cudaStream_t s) {
    if (batch) return lanes<double, false, true>(m, c, a, sms, s);
    return refine ? lanes<double, true, false>(m, c, a, sms, s) : lanes<double, false, false>(m, c, a, sms, s);
}

template <> cudaError_t solve_lanes_fp32_layers<kL>(bool refine, const Models<float>& m, const SolverControls& c,
                                                    const SolveArgs& a, int sms, cudaStream_t s) {
    return refine ? lanes<float, true, false>(m, c, a, sms, s) : lanes<float, false, false>(m, c, a, sms, s);
}

}  // namespace unb
