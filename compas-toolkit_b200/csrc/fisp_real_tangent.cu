// fisp_real_tangent.cu — layouts and launches of the real-phase FISP tangent kernels (fisp_real.cuh).
#include <algorithm>

#include "compas/compas.h"
#include "fisp_real.cuh"
#include "kernels.h"

namespace compas {

namespace {

#define COMPAS_REAL(KP, G)                                                                                  \
    {KP, G, kernels::kRealWarps<KP, 3>, int(kernels::real_smem_bytes<G, 3>(1)),                        \
     kernels::fisp_real_kernel<kernels::RealTangents, KP, G, false>, nullptr,                             \
     kernels::fisp_real_queue_kernel<kernels::RealTangents, KP, G>}
// Three state vectors: up to 6 pairs fit a lane, more states go over 2 or 4 lanes (25 states: 2 lanes
// of 6 pairs, no padding).
const RealLayout kLayouts[] = {
    COMPAS_REAL(1, 1), COMPAS_REAL(2, 1), COMPAS_REAL(3, 1), COMPAS_REAL(4, 1), COMPAS_REAL(5, 1), COMPAS_REAL(6, 1),
    COMPAS_REAL(4, 2), COMPAS_REAL(5, 2), COMPAS_REAL(6, 2), COMPAS_REAL(4, 4),
};
// few (voxel, position) pairs: the states over 4 lanes
const RealLayout kSplitLayouts[] = {
    COMPAS_REAL(1, 4), COMPAS_REAL(2, 4), COMPAS_REAL(3, 4), COMPAS_REAL(4, 4),
};
#undef COMPAS_REAL

const RealLayout& covering(const RealLayout* layouts, int count, int N) {
    for (int i = 0; i < count; i++)
        if (2 * layouts[i].KP * layouts[i].G + 1 >= N) return layouts[i];
    COMPAS_ERROR("no real-phase tangent layout holds the states");
}
const RealLayout& real_layout(int N, bool split) {
    return split ? covering(kSplitLayouts, 4, N) : covering(kLayouts, int(sizeof(kLayouts) / sizeof(kLayouts[0])), N);
}

}  // namespace

bool fisp_real_tangent_split(int64_t pairs) {
    return pairs <= kRealSplitPairs;
}

int fisp_real_tangent_queue_warps(int N, bool split, int P, int64_t tiles) {
    return fisp_real_warps(real_layout(N, split).warps, P, tiles);
}

int fisp_real_tangent_tile_voxels(int N, bool split) {
    return 32 / real_layout(N, split).G;
}

void launch_fisp_real_tangent(const CompasContext& ctx, const kernels::FispArgs& a, const kernels::HostAnswer& ask) {
    const RealLayout* layout = &real_layout(a.N, fisp_real_tangent_split(int64_t(a.nvoxels) * a.P));
    const int ntiles = div_ceil(a.nvoxels, 32 / layout->G);
    const int W = fisp_real_warps(layout->warps, a.P, div_ceil(ntiles, 148));
    const size_t smem = size_t(W) * layout->smem;
    DeviceGuard guard(ctx.device());
    const void* fn = reinterpret_cast<const void*>(layout->fn);
    allow_smem(fn, smem);
    const int grid = std::min(ntiles, resident_ctas(fn, 32 * W, smem, ctx.device()));
    layout->fn<<<grid, 32 * W, smem, ctx.stream()>>>(a, ask, ntiles, nullptr, nullptr);
    check_launch("fisp_real_kernel (tangents)");
}

void launch_fisp_real_tangent_queue(cudaStream_t stream, int device, int W, int max_state, bool split,
                                    const kernels::FispArgs* jobs, const int2* items, int nitems, int* head) {
    if (nitems <= 0) return;
    const RealLayout& layout = real_layout(max_state, split);
    const void* fn = reinterpret_cast<const void*>(layout.queue);
    const size_t smem = size_t(W) * layout.smem;
    DeviceGuard guard(device);
    allow_smem(fn, smem);
    const int grid = std::min(nitems, resident_ctas(fn, 32 * W, smem, device));
    layout.queue<<<grid, 32 * W, smem, stream>>>(jobs, items, nitems, head);
    check_launch("fisp_real_queue_kernel (tangents)");
}

}  // namespace compas
