// fisp_real.cu — layouts and launches of the real-phase FISP value kernels (fisp_real.cuh).
#include <algorithm>
#include <optional>

#include "compas/compas.h"
#include "fisp_real.cuh"
#include "kernels.h"

namespace compas {

namespace {

#define COMPAS_REAL(KP)                                                                                              \
    {KP, 1, kernels::kRealWarps<KP, 1>, int(kernels::real_smem_bytes<1, 1>(1)),                                   \
     kernels::fisp_real_kernel<kernels::RealValue, KP, 1, false>, kernels::fisp_real_kernel<kernels::RealValue, KP, 1, true>, \
     kernels::fisp_real_queue_kernel<kernels::RealValue, KP, 1>}
// entry KP - 1 holds states 0 .. 2·KP: N = 2·KP (one padding state) and 2·KP + 1
const RealLayout kLayouts[] = {
    COMPAS_REAL(1), COMPAS_REAL(2), COMPAS_REAL(3), COMPAS_REAL(4), COMPAS_REAL(5), COMPAS_REAL(6),
    COMPAS_REAL(7), COMPAS_REAL(8), COMPAS_REAL(9), COMPAS_REAL(10), COMPAS_REAL(11), COMPAS_REAL(12),
    COMPAS_REAL(13), COMPAS_REAL(14), COMPAS_REAL(15), COMPAS_REAL(16),
};
#undef COMPAS_REAL
#define COMPAS_REAL_SPLIT(KP)                                                                                        \
    {KP, 4, kernels::kRealWarps<KP, 1>, int(kernels::real_smem_bytes<4, 1>(1)),                                   \
     kernels::fisp_real_kernel<kernels::RealValue, KP, 4, false>, nullptr, nullptr}
// entry KP - 1: the states over 4 lanes, N <= 8·KP + 1
const RealLayout kSplitLayouts[] = {COMPAS_REAL_SPLIT(1), COMPAS_REAL_SPLIT(2), COMPAS_REAL_SPLIT(3), COMPAS_REAL_SPLIT(4)};
#undef COMPAS_REAL_SPLIT
constexpr int kMaxStates = 33;

const RealLayout& real_layout(int N) {
    COMPAS_CHECK(N >= 2 && N <= kMaxStates);
    return kLayouts[N / 2 - 1];
}

}  // namespace

bool fisp_real_covers(const FISPSequence& seq, bool tangents) {
    return seq.max_state >= 2 && seq.max_state <= kMaxStates && !fisp_layout_forced(seq.max_state, tangents) &&
           (seq.repetitions == 1 || seq.inversion_prepulse || seq.wait_spoiling || seq.TW == 0.0f);
}

int fisp_real_warps(int most, int P, int64_t tiles) {
    return int(std::max<int64_t>(1, std::min<int64_t>(most, P * tiles)));
}

int fisp_real_queue_warps(int N, int P, int64_t tiles) {
    return fisp_real_warps(real_layout(N).warps, P, tiles);
}

void launch_fisp_real(const CompasContext& ctx, const kernels::FispArgs& a, const kernels::HostAnswer& ask,
                      bool balance, int* handoff, int handoff_capacity) {
    const RealLayout* layout = &real_layout(a.N);
    // Few (voxel, position) pairs leave most schedulers without a warp, and a lone warp runs at the
    // latency of its instructions: then the states go over 4 lanes.
    if (int64_t(a.nvoxels) * a.P <= kRealSplitPairs) layout = &kSplitLayouts[(a.N + 6) / 8 - 1];
    const int ntiles = div_ceil(a.nvoxels, 32 / layout->G);
    // one position: warps have nothing to share, each is a CTA
    const int W = a.P == 1 ? 1 : fisp_real_warps(layout->warps, a.P, div_ceil(ntiles, 148));
    const size_t smem = size_t(W) * layout->smem;
    DeviceGuard guard(ctx.device());
    const void* fn = reinterpret_cast<const void*>(layout->fn);
    allow_smem(fn, smem);
    int grid = std::min(ntiles, resident_ctas(fn, 32 * W, smem, ctx.device()));
    // the balanced split, as for the general kernels (launch_fisp): all CTAs resident at once, and shares
    // of at least P + W items, which fill more than one round. (A CTA publishes its tail before it waits for its
    // predecessor's, fisp_real_items: it waits on one other, never on a chain.)
    bool balanced = false;
    if (balance && a.P > 1 && layout->balanced != nullptr) {
        const void* bfn = reinterpret_cast<const void*>(layout->balanced);
        allow_smem(bfn, smem);
        const int bgrid = std::min(ntiles, resident_ctas(bfn, 32 * W, smem, ctx.device()));
        const int64_t share = int64_t(ntiles) * a.P / bgrid;  // or one more
        balanced = bgrid > 1 && share >= a.P + W && share < kernels::kFispBalancedItems &&
                   (handoff == nullptr || bgrid <= handoff_capacity);
        if (balanced) grid = bgrid;
    }
    std::optional<Array<int, 1>> flags;
    if (balanced) {
        if (handoff == nullptr) {
            flags.emplace(std::array<int64_t, 1> {grid}, ctx.device(), ctx.stream());
            handoff = flags->data();
        }
        COMPAS_CUDA_CHECK(cudaMemsetAsync(handoff, 0, sizeof(int) * size_t(grid), ctx.stream()));
    }
    (balanced ? layout->balanced : layout->fn)<<<grid, 32 * W, smem, ctx.stream()>>>(a, ask, ntiles, handoff,
                                                                                       ctx.status_word());
    check_launch("fisp_real_kernel");
}

void launch_fisp_real_queue(cudaStream_t stream, int device, int W, int max_state, const kernels::FispArgs* jobs,
                            const int2* items, int nitems, int* head) {
    if (nitems <= 0) return;
    const RealLayout& layout = real_layout(max_state);
    const void* fn = reinterpret_cast<const void*>(layout.queue);
    const size_t smem = size_t(W) * layout.smem;
    DeviceGuard guard(device);
    allow_smem(fn, smem);
    const int grid = std::min(nitems, resident_ctas(fn, 32 * W, smem, device));
    layout.queue<<<grid, 32 * W, smem, stream>>>(jobs, items, nitems, head);
    check_launch("fisp_real_queue_kernel");
}

}  // namespace compas
