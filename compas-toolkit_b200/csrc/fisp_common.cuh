// fisp_common.cuh — what the FISP kernels of fisp.cu and fisp_real.cu share: the phase flag of the
// excitation table and the split of (voxel tile, slice position) items over persistent CTAs.
#pragma once

#include "common.cuh"
#include "job_args.cuh"

namespace compas {
namespace kernels {

// True when every phase of the sequence's table is real (sin φ = 0 exactly: a real RF train and real
// slice profiles, as in the usual MR-STAT FISP sequences).
__device__ __forceinline__ bool fisp_real_phases(const FispArgs& a) {
    return __ldg(&a.table[int64_t(a.P) * a.nTR].x) == 0.0f;
}

// Balanced item split of the one-simulation kernel: the order of a CTA's items (at most
// kFispBalancedItems) and its hand-off points, in shared memory
constexpr int kFispBalancedItems = 2048;
struct FispOrder {
    int item[kFispBalancedItems];  // item of the u-th position in the CTA's order
    int wait_u;                    // first u of the head part (positions of the shared first tile)
    int publish_u;                 // u after the tail part (first positions of the shared last tile)
    int cta;
    int* handoff;                  // per-CTA flags, zero at launch
    unsigned int* status;          // device status word
};

// The share of CTA blockIdx.x when ntiles·P items are split evenly over the grid, in the order tail
// (the first positions of its last tile, shared with the next CTA), whole tiles, head (the last
// positions of its first tile, shared with the previous CTA). Returns the number of items.
__device__ __forceinline__ int fisp_balanced_order(FispOrder& ord, int ntiles, int P, int* handoff,
                                                   unsigned int* status) {
    const int64_t total = int64_t(ntiles) * P;
    const int i0 = int(total * blockIdx.x / gridDim.x), i1 = int(total * (blockIdx.x + 1) / gridDim.x);
    const int n = i1 - i0;
    const int h_end = min(i1, (i0 + P - 1) / P * P);  // end of the head: the first tile's last positions
    const int t_start = max(h_end, i1 / P * P);        // start of the tail: the last tile's first positions
    const int L0 = i1 - t_start, L01 = L0 + (t_start - h_end);
    for (int u = threadIdx.x; u < n; u += blockDim.x)
        ord.item[u] = u < L0 ? t_start + u : (u < L01 ? h_end + (u - L0) : i0 + (u - L01));
    if (threadIdx.x == 0) {
        ord.wait_u = i0 % P != 0 ? L01 : n;      // n: no head, nothing to wait for
        ord.publish_u = i1 % P != 0 ? L0 : -1;   // -1: no tail, nothing to hand over
        ord.cta = blockIdx.x;
        ord.handoff = handoff;
        ord.status = status;
    }
    __syncthreads();
    return n;
}

// Hand-off flags of the balanced item split: a CTA publishes the partial sums of its last, shared
// tile, and the next CTA waits for them before it adds its positions of that tile. The wait is
// bounded: one that gives up records STATUS_WAIT_TIMEOUT in the status word and returns.
__device__ __forceinline__ void handoff_publish(int* flag) {
    __threadfence();  // the CTA's partial-sum stores (ordered before by the barrier) are visible first
    atomicExch(flag, 1);
}
__device__ __forceinline__ void handoff_wait(const int* flag, unsigned int* status) {
    const long long t0 = clock64();
    for (;;) {
        int v;
        asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
        if (v != 0) return;
        if (clock64() - t0 > 4000000000LL) {
            if (status) atomicOr(status, STATUS_WAIT_TIMEOUT);
            return;
        }
        __nanosleep(256);
    }
}

// Range of whole tiles of CTA `cta` when `ntiles` tiles are split over `nctas` CTAs (sizes differ
// by at most one tile).
__device__ __forceinline__ int2 cta_tile_range(int ntiles, int cta, int nctas) {
    return make_int2(int(int64_t(ntiles) * cta / nctas), int(int64_t(ntiles) * (cta + 1) / nctas));
}

}  // namespace kernels

// CTAs of `fn` resident on the device at once with this block size and dynamic shared memory:
// the grid of the persistent one-simulation kernels
inline int resident_ctas(const void* fn, int threads, size_t smem, int device) {
    int per_sm = 1, sms = 148;
    COMPAS_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem));
    COMPAS_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    return std::max(1, per_sm) * sms;
}

// Opt in to `smem` bytes of dynamic shared memory. Without the attribute a launch may use at most
// 48 KB minus the kernel's static shared memory (the work-queue kernels keep their job's argument
// block there), so the attribute is set from 40 KB on.
inline void allow_smem(const void* fn, size_t smem) {
    if (smem > 40 * 1024)
        COMPAS_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
}

}  // namespace compas
