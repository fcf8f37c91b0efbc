// The CUDA translation unit: every __global__ kernel of the library and its launch wrapper.
#include "launch.hpp"

#include <algorithm>
#include <mutex>

#include "combine.cuh"
#include "combine_local.cuh"
#include "combine_push.cuh"
#include "dispatch.cuh"
#include "dispatch_local.cuh"
#include "fused_reduce.cuh"

namespace bep {

std::size_t dispatch_shared_bytes(const SegmentLayout& lay, int tx_warps, int rx_warps, bool use_tma, int stages,
                                  int send_ctas) {
    return dispatch_smem_bytes(lay, tx_warps, rx_warps, use_tma, stages, send_ctas);
}

bool role_profiling_enabled() { return BEP_ENABLE_PROFILING != 0; }

cudaError_t configure_kernels(std::size_t dispatch_smem) {
    // One attribute per kernel per process: several buffers may be alive, so only ever raise it.
    static std::mutex mutex;
    static std::size_t current[64] = {0};
    std::lock_guard<std::mutex> guard(mutex);
    int device = 0;
    cudaError_t status = cudaGetDevice(&device);
    if (status != cudaSuccess) return status;
    if (device < 0 || device >= 64) return cudaErrorInvalidDevice;
    if (dispatch_smem > current[device]) {
        status = cudaFuncSetAttribute(dispatch_kernel<kSmallCtaThreads>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(dispatch_smem));
        if (status != cudaSuccess) return status;
        status = cudaFuncSetAttribute(dispatch_kernel<kMaxWarps * 32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(dispatch_smem));
        if (status != cudaSuccess) return status;
        current[device] = dispatch_smem;
    }
    return cudaSuccess;
}

int dispatch_resident_ctas(int threads, std::size_t smem) {
    int per_sm = 0, device = 0, sms = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
    const cudaError_t status = threads <= kSmallCtaThreads
                                   ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, dispatch_kernel<kSmallCtaThreads>, threads, smem)
                                   : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, dispatch_kernel<kMaxWarps * 32>, threads, smem);
    if (status != cudaSuccess) return 0;
    return per_sm * sms;
}

int combine_resident_ctas(int threads) {
    int per_sm = 0, device = 0, sms = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, combine_kernel, threads, 0) != cudaSuccess) return 0;
    return per_sm * sms;
}

namespace {

template <typename Kernel, typename Args>
cudaError_t cooperative_launch(Kernel kernel, const Args& args, dim3 grid, int threads, std::size_t smem,
                               cudaStream_t stream) {
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = dim3(static_cast<unsigned>(threads), 1, 1);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeCooperative;  // every CTA resident: the waits inside are safe
    attribute[0].val.cooperative = 1;
    config.attrs = attribute;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, args);
}

}  // namespace

cudaError_t launch_dispatch(const DispatchLaunch& launch, int ctas, int threads, std::size_t smem,
                            cudaStream_t stream) {
    const dim3 grid(ctas, launch.num_virtual, 1);
    if (threads <= kSmallCtaThreads) return cooperative_launch(dispatch_kernel<kSmallCtaThreads>, launch, grid, threads, smem, stream);
    return cooperative_launch(dispatch_kernel<kMaxWarps * 32>, launch, grid, threads, smem, stream);
}

LocalPlan plan_dispatch_local(const SegmentLayout& lay, int sms, std::size_t smem_limit, long long l2_bytes) {
    LocalPlan plan = make_local_plan(lay.num_experts, lay.num_channels, lay.num_topk, lay.hidden, lay.num_max_tokens, sms, smem_limit);
    plan.l2_bytes = l2_bytes;
    return plan;
}

std::size_t dispatch_local_hist_ints(const SegmentLayout& lay, int ctas) { return local_hist_ints(ctas, lay.num_experts, lay.num_channels); }

int dispatch_local_width(const SegmentLayout& lay, int tokens, bool padding) {
    return padding && tokens > 0 ? std::max(tokens, lay.num_experts) : tokens;
}

namespace {
using LocalKernel = void (*)(LocalDispatchArgs);
// by mode, then rows that stay E4M3, then more tokens than row buffers
constexpr LocalKernel kernels[12] = {
    local_dispatch_kernel<kLocalTogether, false, false>, local_dispatch_kernel<kLocalTogether, false, true>, local_dispatch_kernel<kLocalTogether, true, false>,
    local_dispatch_kernel<kLocalTogether, true, true>,   local_dispatch_kernel<kLocalWhole, false, false>,   local_dispatch_kernel<kLocalWhole, false, true>,
    local_dispatch_kernel<kLocalWhole, true, false>,     local_dispatch_kernel<kLocalWhole, true, true>,     local_dispatch_kernel<kLocalCached, false, false>,
    local_dispatch_kernel<kLocalCached, false, true>,    local_dispatch_kernel<kLocalCached, true, false>,   local_dispatch_kernel<kLocalCached, true, true>};
}  // namespace

LocalShape shape_dispatch_local(const SegmentLayout& lay, const LocalPlan& plan, int tokens, bool expand, bool recv_fp8, int ctas, bool cached) {
    const long long row_bytes = lay.hidden * (recv_fp8 ? 1ll : 2ll);
    return local_shape(plan, tokens, lay.num_topk, lay.hidden * 2ll + (expand ? lay.num_topk : 1) * row_bytes, ctas, cached);
}

cudaError_t launch_dispatch_local(const DispatchArgs& a, const RankConst& rc, const LocalPlan& plan, int* hist, unsigned long long* counters, int sms, int max_ctas, cudaStream_t stream) {
    const int ctas = std::max(1, std::min(std::min(sms, max_ctas), dispatch_local_width(rc.lay, a.num_tokens, a.do_expand && a.zero_padding && a.alignment > 1)));
    const LocalShape shape = shape_dispatch_local(rc.lay, plan, a.num_tokens, a.do_expand != 0, rc.recv_fp8 != 0, ctas, a.cached != 0);
    const int which = shape.mode * 4 + (rc.recv_fp8 != 0 ? 2 : 0) + (shape.pooled ? 1 : 0);
    const auto kernel = kernels[which];
    static std::mutex mutex;
    static std::size_t configured[12][64] = {{0}};
    {
        std::lock_guard<std::mutex> guard(mutex);
        int device = 0;
        cudaError_t status = cudaGetDevice(&device);
        if (status != cudaSuccess) return status;
        if (device < 0 || device >= 64) return cudaErrorInvalidDevice;
        if (shape.bytes > configured[which][device]) {
            status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(shape.bytes));
            if (status != cudaSuccess) return status;
            configured[which][device] = shape.bytes;
        }
    }
    LocalDispatchArgs args{a, shape.plan, hist, counters, sms, rc.lay.num_experts, rc.lay.num_channels, rc.lay.num_topk, rc.lay.hidden,
                           rc.lay.slots_full, rc.expanded_cap, rc.unique_cap, shape.once};
    // A CTA waits for others at the barrier of a layout that they count together, and for their plans where tokens are claimed:
    // then every CTA has to be resident.  With a cached layout (whose plan is there) and with a small batch no CTA waits.
    if (shape.mode != kLocalCached && (shape.mode == kLocalTogether || shape.pooled)) return cooperative_launch(kernel, args, dim3(ctas), kLocalThreads, shape.bytes, stream);
    kernel<<<ctas, kLocalThreads, shape.bytes, stream>>>(args);
    return cudaGetLastError();
}

cudaError_t launch_combine_local(const CombineLocalArgs& args, cudaStream_t stream) {
    const auto kernel = args.shape.batch == 1 && !args.shape.fixed ? local_combine_push_kernel<1> : local_combine_push_kernel<4>;
    static std::mutex mutex;
    static std::size_t configured[64] = {0};
    {
        std::lock_guard<std::mutex> guard(mutex);
        int device = 0;
        cudaError_t status = cudaGetDevice(&device);
        if (status != cudaSuccess) return status;
        if (device < 0 || device >= 64) return cudaErrorInvalidDevice;
        if (args.shape.bytes > configured[device]) {
            status = cudaFuncSetAttribute(local_combine_push_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(args.shape.bytes));
            if (status == cudaSuccess)
                status = cudaFuncSetAttribute(local_combine_push_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(args.shape.bytes));
            if (status != cudaSuccess) return status;
            configured[device] = args.shape.bytes;
        }
    }
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(static_cast<unsigned>(args.shape.ctas));
    config.blockDim = dim3(kCombineLocalThreads);
    config.dynamicSmemBytes = args.shape.bytes;
    config.stream = stream;
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // its CTAs come where those of the expert GEMM have ended
    attribute[0].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attribute;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, args);
}

cudaError_t launch_combine(const CombineLaunch& launch, int channels, std::size_t crow_stride, cudaStream_t stream) {
    const std::size_t smem = static_cast<std::size_t>(kCombineWarps) * crow_stride;
    static std::mutex mutex;
    static std::size_t configured[64] = {0};
    {
        std::lock_guard<std::mutex> guard(mutex);
        int device = 0;
        cudaError_t status = cudaGetDevice(&device);
        if (status != cudaSuccess) return status;
        if (device >= 0 && device < 64 && smem > configured[device]) {
            status = cudaFuncSetAttribute(combine_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
            if (status != cudaSuccess) return status;
            configured[device] = smem;
        }
    }
    return cooperative_launch(combine_kernel, launch, dim3(channels, launch.num_virtual, 1), kCombineWarps * 32, smem, stream);
}

cudaError_t launch_combine_push(const CombinePushArgs& args, int reduce_ctas, std::size_t smem, cudaStream_t stream) {
    static std::mutex mutex;
    static std::size_t configured[64] = {0};
    {
        std::lock_guard<std::mutex> guard(mutex);
        int device = 0;
        cudaError_t status = cudaGetDevice(&device);
        if (status != cudaSuccess) return status;
        if (device >= 0 && device < 64 && smem > configured[device]) {
            status = cudaFuncSetAttribute(combine_push_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
            if (status != cudaSuccess) return status;
            configured[device] = smem;
        }
    }
    combine_push_kernel<<<args.forward_ctas + reduce_ctas, kFusedReduceThreads, smem, stream>>>(args);
    return cudaGetLastError();
}

cudaError_t launch_fused_reduce(const FusedReduceArgs& args, int ctas, cudaStream_t stream) {
    switch (fused_reduce_groups(args.slots)) {
        case 4: fused_reduce_kernel<4><<<ctas, kFusedReduceThreads, 0, stream>>>(args); break;
        case 2: fused_reduce_kernel<2><<<ctas, kFusedReduceThreads, 0, stream>>>(args); break;
        default: fused_reduce_kernel<1><<<ctas, kFusedReduceThreads, 0, stream>>>(args); break;
    }
    return cudaGetLastError();
}

}  // namespace bep
