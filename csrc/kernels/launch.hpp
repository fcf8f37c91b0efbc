// Host-callable entry points of the CUDA translation unit (csrc/kernels/launch.cu).  The runtime
// (plain C++, built without nvcc) only sees these.
#pragma once

#include <cstddef>

#include <cuda_runtime.h>

#include "combine_local.cuh"
#include "combine_push.cuh"
#include "fused_reduce.cuh"
#include "protocol.cuh"

namespace bep {

// Shared-memory bytes the dispatch kernel needs for this configuration (`stages` row buffers per send warp).
std::size_t dispatch_shared_bytes(const SegmentLayout& lay, int tx_warps, int rx_warps, bool use_tma, int stages,
                                  int send_ctas);

// Raise (never lower) the kernels' dynamic shared-memory limit; thread-safe, idempotent.
cudaError_t configure_kernels(std::size_t dispatch_smem_bytes);

// How many CTAs of `threads` threads and `smem` dynamic bytes fit on the current device at once.
int dispatch_resident_ctas(int threads, std::size_t smem);
int combine_resident_ctas(int threads);

// Cooperative launches: grid = (CTAs per rank, virtual ranks); dispatch: channels + dedicated sender CTAs.
cudaError_t launch_dispatch(const DispatchLaunch& launch, int ctas, int threads, std::size_t smem,
                            cudaStream_t stream);
cudaError_t launch_combine(const CombineLaunch& launch, int channels, std::size_t crow_stride, cudaStream_t stream);

// A group of one rank: how the local dispatch kernel cuts up shared memory, the ints of its scratch, and the two launches.
// `rc` is the host's copy of the rank's constants, `sms` is what the scratch was made for, `max_ctas` bounds the CTAs; `counters` and
// `hist` belong to one buffer, whose launches are stream-ordered.  `shape_dispatch_local`: which kernel `ctas` CTAs run, and with what.
LocalPlan plan_dispatch_local(const SegmentLayout& lay, int sms, std::size_t smem_limit, long long l2_bytes);
std::size_t dispatch_local_hist_ints(const SegmentLayout& lay, int ctas);
// CTAs that a dispatch has work for: one per token, or one per expert where the rows between their segments are zeroed.
int dispatch_local_width(const SegmentLayout& lay, int tokens, bool padding);
LocalShape shape_dispatch_local(const SegmentLayout& lay, const LocalPlan& plan, int tokens, bool expand, bool recv_fp8, int ctas, bool cached);
cudaError_t launch_dispatch_local(const DispatchArgs& a, const RankConst& rc, const LocalPlan& plan, int* hist, unsigned long long* counters, int sms, int max_ctas,
                                  cudaStream_t stream);
cudaError_t launch_combine_local(const CombineLocalArgs& args, cudaStream_t stream);

// Ordinary launches of the combine paths: expert-side gather-reduce-push, owner-side sum.  Any grid size works.
// `reduce_ctas` reducer CTAs follow the args.forward_ctas forwarder CTAs in one grid.
cudaError_t launch_combine_push(const CombinePushArgs& args, int reduce_ctas, std::size_t smem, cudaStream_t stream);
cudaError_t launch_fused_reduce(const FusedReduceArgs& args, int ctas, cudaStream_t stream);
// True when the library was built with the per-role instrumentation (-DBEP_ENABLE_PROFILING=1).
bool role_profiling_enabled();

}  // namespace bep
