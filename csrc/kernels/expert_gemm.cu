// tcgen05 grouped expert GEMM: device code and launcher.  See expert_gemm.cuh for the design.
#include "expert_gemm.cuh"

#include <mutex>
#include <type_traits>

#include "expert_gemm.hpp"
#include "ptx.cuh"

namespace bep {
namespace gemm {

namespace {

// ---- PTX wrappers ---------------------------------------------------------------------------
__device__ __forceinline__ std::uint32_t smem_addr(const void* p) {
    return static_cast<std::uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(std::uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(std::uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(std::uint64_t* bar, unsigned parity) {
    std::uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// bounded wait; returns false (and latches *abort) when the limit is hit or somebody else aborted
__device__ __forceinline__ bool mbar_wait(std::uint64_t* bar, unsigned parity, volatile int* abort) {
    for (std::uint32_t i = 0; i < kWaitLimit; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 1023u) == 1023u && *abort) return false;
    }
    *abort = 1;
    return false;
}

// address of the same shared-memory location in CTA `rank` of the cluster
__device__ __forceinline__ std::uint32_t cluster_addr(const void* p, unsigned rank) {
    std::uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_addr(p)), "r"(rank));
    return remote;
}
__device__ __forceinline__ void mbar_arrive_cluster(std::uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// True in one lane of a converged warp.  Behind a branch on it the compiler knows that tcgen05 and TMA instructions, whose operands are
// uniform registers, are issued once; behind `lane == 0` it does not, and an MMA of a pair took 145 cycles to issue, longer than one of
// 256 x 256 x 16 takes to execute (127).  One pair alone, per K block of 64: 16 to 128 rows 285 -> 131 to 138 ns (weights into an SM at 57 ->
// 125 GB/s), 192 rows 282 -> 207.  64 tokens, top-8 of 32 experts, 7168 x 2048: layer 467 -> 449 us; 555 tokens in E4M3, popular experts,
// 495 -> 458; 4096 tokens in E4M3 1935 -> 1845.  Under the power limit 32 experts of 1024 rows, 7168 -> 4096: 1,205 -> 1,255 TFLOP/s at 1,080
// instead of 1,100 MHz (torch.bmm 1,305 at 1,170).
__device__ __forceinline__ bool elect_one() {
    std::uint32_t elected;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(elected)::"memory");
    return elected != 0;
}
// kPauseLoads loads from shared memory, each at the address that the one before gives: `zero_at` holds a zero.
__device__ __forceinline__ void pause(std::uint32_t& zero_at) {
#pragma unroll
    for (int i = 0; i < kPauseLoads; ++i) {
        std::uint32_t zero;
        asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(zero) : "r"(zero_at) : "memory");
        zero_at += zero;
    }
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Tiled TMA loads, no multicast: the box lands in this CTA's shared memory with the tensor map's swizzle, its bytes are
// counted on `bar`, which may be the other CTA's of the pair.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, int x, int y, std::uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_addr(smem_dst)), "l"(reinterpret_cast<std::uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tma_load_5d(void* smem_dst, const CUtensorMap* map, int x, int group, int expert, std::uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.5d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %3, %4, %5}], [%6];"
        ::"r"(smem_addr(smem_dst)), "l"(reinterpret_cast<std::uint64_t>(map)), "r"(x), "r"(0), "r"(group), "r"(expert), "r"(bar)
        : "memory");
}

__device__ __forceinline__ void tmem_alloc(std::uint32_t* smem_result, unsigned columns) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(smem_result)), "r"(columns)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(std::uint32_t taddr, unsigned columns) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(columns) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[tmem of both CTAs] (+)= A[smem desc] * B[smem desc]; one thread of the leading CTA issues for the pair
template <bool kFp8>
__device__ __forceinline__ void umma(std::uint32_t tmem_d, std::uint64_t desc_a, std::uint64_t desc_b, std::uint32_t idesc, std::uint32_t accumulate) {
    if constexpr (kFp8)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
            : "memory");
}
// all MMAs issued so far by this thread arrive on `bar` of both CTAs when they have completed
__device__ __forceinline__ void umma_commit_pair(std::uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_addr(bar)),
                 "h"(static_cast<std::uint16_t>(3))
                 : "memory");
}
// 16 lanes x 32 columns: thread t gets, for j = 0..3, columns 8j + 2(t % 4) + {0, 1} of lane t / 4 in r[4j], r[4j + 1] and of lane
// t / 4 + 8 in r[4j + 2], r[4j + 3]: the fragments that stmatrix stores
__device__ __forceinline__ void tmem_ld_16x32(std::uint32_t taddr, std::uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr)
                 : "memory");
}
// four transposed 8 x 8 matrices of 16-bit values: lane l gives the address of row l % 8 of matrix l / 8
__device__ __forceinline__ void stmatrix_transposed(std::uint32_t addr, std::uint32_t m0, std::uint32_t m1, std::uint32_t m2, std::uint32_t m3) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(m0), "r"(m1), "r"(m2), "r"(m3) : "memory");
}
// (the registers pass through, so that nothing reads or copies them before the loads have arrived)
__device__ __forceinline__ void tmem_ld_wait(std::uint32_t (&r)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                   "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]),
                   "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]),
                   "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])::"memory");
}

// barrier among the four epilogue warps; true when `ok` held in all of them
__device__ __forceinline__ bool epilogue_all(bool ok) {
    std::uint32_t all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.and.pred.aligned q, 1, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(all)
        : "r"(static_cast<std::uint32_t>(ok))
        : "memory");
    return all != 0;
}
__device__ __forceinline__ void epilogue_sync() { asm volatile("barrier.cta.sync.aligned 1, 128;" ::: "memory"); }

// Shared-memory matrix descriptor of a K-major tile whose rows are 128 bytes (64 bf16) wide, stored
// with the 128-byte swizzle TMA applied: 8-row groups are 1024 bytes apart (stride byte offset), the
// leading byte offset is unused for swizzled K-major operands, descriptor version 1 (sm_100),
// layout type 2 = SWIZZLE_128B.
__device__ __forceinline__ std::uint64_t make_smem_desc(const void* tile) {
    const std::uint64_t addr = smem_addr(tile);
    std::uint64_t desc = 0;
    desc |= (addr & 0x3FFFFull) >> 4;                 // bits  0..13 start address / 16
    desc |= static_cast<std::uint64_t>(0) << 16;      // bits 16..29 leading byte offset / 16
    desc |= static_cast<std::uint64_t>(1024 >> 4) << 32;  // bits 32..45 stride byte offset / 16
    desc |= static_cast<std::uint64_t>(1) << 46;      // bits 46..47 descriptor version
    desc |= static_cast<std::uint64_t>(2) << 61;      // bits 61..63 swizzle mode: 128B
    return desc;
}

// Instruction descriptor, D = F32, both operands K-major, N and M encoded /8 and /16; kind::f16 with A = B = BF16, or
// kind::f8f6f4 with E4M3 operands (format code 0 for both).
template <bool kFp8>
__host__ __device__ constexpr std::uint32_t make_idesc(int m, int n) {
    return (1u << 4)                                   // D format: F32
           | (kFp8 ? 0u : (1u << 7) | (1u << 10))      // A and B format: BF16
           | (static_cast<std::uint32_t>(n >> 3) << 17)
           | (static_cast<std::uint32_t>(m >> 4) << 24);
}

// Walks every pairs-th tile in the order expert, group of eight row chunks, channel tile, row chunk, so that tiles which run at the same
// time share a weight tile.  Eight chunks by nine channel tiles is what 74 pairs can read the least for; with all chunks of an expert in
// one group 74 pairs were at work on as many chunks and read the rows again for every channel tile: one expert of 16384 rows, 7168 -> 4096,
// 920 -> 738 us under the power limit (709 -> 622 without), 8 experts of 4096 rows, gate/up 7168 -> 2048, 1506 -> 1464.  Groups of two lose 3 %
// at 32 experts of 1024 rows, groups of four 1.5 % at 8 x 4096; channel tiles in groups of eight instead lose 5 % at 32 x 1024.
constexpr int kChunkGroup = 8;
struct TileWalk {
    int tile, pairs, m_tiles;
    int next_expert = 0, rows = 0, first_row = 0, first_tile = 0, end_tile = 0;  // of the present expert
    RowChunks chunks{0, 0};
    // the present tile: channel tile, row chunk, first row of the activations, valid rows
    int expert = 0, m_tile = 0, chunk = 0, row0 = 0, tile_rows = 0;

    __device__ __forceinline__ explicit TileWalk(int m_tiles_) : tile(blockIdx.x >> 1), pairs(gridDim.x >> 1), m_tiles(m_tiles_) {}

    __device__ __forceinline__ bool next(const GroupedGemmParams& p) {
        while (tile >= end_tile) {
            if (next_expert >= p.num_experts) return false;
            expert = next_expert++;
            rows = p.expert_counts[expert];
            chunks = row_chunks(rows);
            first_tile = end_tile;
            end_tile += chunks.count * m_tiles;
            first_row = p.expert_offsets[expert];
        }
        const int local = tile - first_tile;
        const int group = local / (kChunkGroup * m_tiles), in_group = local - group * kChunkGroup * m_tiles;
        const int wide = min(kChunkGroup, chunks.count - group * kChunkGroup);
        m_tile = in_group / wide;
        chunk = group * kChunkGroup + in_group - m_tile * wide;
        row0 = first_row + chunk * chunks.rows;
        tile_rows = min(chunks.rows, rows - chunk * chunks.rows);
        tile += pairs;
        return true;
    }
};

}  // namespace

namespace {
// waits (bounded) until the launch before has written all rows of an expert
__device__ __noinline__ bool rows_written(const GroupedGemmParams& p, int expert, unsigned tiles, volatile int* abort) {
    const auto* counter = reinterpret_cast<const std::uint32_t*>(p.progress.counters + expert);
    unsigned long long deadline = 0;
    for (unsigned polls = 1; ptx::ld_acquire_gpu(counter) < tiles; ++polls) {
        if (polls % 64 == 0) {
            const unsigned long long now = ptx::globaltimer_ns();
            if (deadline == 0) deadline = now + p.progress.timeout_ns;
            if (*abort || now > deadline) {
                *abort = 1;
                return false;
            }
        }
        ptx::nanosleep(100);
    }
    asm volatile("fence.proxy.async.global;" ::: "memory");
    return true;
}
}  // namespace

// Launch bounds: at most 128 registers, so that a reducer CTA of the combine (combine_push.cuh) finds room on this CTA's SM.
template <bool kSwiGLU, bool kFp8, bool kScatter>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(256, 2)
grouped_gemm_kernel(const __grid_constant__ ActivationMaps maps_rows, const __grid_constant__ CUtensorMap map_w,
                    const GroupedGemmParams p) {
    static_assert(!kScatter || (!kSwiGLU && !kFp8), "the scatter epilogue exists for the plain BF16 GEMM");
    constexpr int kElemBytes = kFp8 ? 1 : 2;
    constexpr int kBlockK = kBlockKBytes / kElemBytes;  // elements of K per stage
    constexpr int kChannels = kSwiGLU ? kCtaM / 2 : kCtaM;  // output channels of one CTA in a tile
    constexpr int kPitch = staging_pitch(kSwiGLU);

    extern __shared__ __align__(1024) unsigned char smem_unaligned[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<std::uintptr_t>(smem_unaligned) + 1023) & ~std::uintptr_t(1023));
    unsigned char* tiles = smem;
    unsigned char* staging = smem + kRingBytes;
    auto* sh = reinterpret_cast<GemmShared*>(staging + 2 * kChunkRows * kPitch);
    auto* row_factors = reinterpret_cast<float*>(sh + 1);                                        // [2][kMaxRows] scatter and E4M3
    auto* row_targets = reinterpret_cast<unsigned long long*>(row_factors + 2 * kMaxRows);       // [2][kMaxRows] scatter
    volatile int* abort = &sh->abort;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const unsigned rank = cluster_rank();
    const int k_blocks = p.k / kBlockK;
    const int m_tiles = (p.n + 2 * kChannels - 1) / (2 * kChannels);

    if (warp == 0 && lane < kBoxes + 1) {
        const CUtensorMap* map = lane < kBoxes ? &maps_rows.box[lane] : &map_w;
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<std::uint64_t>(map)) : "memory");
    }
    if (threadIdx.x == 64) {
        for (int s = 0; s < kMaxStages; ++s) {
            mbar_init(&sh->full[s], 1);
            mbar_init(&sh->empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&sh->tmem_full[b], 1);
            mbar_init(&sh->tmem_empty[b], 8);
        }
        *abort = 0;
        sh->zero = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        tmem_alloc(&sh->tmem_base, kTmemCols);
        tmem_relinquish();
    }
    // Up to here nothing was read that an earlier launch writes: the launch behind another kernel of the layer gets this far while
    // the last CTAs of that one are still at work (a layer of 64 tokens 459 -> 454 us, of which two launches gain).  What is read from
    // here on is read by ordinary loads, which stay behind the wait (ld.global.nc need not).
    const bool second = p.progress.per_chunk != 0;  // of two linked launches: see Progress
    if (!second) ptx::wait_for_launch_before();
    ptx::let_next_launch_start();
    int most_rows = 1, all_rows = 0;  // of any expert, of all
    for (int e = threadIdx.x; e < p.num_experts; e += kThreads) {
        asm volatile("prefetch.global.L1 [%0];" ::"l"(p.expert_offsets + e));  // asked for again at the first tile
        const int rows = p.expert_counts[e];
        most_rows = max(most_rows, rows);
        all_rows += rows;
    }
    most_rows = __reduce_max_sync(0xffffffffu, most_rows);
    all_rows = __reduce_add_sync(0xffffffffu, all_rows);
    if (lane == 0) {
        sh->most_rows[warp] = most_rows;
        sh->all_rows[warp] = all_rows;
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // barriers of both CTAs are ready before either names the other's
    tc_fence_after();
    const std::uint32_t tmem_base = sh->tmem_base;
    all_rows = 0;
    for (int w = 0; w < kThreads / 32; ++w) {
        most_rows = max(most_rows, sh->most_rows[w]);
        all_rows += sh->all_rows[w];
    }
    const int stage_bytes = kTileW + box_rows(box_of_rows(min(most_rows, kMaxRows))) * kBlockKBytes;
    const int stages = min(kMaxStages, kRingBytes / stage_bytes);
    TileWalk walk(m_tiles);

    if (warp == 0) {
        // ===== TMA producer: this CTA's 128 weight rows and its half of the activation rows =====
        if (elect_one()) {
            int stage = 0;
            unsigned phase = 0;
            bool ok = true;
            int ready = -1;  // second launch: expert whose rows are known to be there
            while (ok && walk.next(p)) {
                if (second && walk.expert != ready) {
                    ok = rows_written(p, walk.expert, static_cast<unsigned>(walk.chunks.count * p.progress.per_chunk), abort);
                    if (!ok) break;
                    ready = walk.expert;
                }
                const int box = box_of_rows(walk.tile_rows);
                const int half = box_rows(box);
                const CUtensorMap* map_rows = &maps_rows.box[box];
                const int row = walk.row0 + static_cast<int>(rank) * half;
                const unsigned pair_bytes = 2u * static_cast<unsigned>(kTileW + half * kBlockKBytes);
                const int group = (walk.m_tile * 2 + static_cast<int>(rank)) * (kChannels / 16);
                const int wrow = walk.expert * p.n + (walk.m_tile * 2 + static_cast<int>(rank)) * kCtaM;
                for (int kb = 0; kb < k_blocks; ++kb) {
                    if (!mbar_wait(&sh->empty[stage], phase ^ 1u, abort)) {
                        ok = false;
                        break;
                    }
                    unsigned char* stage_base = tiles + stage * stage_bytes;
                    if (rank == 0) mbar_expect_tx(&sh->full[stage], pair_bytes);
                    const std::uint32_t bar = cluster_addr(&sh->full[stage], 0);
                    if (kSwiGLU) tma_load_5d(stage_base, &map_w, kb * kBlockK, group, walk.expert, bar);
                    else tma_load_2d(stage_base, &map_w, kb * kBlockK, wrow, bar);
                    tma_load_2d(stage_base + kTileW, map_rows, kb * kBlockK, row, bar);
                    if (++stage == stages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
            }
            // the other roles have taken every stage (and the leading CTA's commits have arrived here) before this CTA ends
            for (int i = 0; ok && i < stages; ++i) {
                ok = mbar_wait(&sh->empty[stage], phase ^ 1u, abort);
                if (++stage == stages) {
                    stage = 0;
                    phase ^= 1u;
                }
            }
            // gave up: what is still on its way gets time to land before shared memory goes away
            if (!ok)
                for (int i = 0; i < 1000; ++i) ptx::nanosleep(1000);
        }
    } else if (warp == 1) {
        // ===== MMA issuer of the pair =====
        auto issue = [&](auto paced) {
            int stage = 0;
            std::uint32_t zero_at = smem_addr(&sh->zero);
            unsigned phase = 0;
            bool ok = true;
            int it = 0;
            for (; ok && walk.next(p); ++it) {
                const int buf = it & 1;
                const unsigned acc_phase = (it >> 1) & 1u;
                if (!mbar_wait(&sh->tmem_empty[buf], acc_phase ^ 1u, abort)) break;
                tc_fence_after();
                const std::uint32_t acc = tmem_base + buf * kAccCols;
                const std::uint32_t idesc = make_idesc<kFp8>(2 * kCtaM, 2 * box_rows(box_of_rows(walk.tile_rows)));
                for (int kb = 0; kb < k_blocks; ++kb) {
                    if (!mbar_wait(&sh->full[stage], phase, abort)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const std::uint64_t desc_w = make_smem_desc(tiles + stage * stage_bytes);
                    const std::uint64_t desc_rows = make_smem_desc(tiles + stage * stage_bytes + kTileW);
#pragma unroll
                    for (int k = 0; k < kBlockKBytes / kUmmaKBytes; ++k) {
                        // 32 bytes further along K inside the swizzle atom: +2 in the address field
                        const std::uint64_t step = static_cast<std::uint64_t>(k * kUmmaKBytes) >> 4;
                        if (decltype(paced)::value && k % 2 == 0) pause(zero_at);
                        umma<kFp8>(acc, desc_w + step, desc_rows + step, idesc, (kb | k) != 0 ? 1u : 0u);
                    }
                    umma_commit_pair(&sh->empty[stage]);  // the stage is free in both CTAs once these MMAs have read it
                    if (++stage == stages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
                if (ok) umma_commit_pair(&sh->tmem_full[buf]);
            }
        };
        // Long BF16 gate/up launches pause in front of every second MMA.  Without a gap the MMAs draw so much power that what follows runs at
        // the lower clock it leaves behind.  4096 tokens, 32 experts, 7168 -> 2 x 2048, for seconds, us without / with the pause: gate/up 1722 /
        // 1720 inside the layer, down projection 1025 / 842, dispatch 148 / 127, combine 162 / 133.  Layers, a few passes (and for seconds), by
        // rows x channels x K of one matrix: 2.4e11 1240 / 1258 (1561 / 1499), 2.7e11 hidden 4096 1275 / 1300 (1551 / 1506), hidden 2048 1227 /
        // 1261 (1429 / 1454), 2.9e11 1436 / 1475 (1787 / 1761), 3.5e11 1712 / 1688 (2119 / 2064), 16 experts with the fused down projection
        // 1672 / 1630 (1995 / 1899), 4.0e11 hidden 4096 1835 / 1801 (2237 / 2094), 5.5e11 2431 / 2431 (2953 / 2828); 1.6e11 893 / 946.  The price
        // is the launch by itself, 32 x 1024 rows 1296 / 1324 us, for seconds 1497 / 1550.  (One load in front of every MMA leaves half of the gain,
        // two in front of each or three cost 5 to 15 %; a gap by the clock register, between K blocks or MMAs, 9 to 20 %.  E4M3 and the down
        // projection gain without.)
        if (rank == 0) {
            if (!kFp8 && kSwiGLU && static_cast<long long>(all_rows) * p.n * p.k >= kLongLaunchPerSm * gridDim.x) {
                if (elect_one()) issue(std::true_type());
            } else if (elect_one()) {
                issue(std::false_type());
            }
        }
    } else {
        // ===== epilogue: 4 warps, warp q owns TMEM lanes [32q, 32q+32); lane = weight row, column = activation row =====
        const int q = warp & 3;
        const ScatterTarget& sc = p.scatter;
        if (kScatter) {
            // every rank must have summed the previous call's rows before its landing area is overwritten
            if (lane < sc.num_ranks) {
                const auto* flag = reinterpret_cast<const std::uint64_t*>(sc.seg[sc.rank] + sc.done_off +
                                                                          static_cast<std::size_t>(lane) * sc.flag_stride);
                const std::uint64_t deadline = ptx::globaltimer_ns() + sc.timeout_ns;
                unsigned polls = 0;
                while (ptx::ld_acquire_sys(flag) + 1 < sc.epoch) {
                    if ((++polls & 63u) == 0 && (*abort || ptx::globaltimer_ns() > deadline)) {
                        if (!*abort) atomicCAS(&p.status[0], 0, 3);
                        *abort = 1;
                        break;
                    }
                    ptx::nanosleep(64);
                }
            }
            __syncwarp();
        }
        const std::uint32_t empty_addr = cluster_addr(&sh->tmem_empty[0], 0);  // in the leading CTA
        constexpr int kLanesPerRow = kChannels / 8;             // 16-byte pieces of a row
        constexpr int kRowsPerStore = 32 / kLanesPerRow;
        const int piece = lane % kLanesPerRow, store_row = q * (kChunkRows / 4) + lane / kLanesPerRow;
        // What belongs to the rows of a tile (scatter: where they go and their weights; E4M3: their scales), two rows per thread, is asked
        // for a tile ahead.  Asked for in their own chunk, every 32 rows waited for L2, and the epilogue was longer than the MMAs of its
        // tile: 2000 tokens, top-8 of 32 experts, 768 -> 2048, scattered down projection and sum 107 -> 91 us.
        constexpr bool kRowFactors = kScatter || kFp8;
        TileWalk ahead = walk;
        int owner[2], token[2], slot[2];
        float factor[2];
        auto ask_rows = [&]() {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int in_tile = static_cast<int>(threadIdx.x) - 64 + 128 * i;
                owner[i] = -1;
                if (in_tile >= ahead.tile_rows) continue;
                const long long r = static_cast<long long>(ahead.row0) + in_tile;
                if constexpr (kScatter) {
                    const long long* meta = sc.source_meta + r * 3;
                    owner[i] = static_cast<int>(meta[0]);
                    token[i] = static_cast<int>(meta[1]);
                    slot[i] = static_cast<int>(meta[2]);
                    factor[i] = sc.row_weights != nullptr ? sc.row_weights[r] : 1.0f;
                } else {
                    factor[i] = p.a_scales[r];
                }
            }
        };
        // into shared memory: what was there was read two tiles ago, and all warps have met since then (epilogue_all)
        auto store_rows = [&](int rows, int buf, int first_channel) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int in_tile = static_cast<int>(threadIdx.x) - 64 + 128 * i;
                if (in_tile >= rows) continue;
                row_factors[buf * kMaxRows + in_tile] = factor[i];
                if constexpr (kScatter) {
                    unsigned long long dst = 0;
                    if (owner[i] >= 0 && owner[i] < sc.num_ranks && slot[i] >= 0 && slot[i] < sc.num_topk && token[i] >= 0)
                        dst = reinterpret_cast<unsigned long long>(sc.seg[owner[i]] + sc.stage_off +
                                                                   (static_cast<std::size_t>(token[i]) * sc.num_topk + slot[i]) * static_cast<std::size_t>(sc.row_stride) +
                                                                   static_cast<std::size_t>(first_channel) * 2);
                    row_targets[buf * kMaxRows + in_tile] = dst;
                }
            }
        };
        if (kRowFactors && ahead.next(p)) ask_rows();
        int it = 0, half = 0;
        for (; walk.next(p); ++it) {
            const int buf = it & 1;
            const unsigned acc_phase = (it >> 1) & 1u;
            const int first_channel = (walk.m_tile * 2 + static_cast<int>(rank)) * kChannels;
            const bool inside = first_channel < p.n;  // n an odd multiple of 128: the last tile has one CTA's channels only
            // E4M3: scales of the weight rows of this thread's channels, lane / 4 + 8 i of its warp's (SwiGLU: two gate, then two up rows)
            float w_scale[4] = {1.0f, 1.0f, 1.0f, 1.0f};
            if (kFp8 && inside) {
                const float* at = p.w_scales + static_cast<long long>(walk.expert) * (kSwiGLU ? 2 : 1) * p.n + first_channel + q * (kChannels / 4) + (lane >> 2);
#pragma unroll
                for (int i = 0; i < 4; ++i) w_scale[i] = kSwiGLU ? at[(i >> 1) * p.n + (i & 1) * 8] : at[i * 8];
            }
            if (kRowFactors) {
                store_rows(walk.tile_rows, buf, first_channel);
                if (ahead.next(p)) ask_rows();
            }
            // all four warps go on or none: they meet at the barriers below
            if (!epilogue_all(mbar_wait(&sh->tmem_full[buf], acc_phase, abort))) break;
            tc_fence_after();
            const std::uint32_t acc = tmem_base + (static_cast<std::uint32_t>(q * 32) << 16) + buf * kAccCols;
            // (2) of a chunk, see below: a few lanes = one row, its channels of this CTA leave as contiguous 16-byte pieces
            auto store_chunk = [&](int c0) {
                epilogue_sync();
#pragma unroll
                for (int i = 0; i < kChunkRows / 4; i += kRowsPerStore) {
                    const int r = store_row + i;
                    unsigned char* dst = nullptr;
                    if (c0 + r < walk.tile_rows && inside) {
                        if constexpr (kScatter) dst = reinterpret_cast<unsigned char*>(row_targets[buf * kMaxRows + c0 + r]);
                        else dst = reinterpret_cast<unsigned char*>(p.out + static_cast<long long>(walk.row0 + c0 + r) * p.n + first_channel);
                    }
                    const uint4 packed = *reinterpret_cast<const uint4*>(staging + (half * kChunkRows + r) * kPitch + piece * 16);
                    if (dst != nullptr) ptx::st_v4(dst + piece * 16, packed);
                }
                half ^= 1;  // the other half was read before the barrier above
            };
#pragma unroll 1
            for (int c0 = 0; c0 < walk.tile_rows; c0 += kChunkRows) {
                // v[16 h + 4 j + 2 i + x]: weight row 16 h + 8 i + lane / 4 of the warp's 32, activation row c0 + 8 j + 2 (lane % 4) + x
                std::uint32_t v[32];
                tmem_ld_16x32(acc + c0, v);
                tmem_ld_16x32(acc + (16u << 16) + c0, v + 16);
                float2 factors[4];  // of the rows that this thread's registers hold
                if constexpr (kRowFactors)
#pragma unroll
                    for (int j = 0; j < 4; ++j) factors[j] = *reinterpret_cast<const float2*>(&row_factors[buf * kMaxRows + c0 + 8 * j + 2 * (lane & 3)]);
                if (c0 > 0) store_chunk(c0 - kChunkRows);  // the chunk before leaves while this one's values are on their way
                tmem_ld_wait(v);
                if (c0 + kChunkRows >= walk.tile_rows) {
                    // the accumulator has been read completely: the MMA warp may start the tile after next
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(empty_addr + buf * 8);
                }
                // (1) 8 rows x 8 channels at a time turned round through shared memory by matrix stores: lane = channel -> staging[row][channel].
                // (A lane per channel with 32 stores of 2 bytes, and as many shuffles of the rows' factors or between gate and up, was slower
                // where K is short: 32 experts of 500 rows, 768 -> 2048 69.9 -> 61.9 us, gate/up 2048 -> 768 97.7 -> 91.5, in E4M3 81.9 -> 76.4.)
                if constexpr (kSwiGLU) {
                    // gate (h = 0) and up (h = 1) of a channel are in one thread
                    const std::uint32_t at = smem_addr(staging + (half * kChunkRows + (lane >> 4) * 8 + (lane & 7)) * kPitch + (q * 16 + (lane >> 3 & 1) * 8) * 2);
#pragma unroll
                    for (int j0 = 0; j0 < 4; j0 += 2) {
                        std::uint32_t m[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int j = j0 + (i >> 1), first = 4 * j + (i & 1) * 2;
                            float silu[2];
#pragma unroll
                            for (int x = 0; x < 2; ++x) {
                                float gate = __uint_as_float(v[first + x]), up = __uint_as_float(v[16 + first + x]);
                                if (kFp8) {
                                    const float a_scale = x == 0 ? factors[j].x : factors[j].y;
                                    gate *= a_scale * w_scale[i & 1];
                                    up *= a_scale * w_scale[2 + (i & 1)];
                                }
                                silu[x] = ptx::quotient(gate, 1.0f + __expf(-gate)) * up;
                            }
                            const __nv_bfloat162 packed = __floats2bfloat162_rn(silu[0], silu[1]);
                            m[i] = *reinterpret_cast<const std::uint32_t*>(&packed);
                        }
                        stmatrix_transposed(at + 8 * j0 * kPitch, m[0], m[1], m[2], m[3]);
                    }
                } else {
                    const std::uint32_t at = smem_addr(staging + (half * kChunkRows + (lane & 7)) * kPitch + (q * 32 + (lane >> 3) * 8) * 2);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        std::uint32_t m[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int first = (i >> 1) * 16 + 4 * j + (i & 1) * 2;
                            float a = __uint_as_float(v[first]), b = __uint_as_float(v[first + 1]);
                            if (kScatter) {
                                a *= factors[j].x;
                                b *= factors[j].y;
                            } else if (kFp8) {
                                a *= factors[j].x * w_scale[i];
                                b *= factors[j].y * w_scale[i];
                            }
                            const __nv_bfloat162 packed = __floats2bfloat162_rn(a, b);
                            m[i] = *reinterpret_cast<const std::uint32_t*>(&packed);
                        }
                        stmatrix_transposed(at + 8 * j * kPitch, m[0], m[1], m[2], m[3]);
                    }
                }
            }
            store_chunk((walk.tile_rows - 1) / kChunkRows * kChunkRows);
            if (!kScatter && p.progress.counters != nullptr && !second) {
                // this CTA's part of the tile, for the TMA loads of other SMs
                asm volatile("fence.proxy.async.global;" ::: "memory");
                __threadfence();
                epilogue_sync();
                if (threadIdx.x == 64) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p.progress.counters + walk.expert) : "memory");
            }
        }
        if (kScatter) ptx::fence_sys();  // this thread's rows before the CTA is counted as finished
    }

    // ---- teardown: every role has left its loop (normally or through the abort latch)
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // nothing of the other CTA names this one's shared memory any more
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kTmemCols);
    }
    if (threadIdx.x == 0 && *abort) atomicCAS(&p.status[0], 0, 1);
    if (second) {
        ptx::wait_for_launch_before();  // whoever waits for this launch has waited for the first one, too
        if (threadIdx.x == 0) {
            __threadfence();
            if (atomicAdd(p.progress.counters + p.num_experts, 1u) + 1u == gridDim.x)
                for (int e = 0; e <= p.num_experts; ++e) p.progress.counters[e] = 0u;
        }
    }
    if (kScatter && threadIdx.x == 0) {
        const ScatterTarget& sc = p.scatter;
        ptx::fence_sys();
        const unsigned long long finished = atomicAdd(sc.cta_done, 1ull) + 1ull;
        if (finished == gridDim.x) {
            // last CTA of this launch: all rows of all CTAs are written; tell every owner (unless something gave up).
            // Launches that share the counter are stream-ordered, so the next one finds it at zero again.
            *sc.cta_done = 0ull;
            ptx::fence_sys();
            if (*reinterpret_cast<volatile int*>(p.status) == 0) {
                for (int r = 0; r < sc.num_ranks; ++r)
                    ptx::st_release_sys(reinterpret_cast<std::uint64_t*>(sc.seg[r] + sc.sig_off + static_cast<std::size_t>(sc.rank) * sc.flag_stride),
                                        sc.epoch);
            }
        }
    }
}

// ---- host side ----------------------------------------------------------------------------------

namespace {

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                 const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_tiled() {
    static EncodeTiled fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* entry = nullptr;
        cudaDriverEntryPointQueryResult result;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &entry, cudaEnableDefault, &result) == cudaSuccess &&
            result == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiled>(entry);
    });
    return fn;
}

template <int kDims>
bool make_map(CUtensorMap* map, const void* base, const cuuint64_t (&dims)[kDims], const cuuint64_t (&strides)[kDims - 1], const cuuint32_t (&box)[kDims], bool fp8) {
    EncodeTiled encode = encode_tiled();
    if (encode == nullptr) return false;
    cuuint32_t elem[kDims];
    for (cuuint32_t& e : elem) e = 1;
    return encode(map, fp8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, kDims, const_cast<void*>(base), dims, strides, box, elem,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// [rows, k] row-major (bf16 or 1-byte fp8), box = 128 bytes of K x box_rows rows, 128-byte swizzle
bool make_row_map(CUtensorMap* map, const void* base, std::uint64_t rows, std::uint64_t k, std::uint32_t box_rows, bool fp8) {
    const std::uint64_t elem_bytes = fp8 ? 1 : 2;
    const cuuint64_t dims[2] = {k, rows}, strides[1] = {k * elem_bytes};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(kBlockKBytes / elem_bytes), box_rows};
    return make_map<2>(map, base, dims, strides, box, fp8);
}

// gate/up weights [experts, 2n, k] seen as [experts][n / 16][gate, up][16][k]: a box of 128 rows alternates sixteen gate and the
// matching sixteen up rows
bool make_gate_up_map(CUtensorMap* map, const void* base, std::uint64_t experts, std::uint64_t n, std::uint64_t k, bool fp8) {
    const std::uint64_t row = k * (fp8 ? 1 : 2);
    const cuuint64_t dims[5] = {k, 16, 2, n / 16, experts}, strides[4] = {row, n * row, 16 * row, 2 * n * row};
    const cuuint32_t box[5] = {static_cast<cuuint32_t>(kBlockKBytes / (fp8 ? 1 : 2)), 16, 2, kCtaM / 32, 1};
    return make_map<5>(map, base, dims, strides, box, fp8);
}

template <bool kSwiGLU, bool kFp8, bool kScatter = false>
cudaError_t launch(const ActivationMaps& maps_rows, const CUtensorMap& map_w, const GroupedGemmParams& p, int sms, cudaStream_t stream) {
    static bool configured[64] = {false};
    int device = 0;
    cudaError_t status = cudaGetDevice(&device);
    if (status != cudaSuccess) return status;
    constexpr int smem = gemm_smem_bytes(kSwiGLU, kFp8, kScatter);
    if (device >= 0 && device < 64 && !configured[device]) {
        status = cudaFuncSetAttribute(grouped_gemm_kernel<kSwiGLU, kFp8, kScatter>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (status != cudaSuccess) return status;
        configured[device] = true;
    }
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(static_cast<unsigned>(sms / 2 * 2));
    config.blockDim = dim3(kThreads);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[0].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attribute;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, grouped_gemm_kernel<kSwiGLU, kFp8, kScatter>, maps_rows, map_w, p);
}

}  // namespace

}  // namespace gemm

namespace {
const char* run_grouped_gemm(const void* a, const void* w, void* out, const float* a_scales, const float* w_scales,
                             const int* expert_offsets, const int* expert_counts, int* status, int rows_capacity,
                             int num_experts, int n, int k, bool swiglu, bool fp8, const gemm::ScatterTarget* target,
                             const gemm::Progress& progress, cudaStream_t stream) {
    using namespace gemm;
    const int block_k = kBlockKBytes / (fp8 ? 1 : 2);
    if (n % 128 != 0 || k % block_k != 0 || n <= 0 || k <= 0)
        return "n must be a multiple of 128 and k a multiple of 64 (bf16) / 128 (fp8)";
    if (reinterpret_cast<std::uintptr_t>(a) % 16 || reinterpret_cast<std::uintptr_t>(w) % 16 ||
        reinterpret_cast<std::uintptr_t>(out) % 16)
        return "operands must be 16-byte aligned";
    if (target != nullptr) {
        if (swiglu || fp8 || n % 256 != 0) return "the scatter epilogue needs a plain BF16 GEMM with n a multiple of 256";
        if (target->num_ranks < 1 || target->num_ranks > kScatterMaxRanks || target->rank < 0 || target->rank >= target->num_ranks)
            return "scatter target: bad rank table";
        if (target->row_stride % 16 != 0 || target->row_stride < 2 * n || target->stage_off % 16 != 0 || target->epoch == 0 ||
            target->cta_done == nullptr || target->source_meta == nullptr)
            return "scatter target: bad landing-area description";
    }
    if (fp8 && (a_scales == nullptr || w_scales == nullptr)) return "fp8 operands need their scales";
    ActivationMaps maps_rows;
    CUtensorMap map_w;
    bool encoded = swiglu ? make_gate_up_map(&map_w, w, num_experts, n, k, fp8)
                          : make_row_map(&map_w, w, static_cast<std::uint64_t>(num_experts) * n, k, kCtaM, fp8);
    for (int i = 0; i < kBoxes; ++i) encoded = encoded && make_row_map(&maps_rows.box[i], a, rows_capacity, k, box_rows(i), fp8);
    if (!encoded) return "cuTensorMapEncodeTiled failed";
    GroupedGemmParams p{};
    p.expert_offsets = expert_offsets;
    p.expert_counts = expert_counts;
    p.out = static_cast<__nv_bfloat16*>(out);
    p.a_scales = a_scales;
    p.w_scales = w_scales;
    p.status = status;
    p.num_experts = num_experts;
    p.n = n;
    p.k = k;
    p.progress = progress;
    if (target != nullptr) p.scatter = *target;
    int device = 0, sms = 0;
    if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
        return "cannot query the device";
    cudaError_t err;
    if (target != nullptr) err = launch<false, false, true>(maps_rows, map_w, p, sms, stream);
    else if (swiglu) err = fp8 ? launch<true, true>(maps_rows, map_w, p, sms, stream) : launch<true, false>(maps_rows, map_w, p, sms, stream);
    else err = fp8 ? launch<false, true>(maps_rows, map_w, p, sms, stream) : launch<false, false>(maps_rows, map_w, p, sms, stream);
    return err == cudaSuccess ? nullptr : cudaGetErrorString(err);
}
}  // namespace

const char* grouped_gemm(const void* a, const void* w, void* out, const float* a_scales, const float* w_scales,
                         const int* expert_offsets, const int* expert_counts, int* status, int rows_capacity,
                         int num_experts, int n, int k, bool swiglu, bool fp8, const gemm::Progress& progress, cudaStream_t stream) {
    return run_grouped_gemm(a, w, out, a_scales, w_scales, expert_offsets, expert_counts, status, rows_capacity, num_experts,
                            n, k, swiglu, fp8, nullptr, progress, stream);
}

const char* grouped_gemm_scatter(const void* a, const void* w, const int* expert_offsets, const int* expert_counts,
                                 int* status, int rows_capacity, int num_experts, int n, int k,
                                 const gemm::ScatterTarget& target, const gemm::Progress& progress, cudaStream_t stream) {
    // `out` is never written by the scatter epilogue; the A pointer stands in to satisfy the alignment check
    return run_grouped_gemm(a, w, const_cast<void*>(a), nullptr, nullptr, expert_offsets, expert_counts, status, rows_capacity,
                            num_experts, n, k, false, false, &target, progress, stream);
}

int grouped_gemm_tiles_per_chunk(int n) { return 2 * ((n + gemm::kCtaM - 1) / gemm::kCtaM); }  // (a pair's tile has 2 x 64 channels)

int grouped_gemm_ctas() {
    int device = 0, sms = 0;
    if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
        return 0;
    return sms;
}

}  // namespace bep
