// Combine of a group of one rank: every token's expert rows, weighted, become its result row in one ordinary launch.  (Large
// batches of short rows: combine_push.cuh, see combine_local_pays.  Launches that share the SMs with other work, too: a CTA
// of this kernel takes nearly all of an SM's shared memory.)
//
// What bounds it: reading the expert rows from HBM (4096 tokens, hidden 7168, top-8: 470 MB in, 59 MB out).  The rows of a token lie
// far apart, so how they are asked for matters more than how many loads are in flight: pieces of 1 KB per row through 16-byte register
// loads read 4.3 TB/s however many of them were outstanding (110 us).  Here a piece is as long as two stages in shared memory allow -- a
// whole row of 7168 with top-8 -- and one bulk copy: 95 us (91 since L2 gives up what was read first), and 104 us with half rows.
//
// Work unit = (entry of the combine map, slice of its rows).  A CTA's first units are its own, the others come from a counter (launches
// of a few units per CTA: in a fixed order, kCombineLocalFixed): SMs do not all get the same share of HBM, and equal shares waited for
// the slowest (125 us).  The producer warp keeps the claim after next and the map entries of the next units on their way while it starts
// the copies of the present ones; a round of that takes 1.4 us, so small units are claimed four at a time (2048 tokens, a row each: 25.5
// -> 21.9 us).  Before, through the multi-rank reducers (combine_push.cuh): 111 us, 139 us for 8192 tokens top-4 (now 103), 22 us for 128
// tokens (now 7.4).  The other warps add the rows out of shared memory in the order of the entry, in FP32, a thread per 16-byte chunk.
#pragma once

#include "protocol.cuh"

namespace bep {

// How a launch cuts its work (host): slices per row and the ring of stages that fits shared memory.
struct CombineLocalShape {
    int slice_chunks = 0;  // 16-byte chunks of a slice
    int slices = 0;        // per row
    int stages = 0;
    int stage_bytes = 0;   // rows of a unit, one slice each
    int ctas = 0;
    int batch = 1;         // consecutive units per claim: 1 or 4
    bool fixed = false;    // nothing is claimed: CTA b takes the units b, b + ctas, ...
    bool once = false;     // the experts' rows leave L2 first, see outgrows_l2
    std::size_t bytes = 0; // dynamic shared memory
};

struct CombineLocalArgs {
    const RankConst* rc;
    const __nv_bfloat16* y;          // expert outputs in the layout of the dispatch's recv_x
    const int* comb_map;             // [C][slots_full][2 + 2K]: token, n, then (row, weight bits) pairs
    const int* recv_chan_counts;     // [C] entries per channel
    const std::uint32_t* plan_mask;  // [Tmax] 0: the token was routed nowhere, its result is zero
    int num_tokens;
    int weighted;
    __nv_bfloat16* out;              // [T, H]
    int* error;                      // [8]
    std::int64_t* stats;             // [8]: rows written, 0, ns from the first CTA's start to the last one's end (without claims: of CTA 0 alone)
    unsigned long long* cta_done;    // CTAs of this launch that have finished; the last one puts it back to zero
    unsigned long long* first_start; // earliest start; all ones between launches
    unsigned long long* next_unit;   // units handed out beyond every CTA's first; zero between launches
    int num_channels, slots_full, num_topk, hidden;
    CombineLocalShape shape;
};

constexpr int kCombineLocalMaxStages = 8;
constexpr int kCombineLocalConsumers = 14;  // warps that add, behind the producer warp: 448 threads, half a row of 7168
constexpr int kCombineLocalThreads = 32 * (1 + kCombineLocalConsumers);
// Units whose stage is at most this large are claimed four at a time, given a dozen per CTA: a claim and the map entries behind
// it are a latency that four units share, 8192 tokens with six rows each 0.9 us a unit at 30 KB (hidden 2560, 68 us) and 1.6
// claimed singly at 34 KB (hidden 2880, 95 us).  Larger units take that long to read anyway (7 stages of 32 KB are in flight),
// and four of them in one CTA would be an uneven end.
constexpr int kCombineLocalSmallStage = 32 * 1024;
// Launches with at most this many units per CTA (the second line: of stages up to kCombineLocalSmallStage) don't claim: CTA b takes the
// units b, b + grid, ...  There is little to even out yet, the map entries of four units are asked for at once, and without counters no
// CTA has to find out whether it is the last one: 16 tokens, 8 rows of 14 KB 7.0 -> 5.2 us.  Singly claimed / in a fixed order:
//   4 units and more: 777 tokens, 4 rows of 8 KB 14.7 / 12.5, 1000 tokens, 2 rows of 4 KB 14.6 / 9.5, 8 rows of 14 KB 30.9 / 28.7;
//   12 units: 1800 tokens, 8 rows of 8 KB 31.4 / 30.0;  14: 2048 tokens, 8 rows of 14 KB, the exchange 102.9 / 103.5.
// Nobody is the last one then, so the duration in `stats` is that of CTA 0 (3.0 us of such a launch of 16 tokens, 16.3 of 2048 single
// rows): counting the CTAs for the sake of that number cost 0.3 to 0.6 us a launch.
constexpr int kCombineLocalFixed = 12;
constexpr int kCombineLocalFixedSmall = 16;

struct CombineLocalHeader {
    int token, n, first_chunk, chunks;  // n < 0: no more units
    float weight[kMaxTopk];
};
struct CombineLocalShared {
    unsigned long long full[kCombineLocalMaxStages], empty[kCombineLocalMaxStages];
    CombineLocalHeader header[kCombineLocalMaxStages];
};
constexpr int kCombineLocalTiles = 2048;  // offset of the stages
static_assert(sizeof(CombineLocalShared) <= kCombineLocalTiles, "the stages start behind the barriers and headers");

// `max_rows`: most rows an entry can have.  Slices are as long as two stages allow, and with few tokens shorter (down to units of 1 KB
// per row) where that spares time.
inline CombineLocalShape combine_local_shape(int tokens, int hidden, int max_rows, int sms, std::size_t smem_limit, long long l2_bytes) {
    CombineLocalShape s;
    const int chunks = hidden / 8;
    auto slices_for = [chunks](int slice) { return (chunks + slice - 1) / slice; };
    int slice = static_cast<int>((smem_limit - kCombineLocalTiles) / 2 - 128) / 16 / max_rows;
    if (slice > chunks) slice = chunks;
    int slices = slices_for(slice);
    // Few tokens: a CTA takes rounds of one unit, each a slice's share of the row and about 0.3 of a row's time on top, and the last round is
    // as long as a full one.  So 16 tokens are cut into eighths and 64 into halves (one round), 75 to 148 not at all (one round of whole
    // rows; some SMs have none), 149 to 222 into halves (three rounds) and 223 to 296 not (two).  8 rows of 14 KB, us, whole / cut as before,
    // into two units per SM or more: 75 tokens 7.0 / 7.7, 100 7.4 / 7.9, 128 7.4 / 8.8, 148 8.3 / 8.2; whole / halves: 149 tokens 9.6 / 9.2, 180
    // 10.7 / 9.9, 200 11.7 / 10.6; 8 rows of 6 KB 75 tokens 6.0 / 7.3, 200 6.9 / 7.6, 4 rows of 8 KB 100 tokens 5.9 / 6.9, 180 6.8 / 7.1.
    const auto cost = [&](int cut) { return static_cast<double>((static_cast<long long>(tokens) * cut + sms - 1) / sms) * (1.0 / cut + 0.3); };
    for (int shorter = slice, cut = slices; static_cast<long long>(tokens) * cut < 2ll * sms && shorter >= 128;) {
        shorter = (shorter + 1) / 2;
        cut = slices_for(shorter);
        if (cost(cut) < cost(slices)) slices = cut;
    }
    s.slice_chunks = (chunks + slices - 1) / slices;  // equal slices
    s.slices = slices_for(s.slice_chunks);
    s.stage_bytes = static_cast<int>(align_up(static_cast<std::size_t>(max_rows) * s.slice_chunks * 16, 128));
    const std::size_t room = (smem_limit - kCombineLocalTiles) / static_cast<std::size_t>(s.stage_bytes);
    s.stages = room < 2 ? 2 : room > kCombineLocalMaxStages ? kCombineLocalMaxStages : static_cast<int>(room);
    s.bytes = kCombineLocalTiles + static_cast<std::size_t>(s.stages) * s.stage_bytes;
    const long long units = static_cast<long long>(tokens) * s.slices;
    s.ctas = units < 1 ? 1 : units < sms ? static_cast<int>(units) : sms;
    s.batch = s.stage_bytes <= kCombineLocalSmallStage && units >= 12ll * sms ? 4 : 1;
    s.fixed = units <= static_cast<long long>(s.stage_bytes <= kCombineLocalSmallStage ? kCombineLocalFixedSmall : kCombineLocalFixed) * s.ctas;
    s.once = outgrows_l2(static_cast<long long>(tokens) * (max_rows + 1) * hidden * 2, l2_bytes);
    return s;
}

// Which calls this kernel is for; the others keep the register loads of combine_push.cuh.  One producer warp hands out a unit
// in 0.8 to 1.1 us (1.6 where units are claimed singly) however short its rows are, while the reducer warps there take an
// entry each and so little time for short rows; they start 4 to 6 us later.  Measured on 148 SMs, us, registers / bulk copies:
//   few tokens (up to 8 per SM): 128 tokens, 8 rows of 1 KB 15.6 / 8.3; 1024 tokens, 8 rows of 2 KB 17.7 / 16.5, one of
//     14 KB 21.4 / 16.5; beyond: 1536 tokens, 2 rows of 1 KB 17.2 / 18.5, 65536 tokens, one of 2 KB 143 / 359;
//   up to 14 per SM with rows of 3 KB and more: 2048 tokens, 8 rows of 4 KB 28.1 / 24.8, of 2 KB 21.6 / 23.7;
//   rows of 10 KB and more: 8192 tokens, one row 69.5 / 58.3, 8 rows of 14 KB 205 / 160; one row of 8 KB 53.3 / 57.5;
//   several rows of 7 KB and more: 8192 tokens, 4 rows of 7 KB 74.9 / 66.3, two 55.0 / 59.5, 8 rows of 5.6 KB 95.5 / 103.7.
inline bool combine_local_pays(int tokens, int hidden, int max_rows, int sms) {
    const int row_bytes = hidden * 2;
    if (tokens <= 8ll * sms || row_bytes >= 10 * 1024) return true;
    return (row_bytes >= 7 * 1024 && max_rows >= 4) || (row_bytes >= 3 * 1024 && tokens <= 14ll * sms);
}

#ifdef __CUDACC__

// kBatch: units whose map entries are asked for at once; consecutive ones, one claim, or in a fixed order `ctas` apart
template <int kBatch>
__global__ void __launch_bounds__(kCombineLocalThreads, 1) local_combine_push_kernel(const __grid_constant__ CombineLocalArgs a) {
    const RankConst* __restrict__ rc = a.rc;
    const int C = a.num_channels, K = a.num_topk, H = a.hidden, T = a.num_tokens;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int chunks = H / 8, stages = a.shape.stages;
    const std::size_t row_bytes = static_cast<std::size_t>(H) * 2;
    extern __shared__ __align__(128) unsigned char combine_smem[];
    auto* sh = reinterpret_cast<CombineLocalShared*>(combine_smem);
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            ptx::mbar_init(reinterpret_cast<std::uint64_t*>(&sh->full[s]), 1);
            ptx::mbar_init(reinterpret_cast<std::uint64_t*>(&sh->empty[s]), kCombineLocalConsumers);
        }
        ptx::mbar_fence_init();
    }
    const int Tc = max(1, (T + C - 1) / C);  // tokens per channel: no channel has more entries
    const long long units = static_cast<long long>((T + Tc - 1) / Tc) * Tc * a.shape.slices;
    const bool fixed = a.shape.fixed;
    const int apart = fixed ? gridDim.x : 1;  // units of a batch
    // The launch before is the expert GEMM, usually, or the dispatch whose map is read below.  Reads of what it may have written are
    // ordinary loads: one that counts on memory staying as it is for the whole kernel (ld.global.nc) may be moved in front of the wait.
    ptx::wait_for_launch_before();
    const std::uint64_t t_start = threadIdx.x == 0 ? ptx::globaltimer_ns() : 0;
    if (threadIdx.x == 0 && !fixed) atomicMin(a.first_start, static_cast<unsigned long long>(t_start));
    const bool aborted = ptx::ld_volatile(&rc->sticky[0]) != 0;
    if (aborted && threadIdx.x == 0 && blockIdx.x == 0) atomicCAS(&a.error[0], 0, kErrAlreadyAborted);
    Health health(rc, a.error);
    __syncthreads();

    bool ok = true;
    auto wait = [&](unsigned long long* bar, unsigned parity) {
        while (!ptx::mbar_try_wait(reinterpret_cast<std::uint64_t*>(bar), parity))
            if (health.give_up(kErrCopyEngine, static_cast<int>(blockIdx.x), 1)) return false;
        return true;
    };
    if (aborted || T == 0) {
        // nothing to do
    } else if (warp == 0) {
        // ---- producer ----------------------------------------------------------------------------------------------
        const int map_stride = 2 + 2 * K;
        const std::uint64_t policy = ptx::l2_policy(a.shape.once);
        struct Entry {
            int count, j;  // the entry exists if j < count
            int2 head;     // token, rows
            int2 pair;     // lane i: row and weight of the entry's i-th row
        };
        auto load_entry = [&](long long u) {
            Entry e{};
            if (u >= units) return e;
            const int entry = static_cast<int>(u / a.shape.slices), c = entry / Tc;
            e.j = entry % Tc;
            // (entries beyond the channel's count hold what an earlier dispatch left: read, not used)
            const int* map = a.comb_map + (static_cast<std::size_t>(c) * a.slots_full + e.j) * map_stride;
            e.count = a.recv_chan_counts[c];
            e.head = *reinterpret_cast<const int2*>(map);
            if (lane < K) e.pair = reinterpret_cast<const int2*>(map)[1 + lane];
            return e;
        };
        auto claim = [&]() {
            unsigned long long got = 0;
            if (lane == 0) got = atomicAdd(a.next_unit, 1ull);
            return got;  // lane 0's value counts
        };
        long long u = static_cast<long long>(blockIdx.x) * (fixed ? 1 : kBatch);
        Entry e[kBatch];
#pragma unroll
        for (int i = 0; i < kBatch; ++i) e[i] = load_entry(u + i * apart);
        unsigned long long claimed = fixed ? 0 : claim();
        int filled = 0;  // stages handed to the consumers
        while (ok && u < units) {
            const long long next_u = fixed ? u + static_cast<long long>(gridDim.x) * kBatch
                                           : (static_cast<long long>(gridDim.x) + static_cast<long long>(__shfl_sync(0xffffffffu, claimed, 0))) * kBatch;
            Entry next[kBatch];
#pragma unroll
            for (int i = 0; i < kBatch; ++i) next[i] = load_entry(next_u + i * apart);
            if (!fixed && next_u < units) claimed = claim();
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
                if (!ok || e[i].j >= e[i].count) continue;
                const int stage = filled % stages;
                ok = __all_sync(0xffffffffu, wait(&sh->empty[stage], (static_cast<unsigned>(filled / stages) & 1u) ^ 1u)) != 0;
                if (!ok) continue;
                const int n = e[i].head.y, first = static_cast<int>((u + i * apart) % a.shape.slices) * a.shape.slice_chunks;
                const int len = min(a.shape.slice_chunks, chunks - first);
                CombineLocalHeader& header = sh->header[stage];
                if (lane < n) header.weight[lane] = a.weighted ? __int_as_float(e[i].pair.y) : 1.0f;
                if (lane == 0) {
                    header.token = e[i].head.x;
                    header.n = n;
                    header.first_chunk = first;
                    header.chunks = len;
                }
                __syncwarp();
                auto* bar = reinterpret_cast<std::uint64_t*>(&sh->full[stage]);
                if (lane == 0) ptx::mbar_expect_tx(bar, static_cast<unsigned>(n * len) * 16u);
                __syncwarp();
                if (lane < n) {
                    unsigned char* const piece = combine_smem + kCombineLocalTiles + static_cast<std::size_t>(stage) * a.shape.stage_bytes + static_cast<std::size_t>(lane) * len * 16;
                    const auto* row = reinterpret_cast<const std::uint8_t*>(a.y) + static_cast<std::size_t>(e[i].pair.x) * row_bytes + static_cast<std::size_t>(first) * 16;
                    ptx::bulk_g2s(piece, row, static_cast<unsigned>(len) * 16u, bar, policy);
                }
                ++filled;
            }
            u = next_u;
#pragma unroll
            for (int i = 0; i < kBatch; ++i) e[i] = next[i];
        }
        if (ok) {  // tell the consumers that this was all
            const int stage = filled % stages;
            ok = __all_sync(0xffffffffu, wait(&sh->empty[stage], (static_cast<unsigned>(filled / stages) & 1u) ^ 1u)) != 0;
            if (ok && lane == 0) {
                sh->header[stage].n = -1;
                ptx::mbar_arrive(reinterpret_cast<std::uint64_t*>(&sh->full[stage]));
            }
        }
        if (!ok)  // copies that are still under way: a bounded time to land before shared memory goes away
            for (int f = max(0, filled - stages); f < filled; ++f)
                for (unsigned polls = 0; !ptx::mbar_try_wait(reinterpret_cast<std::uint64_t*>(&sh->full[f % stages]), static_cast<unsigned>(f / stages) & 1u) &&
                                         polls < (1u << 20); ++polls)
                    ptx::nanosleep(64);
    } else {
        // ---- consumers ---------------------------------------------------------------------------------------------
        const int consumer = warp - 1, rank = consumer * 32 + lane;  // first chunk of this thread in a slice
        const int first_zero = blockIdx.x * kCombineLocalConsumers + consumer, zero_step = gridDim.x * kCombineLocalConsumers;
        const std::uint32_t first_mask = first_zero < T ? a.plan_mask[first_zero] : 1u;  // needed at the end
        for (int f = 0;; ++f) {
            const int stage = f % stages;
            ok = __all_sync(0xffffffffu, wait(&sh->full[stage], static_cast<unsigned>(f / stages) & 1u)) != 0;
            if (!ok) break;
            const CombineLocalHeader& header = sh->header[stage];
            const int n = header.n, len = header.chunks;
            if (n < 0) break;
            const unsigned char* tile = combine_smem + kCombineLocalTiles + static_cast<std::size_t>(stage) * a.shape.stage_bytes;
            std::uint8_t* dst = reinterpret_cast<std::uint8_t*>(a.out) + static_cast<std::size_t>(header.token) * row_bytes + static_cast<std::size_t>(header.first_chunk) * 16;
            for (int q = rank; q < len; q += kCombineLocalConsumers * 32) {
                float acc[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 4
                for (int r = 0; r < n; ++r) {
                    const uint4 v = *reinterpret_cast<const uint4*>(tile + (static_cast<std::size_t>(r) * len + q) * 16);
                    const float w = header.weight[r];
                    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        const float2 p = __bfloat1622float2(h[x]);
                        acc[2 * x] = fmaf(w, p.x, acc[2 * x]);
                        acc[2 * x + 1] = fmaf(w, p.y, acc[2 * x + 1]);
                    }
                }
                uint4 packed;
                __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&packed);
#pragma unroll
                for (int x = 0; x < 4; ++x) h[x] = __floats2bfloat162_rn(acc[2 * x], acc[2 * x + 1]);
                ptx::st_v4(dst + static_cast<std::size_t>(q) * 16, packed);
            }
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(reinterpret_cast<std::uint64_t*>(&sh->empty[stage]));
        }
        // tokens that were routed nowhere have no entry: their result is zero
        for (int t = first_zero; ok && t < T; t += zero_step) {
            if ((t == first_zero ? first_mask : a.plan_mask[t]) != 0) continue;
            for (int q = lane; q < chunks; q += 32)
                ptx::st_v4(reinterpret_cast<std::uint8_t*>(a.out) + static_cast<std::size_t>(t) * row_bytes + static_cast<std::size_t>(q) * 16, make_uint4(0u, 0u, 0u, 0u));
        }
    }

    __syncthreads();
    if (warp == 0) {
        unsigned long long finished = 0;
        if (lane == 0 && !fixed) {
            __threadfence();
            finished = atomicAdd(a.cta_done, 1ull) + 1ull;
        }
        if (fixed ? blockIdx.x == 0 : __shfl_sync(0xffffffffu, finished, 0) == gridDim.x) {
            // launches that share these counters are stream-ordered
            int rows = 0;
            if (!aborted)
                for (int c = lane; c < C; c += 32) rows += a.recv_chan_counts[c];
            rows = __reduce_add_sync(0xffffffffu, rows);
            if (lane == 0) {
                std::uint64_t first = t_start;
                if (!fixed) {
                    __threadfence();
                    first = __ldcg(a.first_start);
                    *a.cta_done = 0ull;
                    *a.next_unit = 0ull;
                    *a.first_start = ~0ull;
                }
                a.stats[0] = rows;
                a.stats[2] = static_cast<std::int64_t>(ptx::globaltimer_ns() - first);
                a.stats[1] = a.stats[3] = a.stats[4] = a.stats[5] = a.stats[6] = a.stats[7] = 0;
                if (ptx::ld_volatile(&rc->sticky[0]) == 0) rc->epochs[1] += 1;
            }
        }
    }
}

#endif  // __CUDACC__

}  // namespace bep
