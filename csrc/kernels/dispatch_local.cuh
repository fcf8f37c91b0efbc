// Dispatch of a group of one rank.  Nothing crosses a link, so of the protocol in dispatch.cuh only the routing layout and
// the expansion are left: no counts message, no READY flags, no send role, no control warp.  Results, routing plan and
// combine map are the ones dispatch.cuh leaves behind, bit for bit; the two kernels may alternate on one buffer.
//
// Grid: one CTA per SM, or one per token where there are fewer tokens (and as many as experts where rows between their
// segments are zeroed); CTA b owns the tokens [T*b/G, T*(b+1)/G).  A launch beside the compute stream has no more CTAs than the
// configuration has channels; where the tables of so many tokens per CTA do not fit, dispatch.cuh takes the call.  (Otherwise the
// channels only number the combine map here: few CTAs would keep a barrier between ranks short, but the SMs that write the
// rows are what sets the pace.)
//   1. token rows are on their way into shared memory before anything about the layout is known;
//   2. expert ids -> histogram and stable ordinals inside the CTA's tokens, 32 tokens at a time, one thread per (token, k);
//   3. one grid barrier; then a prefix over the CTAs before this one and a scan over experts, one thread per bin.  A small batch
//      (kLocalWholePairs) is counted as a whole by every CTA instead, a cached layout skips 2 as well: without the barrier the
//      launch is an ordinary one;
//   4. a warp per token: every lane k < K whose expert is valid starts the bulk store of the row to its expert's segment.
//
// What bounds it.  Large batches: writing the expanded rows to HBM.  4096 tokens, hidden 7168, top-8 move 528 MB.
// Small ones: the chain launch -> ids -> counts -> scan -> rows; between them, from kLocalWholePairs on, a barrier and a prefix.
// Launch to end with a cold L2, general kernel -> this one: 128 tokens 46 -> 10.1 us (no flags to wait for, no prefix by a single warp,
// no barrier), 4096 tokens 131 -> 99 us, the same with E4M3 rows 106 -> 67 us (fourteen row buffers per SM on all SMs instead of eight
// on 128), 256 tokens with a cached layout 45 -> 10.1 us.
#pragma once

#include "dispatch_common.cuh"

namespace bep {

constexpr int kLocalThreads = 512;
constexpr int kLocalWarps = kLocalThreads / 32;
constexpr int kLocalMaxStages = 3;      // row buffers per warp
constexpr int kLocalMinWarps = 4;       // fewer row buffers than this: rows too long, dispatch.cuh takes the call
constexpr int kLocalMaxPairBytes = 64 * 1024;
// Routing tables for a grid of `channels` CTAs (more tokens each) are taken up to this size, so that launches beside other work
// can have this kernel too; beyond it they would cost row buffers (at hidden 7168 fourteen of them leave 26 KB), which large
// batches need more: fourteen on all SMs instead of eight on 128 are 71 instead of 106 us for 4096 E4M3 rows.
constexpr int kLocalSmallPairBytes = 16 * 1024;

// Batches of up to this many (token, k) are counted by every CTA by itself, without a barrier: no CTA waits for another one, and
// where none claims tokens the launch needs no cooperative grid and nobody has to be the last.  Together / by itself, top-8: 16 tokens
// 17.2 / 10.7 us, 128 tokens 17.3 / 10.9, 4096 97.5 / 101 (layout done after 12.6 / 15.8); 777 tokens top-4 20.9 / 13.6.  At the line, 2048
// tokens, the layout is done after 9.2 us (12.5 before ids came eight steps at a time and nothing was read behind the row loads).
constexpr int kLocalWholePairs = 16 * 1024;
constexpr int kLocalFewExperts = 64;  // counted with ballots, without atomics (a warp's 32 pairs meet few counters again and again)

struct LocalDispatchArgs {
    DispatchArgs a;
    LocalPlan plan;
    int* hist;                     // [G][E + 1] counts per CTA, then two copies of [groups][E + 1 + C] sums, then their generation
    unsigned long long* counters;  // barrier arrivals, finished CTAs, complement of the first start, CTAs whose plan is written, tokens claimed (zero between launches)
    int hist_ctas;                 // CTAs the scratch has room for
    int num_experts, num_channels, num_topk, hidden, slots_full, expanded_cap, unique_cap;  // as in the rank's constants
    bool once;                     // rows leave L2 first
};

inline std::size_t local_hist_ints(int ctas, int experts, int channels) {
    const std::size_t groups = static_cast<std::size_t>((ctas + kHistGroup - 1) / kHistGroup);
    return static_cast<std::size_t>(ctas) * (experts + 1) + 2 * groups * (experts + 1 + channels) + 1;
}

struct LocalShared {
    unsigned long long mbar[kLocalWarps * kLocalMaxStages];
    unsigned long long warp_sum[kLocalWarps];
    int flag;        // the CTA leaves without rows
    int routed;      // routed tokens of this CTA
    int token[kLocalWarps * kLocalMaxStages];  // of the row in each buffer
    int first_unique;  // routed tokens of earlier CTAs
    int unique_total;
};

// header | base[E] | total[E] | eoff[E + 1] | chan_base[C] | pair_e[cap*K] | pair_ord[cap*K] | unique[cap] | row buffers
inline LocalPlan make_local_plan(int experts, int channels, int topk, int hidden, int max_tokens, int sms, std::size_t smem_limit) {
    LocalPlan p;
    // tokens per CTA: for a grid of `channels` CTAs (launches beside other work) if their tables stay small, else for all SMs
    const auto cap = [max_tokens](int ctas) { return (max_tokens + ctas - 1) / ctas + 1; };
    const int token_bytes = 8 * topk + 4, few = channels < sms ? channels : sms;
    p.token_cap = cap(few) <= kLocalSmallPairBytes / token_bytes ? cap(few) : cap(sms);
    const std::size_t pair_bytes = static_cast<std::size_t>(p.token_cap) * token_bytes;
    std::size_t bytes = align_up(sizeof(LocalShared), 16) + static_cast<std::size_t>(experts) * 12 + 4 + static_cast<std::size_t>(channels) * 4;
    bytes = align_up(bytes + pair_bytes, 128);
    p.rows_off = bytes;
    p.slot_bytes = static_cast<int>(align_up(static_cast<std::size_t>(hidden) * 2, 128));
    if (pair_bytes > static_cast<std::size_t>(kLocalMaxPairBytes) || bytes >= smem_limit) return p;
    const int slots = static_cast<int>((smem_limit - bytes) / static_cast<std::size_t>(p.slot_bytes));
    p.warps = slots < kLocalWarps ? slots : kLocalWarps;
    p.stages = slots / kLocalWarps < 1 ? 1 : slots / kLocalWarps < kLocalMaxStages ? slots / kLocalWarps : kLocalMaxStages;
    p.bytes = bytes + static_cast<std::size_t>(p.warps) * p.stages * p.slot_bytes;
    p.usable = p.warps >= kLocalMinWarps;
    // what is left over holds the tables of a batch that every CTA counts by itself
    p.whole_off = align_up(p.bytes, 16);
    p.whole_bytes = smem_limit > p.whole_off ? static_cast<int>(smem_limit - p.whole_off) : 0;
    return p;
}

// Those tables: a bit per (token, k), a bit per token, routed tokens before each 32.
__host__ __device__ inline std::size_t local_whole_bytes(int tokens, int topk) {
    const std::size_t pair_words = (static_cast<std::size_t>(tokens) * topk + 31) / 32 + 1, token_words = static_cast<std::size_t>(tokens + 31) / 32;
    return 4 * (pair_words + 2 * token_words + 1);
}
// Whether every CTA of `ctas` counts such a batch by itself.  Where the row buffers leave less than its tables need, `plan` gives up
// the buffers of a warp, if the others still hold all tokens of a CTA: 32 experts, rows of 14 KB, 555 tokens, the layout is done after
// 7.4 us instead of 8.9; 16 experts, rows of 7 KB, 4096 tokens top-2 (28 per CTA, 30 of 32 buffers) 27.6 -> 21.9 us.  Where tokens would
// have to be claimed for it, the barrier is the better one, by itself / together: 2048 tokens top-8, rows of 16 KB in 16 experts (14
// per CTA, 13 buffers) 68.5 / 63.1 us, top-4 in 32 experts 43.6 / 40.9.
inline bool local_counts_whole(int tokens, int topk, int ctas, LocalPlan& plan) {
    if (tokens <= 0 || static_cast<long long>(tokens) * topk > kLocalWholePairs) return false;
    const std::size_t tables = local_whole_bytes(tokens, topk);
    LocalPlan fewer = plan;
    while (tables > static_cast<std::size_t>(fewer.whole_bytes)) {
        if (--fewer.warps < kLocalMinWarps || (tokens + ctas - 1) / ctas > fewer.warps * fewer.stages) return false;
        const std::size_t given = static_cast<std::size_t>(fewer.stages) * fewer.slot_bytes;
        fewer.bytes -= given;
        fewer.whole_off -= given;  // (a multiple of 128)
        fewer.whole_bytes += static_cast<int>(given);
    }
    plan = fewer;
    return true;
}

// What a launch of `ctas` CTAs makes of a plan, for tokens of `token_bytes`, rows as received among them.  `pooled`: a CTA has more tokens
// than row buffers, the rest is claimed.
inline LocalShape local_shape(LocalPlan plan, int tokens, int topk, long long token_bytes, int ctas, bool cached) {
    LocalShape s;
    s.once = outgrows_l2(tokens * token_bytes, plan.l2_bytes);
    const bool whole = !cached && local_counts_whole(tokens, topk, ctas, plan);
    s.mode = cached ? kLocalCached : whole ? kLocalWhole : kLocalTogether;
    s.pooled = (tokens + ctas - 1) / ctas > plan.warps * plan.stages;
    s.bytes = whole ? plan.whole_off + local_whole_bytes(tokens, topk) : plan.bytes;
    s.plan = plan;
    return s;
}

#ifdef __CUDACC__

namespace detail {

__device__ __forceinline__ void local_wait_read(int groups_left) {
    if (groups_left <= 0) bulk_wait_group_read<0>();
    else if (groups_left == 1) bulk_wait_group_read<1>();
    else bulk_wait_group_read<2>();
}

}  // namespace detail

// kFp8: rows stay E4M3.  kPooled: a CTA has more tokens than row buffers.
template <LocalMode kMode, bool kFp8, bool kPooled>
__global__ void __launch_bounds__(kLocalThreads, 1) local_dispatch_kernel(const __grid_constant__ LocalDispatchArgs args) {
    using namespace detail;
    const DispatchArgs& a = args.a;
    const RankConst* __restrict__ rc = a.rc;
    const int E = args.num_experts, C = args.num_channels, K = args.num_topk, H = args.hidden, Qf = args.slots_full;
    const int T = a.num_tokens, G = gridDim.x, b = blockIdx.x;
    const int Tc = max(1, (T + C - 1) / C);
    const int t0 = static_cast<int>(static_cast<long long>(T) * b / G), t1 = static_cast<int>(static_cast<long long>(T) * (b + 1) / G);
    const int nt = t1 - t0;
    const int tid = threadIdx.x, warp = tid >> 5;
    const unsigned lane = ptx::lane_id(), full = 0xffffffffu, lt_mask = (1u << lane) - 1u;
    constexpr bool recv_fp8 = kFp8;
    const bool expand = a.do_expand != 0;
    constexpr bool cached = kMode == kLocalCached, whole = kMode == kLocalWhole;
    const int row_warps = args.plan.warps, stages = args.plan.stages, slot_bytes = args.plan.slot_bytes;
    const unsigned in_bytes = static_cast<unsigned>(H) * 2u;

    extern __shared__ __align__(128) unsigned char local_smem[];
    auto* sh = reinterpret_cast<LocalShared*>(local_smem);
    int* base = reinterpret_cast<int*>(local_smem + align_up(sizeof(LocalShared), 16));  // [E] rows of earlier CTAs in the expert
    int* total = base + E;         // [E] rows of the expert; the bit sets of a 32-token chunk before that
    int* eoff = total + E;         // [E + 1]
    int* chan_base = eoff + E + 1; // [C] routed tokens of earlier channels
    int* pair_e = chan_base + C;   // [cap * K] expert of (token, k), -1: none
    int* pair_ord = pair_e + args.plan.token_cap * K;  // stable ordinal of the pair in its expert: inside the CTA (fresh layout) or overall (cached)
    int* unique = pair_ord + args.plan.token_cap * K;  // [cap] ordinal of the routed token: inside the CTA (fresh) or in its channel (cached); else the complement of it
    unsigned char* rows_sm = local_smem + args.plan.rows_off;

    // what thread 0 has to know about the rank (asked for now, looked at after the histogram)
    const int sticky_before = tid == 0 ? ptx::ld_volatile(&rc->sticky[0]) : 0;
    const std::uint64_t epoch_before = tid == 0 ? __ldcg(rc->epochs) : 0;
    const unsigned long long t_start = ptx::globaltimer_ns();
    // where no CTA needs another one's counts or claims its tokens, nothing has to be settled by the last one
    constexpr bool pooled = kPooled;  // then every CTA has at least as many tokens as row buffers
    constexpr bool alone = (cached || whole) && !pooled;
    if (tid == 0 && !alone) atomicMax(&args.counters[2], ~t_start);
    // profile rows are per channel: CTA b fills the rows b, b + G, ...
#define BEP_PROF(point)                                                                                          \
    do {                                                                                                         \
        const std::int64_t now_ = static_cast<std::int64_t>(ptx::globaltimer_ns());                              \
        for (int r_ = b; r_ < C; r_ += G) a.profile[static_cast<std::size_t>(r_) * 16 + (point)] = now_;         \
    } while (0)
    if (tid == 0)
        for (int r = b; r < C; r += G) {
            std::int64_t* prof = a.profile + static_cast<std::size_t>(r) * 16;
            prof[kProfStart] = prof[kProfGuardDone] = static_cast<std::int64_t>(t_start);
            prof[kProfFirstTxDone] = prof[kProfFirstRxRow] = 0;
        }
    Health health(rc, a.error);

    if (tid < row_warps * stages) {
        ptx::mbar_init(reinterpret_cast<std::uint64_t*>(&sh->mbar[tid]), 1);
        ptx::mbar_fence_init();
    }
    // ids of the first chunk are asked for now; they arrive while shared memory is cleared
    const int first_pairs = min(32, nt) * K;
    const std::int64_t first_id = tid < first_pairs ? __ldg(a.topk_idx + static_cast<std::size_t>(t0) * K + tid) : -1;
    const int W = E + 1, S = W + C;
    const int groups = (args.hist_ctas + kHistGroup - 1) / kHistGroup;
    int* const sums_base = args.hist + static_cast<std::size_t>(args.hist_ctas) * W;
    int* const generation_at = sums_base + static_cast<std::size_t>(2) * groups * S;
    const int generation = cached || whole ? 0 : __ldcg(generation_at);
    auto* const counts = reinterpret_cast<unsigned*>(eoff);  // whole: pairs of the expert, those of earlier CTAs in the upper half
    if (tid == 0) {
        sh->flag = 0;
        sh->routed = 0;
        sh->first_unique = 0;
    }
    for (int i = tid; i < E; i += kLocalThreads) {
        base[i] = 0;
        total[i] = 0;
        counts[i] = 0;
    }
    if (!cached && !whole) {
        // the sums this CTA will add to have been driven out of L2 by the rows of the last launch: fetch both copies' lines
        for (int i = tid * 32; i < S; i += kLocalThreads * 32)
            for (int copy = 0; copy < 2; ++copy)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(sums_base + (static_cast<std::size_t>(copy) * groups + b / kHistGroup) * S + i));
    }
    __syncthreads();

    // ---- 1. the first rows of every warp start their way into shared memory ----------------------------------
    const std::uint64_t policy = ptx::l2_policy(args.once);
    auto start_load = [&](int n, int t) {  // token t as the warp's n-th (lane 0 only)
        auto* bar = reinterpret_cast<std::uint64_t*>(&sh->mbar[warp * stages + n % stages]);
        ptx::mbar_expect_tx(bar, in_bytes);
        std::uint8_t* const slot = rows_sm + static_cast<std::size_t>(warp * stages + n % stages) * slot_bytes;
        // (The stores of BF16 rows as ones that leave L2 first, too: an exchange of 4096 tokens 193 -> 196.5 us.)
        ptx::bulk_g2s(slot, a.x + static_cast<std::size_t>(t) * H, in_bytes, bar, policy);
        sh->token[warp * stages + n % stages] = t;
    };
    int started = 0;  // loads of this warp that are under way or done
    auto start_first_loads = [&]() {
        if (warp >= row_warps) return;
        for (; started < stages && warp + started * row_warps < nt; ++started)
            if (lane == 0) start_load(started, t0 + warp + started * row_warps);
    };
    // Large batches: what does not fit a CTA's row buffers at once is handed out through a counter, a token at a time over
    // all CTAs (SMs do not all get the same share of HBM: with equal shares the slowest finished 17 us behind the others
    // at 4096 tokens: 110 -> 104 us, 8192 tokens top-4 122 -> 117, 4096 with E4M3 rows 73 -> 71).
    const int own_tokens = row_warps * stages, most_tokens = (T + G - 1) / G;

    // a rank that has failed, or has run out of epochs, leaves without rows
    auto leaves = [&]() {  // thread 0
        if (sticky_before != 0) {
            if (b == 0) atomicCAS(&a.error[0], 0, kErrAlreadyAborted);
            return true;
        }
        if (alone && b != G - 1) return false;  // (the last CTA may have advanced the epoch already)
        if (epoch_before + 1 >= (1ull << 32)) record_error(rc, a.error, kErrEpochExhausted, 0, 0);
        return epoch_before + 1 >= (1ull << 32);
    };

    // ---- 2. ordinals inside the CTA ------------------------------------------------------------------------------
    const int all_pairs = T * K, pair_words = (all_pairs + 31) / 32 + 1, token_words = (T + 31) / 32;
    auto* const pair_bits = reinterpret_cast<unsigned*>(local_smem + args.plan.whole_off);  // whole: which pairs name an expert,
    unsigned* const token_bits = pair_bits + pair_words;                                    // which tokens are routed,
    int* const routed_words = reinterpret_cast<int*>(token_bits + token_words);             // [token_words + 1] routed tokens before word w
    if constexpr (whole) {
        // The pairs of the whole batch: 32 per warp and step, the ids of eight steps on their way at once (of four: 2048 tokens top-8 0.8 us
        // more).  Few experts meet in a step again and again: there a lane counts two of them from ballots of the ids' bits.
        const int own_first = t0 * K;
        const bool few = E <= kLocalFewExperts;
        unsigned mine[2] = {0u, 0u};  // few: pairs of the experts lane and lane + 32, those of earlier CTAs in the upper half
        bool bad = false;
        for (int p0 = warp * 32; p0 < all_pairs; p0 += kLocalThreads * 8) {
            std::int64_t id[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int p = p0 + u * kLocalThreads + static_cast<int>(lane);
                id[u] = p < all_pairs ? __ldg(a.topk_idx + p) : -1;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int first = p0 + u * kLocalThreads;
                if (first >= all_pairs) break;
                const bool named = id[u] >= 0 && id[u] < E;
                bad = bad || id[u] < -1 || id[u] >= E;
                const unsigned bits = __ballot_sync(full, named);
                if (lane == 0) pair_bits[first >> 5] = bits;
                if (few) {
                    unsigned same = bits;
#pragma unroll
                    for (int i = 0; i < 5; ++i) {
                        const unsigned plane = __ballot_sync(full, id[u] >> i & 1);
                        same &= lane >> i & 1u ? plane : ~plane;
                    }
                    const unsigned high = __ballot_sync(full, id[u] >> 5 & 1);
                    const int before = own_first - first;  // pairs of the step that belong to earlier CTAs
                    const unsigned earlier = before >= 32 ? full : before <= 0 ? 0u : (1u << before) - 1u;
                    mine[0] += __popc(same & ~high) + (__popc(same & ~high & earlier) << 16);
                    mine[1] += __popc(same & high) + (__popc(same & high & earlier) << 16);
                } else if (named) {
                    atomicAdd(&counts[id[u]], first + static_cast<int>(lane) < own_first ? 0x10001u : 1u);
                }
            }
        }
        if (few)
            for (int i = 0; i < 2; ++i)
                if (mine[i] != 0) atomicAdd(&counts[lane + 32 * i], mine[i]);
        if (tid == 0) pair_bits[pair_words - 1] = 0;
        if (bad) sh->flag = 1;  // (the CTA that owns the token says so)
        start_first_loads();
    }
    if constexpr (!cached) {
        unsigned* bits = reinterpret_cast<unsigned*>(total);
        constexpr int kLastFlag = 1 << 30;  // the pair of the chunk's last token in its expert carries the count forward
        int routed_before = 0;              // (last warp) routed tokens of earlier chunks
        for (int c0 = 0; c0 < nt; c0 += 32) {
            const int pairs = min(32, nt - c0) * K;
            for (int p = tid; p < pairs; p += kLocalThreads) {
                const std::int64_t e = (c0 == 0 && p == tid) ? first_id : __ldg(a.topk_idx + static_cast<std::size_t>(t0 + c0) * K + p);
                const int tl = p / K, k = p % K;
                int mine = -1;
                if (e < -1 || e >= E) {
                    record_error(rc, a.error, kErrInvalidRouting, t0 + c0 + tl, k);
                    sh->flag = 1;
                } else if (e >= 0) {
                    if (atomicOr(&bits[e], 1u << tl) >> tl & 1u) {  // the token names this expert twice
                        int at = k;
                        for (int k2 = k + 1; k2 < K; ++k2)
                            if (a.topk_idx[static_cast<std::size_t>(t0 + c0 + tl) * K + k2] == e) at = k2;
                        record_error(rc, a.error, kErrInvalidRouting, t0 + c0 + tl, at);
                        sh->flag = 1;
                    } else {
                        mine = static_cast<int>(e);
                    }
                }
                pair_e[c0 * K + p] = mine;
            }
            __syncthreads();
            for (int p = tid; p < pairs; p += kLocalThreads) {
                const int e = pair_e[c0 * K + p], tl = p / K;
                if (e < 0) continue;
                const unsigned set = bits[e];
                const int ord = base[e] + __popc(set & ((1u << tl) - 1u));
                pair_ord[c0 * K + p] = ord | (tl == 31 - __clz(set) ? kLastFlag : 0);
            }
            if (warp == kLocalWarps - 1) {
                bool routed = false;
                if (c0 + static_cast<int>(lane) < nt)
                    for (int k = 0; k < K; ++k) routed = routed || pair_e[(c0 + lane) * K + k] >= 0;
                const unsigned m = __ballot_sync(full, routed);
                if (c0 + static_cast<int>(lane) < nt) unique[c0 + lane] = routed ? routed_before + __popc(m & lt_mask) : ~(routed_before + __popc(m & lt_mask));
                routed_before += __popc(m);
                if (lane == 0) sh->routed = routed_before;
            }
            __syncthreads();
            for (int p = tid; p < pairs; p += kLocalThreads) {
                const int e = pair_e[c0 * K + p];
                if (e < 0) continue;
                const int ord = pair_ord[c0 * K + p];
                if (ord & kLastFlag) {
                    pair_ord[c0 * K + p] = ord & ~kLastFlag;
                    base[e] = (ord & ~kLastFlag) + 1;
                    bits[e] = 0;
                }
            }
            __syncthreads();
        }
    }
    if constexpr (whole) {
        __syncthreads();
        for (int i = tid; i < E; i += kLocalThreads) {
            base[i] = static_cast<int>(counts[i] >> 16);
            total[i] = static_cast<int>(counts[i] & 0xffffu);
        }
        const unsigned k_mask = K == 32 ? full : (1u << K) - 1u;
        for (int w = warp; w < token_words; w += kLocalWarps) {
            const int t = w * 32 + static_cast<int>(lane), at = t * K;
            bool routed = false;
            if (t < T) routed = (__funnelshift_r(pair_bits[at >> 5], pair_bits[(at >> 5) + 1], at & 31) & k_mask) != 0;
            const unsigned bits = __ballot_sync(full, routed);
            if (lane == 0) token_bits[w] = bits;
        }
        // (no look at the rank's error word here: a read behind the row loads waits for them, 2048 tokens 2 us.  What this CTA itself
        // has found wrong is in the flag, and so is what was wrong before the launch.)
        if (tid == 0 && leaves()) sh->flag = 1;
        __syncthreads();
        if (warp == kLocalWarps - 1) {
            int before = 0;
            for (int w0 = 0; w0 < token_words; w0 += 32) {
                const int w = w0 + static_cast<int>(lane), n = w < token_words ? __popc(token_bits[w]) : 0;
                int incl = n;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int up = __shfl_up_sync(full, incl, o);
                    if (lane >= static_cast<unsigned>(o)) incl += up;
                }
                if (w < token_words) routed_words[w] = before + incl - n;
                before += __shfl_sync(full, incl, 31);
            }
            if (lane == 0) {
                routed_words[token_words] = before;
                sh->first_unique = 0;
                sh->unique_total = before;
            }
        }
        __syncthreads();
        auto routed_before = [&](int t) {  // t <= T
            const int w = t >> 5;
            return routed_words[w] + (t & 31 ? __popc(token_bits[w] & ((1u << (t & 31)) - 1u)) : 0);
        };
        for (int c = tid; c < C; c += kLocalThreads) chan_base[c] = routed_before(min(T, (c + 1) * Tc)) - routed_before(min(T, c * Tc));
        for (int i = tid; i < nt; i += kLocalThreads) {
            const int t = t0 + i, r = routed_before(t);
            unique[i] = token_bits[t >> 5] >> (t & 31) & 1u ? r : ~r;
        }
        if (tid == 0) {
            BEP_PROF(kProfHistDone);
            BEP_PROF(kProfBarrierDone);
        }
    } else if constexpr (!cached) {
        // ---- 3. prefix over the CTAs before this one.  Two levels (groups of kHistGroup CTAs, then the CTAs of the group),
        // as in dispatch.cuh: a CTA reads G / kHistGroup + kHistGroup rows, all at once, instead of G.
        int* const sums = sums_base + static_cast<std::size_t>(generation & 1) * groups * S;
        int* const sums_next = sums_base + static_cast<std::size_t>((generation + 1) & 1) * groups * S;
        const int my_group = b / kHistGroup;
        for (int i = tid; i < W; i += kLocalThreads) {
            const int v = i < E ? base[i] : sh->routed;
            args.hist[static_cast<std::size_t>(b) * W + i] = v;
            if (v != 0) atomicAdd(sums + static_cast<std::size_t>(my_group) * S + i, v);
        }
        if (nt > 0) {  // routed tokens per channel: a thread per channel that this CTA's tokens touch
            auto routed_before = [&](int i) { return i >= nt ? sh->routed : unique[i] >= 0 ? unique[i] : ~unique[i]; };
            for (int ch = t0 / Tc + tid; ch <= (t1 - 1) / Tc; ch += kLocalThreads) {
                const int v = routed_before(min(t1, (ch + 1) * Tc) - t0) - routed_before(max(t0, ch * Tc) - t0);
                if (v != 0) atomicAdd(sums + static_cast<std::size_t>(my_group) * S + W + ch, v);
            }
        }
        for (int i = b * kLocalThreads + tid; i < groups * S; i += G * kLocalThreads) sums_next[i] = 0;
        __threadfence();  // every thread's own stores and reductions, before the CTA arrives
        if (tid == 0) BEP_PROF(kProfHistDone);
        start_first_loads();
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            atomicAdd(&args.counters[0], 1ull);
            while (ptx::ld_acquire_gpu(reinterpret_cast<const std::uint64_t*>(&args.counters[0])) < static_cast<std::uint64_t>(G))
                if (health.give_up(kErrGridBarrier, b, 0)) break;
            __threadfence();
            sh->flag = leaves() || health.failed() ? 1 : 0;
            BEP_PROF(kProfBarrierDone);
        }
        __syncthreads();
        if (!sh->flag) {
            for (int i = tid; i < S; i += kLocalThreads) {
                int before = 0, all = 0;
                for (int g0 = 0; g0 < groups; g0 += 10) {
                    int v[10];
#pragma unroll
                    for (int u = 0; u < 10; ++u) v[u] = g0 + u < groups ? __ldcg(sums + static_cast<std::size_t>(g0 + u) * S + i) : 0;
#pragma unroll
                    for (int u = 0; u < 10; ++u) {
                        all += v[u];
                        before += g0 + u < my_group ? v[u] : 0;
                    }
                }
                if (i >= W) {  // a channel's routed tokens
                    chan_base[i - W] = all;
                    continue;
                }
                int v[kHistGroup];
#pragma unroll
                for (int u = 0; u < kHistGroup; ++u) {
                    const int b2 = my_group * kHistGroup + u;
                    v[u] = b2 < b ? __ldcg(args.hist + static_cast<std::size_t>(b2) * W + i) : 0;
                }
#pragma unroll
                for (int u = 0; u < kHistGroup; ++u) before += v[u];
                if (i < E) {
                    base[i] = before;
                    total[i] = all;
                } else {
                    sh->first_unique = before;
                    sh->unique_total = all;
                }
            }
        }
    } else {
        start_first_loads();
        if (tid == 0 && leaves()) sh->flag = 1;
        for (int p = tid; p < nt * K; p += kLocalThreads) {
            const std::int64_t e = p == tid && p < first_pairs ? first_id : __ldg(a.topk_idx + static_cast<std::size_t>(t0) * K + p);
            pair_e[p] = e >= 0 && e < E ? static_cast<int>(e) : -1;
            pair_ord[p] = a.plan_expert_ord[static_cast<std::size_t>(t0) * K + p];
        }
        for (int i = tid; i < nt; i += kLocalThreads) unique[i] = (a.plan_mask[t0 + i] & 1u) ? a.plan_slot[t0 + i] : -1;
        for (int i = tid; i < 1 + E + C; i += kLocalThreads) {
            const int v = a.plan_counts[i];
            if (i == 0) sh->unique_total = v;
            else if (i <= E) total[i - 1] = v;
            else chan_base[i - 1 - E] = v;
        }
    }
    __syncthreads();
    bool failed = sh->flag != 0;
    if (tid == 0) BEP_PROF(kProfPrefixScan);

    // ---- aligned scan over experts (a thread takes consecutive bins), scan over channels (last warp) ----------
    int own_from = 0, own_to = 0;
    unsigned long long run = 0;  // padded rows in the upper half, true rows in the lower
    auto padded = [&](int count) { return a.alignment == 1 ? count : (count + a.alignment - 1) / a.alignment * a.alignment; };
    if (!failed) {
        const int per = (E + kLocalThreads - 1) / kLocalThreads;
        own_from = min(E, tid * per);
        own_to = min(E, own_from + per);
        for (int i = own_from; i < own_to; ++i) run += static_cast<unsigned long long>(padded(total[i])) << 32 | static_cast<unsigned>(total[i]);
        unsigned long long incl = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long v = __shfl_up_sync(full, incl, o);
            if (lane >= static_cast<unsigned>(o)) incl += v;
        }
        if (lane == 31) sh->warp_sum[warp] = incl;
        run = incl - run;  // what comes before this thread's bins inside the warp
    }
    __syncthreads();
    unsigned long long all_rows = 0;
    if (!failed) {
#pragma unroll
        for (int w = 0; w < kLocalWarps; ++w) {
            const unsigned long long s = sh->warp_sum[w];
            if (w < warp) run += s;
            all_rows += s;
        }
        int at = static_cast<int>(run >> 32);
        for (int i = own_from; i < own_to; ++i) {
            eoff[i] = at;
            at += padded(total[i]);
        }
        if (tid == 0) eoff[E] = static_cast<int>(all_rows >> 32);
        if (warp == kLocalWarps - 1) {
            int before = 0;
            for (int c0 = 0; c0 < C; c0 += 32) {
                const int v = c0 + static_cast<int>(lane) < C ? chan_base[c0 + lane] : 0;
                if (b == G - 1 && c0 + static_cast<int>(lane) < C) {
                    a.recv_chan_counts[c0 + lane] = v;
                    if (!cached) a.plan_counts[1 + E + c0 + lane] = v;
                }
                int incl = v;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int up = __shfl_up_sync(full, incl, o);
                    if (lane >= static_cast<unsigned>(o)) incl += up;
                }
                if (c0 + static_cast<int>(lane) < C) chan_base[c0 + lane] = before + incl - v;
                before += __shfl_sync(full, incl, 31);
            }
        }
    }
    __syncthreads();
    if (!failed && (static_cast<int>(all_rows >> 32) > args.expanded_cap || sh->unique_total > args.unique_cap)) {
        if (tid == 0) record_error(rc, a.error, kErrCapacity, static_cast<int>(all_rows >> 32), sh->unique_total);
        failed = true;
    }
    if (tid == 0) {
        const std::int64_t now = static_cast<std::int64_t>(ptx::globaltimer_ns());
        for (int r = b; r < C; r += G) {
            std::int64_t* prof = a.profile + static_cast<std::size_t>(r) * 16;
            prof[kProfCountsSent] = prof[kProfOrdinalsDone] = prof[kProfRolesSplit] = now;
            prof[kProfCountsArrived] = prof[kProfPrefixReady] = prof[kProfTxDone] = now;
        }
        if (b == G - 1) {
            a.prefix_tx_ts[0] = static_cast<std::int64_t>(t_start);
            a.prefix_tx_ts[1] = now;
        }
        for (int r = b; r < C; r += G) {
            a.prefix_tx_ts[(r + 1) * 2 + 0] = 0;
            a.prefix_tx_ts[(r + 1) * 2 + 1] = now;
        }
    }

    if (pooled && !cached && !failed) {
        // the plan of the tokens that any CTA may move, before the first of them is claimed
        for (int q = own_tokens * K + tid; q < nt * K; q += kLocalThreads)
            a.plan_expert_ord[static_cast<std::size_t>(t0) * K + q] = pair_e[q] >= 0 ? pair_ord[q] + base[pair_e[q]] : -1;
        for (int i = own_tokens + tid; i < nt; i += kLocalThreads) {
            const bool routed = unique[i] >= 0;
            a.plan_mask[t0 + i] = routed ? 1u : 0u;
            a.plan_slot[t0 + i] = routed ? unique[i] + sh->first_unique - chan_base[(t0 + i) / Tc] : -1;
        }
        __threadfence();
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            atomicAdd(&args.counters[3], 1ull);
        }
    }

    // ---- 4. rows -------------------------------------------------------------------------------------------------------
    const std::size_t out_row_bytes = static_cast<std::size_t>(H) * (recv_fp8 ? 1 : 2);
    auto* const recv_bytes = reinterpret_cast<std::uint8_t*>(a.recv_x);
    const int map_stride = 2 + 2 * K;
    if (warp < row_warps && !failed) {
        bool plans_seen = !pooled || cached, more = pooled;
        for (int n = 0; n < started; ++n) {
            const int buffer = warp * stages + n % stages;
            const int t = sh->token[buffer], c = t / Tc, i = t - t0;
            const bool own = !pooled || n < stages;  // from this CTA's tables, else from the plan in global memory
            int e = -1, ord = -1, j = -1;
            float wgt = 1.0f;
            if (lane < static_cast<unsigned>(K)) {
                const std::size_t at = static_cast<std::size_t>(t) * K + lane;
                if (a.topk_w) wgt = __ldg(a.topk_w + at);
                if (own) {
                    e = pair_e[i * K + lane];
                    if (e >= 0) ord = pair_ord[i * K + lane] + base[e];
                } else {
                    const std::int64_t e64 = __ldg(a.topk_idx + at);
                    ord = __ldcg(a.plan_expert_ord + at);
                    e = e64 >= 0 && e64 < E ? static_cast<int>(e64) : -1;
                }
            }
            if (own) {
                if (unique[i] >= 0) j = cached ? unique[i] : unique[i] + sh->first_unique - chan_base[c];
            } else {
                const int slot = __ldcg(a.plan_slot + t);
                if (__ldcg(a.plan_mask + t) & 1u) j = slot;
            }
            const bool routed = j >= 0;  // j: ordinal in the channel
            const unsigned valid = __ballot_sync(full, e >= 0);
            int row = -1;  // this lane's output row
            if (routed) {
                if (expand) row = e >= 0 ? eoff[e] + ord : -1;
                else if (lane == 0) row = chan_base[c] + j;
            }
            unsigned char* slot = rows_sm + static_cast<std::size_t>(buffer) * slot_bytes;
            if (!__all_sync(full, mbar_wait_bounded(&sh->mbar[buffer], static_cast<unsigned>(n / stages) & 1u, health))) {
                failed = true;
                break;
            }
            float scale = 1.0f;
            if (recv_fp8 && routed) {
                scale = quantise_row_in_place(slot, H);
                ptx::fence_proxy_async_smem();
                __syncwarp();
            }
            // every lane with a row starts its own copy: the bulk groups are the lanes' own
            // (Layers that read E4M3 rows back at once are as fast where they leave L2 first: 555 tokens 456 us, 4096 1870.)
            if (row >= 0) {
                std::uint8_t* const dst = recv_bytes + static_cast<std::size_t>(row) * out_row_bytes;
                if (recv_fp8) ptx::bulk_s2g(dst, slot, static_cast<unsigned>(out_row_bytes), policy);
                else ptx::bulk_s2g(dst, slot, static_cast<unsigned>(out_row_bytes));
            }
            ptx::bulk_commit();
            // the next token: claimed now, its number arrives while this row's copies drain
            const bool refill = more && n + 1 >= stages;
            unsigned long long claim = 0;
            if (refill && lane == 0) claim = atomicAdd(&args.counters[4], 1ull);
            if (routed) {
                int* map = a.comb_map + (static_cast<std::size_t>(c) * Qf + j) * map_stride;
                if (lane == 0) *reinterpret_cast<int2*>(map) = make_int2(t, expand ? __popc(valid) : 1);
                if (expand) {
                    if (row >= 0) {
                        if (recv_fp8) a.recv_scale[row] = scale;
                        a.recv_idx[row] = e;
                        a.recv_w[row] = wgt;
                        std::int64_t* meta = a.source_meta + static_cast<std::size_t>(row) * 3;
                        meta[0] = 0;
                        meta[1] = t;
                        meta[2] = lane;
                        *reinterpret_cast<int2*>(map + 2 + 2 * __popc(valid & lt_mask)) = make_int2(row, __float_as_int(wgt));
                    }
                } else {
                    const int r = __shfl_sync(full, row, 0);
                    if (lane < static_cast<unsigned>(K)) {
                        a.recv_idx[static_cast<std::size_t>(r) * K + lane] = e;
                        a.recv_w[static_cast<std::size_t>(r) * K + lane] = e >= 0 ? wgt : 0.0f;
                    }
                    if (lane == 0) {
                        if (recv_fp8) a.recv_scale[r] = scale;
                        std::int64_t* meta = a.source_meta + static_cast<std::size_t>(r) * 3;
                        meta[0] = 0;
                        meta[1] = t;
                        meta[2] = -1;
                        *reinterpret_cast<int2*>(map + 2) = make_int2(r, __float_as_int(1.0f));
                    }
                }
            }
            if (!cached && own) {
                if (lane < static_cast<unsigned>(K)) a.plan_expert_ord[static_cast<std::size_t>(t) * K + lane] = ord;
                if (lane == 0) {
                    a.plan_mask[t] = routed ? 1u : 0u;
                    a.plan_slot[t] = routed ? j : -1;
                }
            }
            // its load goes into the oldest buffer, once the copies have left that
            if (refill) {
                if (!plans_seen) {  // every CTA has written its part of the plan (they all do before their first row)
                    bool seen = true;
                    if (lane == 0)
                        while (ptx::ld_acquire_gpu(reinterpret_cast<const std::uint64_t*>(&args.counters[3])) < static_cast<std::uint64_t>(G))
                            if (health.give_up(kErrGridBarrier, b, 1)) {
                                seen = false;
                                break;
                            }
                    plans_seen = __all_sync(full, seen) != 0;
                    if (!plans_seen) {
                        failed = true;
                        break;
                    }
                }
                int next_t = -1;
                while (true) {
                    claim = __shfl_sync(full, claim, 0);
                    const int f = static_cast<int>(claim % G), next_i = own_tokens + static_cast<int>(claim / G);
                    more = next_i < most_tokens;
                    const int f_t0 = static_cast<int>(static_cast<long long>(T) * f / G), f_t1 = static_cast<int>(static_cast<long long>(T) * (f + 1) / G);
                    if (more && f_t0 + next_i < f_t1) next_t = f_t0 + next_i;
                    if (!more || next_t >= 0) break;
                    // a CTA with one token less than the others leaves a gap in the numbering: claim again
                    if (lane == 0) claim = atomicAdd(&args.counters[4], 1ull);
                }
                if (next_t >= 0) {
                    local_wait_read(stages - 1);
                    __syncwarp();
                    if (lane == 0) start_load(started, next_t);
                    ++started;
                    __syncwarp();
                }
            }
        }
    }
    if (failed && warp < row_warps) {
        // loads that are still under way: give them a bounded time to land before shared memory goes away
        for (int n = max(0, started - stages); n < started; ++n)
            for (unsigned polls = 0; !ptx::mbar_try_wait(reinterpret_cast<std::uint64_t*>(&sh->mbar[warp * stages + n % stages]),
                                                         static_cast<unsigned>(n / stages) & 1u) && polls < (1u << 20); ++polls)
                ptx::nanosleep(64);
    }
    if (!failed) {
        // Rows between the experts' segments: experts go round the CTAs, their rows round the warps.  (A warp per expert, CTA after
        // CTA, left them to a few SMs: 64 tokens, 32 experts, top-8, hidden 7168, padded to multiples of 256 907 us, now 76;
        // the general kernel, a warp per channel, 148.)
        if (expand && a.zero_padding) {
            for (int el = b; el < E; el += G) {
                for (int row = eoff[el] + total[el] + warp; row < eoff[el + 1]; row += kLocalWarps) {
                    if (recv_fp8) {
                        for (int x = lane; x < H; x += 32) recv_bytes[static_cast<std::size_t>(row) * H + x] = 0;
                        if (lane == 0) a.recv_scale[row] = 0.0f;
                    } else {
                        zero_row(recv_bytes + static_cast<std::size_t>(row) * out_row_bytes, H, true);
                    }
                    if (lane == 0) {
                        a.recv_idx[row] = -1;
                        a.recv_w[row] = 0.0f;
                    }
                    if (lane < 3) a.source_meta[static_cast<std::size_t>(row) * 3 + lane] = -1;
                }
            }
        }
        if (b == G - 1) {
            for (int i = tid; i < E; i += kLocalThreads) {
                a.expert_counts[i] = total[i];
                a.expert_offsets[i] = eoff[i];
                a.expert_prefix[i] = eoff[i] + total[i];
                a.source_expert_prefix[i] = 0;
                if (!cached) a.plan_counts[1 + i] = total[i];
            }
            if (tid == 0) {
                a.expert_offsets[E] = eoff[E];
                a.source_offsets[0] = 0;
                a.source_offsets[1] = sh->unique_total;
                a.unique_count[0] = sh->unique_total;
                a.expanded_count[0] = static_cast<std::int64_t>(all_rows & 0xffffffffull);
                if (!cached) a.plan_counts[0] = sh->unique_total;
            }
        }
    }
    bulk_wait_group_read<0>();  // the row buffers have been read; the rows themselves are complete when the launch is
    const bool any_failed = __syncthreads_or(failed ? 1 : 0) != 0;

    // ---- epilogue: the last CTA settles the launch ---------------------------------------------------------------
    if (tid == 0) {
        BEP_PROF(kProfRxDone);
        BEP_PROF(kProfEnd);
        if (any_failed) return;  // the rank has failed: nothing of it is used again
        if (alone) {
            // launches of a buffer are stream-ordered: the next one sees all of this, whichever CTA wrote it when.  (The end needs no
            // reset: what an earlier launch left in the tensor, or its zeroes, is before any time of this one.)
            atomicMax(reinterpret_cast<unsigned long long*>(&a.timestamps[1]), static_cast<unsigned long long>(ptx::globaltimer_ns()));
            if (b == 0) a.timestamps[0] = static_cast<std::int64_t>(t_start);
            if (b == G - 1) {
                for (int i = 0; i < 8; ++i) a.stats[i] = i == kStatLocalRows ? sh->unique_total : 0;
                if (ptx::ld_volatile(&rc->sticky[0]) == 0) {
                    ptx::st_relaxed_sys(flag_ptr(rc->seg[rc->rank], rc->lay.done_off, rc->rank), epoch_before + 1);
                    rc->epochs[0] = epoch_before + 1;
                }
            }
            return;
        }
        __threadfence();
        if (atomicAdd(&args.counters[1], 1ull) + 1ull == static_cast<unsigned long long>(G)) {
            __threadfence();
            for (int i = 0; i < 8; ++i) a.stats[i] = i == kStatLocalRows ? sh->unique_total : 0;
            a.timestamps[0] = static_cast<std::int64_t>(~__ldcg(&args.counters[2]));
            a.timestamps[1] = static_cast<std::int64_t>(ptx::globaltimer_ns());
            for (int i = 0; i < 5; ++i) args.counters[i] = 0ull;
            if (ptx::ld_volatile(&rc->sticky[0]) == 0) {
                const std::uint64_t epoch = epoch_before + 1;
                ptx::st_release_sys(flag_ptr(rc->seg[rc->rank], rc->lay.done_off, rc->rank), epoch);
                rc->epochs[0] = epoch;
                if (!cached && !whole) *generation_at = generation + 1;
            }
        }
    }
#undef BEP_PROF
}

#endif  // __CUDACC__

}  // namespace bep
