// Grouped expert GEMM for the expanded dispatch layout, on the 5th-generation tensor cores:
// tcgen05.mma issued by one elected thread, operands staged in shared memory by TMA
// (cp.async.bulk.tensor, no multicast), FP32 accumulators in tensor memory (TMEM), read back with
// tcgen05.ld for a fused epilogue.  The reference has no expert GEMM at all (docs/pcie-ep/design.md:304
// puts it out of scope); this is the "grouped SwiGLU expert FFN" that sits between dispatch and combine.
//
//   rows of expert e = A[expert_offsets[e] .. expert_offsets[e] + expert_counts[e])   (device-side ints)
//   plain  : out[row, n]        = sum_k A[row, k] * W[e, n, k]
//   SwiGLU : out[row, n]        = silu(sum_k A[row,k] * W[e, n, k]) * (sum_k A[row,k] * W[e, N + n, k])
//
// A pair of CTAs (a cluster, cta_group::2) multiplies one tile: 256 weight rows x up to 256 activation rows.  The weight rows are
// the M operand (128 per CTA), the activation rows the N operand (half per CTA), so that a tile is as wide as its rows in steps
// of 16: an expert's rows are cut into equal chunks, and nothing is multiplied for rows that are not there beyond those 16.
// For SwiGLU the 256 weight rows are 128 gate and the matching 128 up rows, interleaved in sixteens by the weight's tensor map.
//
// What bounds it.  Few rows per expert: the weights from HBM.  64 tokens, top-8 of 32 experts, 7168 x 2048: gate/up 283 -> 268 us
// (7.0 TB/s), down 154 -> 144.  Many: tensor cores, at the clock that the power limit leaves.  32 experts of 1024 rows, gate/up in BF16:
// 1324 us (1,450 TFLOP/s) for eight launches in a row, 1550 (1,240) for seconds; 2 and 3.5 % of that are the pause between MMAs of such
// launches, which the rest of a layer gets back (see the MMA issuer).  E4M3 inside a layer 910 -> 849 us, down 830 -> 771, without one.
// Between them, and with a short K, the epilogue: 500 rows each, 768 -> 2048 69.9 -> 61.9 us.  Where a few experts have many rows and the
// others about fifty both share a launch, half overlapped: 6 of 500 and 26 of 54 rows, in E4M3 199 -> 181 us (74 and 121 by themselves).
// Where few rows fill the pairs one time and a bit (8 experts of 40 rows, 96 tiles) the last round runs at 125 GB/s of weights per SM:
// 131 -> 72 us.  Stages are as long as the widest tile of the launch needs.  (Stages of each tile's own length in a circle were slower;
// asking weights into L2 ahead of the stages 2 to 80 %.)  Both roles of one thread are entered through elect.sync, see elect_one.
//
// Work decomposition: persistent pairs walk a tile list (expert, channel tile, row chunk) computed on the device from the
// counts -- the host never reads a count.  Per CTA: warp 0 = TMA producer (this CTA's weight rows and its half of the
// activation rows), warp 1 of the leading CTA = MMA issuer for both, warps 2..5 = epilogue.  Shared-memory stages are handed
// over with mbarriers (TMA complete_tx of both CTAs -> the leading CTA's MMA; tcgen05.commit -> both producers), accumulators
// are double buffered in TMEM (tcgen05.commit -> both epilogues; epilogue arrive -> MMA).
//
// Every mbarrier wait is bounded: on expiry the thread latches an abort flag, all roles drain, TMEM
// is released and the kernel returns with status[0] != 0.
#pragma once

#include <cstdint>

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace bep {
namespace gemm {

constexpr int kCtaM = 128;         // weight rows per CTA and tile
constexpr int kMaxRows = 256;      // activation rows per tile
constexpr int kRowStep = 16;       // a tile has a multiple of this many (padded) rows (32: layers of 64 tokens 1.6 % slower, of 4096 0.5 %)
constexpr int kBlockKBytes = 128;  // one 128B-swizzle atom row: 64 bf16 or 128 fp8 elements of K
constexpr int kUmmaKBytes = 32;    // K extent of one tcgen05.mma: 16 bf16 or 32 fp8
constexpr int kThreads = 192;      // 6 warps
constexpr std::uint32_t kWaitLimit = 20u * 1000u * 1000u;  // try_wait probes before giving up (seconds at most)

// Fused down-projection + combine send: instead of writing `out`, the epilogue multiplies every valid row by
// its routing weight and stores it into the slot (token, k) of the token owner's landing area -- local memory or
// a peer's, through the segment table -- so the NVLink transfer of a tile overlaps the MMAs of the next ones.
// When the last CTA of the launch has drained its stores it publishes `epoch` to every rank.
constexpr int kScatterMaxRanks = 16;
struct ScatterTarget {
    unsigned char* seg[kScatterMaxRanks];  // segment of every rank as addressed from this one
    const long long* source_meta;          // [rows][3]: owner rank, token, slot k (-1: padding row)
    const float* row_weights;              // [rows] routing weight of the row; nullptr: 1
    unsigned long long stage_off, sig_off, done_off;  // landing area, "rows are here" flags, "area consumed" flags
    unsigned long long epoch;              // number of this fused call (1, 2, ...), the same on every rank
    unsigned long long* cta_done;          // CTAs of this launch that have finished; the last one puts it back to zero
    unsigned long long timeout_ns;
    int row_stride;                        // bytes between landing slots
    int num_topk, num_ranks, rank, flag_stride;
};

// Two GEMMs of which the second reads what the first writes, launched one behind the other on one stream: the first counts the tiles that
// are written, per expert, and the second starts without waiting for all of the first.  Its CTAs come onto the SMs where the first has ended
// (its pairs do not end together: HBM does not serve all SMs alike), and go on as soon as their own expert is there.  The second finds
// everything from before the first complete: the first has waited for that before it let the second start.
struct Progress {
    unsigned* counters;  // [E + 1]: CTAs' tiles written per expert, CTAs of the second launch that have ended; zero between passes; nullptr: none
    int per_chunk;       // second launch: what the first one counts for a row chunk (2 CTAs x its channel tiles); 0: this launch is the first
    unsigned long long timeout_ns;  // second launch: for the rows of an expert at most, while the first is at work on them
};

struct GroupedGemmParams {
    const int* expert_offsets;  // [E+1] first row of every expert in A / out
    const int* expert_counts;   // [E]   valid rows
    __nv_bfloat16* out;         // [rows, N]
    const float* a_scales;      // FP8 only: one scale per row of A
    const float* w_scales;      // FP8 only: one scale per weight row [E, (2)N]
    int* status;                // [4]: 0 = ok, 1 = a wait expired, 3 = a peer never freed its area
    int num_experts;
    int n;                      // output columns
    int k;                      // reduction length in elements
    Progress progress;
    ScatterTarget scatter;      // only read by the scatter variant
};

// How an expert's rows are cut into tiles: as few as possible, equal but for the last.  (256 each and the rest in one more: the same
// within 1 %, 4096 tokens gate/up 1800 and 1785 us, down 898 and 908.)
struct RowChunks {
    int count, rows;
};
__host__ __device__ constexpr RowChunks row_chunks(int rows) {
    const int count = (rows + kMaxRows - 1) / kMaxRows;
    return {count, count == 0 ? 0 : ((rows + count - 1) / count + kRowStep - 1) / kRowStep * kRowStep};
}
// Each CTA of a pair loads half of a tile's rows: boxes of 8, 16, ... 128 rows, one tensor map each.
constexpr int kBoxes = kMaxRows / kRowStep;
__host__ __device__ constexpr int box_rows(int box) { return (box + 1) * (kRowStep / 2); }
__host__ __device__ constexpr int box_of_rows(int tile_rows) { return (tile_rows + kRowStep - 1) / kRowStep - 1; }
struct ActivationMaps {
    CUtensorMap box[kBoxes];
};

constexpr int kTileW = kCtaM * kBlockKBytes;
// Stages are as long as the widest tile of the launch needs: where all experts have few rows, more of them keep weights on their way.
constexpr int kRingBytes = 6 * (kTileW + kMaxRows / 2 * kBlockKBytes);  // six stages of the widest tiles, more of narrower ones
constexpr int kMaxStages = 10;
// From here on MMAs of a BF16 SwiGLU launch keep a gap, see the MMA issuer: rows x channels x K per SM (222e9 on 148: 0.9 TFLOP, 0.65 ms)
constexpr long long kLongLaunchPerSm = 1500ll * 1000 * 1000;
constexpr int kPauseLoads = 3;
constexpr int kAccCols = kMaxRows;       // TMEM columns of one accumulator set
constexpr int kTmemCols = 2 * kAccCols;  // double buffered
// The epilogue turns the accumulator (lane = channel) round in shared memory, kChunkRows rows at a time in two alternating halves.
// Row pitch: 16 bytes more than a row (a multiple of 128) put the eight rows of a matrix into different banks.
constexpr int kChunkRows = 32;
__host__ __device__ constexpr int staging_pitch(bool swiglu) { return (swiglu ? kCtaM / 2 : kCtaM) * 2 + 16; }
struct alignas(16) GemmShared {
    std::uint64_t full[kMaxStages], empty[kMaxStages], tmem_full[2], tmem_empty[2];
    std::uint32_t tmem_base;
    int abort;
    std::uint32_t zero;
    int most_rows[kThreads / 32];  // of any expert, per warp
    int all_rows[kThreads / 32];   // of all experts, per warp
};
// Behind it, for two tiles in turn: a factor per row (scatter: the routing weight; E4M3: the row's scale) and, for scatter, where the
// row goes (0: nowhere).  Behind the tile's rows lies what was there; what is made of it goes nowhere.
__host__ __device__ constexpr int gemm_smem_bytes(bool swiglu, bool fp8, bool scatter) {
    return 1024 /* alignment slack */ + kRingBytes + 2 * kChunkRows * staging_pitch(swiglu) + static_cast<int>(sizeof(GemmShared)) +
           (fp8 || scatter ? 2 * kMaxRows * 4 : 0) + (scatter ? 2 * kMaxRows * 8 : 0);
}
static_assert(2 * kChunkRows * staging_pitch(true) % 16 == 0 && 2 * kChunkRows * staging_pitch(false) % 16 == 0, "barriers follow the staging");
static_assert(gemm_smem_bytes(false, false, true) <= 227 * 1024 && gemm_smem_bytes(false, true, false) <= 227 * 1024, "one CTA per SM");

}  // namespace gemm
}  // namespace bep
