// Tile geometry of the tcgen05 GEMM family and the shared-memory budget of one launch shape. Host
// and device code share these numbers; the planner uses them to list only shapes that fit.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace tts::b200 {
constexpr int kBlockChannels = 128; // MMA M: weight rows per tile
constexpr int kBlockK = 128;        // bytes of K per pipeline stage (one 128B-swizzled TMA box)
constexpr int kMaxStages = 12;
constexpr int kRowsPerPass = 16;    // token rows the epilogue warps finish per pass (16 threads x 8 channels per row)
constexpr int kMaxSplits = 8;       // portable thread-block cluster size
constexpr int kPrefillTokens = 256; // token tile of the persistent per-row kernel
constexpr int kWeightStreamTokens = 64; // up to here one token tile covers the batch and a decoder chain's plans apply
constexpr int kGroupedTokens = 128; // token tile of the persistent K-group kernel
constexpr size_t kSmemBudget = 224 * 1024; // dynamic part per CTA: all but 3 KiB of the SM, which is what the static barriers and a co-resident quantizer CTA of the next launch need
// CTA-pair prefill kernel. Shared memory: a ring of stages (128 token rows + half of the tile's weight rows) and
// 16 KiB slabs of finished 16-bit rows: two that alternate, or four when the epilogue adds a 16-bit residual (a
// whole tile's residual is prefetched into them).
constexpr int kPairMaxStages = 10, kPairSlabs = 2, kPairResidualSlabs = 4;
constexpr size_t kPairSlabBytes = 16 * 1024, kPairBytes = 6 * 32 * 1024 + kPairSlabs * kPairSlabBytes;
inline int pair_stages(int channels, bool residual) {
    const size_t ring = kPairBytes - (residual ? kPairResidualSlabs : kPairSlabs) * kPairSlabBytes;
    return std::min(kPairMaxStages, int(ring / (size_t(kBlockChannels + channels / 2) * kBlockK)));
}
// Channel tile of the CTA-pair kernel for `rows` tokens on `pairs` pairs: the width out of 64, 128, 192, 256 that
// minimises the estimated cycles. Per 128-byte K block a tile of C channels takes the tensor pipe's 2C cycles and
// never less than 325 (measured at 64 and 128 channels: operand arrival and hand-over), so the widest tile is the
// most efficient one and narrower ones win only where they fill pairs that would idle. The epilogue
// (`column_cycles` per channel) runs under the next tile's K loop where there is one. A launch on all pairs takes
// about a microsecond longer than one on 32 of them, whatever K is. The constants are fitted to launches of 160 to
// 8192 rows on K = 512 to 6144, N = 256 to 12288 (the choice is within 5 % of the best width on nearly all).
constexpr double kPairColumnCycles = 16; // scale, round, store
struct PairTile {
    int channels;
    double cycles;
};
inline PairTile pair_channel_tile(int rows, int channels, int kb_count, int pairs, double column_cycles) {
    PairTile best{256, 0};
    for (int c = 256; c >= kBlockChannels / 2; c -= kBlockChannels / 2) {
        const int64_t tiles = int64_t((channels + c - 1) / c) * ((rows + kPrefillTokens - 1) / kPrefillTokens);
        const int64_t waves = (tiles + pairs - 1) / pairs;
        const double main_loop = double(kb_count) * std::max(2.1 * c, 325.0) + 800, epilogue = column_cycles * c + 800;
        const double cycles = main_loop + epilogue + double(waves - 1) * std::max(main_loop, epilogue) +
                              65.0 * double(std::max<int64_t>(0, std::min<int64_t>(tiles, pairs) - 32));
        if (c == 256 || cycles < 0.97 * best.cycles) best = {c, cycles};
    }
    return best;
}

// Channel tile of the persistent K-group kernel: 128, or 64 while the 64-wide tiles fit one wave (the rescale per K block then
// takes two thirds as long on twice the multiprocessors: 512 x 2048 x 6144 16.1 against 24 us).
inline int grouped_channel_tile(int rows, int channels, int sms) {
    return int64_t((channels + 63) / 64) * ((rows + kGroupedTokens - 1) / kGroupedTokens) <= sms ? 64 : 128;
}

struct LaunchShape {
    bool fits = false;
    int stages = 0, owned_passes = 0;
    size_t tile_region = 0, smem = 0;
};
// K groups per 128-byte K block (1, 2 or 4 for group widths 128, 64, 32): the narrower of the two
// operands' widths decides, an operand without K groups counts as 128.
inline int group_units(int input_group, int weight_group) {
    const int narrow = std::min(input_group ? input_group : kBlockK, weight_group ? weight_group : kBlockK);
    return kBlockK / std::max(32, narrow);
}
// Shared memory of one CTA of the weight-streaming kernel: alignment slack + pipeline stages
// (unsplit: later the transposed [token][channel] tile of 4-byte partials) + split-K slots the
// cluster peers push into + the K-group scales of the CTA's K range, one pair per group.
inline LaunchShape launch_shape(int bn, bool grouped, int kb_per_split, int splits, int units = 1) {
    const size_t stage = size_t(kBlockChannels + bn) * kBlockK;
    const size_t transposed = splits == 1 ? size_t(bn) * kBlockChannels * sizeof(float) : 0;
    const int passes = (bn + kRowsPerPass - 1) / kRowsPerPass;
    const int owned = splits > 1 ? (passes + splits - 1) / splits : 0;
    const size_t reduce = size_t(splits > 1 ? splits : 0) * owned * kRowsPerPass * kBlockChannels * sizeof(float);
    const size_t scales = grouped ? size_t(kb_per_split) * units * (bn + kBlockChannels) * sizeof(float) : 0;
    const size_t fixed = 1024 + reduce + scales;
    LaunchShape shape;
    if (fixed + std::max(2 * stage, transposed) > kSmemBudget) return shape;
    // As many stages as fit (capped by the K blocks of one CTA): the ring is what gets prefetched
    // while the upstream kernel is still running. Measured on the decode chain, deep rings with one
    // CTA per SM beat half-size rings with two co-resident CTAs.
    int stages = int((kSmemBudget - fixed) / stage);
    stages = std::max(2, std::min({stages, kMaxStages, std::max(2, kb_per_split)}));
    shape.fits = true;
    shape.stages = stages;
    shape.owned_passes = owned;
    shape.tile_region = std::max(size_t(stages) * stage, transposed);
    shape.smem = fixed + shape.tile_region;
    return shape;
}
// The same kernel when it quantizes 16-bit activations itself: the ring holds weights only, every K block's token tile stays.
constexpr int dense_tokens(bool grouped) { return grouped ? 32 : 16; } // widest tile; dense_pays takes at most eight rows with one scale per row
struct DenseShape : LaunchShape {
    int token_offset = 0, largest_offset = 0;
};
inline DenseShape dense_launch_shape(int bn, bool grouped, int kb_per_split, int splits) {
    const LaunchShape usual = launch_shape(bn, grouped, kb_per_split, splits);
    const size_t stage = size_t(kBlockChannels) * kBlockK, tokens = size_t(kb_per_split) * bn * kBlockK;
    DenseShape shape;
    if (!usual.fits) return shape;
    const size_t largest = grouped ? 0 : size_t(2) * bn * sizeof(uint32_t);
    const size_t fixed = usual.smem - usual.tile_region + tokens + largest;
    if (fixed + 2 * stage > kSmemBudget) return shape;
    shape.fits = true;
    shape.stages = std::max(2, std::min({int((kSmemBudget - fixed) / stage), kMaxStages, std::max(2, kb_per_split)}));
    shape.owned_passes = usual.owned_passes;
    shape.token_offset = int(shape.stages * stage); // at least the transposed tile of an unsplit launch (32 tokens x 128 channels x 4 bytes)
    shape.tile_region = size_t(shape.token_offset) + tokens;
    shape.smem = fixed - tokens + shape.tile_region;
    shape.largest_offset = int(shape.smem - largest - 1024); // from the 1024-byte aligned start
    return shape;
}
// Whether quantizing inside the GEMM is possible (per-row scales: a thread's registers hold its part of a row) and pays. It takes
// the launch of the quantizer out, 3.1 of 6.2 us on the host; on the device it is no shorter, since every CTA encodes its K range of
// all rows. One call after another, two launches against one: K=2048 -> 2048 in four splits 6.1 -> 5.1 us at one row, 5.4 at eight;
// -> 4096 in two 6.2 -> 5.4, 5.8; -> 12288 unsplit 6.5 -> 6.4 at three rows, but 6.3 -> 6.6 at four and 6.9 at eight; K groups,
// 6144 -> 2048 in six 6.3 -> 6.0 at one, 6.7 -> 6.5 at eight, 7.3 -> 8.2 at sixteen. So the line lies by a CTA's share of blocks.
inline bool dense_pays(int rows, int reduction, int kb_per_split, bool grouped) {
    if (grouped) return rows * kb_per_split <= 64;
    int spread = 1; // rows the eight warps share, one to eight
    while (spread < rows) spread *= 2;
    return spread <= 8 && int64_t(spread) * reduction <= 16384 && rows * kb_per_split <= 48;
}
// In a graph, where the quantizer's launch costs no host time. A decoder layer's four projections, captured, a projection in two launches
// against one: INT8 5.3 -> 5.7 us at one row, 5.5 -> 6.0 at eight (1024 -> 1024 alone 4.1 -> 4.8); K groups FP8 6.0 -> 5.7 at one row, 6.1 ->
// 5.9 at three, but 6.2 -> 6.7 at five, where the widest projection takes two launches whatever the rule.
inline bool dense_pays_captured(int rows, bool grouped) { return grouped && rows <= 4; }
} // namespace tts::b200
