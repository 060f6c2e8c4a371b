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
} // namespace tts::b200
