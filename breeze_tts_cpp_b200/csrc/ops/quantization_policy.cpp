#include "ops/quantization_policy.h"
#include "kernels/quant_linear_geometry.h"
#include <cmath>
#include <limits>
#include <stdexcept>

namespace tts {
using namespace b200;

// Figures measured on a B200 at 1965 MHz: 6.55 TB/s copy bandwidth; one SM pulls about 85 GB/s
// through TMA when it streams alone, about 60 GB/s inside a chain of launches; one `tcgen05.mma` stream per SM adds up to about 4.5 POP/s; a dependent launch costs
// about 4 us that do not scale with bytes (launch boundary, arrival of the first activation tile,
// accumulator drain and store).
ChipModel ChipModel::b200(int multiprocessors) {
    ChipModel chip;
    chip.sms = multiprocessors > 0 ? multiprocessors : 148;
    chip.memory_bytes_per_us = 6.55e6;
    chip.tensor_ops_per_us = 4.5e9 * chip.sms / 148.;
    chip.scalar_ops_per_us = 128. * 2 * 1965 * chip.sms;
    chip.kernel_us = 4.0;
    chip.warp_tensor_ops_per_us = chip.tensor_ops_per_us / chip.sms;
    chip.warp_instructions_per_us = 4. * 1965;
    chip.cache_bytes = size_t(126) << 20;
    chip.cache_bytes_per_us = 60e3 * chip.sms; // per SM while the next launch of a chain prefetches too (85 GB/s alone)
    return chip;
}

std::string path_name(const LinearPath &p) {
    static const char *kinds[] = {"cublaslt", "gemv", "sm80", "hopper", "grouped", "tcgen05"};
    const int kind = int(p.kind);
    if (kind < 0 || kind > 5) throw std::invalid_argument("invalid linear path kind");
    if (p.kind == LinearKind::Lt) return kinds[0];
    if (p.kind == LinearKind::Gemv)
        return "gemv_tokens" + std::to_string(p.tokens) + "_split" + std::to_string(p.splits);
    return std::string(kinds[kind]) + "_channels" + std::to_string(p.channels) + "_tokens" + std::to_string(p.tokens) +
           "_split" + std::to_string(p.splits);
}

namespace {
bool grouped(const KernelProblem &p) { return p.input_group || p.weight_group; }
int blocks(int size, int tile) { return (size + tile - 1) / tile; }
// Which kernel the launcher picks for a path and plain rows (mirrors launch_quant_linear's dispatch).
bool persistent_per_row(const KernelProblem &p, const LinearPath &path) {
    return !grouped(p) && path.tokens == kPrefillTokens && path.splits == 1;
}
bool persistent_grouped(const KernelProblem &p, const LinearPath &path) {
    return p.input_group == kBlockK && p.weight_group == kBlockK && path.tokens == kGroupedTokens && path.splits == 1;
}
} // namespace

std::vector<LinearPath> quant_linear_candidates(KernelProblem p, KernelLimits limits, Type format) {
    if (format != Type::FP8 && format != Type::I8) throw std::invalid_argument("unsupported quantized storage type");
    std::vector<LinearPath> paths;
    if (p.rows < 1 || p.channels < 1 || p.reduction < 1 || p.reduction % 16) return paths;
    const bool group = grouped(p);
    const int kb_total = blocks(p.reduction, kBlockK);
    int cover = 16;
    while (cover < (group ? kGroupedTokens : kPrefillTokens) && cover < p.rows) cover *= 2;
    std::vector<int> token_tiles{cover};
    // K groups: narrower tiles of the split-K kernel beside the persistent kernel's 128 tokens (they pay on short batches).
    if (group && cover == kGroupedTokens) {
        token_tiles.push_back(64);
        if (p.rows <= 256) token_tiles.push_back(32);
    }
    // Between decode and prefill a batch covers a few narrow tiles: several of them per channel slab (and split K)
    // occupy the machine where one or two 256-token tiles would leave most of it idle. Beyond 1024 rows the
    // 256-token tiles fill it by themselves.
    if (!group && p.rows > kWeightStreamTokens && p.rows <= 1024) {
        token_tiles.push_back(64);
        if (cover > 128) token_tiles.push_back(128);
    }
    for (int tokens : token_tiles)
        for (int splits = 1; splits <= std::min(kb_total, kMaxSplits); ++splits) {
            const LaunchShape shape = launch_shape(tokens, group, blocks(kb_total, splits), splits,
                                                   group_units(p.input_group, p.weight_group));
            if (!shape.fits || (limits.shared_bytes && shape.smem > limits.shared_bytes)) continue;
            paths.push_back({LinearKind::Tcgen05, tokens, kBlockChannels, splits});
        }
    return paths;
}

double linear_cost(KernelProblem p, LinearPath path, Type format, const ChipModel &chip) {
    if (path.kind != LinearKind::Tcgen05) return std::numeric_limits<double>::infinity();
    const int sms = std::max(1, chip.sms);
    const int kb_total = blocks(p.reduction, kBlockK);
    if (persistent_per_row(p, path)) {
        // CTA pairs: the estimate the launcher picks the channel tile by, at 1965 MHz, plus launch and fill. Plans know no
        // epilogue, so this is the plain one; the launcher puts 20 to 75 cycles per column in the place of 16 when a chain follows.
        const PairTile tile = pair_channel_tile(p.rows, p.channels, kb_total, std::max(1, sms / 2), kPairColumnCycles);
        return 1.8 + tile.cycles / 1965.;
    }
    if (persistent_grouped(p, path)) {
        // Waves of 128 tokens x 64 or 128 channels, bound by the fp32 rescale of every K128 partial tile (0.28 and 0.42 us per
        // K block, INT8; FP8 is up to 15 % faster). With a single token tile all CTAs pull the same rows: QKV of 103, 111, 119 and 127 rows on
        // this kernel 50.1, 50.3, 50.6 and 51.3 us a decoder layer, in two splits of 64 tokens 47.4, 48.3, 48.6 and 49.1 (FP8 48.2,
        // 48.3, 48.5 and 48.6 against 46.2, 46.4, 47.4 and 48.4); O of 255 rows, as many CTAs on two tiles, FP8 60.6 against 62.1.
        const int channels = grouped_channel_tile(p.rows, p.channels, sms);
        const double tiles = double(blocks(p.channels, channels)) * blocks(p.rows, kGroupedTokens);
        const double per_block = channels != 64 ? 0.42 : p.rows > kGroupedTokens ? 0.28 : 0.2875;
        return (channels == 64 ? 2.9 : 3.2) + std::ceil(tiles / sms) * kb_total * per_block;
    }
    if (p.rows > kWeightStreamTokens) {
        // Weight-streaming kernel with several token tiles per channel slab. Fitted to launches of 65 to 1024 rows on
        // K = 512 to 6144, N = 1024 to 12288: a base per token tile, a slope per K block (the operand bytes one SM
        // pulls; with K groups the rescale), the split-K exchange (per-row scales: 1.0 to 1.6 us at 64 tokens, 2.1 to 2.4 at
        // 128), and contention for L2 as the grid grows. More than one wave does not pay: CTAs own their multiprocessor's shared memory, so nothing of the next wave overlaps.
        const bool group = grouped(p);
        const int splits = std::max(1, path.splits), per_split = blocks(kb_total, splits);
        const int units = group_units(p.input_group, p.weight_group);
        const LaunchShape shape = launch_shape(path.tokens, group, per_split, splits, units);
        if (!shape.fits) return std::numeric_limits<double>::infinity();
        const int64_t ctas = int64_t(blocks(p.channels, kBlockChannels)) * blocks(p.rows, path.tokens) * splits;
        const int resident = (!group && path.tokens <= 64 && shape.smem <= 108 * 1024) ? 2 : 1;
        // Clusters are placed whole inside a GPC (16 to 20 multiprocessors): count what that leaves unusable.
        const int64_t slots = splits > 1 ? std::max<int64_t>(splits, int64_t(sms) * resident * 16 / 18 / splits * splits)
                                         : int64_t(sms) * resident;
        const int tile = path.tokens <= 32 ? 0 : path.tokens <= 64 ? 1 : path.tokens <= 128 ? 2 : 3;
        static constexpr double kBase[2][4] = {{2.3, 2.5, 3.4, 6.2}, {2.7, 3.4, 5.6, 9.0}};
        static constexpr double kSlope[2][4] = {{0.17, 0.17, 0.17, 0.42}, {0.245, 0.31, 0.44, 0.9}};
        // Up to two token tiles with per-row scales a split costs more by its number of CTAs (those that are no power of two are placed later) and
        // the grid's size less. Decoder layers of 87, 103, 119 and 127 rows (INT8) with QKV unsplit / in two splits of 64 tokens: 36.5 / 36.7,
        // 38.0 / 37.9, 38.2 / 38.8 and 38.4 / 39.0 us called one by one, 33.7 / 33.3, 34.4 / 34.3, 35.8 / 35.2 and 36.1 / 35.3 in a graph.
        // K = 2048 -> 512 in six splits / four: blocks of 87 and 103 rows in a graph 18.1 / 17.1 and 18.5 / 16.9.
        const bool short_batch = !group && p.rows <= 2 * kWeightStreamTokens && path.tokens <= 64;
        const double exchange = splits == 1 ? 0.0
                                : group     ? 0.25 + 0.2 * splits
                                : short_batch ? 0.3 + 0.24 * splits + (splits & (splits - 1) ? 0.15 : 0.0)
                                              : path.tokens <= 64 ? 1.0 + 0.08 * splits : 2.2;
        const double contention = (short_batch ? 0.006 : 0.012) * double(std::max<int64_t>(0, std::min(ctas, slots) - 48));
        const double waves = double((ctas + slots - 1) / slots);
        const double one = kBase[group][tile] + per_split * units * kSlope[group][tile] + exchange + contention;
        return one + (waves - 1.0) * (one - 1.0);
    }
    // Weight-streaming kernel, as it runs inside a decoder chain: the launch starts under programmatic
    // dependent launch while its quantizer still runs, so by the time the activations exist the ring
    // already holds `stages` K blocks of weights. What is left on the critical path is
    //   * the K blocks that did not fit the ring, at what one SM can pull or its share of HBM;
    //   * the part of the ring the launches before leave no time for: with few rows they are short (about 1 us + 0.06 us a
    //     row), so more splits, i.e. less weight per SM, pay (down projection, 5 rows: 4 splits 25.4 us a layer, 6 24.1;
    //     QKV 2 splits 25.3, 4 24.7). Per-row INT8 only: its sums are exact whatever the split, while a split moves the
    //     rounding of FP8 and K-group sums, which a stack of requantized layers amplifies to the format's own noise;
    //   * the MMAs, which cost a fixed ~0.12 us per K block up to 64 tokens (four instructions of at
    //     least 48 tensor-pipe cycles each, however few tokens), more for wider tiles;
    //   * the split-K exchange, about 0.3 us per CTA of the cluster at 64 tokens (less for narrower tiles); clusters of seven and eight lose
    //     about 6 us more (their CTAs are placed late and miss the weight prefetch);
    //   * the epilogue, about 0.4 us per 16-token pass a CTA finishes;
    //   * a crowding term: the more SMs a launch holds, the fewer the next launch of the chain finds
    //     free to start its own prefetch early; uneven K splits cost a little as well.
    // Calibrated on the decoder layer's four shapes at 8 to 64 rows, timed inside the chain.
    const int splits = std::max(1, path.splits), per_split = blocks(kb_total, splits);
    const LaunchShape shape = launch_shape(path.tokens, grouped(p), per_split, splits, group_units(p.input_group, p.weight_group));
    if (!shape.fits) return std::numeric_limits<double>::infinity();
    const double stage_bytes = double(kBlockChannels + path.tokens) * kBlockK;
    const int64_t ctas = int64_t(blocks(p.channels, kBlockChannels)) * blocks(p.rows, path.tokens) * splits;
    // Small tiles leave room for two CTAs per SM; clusters are placed whole.
    const int resident = (!grouped(p) && path.tokens <= 64 && shape.smem <= 108 * 1024) ? 2 : 1;
    const int64_t slots = std::max<int64_t>(splits, int64_t(sms) * resident / splits * splits);
    const double waves = double((ctas + slots - 1) / slots);
    const double per_sm = chip.cache_bytes_per_us > 0 ? chip.cache_bytes_per_us / sms : 60e3;
    const int exposed_blocks = std::max(0, per_split - shape.stages);
    const double exposed = exposed_blocks * stage_bytes *
                           std::max(1.0 / per_sm, double(std::min(ctas, slots)) / (0.84 * chip.memory_bytes_per_us));
    const double mma_block = path.tokens <= 64 ? 0.12 : path.tokens <= 128 ? 0.16 : 0.29;
    const bool exact = format == Type::I8 && !grouped(p);
    const double unhidden = !exact ? 0.0 : std::max(0.0, std::min(per_split, shape.stages) * double(kBlockChannels * kBlockK) / per_sm - 1.0 - 0.06 * p.rows);
    const double compute = unhidden + std::max(per_split * mma_block, exposed + mma_block) * (grouped(p) ? 1.5 : 1.0);
    const double exchange = splits > 1 ? (0.15 + 0.15 * path.tokens / 64.0) * splits + (kb_total % splits ? 0.15 : 0.0) + (splits > 6 ? 6.0 : 0.0) : 0.0;
    const int passes = blocks(std::min(p.rows, path.tokens), kRowsPerPass);
    const double epilogue = 0.4 * (splits > 1 ? blocks(passes, splits) : passes);
    const double crowding = 0.01 * double(std::max<int64_t>(0, std::min(ctas, slots) - 64));
    // Later waves see a cold ring: they stream all of their K blocks.
    const double later_wave = per_split * stage_bytes * std::max(1.0 / per_sm, double(slots) / (0.84 * chip.memory_bytes_per_us)) +
                              exchange + epilogue;
    return chip.kernel_us + compute + exchange + epilogue + crowding + (waves - 1.0) * later_wave;
}

double linear_pipeline_cost(KernelProblem p, LinearPath path, Type format, const ChipModel &chip, LinearFinishWork finish,
                            bool fused, LibraryWork, KernelResources) {
    // Row quantizer: one launch, 2 bytes read and 1 written per activation element.
    const double quantize = chip.kernel_us / 2 + (3.0 * p.rows * p.reduction + 4.0 * p.rows) / chip.memory_bytes_per_us;
    const double gemm = linear_cost(p, path, format, chip);
    if (fused) return quantize + gemm; // the epilogue chain rides in the GEMM's own epilogue
    // A separate finishing pass reads and writes every output element once more.
    const double elements = double(p.rows) * p.channels;
    const double pass = chip.kernel_us / 2 + 4.0 * elements / chip.memory_bytes_per_us +
                        elements * finish.instructions_per_output / (32. * chip.warp_instructions_per_us * chip.sms);
    return quantize + gemm + pass;
}

LinearPath select_linear(KernelProblem p, KernelLimits limits, Type format, const ChipModel &chip, bool, LibraryWork) {
    double best = std::numeric_limits<double>::infinity();
    LinearPath selected;
    for (const LinearPath &path : quant_linear_candidates(p, limits, format)) {
        const double cost = linear_cost(p, path, format, chip);
        if (cost < best - 1e-9) { // ties keep the earlier (narrower split) candidate
            best = cost;
            selected = path;
        }
    }
    if (!std::isfinite(best)) throw std::invalid_argument("no supported quantized GEMM implementation");
    return selected;
}
} // namespace tts
