// K-group W8A8 GEMM (group_int8 / group_fp8 beyond decode) for sm_100a: persistent CTAs over tiles of 128 tokens x
// `Channels` (64 or 128) output channels, K-group size 128 on BOTH operands.
//
// Arithmetic (reference grouped_gemm, src/ops/kernels/quant/quant_grouped.cu:16-169): every K block
// of 128 is its own integer/fp8 dot product p_g, and out[m,n] = D(sum_g float(p_g) * (sx_g[m] *
// sw_g[n])) (+ fp32 residual), optionally followed by the finishing chain. The tensor cores therefore produce one
// partial tile per K block, and CUDA cores rescale and add it. What bounds the kernel is both halves together: the rescale alone takes
// 49 (FP8) or 57 us (INT8) of a 4096 x 6144 -> 2048 GEMM's 68 or 80, the operands and MMAs alone 50 (32 KB per K block and SM, 18 TB/s
// from L2), and each waits for the other at times; the clock falls from 1.96 to 1.82-1.9 GHz besides.
//
//   warps 0, 19: producers of the weights and their scales (0) and of the tokens and theirs (19). Per K block one pipeline stage (128
//                token rows + `Channels` weight rows of 128 B, 128-byte swizzle) by TMA and one slot of a small ring for the scales of
//                that K block, on the same barrier: the channels' by TMA, the tokens' by 4-byte asynchronous copies (a row count
//                need not be a multiple of 4). One warp for both was late: 84.7 against 81.3 us (INT8, as above).
//   warp 1     : MMA issuer, whole warp in the loop, elected lane issues. The tokens are the MMA's M rows. The accumulators of a
//                round (two K blocks) change hands together: a barrier test
//                and a hand-over per round instead of per K block take a fifth of the rescale warps' instructions out. It
//                never tests an mbarrier itself: a test waits behind the MMAs in flight.
//   warp 18    : waiter. Tests "accumulators free" and "stage full" for the next K block and hands the
//                result to warp 1 through a named hardware barrier (64 threads), which is free.
//   warps 2-17 : per K block, pull 32 token rows x a quarter of the channels into registers, then result += float(p) * (sx * sw)
//                with packed two-wide fp32 instructions. After the last K block the finished rows leave through swizzled
//                shared-memory slabs and TMA stores, the chain's residual having been prefetched into the same slabs (as in
//                quant_prefill_pair_sm100.cuh).
// Sixteen rescale warps: the chain wait - load - arithmetic of one warp is latency, four warps per scheduler
// hide one another's (eight warps with twice the channels each took about 1100 cycles per K block whatever the format).
// Measured, GEMM alone, one K block per hand-over, one token row per thread and one producer against this: M=4096, 2048 x 6144: INT8 90 ->
// 80 us, FP8 77 -> 68; 12288 x 2048 at M=1021: 50 -> 44, 45 -> 38; at 64 channels 114 -> 95, 107 -> 84. Short sums gain nothing (three
// K blocks, 1305 x 384 -> 1536: 5.4 -> 5.5 us): there the prologue, the epilogue and the code itself are what takes the time.
// CTA pairs with tiles of 256 x 256 (half the operand bytes) were slower, 90 and 94 us with four accumulators of 128 channels and 82
// and 72 with two of 256: the way from a free accumulator to the next full one crosses the two CTAs.
// Every wait is bounded; on expiry the CTA flags the status word and runs to the common exit.
#pragma once
#include "kernels/quant_linear_sm100.cuh"

namespace tts::b200 {

constexpr int kGroupedMaxStages = 7;
__host__ __device__ constexpr int grouped_stages(int channels) { return channels == 64 ? kGroupedMaxStages : 5; } // what shared memory holds
// K blocks per round: the accumulators change hands once per round. Two rounds of 256 tensor-memory columns alternate at 128 channels,
// four of 128 columns at 64 (one of four K blocks each is as fast, but twice the code, which a chain of launches finds cold).
constexpr int kGroupedRound = 2;
__host__ __device__ constexpr int grouped_buffers(int channels) { return 512 / (kGroupedRound * channels); }
// Scale slots need no barriers of their own. They are filled with their stage, so an accumulator that is full implies its
// slot is. And slot c is rewritten for K block c + kScaleSlots only once the MMAs of block b = c + kScaleSlots - stages have
// retired. Those of b's round were issued when the rescale warps had taken the round `buffers` before it out of tensor memory: at
// least block b - buffers * round, and so they had done with the scales of the block before that, which is c or later.
constexpr int kScaleSlots = 16;
constexpr bool grouped_slots_suffice(int channels) { return kScaleSlots - grouped_stages(channels) - grouped_buffers(channels) * kGroupedRound - 1 >= 0; }
static_assert(grouped_slots_suffice(64) && grouped_slots_suffice(128), "a scale slot could be rewritten while it is read");
constexpr int kGroupedWarps = 16;                          // rescale warps
constexpr int kGroupedThreads = 32 * (kGroupedWarps + 4);  // + two producers, MMA issuer, waiter
constexpr int kRescaleThreads = 32 * kGroupedWarps;
constexpr int kScaleSlotBytes = (kBlockChannels + kGroupedTokens) * 4; // channels, then tokens
constexpr uint32_t kGroupedSlabBytes = kGroupedTokens * 128; // 128 token rows x 64 channels of 16 bits
constexpr size_t grouped_smem(int channels) {
    return 1024 + size_t(grouped_stages(channels)) * (kGroupedTokens + channels) * kBlockK + size_t(channels / 64) * kGroupedSlabBytes +
           size_t(kScaleSlots) * kScaleSlotBytes;
}

struct GroupedArgs {
    int m, n, k;
    const float *sx;           // group-major [k / 128, m]
    const float *residual_f32; // [m, n], added before the first rounding
    int *status;
    int early;                 // the weights and their scales are complete (GemmArgs)
    FusedEpilogue ep;          // read by the chain instances only
};

// What a rescale thread holds of a 32-row x Columns partial tile: rows t, t + 8, t + 16 and t + 24 (t = lane / 4) and of every eight
// channels the pair 2 * (lane % 4), as packed pairs [row k][pair j]. In this shape (16x256b) a thread needs a quarter of the
// channels' scales and four tokens'; one token row per thread (32x32b) needs them all, and those shared-memory reads were a fourth of
// the loop (rescale alone, cycles per 128 x 128 K block: FP8 420 -> 335, INT8 504 -> 460).
template <int Columns> using GroupedSums = uint64_t[4][Columns / 8];
// result += float(p) * (sx * sw) for one K block. `hand_back` runs once the partials are in registers.
template <bool Int, int Columns, class HandBack>
__device__ __forceinline__ void grouped_rescale(GroupedSums<Columns> &result, uint32_t partials, uint32_t sx_at, uint32_t sw_at, HandBack hand_back) {
    uint32_t r[2][Columns / 2]; // 16 token rows each
    ptx::tmem_load_rows16<Columns>(partials, r[0]);
    ptx::tmem_load_rows16<Columns>(partials + (16u << 16), r[1]);
    const float4 sx = ptx::ld_shared_4x32(sx_at);
    uint64_t sw[Columns / 8];
#pragma unroll
    for (int j = 0; j < Columns / 8; ++j) sw[j] = ptx::ld_shared_64(sw_at + 32u * j);
    ptx::tmem_load_wait();
    hand_back();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float scale_x = k == 0 ? sx.x : k == 1 ? sx.y : k == 2 ? sx.z : sx.w;
        const uint64_t scale_x2 = ptx::pack2(scale_x, scale_x);
#pragma unroll
        for (int j = 0; j < Columns / 8; ++j) {
            const uint32_t lo = r[k >> 1][4 * j + 2 * (k & 1)], hi = r[k >> 1][4 * j + 2 * (k & 1) + 1];
            const uint64_t p = Int ? ptx::int_to_float2(lo, hi) : ptx::pack2(__uint_as_float(lo), __uint_as_float(hi));
            result[k][j] = ptx::fma2(p, ptx::mul2(sw[j], scale_x2), result[k][j]);
        }
    }
}
// The tokens' scales of a K block, four bytes per lane and 32 tokens, laid down as a rescale thread reads them: tokens t, t + 8, t + 16
// and t + 24 of a quadrant side by side. Arrives on `bar` once they have landed; zeros past the last token.
__device__ __forceinline__ void grouped_copy_token_scales(const GroupedArgs &a, int kb, int m0, int lane, uint32_t slot, uint32_t bar) {
    const float *sx = a.sx + size_t(kb) * a.m + m0 + lane;
    const uint32_t dst = slot + uint32_t((lane & 7) * 4 + (lane >> 3)) * 4u;
#pragma unroll
    for (int i = 0; i < kGroupedTokens / 32; ++i) {
        const bool inside = m0 + lane + 32 * i < a.m;
        ptx::copy_async4(dst + 128u * i, inside ? sx + 32 * i : a.sx, inside ? 4u : 0u);
    }
    ptx::copy_async_arrive(bar);
}
// A warp's finished sums into the slab of its channels (128 token rows x 64 channels, swizzled), through the chain. `row`: the thread's
// first row (all four are the same modulo 8), `token` its token, `channel` its first channel, `chunk` the slab's 16-byte chunk of it.
template <bool F16, int Chain, int Columns>
__device__ __forceinline__ void grouped_rows_to_slab(const GroupedArgs &a, GroupedSums<Columns> &result, uint8_t *slab, int row, int token,
                                                     int channel, int chunk, bool skip16) {
    constexpr int kWords = Columns / 8;
    const int lane = threadIdx.x & 31;
    if (a.residual_f32) {
#pragma unroll
        for (int i = 0; i < 4 * kWords; ++i) {
            const int k = i / kWords, j = i % kWords, m = token + 8 * k, n = channel + 8 * j;
            if (n >= a.n || m >= a.m) continue; // N is a multiple of 16
            const float2 s = __ldg(reinterpret_cast<const float2 *>(a.residual_f32 + size_t(m) * a.n + n));
            result[k][j] = ptx::add2(result[k][j], ptx::pack2(s.x, s.y));
        }
    }
    const auto slab_word = [&](int k, int j) {
        return reinterpret_cast<uint32_t *>(slab + uint32_t(row + 8 * k) * 128u + (((chunk + j) ^ (row & 7)) * 16) + 4 * (lane & 3));
    };
    uint32_t bias_words[kWords]; // the same for all four rows
    if (Chain) {
#pragma unroll
        for (int j = 0; j < kWords; ++j) {
            const uint16_t *b = static_cast<const uint16_t *>(a.ep.bias) + channel + 8 * j;
            bias_words[j] = a.ep.bias && channel + 8 * j < a.n ? uint32_t(__ldg(b)) | (uint32_t(__ldg(b + 1)) << 16) : 0u;
        }
    }
    // The chain works value by value, so four of a thread's channel pairs at a time stand for its eight consecutive channels.
#pragma unroll
    for (int q = 0; q < kWords; ++q) {
        float value[8];
        uint32_t bias[4] = {0u, 0u, 0u, 0u}, gate[4] = {0u, 0u, 0u, 0u}, skip[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = (4 * q + i) / kWords, j = (4 * q + i) % kWords, m = token + 8 * k, n = channel + 8 * j;
            ptx::unpack2(result[k][j], value[2 * i], value[2 * i + 1]);
            if (Chain) {
                bias[i] = bias_words[j];
                if ((Chain & 2) && n < a.n && m < a.m)
                    gate[i] = __ldg(reinterpret_cast<const uint32_t *>(static_cast<const uint16_t *>(a.ep.gate) +
                                                                       size_t(m / a.ep.rows_per_sequence) * a.ep.gate_ld + n));
                if (skip16) skip[i] = *slab_word(k, j);
            }
        }
        uint4 packed = pack8x16<F16>(value);
        if (Chain)
            packed = chain8<F16, (Chain & 2) != 0>(a.ep, packed, make_uint4(bias[0], bias[1], bias[2], bias[3]),
                                                   make_uint4(gate[0], gate[1], gate[2], gate[3]), make_uint4(skip[0], skip[1], skip[2], skip[3]));
        const uint32_t words[4] = {packed.x, packed.y, packed.z, packed.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) *slab_word((4 * q + i) / kWords, (4 * q + i) % kWords) = words[i];
    }
    if (Chain & 4) { // a pass over the warp's rows, one per thread
        __syncwarp();
        const int mine = (row & ~31) + lane;
        activate_chunks<F16, kWords>([&](int q) { return reinterpret_cast<uint4 *>(slab + uint32_t(mine) * 128u + (((chunk + q) ^ (mine & 7)) * 16)); },
                                     a.ep.activation, a.ep.alpha);
    }
}

template <Type F, int Channels, int Chain, bool F16>
__global__ void __launch_bounds__(kGroupedThreads, 1)
w8a8_tcgen05_prefill_grouped(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                             const __grid_constant__ CUtensorMap map_sw, const __grid_constant__ CUtensorMap map_out,
                             const __grid_constant__ CUtensorMap map_residual, const __grid_constant__ GroupedArgs a) {
    constexpr bool kInt = F == Type::I8;
    constexpr int BM = kGroupedTokens;
    constexpr int kStages = grouped_stages(Channels);
    constexpr int kRound = kGroupedRound, kBuffers = grouped_buffers(Channels), kBufferColumns = kRound * Channels;
    constexpr int kColumns = Channels / 4; // kColumns: channels per rescale warp
    constexpr int kWords = kColumns / 8; // packed channel pairs of one token per rescale thread
    constexpr int kSlabs = Channels / 64;
    constexpr int kWeightBytes = Channels * kBlockK, kTokenBytes = BM * kBlockK;
    constexpr int kStageBytes = kWeightBytes + kTokenBytes;
    constexpr uint32_t kRingBytes = kStages * kStageBytes;
    constexpr uint32_t kIdesc = kInt ? ptx::idesc_i8(BM, Channels) : ptx::idesc_e4m3(BM, Channels);

    extern __shared__ uint8_t dynamic_smem[];
    __shared__ alignas(8) uint64_t full_bar[kStages], empty_bar[kStages];
    __shared__ alignas(8) uint64_t acc_full[kBuffers], acc_empty[kBuffers]; // one pair per round in flight
    __shared__ alignas(8) uint64_t residual_full;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;

    // [pipeline stages | slabs | scale slots], 1024-byte aligned for the swizzled boxes.
    const uint32_t raw_base = ptx::smem_u32(dynamic_smem);
    const uint32_t tiles_base = (raw_base + 1023u) & ~1023u;
    uint8_t *aligned = dynamic_smem + (tiles_base - raw_base);
    const uint32_t slab_base = tiles_base + kRingBytes, scale_base = slab_base + kSlabs * kGroupedSlabBytes;
    const int warp = ptx::warp_index(), lane = threadIdx.x & 31;
    const int n_tiles = (a.n + Channels - 1) / Channels, m_tiles = (a.m + BM - 1) / BM;
    const int tiles = n_tiles * m_tiles;
    const int kb_count = (a.k + kBlockK - 1) / kBlockK;
    const bool skip16 = Chain && a.ep.residual != nullptr;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            ptx::mbar_init(ptx::smem_u32(&full_bar[s]), 2 + 32); // both producers with their bytes, every lane of one with its scales
            ptx::mbar_init(ptx::smem_u32(&empty_bar[s]), 1);
        }
        for (int b = 0; b < kBuffers; ++b) {
            ptx::mbar_init(ptx::smem_u32(&acc_full[b]), 1);
            ptx::mbar_init(ptx::smem_u32(&acc_empty[b]), kGroupedWarps);
        }
        ptx::mbar_init(ptx::smem_u32(&residual_full), 1);
        abort_flag = 0;
        ptx::fence_barrier_init();
        ptx::fence_proxy_async_smem();
    }
    if (warp == 1) ptx::tmem_alloc(ptx::smem_u32(&tmem_slot), 512);
    ptx::tcgen05_fence_before();
    __syncthreads();
    ptx::tcgen05_fence_after();
    const uint32_t tmem_base = ptx::warp_uniform(tmem_slot);
    volatile int *abort_ptr = &abort_flag;
    ptx::launch_dependents();
    if (!a.early) ptx::wait_for_upstream();

    if (warp == 0 || warp == kGroupedWarps + 3) {
        // ------------------------------------------------------------ producers: weights and their scales (0), tokens (19)
        // Whole warps run the loop so that addresses and coordinates stay warp-uniform; one elected lane issues. Announced
        // weights need no upstream kernel, so their producer fills the ring ahead of it.
        const bool weights = warp == 0;
        if (ptx::elect_one()) {
            ptx::prefetch_tensormap(weights ? &map_w : &map_x);
            if (weights) ptx::prefetch_tensormap(&map_sw);
        }
        if (!weights) ptx::wait_for_upstream();
        int stage = 0, slot = 0, filled = 0; // filled: K blocks so far, over all tiles
        uint32_t phase = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
            const int n0 = (tile % n_tiles) * Channels, m0 = (tile / n_tiles) * BM;
            for (int kb = 0; kb < kb_count; ++kb, ++filled) {
                ok = filled < kStages || ptx::mbar_wait(ptx::smem_u32(&empty_bar[stage]), phase ^ 1u, abort_ptr);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                const uint32_t bar = ptx::smem_u32(&full_bar[stage]), tile_smem = tiles_base + uint32_t(stage) * kStageBytes;
                const uint32_t scale_slot = scale_base + uint32_t(slot) * kScaleSlotBytes;
                if (weights) {
                    if (ptx::elect_one()) {
                        ptx::mbar_arrive_expect_tx(bar, kWeightBytes + Channels * 4);
                        ptx::tma_load_2d(tile_smem, &map_w, bar, kb * kBlockK, n0);
                        ptx::tma_load_2d(scale_slot, &map_sw, bar, n0, kb);
                    }
                    __syncwarp();
                } else {
                    if (ptx::elect_one()) {
                        ptx::mbar_arrive_expect_tx(bar, kTokenBytes);
                        ptx::tma_load_2d(tile_smem + kWeightBytes, &map_x, bar, kb * kBlockK, m0);
                    }
                    __syncwarp();
                    grouped_copy_token_scales(a, kb, m0, lane, scale_slot + kBlockChannels * 4u, bar);
                }
                slot = (slot + 1) % kScaleSlots;
                if (++stage == kStages) { stage = 0; phase ^= 1u; }
            }
        }
        ptx::copy_async_wait_all();
    } else if (warp == 1 || warp == kGroupedWarps + 2) {
        // ------------------------------------------------------------ MMA issuer (1) and its waiter
        // Both walk the same K-block sequence and meet once per K block at named barrier 4, which also
        // carries the waiter's verdict. Neither leaves its loop early, so the barrier counts always
        // match; after a failed wait the abort flag makes every later wait return at once and the
        // issuer stops issuing.
        int stage = 0;
        uint32_t phase = 0, round = 0; // rounds so far, over all tiles
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            for (int kb = 0; kb < kb_count; ++kb) {
                const int in_round = kb % kRound;
                const bool last = in_round == kRound - 1 || kb + 1 == kb_count;
                const uint32_t buffer = round % kBuffers;
                if (warp != 1) {
                    const bool ready = (in_round || ptx::mbar_wait(ptx::smem_u32(&acc_empty[buffer]), ((round / kBuffers) & 1u) ^ 1u, abort_ptr)) &&
                                       ptx::mbar_wait(ptx::smem_u32(&full_bar[stage]), phase, abort_ptr);
                    (void)ptx::pair_barrier_and(__all_sync(0xffffffffu, ready)); // the vote brings the lanes together
                } else {
                    const bool ready = ptx::pair_barrier_and(true);
                    ptx::tcgen05_fence_after();
                    const uint32_t tile_smem = tiles_base + uint32_t(stage) * kStageBytes;
                    const uint32_t lo_w = ptx::smem_desc_lo_k128(tile_smem), lo_x = ptx::smem_desc_lo_k128(tile_smem + kWeightBytes);
                    const uint32_t d = tmem_base + buffer * kBufferColumns + uint32_t(in_round * Channels);
                    if (ready && ptx::elect_one()) {
                        if (kInt) ptx::mma_i8_k128(d, lo_x, lo_w, kIdesc, 0u);
                        else ptx::mma_f8_k128(d, lo_x, lo_w, kIdesc, 0u);
                        ptx::tcgen05_commit(ptx::smem_u32(&empty_bar[stage]));
                        if (last) ptx::tcgen05_commit(ptx::smem_u32(&acc_full[buffer]));
                    }
                    __syncwarp();
                }
                if (last) ++round;
                if (++stage == kStages) { stage = 0; phase ^= 1u; }
            }
        }
    } else {
        // ------------------------------------------------------------ rescale + epilogue warps
        const int quadrant = warp & 3, quarter = (warp - 2) >> 2; // tensor-memory lanes; which kColumns channels
        const int row = quadrant * 32 + (lane >> 2), c0 = quarter * kColumns, pair = 2 * (lane & 3);
        const uint32_t lane_base = tmem_base + (uint32_t(quadrant * 32) << 16) + uint32_t(c0);
        const bool storer = threadIdx.x == 64; // issues the tile's TMA traffic
        uint8_t *slab = aligned + kRingBytes + uint32_t(c0 / 64) * kGroupedSlabBytes;
        const uint32_t sx_at = uint32_t(kBlockChannels + quadrant * 32 + (lane >> 2) * 4) * 4u, sw_at = uint32_t(c0 + pair) * 4u;
        if (storer) ptx::prefetch_tensormap(&map_out);
        ptx::wait_for_upstream();
        uint32_t round = 0, slot_at = 0, residual_phase = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
            const int n0 = (tile % n_tiles) * Channels, m0 = (tile / n_tiles) * BM;
            const int valid_slabs = min(kSlabs, (a.n - n0 + 63) / 64);
            if (skip16 && storer) { // into the slabs the results will overwrite: the last tile's stores must have left them
                ptx::bulk_wait_read<0>();
                const uint32_t bar = ptx::smem_u32(&residual_full);
                ptx::mbar_arrive_expect_tx(bar, uint32_t(valid_slabs) * kGroupedSlabBytes);
                for (int s = 0; s < valid_slabs; ++s)
                    ptx::tma_load_2d(slab_base + uint32_t(s) * kGroupedSlabBytes, &map_residual, bar, n0 + s * 64, m0);
            }
            GroupedSums<kColumns> result;
#pragma unroll
            for (int i = 0; i < 4 * kWords; ++i) result[i / kWords][i % kWords] = 0ull;
#pragma unroll 1
            for (int first = 0; first < kb_count; first += kRound, ++round) {
                const int blocks = min(kRound, kb_count - first);
                const uint32_t buffer = round % kBuffers;
                ok = ptx::mbar_wait(ptx::smem_u32(&acc_full[buffer]), (round / kBuffers) & 1u, abort_ptr);
                if (!ok) break;
                ptx::tcgen05_fence_after();
                const uint32_t from = lane_base + buffer * kBufferColumns;
#pragma unroll
                for (int u = 0; u < kRound; ++u) {
                    if (u > 0 && u >= blocks) break;
                    const uint32_t scales = ptx::pinned(scale_base + slot_at);
                    slot_at = (slot_at + kScaleSlotBytes) % (kScaleSlots * kScaleSlotBytes);
                    grouped_rescale<kInt, kColumns>(result, from + uint32_t(u * Channels), scales + sx_at, scales + sw_at, [&] {
                        if (u + 1 < blocks) return;
                        ptx::tcgen05_fence_before(); // the tensor cores may have the round's buffers back
                        __syncwarp();
                        if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&acc_empty[buffer]));
                    });
                }
            }
            // ---- tile finished: rows into the slabs, slabs out by TMA.
            if (skip16) {
                if (ok) ok = ptx::mbar_wait(ptx::smem_u32(&residual_full), residual_phase, abort_ptr);
                residual_phase ^= 1u;
            } else if (storer) {
                ptx::bulk_wait_read<0>(); // the last tile's stores have left the slabs
            }
            // All warps decide together whether the tile is stored; the barrier also publishes that the slabs are free.
            ok = ptx::barrier_and(1, kRescaleThreads, ok && !*abort_ptr);
            if (!ok) break;
            grouped_rows_to_slab<F16, Chain, kColumns>(a, result, slab, row, m0 + row, n0 + c0 + pair, (c0 & 63) / 8, skip16);
            ptx::fence_proxy_async_smem(); // the rows are about to be read by the TMA engine
            (void)ptx::barrier_and(1, kRescaleThreads, true);
            if (storer) {
                for (int s = 0; s < valid_slabs; ++s)
                    ptx::tma_store_2d(&map_out, slab_base + uint32_t(s) * kGroupedSlabBytes, n0 + s * 64, m0);
                ptx::bulk_commit();
            }
        }
        if (storer) ptx::bulk_wait_read<0>(); // the slabs must outlive their stores
        ptx::tcgen05_fence_before();
    }

    __syncthreads();
    if (warp == 1) {
        ptx::tcgen05_fence_after();
        ptx::tmem_dealloc(tmem_base, 512);
    }
    if (threadIdx.x == 0 && abort_flag) atomicExch(a.status, 1 + int(blockIdx.x));
}
} // namespace tts::b200
