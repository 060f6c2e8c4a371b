// Compute-bound W8A8 GEMM with per-row scales on CTA pairs (tcgen05 cta_group::2): out[m,n] = D((float(acc) * sx[m])
// * sw[n]) (+ fp32 residual), optionally followed by the finishing chain (bias, 16-bit residual, scales, activation).
// Replaces reference quant_gemm_sm80.cu:14-82 / quant_gemm_sm90.cu:16-69 for compute-bound shapes.
//
// Two SMs share one tile of 256 tokens x `channels` output channels (64 to 256 in steps of 64). The tokens are the
// MMA's M rows: each CTA of the pair loads 128 token rows and HALF of the tile's weight rows into its own shared
// memory and keeps 128 token rows x `channels` accumulators in its own tensor memory; the even CTA issues the
// M=256 MMAs for both. Compared with one-CTA 128x256 tiles this cuts the bytes every SM pulls from L2 per MMA by
// a third, which is what bounds 8-bit GEMMs at these K (the tensor pipe needs 96 B/clk/SM of operands otherwise).
// Persistent clusters, two accumulators in tensor memory so the epilogue of tile i overlaps the MMAs of tile i+1.
// No TMA multicast: each CTA issues its own loads; they carry the cta_group::2 qualifier only so that they can
// signal the barrier in the leader CTA.
//
// Channel tile: chosen per problem by pair_channel_tile (quant_linear_geometry.h). A batch whose 256-wide tiles leave
// many pairs idle takes narrower ones.
//
// Epilogue: one thread = one token row. Per 64-channel slab the eight or sixteen warps (two or four per 32-lane quadrant,
// 32 or 16 channels each) pull their accumulators, finish them and lay the 16-bit rows down in a swizzled shared-memory slab
// that one thread hands to a TMA store, which clips ragged M and N. The 16-bit residual of the chain comes in the
// same way, prefetched by TMA into the slabs the results will overwrite while the MMAs run. What it replaces: direct
// row-wise stores (32 rows per warp instruction: 24 cycles per column of 128 tokens, 84 with a residual) and, for
// wide outputs, a transposition through shared-memory patches with a barrier per 16 tokens (37 and 95 cycles).
// Sixteen warps where the chain follows, because the last tile's epilogue, and that of every tile with an activation, is not hidden:
// eight / sixteen, 750 x 1024 -> 4096 (INT8) with bias 8.1 / 7.6 us, with GELU 9.6 / 8.9; 2048 x 2048 -> 2048 11.7 / 11.2, 13.3 / 12.6;
// a block of 750 x 1024 with GELU 31.4 / 29.5. Plain rows keep eight: a decoder layer of 1025 rows 87.6 / 89.2, of 2048 FP8 137 / 138.
// The producers' split (weights, tokens) is that of quant_prefill_grouped_sm100.cuh.
//
// Barrier protocol (L = leader, even rank; P = peer):
//   full[s]      in L : L's producers arrive with expect_tx for BOTH CTAs' bytes; all four producers'
//                       TMA loads complete their bytes on it.
//   empty[s]     in L and P : one multicast tcgen05.commit after the MMAs that read stage s.
//   acc_full[b]  in L and P : multicast commit after the last MMA of a tile.
//   acc_empty[b] in L : one arrival per epilogue warp of each CTA (the peer's arrive remotely).
//   residual_full[i] in each CTA : the residual slab i of the current tile has landed.
// Every wait is bounded; on expiry the CTA flags the status word and runs to the common exit.
#pragma once
#include "kernels/quant_linear_sm100.cuh"

namespace tts::b200 {

__host__ __device__ constexpr int pair_epilogue_warps(int chain) { return chain ? 16 : 8; }
__host__ __device__ constexpr int pair_threads(int chain) { return 32 * (pair_epilogue_warps(chain) + 4); } // + two producers, MMA issuer, waiter
constexpr int kSlabChannels = 64;
constexpr uint32_t kSlabBytes = kBlockChannels * kSlabChannels * 2; // 128 token rows of 128 bytes

struct PairArgs {
    int m, n, k;
    const float *sx, *sw;
    const float *residual_f32; // [m, n], added before the first rounding (instances without the chain: optional)
    int *status;
    int channels, stages; // channel tile and ring stages
    int early;            // the weights are complete (GemmArgs)
    FusedEpilogue ep;     // read by the chain instances only
};

// Instances: `Chain` compiles the finishing chain into the epilogue (bit 0; bit 1: with a gate, bit 2: with an activation beyond
// ReLU, which cost registers and code that the others would miss: 31.7 against 33.4 us for a 750-row block); `F16` is the output type (else bf16).
template <Type F, int Chain, bool F16>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(pair_threads(Chain), 1)
w8a8_tcgen05_prefill_pair(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                          const __grid_constant__ CUtensorMap map_out, const __grid_constant__ CUtensorMap map_residual,
                          const __grid_constant__ PairArgs a) {
    constexpr bool kInt = F == Type::I8;
    constexpr int kTokens = kPrefillTokens, kMyTokens = kTokens / 2; // per tile, per CTA
    constexpr int kWarps = pair_epilogue_warps(Chain), kColumns = 256 / kWarps; // epilogue warps; channels of a slab that each takes
    constexpr int kAccumulatorColumns = 256;                         // spacing of the two accumulators
    const int channels = a.channels, stages = a.stages;
    const int weight_bytes = channels / 2 * kBlockK, stage_bytes = weight_bytes + kMyTokens * kBlockK; // per CTA
    const bool skip16 = Chain && a.ep.residual != nullptr;
    const int slabs = channels / kSlabChannels, buffers = skip16 ? kPairResidualSlabs : kPairSlabs;
    const uint32_t idesc = kInt ? ptx::idesc_i8(kTokens, channels) : ptx::idesc_e4m3(kTokens, channels);

    extern __shared__ uint8_t dynamic_smem[];
    __shared__ alignas(8) uint64_t full_bar[kPairMaxStages], empty_bar[kPairMaxStages], acc_full[2], acc_empty[2];
    __shared__ alignas(8) uint64_t residual_full[kPairResidualSlabs];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    __shared__ alignas(16) float sw_tile[kAccumulatorColumns]; // weight scales of the tile being finished
    __shared__ alignas(16) uint16_t bias_tile[Chain ? kAccumulatorColumns : 8];

    const uint32_t raw_base = ptx::smem_u32(dynamic_smem);
    const uint32_t tiles_base = (raw_base + 1023u) & ~1023u;
    const uint32_t slab_base = tiles_base + uint32_t(stages * stage_bytes);
    const int warp = ptx::warp_index(), lane = threadIdx.x & 31;
    const uint32_t rank = ptx::cluster_ctarank();
    const bool leader = rank == 0;
    const int n_tiles = (a.n + channels - 1) / channels, m_tiles = (a.m + kTokens - 1) / kTokens;
    const int tiles = n_tiles * m_tiles;
    const int clusters = gridDim.x / 2, cluster_id = blockIdx.x / 2;
    const int kb_count = (a.k + kBlockK - 1) / kBlockK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            ptx::mbar_init(ptx::smem_u32(&full_bar[s]), 2); // the leader's producers with both CTAs' bytes
            ptx::mbar_init(ptx::smem_u32(&empty_bar[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            ptx::mbar_init(ptx::smem_u32(&acc_full[b]), 1);
            ptx::mbar_init(ptx::smem_u32(&acc_empty[b]), 2 * kWarps);
        }
        for (int i = 0; i < kPairResidualSlabs; ++i) ptx::mbar_init(ptx::smem_u32(&residual_full[i]), 1);
        abort_flag = 0;
        ptx::fence_barrier_init();
        ptx::fence_proxy_async_smem();
    }
    if (warp == 1) ptx::tmem_alloc_pair(ptx::smem_u32(&tmem_slot), 512);
    ptx::tcgen05_fence_before();
    __syncthreads();
    ptx::cluster_sync(); // both CTAs' barriers are initialised before either signals the other
    ptx::tcgen05_fence_after();
    const uint32_t tmem_base = ptx::warp_uniform(tmem_slot);
    volatile int *abort_ptr = &abort_flag;
    ptx::launch_dependents();
    if (!a.early) ptx::wait_for_upstream();

    if (warp == 0 || warp == kWarps + 3) {
        // ------------------------------------------------------------ producers: weights (0) and tokens (the last warp); both CTAs
        // Whole warps run the loop so that addresses and coordinates stay warp-uniform (a copy takes them from
        // uniform registers); one elected lane issues. Announced weights need no upstream kernel, so their producer fills the
        // ring ahead of it.
        const bool weights = warp == 0;
        if (ptx::elect_one()) ptx::prefetch_tensormap(weights ? &map_w : &map_x);
        if (!weights) ptx::wait_for_upstream();
        const uint32_t full_leader = ptx::map_to_rank(ptx::smem_u32(&full_bar[0]), 0);
        const uint32_t bytes = uint32_t(weights ? weight_bytes : kMyTokens * kBlockK), place = weights ? 0u : uint32_t(weight_bytes);
        const CUtensorMap *map = weights ? &map_w : &map_x;
        int stage = 0, filled = 0; // filled: K blocks so far, over all tiles
        uint32_t phase = 0;
        bool ok = true;
        for (int tile = cluster_id; tile < tiles && ok; tile += clusters) {
            const int y = weights ? (tile % n_tiles) * channels + int(rank) * (channels / 2) : (tile / n_tiles) * kTokens + int(rank) * kMyTokens;
            for (int kb = 0; kb < kb_count; ++kb, ++filled) {
                if (filled >= stages) {
                    ok = __all_sync(0xffffffffu, ptx::mbar_wait(ptx::smem_u32(&empty_bar[stage]), phase ^ 1u, abort_ptr));
                    if (!ok) break;
                }
                if (ptx::elect_one()) {
                    if (leader) ptx::mbar_arrive_expect_tx(ptx::smem_u32(&full_bar[stage]), 2 * bytes);
                    ptx::tma_load_2d_pair(tiles_base + uint32_t(stage * stage_bytes) + place, map, full_leader + uint32_t(stage) * 8u, kb * kBlockK, y);
                }
                __syncwarp();
                if (++stage == stages) { stage = 0; phase ^= 1u; }
            }
        }
    } else if (warp == 1 || warp == kWarps + 2) {
        // ------------------------------------------------------------ MMA issuer (1) and its waiter, leader CTA only
        // The whole warp runs the loop (warp-uniform stage arithmetic); one elected lane issues the
        // four MMAs of a K block from a single instruction block and commits.
        // A barrier test between MMA issues waits behind them: about 550 cycles per K block, which the 512 MMA cycles of
        // a 256-channel tile hide and a narrower tile's do not (a wait costs such a tile about 200 of them). There
        // the waiter warp tests the barriers and hands its verdict over at a named hardware barrier, once per K block.
        // Both walk the same sequence and neither leaves it early; after a failed wait every later one returns at once.
        const bool use_waiter = channels < 256;
        if (leader && (warp == 1 || use_waiter)) {
            int stage = 0, local = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int tile = cluster_id; tile < tiles; tile += clusters, ++local) {
                const int buffer = local & 1;
                const uint32_t d = tmem_base + uint32_t(buffer * kAccumulatorColumns);
                for (int kb = 0; kb < kb_count; ++kb) {
                    if (warp != 1 || !use_waiter) {
                        if (kb == 0) ok = ok && ptx::mbar_wait(ptx::smem_u32(&acc_empty[buffer]), ((uint32_t(local) >> 1) & 1u) ^ 1u, abort_ptr);
                        ok = ok && ptx::mbar_wait(ptx::smem_u32(&full_bar[stage]), phase, abort_ptr);
                    }
                    if (warp != 1 || !use_waiter) ok = __all_sync(0xffffffffu, ok); // also brings the lanes together
                    if (use_waiter) ok = ptx::pair_barrier_and(ok);
                    if (warp == 1) {
                        ptx::tcgen05_fence_after();
                        const uint32_t tile_smem = tiles_base + uint32_t(stage * stage_bytes);
                        const uint32_t lo_w = ptx::smem_desc_lo_k128(tile_smem), lo_x = ptx::smem_desc_lo_k128(tile_smem + uint32_t(weight_bytes));
                        if (ok && ptx::elect_one()) {
                            if (kInt) ptx::mma_i8_pair_k128(d, lo_x, lo_w, idesc, uint32_t(kb > 0));
                            else ptx::mma_f8_pair_k128(d, lo_x, lo_w, idesc, uint32_t(kb > 0));
                            ptx::tcgen05_commit_pair(ptx::smem_u32(&empty_bar[stage]), 3);
                            if (kb + 1 == kb_count) ptx::tcgen05_commit_pair(ptx::smem_u32(&acc_full[buffer]), 3);
                        }
                        __syncwarp();
                    }
                    if (++stage == stages) { stage = 0; phase ^= 1u; }
                }
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue warps (both CTAs)
        const int e_thread = threadIdx.x - 64;
        const int quadrant = warp & 3, quarter = (warp - 2) >> 2; // tensor-memory lanes; which kColumns channels of a slab
        const int row = quadrant * 32 + lane; // token row of this CTA's half = tensor-memory lane
        const uint32_t lane_base = tmem_base + (uint32_t(quadrant * 32) << 16);
        const bool storer = e_thread == 0; // issues every slab's TMA traffic
        uint8_t *slab_ptr = dynamic_smem + (slab_base - raw_base);
        const float *__restrict__ residual = a.residual_f32;
        if (storer) ptx::prefetch_tensormap(&map_out);
        ptx::wait_for_upstream();
        uint32_t slab_count = 0;      // slabs stored so far, over all tiles
        uint32_t residual_phase = 0;  // bit i: parity of residual_full[i]'s next completion (ragged tiles use fewer slabs)
        int local = 0;
        for (int tile = cluster_id; tile < tiles; tile += clusters, ++local) {
            const int buffer = local & 1;
            const int n0 = (tile % n_tiles) * channels;
            const int m0 = (tile / n_tiles) * kTokens + int(rank) * kMyTokens;
            const int token = m0 + row;
            const bool token_ok = token < a.m;
            const int valid_slabs = m0 < a.m ? min(slabs, (a.n - n0 + kSlabChannels - 1) / kSlabChannels) : 0;
            if (skip16 && storer) {
                // This tile's residual slabs, into the buffers its results will overwrite: the last tile's stores
                // must have been read out of them.
                ptx::bulk_wait_read<0>();
                for (int i = 0; i < valid_slabs; ++i) {
                    const uint32_t bar = ptx::smem_u32(&residual_full[i]);
                    ptx::mbar_arrive_expect_tx(bar, kSlabBytes);
                    ptx::tma_load_2d(slab_base + uint32_t(i) * kSlabBytes, &map_residual, bar, n0 + i * kSlabChannels, m0);
                }
            }
            const float scale_x = token_ok ? a.sx[token] : 0.f;
            if (e_thread < kAccumulatorColumns) sw_tile[e_thread] = n0 + e_thread < a.n && e_thread < channels ? a.sw[n0 + e_thread] : 0.f;
            if (Chain && e_thread < kAccumulatorColumns)
                bias_tile[e_thread] = a.ep.bias && n0 + e_thread < a.n && e_thread < channels
                                          ? static_cast<const uint16_t *>(a.ep.bias)[n0 + e_thread] : uint16_t(0);
            // One barrier publishes the scales and makes the verdict of the wait common to all epilogue
            // warps: they leave the loop together or not at all.
            if (!ptx::barrier_and(1, 32 * kWarps, ptx::mbar_wait(ptx::smem_u32(&acc_full[buffer]), (uint32_t(local) >> 1) & 1u, abort_ptr)))
                break;
            ptx::tcgen05_fence_after();
            bool ok = true;
#pragma unroll 1
            for (int slab = 0; slab < valid_slabs; ++slab, ++slab_count) {
                const int c0 = slab * kSlabChannels + quarter * kColumns; // this thread's columns of the tile
                uint32_t r[kColumns];
                ptx::tmem_load<kColumns>(lane_base + uint32_t(buffer * kAccumulatorColumns + c0), r);
                const uint32_t place = skip16 ? uint32_t(slab) : slab_count % kPairSlabs;
                uint8_t *out_row = slab_ptr + place * kSlabBytes + uint32_t(row) * 128u;
                ptx::tmem_load_wait();
                if (skip16) {
                    ok = ptx::mbar_wait(ptx::smem_u32(&residual_full[slab]), (residual_phase >> slab) & 1u, abort_ptr);
                    residual_phase ^= 1u << slab;
                }
                const uint4 *gate_row = (Chain & 2) && token_ok ? gate_at(a.ep, token, n0 + c0) : nullptr;
                const float *skip_row = residual && token_ok && n0 + c0 < a.n ? residual + size_t(token) * a.n + n0 + c0 : nullptr;
#pragma unroll
                for (int q = 0; q < kColumns / 8; ++q) { // eight channels = one 16-byte chunk of the slab row
                    uint4 *chunk = reinterpret_cast<uint4 *>(out_row + (((quarter * (kColumns / 8) + q) ^ (row & 7)) * 16));
                    const float4 w_lo = *reinterpret_cast<const float4 *>(&sw_tile[c0 + 8 * q]);
                    const float4 w_hi = *reinterpret_cast<const float4 *>(&sw_tile[c0 + 8 * q + 4]);
                    const float w8[8] = {w_lo.x, w_lo.y, w_lo.z, w_lo.w, w_hi.x, w_hi.y, w_hi.z, w_hi.w};
                    float value[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float acc = kInt ? float(int(r[8 * q + i])) : __uint_as_float(r[8 * q + i]);
                        value[i] = __fmul_rn(__fmul_rn(acc, scale_x), w8[i]);
                    }
                    if (skip_row && n0 + c0 + 8 * q < a.n) { // N is a multiple of 16
                        const float4 s_lo = __ldg(reinterpret_cast<const float4 *>(skip_row + 8 * q));
                        const float4 s_hi = __ldg(reinterpret_cast<const float4 *>(skip_row + 8 * q + 4));
                        const float s8[8] = {s_lo.x, s_lo.y, s_lo.z, s_lo.w, s_hi.x, s_hi.y, s_hi.z, s_hi.w};
#pragma unroll
                        for (int i = 0; i < 8; ++i) value[i] = __fadd_rn(value[i], s8[i]);
                    }
                    uint4 packed = pack8x16<F16>(value);
                    if (Chain)
                        packed = chain8<F16, (Chain & 2) != 0>(a.ep, packed, *reinterpret_cast<const uint4 *>(&bias_tile[c0 + 8 * q]),
                                             gate_row && n0 + c0 + 8 * q < a.n ? __ldg(gate_row + q) : make_uint4(0, 0, 0, 0),
                                             skip16 ? *chunk : make_uint4(0, 0, 0, 0));
                    *chunk = packed;
                }
                if (Chain & 4) {
                    // A pass of its own over the thread's finished row: nothing but its values is live in it.
                    activate_chunks<F16, kColumns / 8>([&](int q) { return reinterpret_cast<uint4 *>(out_row + (((quarter * (kColumns / 8) + q) ^ (row & 7)) * 16)); },
                                            a.ep.activation, a.ep.alpha);
                }
                ptx::fence_proxy_async_smem(); // the rows are about to be read by the TMA engine
                // With two buffers the next slab's must be free by the time this barrier lets anyone write it.
                if (!skip16 && storer) ptx::bulk_wait_read<0>();
                ok = ptx::barrier_and(1, 32 * kWarps, ok);
                if (!ok) break;
                if (storer) {
                    ptx::tma_store_2d(&map_out, slab_base + place * kSlabBytes, n0 + slab * kSlabChannels, m0);
                    ptx::bulk_commit();
                }
            }
            if (!ok) break;
            // Hand the accumulator back to the leader's MMA issuer (remote arrive from the peer CTA).
            ptx::tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive_cluster(ptx::map_to_rank(ptx::smem_u32(&acc_empty[buffer]), 0));
        }
        if (storer) ptx::bulk_wait_read<0>(); // the slabs must outlive their stores
        ptx::tcgen05_fence_before();
    }

    // Neither CTA may leave while the other can still signal its barriers or read its shared memory.
    __syncthreads();
    ptx::cluster_sync();
    if (warp == 1) {
        ptx::tcgen05_fence_after();
        ptx::tmem_dealloc_pair(tmem_base, 512);
    }
    if (threadIdx.x == 0 && abort_flag) atomicExch(a.status, 1 + int(blockIdx.x));
}
} // namespace tts::b200
