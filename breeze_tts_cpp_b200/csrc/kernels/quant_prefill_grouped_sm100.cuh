// K-group W8A8 GEMM (group_int8 / group_fp8 beyond decode) for sm_100a: persistent CTAs over tiles of 128 tokens x
// `Channels` (64 or 128) output channels, K-group size 128 on BOTH operands.
//
// Arithmetic (reference grouped_gemm, src/ops/kernels/quant/quant_grouped.cu:16-169): every K block
// of 128 is its own integer/fp8 dot product p_g, and out[m,n] = D(sum_g float(p_g) * (sx_g[m] *
// sw_g[n])) (+ fp32 residual), optionally followed by the finishing chain. The tensor cores therefore produce one
// partial tile per K block, and CUDA cores rescale and add it; that second part is what bounds this kernel (INT8: issue,
// 147 instructions per rescale warp and K block, 88 of them the arithmetic and its scale reads, 69 % of the slots; FP8 and many waves: the 32 KB per K block each SM
// pulls from L2).
//
//   warp 0     : producer. Per K block one pipeline stage (128 token rows + `Channels` weight rows of 128 B, 128-byte
//                swizzle) by TMA and one slot of a small ring for the scales of that K block, on the same barrier: the
//                channels' by TMA, the tokens' by 4-byte asynchronous copies (a row count need not be a multiple of 4).
//   warp 1     : MMA issuer, whole warp in the loop, elected lane issues. The tokens are the MMA's M rows. Four (eight)
//                accumulators rotate through tensor memory, so the tensor cores run that many K blocks
//                ahead of the rescale. It never tests an mbarrier itself: a test waits behind the MMAs in flight.
//   warp 18    : waiter. Tests "accumulator free" and "stage full" for the next K block and hands the
//                result to warp 1 through a named hardware barrier (64 threads), which is free.
//   warps 2-17 : per K block, pull the accumulator into registers (lane = token, a quarter of the channels per
//                warp), hand the buffer back at once, then result += float(p) * (sx * sw) with packed
//                two-wide fp32 instructions. After the last K block the finished rows leave through swizzled
//                shared-memory slabs and TMA stores, the chain's residual having been prefetched into the same slabs (as in
//                quant_prefill_pair_sm100.cuh).
// Sixteen rescale warps: the chain wait - load - hand back - arithmetic of one warp is latency, four warps per scheduler
// hide one another's (eight warps with twice the channels each took about 1100 cycles per K block whatever the format).
// Measured, GEMM alone, M=4096: INT8 12288 x 2048 220 -> 164 us, 2048 x 6144 110 -> 88; FP8 192 -> 144 and 92 -> 76; with a row
// count that is no multiple of four (1021) the weight-streaming kernel used to run: FP8 102 -> 44 us.
// Every wait is bounded; on expiry the CTA flags the status word and runs to the common exit.
#pragma once
#include "kernels/quant_linear_sm100.cuh"

namespace tts::b200 {

constexpr int kGroupedMaxStages = 7;
__host__ __device__ constexpr int grouped_stages(int channels) { return channels == 64 ? kGroupedMaxStages : 5; } // what shared memory holds
// Scale slots need no barriers of their own. They are filled with their stage, so an accumulator that is full implies its
// slot is. And slot c is rewritten for K block c + kScaleSlots only once the MMAs of block c + kScaleSlots - stages
// have retired, which the rescale warps allowed by emptying the accumulator of a block at most 8 before that, after they were
// done with the block before that one: c + kScaleSlots - stages - 9 >= c.
constexpr int kScaleSlots = 16;
static_assert(kScaleSlots >= kGroupedMaxStages + 9, "a scale slot could be rewritten while it is read");
constexpr int kGroupedWarps = 16;                          // rescale warps
constexpr int kGroupedThreads = 32 * (kGroupedWarps + 3);  // + producer, MMA issuer, waiter
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

template <Type F, int Channels, int Chain, bool F16>
__global__ void __launch_bounds__(kGroupedThreads, 1)
w8a8_tcgen05_prefill_grouped(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                             const __grid_constant__ CUtensorMap map_sw, const __grid_constant__ CUtensorMap map_out,
                             const __grid_constant__ CUtensorMap map_residual, const __grid_constant__ GroupedArgs a) {
    constexpr bool kInt = F == Type::I8;
    constexpr int BM = kGroupedTokens;
    constexpr int kStages = grouped_stages(Channels);
    constexpr int kAccumulators = 512 / Channels, kColumns = Channels / 4; // kColumns: channels per rescale thread
    constexpr int kSlabs = Channels / 64;
    constexpr int kWeightBytes = Channels * kBlockK, kTokenBytes = BM * kBlockK;
    constexpr int kStageBytes = kWeightBytes + kTokenBytes;
    constexpr uint32_t kRingBytes = kStages * kStageBytes;
    constexpr uint32_t kIdesc = kInt ? ptx::idesc_i8(BM, Channels) : ptx::idesc_e4m3(BM, Channels);

    extern __shared__ uint8_t dynamic_smem[];
    __shared__ alignas(8) uint64_t full_bar[kStages], empty_bar[kStages];
    __shared__ alignas(8) uint64_t acc_full[kAccumulators], acc_empty[kAccumulators];
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
            ptx::mbar_init(ptx::smem_u32(&full_bar[s]), 1 + 32); // the elected lane with the bytes, every lane with its scales
            ptx::mbar_init(ptx::smem_u32(&empty_bar[s]), 1);
        }
        for (int b = 0; b < kAccumulators; ++b) {
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

    if (warp == 0) {
        // ------------------------------------------------------------ producer
        // The whole warp runs the loop so that addresses and coordinates stay warp-uniform; one elected lane issues.
        // The first round of the ring fetches announced weights and their scales before the wait on upstream.
        if (ptx::elect_one()) {
            ptx::prefetch_tensormap(&map_w);
            ptx::prefetch_tensormap(&map_x);
            ptx::prefetch_tensormap(&map_sw);
        }
        const int ahead = int(blockIdx.x) < tiles ? min(kStages, kb_count) : 0;
        const int first_n0 = (int(blockIdx.x) % n_tiles) * Channels;
        const auto load_weights = [&](int stage, int slot, int kb, int n0) {
            const uint32_t bar = ptx::smem_u32(&full_bar[stage]);
            ptx::mbar_arrive_expect_tx(bar, kStageBytes + Channels * 4);
            ptx::tma_load_2d(tiles_base + uint32_t(stage) * kStageBytes, &map_w, bar, kb * kBlockK, n0);
            ptx::tma_load_2d(scale_base + uint32_t(slot) * kScaleSlotBytes, &map_sw, bar, n0, kb);
        };
        for (int i = 0; i < ahead; ++i) {
            if (ptx::elect_one()) load_weights(i, i, i, first_n0);
            __syncwarp();
        }
        ptx::wait_for_upstream();
        int stage = 0, slot = 0, filled = 0; // filled: K blocks so far, over all tiles
        uint32_t phase = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
            const int n0 = (tile % n_tiles) * Channels, m0 = (tile / n_tiles) * BM;
            for (int kb = 0; kb < kb_count; ++kb, ++filled) {
                ok = filled < kStages || ptx::mbar_wait(ptx::smem_u32(&empty_bar[stage]), phase ^ 1u, abort_ptr);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                if (ptx::elect_one()) {
                    if (filled >= ahead) load_weights(stage, slot, kb, n0);
                    ptx::tma_load_2d(tiles_base + uint32_t(stage) * kStageBytes + kWeightBytes, &map_x,
                                     ptx::smem_u32(&full_bar[stage]), kb * kBlockK, m0);
                }
                __syncwarp();
                const float *sx = a.sx + size_t(kb) * a.m + m0 + lane;
                const uint32_t sx_slot = scale_base + uint32_t(slot) * kScaleSlotBytes + uint32_t(kBlockChannels + lane) * 4u;
#pragma unroll
                for (int i = 0; i < BM / 32; ++i) {
                    const bool inside = m0 + lane + 32 * i < a.m;
                    ptx::copy_async4(sx_slot + 128u * i, inside ? sx + 32 * i : a.sx, inside ? 4u : 0u);
                }
                ptx::copy_async_arrive(ptx::smem_u32(&full_bar[stage]));
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
        uint32_t phase = 0, count = 0; // count: K blocks so far, over all tiles
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            for (int kb = 0; kb < kb_count; ++kb, ++count) {
                const uint32_t buffer = count % kAccumulators;
                if (warp != 1) {
                    const uint32_t use = (count / kAccumulators) & 1u;
                    const bool ready = ptx::mbar_wait(ptx::smem_u32(&acc_empty[buffer]), use ^ 1u, abort_ptr) &&
                                       ptx::mbar_wait(ptx::smem_u32(&full_bar[stage]), phase, abort_ptr);
                    (void)ptx::pair_barrier_and(__all_sync(0xffffffffu, ready)); // the vote brings the lanes together
                } else {
                    const bool ready = ptx::pair_barrier_and(true);
                    ptx::tcgen05_fence_after();
                    const uint32_t tile_smem = tiles_base + uint32_t(stage) * kStageBytes;
                    const uint32_t lo_w = ptx::smem_desc_lo_k128(tile_smem), lo_x = ptx::smem_desc_lo_k128(tile_smem + kWeightBytes);
                    const uint32_t d = tmem_base + buffer * uint32_t(Channels);
                    if (ready && ptx::elect_one()) {
                        if (kInt) ptx::mma_i8_k128(d, lo_x, lo_w, kIdesc, 0u);
                        else ptx::mma_f8_k128(d, lo_x, lo_w, kIdesc, 0u);
                        ptx::tcgen05_commit(ptx::smem_u32(&empty_bar[stage]));
                        ptx::tcgen05_commit(ptx::smem_u32(&acc_full[buffer]));
                    }
                    __syncwarp();
                }
                if (++stage == kStages) { stage = 0; phase ^= 1u; }
            }
        }
    } else {
        // ------------------------------------------------------------ rescale + epilogue warps
        const int quadrant = warp & 3, quarter = (warp - 2) >> 2; // tensor-memory lanes; which kColumns channels
        const int row = quadrant * 32 + lane, c0 = quarter * kColumns;
        const uint32_t lane_base = tmem_base + (uint32_t(quadrant * 32) << 16) + uint32_t(c0);
        const bool storer = threadIdx.x == 64; // issues the tile's TMA traffic
        const float *__restrict__ residual = a.residual_f32;
        const float *scales = reinterpret_cast<const float *>(aligned + (scale_base - tiles_base));
        uint8_t *slab_row = aligned + kRingBytes + uint32_t(c0 / 64) * kGroupedSlabBytes + uint32_t(row) * 128u;
        const ptx::IntBias bias_of_int = ptx::int_bias(raw_base);
        if (storer) ptx::prefetch_tensormap(&map_out);
        ptx::wait_for_upstream();
        uint32_t count = 0, residual_phase = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
            const int n0 = (tile % n_tiles) * Channels, m0 = (tile / n_tiles) * BM;
            const int token = m0 + row;
            const bool token_ok = token < a.m;
            const int valid_slabs = min(kSlabs, (a.n - n0 + 63) / 64);
            if (skip16 && storer) { // into the slabs the results will overwrite: the last tile's stores must have left them
                ptx::bulk_wait_read<0>();
                const uint32_t bar = ptx::smem_u32(&residual_full);
                ptx::mbar_arrive_expect_tx(bar, uint32_t(valid_slabs) * kGroupedSlabBytes);
                for (int s = 0; s < valid_slabs; ++s)
                    ptx::tma_load_2d(slab_base + uint32_t(s) * kGroupedSlabBytes, &map_residual, bar, n0 + s * 64, m0);
            }
            uint64_t result[kColumns / 2];
#pragma unroll
            for (int i = 0; i < kColumns / 2; ++i) result[i] = 0ull;
#pragma unroll 1
            for (int kb = 0; kb < kb_count; ++kb, ++count) {
                const uint32_t buffer = count % kAccumulators;
                ok = ptx::mbar_wait(ptx::smem_u32(&acc_full[buffer]), (count / kAccumulators) & 1u, abort_ptr);
                if (!ok) break;
                ptx::tcgen05_fence_after();
                uint32_t r[kColumns];
                ptx::tmem_load<kColumns>(lane_base + buffer * uint32_t(Channels), r);
                ptx::tmem_load_wait();
                // Everything is in registers: the tensor cores may have the buffer back.
                ptx::tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&acc_empty[buffer]));
                const float scale_x = scales[(count % kScaleSlots) * (kScaleSlotBytes / 4) + kBlockChannels + row];
                const uint64_t scale_x2 = ptx::pack2(scale_x, scale_x);
                const uint32_t sw = ptx::pinned(scale_base + (count % kScaleSlots) * kScaleSlotBytes + uint32_t(c0) * 4u);
#pragma unroll
                for (int q = 0; q < kColumns / 4; ++q) {
                    const ulonglong2 sw4 = ptx::ld_shared_2x64(sw + 16u * q); // the same address in every lane: a broadcast
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int i = 4 * q + 2 * h;
                        const uint64_t p = kInt ? ptx::int_to_float2(r[i], r[i + 1], bias_of_int)
                                                : ptx::pack2(__uint_as_float(r[i]), __uint_as_float(r[i + 1]));
                        result[i / 2] = ptx::fma2(p, ptx::mul2(h ? sw4.y : sw4.x, scale_x2), result[i / 2]);
                    }
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
            const uint4 *gate_row = (Chain & 2) && token_ok ? gate_at(a.ep, token, n0 + c0) : nullptr;
            const float *skip_row = residual && token_ok ? residual + size_t(token) * a.n + n0 + c0 : nullptr;
#pragma unroll
            for (int q = 0; q < kColumns / 8; ++q) { // eight channels = one 16-byte chunk of the slab row
                uint4 *chunk = reinterpret_cast<uint4 *>(slab_row + ((((c0 & 63) / 8 + q) ^ (row & 7)) * 16));
                const bool inside = n0 + c0 + 8 * q < a.n; // N is a multiple of 16
                float value[8];
#pragma unroll
                for (int i = 0; i < 4; ++i) ptx::unpack2(result[4 * q + i], value[2 * i], value[2 * i + 1]);
                if (skip_row && inside) {
                    const float4 lo = __ldg(reinterpret_cast<const float4 *>(skip_row + 8 * q)), hi = __ldg(reinterpret_cast<const float4 *>(skip_row + 8 * q + 4));
                    const float s8[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
                    for (int i = 0; i < 8; ++i) value[i] = __fadd_rn(value[i], s8[i]);
                }
                uint4 packed = pack8x16<F16>(value);
                if (Chain) {
                    uint4 bias = make_uint4(0, 0, 0, 0);
                    if (a.ep.bias && inside) {
                        const uint16_t *b = static_cast<const uint16_t *>(a.ep.bias) + n0 + c0 + 8 * q;
                        uint32_t w[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) w[i] = uint32_t(b[2 * i]) | (uint32_t(b[2 * i + 1]) << 16);
                        bias = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                    packed = chain8<F16, (Chain & 2) != 0>(a.ep, packed, bias, gate_row && inside ? __ldg(gate_row + q) : make_uint4(0, 0, 0, 0), skip16 ? *chunk : make_uint4(0, 0, 0, 0));
                }
                *chunk = packed;
            }
            if (Chain & 4)
                activate_chunks<F16, kColumns / 8>(
                    [&](int q) { return reinterpret_cast<uint4 *>(slab_row + ((((c0 & 63) / 8 + q) ^ (row & 7)) * 16)); }, a.ep.activation, a.ep.alpha);
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
