// W8A8 GEMM + dequant epilogue for sm_100a: tcgen05 MMA (kind::i8 / kind::f8f6f4), accumulators in
// tensor memory, operands brought in by TMA with the 128-byte swizzle, split-K with an in-kernel,
// fixed-order reduction.
//
// Orientation: the 128-row MMA operand is a slab of 128 output channels of the weight matrix
// W[N,K]; the MMA "N" operand is a tile of BN tokens of X[M,K]. Both are K-contiguous exactly as
// the reference stores them, so no repacking is needed. One accumulator lane = one output channel,
// one accumulator column = one token; a warp storing one token writes 32 consecutive channels.
//
//   per-row scales : out[m,n] = D((float(acc) * sx[m]) * sw[n])
//                    (reference order: src/ops/kernels/quant/quant_gemm_sm80.cu:22-29)
//   K groups       : r += float(p_g) * (sx[g,m] * sw[g,n]) for g ascending, out = D(r)
//                    (reference: src/ops/kernels/quant/quant_grouped.cu:85-168); every group of
//                    128, 64 or 32 along K (the narrower of the two operands' group widths, as in
//                    the reference, :185-199) accumulates into a fresh tensor-memory buffer that the
//                    epilogue warps drain and rescale while the next group's MMAs run. A 128-byte K
//                    block is four 32-byte MMAs, so it splits into one, two or four such units.
//   split-K        : the splits of one output tile form a thread-block cluster. Token rows are dealt
//                    to the CTAs in blocks of 16; every CTA pushes its partial rows straight from
//                    tensor memory into the owner's shared memory (one slot per split, remote
//                    stores over distributed shared memory), one cluster barrier later the owner
//                    sums its slots in split order and finishes the rows. No workspace traffic, no
//                    second launch (replaces reference quant_reduce.cuh:9-29), deterministic.
//   launch overlap : the kernel starts under programmatic dependent launch: barriers, tensor
//                    memory and the first pipeline stages of WEIGHT tiles are set up while the
//                    producer of the activations is still running; only the activation tiles, the
//                    scales and the residual wait for it. Weights nobody has announced as complete
//                    (WeightMaps) wait too: every kernel lets its successor start at once, so an
//                    upstream kernel, or the one before it, may still be writing them.
//   epilogue       : accumulators leave tensor memory lane-per-channel, are transposed through
//                    shared memory, and are finished token-row-wise so that every global access
//                    (fp32 residual, bias, bf16 store) is a coalesced 16-byte vector.
#pragma once
#include "kernels/sm100_ptx.cuh"
#include "kernels/quant_blocks.cuh"
#include "kernels/quant_linear_geometry.h"
#include "kernels/sequence_finish.cuh"
#include "core/tensor.h"
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <type_traits>

namespace tts::b200 {

constexpr int kGemmThreads = 320;   // warp 0 TMA, warp 1 MMA + TMEM, warps 2-9 epilogue
constexpr int kEpilogueThreads = 256;

// Workspace carve-up (owner zeroes the first kWorkspaceHeader bytes once). The GEMM itself needs
// no scratch; only the status word lives here.
constexpr size_t kStatusOffset = 16384;    // int status[4]: nonzero after a bounded wait gave up
constexpr size_t kSettleOffset = 16640;    // int: written by quant_linear_settle, read by nobody
constexpr size_t kWorkspaceHeader = 32768;

struct FusedEpilogue {
    const void *bias = nullptr;         // [N], output dtype
    const void *residual = nullptr;     // [M, residual_ld], output dtype
    const void *gate = nullptr;         // [sequences or 1, gate_ld], output dtype, 16-byte rows
    const float *residual_f32 = nullptr; // [M, N] fp32, added before the first rounding
    float value_scale = 1.f, residual_scale = 1.f, output_scale = 1.f, alpha = .1f;
    int activation = 0;                 // ops::Activation
    int residual_ld = 0;
    int gate_ld = 0, rows_per_sequence = 1; // gate_ld is 0 for a gate that all sequences share
    int residual_vector = 0;            // residual rows are 16-byte aligned
    int plain_residual = 0;             // a residual with value_scale == residual_scale == 1
    int chain = 0;                      // nonzero when anything beyond residual_f32 is requested
};

struct GemmArgs {
    int m, n, k;
    const float *sx, *sw;
    void *out;
    int out_type; // Type::BF16, Type::F16, or Type::I32 (raw accumulators, per-row INT8 only)
    int input_group, weight_group;
    int splits, stages;
    int tile_region; // bytes of shared memory holding the pipeline stages (and, unsplit, the transposed tile)
    int owned_passes; // split-K: 16-row passes each CTA of the cluster may own (slots per split)
    int vector_io;   // every global row touched by the epilogue is 16-byte aligned
    int *status;
    int early; // the weights and their scales are complete: fetch them before the upstream kernel is
    // Failure-path exercise (host-side injection, see quant_linear_inject_wait_expiry): the first weight
    // barrier expects `expiry_extra_bytes` more than its copy delivers, and every wait gives up after
    // `wait_limit_cycles` (0 = the regular limit). Both zero in normal operation.
    int expiry_extra_bytes;
    long long wait_limit_cycles;
    unsigned refill_delay_ns; // the refill waiter's start held back (quant_linear_inject_refill_delay); 0 in normal operation
    FusedEpilogue ep;
};
// Of the instances that quantize 16-bit activations: those, their row stride in elements, and where in the dynamic shared memory
// their quantized tiles lie (behind the weight ring) and the rows' largest magnitudes (behind everything).
struct DenseArgs : GemmArgs {
    const void *x;
    int x_ld, token_offset, largest_offset;
};

// Two 16-bit values in one word -> fp32.
template <bool F16> __device__ __forceinline__ float2 unpack16(uint32_t word) {
    return F16 ? __half22float2(*reinterpret_cast<const __half2 *>(&word))
               : make_float2(__uint_as_float(word << 16), __uint_as_float(word & 0xffff0000u));
}
template <bool F16> __device__ __forceinline__ uint32_t pack2x16(float lo, float hi) {
    if (F16) {
        __half2 h = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<uint32_t *>(&h);
    }
    __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&b);
}
// Sum of two pairs, rounded once. Equal to the finishing pass's fp32 sum rounded to storage: fp32 carries more than
// twice the storage type's precision plus two bits, so its intermediate rounding cannot show.
template <bool F16> __device__ __forceinline__ uint32_t add2x16(uint32_t a, uint32_t b) {
    if (F16) {
        __half2 h = __hadd2(*reinterpret_cast<__half2 *>(&a), *reinterpret_cast<__half2 *>(&b));
        return *reinterpret_cast<uint32_t *>(&h);
    }
    __nv_bfloat162 h = __hadd2(*reinterpret_cast<__nv_bfloat162 *>(&a), *reinterpret_cast<__nv_bfloat162 *>(&b));
    return *reinterpret_cast<uint32_t *>(&h);
}
template <bool F16> __device__ __forceinline__ uint32_t relu2x16(uint32_t v) {
    const float2 f = unpack16<F16>(v);
    return pack2x16<F16>(fmaxf(f.x, 0.f), fmaxf(f.y, 0.f));
}
// Post-GEMM chain on eight consecutive channels of one row, already rounded to storage and packed, up to and
// including ReLU; rounding points follow the reference's separate pass
// (src/ops/kernels/sequence/sequence_internal.cuh:52-74), so a kernel's GEMM + fused chain equals the same kernel's
// GEMM followed by that pass bit for bit (FP8 plans of 128 tokens run another kernel when a chain follows, launch_quant_linear, and its fp32 sums
// may round differently). Every step ends in a storage value, which is why the row can stay packed between them.
// The gate is one more rounding step here instead of a launch and a pass over the output: modulated FP8 block of 4 x 93 x 512,
// 23.7 -> 18.8 us.
template <bool F16, bool Gate = true> __device__ __forceinline__ uint4 chain8(const FusedEpilogue &e, uint4 row, uint4 bias, uint4 gate, uint4 skip) {
    uint32_t v[4] = {row.x, row.y, row.z, row.w};
    const uint32_t b[4] = {bias.x, bias.y, bias.z, bias.w}, k[4] = {skip.x, skip.y, skip.z, skip.w};
    if (e.bias) {
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = add2x16<F16>(v[i], b[i]);
    }
    if (Gate && e.gate) {
        const uint32_t g[4] = {gate.x, gate.y, gate.z, gate.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 x = unpack16<F16>(v[i]), y = unpack16<F16>(g[i]);
            v[i] = pack2x16<F16>(__fmul_rn(x.x, y.x), __fmul_rn(x.y, y.y));
        }
    }
    if (e.plain_residual) {
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = add2x16<F16>(v[i], k[i]);
    } else if (e.residual || e.value_scale != 1.f) { // contracted as in the reference's finishing pass
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 x = unpack16<F16>(v[i]), s = unpack16<F16>(k[i]);
            v[i] = pack2x16<F16>(__fmaf_rn(e.value_scale, x.x, __fmul_rn(e.residual_scale, s.x)),
                                 __fmaf_rn(e.value_scale, x.y, __fmul_rn(e.residual_scale, s.y)));
        }
    }
    if (e.output_scale != 1.f) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 x = unpack16<F16>(v[i]);
            v[i] = pack2x16<F16>(__fmul_rn(x.x, e.output_scale), __fmul_rn(x.y, e.output_scale));
        }
    }
    if (e.activation == 1) {
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = relu2x16<F16>(v[i]);
    }
    return make_uint4(v[0], v[1], v[2], v[3]);
}
// The gate of row `m`, from channel `n` on (n a multiple of 8).
__device__ __forceinline__ const uint4 *gate_at(const FusedEpilogue &e, int m, int n) {
    return reinterpret_cast<const uint4 *>(static_cast<const uint16_t *>(e.gate) + size_t(m / e.rows_per_sequence) * e.gate_ld + n);
}
// n / d for d between 1 and 2^120: an approximate reciprocal and one correction by the exact remainder of the quotient
// (P. Markstein, IBM J. Res. Dev. 34, 1990). It has no branch, unlike __fdiv_rn, whose guard keeps one quotient of a thread from
// overlapping the next.
__device__ __forceinline__ float quotient(float n, float d) {
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(d));
    const float q = __fmul_rn(n, r);
    return __fmaf_rn(__fmaf_rn(-d, q, n), r, q);
}
// SiLU and sigmoid of eight packed values, none of them beyond +-80 (e^80 is far from overflow); over all 65536 values of both
// storage types the results are the finishing pass's. Up projection of a 750 x 1024 block with SiLU: 27.6 -> 13 us.
template <bool F16, bool Sigmoid, int Words> __device__ __forceinline__ void logistic(uint32_t (&v)[Words]) {
    const auto one = [](float x) { return quotient(Sigmoid ? 1.f : x, __fadd_rn(1.f, expf(-x))); };
#pragma unroll
    for (int i = 0; i < Words; ++i) {
        const float2 x = unpack16<F16>(v[i]);
        v[i] = pack2x16<F16>(one(x.x), one(x.y));
    }
}
template <bool F16, int Words> __device__ __forceinline__ bool within80(const uint32_t (&v)[Words]) {
    bool all = true;
#pragma unroll
    for (int i = 0; i < Words; ++i) {
        const float2 x = unpack16<F16>(v[i]);
        all = all && fabsf(x.x) < 80.f && fabsf(x.y) < 80.f; // false for a NaN
    }
    return all;
}
// The finishing pass's other activations (its own instruction sequences) on packed values, all of a call's evaluations
// independent of one another.
template <bool F16, int Words> __device__ __forceinline__ void activate(uint32_t (&v)[Words], int kind, float alpha) {
    if ((kind == 3 || kind == 8) && within80<F16>(v)) {
        if (kind == 3) logistic<F16, false>(v);
        else logistic<F16, true>(v);
        return;
    }
    switch (kind) {
#define B200Q_ACTIVATION(K)                                                                                          \
    case K:                                                                                                          \
        _Pragma("unroll") for (int i = 0; i < Words; ++i) {                                                          \
            const float2 x = unpack16<F16>(v[i]);                                                                    \
            v[i] = pack2x16<F16>(finish_activation(x.x, K, alpha), finish_activation(x.y, K, alpha));                \
        }                                                                                                            \
        break;
        B200Q_ACTIVATION(2)
        B200Q_ACTIVATION(3)
        B200Q_ACTIVATION(4)
        B200Q_ACTIVATION(5)
        B200Q_ACTIVATION(7)
        B200Q_ACTIVATION(8)
#undef B200Q_ACTIVATION
    default: break;
    }
}
// Out of line because it is large and called from several places: one copy per kernel, arguments and result in registers.
template <bool F16> __device__ __noinline__ uint4 activate8(uint4 row, int kind, float alpha) {
    uint32_t v[4] = {row.x, row.y, row.z, row.w};
    activate<F16>(v, kind, alpha);
    return make_uint4(v[0], v[1], v[2], v[3]);
}
// A thread's finished chunks of eight values in a slab. In line, eight values at a time: four chunks at a time keep more in flight
// (GEMM 3000 x 2048 -> 8192 with SiLU / tanh GELU: a call per chunk 69 / 53 us, this 66 / 50, four chunks 63 / 45), but their code
// is met cold when a block has only a few tiles per pair (block of 750 x 1024 with GELU: 32.6, 32.2 and 33.2 us).
template <bool F16, int Chunks, class At> __device__ __forceinline__ void activate_chunks(At at, int kind, float alpha) {
#pragma unroll 1
    for (int q = 0; q < Chunks; ++q) {
        const uint4 row = *at(q);
        uint32_t v[4] = {row.x, row.y, row.z, row.w};
        activate<F16>(v, kind, alpha);
        *at(q) = make_uint4(v[0], v[1], v[2], v[3]);
    }
}
template <bool F16> __device__ __forceinline__ uint4 pack8x16(const float (&v)[8]) {
    return make_uint4(pack2x16<F16>(v[0], v[1]), pack2x16<F16>(v[2], v[3]), pack2x16<F16>(v[4], v[5]), pack2x16<F16>(v[6], v[7]));
}
// The MMA issuer never tests an mbarrier for a refilled stage: the test waits behind the MMAs in flight (200 to 300 cycles per
// K block). A waiter tests for it and hands the verdict over at a named hardware barrier. K-group mode has a warp of its own
// for that, because its epilogue warps are busy; per-row mode uses the last epilogue warp, which is idle until the end.
template <bool Grouped> constexpr int kStreamThreads = kGemmThreads + (Grouped ? 32 : 0);

// `Plain` instances serve what a decoder chain asks for: aligned 16-bit rows, nothing behind the product but an fp32 residual,
// K groups of 128 or none. They carry no other code: in a chain every launch finds the instruction caches cold, and the
// general kernel's extra paths cost time although they are not taken.
// `Split` says the same about split K. K-group tiles below 64 tokens keep one instance for both: their chain alternates split
// and unsplit launches, and one resident copy of that larger kernel beats two (28 layers, 3 / 16 / 32 rows: 729 / 796 / 830
// against 756 / 833 / 855 us; at 57 rows, in the 64-token tile, two are better, 1024 against 1040).
template <bool Grouped, int BN> constexpr bool kOneInstance = Grouped && BN < 64;
constexpr int kDenseLoads = 8; // 16-byte pieces of a row that a thread holds: 16384 values per CTA
// `X`, when not void, is the type of 16-bit activations that this launch quantizes itself (GemmArgs::x): the epilogue warps, idle until
// the accumulators are full, encode the CTA's K range into resident token tiles while the weights arrive. A few rows only: every
// CTA of a channel slab encodes the same rows again, and with one scale per row reads them whole.
template <Type F, bool Grouped, int BN, bool Plain, bool Split, class X = void>
__global__ void __launch_bounds__(kStreamThreads<Grouped>, (!Grouped && BN <= 64 && std::is_void_v<X>) ? 2 : 1)
w8a8_tcgen05_gemm(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                  const __grid_constant__ std::conditional_t<std::is_void_v<X>, GemmArgs, DenseArgs> a) {
    constexpr bool kInt = F == Type::I8;
    constexpr bool kIntAcc = kInt && !Grouped; // partial tiles / raw outputs carry int32 bit patterns
    constexpr int kWeightBytes = kBlockChannels * kBlockK, kTokenBytes = BN * kBlockK;
    constexpr bool kDense = !std::is_void_v<X>, kOne = kOneInstance<Grouped, BN> || kDense;
    constexpr int kStageBytes = kWeightBytes + (kDense ? 0 : kTokenBytes);
    // K-group mode gives every K block its own accumulator for as long as tensor memory lasts (512
    // columns: 32 buffers at BN=16 ... 4 at BN=128) and reuses them round-robin after that.
    constexpr int kAccBuffers = Grouped ? (512 / BN > 32 ? 32 : 512 / BN) : 1;
    constexpr int kAccColumns = Grouped ? kAccBuffers * BN : BN;
    constexpr uint32_t kTmemColumns = kAccColumns <= 32 ? 32 : kAccColumns <= 64 ? 64 : kAccColumns <= 128 ? 128
                                      : kAccColumns <= 256 ? 256 : 512;
    constexpr uint32_t kIdesc = kInt ? ptx::idesc_i8(kBlockChannels, BN) : ptx::idesc_e4m3(kBlockChannels, BN);
    constexpr int kChunks = BN / 16;               // 16-token column chunks of the accumulator
    constexpr uint32_t kPassBytes = kRowsPerPass * kBlockChannels * 4;

    extern __shared__ uint8_t dynamic_smem[];
    __shared__ alignas(8) uint64_t full_bar[kMaxStages], empty_bar[kMaxStages], acc_full[kAccBuffers], acc_empty[kAccBuffers];
    __shared__ alignas(8) uint64_t w_full, x_full; // the first fill of all stages: weights, activations
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    __shared__ float sx_tile[BN]; // per-row activation scales of this token tile

    // Dynamic shared memory, 1024-byte aligned for the swizzled TMA boxes:
    //   [pipeline stages | dense: token tiles | split-K slots pushed by the cluster peers | K-group scales]
    // Unsplit launches reuse the stage memory for the transposed tile once the last MMA retired;
    // split launches must not, because peers push while this CTA may still be in its main loop.
    const uint32_t raw_base = ptx::smem_u32(dynamic_smem);
    const uint32_t tiles_base = (raw_base + 1023u) & ~1023u;
    uint8_t *tiles_ptr = dynamic_smem + (tiles_base - raw_base);
    const int splits = Split ? a.splits : 1;
    const bool split_k = Split && (!kOne || splits > 1);
    const uint32_t reduce_bytes = split_k ? uint32_t(splits * a.owned_passes) * kPassBytes : 0u;
    const uint32_t reduce_base = tiles_base + uint32_t(a.tile_region);
    uint8_t *reduce_ptr = tiles_ptr + a.tile_region;
    float *scale_smem = reinterpret_cast<float *>(reduce_ptr + reduce_bytes);

    const int warp = ptx::warp_index(), lane = threadIdx.x & 31;
    const int split = split_k ? int(ptx::cluster_ctarank()) : 0; // cluster = (1,1,splits): rank == blockIdx.z
    const int n0 = blockIdx.x * kBlockChannels, m0 = blockIdx.y * BN;
    const int kb_total = (a.k + kBlockK - 1) / kBlockK;
    const int kb_begin = int(int64_t(kb_total) * split / splits);
    const int kb_end = int(int64_t(kb_total) * (split + 1) / splits);
    const int kb_count = kb_end - kb_begin;
    // K-group mode: accumulation units per 128-byte K block (1, 2 or 4) and MMAs per unit.
    const int unit_k = Grouped && !Plain && !kDense ? min(a.input_group ? a.input_group : kBlockK, a.weight_group ? a.weight_group : kBlockK) : kBlockK;
    const int units = kBlockK / unit_k, unit_mmas = 4 / units;
    const int tile_linear = blockIdx.y * gridDim.x + blockIdx.x;
    const int valid_tokens = min(BN, a.m - m0);

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            ptx::mbar_init(ptx::smem_u32(&full_bar[s]), 1);
            ptx::mbar_init(ptx::smem_u32(&empty_bar[s]), 1);
        }

        for (int b = 0; b < kAccBuffers; ++b) {
            ptx::mbar_init(ptx::smem_u32(&acc_full[b]), 1);
            ptx::mbar_init(ptx::smem_u32(&acc_empty[b]), kEpilogueThreads / 32);
        }
        ptx::mbar_init(ptx::smem_u32(&w_full), 1);
        ptx::mbar_init(ptx::smem_u32(&x_full), kDense ? kEpilogueThreads / 32 : 1);
        abort_flag = 0;
        ptx::fence_barrier_init();
        ptx::fence_proxy_async_smem();
    }
    // Per-row dense instances: the rows' largest magnitudes as bits, without NaN from BN on.
    [[maybe_unused]] uint32_t *row_largest = nullptr;
    if constexpr (kDense && !Grouped) {
        row_largest = reinterpret_cast<uint32_t *>(tiles_ptr + a.largest_offset);
        if (threadIdx.x >= 64 && threadIdx.x < 64 + 2 * BN) row_largest[threadIdx.x - 64] = 0u;
    }
    if (warp == 1) ptx::tmem_alloc(ptx::smem_u32(&tmem_slot), kTmemColumns);
    ptx::tcgen05_fence_before();
    __syncthreads();
    ptx::tcgen05_fence_after();
    const uint32_t tmem_base = ptx::warp_uniform(tmem_slot);
    [[maybe_unused]] uint32_t token_base = 0; // dense: the token tiles, one per K block
    if constexpr (kDense) token_base = tiles_base + uint32_t(a.token_offset);
    volatile int *abort_ptr = &abort_flag;
    // K blocks whose MMAs go out in one burst: prefetched, and with an accumulator nobody used before. The others are waited for.
    const int refill_from = Grouped ? min(min(a.stages, kb_count), kAccBuffers / units) : min(a.stages, kb_count);
    const auto wait_for_refills = [&](bool ok, long long limit) {
        int stage = refill_from == a.stages ? 0 : refill_from;
        uint32_t phase = refill_from == a.stages ? 0u : 1u;
        const int ahead = min(a.stages, kb_count);
        // A parity test cannot tell a phase from the second one after it, so this warp, however late it comes, must find no barrier
        // two phases on. It does not: full_bar counts refills only (the first fill has barriers of its own), and the next refill of
        // a stage needs MMAs that wait for the verdict on this one; likewise the accumulators.
        if (a.refill_delay_ns) __nanosleep(a.refill_delay_ns);
        for (int it = refill_from; it < kb_count; ++it) {
            if (Grouped && it * units >= kAccBuffers) // the epilogue drained these accumulators' previous groups
                for (int u = 0; u < units && ok; ++u)
                    ok = ptx::mbar_wait(ptx::smem_u32(&acc_empty[(it * units + u) % kAccBuffers]),
                                        (uint32_t((it * units + u) / kAccBuffers) & 1u) ^ 1u, abort_ptr, limit);
            if (it >= ahead) ok = ok && ptx::mbar_wait(ptx::smem_u32(&full_bar[stage]), phase, abort_ptr, limit);
            ok = ptx::pair_barrier_and(__all_sync(0xffffffffu, ok)); // the vote brings the lanes together for the aligned barrier
            if (++stage == a.stages) { stage = 0; phase ^= 1u; }
        }
    };
    const long long wait_limit = a.wait_limit_cycles > 0 ? a.wait_limit_cycles : ptx::kWaitLimitCycles;
    // The next kernel in the stream may begin its own prologue; peers learn that this CTA is running.
    ptx::launch_dependents();
    if (split_k) ptx::cluster_arrive();
    if (!a.early) ptx::wait_for_upstream();

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        // The whole warp runs the loops so that addresses and coordinates stay warp-uniform (a copy takes them from
        // uniform registers; issued from a single-lane branch it took about 190 cycles, most of it moving operands
        // there); one elected lane issues.
        if (ptx::elect_one()) {
            ptx::prefetch_tensormap(&map_w);
            if (!kDense) ptx::prefetch_tensormap(&map_x);
        }
        // Weights do not depend on the upstream kernel: fill the ring with weight tiles first, then wait for upstream
        // and add the activation tiles of all those stages, each under ONE barrier. A barrier test between MMA issues
        // costs the issuing thread about 200 cycles, so the burst over the prefetched stages must not need any.
        // Weights are streamed once: they are marked first-to-evict so that the few megabytes of
        // activations the chain keeps passing from kernel to kernel stay in L2.
        const uint64_t stream_once = ptx::policy_evict_first();
        const int ahead = min(a.stages, kb_count);
        if (ptx::elect_one()) { // one election around a burst: per copy or per MMA it costs some 20 cycles
            const uint32_t bar = ptx::smem_u32(&w_full);
            ptx::mbar_arrive_expect_tx(bar, uint32_t(ahead) * kWeightBytes + uint32_t(a.expiry_extra_bytes));
            for (int i = 0; i < ahead; ++i)
                ptx::tma_load_2d_hint(tiles_base + uint32_t(i) * kStageBytes, &map_w, bar, (kb_begin + i) * kBlockK, n0, stream_once);
        }
        __syncwarp();
        if constexpr (!kDense) {
            ptx::wait_for_upstream();
            if (ptx::elect_one()) {
                ptx::mbar_arrive_expect_tx(ptx::smem_u32(&x_full), uint32_t(ahead) * kTokenBytes);
                for (int i = 0; i < ahead; ++i)
                    ptx::tma_load_2d(tiles_base + uint32_t(i) * kStageBytes + kWeightBytes, &map_x,
                                     ptx::smem_u32(&x_full), (kb_begin + i) * kBlockK, m0);
            }
            __syncwarp();
        }
        int stage = ahead == a.stages ? 0 : ahead;
        uint32_t phase = ahead == a.stages ? 1u : 0u;
        for (int kb = kb_begin + ahead; kb < kb_end; ++kb) {
            if (!__all_sync(0xffffffffu, ptx::mbar_wait(ptx::smem_u32(&empty_bar[stage]), phase ^ 1u, abort_ptr, wait_limit))) break;
            const uint32_t bar = ptx::smem_u32(&full_bar[stage]);
            const uint32_t dst = tiles_base + uint32_t(stage) * kStageBytes;
            if (ptx::elect_one()) {
                ptx::mbar_arrive_expect_tx(bar, kStageBytes);
                ptx::tma_load_2d_hint(dst, &map_w, bar, kb * kBlockK, n0, stream_once);
                if (!kDense) ptx::tma_load_2d(dst + kWeightBytes, &map_x, bar, kb * kBlockK, m0);
            }
            __syncwarp();
            if (++stage == a.stages) { stage = 0; phase ^= 1u; }
        }
        if (split_k) ptx::cluster_wait();
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        // The whole warp runs the loop so that stage indices and descriptors stay warp-uniform (the
        // tensor-core instructions take them from uniform registers); one elected lane issues.
        {
            // The weight tiles of the prefetched stages land while the upstream kernel still runs: they are waited
            // for first, off the critical path, then the activations.
            bool ok = ptx::mbar_wait(ptx::smem_u32(&w_full), 0u, abort_ptr, wait_limit);
            ok = ok && ptx::mbar_wait(ptx::smem_u32(&x_full), 0u, abort_ptr, wait_limit);
            ok = __all_sync(0xffffffffu, ok);
            // The prefetched stages need no barrier at all any more, so their MMAs go out back to back
            // (any shared-memory access between MMA issues stalls the issuing warp for a couple of
            // hundred cycles). Stage i holds K block i here; in K-group mode K block i also has
            // accumulator i to itself while fresh accumulators last.
            const int burst = refill_from; // min(ahead, K blocks with a fresh accumulator)
            int stage = burst == a.stages ? 0 : burst;
            if (!Grouped || Plain || kDense || units == 1) {
                // One K block: four MMAs into its accumulator and its reports. A loop of its own: one that also served the
                // narrow groups issued K-group blocks at half the rate.
                const auto issue = [&](int it, int at, uint32_t buffer) {
                    const uint32_t tile = tiles_base + uint32_t(at) * kStageBytes;
                    const uint32_t lo_w = ptx::smem_desc_lo_k128(tile), lo_x = ptx::smem_desc_lo_k128(kDense ? token_base + uint32_t(it) * kTokenBytes : tile + kWeightBytes);
                    const uint32_t d = tmem_base + buffer * uint32_t(BN), accumulate = Grouped ? 0u : uint32_t(it > 0);
                    if (kInt) ptx::mma_i8_k128(d, lo_w, lo_x, kIdesc, accumulate);
                    else ptx::mma_f8_k128(d, lo_w, lo_x, kIdesc, accumulate);
                    // Only a stage that will be refilled needs to report that its MMAs retired.
                    if (it + a.stages < kb_count) ptx::tcgen05_commit(ptx::smem_u32(&empty_bar[at]));
                    if (Grouped) ptx::tcgen05_commit(ptx::smem_u32(&acc_full[buffer]));
                };
                ptx::tcgen05_fence_after();
                if (ok && ptx::elect_one())
                    for (int it = 0; it < burst; ++it) issue(it, it, Grouped ? uint32_t(it) : 0u);
                __syncwarp();
                // Refilled stages arrive at the rate memory delivers them.
                for (int it = burst; it < kb_count; ++it) {
                    ok = ptx::pair_barrier_and(ok);
                    ptx::tcgen05_fence_after();
                    if (ok && ptx::elect_one()) issue(it, stage, Grouped ? uint32_t(it) % kAccBuffers : 0u);
                    __syncwarp();
                    if (++stage == a.stages) stage = 0;
                }
            } else {
                // Narrow K groups: the MMAs of one 128-byte K block go to `units` accumulators, `unit_mmas`
                // each; every accumulator reports on its own barrier.
                for (int it = 0; it < kb_count; ++it) {
                    const int at = it < burst ? it : stage, buffer = (it * units) % kAccBuffers;
                    if (it >= burst) ok = ptx::pair_barrier_and(ok);
                    ptx::tcgen05_fence_after();
                    const uint32_t tile = tiles_base + uint32_t(at) * kStageBytes;
                    const uint32_t lo_w = ptx::smem_desc_lo_k128(tile), lo_x = ptx::smem_desc_lo_k128(tile + kWeightBytes);
                    if (ok && ptx::elect_one()) {
                        for (int u = 0; u < units; ++u) {
                            const uint32_t d = tmem_base + uint32_t((buffer + u) * BN);
                            for (int m = 0; m < unit_mmas; ++m) {
                                const uint32_t step = uint32_t(2 * (u * unit_mmas + m)); // 32 bytes of K = 2 descriptor units
                                if (kInt) ptx::mma_i8_lo(d, lo_w + step, lo_x + step, kIdesc, uint32_t(m > 0));
                                else ptx::mma_f8_lo(d, lo_w + step, lo_x + step, kIdesc, uint32_t(m > 0));
                            }
                            ptx::tcgen05_commit(ptx::smem_u32(&acc_full[buffer + u]));
                        }
                        if (it + a.stages < kb_count) ptx::tcgen05_commit(ptx::smem_u32(&empty_bar[at]));
                    }
                    __syncwarp();
                    if (it >= burst && ++stage == a.stages) stage = 0;
                }
            }
            if (ptx::elect_one()) {
                if (!Grouped) ptx::tcgen05_commit(ptx::smem_u32(&acc_full[0]));
            }
            __syncwarp();
        }
        if (split_k) ptx::cluster_wait();
    } else if (Grouped && warp == kGemmThreads / 32) {
        // ------------------------------------------------------------ waiter (K-group mode)
        wait_for_refills(true, wait_limit);
        if (split_k) ptx::cluster_wait();
    } else {
        // ------------------------------------------------------------ epilogue warps (8 warps)
        const int e_thread = threadIdx.x - 64;
        const int quadrant = warp & 3;      // tensor-memory lanes this warp may read
        const int half = (warp - 2) >> 2;   // the two warps of a quadrant take alternate 16-token chunks
        const int channel_in_tile = quadrant * 32 + lane;
        const uint32_t lane_base = tmem_base + (uint32_t(quadrant * 32) << 16);
        uint32_t *tile_words = reinterpret_cast<uint32_t *>(tiles_ptr);
        bool ok = true;

        // Phase-2 ownership of this thread: 8 consecutive channels of one token row per pass.
        const int j = e_thread & 15, row_in_pass = e_thread >> 4;
        const int n = n0 + 8 * j;
        const bool columns_ok = n < a.n;
        const FusedEpilogue &e = a.ep;
        const int type = a.out_type;
        const int passes = (valid_tokens + kRowsPerPass - 1) / kRowsPerPass;
        // Weights' scales are fetched before anything else so their latency hides behind the main loop.
        float sw8[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) sw8[i] = (!Grouped && columns_ok) ? a.sw[n + i] : 1.f;
        // K-group mode: the weights' group scales of this CTA's K range are static too, one entry per
        // accumulation unit (zero for a unit past the end of K, whose accumulator holds zeros). They come by asynchronous
        // copies, so that nothing waits for them until the activations' have been asked for too.
        const int unit_count = kb_count * units;
        float *sx_smem = scale_smem, *sw_smem = scale_smem + size_t(unit_count) * BN;
        if constexpr (Grouped) {
            const int shift = __ffs(a.weight_group) - 1; // group widths are powers of two
            const uint32_t dst = ptx::smem_u32(sw_smem);
            for (int i = e_thread; i < unit_count * kBlockChannels; i += kEpilogueThreads) {
                const int unit = i / kBlockChannels, channel = n0 + i % kBlockChannels, k0 = kb_begin * kBlockK + unit * unit_k;
                const bool inside = channel < a.n && k0 < a.k;
                if (a.weight_group) ptx::copy_async4(dst + 4u * i, inside ? a.sw + size_t(k0 >> shift) * a.n + channel : a.sw, inside ? 4u : 0u);
                else sw_smem[i] = 1.f;
            }
        }
        ptx::wait_for_upstream(); // activation scales, residuals, bias and the output buffer belong to upstream
        uint4 bias8 = make_uint4(0, 0, 0, 0);
        float first_residual[8];
        uint4 first_skip = make_uint4(0, 0, 0, 0); // 16-bit residual of that pass
        uint4 first_gate = make_uint4(0, 0, 0, 0);
        {
            const int c = split * kRowsPerPass + row_in_pass; // first pass this CTA owns
#pragma unroll
            for (int i = 0; i < 8; ++i) first_residual[i] = 0.f;
            if (!Plain && e.residual && e.residual_vector && columns_ok && c < valid_tokens)
                first_skip = *reinterpret_cast<const uint4 *>(static_cast<const uint16_t *>(e.residual) +
                                                              size_t(m0 + c) * e.residual_ld + n);
            if (!Plain && e.gate && columns_ok && c < valid_tokens) first_gate = *gate_at(e, m0 + c, n);
            if (!Plain && e.bias && columns_ok) {
                const uint16_t *bias16 = static_cast<const uint16_t *>(e.bias) + n;
                uint32_t w[4]; // packed pairs
#pragma unroll
                for (int i = 0; i < 4; ++i) w[i] = uint32_t(bias16[2 * i]) | (uint32_t(bias16[2 * i + 1]) << 16);
                bias8 = make_uint4(w[0], w[1], w[2], w[3]);
            }
            if (e.residual_f32 && columns_ok && c < valid_tokens) {
                const float *src = e.residual_f32 + size_t(m0 + c) * a.n + n;
                if (a.vector_io) {
                    const float4 lo = *reinterpret_cast<const float4 *>(src), hi = *reinterpret_cast<const float4 *>(src + 4);
                    first_residual[0] = lo.x; first_residual[1] = lo.y; first_residual[2] = lo.z; first_residual[3] = lo.w;
                    first_residual[4] = hi.x; first_residual[5] = hi.y; first_residual[6] = hi.z; first_residual[7] = hi.w;
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) first_residual[i] = src[i];
                }
            }
        }

        // ---- dense activations: this CTA's K range of the rows into the token tiles, bytes and scales as the row quantizers write them.
        if constexpr (kDense) {
            const X *x = static_cast<const X *>(a.x) + size_t(m0) * a.x_ld;
            const auto chunk_at = [&](int kb, int row, int chunk) { // 16 columns of a 128-byte swizzled row
                return token_base + uint32_t(kb) * kTokenBytes + uint32_t(row) * 128u + uint32_t((chunk ^ (row & 7)) * 16);
            };
            if constexpr (Grouped) {
                float *scales = scale_smem; // [K block][token]
                const int blocks = kb_count * valid_tokens;
#pragma unroll 1
                for (int first = (warp - 2) * 8; first < blocks; first += kEpilogueThreads / 4) { // four lanes per block of 128
                    const int block = first + (lane >> 2), part = lane & 3;
                    const bool active = block < blocks;
                    const int kb = active ? block / valid_tokens : 0, row = active ? block - kb * valid_tokens : 0;
                    const int column = (kb_begin + kb) * kBlockK + part * 32;
                    uint32_t mask[16], raw[16];
                    load_masks(column, mask);
                    load_row32(x + size_t(row) * a.x_ld + column, raw);
#pragma unroll
                    for (int i = 0; i < 16; ++i) raw[i] ^= mask[i];
                    rotate_quantize32<F, X>(raw, [&](const Words8 &bytes, float step) {
                        if (!active) return;
                        ptx::st_shared_2x64(chunk_at(kb, row, 2 * part), bytes.w[0], bytes.w[1]);
                        ptx::st_shared_2x64(chunk_at(kb, row, 2 * part + 1), bytes.w[2], bytes.w[3]);
                        if (!part) scales[kb * BN + row] = step;
                    });
                }
            } else {
                // A row per warp, or up to eight warps: each thread keeps its columns in registers between the maximum and the bytes.
                const int log = valid_tokens > 4 ? 5 : valid_tokens > 2 ? 6 : valid_tokens > 1 ? 7 : 8; // threads per row
                const int row = e_thread >> log, mine = (e_thread & ((1 << log) - 1)) * 8;
                const X *source = x + size_t(row) * a.x_ld;
                uint4 v[kDenseLoads];
                uint32_t largest = 0u;
#pragma unroll
                for (int j = 0; j < kDenseLoads; ++j) {
                    const int column = (j << (log + 3)) + mine;
                    v[j] = row < valid_tokens && column < a.k ? *reinterpret_cast<const uint4 *>(source + column) : make_uint4(0, 0, 0, 0);
                }
#pragma unroll
                for (int j = 0; j < kDenseLoads; ++j)
                    largest = max_magnitude16x2(max_magnitude16x2(max_magnitude16x2(max_magnitude16x2(largest, v[j].x), v[j].y), v[j].z), v[j].w);
                uint32_t bits = __reduce_max_sync(0xffffffffu, fold_magnitude(largest));
                if (!lane) atomicMax(&row_largest[row], bits);
                const bool finite = ptx::barrier_and(1, kEpilogueThreads, magnitude_finite<X>(bits));
                bits = row_largest[row];
                float amax = magnitude_value<X>(bits);
                if (!finite) { // infinities or NaN somewhere: also the maximum that skips NaN
                    float known = 0.f;
#pragma unroll
                    for (int j = 0; j < kDenseLoads; ++j)
                        for (uint32_t word : {v[j].x, v[j].y, v[j].z, v[j].w}) known = max_skipping_nan<X>(known, word);
                    const uint32_t known_bits = __reduce_max_sync(0xffffffffu, __float_as_uint(known)); // non-negative floats order like their bits
                    if (!lane) atomicMax(&row_largest[BN + row], known_bits);
                    asm volatile("bar.sync 1, 256;" ::: "memory");
                    if (!magnitude_finite<X>(bits)) amax = __uint_as_float(row_largest[BN + row]);
                }
                const float step = quant_scale<F>(amax), inverse = __fdiv_rn(1.f, step);
                const uint64_t inverse2 = f32x2(inverse, inverse);
                if (!mine && row < valid_tokens) sx_tile[row] = step;
#pragma unroll
                for (int j = 0; j < kDenseLoads; ++j) {
                    const int column = (j << (log + 3)) + mine - kb_begin * kBlockK, chunk = column >> 4;
                    if (row < valid_tokens && column >= 0 && column < kb_count * kBlockK)
                        ptx::st_shared_64(chunk_at(chunk >> 3, row, chunk & 7) + uint32_t(column & 8), encode_words<F, X>(v[j], inverse2, magnitude_finite<X>(bits)));
                }
            }
            ptx::fence_proxy_async_smem(); // the tiles are about to be read by the tensor cores
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&x_full));
        }

        // ---- phase 1: accumulators (one lane = one channel) -> [token][channel] rows, either in this
        // CTA's shared memory (unsplit) or pushed into the owning peer's slot for this split.
        auto emit_chunk = [&](int chunk, const uint32_t (&words)[16]) {
            if (!split_k) {
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    if (chunk * 16 + i < valid_tokens) tile_words[(chunk * 16 + i) * kBlockChannels + channel_in_tile] = words[i];
            } else {
                const int owner = chunk % splits, local_pass = chunk / splits;
                const uint32_t slot = reduce_base + uint32_t(split * a.owned_passes + local_pass) * kPassBytes +
                                      uint32_t(channel_in_tile) * 4u;
                const uint32_t remote = ptx::map_to_rank(slot, uint32_t(owner));
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    if (chunk * 16 + i < valid_tokens) ptx::st_cluster_u32(remote + uint32_t(i) * (kBlockChannels * 4u), words[i]);
            }
        };

        if constexpr (!Grouped) {
            if constexpr (!kDense)
                for (int c = e_thread; c < BN; c += kEpilogueThreads) sx_tile[c] = c < valid_tokens ? a.sx[m0 + c] : 0.f;
            if (warp == kGemmThreads / 32 - 1) wait_for_refills(true, wait_limit);
            ok = ptx::mbar_wait(ptx::smem_u32(&acc_full[0]), 0, abort_ptr, wait_limit);
            ptx::tcgen05_fence_after();
            if (split_k) ptx::cluster_wait(); // every peer is running: its shared memory may be written
            if (ok) {
                // Two chunks per round: both loads are in flight before the single wait.
#pragma unroll 1
                for (int chunk = half; chunk < kChunks; chunk += 4) {
                    if (chunk * 16 >= valid_tokens) break;
                    const bool second = chunk + 2 < kChunks && (chunk + 2) * 16 < valid_tokens;
                    uint32_t r0[16], r1[16];
                    ptx::tmem_load16(lane_base + uint32_t(chunk * 16), r0);
                    if (second) ptx::tmem_load16(lane_base + uint32_t((chunk + 2) * 16), r1);
                    ptx::tmem_load_wait();
                    emit_chunk(chunk, r0);
                    if (second) emit_chunk(chunk + 2, r1);
                }
            }
        } else {
            // Stage the activations' group scales of this split (the weights' were staged before the wait):
            // sx_g[unit][token], each operand indexed by its own group width.
            const int shift = __ffs(a.input_group) - 1;
            const uint32_t dst = ptx::smem_u32(sx_smem);
            for (int i = e_thread; !kDense && i < unit_count * BN; i += kEpilogueThreads) {
                const int unit = i / BN, token = i % BN, k0 = kb_begin * kBlockK + unit * unit_k;
                const bool inside = token < valid_tokens && k0 < a.k;
                if (a.input_group) ptx::copy_async4(dst + 4u * i, inside ? a.sx + size_t(k0 >> shift) * a.m + m0 + token : a.sx, inside ? 4u : 0u);
                else sx_smem[i] = 1.f;
            }
            ptx::copy_async_wait_all();
            asm volatile("bar.sync 1, 256;" ::: "memory");
            // The two warps of a lane quadrant take half of the tokens each. A round drains kRound units with one wait: a
            // commit completes after all earlier MMAs, so the last unit's barrier stands for the round. The arithmetic is
            // packed two-wide.
            constexpr int kHalf = BN / 2, kRound = BN == 16 ? 4 : BN == 32 ? 2 : 1;
            uint64_t result[kHalf / 2];
#pragma unroll
            for (int c = 0; c < kHalf / 2; ++c) result[c] = 0ull;
#pragma unroll 1
            for (int first = 0; first < unit_count && ok; first += kRound) {
                const int last = min(first + kRound, unit_count) - 1;
                ok = ptx::mbar_wait(ptx::smem_u32(&acc_full[last % kAccBuffers]), uint32_t(last / kAccBuffers) & 1u, abort_ptr, wait_limit);
                if (!ok) break;
                ptx::tcgen05_fence_after();
                uint32_t r[kRound][kHalf];
#pragma unroll
                for (int u = 0; u < kRound; ++u)
                    if (first + u <= last) ptx::tmem_load<kHalf>(lane_base + uint32_t(((first + u) % kAccBuffers) * BN + half * kHalf), r[u]);
                ptx::tmem_load_wait();
                // Everything this warp needs is in registers: hand the buffers that are used again back before the arithmetic.
                if (first + kAccBuffers < unit_count) {
                    ptx::tcgen05_fence_before();
                    __syncwarp();
                    if (lane == 0)
                        for (int u = first; u <= last; ++u) ptx::mbar_arrive(ptx::smem_u32(&acc_empty[u % kAccBuffers]));
                }
#pragma unroll
                for (int u = 0; u < kRound; ++u) {
                    if (first + u <= last) {
                        const int it = first + u;
                        const float scale_w = sw_smem[it * kBlockChannels + channel_in_tile];
                        const uint64_t scale_w2 = ptx::pack2(scale_w, scale_w);
                        const uint32_t scale_x = ptx::pinned(ptx::smem_u32(sx_smem + it * BN + half * kHalf));
#pragma unroll
                        for (int q = 0; q < kHalf / 4; ++q) {
                            const ulonglong2 sx4 = ptx::ld_shared_2x64(scale_x + 16u * q); // a broadcast
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                const int i = 4 * q + 2 * h;
                                const uint64_t p = kInt ? ptx::int_to_float2(r[u][i], r[u][i + 1])
                                                        : ptx::pack2(__uint_as_float(r[u][i]), __uint_as_float(r[u][i + 1]));
                                result[i / 2] = ptx::fma2(p, ptx::mul2(h ? sx4.y : sx4.x, scale_w2), result[i / 2]);
                            }
                        }
                    }
                }
            }
            if (split_k) ptx::cluster_wait();
            if (ok) {
                // Outer scales exist only when just one operand carries K-group scales.
                const int channel = n0 + channel_in_tile;
                const float outer_w = (!a.weight_group && channel < a.n) ? a.sw[channel] : 1.f;
                constexpr int kRows = kHalf < 16 ? kHalf : 16; // tokens of one 16-row pass this thread holds
#pragma unroll
                for (int k = 0; k < kHalf / kRows; ++k) {
                    const int token0 = half * kHalf + k * kRows, chunk = token0 / 16;
                    if (token0 < valid_tokens) {
                        uint32_t words[kRows];
#pragma unroll
                        for (int i = 0; i < kRows; i += 2) {
                            float v[2];
                            ptx::unpack2(result[(k * kRows + i) / 2], v[0], v[1]);
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                const int c = token0 + i + h;
                                const float outer = (a.input_group || c >= valid_tokens) ? 1.f : a.sx[m0 + c];
                                words[i + h] = __float_as_uint(v[h] * (outer * outer_w));
                            }
                        }
                        if (!split_k) {
#pragma unroll
                            for (int i = 0; i < kRows; ++i)
                                if (token0 + i < valid_tokens) tile_words[(token0 + i) * kBlockChannels + channel_in_tile] = words[i];
                        } else {
                            const uint32_t remote = ptx::map_to_rank(reduce_base + uint32_t(split * a.owned_passes + chunk / splits) * kPassBytes +
                                                                         uint32_t((token0 & 15) * kBlockChannels + channel_in_tile) * 4u,
                                                                     uint32_t(chunk % splits));
#pragma unroll
                            for (int i = 0; i < kRows; ++i)
                                if (token0 + i < valid_tokens) ptx::st_cluster_u32(remote + uint32_t(i) * (kBlockChannels * 4u), words[i]);
                        }
                    }
                }
            }
        }
        ptx::tcgen05_fence_before();

        // ---- phase boundary: rows are where their finisher will read them.
        if (split_k) ptx::cluster_sync();
        else asm volatile("bar.sync 1, 256;" ::: "memory");

        // ---- phase 2: finish token rows; every global access is a 16-byte vector on a 256-byte row.
        // Aligned 16-bit rows take a loop specialised for the output type and for whether the finishing chain
        // follows; raw accumulators and unaligned rows take the general loop below it.
        const bool lean = Plain || (type != int(Type::I32) && a.vector_io && (!e.residual || e.residual_vector));
        const auto finish_rows = [&](auto f16_tag, auto chain_tag) {
            constexpr bool kF16 = decltype(f16_tag)::value, kChain = decltype(chain_tag)::value;
            const float *__restrict__ residual = e.residual_f32; // never aliases the output rows
            uint16_t *out16 = static_cast<uint16_t *>(a.out);
            const size_t slot_stride = size_t(a.owned_passes) * kPassBytes;
#pragma unroll 2
            for (int local_pass = 0;; ++local_pass) {
                const int pass = local_pass * splits + split;
                if (pass >= passes) break;
                const int c = pass * kRowsPerPass + row_in_pass;
                if (c >= valid_tokens) continue;
                const size_t at = size_t(m0 + c) * a.n + n;
                float r8[8];
                if (residual && local_pass > 0) {
                    const float4 lo = *reinterpret_cast<const float4 *>(residual + at), hi = *reinterpret_cast<const float4 *>(residual + at + 4);
                    r8[0] = lo.x; r8[1] = lo.y; r8[2] = lo.z; r8[3] = lo.w; r8[4] = hi.x; r8[5] = hi.y; r8[6] = hi.z; r8[7] = hi.w;
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) r8[i] = first_residual[i];
                }
                uint4 skip16 = first_skip;
                if (kChain && e.residual && local_pass > 0)
                    skip16 = *reinterpret_cast<const uint4 *>(static_cast<const uint16_t *>(e.residual) +
                                                              size_t(m0 + c) * e.residual_ld + n);
                const uint4 gate = kChain && e.gate && local_pass > 0 ? *gate_at(e, m0 + c, n) : first_gate;
                uint32_t raw[8];
                if (!split_k) {
                    const uint8_t *src = tiles_ptr + size_t(c * kBlockChannels + 8 * j) * 4;
                    const uint4 lo = *reinterpret_cast<const uint4 *>(src), hi = *reinterpret_cast<const uint4 *>(src + 16);
                    raw[0] = lo.x; raw[1] = lo.y; raw[2] = lo.z; raw[3] = lo.w; raw[4] = hi.x; raw[5] = hi.y; raw[6] = hi.z; raw[7] = hi.w;
                } else {
                    const uint8_t *src = reduce_ptr + size_t(local_pass) * kPassBytes + size_t(row_in_pass * kBlockChannels + 8 * j) * 4;
#pragma unroll
                    for (int i = 0; i < 8; ++i) raw[i] = 0u;
                    for (int s = 0; s < splits; ++s) {
                        const uint4 lo = *reinterpret_cast<const uint4 *>(src + s * slot_stride);
                        const uint4 hi = *reinterpret_cast<const uint4 *>(src + s * slot_stride + 16);
                        const uint32_t part[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            raw[i] = kIntAcc ? uint32_t(int(raw[i]) + int(part[i]))
                                             : __float_as_uint(__fadd_rn(__uint_as_float(raw[i]), __uint_as_float(part[i])));
                    }
                }
                const float scale_x = sx_tile[Grouped ? 0 : c];
                float value[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float acc = kIntAcc ? float(int(raw[i])) : __uint_as_float(raw[i]);
                    value[i] = Grouped ? acc : __fmul_rn(__fmul_rn(acc, scale_x), sw8[i]);
                    if (residual) value[i] = __fadd_rn(value[i], r8[i]);
                }
                uint4 packed = Plain && type == int(Type::F16) ? pack8x16<true>(value) : pack8x16<kF16>(value);
                if (kChain) {
                    packed = chain8<kF16>(e, packed, bias8, gate, skip16);
                    if (e.activation > 1) packed = activate8<kF16>(packed, e.activation, e.alpha);
                }
                *reinterpret_cast<uint4 *>(out16 + at) = packed;
            }
        };
        if (ok && !*abort_ptr && columns_ok && lean) {
            using std::bool_constant;
            if (Plain) finish_rows(bool_constant<false>{}, bool_constant<false>{});
            else if (type == int(Type::F16)) finish_rows(bool_constant<true>{}, bool_constant<true>{});
            else finish_rows(bool_constant<false>{}, bool_constant<true>{});
        } else if (!Plain && ok && !*abort_ptr && columns_ok) {
            for (int local_pass = 0;; ++local_pass) {
                const int pass = local_pass * splits + split;
                if (pass >= passes) break;
                const int c = pass * kRowsPerPass + row_in_pass;
                if (c >= valid_tokens) continue;
                const int m = m0 + c;
                uint32_t raw[8];
                if (!split_k) {
                    const uint8_t *src = tiles_ptr + size_t(c * kBlockChannels + 8 * j) * 4;
                    const uint4 lo = *reinterpret_cast<const uint4 *>(src), hi = *reinterpret_cast<const uint4 *>(src + 16);
                    raw[0] = lo.x; raw[1] = lo.y; raw[2] = lo.z; raw[3] = lo.w;
                    raw[4] = hi.x; raw[5] = hi.y; raw[6] = hi.z; raw[7] = hi.w;
                } else {
                    // Slots of this pass, one per split, summed in split order (deterministic).
                    const uint8_t *src = reduce_ptr + size_t(local_pass) * kPassBytes + size_t(row_in_pass * kBlockChannels + 8 * j) * 4;
                    const size_t slot_stride = size_t(a.owned_passes) * kPassBytes;
#pragma unroll
                    for (int i = 0; i < 8; ++i) raw[i] = 0u; // int 0 and +0.f share this pattern
                    for (int s = 0; s < splits; ++s) {
                        const uint4 lo = *reinterpret_cast<const uint4 *>(src + s * slot_stride);
                        const uint4 hi = *reinterpret_cast<const uint4 *>(src + s * slot_stride + 16);
                        const uint32_t part[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            raw[i] = kIntAcc ? uint32_t(int(raw[i]) + int(part[i]))
                                             : __float_as_uint(__fadd_rn(__uint_as_float(raw[i]), __uint_as_float(part[i])));
                    }
                }
                const size_t at = size_t(m) * a.n + n;
                if (type == int(Type::I32)) {
                    uint32_t *dst = static_cast<uint32_t *>(a.out) + at;
                    if (a.vector_io) {
                        *reinterpret_cast<uint4 *>(dst) = make_uint4(raw[0], raw[1], raw[2], raw[3]);
                        *reinterpret_cast<uint4 *>(dst + 4) = make_uint4(raw[4], raw[5], raw[6], raw[7]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 8; ++i) dst[i] = raw[i];
                    }
                    continue;
                }
                float value[8];
                const float scale_x = sx_tile[Grouped ? 0 : c];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float acc = kIntAcc ? float(int(raw[i])) : __uint_as_float(raw[i]);
                    value[i] = Grouped ? acc : __fmul_rn(__fmul_rn(acc, scale_x), sw8[i]);
                }
                if (e.residual_f32) {
                    float r8[8];
                    if (local_pass == 0) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) r8[i] = first_residual[i];
                    } else if (a.vector_io) {
                        const float4 lo = *reinterpret_cast<const float4 *>(e.residual_f32 + at);
                        const float4 hi = *reinterpret_cast<const float4 *>(e.residual_f32 + at + 4);
                        r8[0] = lo.x; r8[1] = lo.y; r8[2] = lo.z; r8[3] = lo.w;
                        r8[4] = hi.x; r8[5] = hi.y; r8[6] = hi.z; r8[7] = hi.w;
                    } else {
#pragma unroll
                        for (int i = 0; i < 8; ++i) r8[i] = e.residual_f32[at + i];
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i) value[i] = __fadd_rn(value[i], r8[i]);
                }
                const auto finish = [&](auto f16_tag) {
                    constexpr bool kF16 = decltype(f16_tag)::value;
                    uint4 row = pack8x16<kF16>(value);
                    if (e.chain) {
                        uint32_t skip[4] = {0u, 0u, 0u, 0u};
                        if (e.residual) {
                            const uint16_t *src = static_cast<const uint16_t *>(e.residual) + size_t(m) * e.residual_ld + n;
#pragma unroll
                            for (int i = 0; i < 4; ++i) skip[i] = uint32_t(src[2 * i]) | (uint32_t(src[2 * i + 1]) << 16);
                        }
                        const uint4 gate = e.gate ? *gate_at(e, m, n) : make_uint4(0, 0, 0, 0);
                        row = chain8<kF16>(e, row, bias8, gate, make_uint4(skip[0], skip[1], skip[2], skip[3]));
                        if (e.activation > 1) row = activate8<kF16>(row, e.activation, e.alpha);
                    }
                    return row;
                };
                uint16_t *dst = static_cast<uint16_t *>(a.out) + at;
                const uint4 packed = type == int(Type::F16) ? finish(std::true_type{}) : finish(std::false_type{});
                if (a.vector_io) {
                    *reinterpret_cast<uint4 *>(dst) = packed;
                } else {
                    dst[0] = uint16_t(packed.x); dst[1] = uint16_t(packed.x >> 16);
                    dst[2] = uint16_t(packed.y); dst[3] = uint16_t(packed.y >> 16);
                    dst[4] = uint16_t(packed.z); dst[5] = uint16_t(packed.z >> 16);
                    dst[6] = uint16_t(packed.w); dst[7] = uint16_t(packed.w >> 16);
                }
            }
        }
    }
    if ((warp < 2 || warp >= kGemmThreads / 32) && split_k) ptx::cluster_sync(); // the other warps' share of the phase barrier

    __syncthreads(); // tensor memory is drained and nobody else will touch this CTA's shared memory
    if (warp == 1) {
        ptx::tcgen05_fence_after();
        ptx::tmem_dealloc(tmem_base, kTmemColumns);
    }
    if (threadIdx.x == 0 && abort_flag) atomicExch(a.status, 1 + tile_linear);
}
} // namespace tts::b200
