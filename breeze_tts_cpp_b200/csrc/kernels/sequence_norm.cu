// LayerNorm fused with quantization, and the fused LayerNorm + quantize + projection for narrow
// models (K <= 512), as sm_100a kernels behind the reference's operators.
//
// Replaces the reference's `norm_kernel<T, RowOutput>` (src/ops/kernels/sequence/sequence_norm.cu:64-204,
// launcher :412-440) and `norm_project_kernel<T, QuantProjection>` (:261-370, launcher :518-575).
// The statistics keep the reference's arithmetic so that the bytes match it: thread t sums columns
// t, t+256, ... in that order, warps are reduced by a shuffle-down tree with distances 1, 2, 4, 8, 16,
// thread 0 adds the eight warp sums in order, the variance accumulates fma(delta, delta, sum), the
// norm uses the hardware reciprocal square root, and every storage rounding point of the row
// pipeline (projection bias, gate, residual, weight, bias, scale, shift) is kept. The quantizing tail
// then works on eight consecutive columns per thread (128-bit accesses); maxima are exact, so the
// regrouping changes no bit. Compile with --fmad=false: contractions are written out.
#include "kernels/sequence_pointwise.h"
#include "kernels/launch.cuh"
#include "kernels/quant_blocks.cuh"
#include "kernels/sequence_finish.cuh"
#include <stdexcept>
#include <string>
#include <type_traits>

namespace tts {
namespace b200 {
namespace {
constexpr int kThreads = 256;
constexpr int kCached = 8; // strided values a thread keeps between the two statistics passes (2048 columns)

struct NormArgs {
    FinishOperand input, weight, bias, projection, residual, gate, shift, scale;
    void *output = nullptr, *raw = nullptr;
    int output_stride = 0, raw_stride = 0, rows_per_sequence = 1, input_rows = 0;
    const int *source_rows = nullptr;
    float eps = 0.f;
};

template <class T> struct NormRow {
    const T *input, *projection, *residual, *gate, *weight, *bias, *scale, *shift;
    template <class U> __device__ static const U *row_of(const FinishOperand &o, int row) {
        return o.data ? static_cast<const U *>(o.data) + size_t(o.rows == 1 ? 0 : row) * o.stride : nullptr;
    }
    __device__ NormRow(const NormArgs &a, int row) {
        const int sequence = row / a.rows_per_sequence;
        input = row_of<T>(a.input, row);
        projection = row_of<T>(a.projection, 0);
        residual = row_of<T>(a.residual, row);
        gate = row_of<T>(a.gate, sequence);
        weight = row_of<T>(a.weight, 0);
        bias = row_of<T>(a.bias, 0);
        scale = row_of<T>(a.scale, sequence);
        shift = row_of<T>(a.shift, sequence);
    }
    __device__ __forceinline__ static float read(const T *p, int c) { return p ? float(p[c]) : 0.f; }
    // The value that is normalized: input + projection bias, times gate, plus residual, rounded to
    // storage after every step (reference: NormRow::load, sequence_norm.cu:43-47).
    __device__ __forceinline__ float load(int c) const {
        float value = round_storage<T>(__fadd_rn(float(input[c]), read(projection, c)));
        if (gate) value = round_storage<T>(__fmul_rn(value, float(gate[c])));
        return round_storage<T>(__fadd_rn(value, read(residual, c)));
    }
    // reference: NormRow::transform, sequence_norm.cu:48-57
    __device__ __forceinline__ float transform(int c, float value, float mean, float inverse) const {
        value = __fmul_rn(__fsub_rn(value, mean), inverse);
        if (weight) value = __fmul_rn(value, float(weight[c]));
        value = round_storage<T>(__fadd_rn(value, read(bias, c)));
        if (scale) value = round_storage<T>(__fmul_rn(value, round_storage<T>(__fadd_rn(1.f, float(scale[c])))));
        return round_storage<T>(__fadd_rn(value, read(shift, c)));
    }
};

// Sum over the CTA in the order of a block reduction built from warp shuffle-down trees: the result is
// returned to every thread.
__device__ __forceinline__ float block_sum(float v, float *slots, float *broadcast) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) v = __fadd_rn(__shfl_down_sync(0xffffffffu, v, d), v);
    if (!(threadIdx.x & 31)) slots[threadIdx.x >> 5] = v;
    __syncthreads();
    if (!threadIdx.x) {
        float total = slots[0];
#pragma unroll
        for (int w = 1; w < kThreads / 32; ++w) total = __fadd_rn(total, slots[w]);
        *broadcast = total;
    }
    __syncthreads();
    return *broadcast;
}

// Mean and reciprocal standard deviation of one row.
template <class T>
__device__ __forceinline__ void row_statistics(const NormRow<T> &row, int cols, float eps, float *slots, float *shared,
                                               float &mean, float &inverse) {
    float cached[kCached], sum = 0.f;
#pragma unroll
    for (int i = 0; i < kCached; ++i) {
        const int c = int(threadIdx.x) + i * kThreads;
        cached[i] = c < cols ? row.load(c) : 0.f;
        sum = __fadd_rn(sum, cached[i]);
    }
    for (int c = int(threadIdx.x) + kCached * kThreads; c < cols; c += kThreads) sum = __fadd_rn(sum, row.load(c));
    mean = __fdiv_rn(block_sum(sum, slots, shared), float(cols));
    sum = 0.f;
#pragma unroll
    for (int i = 0; i < kCached; ++i) {
        if (int(threadIdx.x) + i * kThreads < cols) {
            const float delta = __fsub_rn(cached[i], mean);
            sum = __fmaf_rn(delta, delta, sum);
        }
    }
    for (int c = int(threadIdx.x) + kCached * kThreads; c < cols; c += kThreads) {
        const float delta = __fsub_rn(row.load(c), mean);
        sum = __fmaf_rn(delta, delta, sum);
    }
    inverse = rsqrtf(__fadd_rn(__fdiv_rn(block_sum(sum, slots, shared + 1), float(cols)), eps));
}

template <class T> __device__ __forceinline__ void store16(T *p, int remaining, const float (&v)[8]) {
    if ((reinterpret_cast<uintptr_t>(p) & 15) == 0 && remaining >= 8) {
        uint4 packed;
        T *e = reinterpret_cast<T *>(&packed);
#pragma unroll
        for (int i = 0; i < 8; ++i) e[i] = T(v[i]);
        *reinterpret_cast<uint4 *>(p) = packed;
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (i < remaining) p[i] = T(v[i]);
    }
}

template <Type F, class T, int Items, bool Rotate>
__global__ void __launch_bounds__(kThreads)
layer_norm_quantize_rows(NormArgs a, unsigned char *__restrict__ q, float *__restrict__ scales, int rows, int cols, int group) {
    __shared__ float slots[kThreads / 32];
    __shared__ float shared[2];
    pdl_launch_dependents();
    pdl_wait_upstream();
    const int output_row = blockIdx.x;
    const int row = a.source_rows ? a.source_rows[output_row] : output_row;
    T *output = a.output ? static_cast<T *>(a.output) + size_t(output_row) * a.output_stride : nullptr;
    T *raw = a.raw ? static_cast<T *>(a.raw) + size_t(output_row) * a.raw_stride : nullptr;
    const bool aligned = cols % 8 == 0 && (reinterpret_cast<uintptr_t>(q) & 7) == 0;
    float v[Items][8];
    if (row < 0 || row >= a.input_rows) {
        // A gathered row that does not exist poisons its output (reference: sequence_norm.cu:74-84).
        for (int c = threadIdx.x; c < cols; c += kThreads) {
            if (output) output[c] = T(nanf(""));
            q[size_t(output_row) * cols + c] = (unsigned char)Codec<F>::one(nanf(""));
        }
        const int groups = group ? (cols + group - 1) / group : 1;
        for (int g = threadIdx.x; g < groups; g += kThreads) scales[size_t(g) * rows + output_row] = 1.f;
        return;
    }
    const NormRow<T> fusion(a, row);
    float mean, inverse;
    row_statistics(fusion, cols, a.eps, slots, shared, mean, inverse);
#pragma unroll
    for (int j = 0; j < Items; ++j) {
        const int col = (j * kThreads + int(threadIdx.x)) * 8;
        float before[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const bool inside = col + i < cols;
            before[i] = inside ? fusion.load(col + i) : 0.f;
            v[j][i] = inside ? fusion.transform(col + i, before[i], mean, inverse) : 0.f;
        }
        if (col < cols) {
            if (raw) store16(raw + col, cols - col, before);
            if (output) store16(output + col, cols - col, v[j]);
        }
    }
    quantize_tail<F, kThreads, Items, Rotate>(v, q, scales, output_row, rows, cols, group, 0, 1, aligned, slots);
}

// Four words (eight storage values) of an optional operand row (16-byte aligned), zeros when absent.
template <class T> __device__ __forceinline__ uint4 row_words(const T *p, int c) {
    return p ? *reinterpret_cast<const uint4 *>(p + c) : make_uint4(0, 0, 0, 0);
}

// The same operator for aligned rows of up to 2048 columns, `Lanes` (32 or 128) threads per row, one row per warp or per
// CTA. Thread l owns columns (j*Lanes+l)*8..+7 of every stretch j: each operand is read once, by 128-bit loads. Sums and
// products that the row pipeline rounds to storage are packed 16-bit instructions (their single rounding equals the
// fp32 result rounded to storage, see add2x16 of the GEMM epilogue). The statistics keep the order of the CTA kernel
// above: the row goes through shared memory, this thread adds up the columns its threads 2l and 2l+1 (of every 2*Lanes)
// would have, in their order; their shuffle distance 1 falls inside the thread and 2 to 16 become lane distances 1 to 8,
// and the eight warp sums are added in order. That kernel reads every operand three times, two bytes at a time.
// Measured, kernel alone: 750 x 1024 8.6 -> about 4 us, 4096 x 2048 bf16 59 -> 14.5, 16 x 1024 4.7 -> 2.2.
template <Type F, class T, int Lanes, int Chunks, bool Rotate>
__global__ void __launch_bounds__(128)
layer_norm_quantize_packed(NormArgs a, unsigned char *__restrict__ q, float *__restrict__ scales, int rows, int cols, int group, bool rehearse) {
    extern __shared__ uint4 row_values[];       // per row: its storage values
    __shared__ float warp_sums[2][8];           // Lanes == 128: sums of the emulated warps, then mean and spread in turn
    __shared__ uint32_t warp_max[4];
    constexpr int kPairs = 128 / Lanes;          // emulated thread pairs per thread
    const int slot = Lanes == 32 ? int(threadIdx.x) / 32 : 0, lane = Lanes == 32 ? int(threadIdx.x) & 31 : int(threadIdx.x);
    const int output_row = Lanes == 32 ? int(blockIdx.x) * int(blockDim.x / 32) + slot : int(blockIdx.x);
    pdl_launch_dependents();
    if (output_row >= rows) { // a whole warp (Lanes == 32) or nobody
        pdl_wait_upstream();
        return;
    }
    const auto row_sync = [] {
        if (Lanes == 32) __syncwarp();
        else __syncthreads();
    };
    // `rehearse`: once through on zeros before the wait, without a global access, so that the code is in the instruction caches when
    // the input is there. (The operands' pointers are not __restrict__, so their plain loads stay behind the wait.)
#pragma unroll 1
    for (int pass = rehearse ? 0 : 1; pass < 2; ++pass) {
        const bool real = pass;
        const auto operand = [&](const T *p, int c) { return real ? row_words(p, c) : make_uint4(0, 0, 0, 0); };
        if (real) {
            row_sync(); // the rehearsal is done with the shared memory
            pdl_wait_upstream();
        }
        const int row = !real ? 0 : a.source_rows ? a.source_rows[output_row] : output_row;
        T *output = a.output ? static_cast<T *>(a.output) + size_t(output_row) * a.output_stride : nullptr;
        T *raw = a.raw ? static_cast<T *>(a.raw) + size_t(output_row) * a.raw_stride : nullptr;
        if (row < 0 || row >= a.input_rows) { // a gathered row that does not exist poisons its output
            for (int c = lane; c < cols; c += Lanes) {
                if (output) output[c] = T(nanf(""));
                q[size_t(output_row) * cols + c] = (unsigned char)Codec<F>::one(nanf(""));
            }
            const int groups = group ? (cols + group - 1) / group : 1;
            for (int g = lane; g < groups; g += Lanes) scales[size_t(g) * rows + output_row] = 1.f;
            return;
        }
        const NormRow<T> fusion(a, row);
        uint4 *mine = row_values + size_t(slot) * (cols / 8);
        uint4 v[Chunks];
#pragma unroll
        for (int j = 0; j < Chunks; ++j) {
            const int col = (j * Lanes + lane) * 8;
            v[j] = make_uint4(0, 0, 0, 0);
            if (real && col < cols) v[j] = *reinterpret_cast<const uint4 *>(fusion.input + col);
        }
#pragma unroll
        for (int j = 0; j < Chunks; ++j) {
            const int col = (j * Lanes + lane) * 8;
            if (col < cols) { // NormRow::load
                const uint4 p = operand(fusion.projection, col), g = operand(fusion.gate, col), r = operand(fusion.residual, col);
                uint32_t *w = reinterpret_cast<uint32_t *>(&v[j]);
                const uint32_t *pw = reinterpret_cast<const uint32_t *>(&p), *gw = reinterpret_cast<const uint32_t *>(&g),
                               *rw = reinterpret_cast<const uint32_t *>(&r);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    w[i] = add16x2<T>(w[i], pw[i]);
                    if (fusion.gate) w[i] = mul16x2<T>(w[i], gw[i]);
                    w[i] = add16x2<T>(w[i], rw[i]); // also without a residual: -0 + 0 is +0
                }
                mine[col / 8] = v[j];
                if (raw && real) *reinterpret_cast<uint4 *>(raw + col) = v[j];
            }
        }
        row_sync();
        const uint32_t *words = reinterpret_cast<const uint32_t *>(mine);
        // Sum over the row of per-pair partial sums, in the CTA kernel's order; the same value in every thread.
        const auto row_sum = [&](uint64_t (&pair)[kPairs], float *shared_sums) {
            float s[kPairs];
#pragma unroll
            for (int g = 0; g < kPairs; ++g) {
                const float2 f = unpack_f32x2(pair[g]);
                s[g] = __fadd_rn(f.x, f.y);
            }
#pragma unroll
            for (int d = 1; d < 16; d <<= 1)
#pragma unroll
                for (int g = 0; g < kPairs; ++g) s[g] = __fadd_rn(__shfl_down_sync(0xffffffffu, s[g], d), s[g]);
            // Lane 0 of every 16 holds a warp sum: warps 2g and 2g+1 of the order for Lanes == 32.
            if (Lanes == 32) {
                float total = 0.f;
#pragma unroll
                for (int g = 0; g < kPairs; ++g) {
                    const float lo = __shfl_sync(0xffffffffu, s[g], 0), hi = __shfl_sync(0xffffffffu, s[g], 16);
                    total = g ? __fadd_rn(total, lo) : lo;
                    total = __fadd_rn(total, hi);
                }
                return total;
            }
            if (!(lane & 15)) shared_sums[lane >> 4] = s[0];
            __syncthreads();
            float total = shared_sums[0];
#pragma unroll
            for (int w = 1; w < 8; ++w) total = __fadd_rn(total, shared_sums[w]);
            return total;
        };
        constexpr int kTerms = Chunks * Lanes * 8 / 256 > 0 ? Chunks * Lanes * 8 / 256 : 1; // columns per emulated thread
        uint64_t pair[kPairs], kept[kTerms][kPairs];
#pragma unroll
        for (int g = 0; g < kPairs; ++g) pair[g] = 0ull;
#pragma unroll
        for (int i = 0; i < kTerms; ++i)
#pragma unroll
            for (int g = 0; g < kPairs; ++g) {
                const int at = i * 128 + g * 32 + lane; // word index = column pair
                kept[i][g] = 0ull;
                if (2 * at < cols) {
                    kept[i][g] = widen2<T>(words[at]);
                    pair[g] = add_f32x2(pair[g], kept[i][g]);
                }
            }
        const float mean = __fdiv_rn(row_sum(pair, warp_sums[0]), float(cols));
        const uint64_t minus_mean = f32x2(-mean, -mean);
#pragma unroll
        for (int g = 0; g < kPairs; ++g) pair[g] = 0ull;
#pragma unroll
        for (int i = 0; i < kTerms; ++i)
#pragma unroll
            for (int g = 0; g < kPairs; ++g)
                if (2 * (i * 128 + g * 32 + lane) < cols) {
                    const uint64_t delta = add_f32x2(kept[i][g], minus_mean);
                    pair[g] = fma_f32x2(delta, delta, pair[g]);
                }
        const float inverse = rsqrtf(__fadd_rn(__fdiv_rn(row_sum(pair, warp_sums[1]), float(cols)), a.eps));
        const uint64_t inverse2 = f32x2(inverse, inverse);
        const uint32_t one16 = Packed16<T>::pack(1.f, 1.f);
        uint32_t largest = 0u;
#pragma unroll
        for (int j = 0; j < Chunks; ++j) {
            const int col = (j * Lanes + lane) * 8;
            if (col < cols) { // NormRow::transform
                const uint4 wt = operand(fusion.weight, col), bs = operand(fusion.bias, col), sc = operand(fusion.scale, col),
                            sh = operand(fusion.shift, col);
                uint32_t *w = reinterpret_cast<uint32_t *>(&v[j]);
                const uint32_t *ww = reinterpret_cast<const uint32_t *>(&wt), *bw = reinterpret_cast<const uint32_t *>(&bs),
                               *cw = reinterpret_cast<const uint32_t *>(&sc), *hw = reinterpret_cast<const uint32_t *>(&sh);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    uint64_t value = mul_f32x2(add_f32x2(widen2<T>(w[i]), minus_mean), inverse2);
                    if (fusion.weight) value = mul_f32x2(value, widen2<T>(ww[i]));
                    // Scalar adds: a packed one would be contracted with the product.
                    const float2 f = unpack_f32x2(value), b = unpack_f32x2(widen2<T>(bw[i]));
                    w[i] = Packed16<T>::pack(__fadd_rn(f.x, b.x), __fadd_rn(f.y, b.y));
                    if (fusion.scale) w[i] = mul16x2<T>(w[i], add16x2<T>(one16, cw[i]));
                    w[i] = add16x2<T>(w[i], hw[i]);
                    largest = max_magnitude16x2(largest, w[i]);
                }
                if (output && real) *reinterpret_cast<uint4 *>(output + col) = v[j];
            }
        }
        unsigned char *out = q + size_t(output_row) * cols;
        if (!group) {
            uint32_t bits = __reduce_max_sync(0xffffffffu, fold_magnitude(largest));
            if (Lanes > 32) {
                if (!(threadIdx.x & 31)) warp_max[threadIdx.x >> 5] = bits;
                __syncthreads();
                bits = max(max(warp_max[0], warp_max[1]), max(warp_max[2], warp_max[3]));
            }
            const bool finite = magnitude_finite<T>(bits);
            float amax = magnitude_value<T>(bits);
            if (!finite) { // uniform over the row's threads
                amax = 0.f;
#pragma unroll
                for (int j = 0; j < Chunks; ++j)
                    for (uint32_t word : {v[j].x, v[j].y, v[j].z, v[j].w}) amax = max_skipping_nan<T>(amax, word);
                uint32_t known = __reduce_max_sync(0xffffffffu, __float_as_uint(amax));
                if (Lanes > 32) {
                    __syncthreads();
                    if (!(threadIdx.x & 31)) warp_max[threadIdx.x >> 5] = known;
                    __syncthreads();
                    known = max(max(warp_max[0], warp_max[1]), max(warp_max[2], warp_max[3]));
                }
                amax = __uint_as_float(known);
            }
            const float step = quant_scale<F>(amax), reciprocal = __fdiv_rn(1.f, step);
            const uint64_t reciprocal2 = f32x2(reciprocal, reciprocal);
            if (!lane && real) scales[output_row] = step;
#pragma unroll
            for (int j = 0; j < Chunks; ++j) {
                const int col = (j * Lanes + lane) * 8;
                if (col < cols && real) *reinterpret_cast<uint64_t *>(out + col) = encode_words<F, T>(v[j], reciprocal2, finite);
            }
            continue;
        }
        if (Rotate && group == 128 && cols % 128 == 0 && (reinterpret_cast<uintptr_t>(q) & 31) == 0) {
            // Through shared memory once more, to 32 consecutive columns per thread.
            row_sync(); // everybody has read the statistics' copy
#pragma unroll
            for (int j = 0; j < Chunks; ++j) {
                const int col = (j * Lanes + lane) * 8;
                if (col < cols) mine[col / 8] = v[j];
            }
            row_sync();
            for (int first = 0; first < cols; first += Lanes * 32) {
                if (Lanes > 32 && first + int(threadIdx.x & ~31u) * 32 >= cols) break; // a whole warp without columns
                const int column = first + lane * 32;
                const bool active = column < cols;
                uint32_t w[16], mask[16];
                load_masks(active ? column : 0, mask);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint4 x = mine[(active ? column : 0) / 8 + i];
                    w[4 * i] = x.x ^ mask[4 * i]; w[4 * i + 1] = x.y ^ mask[4 * i + 1];
                    w[4 * i + 2] = x.z ^ mask[4 * i + 2]; w[4 * i + 3] = x.w ^ mask[4 * i + 3];
                }
                rotate_quantize32<F, T>(w, out + column, scales + size_t(column / 128) * rows + output_row, active && real);
            }
            continue;
        }
#pragma unroll
        for (int j = 0; j < Chunks; ++j) {
            const int col = (j * Lanes + lane) * 8;
            float f[8];
            unpack8<T>(v[j], f);
            if (Rotate) hadamard128(f, col);
            const float gmax = group_max(col < cols ? abs_max8(f) : 0.f, group >> 3);
            if (col < cols && real) {
                const float step = quant_scale<F>(gmax);
                if (!(col & (group - 1))) scales[size_t(col / group) * rows + output_row] = step;
                store8<F>(out + col, 8, true, f, __fdiv_rn(1.f, step));
            }
        }
    }
}

// Every row of every operand present starts on a 16-byte boundary and holds whole 8-column chunks.
bool rows_aligned(const NormArgs &a, int cols, const void *q) {
    auto ok = [](const void *p, int stride) { return !p || (reinterpret_cast<uintptr_t>(p) % 16 == 0 && stride % 8 == 0); };
    for (const FinishOperand *o : {&a.input, &a.weight, &a.bias, &a.projection, &a.residual, &a.gate, &a.shift, &a.scale})
        if (!ok(o->data, o->rows == 1 ? 0 : o->stride)) return false;
    return cols % 8 == 0 && ok(a.output, a.output_stride) && ok(a.raw, a.raw_stride) && reinterpret_cast<uintptr_t>(q) % 8 == 0;
}

template <Type F, class T, bool Rotate>
void launch_norm(const NormArgs &a, RowScaledView out, int sms, cudaStream_t stream) {
    const int rows = out.values.rows, cols = out.values.cols;
    auto *q = out.values.ptr<unsigned char>();
    auto *s = out.scales.ptr<float>();
    // Aligned rows of up to 2048 columns: one warp per row up to 512 columns, 128 threads per row beyond (a single warp
    // takes too long over a wide row, 9.4 us at 2048 columns however few the rows). Four warp rows per CTA once that still
    // leaves every multiprocessor one.
    if (cols <= 2048 && rows_aligned(a, cols, q)) {
        const int chunks = (cols + 255) / 256;
        const int per_cta = rows >= 4 * sms ? 4 : 1;
        // The rehearsal pays while the launch waits for the host or for a GEMM that leaves room beside it, which a row per warp does over the whole
        // range measured and a CTA per row up to one per multiprocessor: feed-forward blocks without / with it, 300 x 512 18.6 / 17.4 us,
        // 1000 x 256 2 %, 100 x 1536 3 %, 148 x 1024 1.5 %, but 200 x 2048 25.5 / 26.0, 296 x 768 (K groups) 20.7 / 21.6 and 900 x 1024 25.9 / 27.1.
        // In a graph it costs 2 to 12 % above these limits too, and changes little below them.
        const bool rehearse = rows <= (chunks <= 2 ? 8 : 1) * sms;
        const auto run = [&](auto lanes, auto count, int rows_per_cta) {
            constexpr int kLanes = decltype(lanes)::value, kCount = decltype(count)::value;
            launch_pdl("layer norm + quantize launch", layer_norm_quantize_packed<F, T, kLanes, kCount, Rotate>,
                       dim3(unsigned((rows + rows_per_cta - 1) / rows_per_cta)), dim3(unsigned(kLanes * rows_per_cta)),
                       size_t(rows_per_cta) * cols * 2, stream, a, q, s, rows, cols, out.group_size, rehearse);
        };
        using std::integral_constant;
        if (chunks <= 1) run(integral_constant<int, 32>{}, integral_constant<int, 1>{}, per_cta);
        else if (chunks <= 2) run(integral_constant<int, 32>{}, integral_constant<int, 2>{}, per_cta);
        else if (chunks <= 4) run(integral_constant<int, 128>{}, integral_constant<int, 1>{}, 1);
        else run(integral_constant<int, 128>{}, integral_constant<int, 2>{}, 1);
        return;
    }
#define B200Q_RUN(I)                                                                                                 \
    launch_pdl("layer norm + quantize launch", layer_norm_quantize_rows<F, T, I, Rotate>, dim3(rows), dim3(kThreads), 0, \
               stream, a, q, s, rows, cols, out.group_size)
    switch ((cols + kThreads * 8 - 1) / (kThreads * 8)) {
    case 1: B200Q_RUN(1); break;
    case 2: B200Q_RUN(2); break;
    case 3: B200Q_RUN(3); break;
    case 4: B200Q_RUN(4); break;
    default: throw std::invalid_argument("layer norm + quantize holds rows of up to 8192 columns");
    }
#undef B200Q_RUN
}

// ---------------------------------------------------------------- norm + quantize + projection, K <= 512
constexpr int kProjectionValues = 2;               // columns per thread: K <= 512
constexpr int kChannelsPerWarp = 8, kChannelsPerBlock = (kThreads / 32) * kChannelsPerWarp;

struct ProjectionArgs {
    const unsigned char *weight;
    const float *weight_scales;
    unsigned char *encoded;
    float *encoded_scales;
    void *output;
    int output_stride, channels, cols;
};

// Grid (ceil(N / 64), rows). Every CTA of a row normalizes and quantizes the row into shared memory
// (the first one also stores the row-level results), then each warp produces eight output channels:
// lanes stride the K axis four bytes at a time exactly as the reference's warp does, so FP8 sums are
// added in the same order; INT8 sums are exact integers. (A layer that was prepared for its rows runs LayerNorm +
// quantize and the GEMM instead, Linear::normalized_forward; its FP8 sums are the tensor cores'.)
template <Type F, class T>
__global__ void __launch_bounds__(kThreads)
norm_quantize_project(NormArgs a, ProjectionArgs p, FinishArgs finish) {
    __shared__ float slots[kThreads / 32];
    __shared__ float shared[3];
    __shared__ __align__(16) T activation[kThreads * kProjectionValues]; // FP8: decoded values; INT8: the bytes
    pdl_launch_dependents();
    pdl_wait_upstream();
    const int row = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, cols = p.cols;
    const NormRow<T> fusion(a, row);
    float values[kProjectionValues], sum = 0.f;
#pragma unroll
    for (int i = 0; i < kProjectionValues; ++i) {
        const int c = int(threadIdx.x) + i * kThreads;
        values[i] = c < cols ? fusion.load(c) : 0.f;
        sum = __fadd_rn(sum, values[i]);
    }
    const float mean = __fdiv_rn(block_sum(sum, slots, shared), float(cols));
    sum = 0.f;
#pragma unroll
    for (int i = 0; i < kProjectionValues; ++i)
        if (int(threadIdx.x) + i * kThreads < cols) {
            const float delta = __fsub_rn(values[i], mean);
            sum = __fmaf_rn(delta, delta, sum);
        }
    const float inverse = rsqrtf(__fadd_rn(__fdiv_rn(block_sum(sum, slots, shared + 1), float(cols)), a.eps));
    float rounded[kProjectionValues], amax = 0.f;
    T *normalized = a.output ? static_cast<T *>(a.output) + size_t(row) * a.output_stride : nullptr;
    T *raw = a.raw ? static_cast<T *>(a.raw) + size_t(row) * a.raw_stride : nullptr;
#pragma unroll
    for (int i = 0; i < kProjectionValues; ++i) {
        const int c = int(threadIdx.x) + i * kThreads;
        rounded[i] = 0.f;
        if (c < cols) {
            rounded[i] = fusion.transform(c, values[i], mean, inverse);
            amax = fmaxf(amax, fabsf(rounded[i]));
            if (!blockIdx.x) {
                if (raw) raw[c] = T(values[i]);
                if (normalized) normalized[c] = T(rounded[i]);
            }
        }
    }
    const float step = quant_scale<F>(cta_max<kThreads>(amax, slots));
    const float reciprocal = __fdiv_rn(1.f, step);
    if (!threadIdx.x && !blockIdx.x && p.encoded_scales) p.encoded_scales[row] = step;
#pragma unroll
    for (int i = 0; i < kProjectionValues; ++i) {
        const int c = int(threadIdx.x) + i * kThreads;
        if (c < cols) {
            const unsigned char byte = (unsigned char)Codec<F>::one(__fmul_rn(rounded[i], reciprocal));
            if (F == Type::I8) {
                reinterpret_cast<unsigned char *>(activation)[c] = byte;
            } else {
                const __half_raw decoded = __nv_cvt_fp8_to_halfraw(byte, __NV_E4M3);
                activation[c] = T(__half2float(__half(decoded)));
            }
            if (!blockIdx.x && p.encoded) p.encoded[size_t(row) * cols + c] = byte;
        }
    }
    __syncthreads();
    const FinishRow finish_of_row = finish_row(finish, row);
    T *out = static_cast<T *>(p.output) + size_t(row) * p.output_stride;
#pragma unroll 1
    for (int k = 0; k < kChannelsPerWarp; ++k) {
        const int channel = (blockIdx.x * (kThreads / 32) + warp) * kChannelsPerWarp + k;
        if (channel >= p.channels) break; // warp-uniform
        const unsigned char *w = p.weight + size_t(channel) * cols;
        float result;
        if (F == Type::I8) {
            int acc = 0;
            for (int c = lane * 4; c < cols; c += 128)
                acc = __dp4a(*reinterpret_cast<const int *>(reinterpret_cast<const unsigned char *>(activation) + c),
                             *reinterpret_cast<const int *>(w + c), acc);
            acc = __reduce_add_sync(0xffffffffu, acc);
            result = __fmul_rn(__fmul_rn(float(acc), p.weight_scales[channel]), step);
        } else {
            float acc = 0.f;
            for (int c = lane * 4; c < cols; c += 128) {
                const unsigned packed = *reinterpret_cast<const unsigned *>(w + c);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const __half_raw decoded = __nv_cvt_fp8_to_halfraw((packed >> (8 * i)) & 0xffu, __NV_E4M3);
                    acc = __fmaf_rn(float(activation[c + i]), __half2float(__half(decoded)), acc);
                }
            }
#pragma unroll
            for (int d = 16; d; d >>= 1) acc = __fadd_rn(acc, __shfl_down_sync(0xffffffffu, acc, d));
            result = __fmul_rn(__fmul_rn(acc, p.weight_scales[channel]), step);
        }
        if (!lane) out[channel] = T(finish_apply<T>(finish, finish_of_row, round_storage<T>(result), row, channel));
    }
}

NormArgs norm_args(TensorView x, TensorView weight, TensorView bias, float eps, const ops::NormFusion &f, TensorView output) {
    NormArgs a;
    a.input = FinishOperand(x);
    a.weight = FinishOperand(weight);
    a.bias = FinishOperand(bias);
    a.projection = FinishOperand(f.projection_bias);
    a.residual = FinishOperand(f.residual);
    a.gate = FinishOperand(f.gate);
    a.shift = FinishOperand(f.shift);
    a.scale = FinishOperand(f.scale);
    a.output = output.data;
    a.output_stride = output.ld();
    a.raw = f.raw.data;
    a.raw_stride = f.raw.ld();
    a.rows_per_sequence = f.rows_per_sequence;
    a.input_rows = x.rows;
    a.source_rows = f.source_rows;
    a.eps = eps;
    return a;
}
} // namespace
} // namespace b200

void launch_layer_norm_quantize(TensorView x, RowScaledView q, TensorView weight, TensorView bias, float eps,
                                const ops::NormFusion &f, TensorView retained, int multiprocessors, cudaStream_t stream) {
    const b200::NormArgs a = b200::norm_args(x, weight, bias, eps, f, retained);
    const bool fp8 = q.values.type == Type::FP8, rotate = q.rotation_size != 0;
    auto run = [&](auto tag) {
        using T = decltype(tag);
        if (fp8) {
            if (rotate) b200::launch_norm<Type::FP8, T, true>(a, q, multiprocessors, stream);
            else b200::launch_norm<Type::FP8, T, false>(a, q, multiprocessors, stream);
        } else {
            if (rotate) b200::launch_norm<Type::I8, T, true>(a, q, multiprocessors, stream);
            else b200::launch_norm<Type::I8, T, false>(a, q, multiprocessors, stream);
        }
    };
    if (x.type == Type::F16) run(__half{});
    else run(__nv_bfloat16{});
}

void launch_normalized_quantized_linear(TensorView x, TensorView normalized, TensorView norm_weight, TensorView norm_bias,
                                        float eps, const ops::NormFusion &f, RowScaledView weight, TensorView output,
                                        const ops::Epilogue &e, RowScaledView encoded, cudaStream_t stream) {
    const b200::NormArgs a = b200::norm_args(x, norm_weight, norm_bias, eps, f, normalized);
    b200::ProjectionArgs p{weight.values.ptr<unsigned char>(), weight.scales.ptr<float>(), encoded.values.ptr<unsigned char>(),
                           encoded.scales.ptr<float>(), output.data, output.ld(), weight.values.rows, weight.values.cols};
    const dim3 grid(unsigned((p.channels + b200::kChannelsPerBlock - 1) / b200::kChannelsPerBlock), unsigned(x.rows));
    const b200::FinishArgs finish(e);
    auto run = [&](auto tag) {
        using T = decltype(tag);
        if (weight.values.type == Type::FP8)
            b200::launch_pdl("norm + quantize + projection launch", b200::norm_quantize_project<Type::FP8, T>, grid,
                             dim3(b200::kThreads), 0, stream, a, p, finish);
        else
            b200::launch_pdl("norm + quantize + projection launch", b200::norm_quantize_project<Type::I8, T>, grid,
                             dim3(b200::kThreads), 0, stream, a, p, finish);
    };
    if (x.type == Type::F16) run(__half{});
    else run(__nv_bfloat16{});
}
} // namespace tts
