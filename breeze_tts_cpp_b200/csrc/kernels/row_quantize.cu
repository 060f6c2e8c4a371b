// Stage 1 (and the stage-3 producer) of the quantized linear path: dynamic per-token quantization
// of a 16-bit [rows,K] matrix to one-byte values plus fp32 scales, optionally after the matched
// H128 rotation and optionally with K-group scales. One pass over HBM: each thread keeps its
// 128-bit loads in registers across the amax reduction, so the row is read once and written once.
//
// Replaces the reference launcher `launch_row_quantize`
// (src/ops/kernels/quant/row_quantize.cu:167-193) and the four kernels behind it
// (:24-37 scalar, :42-87 register-cached, :90-115 rotated per-row, :145-165 K-group).
#include "kernels/row_quantize.h"
#include "kernels/quant_blocks.cuh"
#include "kernels/launch.cuh"
#include <stdexcept>

namespace tts {
namespace b200 {
namespace {
constexpr int kThreads = 256;

// Register-resident rows: K <= Items * 2048 * parts.
// `Packed`: aligned rows, one scale per row, no rotation; an instance of its own without the other paths (in a decoder chain
// every launch finds the instruction caches cold).
template <Type F, class T, int Items, bool Rotate, bool Packed>
__global__ void __launch_bounds__(kThreads)
row_quantize_cached(const T *__restrict__ x, unsigned char *__restrict__ q, float *__restrict__ scales,
                    int rows, int cols, int stride, int group, int parts, bool aligned, bool rehearse) {
    __shared__ float slots[kThreads / 32];
    pdl_launch_dependents();
    if (Packed) {
        const T *source = x + size_t(blockIdx.x) * stride;
#pragma unroll 1
        for (int pass = rehearse ? 0 : 1; pass < 2; ++pass) {
            if (pass) pdl_wait_upstream();
            uint4 raw[Items];
#pragma unroll
            for (int j = 0; j < Items; ++j) {
                const int column = (j * kThreads + int(threadIdx.x)) * 8;
                raw[j] = make_uint4(0, 0, 0, 0);
                if (pass && column < cols) raw[j] = load_upstream16(source + column);
            }
            quantize_row_packed<F, T, kThreads, Items>(raw, q + size_t(blockIdx.x) * cols, scales + blockIdx.x, cols, reinterpret_cast<uint32_t *>(slots), pass);
            __syncthreads();
        }
        return;
    }
    pdl_wait_upstream();
    const int row = blockIdx.x / parts, shard = blockIdx.x % parts;
    const T *source = x + size_t(row) * stride;
    float v[Items][8];
    if (Packed || aligned) {
        // All loads of the row shard are issued before the first value is used.
        uint4 raw[Items];
#pragma unroll
        for (int j = 0; j < Items; ++j) {
            int column = ((j * parts + shard) * kThreads + int(threadIdx.x)) * 8;
            raw[j] = column < cols ? load_upstream16(source + column) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int j = 0; j < Items; ++j) unpack8<T>(raw[j], v[j]);
    } else {
#pragma unroll
        for (int j = 0; j < Items; ++j) {
            int column = ((j * parts + shard) * kThreads + int(threadIdx.x)) * 8;
            if (column < cols) {
                load8(source + column, cols - column, false, v[j]);
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) v[j][i] = 0.f;
            }
        }
    }
    quantize_tail<F, kThreads, Items, Rotate>(v, q, scales, row, rows, cols, group, shard, parts,
                                              aligned, slots);
}

// Arbitrarily wide rows with one scale per row: two passes over the row (the second one mostly
// served by L2), the rotation recomputed rather than spilled.
template <Type F, class T, bool Rotate>
__global__ void __launch_bounds__(kThreads)
row_quantize_wide(const T *__restrict__ x, unsigned char *__restrict__ q, float *__restrict__ scales,
                  int cols, int stride, bool aligned) {
    __shared__ float slots[kThreads / 32];
    pdl_launch_dependents();
    pdl_wait_upstream();
    const int row = blockIdx.x;
    const T *source = x + size_t(row) * stride;
    const int padded = (cols + kThreads * 8 - 1) / (kThreads * 8) * (kThreads * 8);
    float amax = 0.f, v[8];
    for (int column = threadIdx.x * 8; column < padded; column += kThreads * 8) {
        load8(source + (column < cols ? column : 0), column < cols ? cols - column : 0, aligned, v);
        if (Rotate) hadamard128(v, column);
        if (column < cols) amax = fmaxf(amax, abs_max8(v));
    }
    float step = quant_scale<F>(cta_max<kThreads>(amax, slots));
    float inverse = __fdiv_rn(1.f, step);
    if (!threadIdx.x) scales[row] = step;
    for (int column = threadIdx.x * 8; column < padded; column += kThreads * 8) {
        load8(source + (column < cols ? column : 0), column < cols ? cols - column : 0, aligned, v);
        if (Rotate) hadamard128(v, column);
        if (column < cols)
            store8<F>(q + size_t(row) * cols + column, cols - column, aligned, v, inverse);
    }
}

// Long batches with one scale per row: one WARP per row, eight rows per CTA. The row stays in the
// lane's registers (up to 16 128-bit loads, all issued before the first use) and the amax needs only a
// warp reduction, so no CTA-wide barrier sits between the read and the write; with thousands of rows
// this keeps far more bytes in flight per SM than one small CTA per row. Max is exact, so the bytes
// and scales are the same as the CTA-per-row kernel's.
// `Resident` = CTAs per multiprocessor the register budget is cut for. More resident warps beat a spill-free
// kernel once there are rows enough to fill them (M=8192: K=2048 11.2 -> 9.5 us = 0.81 of the measured HBM rate
// with three CTAs; K=4096 14.4 -> 11.5 us with two); short batches keep the unconstrained kernel.
template <Type F, class T, int Loads, int Resident>
__global__ void __launch_bounds__(kThreads, Resident)
row_quantize_warp_rows(const T *__restrict__ x, unsigned char *__restrict__ q, float *__restrict__ scales, int rows,
                       int cols, int stride) {
    pdl_launch_dependents();
    pdl_wait_upstream();
    const int row = blockIdx.x * (kThreads / 32) + int(threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= rows) return;
    const T *source = x + size_t(row) * stride;
    uint4 raw[Loads];
#pragma unroll
    for (int j = 0; j < Loads; ++j) {
        const int column = (j * 32 + lane) * 8;
        raw[j] = column < cols ? load_upstream16(source + column) : make_uint4(0, 0, 0, 0);
    }
    uint32_t largest = 0u;
#pragma unroll
    for (int j = 0; j < Loads; ++j)
        largest = max_magnitude16x2(max_magnitude16x2(max_magnitude16x2(max_magnitude16x2(largest, raw[j].x), raw[j].y), raw[j].z), raw[j].w);
    const uint32_t bits = __reduce_max_sync(0xffffffffu, fold_magnitude(largest));
    const bool finite = magnitude_finite<T>(bits);
    float amax = magnitude_value<T>(bits);
    if (!finite) { // infinities or NaN: the maximum that skips NaN, and the clamping encoder
        amax = 0.f;
#pragma unroll
        for (int j = 0; j < Loads; ++j)
            for (uint32_t word : {raw[j].x, raw[j].y, raw[j].z, raw[j].w}) amax = max_skipping_nan<T>(amax, word);
        amax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(amax))); // non-negative floats order like their bits
    }
    const float step = quant_scale<F>(amax), inverse = __fdiv_rn(1.f, step);
    const uint64_t inverse2 = f32x2(inverse, inverse);
    if (!lane) scales[row] = step;
#pragma unroll
    for (int j = 0; j < Loads; ++j) {
        const int column = (j * 32 + lane) * 8;
        if (column < cols) *reinterpret_cast<uint64_t *>(q + size_t(row) * cols + column) = encode_words<F, T>(raw[j], inverse2, finite);
    }
}

// K-group mode with rotation (group 128): the blocks of all rows in one list, block i = K group i / rows of row i %
// rows, four lanes per block, eight blocks per warp. A block's scale then belongs at scales[i], a warp's eight scales
// share one 32-byte sector, and neither rows nor columns leave lanes idle. Against eight columns per lane: 8192 x 2048 11.5 us, 1021 x
// 2048 5.1 -> 3.1, 16 x 2048 1.7 -> 1.4; 12288 x 2048, which takes row_quantize_lanes now, 43.9 -> 19.6 (3.9 TB/s). One set of eight per warp: looping over four with the next one's loads in flight
// took 24.9 us, resident warps hide more. What is left is issue (491 instructions per 32 columns, 57 % busy).
template <Type F, class T>
__global__ void __launch_bounds__(kThreads, 3)
row_quantize_blocks(const T *__restrict__ x, unsigned char *__restrict__ q, float *__restrict__ scales, int rows, int cols,
                    int stride, int blocks, bool rehearse) {
    pdl_launch_dependents();
    const int first = (int(blockIdx.x) * int(blockDim.x >> 5) + int(threadIdx.x >> 5)) * 8;
    const int block = first + (int(threadIdx.x & 31) >> 2);
    const bool active = block < blocks;
    const int group = active ? block / rows : 0, row = active ? block - group * rows : 0;
    const int column = group * 128 + int(threadIdx.x & 3) * 32;
    uint32_t mask[16], raw[16];
    load_masks(column, mask); // static: may precede the wait
    if (first >= blocks) {
        pdl_wait_upstream();
        return;
    }
    // `rehearse` (kRehearsedRows): once through on the masks before the wait, without a global access.
#pragma unroll 1
    for (int pass = rehearse ? 0 : 1; pass < 2; ++pass) {
#pragma unroll
        for (int i = 0; i < 16; ++i) raw[i] = 0u;
        if (pass) {
            pdl_wait_upstream();
            load_row32(x + size_t(row) * stride + column, raw);
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) raw[i] ^= mask[i];
        rotate_quantize32<F, T>(raw, q + size_t(row) * cols + column, scales + block, active && pass);
    }
}

// The same with one lane per block for long lists (lane_blocks_pay): persistent warps over tasks of 32 rows x one K group, neighbouring
// warps on neighbouring groups. Bound by the fp32 pipe and issue; 12288 x 2048 20.2 -> 18.5 us against four lanes per block.
template <Type F, class T>
__global__ void __launch_bounds__(kLaneBlockThreads, kLaneBlockResident)
row_quantize_lanes(const T *__restrict__ x, unsigned char *__restrict__ q, float *__restrict__ scales, int rows, int cols, int stride,
                   int groups, int tasks) {
    extern __shared__ uint4 lane_buffers[];
    pdl_launch_dependents();
    const uint32_t buffer = uint32_t(__cvta_generic_to_shared(lane_buffers)) + (threadIdx.x >> 5) * kLaneBlockBytes;
    const int warps = int(gridDim.x) * (kLaneBlockThreads / 32);
    int task = __shfl_sync(0xffffffffu, int(blockIdx.x) * (kLaneBlockThreads / 32) + int(threadIdx.x >> 5), 0);
    pdl_wait_upstream();
    const auto fetch = [&](int t) {
        const int row0 = t / groups * 32;
        lane_blocks_fetch(buffer, x + size_t(row0) * stride + t % groups * 128, stride, rows - row0);
    };
    if (task < tasks) fetch(task);
#pragma unroll 1
    for (; task < tasks; task += warps) {
        const int group = task % groups, row = task / groups * 32 + int(threadIdx.x & 31);
        uint32_t raw[64];
        lane_blocks_landed();
#pragma unroll
        for (int p = 0; p < 16; ++p) {
            const uint4 w = lane_blocks_read(buffer, p);
            raw[4 * p] = w.x; raw[4 * p + 1] = w.y; raw[4 * p + 2] = w.z; raw[4 * p + 3] = w.w;
        }
        __syncwarp(); // everybody's row is in registers
        if (task + warps < tasks) fetch(task + warps);
        rotate_quantize128<F, T>(raw, group, q + size_t(row) * cols + group * 128, scales + size_t(group) * rows + row, row < rows);
    }
}

template <Type F, class T, bool Rotate>
void launch_typed(const T *x, unsigned char *q, float *scales, int rows, int cols, int stride,
                  int group, int multiprocessors, cudaStream_t stream) {
    const bool aligned = cols % 8 == 0 && stride % 8 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0 &&
                         reinterpret_cast<uintptr_t>(q) % 8 == 0;
    const int chunks = (cols + kThreads * 8 - 1) / (kThreads * 8); // 2048-column slabs per row
    if (!group && !Rotate && aligned && cols <= 4096 && rows >= 8 * multiprocessors) {
        const dim3 grid(unsigned((rows + kThreads / 32 - 1) / (kThreads / 32)));
#define B200Q_WARP_ROWS(L, R)                                                                                          \
    launch_pdl("row quantize launch", row_quantize_warp_rows<F, T, L, R>, grid, dim3(kThreads), 0, stream, x, q, scales,   \
               rows, cols, stride)
        const int loads = (cols + 255) / 256;
        const bool many = rows >= 24 * multiprocessors; // three CTAs of eight rows on every multiprocessor
        if (loads <= 4) B200Q_WARP_ROWS(4, 1);
        else if (loads <= 8) { if (many) B200Q_WARP_ROWS(8, 3); else B200Q_WARP_ROWS(8, 1); }
        else B200Q_WARP_ROWS(16, 2);
#undef B200Q_WARP_ROWS
        return;
    }
    if (Rotate && group == 128 && cols % 128 == 0 && stride % 16 == 0 && reinterpret_cast<uintptr_t>(x) % 32 == 0 &&
        reinterpret_cast<uintptr_t>(q) % 32 == 0 && int64_t(rows) * (cols / 128) < INT32_MAX - 4096) {
        const int blocks = rows * (cols / 128), tasks = (rows + 31) / 32 * (cols / 128);
        if (lane_blocks_pay(tasks, cols, multiprocessors)) {
            launch_pdl("row quantize launch", row_quantize_lanes<F, T>, dim3(unsigned(lane_blocks_grid(tasks, multiprocessors))), dim3(kLaneBlockThreads),
                       kLaneBlockThreads / 32 * kLaneBlockBytes, stream, x, q, scales, rows, cols, stride, cols / 128, tasks);
            return;
        }
        // Short batches take small CTAs, so that they spread over the machine.
        const int threads = blocks >= 8 * (kThreads / 32) * multiprocessors ? kThreads : 64;
        const int per_cta = 8 * (threads / 32);
        launch_pdl("row quantize launch", row_quantize_blocks<F, T>, dim3(unsigned((blocks + per_cta - 1) / per_cta)),
                   dim3(unsigned(threads)), 0, stream, x, q, scales, rows, cols, stride, blocks, rows <= kRehearsedRows);
        return;
    }
    int parts = 1;
    if (group) {
        // K groups never cross a 2048-column slab, so slabs of one row can go to different CTAs.
        // Spread short batches over the machine; long batches keep whole rows per CTA.
        while (parts < chunks && int64_t(rows) * parts * 2 <= multiprocessors) parts *= 2;
        if (chunks > 4 * parts) parts = (chunks + 3) / 4;
    } else if (chunks > 4) {
        launch_pdl("row quantize launch", row_quantize_wide<F, T, Rotate>, dim3(rows), dim3(kThreads), 0, stream, x, q, scales,
                   cols, stride, aligned);
        return;
    }
    const int items = (chunks + parts - 1) / parts;
    const unsigned grid = unsigned(rows) * unsigned(parts);
#define B200Q_LAUNCH(I)                                                                            \
    launch_pdl("row quantize launch", aligned && !group && !Rotate ? row_quantize_cached<F, T, I, false, true>                   \
                                                                    : row_quantize_cached<F, T, I, Rotate, false>, dim3(grid), dim3(kThreads), 0, stream, x, q, \
               scales, rows, cols, stride, group, parts, aligned, rows <= kRehearsedRows)
    switch (items) {
    case 1: B200Q_LAUNCH(1); break;
    case 2: B200Q_LAUNCH(2); break;
    case 3: B200Q_LAUNCH(3); break;
    default: B200Q_LAUNCH(4); break;
    }
#undef B200Q_LAUNCH
}

template <Type F, class T>
void launch_rotation(const T *x, unsigned char *q, float *scales, int rows, int cols, int stride,
                     int group, int rotation, int sms, cudaStream_t stream) {
    if (rotation) launch_typed<F, T, true>(x, q, scales, rows, cols, stride, group, sms, stream);
    else launch_typed<F, T, false>(x, q, scales, rows, cols, stride, group, sms, stream);
}
} // namespace
} // namespace b200

void launch_row_quantize(TensorView source, RowScaledView destination, cudaStream_t stream,
                         int multiprocessors) {
    destination.validate();
    if ((source.type != Type::BF16 && source.type != Type::F16) || !source.data ||
        !destination.values.data || !destination.scales.data || source.rows < 1 || source.cols < 1 ||
        source.rows != destination.values.rows || source.cols != destination.values.cols)
        throw std::invalid_argument("row quantization shape/type mismatch");
    if (int64_t(source.rows) * ((source.cols + 2047) / 2048) > INT32_MAX)
        throw std::invalid_argument("quantization grid exceeds capacity");
    if (multiprocessors <= 0) multiprocessors = 148;
    auto *q = destination.values.ptr<unsigned char>();
    auto *s = destination.scales.ptr<float>();
    const int rows = source.rows, cols = source.cols, ld = source.ld();
    const int group = destination.group_size, rotation = destination.rotation_size;
    const bool fp8 = destination.values.type == Type::FP8;
    if (source.type == Type::F16) {
        auto *x = source.ptr<const __half>();
        if (fp8) b200::launch_rotation<Type::FP8>(x, q, s, rows, cols, ld, group, rotation, multiprocessors, stream);
        else b200::launch_rotation<Type::I8>(x, q, s, rows, cols, ld, group, rotation, multiprocessors, stream);
    } else {
        auto *x = source.ptr<const __nv_bfloat16>();
        if (fp8) b200::launch_rotation<Type::FP8>(x, q, s, rows, cols, ld, group, rotation, multiprocessors, stream);
        else b200::launch_rotation<Type::I8>(x, q, s, rows, cols, ld, group, rotation, multiprocessors, stream);
    }
    cudaError_t status = cudaGetLastError();
    if (status != cudaSuccess)
        throw std::runtime_error(std::string("row quantize launch: ") + cudaGetErrorString(status));
}
} // namespace tts
