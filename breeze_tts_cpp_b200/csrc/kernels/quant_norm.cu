// Fused producer of the QKV / gate-up activations: x += update (optionally scaled, written back),
// RMSNorm, then per-row / K-group / rotated quantization of the normalized 16-bit value, all with
// the row held in registers (one 128-bit load and one 64-bit store per thread).
//
// Replaces the reference kernel `residual_rms_quantize` (src/ops/kernels/quant/quant_norm.cu:14-123).
// Rounding points and reduction order are kept so the bytes match that kernel bit for bit:
// the residual sum and the weight product happen in storage precision, squares are summed per
// thread over its four pairs, then a shuffle-down tree per warp, then serially over the eight
// warps; the norm uses the hardware reciprocal square root. Compile with --fmad=false.
#include "kernels/quant_norm.h"
#include "kernels/quant_blocks.cuh"
#include "kernels/launch.cuh"
#include <stdexcept>
#include <string>

namespace tts {
namespace b200 {
namespace {
constexpr int kThreads = 256;
template <class T> struct Pair16;
template <> struct Pair16<__nv_bfloat16> {
    using P = __nv_bfloat162;
    __device__ static float2 unpack(P v) { return __bfloat1622float2(v); }
    __device__ static P pack(float x, float y) { return __floats2bfloat162_rn(x, y); }
};
template <> struct Pair16<__half> {
    using P = __half2;
    __device__ static float2 unpack(P v) { return __half22float2(v); }
    __device__ static P pack(float x, float y) { return __floats2half2_rn(x, y); }
};

template <class T> __device__ __forceinline__ uint4 load_raw8(const T *p, int remaining, bool aligned) {
    uint4 raw = make_uint4(0, 0, 0, 0);
    if (aligned && remaining >= 8) return load_upstream16(p);
    T *e = reinterpret_cast<T *>(&raw);
    for (int i = 0; i < 8; ++i)
        if (i < remaining) e[i] = load_upstream(p + i);
    return raw;
}
template <class T> __device__ __forceinline__ void store_raw8(T *p, uint4 raw, int remaining, bool aligned) {
    if (aligned && remaining >= 8) {
        *reinterpret_cast<uint4 *>(p) = raw;
        return;
    }
    const T *e = reinterpret_cast<const T *>(&raw);
    for (int i = 0; i < 8; ++i)
        if (i < remaining) p[i] = e[i];
}

// `Packed`: aligned rows, one scale per row, no rotation. An instance of its own without the other paths (in a decoder chain
// every launch finds the instruction caches cold).
template <Type F, class T, bool Add, bool Rotate, bool Packed>
__global__ void __launch_bounds__(kThreads)
rms_quantize(T *__restrict__ x, const T *__restrict__ update, const T *__restrict__ weight,
             const T *__restrict__ update_scale, unsigned char *__restrict__ out, float *__restrict__ scales,
             int rows, int cols, float eps, bool gemma, int group, bool any_aligned, bool rehearse) {
    const bool aligned = Packed || any_aligned;
    using M = Pair16<T>;
    using P = typename M::P;
    __shared__ float slots[kThreads / 32];
    pdl_launch_dependents();
    const int row = blockIdx.x, column = threadIdx.x * 8;
    uint4 w = make_uint4(0, 0, 0, 0);
    if (column < cols) w = load_raw8(weight + column, cols - column, aligned); // a parameter: may precede the wait
    // `rehearse` (kRehearsedRows): once through on zeros before the wait, without a global access.
#pragma unroll 1
    for (int pass = Packed && rehearse ? 0 : 1; pass < 2; ++pass) {
        const bool real = !Packed || pass;
        if (Packed && rehearse && real) __syncthreads(); // the rehearsal's maxima have been read
        if (real) pdl_wait_upstream();
        uint4 value = make_uint4(0, 0, 0, 0);
        if (real && column < cols) {
            const int remaining = cols - column;
            value = load_raw8(x + size_t(row) * cols + column, remaining, aligned);
            if (Add) {
                uint4 u = load_raw8(update + size_t(row) * cols + column, remaining, aligned);
                uint4 s = update_scale ? load_raw8(update_scale + column, remaining, aligned) : make_uint4(0, 0, 0, 0);
                P *vp = reinterpret_cast<P *>(&value), *up = reinterpret_cast<P *>(&u), *sp = reinterpret_cast<P *>(&s);
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    P b = up[p];
                    if (update_scale) b = __hmul2(b, sp[p]);
                    vp[p] = __hadd2(vp[p], b);
                }
                store_raw8(x + size_t(row) * cols + column, value, remaining, aligned);
            }
        }
        float sum = 0.f;
        {
            const P *vp = reinterpret_cast<const P *>(&value);
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                float2 f = M::unpack(vp[p]);
                sum = __fadd_rn(sum, __fadd_rn(__fmul_rn(f.x, f.x), __fmul_rn(f.y, f.y)));
            }
        }
#pragma unroll
        for (int d = 16; d; d >>= 1) sum = __fadd_rn(sum, __shfl_down_sync(0xffffffffu, sum, d));
        if (!(threadIdx.x & 31)) slots[threadIdx.x >> 5] = sum;
        __syncthreads();
        float total = 0.f;
#pragma unroll
        for (int p = 0; p < kThreads / 32; ++p) total = __fadd_rn(total, slots[p]);
        __syncthreads();
        const float inv_norm = rsqrtf(__fadd_rn(__fdiv_rn(total, float(cols)), eps));
        float v[1][8];
        {
            const P *vp = reinterpret_cast<const P *>(&value), *wp = reinterpret_cast<const P *>(&w);
            if (Packed) { // the normalized row stays in packed storage precision
                uint4 row_words[1];
                P *np = reinterpret_cast<P *>(&row_words[0]);
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    const float2 f = M::unpack(vp[p]), wf = M::unpack(wp[p]);
                    np[p] = gemma ? M::pack(__fmul_rn(__fmul_rn(f.x, inv_norm), __fadd_rn(wf.x, 1.f)),
                                            __fmul_rn(__fmul_rn(f.y, inv_norm), __fadd_rn(wf.y, 1.f)))
                                  : __hmul2(M::pack(__fmul_rn(f.x, inv_norm), __fmul_rn(f.y, inv_norm)), wp[p]);
                }
                if (column >= cols) row_words[0] = make_uint4(0, 0, 0, 0);
                quantize_row_packed<F, T, kThreads, 1>(row_words, out + size_t(row) * cols, scales + row, cols,
                                                       reinterpret_cast<uint32_t *>(slots), real);
                continue;
            }
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                float2 f = M::unpack(vp[p]);
                P normalized;
                if (gemma) {
                    float2 wf = M::unpack(wp[p]);
                    normalized = M::pack(__fmul_rn(__fmul_rn(f.x, inv_norm), __fadd_rn(wf.x, 1.f)),
                                         __fmul_rn(__fmul_rn(f.y, inv_norm), __fadd_rn(wf.y, 1.f)));
                } else {
                    normalized = __hmul2(M::pack(__fmul_rn(f.x, inv_norm), __fmul_rn(f.y, inv_norm)), wp[p]);
                }
                float2 r = M::unpack(normalized);
                v[0][2 * p] = column < cols ? r.x : 0.f;
                v[0][2 * p + 1] = column < cols ? r.y : 0.f;
            }
        }
        quantize_tail<F, kThreads, 1, Rotate>(v, out, scales, row, rows, cols, group, 0, 1, aligned, slots);
    }
}

// K-group mode with rotation: 64 threads per row, 32 consecutive columns each, so that four lanes hold a block for the
// shared rotate-and-quantize step; one to four rows per CTA. The squares are added up in the order of rms_quantize: a
// lane's 32 columns are four of that kernel's threads (eight columns each, summed alike), its shuffle distances 16, 8 and
// 4 are lane distances 4, 2 and 1 here and 2 and 1 fall inside a lane; the eight warp sums are added in order.
template <Type F, class T, bool Add>
__global__ void __launch_bounds__(kThreads)
rms_quantize_blocks(T *__restrict__ x, const T *__restrict__ update, const T *__restrict__ weight, const T *__restrict__ update_scale,
                    unsigned char *__restrict__ out, float *__restrict__ scales, int rows, int cols, float eps, bool gemma, bool rehearse) {
    __shared__ float slots[kThreads / 64][8];
    pdl_launch_dependents();
    const int slot = int(threadIdx.x) / 64, lane = int(threadIdx.x) % 64;
    const int row = int(blockIdx.x) * int(blockDim.x / 64) + slot, column = lane * 32;
    const bool active = row < rows && column < cols;
    uint32_t mask[16], w[16], value[16];
    if (active) { // a table and a parameter: may precede the wait (behind it the weight costs 2 % of a K-group decode step)
        load_masks(column, mask);
        load_row32(weight + column, w);
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) mask[i] = w[i] = 0u;
    }
    T *mine = x + size_t(row) * cols + column;
#pragma unroll 1
    for (int pass = rehearse ? 0 : 1; pass < 2; ++pass) { // as in rms_quantize
        if (pass) {
            __syncthreads(); // the rehearsal's sums have been read
            pdl_wait_upstream();
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) value[i] = 0u;
        if (active && pass) {
            load_row32(mine, value);
            if (Add) {
                uint32_t u[16];
                load_row32(update + size_t(row) * cols + column, u);
                if (update_scale) {
                    uint32_t s[16];
                    load_row32(update_scale + column, s);
#pragma unroll
                    for (int i = 0; i < 16; ++i) u[i] = mul16x2<T>(u[i], s[i]);
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) value[i] = add16x2<T>(value[i], u[i]);
                store_row32(mine, value);
            }
        }
        float sum[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            sum[t] = 0.f;
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                const float2 f = unpack_f32x2(widen2<T>(value[4 * t + p]));
                sum[t] = __fadd_rn(sum[t], __fadd_rn(__fmul_rn(f.x, f.x), __fmul_rn(f.y, f.y)));
            }
        }
#pragma unroll
        for (int d = 4; d; d >>= 1)
#pragma unroll
            for (int t = 0; t < 4; ++t) sum[t] = __fadd_rn(sum[t], __shfl_down_sync(0xffffffffu, sum[t], d));
        if (!(lane & 7)) slots[slot][lane >> 3] = __fadd_rn(__fadd_rn(sum[0], sum[2]), __fadd_rn(sum[1], sum[3]));
        __syncthreads();
        float total = 0.f;
#pragma unroll
        for (int p = 0; p < 8; ++p) total = __fadd_rn(total, slots[slot][p]);
        const float inv_norm = rsqrtf(__fadd_rn(__fdiv_rn(total, float(cols)), eps));
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float2 f = unpack_f32x2(widen2<T>(value[i]));
            if (gemma) {
                const float2 wf = unpack_f32x2(widen2<T>(w[i]));
                value[i] = Packed16<T>::pack(__fmul_rn(__fmul_rn(f.x, inv_norm), __fadd_rn(wf.x, 1.f)),
                                             __fmul_rn(__fmul_rn(f.y, inv_norm), __fadd_rn(wf.y, 1.f)));
            } else {
                value[i] = mul16x2<T>(Packed16<T>::pack(__fmul_rn(f.x, inv_norm), __fmul_rn(f.y, inv_norm)), w[i]);
            }
            value[i] ^= mask[i];
        }
        rotate_quantize32<F, T>(value, out + size_t(row) * cols + column, scales + size_t(column / 128) * rows + row, active && pass);
    }
}

template <Type F, class T>
void launch(T *x, const T *update, const T *weight, const T *update_scale, unsigned char *q, float *s, int rows,
            int cols, float eps, bool gemma, int group, int rotation, int sms, cudaStream_t stream) {
    const bool aligned = cols % 8 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0 &&
                         reinterpret_cast<uintptr_t>(weight) % 16 == 0 && reinterpret_cast<uintptr_t>(q) % 8 == 0 &&
                         (!update || reinterpret_cast<uintptr_t>(update) % 16 == 0) &&
                         (!update_scale || reinterpret_cast<uintptr_t>(update_scale) % 16 == 0);
    const auto aligned32 = [](const void *p) { return reinterpret_cast<uintptr_t>(p) % 32 == 0; };
    if (rotation && group == 128 && cols % 128 == 0 && aligned32(x) && aligned32(weight) && aligned32(q) && aligned32(update) &&
        aligned32(update_scale)) {
        // Four rows per CTA once that still leaves every multiprocessor one.
        const int per_cta = rows >= 4 * sms ? 4 : rows >= 2 * sms ? 2 : 1;
        const dim3 grid(unsigned((rows + per_cta - 1) / per_cta)), block(unsigned(64 * per_cta));
        if (update)
            launch_pdl("quantized norm launch", rms_quantize_blocks<F, T, true>, grid, block, 0, stream, x, update, weight, update_scale, q,
                       s, rows, cols, eps, gemma, rows <= kRehearsedRows);
        else
            launch_pdl("quantized norm launch", rms_quantize_blocks<F, T, false>, grid, block, 0, stream, x, update, weight, update_scale,
                       q, s, rows, cols, eps, gemma, rows <= kRehearsedRows);
        return;
    }
#define B200Q_RUN(ADD, ROT)                                                                        \
    launch_pdl("quantized norm launch", aligned && !group && !ROT ? rms_quantize<F, T, ADD, false, true> : rms_quantize<F, T, ADD, ROT, false>, dim3(rows), dim3(kThreads), 0, stream, x, update,   \
               weight, update_scale, q, s, rows, cols, eps, gemma, group, aligned, rows <= kRehearsedRows)
    if (update) { if (rotation) B200Q_RUN(true, true); else B200Q_RUN(true, false); }
    else { if (rotation) B200Q_RUN(false, true); else B200Q_RUN(false, false); }
#undef B200Q_RUN
}
} // namespace
} // namespace b200

void launch_quantized_norm(TensorView residual, TensorView update, TensorView weight, RowScaledView output,
                           float epsilon, bool gemma, TensorView update_scale, cudaStream_t stream, int multiprocessors) {
    output.validate();
    if (multiprocessors <= 0) multiprocessors = 148;
    // reference: quant_norm.cu:170-180
    if ((residual.type != Type::BF16 && residual.type != Type::F16) || !residual.data || !weight.data ||
        !output.values.data || !output.scales.data || !residual.dense() || residual.cols < 1 ||
        residual.cols > 2048 || residual.rows < 1 || residual.cols != output.values.cols ||
        residual.rows != output.values.rows || weight.type != residual.type || !weight.dense() ||
        weight.numel() != size_t(residual.cols) ||
        (update.data && (update.type != residual.type || update.rows != residual.rows ||
                         update.cols != residual.cols || !update.dense())) ||
        (update_scale.data && (update_scale.type != residual.type || !update_scale.dense() ||
                               update_scale.numel() != size_t(residual.cols))))
        throw std::invalid_argument("quantized RMS shape/type mismatch");
    auto *q = output.values.ptr<unsigned char>();
    auto *s = output.scales.ptr<float>();
    const bool fp8 = output.values.type == Type::FP8;
    auto run = [&](auto tag) {
        using T = decltype(tag);
        if (fp8)
            b200::launch<Type::FP8, T>(residual.ptr<T>(), update.ptr<const T>(), weight.ptr<const T>(),
                                       update_scale.ptr<const T>(), q, s, residual.rows, residual.cols, epsilon, gemma,
                                       output.group_size, output.rotation_size, multiprocessors, stream);
        else
            b200::launch<Type::I8, T>(residual.ptr<T>(), update.ptr<const T>(), weight.ptr<const T>(),
                                      update_scale.ptr<const T>(), q, s, residual.rows, residual.cols, epsilon, gemma,
                                      output.group_size, output.rotation_size, multiprocessors, stream);
    };
    if (residual.type == Type::F16) run(__half{});
    else run(__nv_bfloat16{});
    cudaError_t status = cudaGetLastError();
    if (status != cudaSuccess) throw std::runtime_error(std::string("quantized norm launch: ") + cudaGetErrorString(status));
}
} // namespace tts
