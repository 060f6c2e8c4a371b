// Rotation + quantization of 128-column K blocks: what the K-group modes (group 128, H128 rotation) run on every activation and weight.
// FOUR lanes per block, 32 consecutive columns per lane, and for long lists ONE lane per block (further down).
//
// Bound: instruction issue, then HBM. With eight columns per lane (quant_codec.cuh) a block takes four shuffle stages
// of eight values per lane, a hash per column for its sign and scalar fp32 throughout: about 300 instructions per
// 8 columns, 44 us for 12288 x 2048 where the traffic takes 12. Here five of the seven butterfly stages are inside
// a lane, most arithmetic is two-wide (add / mul / fma .f32x2), signs come from a table as masks for packed pairs,
// and INT8 bytes come from adding a constant instead of the conversion pipe: about 95 instructions per 8 columns.
// The arithmetic is that of quant_codec.cuh step for step (same butterfly order, same roundings), so bytes and scales
// are bit-identical to it.
#pragma once
#include "kernels/quant_codec.cuh"
#include <algorithm>

namespace tts::b200 {

__device__ __forceinline__ uint64_t f32x2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack_f32x2(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t sub_f32x2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// Largest magnitude of three, NaN if any is.
__device__ __forceinline__ float max_magnitude3(float a, float b, float c) {
    float r;
    asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
// Larger magnitude of the two, NaN if either is; the sign of the result means nothing.
__device__ __forceinline__ float max_magnitude(float a, float b) {
    float r;
    asm("max.NaN.xorsign.abs.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
// Two 16-bit values in one word -> fp32 pair.
template <class T> __device__ __forceinline__ uint64_t widen2(uint32_t word);
template <> __device__ __forceinline__ uint64_t widen2<__nv_bfloat16>(uint32_t word) {
    return f32x2(__uint_as_float(word << 16), __uint_as_float(word & 0xffff0000u));
}
template <> __device__ __forceinline__ uint64_t widen2<__half>(uint32_t word) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&word));
    return f32x2(f.x, f.y);
}

// Eight 16-bit words (32 bytes) per access.
struct alignas(32) Words8 {
    uint64_t w[4];
};
__device__ __forceinline__ Words8 load_words8(const void *p) {
    Words8 r;
    asm volatile("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(r.w[0]), "=l"(r.w[1]), "=l"(r.w[2]), "=l"(r.w[3]) : "l"(p));
    return r;
}
__device__ __forceinline__ void store_words8(void *p, const Words8 &v) {
    asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(v.w[0]), "l"(v.w[1]), "l"(v.w[2]), "l"(v.w[3]) : "memory");
}
// 32 consecutive 16-bit elements (64 bytes, 32-byte aligned) as 16 packed words.
__device__ __forceinline__ void load_row32(const void *p, uint32_t (&raw)[16]) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const Words8 v = load_words8(static_cast<const char *>(p) + 32 * h);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            raw[8 * h + 2 * i] = uint32_t(v.w[i]);
            raw[8 * h + 2 * i + 1] = uint32_t(v.w[i] >> 32);
        }
    }
}

__device__ __forceinline__ void store_row32(void *p, const uint32_t (&raw)[16]) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        Words8 v;
#pragma unroll
        for (int i = 0; i < 4; ++i) v.w[i] = uint64_t(raw[8 * h + 2 * i]) | (uint64_t(raw[8 * h + 2 * i + 1]) << 32);
        store_words8(static_cast<char *>(p) + 32 * h, v);
    }
}
// Packed 16-bit arithmetic on a word of two values.
template <class T> struct Packed16;
template <> struct Packed16<__nv_bfloat16> {
    using P = __nv_bfloat162;
    __device__ __forceinline__ static uint32_t pack(float x, float y) {
        const P p = __floats2bfloat162_rn(x, y);
        return *reinterpret_cast<const uint32_t *>(&p);
    }
};
template <> struct Packed16<__half> {
    using P = __half2;
    __device__ __forceinline__ static uint32_t pack(float x, float y) {
        const P p = __floats2half2_rn(x, y);
        return *reinterpret_cast<const uint32_t *>(&p);
    }
};
template <class T> __device__ __forceinline__ uint32_t add16x2(uint32_t a, uint32_t b) {
    using P = typename Packed16<T>::P;
    const P r = __hadd2(*reinterpret_cast<const P *>(&a), *reinterpret_cast<const P *>(&b));
    return *reinterpret_cast<const uint32_t *>(&r);
}
template <class T> __device__ __forceinline__ uint32_t mul16x2(uint32_t a, uint32_t b) {
    using P = typename Packed16<T>::P;
    const P r = __hmul2(*reinterpret_cast<const P *>(&a), *reinterpret_cast<const P *>(&b));
    return *reinterpret_cast<const uint32_t *>(&r);
}

// Sign flips of the rotation as XOR masks for packed pairs of 16-bit values (column 2i in the low half).
constexpr int kMaskedColumns = 8192;
struct alignas(16) RotationMasks { // load_masks reads 16 bytes at a time
    uint32_t pair[kMaskedColumns / 2];
};
__host__ __device__ constexpr uint32_t rotation_flip(uint32_t column) { // 1 = the column's sign is flipped (rotation_sign == -1)
    uint32_t h = column * 0x45d9f3bu;
    h = (h ^ (h >> 16)) * 0x45d9f3bu;
    return ((h ^ (h >> 16)) & 1u) ^ 1u;
}
constexpr RotationMasks make_rotation_masks() {
    RotationMasks m{};
    for (int i = 0; i < kMaskedColumns / 2; ++i)
        m.pair[i] = (rotation_flip(uint32_t(2 * i)) << 15) | (rotation_flip(uint32_t(2 * i + 1)) << 31);
    return m;
}
static __device__ const RotationMasks rotation_masks = make_rotation_masks();
__device__ __forceinline__ void load_masks(int column, uint32_t (&mask)[16]) {
    if (column + 32 <= kMaskedColumns) {
        const uint4 *src = reinterpret_cast<const uint4 *>(&rotation_masks.pair[column / 2]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint4 v = __ldg(src + i);
            mask[4 * i] = v.x; mask[4 * i + 1] = v.y; mask[4 * i + 2] = v.z; mask[4 * i + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i)
            mask[i] = (rotation_flip(uint32_t(column + 2 * i)) << 15) | (rotation_flip(uint32_t(column + 2 * i + 1)) << 31);
    }
}

// Eight values -> eight bytes. `Finite`: every |v * inverse| is known to be at most 127.5 (no NaN), which a finite
// maximum guarantees.
template <Type F, bool Finite> __device__ __forceinline__ uint64_t encode8(const uint64_t *v, uint64_t inverse2) {
    uint64_t scaled[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) scaled[i] = mul_f32x2(v[i], inverse2);
    if constexpr (F == Type::I8 && Finite) {
        // 1.5 * 2^23 + x rounds x to an integer, half to even, and leaves it in the low bits: one add per value pair
        // instead of clamp and conversion. Scalar adds: the assembler contracts a packed multiply and a packed add
        // into one rounding, which would change ties (seen as one byte in 50,000).
        uint32_t b[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = unpack_f32x2(scaled[i]);
            b[2 * i] = __float_as_uint(__fadd_rn(f.x, 12582912.f));
            b[2 * i + 1] = __float_as_uint(__fadd_rn(f.y, 12582912.f));
        }
        const uint32_t lo = __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410);
        const uint32_t hi = __byte_perm(__byte_perm(b[4], b[5], 0x0040), __byte_perm(b[6], b[7], 0x0040), 0x5410);
        return uint64_t(lo) | (uint64_t(hi) << 32);
    } else {
        const float2 a = unpack_f32x2(scaled[0]), b = unpack_f32x2(scaled[1]), c = unpack_f32x2(scaled[2]), d = unpack_f32x2(scaled[3]);
        return uint64_t(Codec<F>::four(a.x, a.y, b.x, b.y)) | (uint64_t(Codec<F>::four(c.x, c.y, d.x, d.y)) << 32);
    }
}

// Rotates and quantizes the 128-column block this lane's group of four holds (lane & 3 = which 32 columns). `raw` = its 32 storage
// values with the signs already flipped (XOR with load_masks: the product with +-1). Hands every lane's 32 bytes and the block's
// scale to `store`. Every lane of the warp must call this.
template <Type F, class T, class Store> __device__ __forceinline__ void rotate_quantize32(const uint32_t (&raw)[16], Store store) {
    uint64_t v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = widen2<T>(raw[i]);
#pragma unroll
    for (int i = 0; i < 16; ++i) { // span 1: inside a pair
        const float2 f = unpack_f32x2(v[i]);
        v[i] = f32x2(__fadd_rn(f.x, f.y), __fsub_rn(f.x, f.y));
    }
    const uint64_t minus = f32x2(-1.f, -1.f);
#pragma unroll
    for (int span = 1; span < 16; span <<= 1) { // spans 2 to 16
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if (!(i & span)) {
                const uint64_t a = v[i], b = v[i | span];
                v[i] = add_f32x2(a, b);
                v[i | span] = fma_f32x2(b, minus, a); // a - b, rounded once
            }
        }
    }
#pragma unroll
    for (int span = 1; span < 4; span <<= 1) { // spans 32 and 64: across lanes
        const float sign = (threadIdx.x & span) ? -1.f : 1.f;
        const uint64_t sign2 = f32x2(sign, sign);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float2 f = unpack_f32x2(v[i]);
            const uint64_t other = f32x2(__shfl_xor_sync(0xffffffffu, f.x, span), __shfl_xor_sync(0xffffffffu, f.y, span));
            v[i] = fma_f32x2(v[i], sign2, other); // v + other, or other - v in the upper lane
        }
    }
    const uint64_t norm = f32x2(0.08838834764831845f, 0.08838834764831845f);
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        v[i] = mul_f32x2(v[i], norm);
        const float2 f = unpack_f32x2(v[i]);
        amax = max_magnitude(max_magnitude(amax, f.x), f.y);
    }
    amax = max_magnitude(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fabsf(max_magnitude(amax, __shfl_xor_sync(0xffffffffu, amax, 2)));
    const bool finite = amax <= FLT_MAX; // false for infinities and NaN
    if (__all_sync(0xffffffffu, finite)) {
        const float step = quant_scale<F>(amax);
        const float inverse = __fdiv_rn(1.f, step);
        const uint64_t inverse2 = f32x2(inverse, inverse);
        Words8 bytes;
#pragma unroll
        for (int i = 0; i < 4; ++i) bytes.w[i] = encode8<F, true>(v + 4 * i, inverse2);
        store(bytes, step);
        return;
    }
    // Infinities or NaN somewhere in the warp: the maximum that skips NaN, and the clamping encoder.
    float known = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float2 f = unpack_f32x2(v[i]);
        known = fmaxf(known, fmaxf(fabsf(f.x), fabsf(f.y)));
    }
    known = fmaxf(known, __shfl_xor_sync(0xffffffffu, known, 1));
    known = fmaxf(known, __shfl_xor_sync(0xffffffffu, known, 2));
    const float step = quant_scale<F>(known);
    const float inverse = __fdiv_rn(1.f, step);
    const uint64_t inverse2 = f32x2(inverse, inverse);
    Words8 bytes;
#pragma unroll
    for (int i = 0; i < 4; ++i) bytes.w[i] = encode8<F, false>(v + 4 * i, inverse2);
    store(bytes, step);
}
// The same into global memory: 32 bytes at `q` (32-byte aligned) and, from the first lane of the four, the scale; lanes with `active`
// false store nothing.
template <Type F, class T>
__device__ __forceinline__ void rotate_quantize32(const uint32_t (&raw)[16], unsigned char *q, float *scale, bool active) {
    rotate_quantize32<F, T>(raw, [&](const Words8 &bytes, float step) {
        if (!active) return;
        store_words8(q, bytes);
        if (!(threadIdx.x & 3)) *scale = step;
    });
}

// ---------------------------------------------------------------- long lists of blocks: one lane per block
// A warp takes 32 rows of one K group, a lane one row's whole 128 columns: no shuffle stage, signs that are the same for the warp, and
// one scale, division and address per 128 columns instead of per 32. 1570 instructions per 32 blocks, loads included, against 1960 with
// four lanes each. What that costs is warps (160 to 166 registers by type, three per scheduler), so the rows come by asynchronous copies, the next task's while
// this one is computed.
constexpr int kLaneBlockThreads = 64, kLaneBlockResident = 6; // CTAs per multiprocessor
constexpr int kLaneBlockBytes = 32 * 256;                      // 32 rows of 128 16-bit columns, per warp and operand
inline int lane_blocks_grid(int tasks, int sms) { return std::min((tasks + kLaneBlockThreads / 32 - 1) / (kLaneBlockThreads / 32), kLaneBlockResident * sms); }
// From three tasks per warp on: 12288 x 2048 20.2 -> 18.4 us and 4096 x 6144 17.2 -> 15.6, but 8192 x 2048 11.5 -> 12.2.
inline bool lane_blocks_pay(int tasks, int cols, int sms) { return cols <= kMaskedColumns && tasks >= 3 * kLaneBlockResident * (kLaneBlockThreads / 32) * sms; }

// 32 rows x 256 bytes from `source` (the first row's block, rows `stride` elements apart, `rows` of them left) into `buffer`; 16-byte
// pieces, XOR-swizzled by the row so that lanes read their rows without bank conflicts. Rows past the last one repeat it.
template <class T> __device__ __forceinline__ void lane_blocks_fetch(uint32_t buffer, const T *source, int stride, int rows) {
    const int lane = threadIdx.x & 31, piece = lane & 15;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int r = 2 * i + (lane >> 4), row = min(r, rows - 1);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(buffer + uint32_t((r * 16 + (piece ^ (r & 7))) * 16)),
                     "l"(source + size_t(row) * stride + piece * 8)
                     : "memory");
    }
}
__device__ __forceinline__ void lane_blocks_landed() {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
}
// Piece `p` (eight columns) of this lane's row.
__device__ __forceinline__ uint4 lane_blocks_read(uint32_t buffer, int p) {
    const int lane = threadIdx.x & 31;
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(buffer + uint32_t((lane * 16 + (p ^ (lane & 7))) * 16))
                 : "memory");
    return v;
}
// Rotates and quantizes a lane's block (K group `group`; the arithmetic of rotate_quantize32, butterfly by butterfly). Writes 128 bytes
// at `q` (32-byte aligned) and the scale; lanes with `active` false store nothing. All lanes of the warp call this.
template <Type F, class T>
__device__ __forceinline__ void rotate_quantize128(const uint32_t (&raw)[64], int group, unsigned char *q, float *scale, bool active) {
    uint64_t v[64];
    const uint4 *masks = reinterpret_cast<const uint4 *>(&rotation_masks.pair[group * 64]); // one address for the warp
#pragma unroll
    for (int p = 0; p < 16; ++p) { // span 1: inside a pair
        const uint4 m = __ldg(masks + p);
        const uint32_t flip[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = unpack_f32x2(widen2<T>(raw[4 * p + i] ^ flip[i]));
            v[4 * p + i] = f32x2(__fadd_rn(f.x, f.y), __fsub_rn(f.x, f.y));
        }
    }
#pragma unroll
    for (int span = 1; span < 64; span <<= 1) { // spans 2 to 64
#pragma unroll
        for (int i = 0; i < 64; ++i) {
            if (!(i & span)) {
                const uint64_t a = v[i], b = v[i | span];
                v[i] = add_f32x2(a, b);
                v[i | span] = sub_f32x2(a, b);
            }
        }
    }
    const uint64_t norm = f32x2(0.08838834764831845f, 0.08838834764831845f);
    float m[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 64; ++i) {
        v[i] = mul_f32x2(v[i], norm);
        const float2 f = unpack_f32x2(v[i]);
        m[i & 3] = max_magnitude3(m[i & 3], f.x, f.y);
    }
    float amax = max_magnitude3(max_magnitude3(m[0], m[1], m[2]), m[3], 0.f);
    const bool finite = __all_sync(0xffffffffu, amax <= FLT_MAX); // false for infinities and NaN anywhere in the warp
    if (!finite) {                                                // the maximum that skips NaN, and the clamping encoder
        amax = 0.f;
#pragma unroll
        for (int i = 0; i < 64; ++i) {
            const float2 f = unpack_f32x2(v[i]);
            amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
        }
    }
    const float step = quant_scale<F>(amax), inverse = __fdiv_rn(1.f, step);
    const uint64_t inverse2 = f32x2(inverse, inverse);
    if (active) *scale = step;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        Words8 bytes;
        if (finite) {
#pragma unroll
            for (int i = 0; i < 4; ++i) bytes.w[i] = encode8<F, true>(v + 16 * p + 4 * i, inverse2);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) bytes.w[i] = encode8<F, false>(v + 16 * p + 4 * i, inverse2);
        }
        if (active) store_words8(q + 32 * p, bytes);
    }
}

// ---------------------------------------------------------------- unrotated rows, kept in packed storage precision
// Running maximum of magnitudes, two per word, as unsigned 16-bit patterns: storage values order like their bits, and
// infinities and NaN come out on top instead of vanishing, which tells whether the fast encoder may be used.
__device__ __forceinline__ uint32_t max_magnitude16x2(uint32_t m, uint32_t word) {
    uint32_t r;
    asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(m), "r"(word & 0x7fff7fffu));
    return r;
}
__device__ __forceinline__ uint32_t fold_magnitude(uint32_t m) { return max(m & 0xffffu, m >> 16); }
template <class T> __device__ __forceinline__ float magnitude_value(uint32_t bits);
template <> __device__ __forceinline__ float magnitude_value<__nv_bfloat16>(uint32_t bits) { return __uint_as_float(bits << 16); }
template <> __device__ __forceinline__ float magnitude_value<__half>(uint32_t bits) { return __half2float(__ushort_as_half((unsigned short)bits)); }
template <class T> __device__ __forceinline__ bool magnitude_finite(uint32_t bits);
template <> __device__ __forceinline__ bool magnitude_finite<__nv_bfloat16>(uint32_t bits) { return bits < 0x7f80u; }
template <> __device__ __forceinline__ bool magnitude_finite<__half>(uint32_t bits) { return bits < 0x7c00u; }
// The maximum the scale rule uses when NaN are present: of everything that is not NaN.
template <class T> __device__ __forceinline__ float max_skipping_nan(float m, uint32_t word) {
    const float2 f = unpack_f32x2(widen2<T>(word));
    return fmaxf(m, fmaxf(fabsf(f.x), fabsf(f.y)));
}
// Eight storage values (four words) -> eight bytes.
template <Type F, class T> __device__ __forceinline__ uint64_t encode_words(uint4 words, uint64_t inverse2, bool finite) {
    const uint64_t v[4] = {widen2<T>(words.x), widen2<T>(words.y), widen2<T>(words.z), widen2<T>(words.w)};
    return finite ? encode8<F, true>(v, inverse2) : encode8<F, false>(v, inverse2);
}
// Tail of the per-row producers: the CTA holds one row as packed storage values, thread t, item j owning columns
// (j*Threads + t)*8 .. +7 (zeros past the end); one scale. `slots` holds one word per warp and is still being
// read on return: a barrier has to come before it is written again. Equals quantize_tail (quant_codec.cuh)
// bit for bit with about a third of its instructions.
template <Type F, class T, int Threads, int Items>
__device__ __forceinline__ void quantize_row_packed(const uint4 (&v)[Items], unsigned char *out, float *scale, int cols, uint32_t *slots,
                                                    bool store = true) {
    const auto cta_largest = [&](uint32_t bits) {
        bits = __reduce_max_sync(0xffffffffu, bits);
        if (!(threadIdx.x & 31)) slots[threadIdx.x >> 5] = bits;
        __syncthreads();
        uint32_t r = 0u;
#pragma unroll
        for (int w = 0; w < Threads / 32; ++w) r = max(r, slots[w]);
        return r;
    };
    uint32_t largest = 0u;
#pragma unroll
    for (int j = 0; j < Items; ++j)
        largest = max_magnitude16x2(max_magnitude16x2(max_magnitude16x2(max_magnitude16x2(largest, v[j].x), v[j].y), v[j].z), v[j].w);
    const uint32_t bits = cta_largest(fold_magnitude(largest));
    const bool finite = magnitude_finite<T>(bits);
    float amax = magnitude_value<T>(bits);
    if (!finite) { // infinities or NaN: the maximum that skips NaN, and the clamping encoder
        amax = 0.f;
#pragma unroll
        for (int j = 0; j < Items; ++j)
            for (uint32_t word : {v[j].x, v[j].y, v[j].z, v[j].w}) amax = max_skipping_nan<T>(amax, word);
        __syncthreads();
        amax = __uint_as_float(cta_largest(__float_as_uint(amax))); // non-negative floats order like their bits
    }
    const float step = quant_scale<F>(amax), inverse = __fdiv_rn(1.f, step);
    const uint64_t inverse2 = f32x2(inverse, inverse);
    if (!threadIdx.x && store) *scale = step;
#pragma unroll
    for (int j = 0; j < Items; ++j) {
        const int column = (j * Threads + int(threadIdx.x)) * 8;
        if (column < cols && store) *reinterpret_cast<uint64_t *>(out + column) = encode_words<F, T>(v[j], inverse2, finite);
    }
}
} // namespace tts::b200
