// Host launchers of the quantized GEMM. Signatures follow the reference's
// (src/ops/kernels/quant/quant_dispatch.h:7-17) so `QuantizedGemm` and any direct caller can
// switch without edits; `LinearKind::Tcgen05` is the only kind this build executes.
#pragma once
#include "core/quantization.h"
#include "core/tensor.h"
#include <cuda.h>
#include <cuda_runtime.h>

namespace tts {
namespace ops { struct Epilogue; }

void grouped_quant_gemm(KernelProblem, const void *input, const float *input_scales,
                        const void *weights, const float *weight_scales, void *output,
                        cudaStream_t, Type format, Type output_type, int tokens = 16, int splits = 1,
                        void *workspace = nullptr, size_t workspace_bytes = 0);
void launch_quant_linear(LinearPath config, KernelProblem shape, const void *input,
                         const float *input_scales, const void *weights, const float *weight_scales,
                         void *output, void *workspace, size_t workspace_bytes, cudaStream_t stream,
                         Type format = Type::FP8, Type output_type = Type::BF16,
                         const ops::Epilogue *finish = nullptr, const struct WeightMaps *prepared = nullptr);
// Initialization only; the fused finish needs no extra resources on this path.
KernelResources quant_linear_finish_resources(LinearPath, Type format, Type output_type);

// --- additions of this build -------------------------------------------------------------------
// An announced weight matrix, handed to `launch_quant_linear` through its last, optional argument. It says two things: here
// is the matrix's TMA descriptor (the weight-streaming kernel's), and the matrix and its scales were complete when it was made,
// so that a launch may fetch them before the kernels upstream of it are done. A launch whose weights it does not describe (or
// that passes none) builds the descriptor itself and reads nothing before its wait.
struct WeightMaps {
    CUtensorMap values; // 128 bytes of K x 128 rows
    const void *weights = nullptr;
    int channels = 0, reduction = 0;
};
// The GEMM on 16-bit activations, quantized inside the launch (a few rows): the bytes, scales and sums of launch_row_quantize and
// launch_quant_linear with this path. False when the launch does not take the operands or two launches are faster.
bool launch_dense_linear(LinearPath config, KernelProblem shape, int rotation, TensorView x, const void *weights, const float *weight_scales,
                         void *output, void *workspace, size_t workspace_bytes, cudaStream_t stream, Type format, Type output_type,
                         const ops::Epilogue *finish, const WeightMaps *prepared);
WeightMaps quant_linear_weight_maps(const void *weights, int channels, int reduction);
// Tile/split choice for a problem with the B200 chip model: tokens = token tile (16..256),
// channels = 128, splits = split-K. Shorthand for `select_linear` (ops/quantization_policy.h).
LinearPath select_tcgen05_path(KernelProblem, Type format, int multiprocessors, size_t workspace_bytes);
// Bytes of caller workspace a path needs (header + split-K partials).
size_t quant_linear_workspace_bytes(LinearPath, KernelProblem);
// One-time set-up per device and process: raises the dynamic shared-memory limit of every kernel
// instance and resolves the driver entry point for tensor maps. Call before stream capture.
void quant_linear_initialize(int device);
// Zeroes the ticket/status header of a fresh workspace (asynchronously on `stream`).
void quant_linear_reset_workspace(void *workspace, size_t workspace_bytes, cudaStream_t stream);
// Failure-path exercise without a GPU fault: the NEXT weight-streaming GEMM launched from this thread
// arms its first weight barrier for `extra_bytes` more than its (fully completing) copy delivers and
// lets every device-side wait give up after `limit_cycles` SM cycles, so the kernel runs to its normal
// teardown, stores nothing and raises the status word. One-shot; nothing is left in flight.
void quant_linear_inject_wait_expiry(int extra_bytes, long long limit_cycles);
// The same for scheduling: in the NEXT weight-streaming GEMM of this thread the warp that waits for refilled stages starts
// about that many nanoseconds late (at most 10^6), as it may when its multiprocessor is busy. Results do not depend on it.
void quant_linear_inject_refill_delay(int nanoseconds);
// Orders everything enqueued on `stream` so far before the start of everything after. The kernels of this library let their
// successors start while they still run, and pass that on: two launches after a kernel its results may not be there yet. A
// memory operation between them is an ordinary dependency on either side.
void quant_linear_settle(void *workspace, cudaStream_t stream);
// Blocking read of the status word: 0 = clean, otherwise 1 + index of the tile whose bounded wait gave up.
int quant_linear_status(const void *workspace, cudaStream_t stream);
} // namespace tts
