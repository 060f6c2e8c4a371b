// Launch helper shared by every kernel of the path: all of them are launched with the
// programmatic-stream-serialization attribute, so a kernel's prologue may overlap the tail of the
// kernel before it in the stream. The contract each kernel keeps in return:
//   * it executes `pdl_launch_dependents()` early, and
//   * it executes `pdl_wait_upstream()` before its first read of data a previous kernel may have
//     written and before its first global write. Only parameters that are complete by contract are read
//     earlier: announced weights with their scales (GEMMs) and RMSNorm weights. A kernel whose inputs are pointers to const
//     __restrict__ reads them by load_upstream16 and its kin (quant_codec.cuh): the compiler may move a plain load in front of the wait.
// Because every kernel waits for its predecessor to finish before it finishes itself, ordering
// stays transitive along the whole chain. Outside such a launch both instructions do nothing.
#pragma once
#include <cuda_runtime.h>
#include <stdexcept>
#include <string>

namespace tts::b200 {
__device__ __forceinline__ void pdl_launch_dependents() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait_upstream() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Quantizers of batches this short walk their code once before the wait (`rehearse`): a launch finds the instruction caches cold, and fetching the
// code while the GEMM in front still runs takes that off the chain's critical path. 28 layers, K groups INT8: 40 rows 1033 -> 966 us, 64 rows
// 1041 -> 1001; one scale per row 0.3 % at most. Beyond 64 rows the GEMMs in front leave no room to do it ahead of time, and it
// comes on top: a decoder layer of 79, 127 and 148 rows (INT8) 37.4, 39.3 and 42.2 us with it, 36.1, 38.2 and 40.2 without, K groups FP8
// 44.6, 48.3 and 58.6 against 43.8, 47.0 and 57.3; from 149 rows on no difference.
constexpr int kRehearsedRows = 64;

// Whether launches on `stream` are being recorded into a graph: they cost no host time then and follow one another without gaps.
inline bool being_captured(cudaStream_t stream) {
    if (!stream || stream == cudaStreamLegacy) return false; // never captured
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &status) == cudaSuccess) return status != cudaStreamCaptureStatusNone;
    (void)cudaGetLastError(); // the launch itself will say so
    return false;
}

template <class... Params, class... Args>
void launch_pdl(const char *what, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                Args... args) {
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    config.attrs = &attribute;
    config.numAttrs = 1;
    cudaError_t status = cudaLaunchKernelEx(&config, kernel, Params(args)...);
    if (status != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(status));
}
} // namespace tts::b200
