// Instances of the weight-streaming kernel that quantize their activations themselves, in a translation unit of their own.
#pragma once
#include "kernels/quant_linear_sm100.cuh"

namespace tts::b200 {
void raise_dense_limits(); // dynamic shared memory, on the current device
void launch_dense_instance(Type format, bool grouped, int tokens, Type input_type, const CUtensorMap &map_w, const DenseArgs &args, dim3 grid,
                           size_t smem, cudaStream_t stream);
} // namespace tts::b200
