#include "kernels/quant_linear_dense.h"
#include <stdexcept>
#include <string>

namespace tts::b200 {
namespace {
void check(cudaError_t status, const char *what) {
    if (status != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(status));
}
template <Type F, bool Grouped, int BN, class X> constexpr auto *instance() { return w8a8_tcgen05_gemm<F, Grouped, BN, false, true, X>; }
template <class Pick> auto by_instance(Type format, bool grouped, int tokens, Type input, Pick pick) {
    const auto typed = [&](auto f, auto g, auto bn) {
        constexpr Type F = decltype(f)::value;
        constexpr bool G = decltype(g)::value;
        constexpr int BN = decltype(bn)::value;
        return input == Type::F16 ? pick(instance<F, G, BN, __half>()) : pick(instance<F, G, BN, __nv_bfloat16>());
    };
    const auto of = [&](auto f) { // 32 tokens for K groups only
        if (!grouped) return typed(f, std::false_type{}, std::integral_constant<int, 16>{});
        return tokens == 16 ? typed(f, std::true_type{}, std::integral_constant<int, 16>{}) : typed(f, std::true_type{}, std::integral_constant<int, 32>{});
    };
    return format == Type::I8 ? of(std::integral_constant<Type, Type::I8>{}) : of(std::integral_constant<Type, Type::FP8>{});
}
} // namespace

void raise_dense_limits() {
    for (Type format : {Type::I8, Type::FP8})
        for (bool grouped : {false, true})
            for (int tokens : {dense_tokens(false), dense_tokens(grouped)})
                for (Type input : {Type::BF16, Type::F16})
                    by_instance(format, grouped, tokens, input, [](auto *kernel) {
                        check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemBudget)), "cudaFuncSetAttribute(shared memory)");
                    });
}

void launch_dense_instance(Type format, bool grouped, int tokens, Type input_type, const CUtensorMap &map_w, const DenseArgs &args, dim3 grid,
                           size_t smem, cudaStream_t stream) {
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = dim3(grouped ? kStreamThreads<true> : kStreamThreads<false>);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attributes[2];
    attributes[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[0].val.programmaticStreamSerializationAllowed = 1;
    attributes[1].id = cudaLaunchAttributeClusterDimension;
    attributes[1].val.clusterDim.x = attributes[1].val.clusterDim.y = 1;
    attributes[1].val.clusterDim.z = unsigned(args.splits);
    config.attrs = attributes;
    config.numAttrs = args.splits > 1 ? 2 : 1;
    by_instance(format, grouped, tokens, input_type, [&](auto *kernel) {
        check(cudaLaunchKernelEx(&config, kernel, map_w, map_w, args), "quantized GEMM launch");
    });
}
} // namespace tts::b200
