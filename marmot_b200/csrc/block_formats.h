// The GGUF block formats of the weights (layouts: include/marmot/quant_block.h:48-52,91-97,111-117 in the reference tree).  Plain C++
// apart from the qualifiers, so that host code without CUDA can include it.
#pragma once

#ifdef __CUDACC__
#define MCU_HD __host__ __device__ __forceinline__
#else
#define MCU_HD inline
#endif

namespace mcu {

constexpr int QK_K = 256;
constexpr int Q8_0_VALUES = 32;
constexpr int Q4_K_BYTES = 144;
constexpr int Q6_K_BYTES = 210;
constexpr int Q8_0_BYTES = 34;

enum Kind : int { KIND_Q8_0 = 5, KIND_Q4_K = 9, KIND_Q6_K = 11 };

MCU_HD int block_values(int kind) { return kind == KIND_Q8_0 ? Q8_0_VALUES : QK_K; }
MCU_HD int block_bytes(int kind) {
    return kind == KIND_Q4_K ? Q4_K_BYTES : kind == KIND_Q6_K ? Q6_K_BYTES : Q8_0_BYTES;
}
MCU_HD bool kind_supported(int kind) {
    return kind == KIND_Q8_0 || kind == KIND_Q4_K || kind == KIND_Q6_K;
}

}  // namespace mcu
