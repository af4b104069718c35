// W4A16 contraction for few rows of activations on the 5th-generation tensor cores (fq_awq_skinny.cu).
#pragma once
#include "fq_common.cuh"

namespace fq {

constexpr int SK_MAX_PROJ = 4;

struct SkinnyCall {
    const void* x; int M, K, group, n_proj, interleaved;
    const int32_t* qweight[SK_MAX_PROJ]; const void* scales[SK_MAX_PROJ]; const int32_t* qzeros[SK_MAX_PROJ]; const void* bias[SK_MAX_PROJ];
    int N[SK_MAX_PROJ]; void* y[SK_MAX_PROJ];
};

// Whether the kernel takes this call.
bool awq_skinny_supported(const SkinnyCall& c);
int awq_skinny_launch(const SkinnyCall& c, void* stream, const char* fn);

}  // namespace fq
