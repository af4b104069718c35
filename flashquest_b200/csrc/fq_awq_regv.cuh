// AWQ W4A16 linears for 1..8 rows with the weights in registers (fq_awq_regv.cu).
#pragma once
#include "fq_common.cuh"

namespace fq {

constexpr int RV_MAX_PROJ = 4;

struct RegvCall {
    const void* x; int M, K, group, n_proj, interleaved;
    const int32_t* qweight[RV_MAX_PROJ]; const void* scales[RV_MAX_PROJ]; const int32_t* qzeros[RV_MAX_PROJ]; const void* bias[RV_MAX_PROJ];
    int N[RV_MAX_PROJ]; void* y[RV_MAX_PROJ];
    const fq_gemv_prologue* pro; const fq_gemv_rope* rope;       // or null
};

bool awq_regv_supported(const RegvCall& c);
int awq_regv_launch(const RegvCall& c, void* stream, const char* fn);

}  // namespace fq
