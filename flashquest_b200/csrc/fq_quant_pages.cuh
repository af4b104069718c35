// Bulk packing of whole pages (fq_quant_pages.cu), shared by the INT4, INT8 and TurboQuant append paths.
#pragma once
#include "fq_common.cuh"
#include "fq_exact_div.cuh"

namespace fq {

struct QuantPagesParams {
    // token stream head[0:n_head] ++ new, element strides of (b, h, token); K or V may be null
    const void *K_head, *V_head, *K_new, *V_new;
    int64_t hd_sb, hd_sh, hd_ss, nw_sb, nw_sh, nw_ss;
    int n_head, n_new, n_quant;              // n_quant: a multiple of the page size
    int B, H, D, page, bits;                 // bits: 4 or 8
    uint8_t *K_codes, *V_codes;              // K_codes null: page metadata only; V_codes null: no V
    int64_t cd_sb, cd_sh, cd_ss;             // bytes
    uint16_t *K_scale, *K_mn; int64_t km_sb, km_sh, km_sp;
    uint16_t *V_scale, *V_mn; int64_t vm_sb, vm_sh, vm_ss;
    void *stage_K, *stage_V; int64_t st_sb, st_sh, st_ss;     // rows for the n_head + n_new - n_quant tokens left over, or null
    int zero_rest;                           // also zero the staging rows behind them
};

template <typename T> struct Q2;
template <> struct Q2<__half> {
    using type = __half2;
    __device__ static float2 f2(uint32_t u) { return __half22float2(*reinterpret_cast<__half2*>(&u)); }
    __device__ static uint32_t mn(uint32_t a, uint32_t b) { uint32_t r; asm("min.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
    __device__ static uint32_t mx(uint32_t a, uint32_t b) { uint32_t r; asm("max.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
    static constexpr uint32_t POS_INF = 0x7c007c00u;
};
template <> struct Q2<__nv_bfloat16> {
    using type = __nv_bfloat162;
    __device__ static float2 f2(uint32_t u) { return make_float2(bf16_lo(u), bf16_hi(u)); }
    __device__ static uint32_t mn(uint32_t a, uint32_t b) { uint32_t r; asm("min.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
    __device__ static uint32_t mx(uint32_t a, uint32_t b) { uint32_t r; asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
    static constexpr uint32_t POS_INF = 0x7f807f80u;
};

// Scale of a page's channel, in the input dtype: max(rn(rn(hi - lo) / top), eps).
template <typename T>
__device__ __forceinline__ float page_scale(float hi, float lo, float top, float rtop, float eps) {
    return fmaxf(Dt<T>::rn(div_by_top(Dt<T>::rn(__fsub_rn(hi, lo)), top, rtop)), eps);
}

// Whether the kernel takes this call (else: the general kernels).
bool quant_pages_supported(const QuantPagesParams& p, int dtype);
int quant_pages_launch(const QuantPagesParams& p, int dtype, void* stream, const char* fn);

}  // namespace fq
