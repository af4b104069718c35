// One new token of the patched attention forward around the decode layer
// (flashquest/eager/llama_persistent_patch.py:164-245): the rotary embedding of q and k with Hugging Face's
// roundings, the cast to the cache's dtype, and the decode layer of the INT8 cache (append, page scores, selection,
// attention with the staged tail in the same softmax) as one host call.
#include "fq_append.cuh"
#include "fq_quant_pages.cuh"

namespace fq {

// q*cos + rotate_half(q)*sin, every product and the sum rounded to the model's dtype TM, then cast to the cache's
// dtype TC; v is only cast.  One CTA per (head, batch), a thread per channel pair (i, i + D/2).  Latency-bound: it
// replaces eleven element-wise launches of a few hundred values each.
// `pattern` (one byte per KV head, not 0: a retrieval head) is turned into the retention of every query head here, at each
// call: the caller's tensor may have changed since the last one.  The selection, two launches on or three, reads the result.
template <typename TM, typename TC>
__global__ void __launch_bounds__(64) rope_qkv_kernel(const TM* __restrict__ q, int64_t q_sb, const TM* __restrict__ k, int64_t k_sb,
                                                      const TM* __restrict__ v, int64_t v_sb, const TM* __restrict__ cosv, int64_t c_sb,
                                                      const TM* __restrict__ sinv, int64_t s_sb, int Hq, int Hkv, int D,
                                                      TC* __restrict__ q_out, TC* __restrict__ k_out, TC* __restrict__ v_out,
                                                      const uint8_t* __restrict__ pattern, int64_t pt_s, int n_rep, float retention, float* __restrict__ ret_out) {
    const int head = blockIdx.x, b = blockIdx.y, half = D / 2, i = threadIdx.x;
    pdl_wait();
    pdl_trigger();
    if (i >= half) return;
    const bool is_q = head < Hq, is_v = head >= Hq + Hkv;
    const int hh = is_q ? head : is_v ? head - Hq - Hkv : head - Hq;
    const TM* src = (is_q ? q + b * q_sb : is_v ? v + b * v_sb : k + b * k_sb) + (int64_t)hh * D;
    TC* dst = is_q ? q_out + ((int64_t)b * Hq + hh) * D : (is_v ? v_out : k_out) + ((int64_t)b * Hkv + hh) * D;
    const float x1 = Dt<TM>::to_f32(src[i]), x2 = Dt<TM>::to_f32(src[i + half]);
    const bool ret = pattern != nullptr && is_q && (i | b) == 0;
    const uint8_t keep = ret ? pattern[head / n_rep * pt_s] : 0;              // in flight with the rest
    float a = x1, c = x2;
    if (!is_v) {
        const float c1 = Dt<TM>::to_f32(cosv[b * c_sb + i]), c2 = Dt<TM>::to_f32(cosv[b * c_sb + i + half]);
        const float s1 = Dt<TM>::to_f32(sinv[b * s_sb + i]), s2 = Dt<TM>::to_f32(sinv[b * s_sb + i + half]);
        a = Dt<TM>::rn(__fadd_rn(Dt<TM>::rn(__fmul_rn(x1, c1)), Dt<TM>::rn(__fmul_rn(-x2, s1))));
        c = Dt<TM>::rn(__fadd_rn(Dt<TM>::rn(__fmul_rn(x2, c2)), Dt<TM>::rn(__fmul_rn(x1, s2))));
    }
    dst[i] = from_f32<TC>(a);
    dst[i + half] = from_f32<TC>(c);
    if (ret) ret_out[head] = keep ? retention : 0.0f;
}

template <typename TM, typename TC>
static void launch_rope_qkv(const void* q, int64_t q_sb, const void* k, int64_t k_sb, const void* v, int64_t v_sb, const void* c, int64_t c_sb,
                            const void* s, int64_t s_sb, int B, int Hq, int Hkv, int D, void* qo, void* ko, void* vo,
                            const uint8_t* pattern, int64_t pt_s, float retention, float* ret_out, cudaStream_t st) {
    launch_k(PDL_QUANT, rope_qkv_kernel<TM, TC>, dim3((unsigned)(Hq + 2 * Hkv), (unsigned)B), dim3(64), 0, st,
             static_cast<const TM*>(q), q_sb, static_cast<const TM*>(k), k_sb, static_cast<const TM*>(v), v_sb,
             static_cast<const TM*>(c), c_sb, static_cast<const TM*>(s), s_sb, Hq, Hkv, D,
             static_cast<TC*>(qo), static_cast<TC*>(ko), static_cast<TC*>(vo), pattern, pt_s, Hq / Hkv, retention, ret_out);
}

}  // namespace fq

extern "C" int fq_rope_qkv(const void* q, int64_t q_sb, const void* k, int64_t k_sb, const void* v, int64_t v_sb, int dtype,
                           const void* cosv, int64_t cos_sb, const void* sinv, int64_t sin_sb, int B, int Hq, int Hkv, int D,
                           void* q_out, void* k_out, void* v_out, int out_dtype, void* stream) {
    return fq_rope_qkv_pattern(q, q_sb, k, k_sb, v, v_sb, dtype, cosv, cos_sb, sinv, sin_sb, B, Hq, Hkv, D, q_out, k_out, v_out, out_dtype,
                               nullptr, 0, 0.0f, nullptr, stream);
}

extern "C" int fq_rope_qkv_pattern(const void* q, int64_t q_sb, const void* k, int64_t k_sb, const void* v, int64_t v_sb, int dtype,
                                   const void* cosv, int64_t cos_sb, const void* sinv, int64_t sin_sb, int B, int Hq, int Hkv, int D,
                                   void* q_out, void* k_out, void* v_out, int out_dtype,
                                   const uint8_t* pattern, int64_t pattern_stride, float retention, float* retention_per_head, void* stream) {
    using namespace fq;
    const char* fn = "fq_rope_qkv";
    FQ_CHECK_ARG(!pattern || (retention_per_head && Hkv > 0 && Hq % Hkv == 0), FQ_ERR_ARG, "%s: a head pattern needs H_q a multiple of H_kv and an output", fn);
    FQ_CHECK_ARG(q && k && v && cosv && sinv && q_out && k_out && v_out, FQ_ERR_ARG, "%s: null pointer", fn);
    FQ_CHECK_ARG(B > 0 && Hq > 0 && Hkv > 0 && D > 0 && D % 2 == 0 && D <= 128 && B <= 65535, FQ_ERR_ARG, "%s: bad sizes", fn);
    FQ_CHECK_ARG((dtype == FQ_F16 || dtype == FQ_BF16) && (out_dtype == FQ_F16 || out_dtype == FQ_BF16), FQ_ERR_DTYPE, "%s: fp16 or bf16 only", fn);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    using hf = __half; using bf = __nv_bfloat16;
    auto go = dtype == FQ_F16 ? (out_dtype == FQ_F16 ? launch_rope_qkv<hf, hf> : launch_rope_qkv<hf, bf>)
                              : (out_dtype == FQ_F16 ? launch_rope_qkv<bf, hf> : launch_rope_qkv<bf, bf>);
    go(q, q_sb, k, k_sb, v, v_sb, cosv, cos_sb, sinv, sin_sb, B, Hq, Hkv, D, q_out, k_out, v_out, pattern, pattern_stride, retention, retention_per_head, st);
    FQ_CHECK_LAUNCH(fn);
    return FQ_OK;
}

// Append to an INT8 cache (code rows of D bytes in the fq_int4_cache record), one launch.
extern "C" int fq_append_kv_int8(const fq_int4_cache* c, int layer, int seen, const void* K_new, const void* V_new,
                                 int64_t nw_sb, int64_t nw_sh, int64_t nw_ss, int n_new, void* stream) {
    using namespace fq;
    const char* fn = "fq_append_kv_int8";
    FQ_CHECK_ARG(c && K_new && V_new, FQ_ERR_ARG, "%s: null pointer", fn);
    FQ_CHECK_ARG(layer >= 0 && layer < c->L, FQ_ERR_ARG, "%s: layer_idx %d out of range [0, %d)", fn, layer, c->L);
    FQ_CHECK_ARG(seen >= 0 && n_new > 0 && seen + n_new <= c->max_seq_len, FQ_ERR_ARG, "%s: seen+new=%d exceeds max_seq_len=%d", fn, seen + n_new, c->max_seq_len);
    const int page = c->page, partial = seen % page, tok0 = seen - partial;
    QuantPagesParams f{};
    char* Kt = static_cast<char*>(c->K_partial) + layer * c->pt_sl * 2;
    char* Vt = static_cast<char*>(c->V_partial) + layer * c->pt_sl * 2;
    f.K_head = Kt; f.V_head = Vt; f.hd_sb = c->pt_sb; f.hd_sh = c->pt_sh; f.hd_ss = c->pt_ss; f.n_head = partial;
    f.K_new = K_new; f.V_new = V_new; f.nw_sb = nw_sb; f.nw_sh = nw_sh; f.nw_ss = nw_ss; f.n_new = n_new;
    f.n_quant = (partial + n_new) / page * page; f.B = c->B; f.H = c->Hkv; f.D = c->D; f.page = page; f.bits = 8;
    f.K_codes = c->K_packed + layer * c->pk_sl + (int64_t)tok0 * c->pk_ss; f.V_codes = c->V_packed + layer * c->pk_sl + (int64_t)tok0 * c->pk_ss;
    f.cd_sb = c->pk_sb; f.cd_sh = c->pk_sh; f.cd_ss = c->pk_ss;
    f.K_scale = static_cast<uint16_t*>(c->K_scale) + layer * c->km_sl + (int64_t)(tok0 / page) * c->km_sp;
    f.K_mn = static_cast<uint16_t*>(c->K_mn) + layer * c->km_sl + (int64_t)(tok0 / page) * c->km_sp;
    f.km_sb = c->km_sb; f.km_sh = c->km_sh; f.km_sp = c->km_sp;
    f.V_scale = static_cast<uint16_t*>(c->V_scale) + layer * c->vm_sl + tok0; f.V_mn = static_cast<uint16_t*>(c->V_mn) + layer * c->vm_sl + tok0;
    f.vm_sb = c->vm_sb; f.vm_sh = c->vm_sh; f.vm_ss = 1;
    f.stage_K = Kt; f.stage_V = Vt; f.st_sb = c->pt_sb; f.st_sh = c->pt_sh; f.st_ss = c->pt_ss;
    f.zero_rest = f.n_quant > 0;
    FQ_CHECK_ARG(quant_pages_supported(f, c->kv_dtype), FQ_ERR_UNSUPPORTED,
                 "%s: takes 16-bit rows, head_dim 64 or 128, page 16, 32 or 64 and 16-byte aligned rows", fn);
    return quant_pages_launch(f, c->kv_dtype, stream, fn);
}

extern "C" int fq_decode_layer_int8(
    const fq_int4_cache* c, int layer, int seen,
    const void* K_new, const void* V_new, int64_t nw_sb, int64_t nw_sh, int64_t nw_ss, int n_new,
    const void* Q, int q_dtype, int64_t q_sb, int64_t q_sh, const fq_decode_params* prm,
    float* scores, int32_t* compact, void* O, float* lse, void* workspace, size_t workspace_bytes, void* stream) {
    using namespace fq;
    const char* fn = "fq_decode_layer_int8";
    FQ_CHECK_ARG(c && prm, FQ_ERR_ARG, "%s: null descriptor", fn);
    FQ_CHECK_ARG(layer >= 0 && layer < c->L, FQ_ERR_ARG, "%s: layer_idx %d out of range [0, %d)", fn, layer, c->L);
    const int page = c->page, D = c->D, B = c->B, Hkv = c->Hkv, Hq = prm->Hq;
    int rc;
    const int now = seen + n_new, tail = now % page, completed = now - tail, P = completed / page;
    char* Kt = static_cast<char*>(c->K_partial) + layer * c->pt_sl * 2;
    char* Vt = static_cast<char*>(c->V_partial) + layer * c->pt_sl * 2;
    // tokens that complete no page are staged in the launch of the scores
    QuantParams staged;
    const bool along = seen >= 0 && now <= c->max_seq_len && (page == 16 || page == 32 || page == 64) && page_scores_take_append(q_dtype, B, Hq, Hkv, P, D) &&
                       append_stage_params(staged, Kt, Vt, c->pt_sb, c->pt_sh, c->pt_ss, K_new, V_new, nw_sb, nw_sh, nw_ss, c->kv_dtype, B, Hkv, D, page, seen, n_new);
    if (n_new > 0 && !along) {
        rc = fq_append_kv_int8(c, layer, seen, K_new, V_new, nw_sb, nw_sh, nw_ss, n_new, stream);
        if (rc != FQ_OK) return rc;
    }
    const uint16_t* Ks = static_cast<const uint16_t*>(c->K_scale) + layer * c->km_sl;
    const uint16_t* Km = static_cast<const uint16_t*>(c->K_mn) + layer * c->km_sl;
    if (P > 0) {
        rc = page_scores_int4_launch(Q, q_dtype, q_sb, q_sh, Ks, Km, c->km_sb, c->km_sh, c->km_sp, B, Hq, Hkv, P, D, scores, (int64_t)Hq * P, P, stream,
                                     DynPos{}, 255.0f, along ? &staged : nullptr, c->kv_dtype);
        if (rc != FQ_OK) return rc;
        rc = fq_select_pages(scores, (int64_t)Hq * P, P, B, Hq, P, prm->retention_per_head, prm->retention,
                             prm->k_max_static < P ? prm->k_max_static : P, prm->sinks, prm->window, nullptr, 0, 0,
                             compact, (int64_t)Hq * prm->bucket, prm->bucket, prm->bucket, nullptr, stream);
        if (rc != FQ_OK) return rc;
    }
    return fq_sparse_decode_int8(
        Q, q_dtype, q_sb, q_sh, c->K_packed + layer * c->pk_sl, c->V_packed + layer * c->pk_sl, c->pk_sb, c->pk_sh, c->pk_ss,
        Ks, Km, c->km_sb, c->km_sh, c->km_sp, static_cast<const uint16_t*>(c->V_scale) + layer * c->vm_sl,
        static_cast<const uint16_t*>(c->V_mn) + layer * c->vm_sl, c->vm_sb, c->vm_sh,
        compact, (int64_t)Hq * prm->bucket, prm->bucket, P > 0 ? prm->bucket : 0,
        tail ? Kt : nullptr, tail ? Vt : nullptr, c->kv_dtype, c->pt_sb, c->pt_sh, c->pt_ss, tail,
        B, Hq, Hkv, completed, P, D, page, prm->sm_scale, O, lse, workspace, workspace_bytes, prm->n_split, stream);
}
