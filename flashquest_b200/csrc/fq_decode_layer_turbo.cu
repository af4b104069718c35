// Host-side chaining of one decode step of one layer on a persistent TurboQuant (K3-V3) cache:
// pack-on-append, page scores from the raw
// metadata, top-k + compact index, rotation of Q, sparse attention over the selected planes in
// the rotated basis, rotation of O back, tail attention over the staged tokens and the LSE merge.
// No device code of its own: it exists so that a caller pays one foreign call per layer.
#include "fq_append.cuh"

extern "C" size_t fq_decode_layer_turbo_scratch_bytes(int B, int Hq, int D) {
    if (B <= 0 || Hq <= 0 || D <= 0) return 0;
    const size_t rows = (size_t)B * Hq;
    return ((rows * D * 2 + 255) & ~(size_t)255) + rows * 4;     // O in the rotated basis (16-bit) | lse of its part
}

extern "C" int fq_decode_layer_turbo(
    const fq_turbo_cache* c, int layer, int seen,
    const void* K_new, const void* V_new, int64_t nw_sb, int64_t nw_sh, int64_t nw_ss, int n_new,
    const void* Q, int q_dtype, int64_t q_sb, int64_t q_sh,
    const fq_decode_params* prm,
    float* scores, int32_t* compact, void* scratch, size_t scratch_bytes, void* O, float* lse,
    void* workspace, size_t workspace_bytes, void* stream) {
    using namespace fq;
    const char* fn = "fq_decode_layer_turbo";
    FQ_CHECK_ARG(c && prm, FQ_ERR_ARG, "%s: null descriptor", fn);
    FQ_CHECK_ARG(layer >= 0 && layer < c->L, FQ_ERR_ARG, "%s: layer_idx %d out of range [0, %d)", fn, layer, c->L);
    FQ_CHECK_ARG(seen >= 0 && n_new >= 0 && seen + n_new <= c->max_seq_len, FQ_ERR_ARG,
                 "%s: seen+new=%d exceeds max_seq_len=%d", fn, seen + n_new, c->max_seq_len);
    FQ_CHECK_ARG(c->kv_dtype == FQ_F16 || c->kv_dtype == FQ_BF16, FQ_ERR_DTYPE, "%s: cache dtype code %d", fn, c->kv_dtype);
    FQ_CHECK_ARG(q_dtype == FQ_F16 || q_dtype == FQ_BF16, FQ_ERR_DTYPE, "%s: Q must be fp16 or bf16 (code %d)", fn, q_dtype);
    const int page = c->page, D = c->D, B = c->B, Hkv = c->Hkv, Hq = prm->Hq;
    FQ_CHECK_ARG(Q && O && scratch && scratch_bytes >= fq_decode_layer_turbo_scratch_bytes(B, Hq, D), FQ_ERR_WORKSPACE,
                 "%s: scratch of %zu B needed, %zu given", fn, fq_decode_layer_turbo_scratch_bytes(B, Hq, D), scratch_bytes);
    FQ_CHECK_ARG(q_sh == D && q_sb == (int64_t)Hq * D, FQ_ERR_ARG, "%s: Q must be dense (B,H_q,D)", fn);
    const size_t esz = 2;
    uint8_t* Kms = c->K_msb + layer * c->ms_sl; uint8_t* Kls = c->K_lsb + layer * c->ls_sl;
    uint8_t* Vms = c->V_msb + layer * c->ms_sl; uint8_t* Vls = c->V_lsb + layer * c->ls_sl;
    uint16_t* Kst = static_cast<uint16_t*>(c->K_scale_turbo) + layer * c->st_sl;
    uint16_t* Vst = static_cast<uint16_t*>(c->V_scale_turbo) + layer * c->st_sl;
    uint16_t* Ksr = static_cast<uint16_t*>(c->K_scale_raw) + layer * c->km_sl;
    uint16_t* Kmr = static_cast<uint16_t*>(c->K_mn_raw) + layer * c->km_sl;
    char* Kt = static_cast<char*>(c->K_partial) + layer * c->pt_sl * esz;
    char* Vt = static_cast<char*>(c->V_partial) + layer * c->pt_sl * esz;
    int rc;
    const int now = seen + n_new;
    const int tail = now % page;
    const int completed = now - tail;
    const int P = completed / page;
    // tokens that complete no page are staged in the launch of the scores
    QuantParams staged;
    const bool along = page_scores_take_append(q_dtype, B, Hq, Hkv, P, D) &&
                       append_stage_params(staged, Kt, Vt, c->pt_sb, c->pt_sh, c->pt_ss, K_new, V_new, nw_sb, nw_sh, nw_ss, c->kv_dtype, B, Hkv, D, page, seen, n_new);
    if (n_new > 0 && !along) {
        rc = fq_append_kv_turbo(c, layer, seen, K_new, V_new, nw_sb, nw_sh, nw_ss, n_new, stream);
        if (rc != FQ_OK) return rc;
    }
    const int64_t rows = (int64_t)B * Hq;
    char* sb = static_cast<char*>(scratch);
    void* O_rot = sb;
    float* lse_rot = reinterpret_cast<float*>(sb + ((rows * D * 2 + 255) & ~(int64_t)255));
    const bool sparse = P > 0, both = sparse && tail > 0;
    if (sparse) {
        rc = page_scores_int4_launch(Q, q_dtype, q_sb, q_sh, Ksr, Kmr, c->km_sb, c->km_sh, c->km_sp, B, Hq, Hkv, P, D, scores, (int64_t)Hq * P, P, stream,
                                     DynPos{}, 15.0f, along ? &staged : nullptr, c->kv_dtype);
        if (rc != FQ_OK) return rc;
        const int k_max = prm->k_max_static < P ? prm->k_max_static : P;
        rc = fq_select_pages(scores, (int64_t)Hq * P, P, B, Hq, P, prm->retention_per_head, prm->retention, k_max, prm->sinks, prm->window,
                             nullptr, 0, 0, compact, (int64_t)Hq * prm->bucket, prm->bucket, prm->bucket, nullptr, stream);
        if (rc != FQ_OK) return rc;
        int n_split = prm->n_split > 0 ? prm->n_split : fq_sparse_decode_default_splits(B, Hq, prm->bucket, page);
        if (n_split > 64) n_split = 64;
        // Q is rotated by the attention's own CTAs
        rc = sparse_decode_turbo_launch(Q, q_dtype, (int64_t)Hq * D, D,
                                    Kms, c->ms_sb, c->ms_sh, c->ms_ss, Kls, c->ls_sb, c->ls_sh, c->ls_ss, Kst, c->st_sb, c->st_sh,
                                    Vms, c->ms_sb, c->ms_sh, c->ms_ss, Vls, c->ls_sb, c->ls_sh, c->ls_ss, Vst, c->st_sb, c->st_sh,
                                    compact, (int64_t)Hq * prm->bucket, prm->bucket, prm->bucket,
                                    B, Hq, Hkv, completed, P, D, page, prm->sm_scale,
                                    O_rot, (int64_t)Hq * D, D, both ? lse_rot : lse, workspace, workspace_bytes, n_split, stream, true);
        if (rc != FQ_OK) return rc;
        if (both)
            return turbo_finish_launch(O_rot, lse_rot, Q, q_dtype, Kt, Vt, c->kv_dtype, c->pt_sb, c->pt_sh, c->pt_ss, tail, B, Hq, Hkv, D, prm->sm_scale, O, lse, stream);
        return fq_wht(O_rot, O, q_dtype, rows, D, stream);
    }
    // no page yet: dense attention over the staged tokens, the tail-only case of the INT4 kernel
    return fq_sparse_decode_int4(Q, q_dtype, q_sb, q_sh, nullptr, 0, 0, nullptr, nullptr, 0, 0, 0, nullptr, 0, 0, nullptr, nullptr, 0, 0,
                                 nullptr, 0, 0, 0, tail ? Kt : nullptr, tail ? Vt : nullptr, c->kv_dtype, c->pt_sb, c->pt_sh, c->pt_ss, tail,
                                 B, Hq, Hkv, 0, 0, D, page < 16 ? 16 : page, prm->sm_scale, O, (int64_t)Hq * D, D, lse, nullptr, 0, 1, stream);
}
