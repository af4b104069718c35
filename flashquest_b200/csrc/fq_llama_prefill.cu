// Prefill of one prompt through a Llama-shaped model in ONE foreign call (the S_q > 1 branch of
// flashquest/eager/llama_persistent_patch.py:196-201 inside Hugging Face's layer loop).  The loop issued from Python cost
// about 360 us of host time per layer, which bounded every prompt below roughly 1500 tokens (10 ms whatever its length);
// here it is ten launches per layer.
//
// K and V of the attention are the bf16-rounded dequantised values of the completed pages followed by the staged tail:
// one kernel writes both tensors from the cache in the attention's dtype, instead of a dequantise, a cast and a
// concatenation for each.  After the last layer's attention only the last token is carried on: nothing else of the
// block's output is read by anybody.
#include "fq_common.cuh"

namespace fq {

// (H_kv, S, D) fp16 K and V of one layer from the INT4 pages [0, done) and the staged rows behind them.  HBM/L2-bound:
// 8 channels per thread, one 4-byte load of codes, one 16-byte store.
__global__ void __launch_bounds__(256) gather_kv_f16_kernel(const fq_int4_cache c, int layer, int S, int done, __half* __restrict__ Kf, __half* __restrict__ Vf) {
    const int ch = c.D >> 3;
    const int64_t total = (int64_t)c.Hkv * S * ch;
    const int is_v = blockIdx.y;
    pdl_wait();
    pdl_trigger();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int cc = (int)(i % ch);
        const int64_t r = i / ch;
        const int t = (int)(r % S), h = (int)(r / S);
        uint4 o;
        if (t >= done) {
            const __half* src = static_cast<const __half*>(is_v ? c.V_partial : c.K_partial) + layer * c.pt_sl + h * c.pt_sh + (int64_t)(t - done) * c.pt_ss + 8 * cc;
            o = *reinterpret_cast<const uint4*>(src);
        } else {
            const uint32_t w = *reinterpret_cast<const uint32_t*>((is_v ? c.V_packed : c.K_packed) + layer * c.pk_sl + h * c.pk_sh + (int64_t)t * c.pk_ss + 4 * cc);
            float sc[8], mn[8];
            if (is_v) {
                const int64_t mo = layer * c.vm_sl + h * c.vm_sh + t;
                const float s = bf16_lo(static_cast<const uint16_t*>(c.V_scale)[mo]), m = bf16_lo(static_cast<const uint16_t*>(c.V_mn)[mo]);
#pragma unroll
                for (int k = 0; k < 8; ++k) { sc[k] = s; mn[k] = m; }
            } else {
                const int64_t mo = layer * c.km_sl + h * c.km_sh + (int64_t)(t / c.page) * c.km_sp + 8 * cc;
                load8<__nv_bfloat16>(static_cast<const __nv_bfloat16*>(c.K_scale) + mo, sc);
                load8<__nv_bfloat16>(static_cast<const __nv_bfloat16*>(c.K_mn) + mo, mn);
            }
            uint32_t p[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float a = Dt<__nv_bfloat16>::rn(__fadd_rn(__fmul_rn((float)((w >> (8 * k)) & 15u), sc[2 * k]), mn[2 * k]));
                const float b = Dt<__nv_bfloat16>::rn(__fadd_rn(__fmul_rn((float)((w >> (8 * k + 4)) & 15u), sc[2 * k + 1]), mn[2 * k + 1]));
                const __half2 h2 = __floats2half2_rn(a, b);
                p[k] = *reinterpret_cast<const uint32_t*>(&h2);
            }
            o = make_uint4(p[0], p[1], p[2], p[3]);
        }
        *reinterpret_cast<uint4*>((is_v ? Vf : Kf) + r * c.D + 8 * cc) = o;
    }
}

// y_i = x @ W_i for up to three linears sharing x: the GEMV for up to 8 rows, the tensor-core GEMM above.  The one row behind
// the last attention of a longer prompt stays on the GEMM with groups of 256, which the GEMV is not built for.
static int linears(const fq_llama_model* m, const void* x, int rows, bool one_of_many, const fq_awq_linear* const* w, int n, void* const* y, void* stream) {
    const int32_t* qw[3]; const void* sc[3]; const int32_t* qz[3]; const void* bs[3]; int N[3];
    bool bias = false;
    for (int i = 0; i < n; ++i) {
        qw[i] = w[i]->qweight; sc[i] = w[i]->scales; qz[i] = w[i]->qzeros; bs[i] = w[i]->bias; N[i] = w[i]->N;
        bias |= bs[i] != nullptr;
    }
    if (rows <= 8 && !(one_of_many && m->group > 128)) {
        int total = 0;
        for (int i = 0; i < n; ++i) total += N[i];
        return fq_awq_gemv(x, rows, w[0]->K, m->group, n, qw, sc, qz, bias ? bs : nullptr, N, y, m->interleaved,
                           fq_awq_gemv_default_splits(w[0]->K, total, m->group), stream);
    }
    return fq_awq_gemm(x, rows, w[0]->K, m->group, n, qw, sc, qz, bias ? bs : nullptr, N, y, m->interleaved, stream);
}

static size_t up256(size_t n) { return (n + 255) & ~(size_t)255; }

struct PrefillBuffers {
    char *x0, *x1, *normed, *q, *k, *v, *Kf, *Vf, *attn, *delta, *gate, *up, *act;
    size_t bytes;
    PrefillBuffers(const fq_llama_model* m, int S, char* base) {
        const size_t n = (size_t)S, H = m->hidden, nq = (size_t)m->q_heads * m->head_dim, nkv = (size_t)m->kv_heads * m->head_dim, F = m->ffn;
        size_t at = 0;
        auto take = [&](size_t halves) { char* p = base + at; at += up256(halves * 2); return p; };
        x0 = take(n * H); x1 = take(n * H); normed = take(n * H);
        q = take(n * nq); k = take(n * nkv); v = take(n * nkv); Kf = take(n * nkv); Vf = take(n * nkv);
        attn = take(n * nq); delta = take(n * H);
        gate = take(n * F); up = take(n * F); act = take(n * F);
        bytes = at;
    }
};

}  // namespace fq

extern "C" size_t fq_llama_prefill_workspace_bytes(const fq_llama_model* m, int S) {
    if (!m || S <= 0) return 0;
    return fq::PrefillBuffers(m, S, nullptr).bytes;
}

extern "C" int fq_llama_prefill(const fq_llama_model* m, const fq_int4_cache* c, const void* x, int S, float sm_scale,
                                void* workspace, size_t workspace_bytes, void* logits, int32_t* next_id, void* stream) {
    using namespace fq;
    const char* fn = "fq_llama_prefill";
    FQ_CHECK_ARG(m && c && x && workspace && logits && next_id && m->layers, FQ_ERR_ARG, "%s: null argument", fn);
    FQ_CHECK_ARG(S >= 1 && S <= c->max_seq_len, FQ_ERR_ARG, "%s: seen+new=%d exceeds max_seq_len=%d", fn, S, c->max_seq_len);
    FQ_CHECK_ARG(c->B == 1 && m->n_layers >= 1 && m->n_layers <= c->L && m->kv_heads == c->Hkv && m->head_dim == c->D, FQ_ERR_ARG,
                 "%s: model and cache shapes differ, or more than one sequence", fn);
    FQ_CHECK_ARG(c->kv_dtype == FQ_F16, FQ_ERR_DTYPE, "%s: computes in fp16; the cache stages dtype code %d", fn, c->kv_dtype);
    FQ_CHECK_ARG(c->D % 8 == 0 && aligned(workspace, 256) && aligned(x, 16), FQ_ERR_ALIGN, "%s: workspace and x alignment", fn);
    const PrefillBuffers w(m, S, static_cast<char*>(workspace));
    FQ_CHECK_ARG(workspace_bytes >= w.bytes, FQ_ERR_WORKSPACE, "%s: workspace of %zu B needed, %zu given", fn, w.bytes, workspace_bytes);
    const int H = m->hidden, D = m->head_dim, Hq = m->q_heads, Hkv = m->kv_heads, page = c->page;
    const int nq = Hq * D, nkv = Hkv * D, done = S - S % page;
    const char* xin = static_cast<const char*>(x);      // residual stream; alternates between two buffers
    const char* delta = nullptr;                         // output of the previous block, added by the next norm
    int flip = 0, rc;
    // rows [first, first + n) of the residual stream: add the block output, normalise into w.normed
    auto add_norm = [&](const void* weight, int first, int n) -> int {
        char* out = delta ? (flip ? w.x1 : w.x0) : nullptr;
        const size_t off = (size_t)first * H * 2;
        const int r = fq_add_rmsnorm(xin + off, delta ? delta + off : nullptr, weight, m->rms_eps, n, H, out ? out + off : nullptr, w.normed, stream);
        if (out) { xin = out; flip ^= 1; }
        return r;
    };
    for (int l = 0; l < m->n_layers; ++l) {
        const fq_llama_layer& L = m->layers[l];
        FQ_CHECK_ARG(L.q.K == H && L.q.N == nq && L.k.N == nkv && L.v.N == nkv && L.o.K == nq && L.o.N == H &&
                     L.gate.N == m->ffn && L.up.N == m->ffn && L.down.K == m->ffn && L.down.N == H, FQ_ERR_ARG,
                     "%s: layer %d has unexpected projection shapes", fn, l);
        if ((rc = add_norm(L.input_norm, 0, S)) != FQ_OK) return rc;
        {
            const fq_awq_linear* ws[3] = {&L.q, &L.k, &L.v};
            void* y[3] = {w.q, w.k, w.v};
            if ((rc = linears(m, w.normed, S, false, ws, 3, y, stream)) != FQ_OK) return rc;
        }
        if ((rc = fq_rope_tokens(w.q, nq, D, Hq, w.k, nkv, D, Hkv, S, D, 0, m->rope_theta, stream)) != FQ_OK) return rc;
        uint8_t* Kp = c->K_packed + l * c->pk_sl; uint8_t* Vp = c->V_packed + l * c->pk_sl;
        uint16_t* Ks = static_cast<uint16_t*>(c->K_scale) + l * c->km_sl; uint16_t* Km = static_cast<uint16_t*>(c->K_mn) + l * c->km_sl;
        uint16_t* Vs = static_cast<uint16_t*>(c->V_scale) + l * c->vm_sl; uint16_t* Vm = static_cast<uint16_t*>(c->V_mn) + l * c->vm_sl;
        char* Kt = static_cast<char*>(c->K_partial) + l * c->pt_sl * 2; char* Vt = static_cast<char*>(c->V_partial) + l * c->pt_sl * 2;
        rc = fq_quantize_kv_int4(nullptr, nullptr, 0, 0, 0, 0, w.k, w.v, (int64_t)S * nkv, D, nkv, S, FQ_F16, 1, Hkv, D, page, done,
                                 Kp, Vp, c->pk_sb, c->pk_sh, c->pk_ss, Ks, Km, c->km_sb, c->km_sh, c->km_sp, Vs, Vm, c->vm_sb, c->vm_sh, 1,
                                 Kt, Vt, c->pt_sb, c->pt_sh, c->pt_ss, stream);
        if (rc != FQ_OK) return rc;
        {
            const int64_t n = (int64_t)Hkv * S * (D / 8), want = (n + 255) / 256;
            launch_k(PDL_QUANT, gather_kv_f16_kernel, dim3((unsigned)(want < 148 * 8 ? want : 148 * 8), 2), dim3(256), 0, static_cast<cudaStream_t>(stream),
                     *c, l, S, done, reinterpret_cast<__half*>(w.Kf), reinterpret_cast<__half*>(w.Vf));
            FQ_CHECK_LAUNCH(fn);
        }
        rc = fq_prefill_attention(w.q, (int64_t)S * nq, D, nq, w.Kf, (int64_t)S * nkv, (int64_t)S * D, D, w.Vf, (int64_t)S * nkv, (int64_t)S * D, D,
                                  FQ_F16, 1, Hq, Hkv, S, S, D, sm_scale, w.attn, (int64_t)S * nq, D, nq, stream);
        if (rc != FQ_OK) return rc;
        // behind the last attention only the last token goes on
        const int first = l + 1 == m->n_layers ? S - 1 : 0, rows = S - first;
        {
            const fq_awq_linear* ws[1] = {&L.o};
            void* y[1] = {w.delta + (size_t)first * H * 2};
            if ((rc = linears(m, w.attn + (size_t)first * nq * 2, rows, S > 8, ws, 1, y, stream)) != FQ_OK) return rc;
        }
        delta = w.delta;
        if ((rc = add_norm(L.post_norm, first, rows)) != FQ_OK) return rc;
        if (rows <= 8) {
            const fq_awq_linear* ws[2] = {&L.gate, &L.up};
            void* y[2] = {w.gate, w.up};
            if ((rc = linears(m, w.normed, rows, S > 8, ws, 2, y, stream)) != FQ_OK) return rc;
            if ((rc = fq_swiglu(w.gate, w.up, (int64_t)rows * m->ffn, w.act, stream)) != FQ_OK) return rc;
        } else {
            const int32_t* qw[2] = {L.gate.qweight, L.up.qweight}; const void* sc[2] = {L.gate.scales, L.up.scales};
            const int32_t* qz[2] = {L.gate.qzeros, L.up.qzeros}; const void* bs[2] = {L.gate.bias, L.up.bias};
            if ((rc = fq_awq_gate_up_swiglu(w.normed, rows, H, m->group, qw, sc, qz, bs, m->ffn, w.gate, w.up, w.act, m->interleaved, stream)) != FQ_OK) return rc;
        }
        {
            const fq_awq_linear* ws[1] = {&L.down};
            void* y[1] = {w.delta + (size_t)first * H * 2};
            if ((rc = linears(m, w.act, rows, S > 8, ws, 1, y, stream)) != FQ_OK) return rc;
        }
    }
    if ((rc = add_norm(m->final_norm, S - 1, 1)) != FQ_OK) return rc;
    if ((rc = fq_gemv_f16(w.normed, m->lm_head, 1, H, m->vocab, logits, stream)) != FQ_OK) return rc;
    return fq_argmax_f16(logits, 1, m->vocab, next_id, stream);
}
