// INT4 KV quantisation on append, and the inverse used by prefill.
//
// One warp owns one page of one (batch, kv head).  A lane owns 8 consecutive channels
// (one 16-byte load per token); D/8 lanes cover a token, so a warp reads 32/(D/8) tokens
// per load instruction, fully coalesced.  K needs the page's per-channel min/max before any
// code can be produced, so the page is read twice (the second read is served by L1/L2);
// V is per token and needs one read.  HBM traffic per page: 2*page*D*sizeof(T) in,
// page*D (codes) + 2*D*2 (K metadata) + page*4 (V metadata) out.
#include "fq_append.cuh"
#include "fq_quant_pages.cuh"

namespace fq {

template <typename T>
__global__ void __launch_bounds__(128) quant_int4_kernel(QuantParams p) {
    int b = blockIdx.z;
    if (p.n_layers > 1) {              // one launch appends to every layer
        const int layer = b / p.B;
        b -= layer * p.B;
        p.pos += layer;
        p.K_head = static_cast<const T*>(p.K_head) + layer * p.hd_sl; p.V_head = static_cast<const T*>(p.V_head) + layer * p.hd_sl;
        p.K_new = static_cast<const T*>(p.K_new) + layer * p.nw_sl;   p.V_new = static_cast<const T*>(p.V_new) + layer * p.nw_sl;
        p.K_packed += layer * p.pk_sl; p.V_packed += layer * p.pk_sl;
        p.K_scale += layer * p.km_sl;  p.K_mn += layer * p.km_sl;
        p.V_scale += layer * p.vm_sl;  p.V_mn += layer * p.vm_sl;
        p.stage_K = static_cast<T*>(p.stage_K) + layer * p.st_sl;     p.stage_V = static_cast<T*>(p.stage_V) + layer * p.st_sl;
    }
    pdl_wait();        // inputs and the staging rows may come from the previous kernel
    pdl_trigger();
    if (p.pos && !quant_locate(p)) return;                          // full: nothing is written (the host checks its own count)
    quant_int4_cta<T>(p, b, blockIdx.y, blockIdx.x);
}

// out = bf16(code * scale + mn); one thread per 8 output elements.
__global__ void __launch_bounds__(256) dequant_int4_kernel(
    const uint8_t* packed, int64_t pk_sb, int64_t pk_sh, int64_t pk_ss,
    const uint16_t* scale, const uint16_t* mn, int64_t m_sb, int64_t m_sh, int64_t m_s2,
    int per_page, int B, int H, int S, int D, int page,
    uint16_t* out, int64_t o_sb, int64_t o_sh, int64_t o_ss) {
    const int chunks = D >> 3;
    const int64_t total = (int64_t)B * H * S * chunks;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int c = (int)(i % chunks);
        int64_t r = i / chunks;
        const int t = (int)(r % S);
        r /= S;
        const int h = (int)(r % H), b = (int)(r / H);
        const uint32_t w = *reinterpret_cast<const uint32_t*>(packed + b * pk_sb + h * pk_sh + (int64_t)t * pk_ss + 4 * c);
        float sc[8], m[8];
        if (per_page) {
            const int64_t mo = b * m_sb + h * m_sh + (int64_t)(t / page) * m_s2 + 8 * c;
            const uint4 s4 = *reinterpret_cast<const uint4*>(scale + mo);
            const uint4 m4 = *reinterpret_cast<const uint4*>(mn + mo);
            const uint32_t sa[4] = {s4.x, s4.y, s4.z, s4.w}, ma[4] = {m4.x, m4.y, m4.z, m4.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                sc[2 * k] = bf16_lo(sa[k]); sc[2 * k + 1] = bf16_hi(sa[k]);
                m[2 * k] = bf16_lo(ma[k]); m[2 * k + 1] = bf16_hi(ma[k]);
            }
        } else {
            const int64_t mo = b * m_sb + h * m_sh + (int64_t)t * m_s2;
            const float s0 = bf16_lo(scale[mo]), m0 = bf16_lo(mn[mo]);
#pragma unroll
            for (int k = 0; k < 8; ++k) { sc[k] = s0; m[k] = m0; }
        }
        uint32_t o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float a = __fadd_rn(__fmul_rn((float)((w >> (8 * k)) & 15u), sc[2 * k]), m[2 * k]);
            float bb = __fadd_rn(__fmul_rn((float)((w >> (8 * k + 4)) & 15u), sc[2 * k + 1]), m[2 * k + 1]);
            o[k] = f32_to_bf16_bits(a) | ((uint32_t)f32_to_bf16_bits(bb) << 16);
        }
        *reinterpret_cast<uint4*>(out + b * o_sb + h * o_sh + (int64_t)t * o_ss + 8 * c) =
            make_uint4(o[0], o[1], o[2], o[3]);
    }
}

}  // namespace fq

namespace fq {
int quantize_kv_int4_launch(
    const void* K_head, const void* V_head, int64_t hd_sb, int64_t hd_sh, int64_t hd_ss, int n_head,
    const void* K_new, const void* V_new, int64_t nw_sb, int64_t nw_sh, int64_t nw_ss, int n_new,
    int dtype, int B, int H, int D, int page, int n_quant,
    uint8_t* K_packed, uint8_t* V_packed, int64_t pk_sb, int64_t pk_sh, int64_t pk_ss,
    void* K_scale, void* K_mn, int64_t km_sb, int64_t km_sh, int64_t km_sp,
    void* V_scale, void* V_mn, int64_t vm_sb, int64_t vm_sh, int64_t vm_ss,
    void* stage_K, void* stage_V, int64_t st_sb, int64_t st_sh, int64_t st_ss,
    void* stream, const DynPos& dp) {
    using namespace fq;
    const char* fn = "fq_quantize_kv_int4";
    FQ_CHECK_ARG(B > 0 && H > 0 && page > 0 && n_head >= 0 && n_new >= 0 && n_quant >= 0, FQ_ERR_ARG,
                 "%s: bad sizes B=%d H=%d page=%d n_head=%d n_new=%d n_quant=%d", fn, B, H, page, n_head, n_new, n_quant);
    FQ_CHECK_ARG(D % 2 == 0, FQ_ERR_ARG, "%s: requires even head_dim; got %d", fn, D);
    FQ_CHECK_ARG(D >= 8 && D <= 256 && (D & (D - 1)) == 0, FQ_ERR_UNSUPPORTED,
                 "%s: head_dim %d not in {8,16,32,64,128,256}", fn, D);
    FQ_CHECK_ARG(n_quant <= n_head + n_new, FQ_ERR_ARG, "%s: n_quant %d exceeds the stream length %d", fn, n_quant, n_head + n_new);
    FQ_CHECK_ARG(n_head == 0 || n_quant == 0 || n_head < page, FQ_ERR_ARG,
                 "%s: a staged head (%d tokens) must be shorter than a page (%d)", fn, n_head, page);
    FQ_CHECK_ARG(dtype == FQ_F32 || dtype == FQ_F16 || dtype == FQ_BF16, FQ_ERR_DTYPE, "%s: dtype code %d", fn, dtype);
    const bool doK = K_packed != nullptr || K_scale != nullptr, doV = V_packed != nullptr;
    if (n_quant > 0) {
        FQ_CHECK_ARG(doK || doV, FQ_ERR_ARG, "%s: neither K nor V outputs given", fn);
        FQ_CHECK_ARG(!doK || (K_scale && K_mn && (K_new || n_new == 0)), FQ_ERR_ARG, "%s: K outputs/inputs missing", fn);
        FQ_CHECK_ARG(!doV || (V_scale && V_mn && (V_new || n_new == 0)), FQ_ERR_ARG, "%s: V outputs/inputs missing", fn);
    }
    const size_t esz = dtype == FQ_F32 ? 4 : 2;
    const size_t row_align = 16 / esz;  // elements per 16 bytes
    FQ_CHECK_ARG(hd_sb % row_align == 0 && hd_sh % row_align == 0 && hd_ss % row_align == 0 &&
                 nw_sb % row_align == 0 && nw_sh % row_align == 0 && nw_ss % row_align == 0 &&
                 st_sb % row_align == 0 && st_sh % row_align == 0 && st_ss % row_align == 0,
                 FQ_ERR_ALIGN, "%s: input/staging strides must keep rows 16-byte aligned", fn);
    FQ_CHECK_ARG(aligned(K_head, 16) && aligned(V_head, 16) && aligned(K_new, 16) && aligned(V_new, 16) &&
                 aligned(stage_K, 16) && aligned(stage_V, 16), FQ_ERR_ALIGN, "%s: input pointers must be 16-byte aligned", fn);
    FQ_CHECK_ARG(pk_sb % 4 == 0 && pk_sh % 4 == 0 && pk_ss % 4 == 0 && aligned(K_packed, 4) && aligned(V_packed, 4),
                 FQ_ERR_ALIGN, "%s: packed rows must be 4-byte aligned", fn);
    FQ_CHECK_ARG(km_sb % 8 == 0 && km_sh % 8 == 0 && km_sp % 8 == 0 && aligned(K_scale, 16) && aligned(K_mn, 16),
                 FQ_ERR_ALIGN, "%s: K metadata rows must be 16-byte aligned", fn);

    // whole pages of a prompt: the register-resident kernel.  The general one below takes ragged last pages, other
    // page sizes, head dimensions and fp32, appends that complete no page, and positions read on the device.
    if (dp.pos == nullptr && n_quant > 0) {
        QuantPagesParams f{};
        f.K_head = K_head; f.V_head = V_head; f.K_new = K_new; f.V_new = V_new;
        f.hd_sb = hd_sb; f.hd_sh = hd_sh; f.hd_ss = hd_ss; f.nw_sb = nw_sb; f.nw_sh = nw_sh; f.nw_ss = nw_ss;
        f.n_head = n_head; f.n_new = n_new; f.n_quant = n_quant; f.B = B; f.H = H; f.D = D; f.page = page; f.bits = 4;
        f.K_codes = K_packed; f.V_codes = V_packed; f.cd_sb = pk_sb; f.cd_sh = pk_sh; f.cd_ss = pk_ss;
        f.K_scale = static_cast<uint16_t*>(K_scale); f.K_mn = static_cast<uint16_t*>(K_mn); f.km_sb = km_sb; f.km_sh = km_sh; f.km_sp = km_sp;
        f.V_scale = static_cast<uint16_t*>(V_scale); f.V_mn = static_cast<uint16_t*>(V_mn); f.vm_sb = vm_sb; f.vm_sh = vm_sh; f.vm_ss = vm_ss;
        f.stage_K = stage_K; f.stage_V = stage_V; f.st_sb = st_sb; f.st_sh = st_sh; f.st_ss = st_ss;
        if (quant_pages_supported(f, dtype)) return quant_pages_launch(f, dtype, stream, fn);
    }
    QuantParams p;
    p.K_head = K_head; p.V_head = V_head; p.K_new = K_new; p.V_new = V_new;
    p.hd_sb = hd_sb; p.hd_sh = hd_sh; p.hd_ss = hd_ss; p.nw_sb = nw_sb; p.nw_sh = nw_sh; p.nw_ss = nw_ss;
    p.n_head = n_head; p.n_new = n_new;
    p.B = B; p.H = H; p.D = D; p.page = page; p.n_quant = n_quant;
    p.n_pages = (n_quant + page - 1) / page;
    p.K_packed = K_packed; p.V_packed = V_packed; p.pk_sb = pk_sb; p.pk_sh = pk_sh; p.pk_ss = pk_ss;
    p.K_scale = static_cast<uint16_t*>(K_scale); p.K_mn = static_cast<uint16_t*>(K_mn);
    p.km_sb = km_sb; p.km_sh = km_sh; p.km_sp = km_sp;
    p.V_scale = static_cast<uint16_t*>(V_scale); p.V_mn = static_cast<uint16_t*>(V_mn);
    p.vm_sb = vm_sb; p.vm_sh = vm_sh; p.vm_ss = vm_ss;
    p.stage_K = stage_K; p.stage_V = stage_V; p.st_sb = st_sb; p.st_sh = st_sh; p.st_ss = st_ss;
    p.pos = dp.pos; p.max_tokens = dp.pos ? dp.max_tokens : 0x7fffffff;
    p.n_layers = 1; p.hd_sl = p.nw_sl = p.pk_sl = p.km_sl = p.vm_sl = p.st_sl = 0;
    if (p.pos == nullptr && n_quant == 0 && (n_head + n_new == 0 || (!stage_K && !stage_V))) return FQ_OK;

    dim3 grid((unsigned)max(1, (p.n_pages + 3) / 4), (unsigned)H, (unsigned)B);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (dtype == FQ_F32) launch_k(PDL_QUANT, quant_int4_kernel<float>, grid, dim3(128), 0, st, p);
    else if (dtype == FQ_F16) launch_k(PDL_QUANT, quant_int4_kernel<__half>, grid, dim3(128), 0, st, p);
    else launch_k(PDL_QUANT, quant_int4_kernel<__nv_bfloat16>, grid, dim3(128), 0, st, p);
    FQ_CHECK_LAUNCH(fn);
    return FQ_OK;
}

}  // namespace fq

extern "C" int fq_quantize_kv_int4(
    const void* K_head, const void* V_head, int64_t hd_sb, int64_t hd_sh, int64_t hd_ss, int n_head,
    const void* K_new, const void* V_new, int64_t nw_sb, int64_t nw_sh, int64_t nw_ss, int n_new,
    int dtype, int B, int H, int D, int page, int n_quant,
    uint8_t* K_packed, uint8_t* V_packed, int64_t pk_sb, int64_t pk_sh, int64_t pk_ss,
    void* K_scale, void* K_mn, int64_t km_sb, int64_t km_sh, int64_t km_sp,
    void* V_scale, void* V_mn, int64_t vm_sb, int64_t vm_sh, int64_t vm_ss,
    void* stage_K, void* stage_V, int64_t st_sb, int64_t st_sh, int64_t st_ss,
    void* stream) {
    return fq::quantize_kv_int4_launch(K_head, V_head, hd_sb, hd_sh, hd_ss, n_head, K_new, V_new, nw_sb, nw_sh, nw_ss, n_new,
                                       dtype, B, H, D, page, n_quant, K_packed, V_packed, pk_sb, pk_sh, pk_ss,
                                       K_scale, K_mn, km_sb, km_sh, km_sp, V_scale, V_mn, vm_sb, vm_sh, vm_ss,
                                       stage_K, stage_V, st_sb, st_sh, st_ss, stream, fq::DynPos{});
}

namespace fq {
static bool append_aligned(const void* a, const void* b, int64_t sb, int64_t sh, int64_t ss) {
    return a && b && aligned(a, 16) && aligned(b, 16) && sb % 8 == 0 && sh % 8 == 0 && ss % 8 == 0;
}

bool append_stage_params(QuantParams& q, void* K_partial, void* V_partial, int64_t pt_sb, int64_t pt_sh, int64_t pt_ss, const void* K_new, const void* V_new,
                         int64_t nw_sb, int64_t nw_sh, int64_t nw_ss, int dtype, int B, int H, int D, int page, int seen, int n_new) {
    if (n_new < 1 || page < 1 || seen % page + n_new >= page || (dtype != FQ_F16 && dtype != FQ_BF16) || (D != 64 && D != 128)) return false;
    if (!append_aligned(K_new, V_new, nw_sb, nw_sh, nw_ss) || !append_aligned(K_partial, V_partial, pt_sb, pt_sh, pt_ss)) return false;
    q = QuantParams{};
    q.K_head = K_partial; q.V_head = V_partial; q.hd_sb = pt_sb; q.hd_sh = pt_sh; q.hd_ss = pt_ss;
    q.K_new = K_new; q.V_new = V_new; q.nw_sb = nw_sb; q.nw_sh = nw_sh; q.nw_ss = nw_ss;
    q.n_head = seen % page; q.n_new = n_new; q.B = B; q.H = H; q.D = D; q.page = page;
    q.stage_K = K_partial; q.stage_V = V_partial; q.st_sb = pt_sb; q.st_sh = pt_sh; q.st_ss = pt_ss;
    q.n_layers = 1; q.max_tokens = 0x7fffffff;
    return true;
}

bool append_dyn_params(QuantParams& q, const fq_int4_cache* c, int layer, const int* pos, const void* K_new, const void* V_new,
                       int64_t nw_sb, int64_t nw_sh, int64_t nw_ss, int n_new) {
    char* Kt = static_cast<char*>(c->K_partial) + layer * c->pt_sl * 2;
    char* Vt = static_cast<char*>(c->V_partial) + layer * c->pt_sl * 2;
    if (n_new >= c->page || !append_stage_params(q, Kt, Vt, c->pt_sb, c->pt_sh, c->pt_ss, K_new, V_new, nw_sb, nw_sh, nw_ss, c->kv_dtype, c->B, c->Hkv, c->D, c->page, 0, n_new)) return false;
    q.K_packed = c->K_packed + layer * c->pk_sl; q.V_packed = c->V_packed + layer * c->pk_sl; q.pk_sb = c->pk_sb; q.pk_sh = c->pk_sh; q.pk_ss = c->pk_ss;
    q.K_scale = static_cast<uint16_t*>(c->K_scale) + layer * c->km_sl; q.K_mn = static_cast<uint16_t*>(c->K_mn) + layer * c->km_sl;
    q.km_sb = c->km_sb; q.km_sh = c->km_sh; q.km_sp = c->km_sp;
    q.V_scale = static_cast<uint16_t*>(c->V_scale) + layer * c->vm_sl; q.V_mn = static_cast<uint16_t*>(c->V_mn) + layer * c->vm_sl;
    q.vm_sb = c->vm_sb; q.vm_sh = c->vm_sh; q.vm_ss = 1;
    q.pos = pos; q.max_tokens = c->max_seq_len;
    return c->pk_sb % 4 == 0 && c->pk_sh % 4 == 0 && c->pk_ss % 4 == 0 && aligned(q.K_packed, 4) && aligned(q.V_packed, 4) &&
           c->km_sb % 8 == 0 && c->km_sh % 8 == 0 && c->km_sp % 8 == 0 && aligned(q.K_scale, 16) && aligned(q.K_mn, 16);
}

// Append n_new tokens (1 <= n_new < page) to layers [0, n_layers) in ONE launch, positions read from pos[layer].
int quant_append_layers_dyn(const fq_int4_cache* c, int n_layers, const int* pos, const void* K_new, const void* V_new,
                            int64_t nw_sl, int64_t nw_sb, int64_t nw_sh, int64_t nw_ss, int n_new, void* stream) {
    const char* fn = "fq_decode_step_int4_dev";
    FQ_CHECK_ARG(aligned(K_new, 16) && aligned(V_new, 16) && nw_sl % 8 == 0 && nw_sb % 8 == 0 && nw_sh % 8 == 0 && nw_ss % 8 == 0,
                 FQ_ERR_ALIGN, "%s: new K/V rows must be 16-byte aligned", fn);
    QuantParams p;
    p.K_head = c->K_partial; p.V_head = c->V_partial; p.K_new = K_new; p.V_new = V_new;
    p.hd_sb = c->pt_sb; p.hd_sh = c->pt_sh; p.hd_ss = c->pt_ss; p.nw_sb = nw_sb; p.nw_sh = nw_sh; p.nw_ss = nw_ss;
    p.n_head = 0; p.n_new = n_new;
    p.B = c->B; p.H = c->Hkv; p.D = c->D; p.page = c->page; p.n_quant = 0; p.n_pages = 1;
    p.K_packed = c->K_packed; p.V_packed = c->V_packed; p.pk_sb = c->pk_sb; p.pk_sh = c->pk_sh; p.pk_ss = c->pk_ss;
    p.K_scale = static_cast<uint16_t*>(c->K_scale); p.K_mn = static_cast<uint16_t*>(c->K_mn);
    p.km_sb = c->km_sb; p.km_sh = c->km_sh; p.km_sp = c->km_sp;
    p.V_scale = static_cast<uint16_t*>(c->V_scale); p.V_mn = static_cast<uint16_t*>(c->V_mn);
    p.vm_sb = c->vm_sb; p.vm_sh = c->vm_sh; p.vm_ss = 1;
    p.stage_K = c->K_partial; p.stage_V = c->V_partial; p.st_sb = c->pt_sb; p.st_sh = c->pt_sh; p.st_ss = c->pt_ss;
    p.pos = pos; p.max_tokens = c->max_seq_len;
    p.n_layers = n_layers; p.hd_sl = c->pt_sl; p.nw_sl = nw_sl; p.pk_sl = c->pk_sl; p.km_sl = c->km_sl; p.vm_sl = c->vm_sl; p.st_sl = c->pt_sl;
    FQ_CHECK_ARG((int64_t)c->B * n_layers <= 65535, FQ_ERR_ARG, "%s: batch x layers = %lld too large for one launch", fn, (long long)c->B * n_layers);
    dim3 grid(1u, (unsigned)c->Hkv, (unsigned)(c->B * n_layers));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (c->kv_dtype == FQ_F16) launch_k(PDL_QUANT, quant_int4_kernel<__half>, grid, dim3(128), 0, st, p);
    else launch_k(PDL_QUANT, quant_int4_kernel<__nv_bfloat16>, grid, dim3(128), 0, st, p);
    FQ_CHECK_LAUNCH(fn);
    return FQ_OK;
}
}  // namespace fq

extern "C" int fq_dequantize_int4(
    const uint8_t* packed, int64_t pk_sb, int64_t pk_sh, int64_t pk_ss,
    const void* scale, const void* mn, int64_t m_sb, int64_t m_sh, int64_t m_s2,
    int per_page, int B, int H, int S, int D, int page,
    void* out, int64_t o_sb, int64_t o_sh, int64_t o_ss, void* stream) {
    using namespace fq;
    const char* fn = "fq_dequantize_int4";
    FQ_CHECK_ARG(B > 0 && H > 0 && S >= 0 && page > 0, FQ_ERR_ARG, "%s: bad sizes", fn);
    FQ_CHECK_ARG(D >= 8 && D % 8 == 0, FQ_ERR_UNSUPPORTED, "%s: head_dim %d must be a multiple of 8", fn, D);
    FQ_CHECK_ARG(packed && scale && mn && out, FQ_ERR_ARG, "%s: null pointer", fn);
    FQ_CHECK_ARG(pk_sb % 4 == 0 && pk_sh % 4 == 0 && pk_ss % 4 == 0 && aligned(packed, 4), FQ_ERR_ALIGN, "%s: packed rows must be 4-byte aligned", fn);
    FQ_CHECK_ARG(o_sb % 8 == 0 && o_sh % 8 == 0 && o_ss % 8 == 0 && aligned(out, 16), FQ_ERR_ALIGN, "%s: output rows must be 16-byte aligned", fn);
    if (per_page)
        FQ_CHECK_ARG(m_sb % 8 == 0 && m_sh % 8 == 0 && m_s2 % 8 == 0 && aligned(scale, 16) && aligned(mn, 16), FQ_ERR_ALIGN,
                     "%s: K metadata rows must be 16-byte aligned", fn);
    if (S == 0) return FQ_OK;
    const int64_t total = (int64_t)B * H * S * (D / 8);
    const int64_t want = (total + 255) / 256;
    const int blocks = (int)(want < 148 * 16 ? want : 148 * 16);
    count_launch();
    dequant_int4_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        packed, pk_sb, pk_sh, pk_ss, static_cast<const uint16_t*>(scale), static_cast<const uint16_t*>(mn),
        m_sb, m_sh, m_s2, per_page, B, H, S, D, page, static_cast<uint16_t*>(out), o_sb, o_sh, o_ss);
    FQ_CHECK_LAUNCH(fn);
    return FQ_OK;
}
