// Append of tokens to an INT4 cache by the threads of one CTA: pages that fill are packed, the rest is staged.  Shared by the append
// launch (fq_quant_int4.cu) and the page scores of a decode step, which append in the same launch (fq_scores.cu).
#pragma once
#include "fq_common.cuh"

namespace fq {

struct QuantParams {
    const void *K_head, *V_head, *K_new, *V_new;
    int64_t hd_sb, hd_sh, hd_ss, nw_sb, nw_sh, nw_ss;
    int n_head, n_new;
    int B, H, D, page, n_quant, n_pages;
    uint8_t *K_packed, *V_packed;
    int64_t pk_sb, pk_sh, pk_ss;
    uint16_t *K_scale, *K_mn;
    int64_t km_sb, km_sh, km_sp;
    uint16_t *V_scale, *V_mn;
    int64_t vm_sb, vm_sh, vm_ss;
    void *stage_K, *stage_V;
    int64_t st_sb, st_sh, st_ss;
    const int* pos;      // non-null: tokens already cached, read on the device (see DynPos); outputs then point at token 0
    int n_layers;        // > 1 (only with pos): grid.z = n_layers * B, pos[layer], every tensor offset by its layer stride
    int64_t hd_sl, nw_sl, pk_sl, km_sl, vm_sl, st_sl;
    int max_tokens;      // capacity of the cache rows (device-side guard in that mode)
};

// Code of one element: rint((x - mn) / sc) clamped to 0..15, where the quotient is the IEEE
// fp32 quotient (what the reference computes).  The division is replaced by a multiplication
// with the correctly rounded reciprocal: that product is within 3e-6 of the IEEE quotient for
// quotients below 16, so both round to the same integer unless the product lies within 2e-5
// of a half-integer; only then (about 4 elements in 100 000) is the exact division done.
// Rounding to nearest even through the 1.5 * 2^23 constant.  Returns the code as a float.
__device__ __forceinline__ float code4f(float x, float mn, float sc, float rsc) {
    const float d = __fsub_rn(x, mn);
    const float t = __fmul_rn(d, rsc);
    float r = __fsub_rn(__fadd_rn(t, 12582912.0f), 12582912.0f);
    if (!(fabsf(__fsub_rn(t, r)) < 0.49998f) || !(t < 16.0f))     // near a tie, huge, or NaN
        r = rintf(__fdiv_rn(d, sc));
    return fminf(fmaxf(r, 0.0f), 15.0f);
}
// eight codes -> one 32-bit word, nibble i = code i; two exact fp32 sums of four nibbles each
__device__ __forceinline__ uint32_t pack8(const float (&q)[8]) {
    const float lo = fmaf(q[3], 4096.f, fmaf(q[2], 256.f, fmaf(q[1], 16.f, q[0])));
    const float hi = fmaf(q[7], 4096.f, fmaf(q[6], 256.f, fmaf(q[5], 16.f, q[4])));
    return (uint32_t)lo | ((uint32_t)hi << 16);
}

template <typename T>
__device__ __forceinline__ const T* stream_row(const T* head, const T* nw, const QuantParams& p,
                                               int b, int h, int t) {
    return t < p.n_head ? head + b * p.hd_sb + h * p.hd_sh + (int64_t)t * p.hd_ss
                        : nw + b * p.nw_sb + h * p.nw_sh + (int64_t)(t - p.n_head) * p.nw_ss;
}

// Positions read on the device: append of n_new tokens behind *pos cached ones; the staged head is the partial page.  false: the
// cache is full.
__device__ __forceinline__ bool quant_locate(QuantParams& p) {
    const int seen = *p.pos;
    if (seen < 0 || seen + p.n_new > p.max_tokens) return false;
    const int partial = seen % p.page;
    const int tok_start = seen - partial, pg_start = tok_start / p.page;
    p.n_head = partial;
    p.n_quant = ((partial + p.n_new) / p.page) * p.page;
    p.n_pages = p.n_quant / p.page;
    if (p.K_packed) p.K_packed += (int64_t)tok_start * p.pk_ss;
    if (p.V_packed) p.V_packed += (int64_t)tok_start * p.pk_ss;
    if (p.K_scale) { p.K_scale += (int64_t)pg_start * p.km_sp; p.K_mn += (int64_t)pg_start * p.km_sp; }
    if (p.V_scale) { p.V_scale += (int64_t)tok_start * p.vm_ss; p.V_mn += (int64_t)tok_start * p.vm_ss; }
    return true;
}

// (b, h) of the batch; a warp per page: pages 4 bx .. of this call, the left-over tokens by bx 0.  128 threads.
template <typename T>
__device__ __forceinline__ void quant_int4_cta(const QuantParams& p, int b, int h, int bx) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int page_idx = bx * 4 + warp;
    const int LPT = p.D >> 3;          // lanes per token
    const int TPI = 32 / LPT;          // tokens per warp iteration
    const int ti = lane / LPT, c = lane % LPT;
    const T* Kh = static_cast<const T*>(p.K_head);
    const T* Kn = static_cast<const T*>(p.K_new);
    const T* Vh = static_cast<const T*>(p.V_head);
    const T* Vn = static_cast<const T*>(p.V_new);
    if (page_idx < p.n_pages) {
        const int t0 = page_idx * p.page;
        const int n_tok = min(p.page, p.n_quant - t0);
        // ---------------- K: per page, per channel ----------------
        if (p.K_scale != nullptr) {      // K_packed may be NULL: metadata only
            float mn[8], mx[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) { mn[i] = INFINITY; mx[i] = -INFINITY; }
            for (int tt = ti; tt < n_tok; tt += TPI) {
                float v[8];
                load8<T>(stream_row<T>(Kh, Kn, p, b, h, t0 + tt) + 8 * c, v);
#pragma unroll
                for (int i = 0; i < 8; ++i) { mn[i] = fminf(mn[i], v[i]); mx[i] = fmaxf(mx[i], v[i]); }
            }
            for (int off = LPT; off < 32; off <<= 1) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    mn[i] = fminf(mn[i], __shfl_xor_sync(0xffffffffu, mn[i], off));
                    mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], off));
                }
            }
            float sc[8];
            const float eps = Dt<T>::rn(1e-6f);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float diff = Dt<T>::rn(__fsub_rn(mx[i], mn[i]));
                sc[i] = fmaxf(Dt<T>::rn(__fdiv_rn(diff, 15.0f)), eps);
            }
            float rsc[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) rsc[i] = __frcp_rn(sc[i]);
            if (ti == 0) {
                uint32_t s4[4], m4[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    s4[i] = f32_to_bf16_bits(sc[2 * i]) | ((uint32_t)f32_to_bf16_bits(sc[2 * i + 1]) << 16);
                    m4[i] = f32_to_bf16_bits(mn[2 * i]) | ((uint32_t)f32_to_bf16_bits(mn[2 * i + 1]) << 16);
                }
                int64_t mo = b * p.km_sb + h * p.km_sh + (int64_t)page_idx * p.km_sp + 8 * c;
                *reinterpret_cast<uint4*>(p.K_scale + mo) = make_uint4(s4[0], s4[1], s4[2], s4[3]);
                *reinterpret_cast<uint4*>(p.K_mn + mo) = make_uint4(m4[0], m4[1], m4[2], m4[3]);
            }
            for (int tt = ti; tt < n_tok && p.K_packed != nullptr; tt += TPI) {
                float v[8];
                load8<T>(stream_row<T>(Kh, Kn, p, b, h, t0 + tt) + 8 * c, v);
                float q[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) q[i] = code4f(v[i], mn[i], sc[i], rsc[i]);
                uint8_t* row = p.K_packed + b * p.pk_sb + h * p.pk_sh + (int64_t)(t0 + tt) * p.pk_ss;
                *reinterpret_cast<uint32_t*>(row + 4 * c) = pack8(q);
            }
        }
        // ---------------- V: per token ----------------
        if (p.V_packed != nullptr) {
            for (int tt = ti; tt < n_tok + ti; tt += TPI) {   // uniform trip count for the shuffles
                const bool live = tt < n_tok;
                float v[8];
                if (live) {
                    load8<T>(stream_row<T>(Vh, Vn, p, b, h, t0 + tt) + 8 * c, v);
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[i] = 0.f;
                }
                float lo = v[0], hi = v[0];
#pragma unroll
                for (int i = 1; i < 8; ++i) { lo = fminf(lo, v[i]); hi = fmaxf(hi, v[i]); }
                for (int off = 1; off < LPT; off <<= 1) {
                    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, off));
                    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, off));
                }
                if (live) {
                    float sc = fmaxf(__fdiv_rn(__fsub_rn(hi, lo), 15.0f), 1e-6f);
                    const float rsc = __frcp_rn(sc);
                    float q[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) q[i] = code4f(v[i], lo, sc, rsc);
                    uint8_t* row = p.V_packed + b * p.pk_sb + h * p.pk_sh + (int64_t)(t0 + tt) * p.pk_ss;
                    *reinterpret_cast<uint32_t*>(row + 4 * c) = pack8(q);
                    if (c == 0) {
                        int64_t mo = b * p.vm_sb + h * p.vm_sh + (int64_t)(t0 + tt) * p.vm_ss;
                        p.V_scale[mo] = f32_to_bf16_bits(sc);
                        p.V_mn[mo] = f32_to_bf16_bits(lo);
                    }
                }
            }
        }
    }
    // ---------------- staging of the tokens that do not fill a page ----------------
    // Stream token t >= n_quant goes to staging row t - n_quant.  With n_quant == 0 the head
    // tokens are already in place (the head IS the staging buffer) and only the new tokens are
    // copied behind them.  Done by the CTA that owns page 0 (the only page that can read the
    // staged head, which may alias the staging buffer), after all of its reads.
    if (bx != 0) return;
    __syncthreads();
    const int total = p.n_head + p.n_new;
    const int rem = total - p.n_quant;
    if (rem <= 0) return;
    const int chunks = p.D >> 3;
    for (int i = threadIdx.x; i < rem * chunks; i += blockDim.x) {
        const int r = i / chunks, cc = i % chunks;
        const int t = p.n_quant + r;
        if (p.n_quant == 0 && t < p.n_head) continue;
        const int64_t so = b * p.st_sb + h * p.st_sh + (int64_t)r * p.st_ss + 8 * cc;
        if (p.stage_K != nullptr) {
            const T* src = stream_row<T>(Kh, Kn, p, b, h, t) + 8 * cc;
            T* dst = static_cast<T*>(p.stage_K) + so;
            if (sizeof(T) == 2) {
                *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(src);
            } else {
                reinterpret_cast<uint4*>(dst)[0] = reinterpret_cast<const uint4*>(src)[0];
                reinterpret_cast<uint4*>(dst)[1] = reinterpret_cast<const uint4*>(src)[1];
            }
        }
        if (p.stage_V != nullptr) {
            const T* src = stream_row<T>(Vh, Vn, p, b, h, t) + 8 * cc;
            T* dst = static_cast<T*>(p.stage_V) + so;
            if (sizeof(T) == 2) {
                *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(src);
            } else {
                reinterpret_cast<uint4*>(dst)[0] = reinterpret_cast<const uint4*>(src)[0];
                reinterpret_cast<uint4*>(dst)[1] = reinterpret_cast<const uint4*>(src)[1];
            }
        }
    }
}

}  // namespace fq
