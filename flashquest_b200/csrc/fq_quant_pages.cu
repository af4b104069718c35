// Packing of whole pages of 16-bit K / V rows into 4-bit or 8-bit codes: the bulk append of a prompt.
//
// Same results, bit for bit, as the general kernels (quant_int4_kernel, quant_k_int8_kernel, quant_v_int8_kernel), for
// head_dim 64 or 128, pages of 16, 32 or 64 tokens and 16-bit inputs.  What bounds it is instruction issue and the warps in
// flight to fill it (67 M elements of a 32k-token layer against 172 MB, 26 us at the measured copy rate), so the work per
// element is what this kernel removes:
//  * a warp owns 16 tokens of K or of V and keeps them in registers (32 per lane, packed): one read of the input, 8 loads of
//    16 bytes in flight per lane, no second pass.  K and V in one warp needed 120 registers, 16 warps per SM; apart 24 to 28 fit
//    (quant_pages_ctas);
//  * minima and maxima on packed pairs; the page's other tiles (page 32 / 64) join through shared memory;
//  * a code is the quotient by one residual step (two for V, whose scales are fp32) from the approximate reciprocal, which rounds
//    like the IEEE one (fq_exact_div.cuh), two elements per instruction, rounded by adding 1.5 * 2^23.  Redoing the elements near
//    a half-integer with a division instead costs little in fp16 (1 group of 8 in 3000), but coarse bf16 values lie on
//    half-integers so often that nearly every warp divided;
//  * per-token scales of V: the 16 lanes of a token reduce-scatter (min, -max) pairs, so each lane divides for one token
//    and the others read the result from shared memory.
// Measured, one layer of 32 765 tokens, K + V, 8 heads x 128, the division form with K and V in a warp -> this: 4-bit fp16 page 16
// 57.7 -> 43.3 us (4.0 TB/s), 4-bit bf16 page 64 98.5 -> 45.5, 8-bit bf16 102.1 -> 42.4.
#include "fq_quant_pages.cuh"

namespace fq {

__device__ __forceinline__ float rcp_approx(float x) { float y; asm("rcp.approx.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
// max(|a|, |b|, c), NaN if any is NaN
__device__ __forceinline__ float absmax_nan(float a, float b, float c) {
    float y;
    asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
    return y;
}

__device__ __forceinline__ float min_nan(float a, float b) { float y; asm("min.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b)); return y; }

// The code of one element as the reference computes it: rint of the IEEE quotient, clamped.
__device__ __noinline__ uint32_t code_exact(float x, float mn, float sc, float top) {
    const float r = rintf(__fdiv_rn(__fsub_rn(x, mn), sc));
    return (uint32_t)fminf(fmaxf(r, 0.0f), top);
}

// Codes of eight consecutive elements (four packed words) against per-element or common minima, negated scales and reciprocals:
// code_quotient16 (STEPS 1) or code_quotient32 (STEPS 2) of two elements per instruction, rounded by adding 1.5 * 2^23.
// Returns them packed: BITS 4: one word in out.x; BITS 8: two words.
template <typename T, int BITS, int STEPS>
__device__ __forceinline__ uint2 encode8(const uint32_t (&w)[4], const float2 (&mn)[4], const float2 (&rsc)[4], const float2 (&nsc)[4]) {
    constexpr float MAGIC = 12582912.0f;
    constexpr float TOP = BITS == 4 ? 15.0f : 255.0f;
    const float2 magic = make_float2(MAGIC, MAGIC), neg1 = make_float2(-1.f, -1.f);
    uint32_t u[8];
    float worst = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 d = __ffma2_rn(mn[i], neg1, Q2<T>::f2(w[i]));              // x - mn, rounded once
        float2 t = __fmul2_rn(d, rsc[i]);
#pragma unroll
        for (int s = 0; s < STEPS; ++s) t = __ffma2_rn(__ffma2_rn(t, nsc[i], d), rsc[i], t);
        if (BITS == 8) { t.x = min_nan(t.x, 255.25f); t.y = min_nan(t.y, 255.25f); }    // a rounded-down scale can give 255.99
        worst = absmax_nan(t.x, t.y, worst);
        const float2 m = __fadd2_rn(t, magic);
        u[2 * i] = __float_as_uint(m.x);
        u[2 * i + 1] = __float_as_uint(m.y);
    }
    uint2 out = make_uint2(0u, 0u);
    if (!(worst < 256.f)) {             // infinities and NaNs among the inputs
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 x = Q2<T>::f2(w[i]);
            u[2 * i] = code_exact(x.x, mn[i].x, -nsc[i].x, TOP);
            u[2 * i + 1] = code_exact(x.y, mn[i].y, -nsc[i].y, TOP);
        }
        if (BITS == 4) {
#pragma unroll
            for (int i = 0; i < 8; ++i) out.x |= u[i] << (4 * i);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) { out.x |= u[i] << (8 * i); out.y |= u[4 + i] << (8 * i); }
        }
    } else if (BITS == 4) {
        // u[i] = bits(1.5 * 2^23) + code: shift-add, the constants taken off once
        uint32_t a = 0u;
        constexpr uint32_t C = 0x4b400000u;
        constexpr uint32_t SUM = C + (C << 4) + (C << 8) + (C << 12) + (C << 16) + (C << 20) + (C << 24) + (C << 28);
#pragma unroll
        for (int i = 7; i >= 0; --i) a = (a << 4) + u[i];
        out.x = a - SUM;
    } else {
        out.x = __byte_perm(__byte_perm(u[0], u[1], 0x0040), __byte_perm(u[2], u[3], 0x0040), 0x5410);
        out.y = __byte_perm(__byte_perm(u[4], u[5], 0x0040), __byte_perm(u[6], u[7], 0x0040), 0x5410);
    }
    return out;
}

// CTAs of four warps per SM that the registers are cut for: six have 80 a thread, seven 72.  One layer of 32k tokens, 8 heads, L2
// flushed in between, six against seven: 8-bit bf16 of 128 channels 51.2 -> 49.2 us although 100 bytes spill, of 64 channels (no spills) 35.6 -> 33.6,
// fp16 of 64 channels 33.6 both; 8-bit fp16 of 128 channels spills 340 bytes at 72, 51.2 -> 53.2.  4-bit codes need the 80.
template <typename T, int D, int BITS>
constexpr int quant_pages_ctas() { return BITS == 8 && !(std::is_same_v<T, __half> && D == 128) ? 7 : 6; }

// 16 tokens of one (b, h) per warp.  A lane owns 8 channels (one 16-byte load) of every RPI-th token.
template <typename T, int D, int BITS, int NT>      // NT: 16-token tiles per page
__global__ void __launch_bounds__(128, quant_pages_ctas<T, D, BITS>()) quant_pages_kernel(QuantPagesParams p) {
    constexpr int LPT = D / 8;            // lanes per token
    constexpr int RPI = 32 / LPT;         // tokens per load instruction
    constexpr int NI = 16 / RPI;          // loads per lane for a tile (8 at D 128, 4 at D 64)
    constexpr float TOP = BITS == 4 ? 15.0f : 255.0f, RTOP = 1.0f / TOP;
    __shared__ __align__(16) uint32_t s_mn[NT > 1 ? 4 * 32 * 4 : 4], s_mx[NT > 1 ? 4 * 32 * 4 : 4];    // per-channel extrema of each tile
    __shared__ float4 s_tok[4][16];                                                                   // (min, -scale, 1/scale) of each V token
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int b = blockIdx.z, h = blockIdx.y;
    // K and V of the same tokens are different CTAs
    const bool both = p.K_scale != nullptr && p.V_codes != nullptr;
    const int bx = both ? blockIdx.x >> 1 : blockIdx.x;
    const bool doK = p.K_scale != nullptr && !(both && (blockIdx.x & 1)), doV = p.V_codes != nullptr && !doK;
    const int tile = bx * 4 + warp;
    const int ti = lane / LPT, c = lane % LPT;
    const T* Kh = static_cast<const T*>(p.K_head) + b * p.hd_sb + h * p.hd_sh;
    const T* Vh = static_cast<const T*>(p.V_head) + b * p.hd_sb + h * p.hd_sh;
    const T* Kn = static_cast<const T*>(p.K_new) + b * p.nw_sb + h * p.nw_sh;
    const T* Vn = static_cast<const T*>(p.V_new) + b * p.nw_sb + h * p.nw_sh;
    pdl_wait();        // inputs and the staging rows may come from the previous kernel
    pdl_trigger();
    const int t0 = tile * 16;
    const bool live = t0 < p.n_quant && (doK || doV);
    uint32_t x[NI][4];
    const T *head = doV ? Vh : Kh, *fresh_rows = doV ? Vn : Kn;
    if (live) {
        // only the first page can hold staged tokens
        const bool fresh = t0 >= p.n_head;
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            const int t = t0 + ti + RPI * i;
            const int64_t on = (int64_t)(t - p.n_head) * p.nw_ss + 8 * c, oh = (int64_t)t * p.hd_ss + 8 * c;
            const bool nw = fresh || t >= p.n_head;
            const uint4 u = *reinterpret_cast<const uint4*>(nw ? fresh_rows + on : head + oh);
            x[i][0] = u.x; x[i][1] = u.y; x[i][2] = u.z; x[i][3] = u.w;
        }
    }
    // ---------------- K: per page and channel ----------------
    if (doK) {
        uint32_t mn[4], mx[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) { mn[j] = Q2<T>::POS_INF; mx[j] = Q2<T>::POS_INF | 0x80008000u; }
        if (live) {
#pragma unroll
            for (int i = 0; i < NI; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) { mn[j] = Q2<T>::mn(mn[j], x[i][j]); mx[j] = Q2<T>::mx(mx[j], x[i][j]); }
        }
#pragma unroll
        for (int off = LPT; off < 32; off <<= 1)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                mn[j] = Q2<T>::mn(mn[j], __shfl_xor_sync(0xffffffffu, mn[j], off));
                mx[j] = Q2<T>::mx(mx[j], __shfl_xor_sync(0xffffffffu, mx[j], off));
            }
        if constexpr (NT > 1) {           // the other tiles of the page
            uint4* smn = reinterpret_cast<uint4*>(s_mn);
            uint4* smx = reinterpret_cast<uint4*>(s_mx);
            smn[warp * 32 + lane] = make_uint4(mn[0], mn[1], mn[2], mn[3]);
            smx[warp * 32 + lane] = make_uint4(mx[0], mx[1], mx[2], mx[3]);
            __syncthreads();
#pragma unroll
            for (int o = 1; o < NT; ++o) {
                const uint4 a = smn[(warp ^ o) * 32 + lane], e = smx[(warp ^ o) * 32 + lane];
                mn[0] = Q2<T>::mn(mn[0], a.x); mn[1] = Q2<T>::mn(mn[1], a.y); mn[2] = Q2<T>::mn(mn[2], a.z); mn[3] = Q2<T>::mn(mn[3], a.w);
                mx[0] = Q2<T>::mx(mx[0], e.x); mx[1] = Q2<T>::mx(mx[1], e.y); mx[2] = Q2<T>::mx(mx[2], e.z); mx[3] = Q2<T>::mx(mx[3], e.w);
            }
        }
        if (live) {
            float2 m2[4], sc[4], rs[4];
            const float eps = Dt<T>::rn(1e-6f);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                m2[j] = Q2<T>::f2(mn[j]);
                const float2 hi = Q2<T>::f2(mx[j]);
                const float s[2] = {page_scale<T>(hi.x, m2[j].x, TOP, RTOP, eps), page_scale<T>(hi.y, m2[j].y, TOP, RTOP, eps)};
                sc[j] = make_float2(-s[0], -s[1]);
                rs[j] = make_float2(rcp_approx(s[0]), rcp_approx(s[1]));
            }
            if (ti == 0 && (NT == 1 || (tile & (NT - 1)) == 0)) {
                uint32_t s4[4], m4[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    s4[j] = f32_to_bf16_bits(-sc[j].x) | ((uint32_t)f32_to_bf16_bits(-sc[j].y) << 16);
                    m4[j] = f32_to_bf16_bits(m2[j].x) | ((uint32_t)f32_to_bf16_bits(m2[j].y) << 16);
                }
                const int64_t mo = b * p.km_sb + h * p.km_sh + (int64_t)(tile / NT) * p.km_sp + 8 * c;
                *reinterpret_cast<uint4*>(p.K_scale + mo) = make_uint4(s4[0], s4[1], s4[2], s4[3]);
                *reinterpret_cast<uint4*>(p.K_mn + mo) = make_uint4(m4[0], m4[1], m4[2], m4[3]);
            }
            if (p.K_codes != nullptr) {
                uint8_t* row = p.K_codes + b * p.cd_sb + h * p.cd_sh + (int64_t)(t0 + ti) * p.cd_ss + BITS * c;
#pragma unroll
                for (int i = 0; i < NI; ++i) {
                    const uint2 w = encode8<T, BITS, 1>(x[i], m2, rs, sc);
                    if (BITS == 4) *reinterpret_cast<uint32_t*>(row + (int64_t)(RPI * i) * p.cd_ss) = w.x;
                    else *reinterpret_cast<uint2*>(row + (int64_t)(RPI * i) * p.cd_ss) = w;
                }
            }
        }
    }
    // ---------------- V: per token ----------------
    if (doV && live) {
        uint32_t mm[NI];                  // (min, -max) of this lane's 8 channels, per token
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            const uint32_t lo = Q2<T>::mn(Q2<T>::mn(x[i][0], x[i][1]), Q2<T>::mn(x[i][2], x[i][3]));
            const uint32_t hi = Q2<T>::mx(Q2<T>::mx(x[i][0], x[i][1]), Q2<T>::mx(x[i][2], x[i][3]));
            mm[i] = Q2<T>::mn(__byte_perm(lo, hi, 0x5410) ^ 0x80000000u, __byte_perm(lo, hi, 0x7632) ^ 0x80000000u);
        }
        // reduce-scatter over the token's LPT lanes: lane bit k of c keeps half of the remaining tokens
#pragma unroll
        for (int k = 0, n = NI; (1 << k) < LPT; ++k) {
            if (n > 1) {
                n >>= 1;
                const bool up = (c >> k) & 1;
#pragma unroll
                for (int i = 0; i < NI / 2; ++i) {
                    if (i < n) {
                        const uint32_t send = up ? mm[i] : mm[i + n], keep = up ? mm[i + n] : mm[i];
                        mm[i] = Q2<T>::mn(keep, __shfl_xor_sync(0xffffffffu, send, 1 << k));
                    }
                }
            } else {
                mm[0] = Q2<T>::mn(mm[0], __shfl_xor_sync(0xffffffffu, mm[0], 1 << k));
            }
        }
        // the token left with this lane: bit 0 of c chose the upper half of NI, bit 1 the next half, ...
        int own = 0;
#pragma unroll
        for (int k = 0, n = NI; n > 1; ++k) { n >>= 1; own += ((c >> k) & 1) ? n : 0; }
        const int tok = ti + RPI * own;
        const float2 ext = Q2<T>::f2(mm[0] ^ 0x80000000u);            // (min, max)
        const float vsc = fmaxf(__fdiv_rn(__fsub_rn(ext.y, ext.x), TOP), 1e-6f);
        if (c < NI) {
            s_tok[warp][tok] = make_float4(ext.x, -vsc, refine_rcp(vsc, rcp_approx(vsc)), 0.f);
            const int64_t mo = b * p.vm_sb + h * p.vm_sh + (int64_t)(t0 + tok) * p.vm_ss;
            p.V_scale[mo] = f32_to_bf16_bits(vsc);
            p.V_mn[mo] = f32_to_bf16_bits(ext.x);
        }
        __syncwarp();
        uint8_t* row = p.V_codes + b * p.cd_sb + h * p.cd_sh + (int64_t)(t0 + ti) * p.cd_ss + BITS * c;
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            const float4 q = s_tok[warp][ti + RPI * i];
            float2 m2[4], sc[4], rs[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) { m2[j] = make_float2(q.x, q.x); sc[j] = make_float2(q.y, q.y); rs[j] = make_float2(q.z, q.z); }
            const uint2 w = encode8<T, BITS, 2>(x[i], m2, rs, sc);
            if (BITS == 4) *reinterpret_cast<uint32_t*>(row + (int64_t)(RPI * i) * p.cd_ss) = w.x;
            else *reinterpret_cast<uint2*>(row + (int64_t)(RPI * i) * p.cd_ss) = w;
        }
    }
    // ---------------- staging of the tokens that do not fill a page (the CTA that has read the staged head) ----------------
    if (bx != 0) return;
    __syncthreads();
    const int rem = p.n_head + p.n_new - p.n_quant;
    constexpr int CH = D / 8;
    for (int i = threadIdx.x; i < rem * CH; i += 128) {
        const int r = i / CH, cc = i % CH, t = p.n_quant + r;
        if (p.n_quant == 0 && t < p.n_head) continue;              // already in place
        const int64_t on = (int64_t)(t - p.n_head) * p.nw_ss + 8 * cc, oh = (int64_t)t * p.hd_ss + 8 * cc;
        const int64_t so = b * p.st_sb + h * p.st_sh + (int64_t)r * p.st_ss + 8 * cc;
        if (p.stage_K && !(both && doV)) *reinterpret_cast<uint4*>(static_cast<T*>(p.stage_K) + so) = *reinterpret_cast<const uint4*>(t >= p.n_head ? Kn + on : Kh + oh);
        if (p.stage_V && !(both && doK)) *reinterpret_cast<uint4*>(static_cast<T*>(p.stage_V) + so) = *reinterpret_cast<const uint4*>(t >= p.n_head ? Vn + on : Vh + oh);
    }
    if (p.zero_rest) {
        for (int i = rem * CH + threadIdx.x; i < p.page * CH; i += 128) {
            const int64_t so = b * p.st_sb + h * p.st_sh + (int64_t)(i / CH) * p.st_ss + 8 * (i % CH);
            if (!(both && doV)) *reinterpret_cast<uint4*>(static_cast<T*>(p.stage_K) + so) = make_uint4(0u, 0u, 0u, 0u);
            if (!(both && doK)) *reinterpret_cast<uint4*>(static_cast<T*>(p.stage_V) + so) = make_uint4(0u, 0u, 0u, 0u);
        }
    }
}

bool quant_pages_supported(const QuantPagesParams& p, int dtype) {
    auto a16 = [](const void* x) { return aligned(x, 16); };
    return (dtype == FQ_F16 || dtype == FQ_BF16) && (p.D == 64 || p.D == 128) && (p.page == 16 || p.page == 32 || p.page == 64) &&
           p.n_quant >= 0 && p.n_quant % p.page == 0 && p.B <= 65535 && p.H <= 65535 &&
           a16(p.K_head) && a16(p.V_head) && a16(p.K_new) && a16(p.V_new) && a16(p.stage_K) && a16(p.stage_V) && a16(p.K_scale) && a16(p.K_mn) &&
           p.hd_sb % 8 == 0 && p.hd_sh % 8 == 0 && p.hd_ss % 8 == 0 && p.nw_sb % 8 == 0 && p.nw_sh % 8 == 0 && p.nw_ss % 8 == 0 &&
           p.st_sb % 8 == 0 && p.st_sh % 8 == 0 && p.st_ss % 8 == 0 && p.km_sb % 8 == 0 && p.km_sh % 8 == 0 && p.km_sp % 8 == 0 &&
           p.cd_sb % p.bits == 0 && p.cd_sh % p.bits == 0 && p.cd_ss % p.bits == 0 && aligned(p.K_codes, p.bits) && aligned(p.V_codes, p.bits);
}

template <typename T, int D, int BITS>
static cudaError_t launch_nt(const QuantPagesParams& p, dim3 grid, cudaStream_t st) {
    if (p.page == 16) return launch_k(PDL_QUANT, quant_pages_kernel<T, D, BITS, 1>, grid, dim3(128), 0, st, p);
    if (p.page == 32) return launch_k(PDL_QUANT, quant_pages_kernel<T, D, BITS, 2>, grid, dim3(128), 0, st, p);
    return launch_k(PDL_QUANT, quant_pages_kernel<T, D, BITS, 4>, grid, dim3(128), 0, st, p);
}
template <typename T>
static cudaError_t launch_t(const QuantPagesParams& p, dim3 grid, cudaStream_t st) {
    if (p.D == 128) return p.bits == 4 ? launch_nt<T, 128, 4>(p, grid, st) : launch_nt<T, 128, 8>(p, grid, st);
    return p.bits == 4 ? launch_nt<T, 64, 4>(p, grid, st) : launch_nt<T, 64, 8>(p, grid, st);
}

int quant_pages_launch(const QuantPagesParams& p, int dtype, void* stream, const char* fn) {
    const dim3 grid((unsigned)(max(1, (p.n_quant / 16 + 3) / 4) * (p.K_scale && p.V_codes ? 2 : 1)), (unsigned)p.H, (unsigned)p.B);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (dtype == FQ_F16) launch_t<__half>(p, grid, st);
    else launch_t<__nv_bfloat16>(p, grid, st);
    FQ_CHECK_LAUNCH(fn);
    return FQ_OK;
}

}  // namespace fq
