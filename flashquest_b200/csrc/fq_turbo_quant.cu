// Walsh-Hadamard rotation and TurboQuant K3-V3 packing (3-bit Lloyd-Max codes in a 1-bit and
// a 2-bit plane, per-token RMS scale).
//
// One warp owns one token row of D values; lane l holds the D/32 consecutive values starting
// at l*D/32.  The butterfly stages with a stride inside a lane are register-only, the others
// exchange with lane ^ (stride / values-per-lane) by shuffle.  Every stage is rounded to the
// tensor's dtype exactly as the reference's eager ops do (kernel/wht.py:26-41), so results are
// bit-identical.  HBM-bound: D*sizeof(T) in, 3*D/8 + 2 bytes out per token.
#include "fq_quant_pages.cuh"
#include "fq_wht.cuh"

namespace fq {

// kernel/kv_quant.py:225-229
__device__ __constant__ float c_turbo_codebook[8] = {-2.1519f, -1.3439f, -0.7560f, -0.2451f,
                                                     0.2451f, 0.7560f, 1.3439f, 2.1519f};

// wht_along_head_dim (kernel/wht.py:17): rows of D values, dtype preserved.  Launched early like the rest of the decode chain
// (a TurboQuant step of 16 x 32k: 252 -> 246 us together with the merge).
template <typename T, int EPL>
__global__ void __launch_bounds__(128) wht_kernel(const T* __restrict__ x, T* __restrict__ out, int64_t n_rows, int D) {
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    pdl_wait();
    pdl_trigger();
    if (row >= n_rows) return;
    float v[EPL];
    load_row<T, EPL>(x + row * D, lane, D, v);
    wht_lanes<T, EPL>(v, lane, D);
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
        const int i = lane * EPL + j;
        if (i < D) out[row * D + i] = from_f32<T>(v[j]);
    }
}

struct TurboParams {
    // token streams head[0:n_head] ++ new; the packed kernel takes K and V in one launch (n_streams 2), the other one stream 0
    const void *head[2], *nw[2];
    int64_t hd_sb, hd_sh, hd_ss, nw_sb, nw_sh, nw_ss;
    int n_streams, n_head, n_quant, D;
    uint8_t *msb[2], *lsb[2];                    // (B,H,n,D/8), (B,H,n,D/4)
    int64_t ms_sb, ms_sh, ms_ss, ls_sb, ls_sh, ls_ss;
    uint16_t* scale[2];                          // (B,H,n) bf16
    int64_t sc_sb, sc_sh, sc_ss;
    // with pages of 16 tokens: minimum and scale of stream 0 per page and channel (null: none), and the rows
    // behind n_quant written to the head buffers
    uint16_t *raw_scale, *raw_mn;
    int64_t km_sb, km_sh, km_sp;
    int n_stage;
};

// quantize_k_turbo / quantize_v_turbo without the raw page metadata
// (kernel/kv_quant.py:327-405): rot = WHT(x) in x's dtype; s = max(sqrt(mean(rot^2)), 1e-6) in
// fp32 (lane partial sums in ascending order, then an xor butterfly 16,8,4,2,1);
// idx = first index of min |rot/s - c_j|; planes per kv_quant.py:253-279.
template <typename T, int EPL>
__global__ void __launch_bounds__(128) turbo_quant_kernel(TurboParams p) {
    __shared__ uint8_t s_idx[4][1024];
    __shared__ float s_cb[9];          // the codebook where lanes may index it independently, +inf behind it
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int b = blockIdx.z, h = blockIdx.y;
    const int t = blockIdx.x * 4 + warp;
    if (threadIdx.x < 9) s_cb[threadIdx.x] = threadIdx.x < 8 ? c_turbo_codebook[threadIdx.x] : INFINITY;
    __syncthreads();
    if (t >= p.n_quant) return;
    const int D = p.D;
    const T* row = t < p.n_head
        ? static_cast<const T*>(p.head[0]) + b * p.hd_sb + h * p.hd_sh + (int64_t)t * p.hd_ss
        : static_cast<const T*>(p.nw[0]) + b * p.nw_sb + h * p.nw_sh + (int64_t)(t - p.n_head) * p.nw_ss;
    float v[EPL];
    load_row<T, EPL>(row, lane, D, v);
    wht_lanes<T, EPL>(v, lane, D);
    float a = 0.f;
#pragma unroll
    for (int j = 0; j < EPL; ++j) a = __fmaf_rn(v[j], v[j], a);
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) a = __fadd_rn(a, __shfl_xor_sync(0xffffffffu, a, off));
    const float s = fmaxf(__fsqrt_rn(__fdiv_rn(a, (float)D)), 1e-6f);
    // Nearest codebook entry, first index on ties (torch.argmin): the codebook is sorted, so
    // the winner is one of the two entries around y; which one is decided by the same fp32
    // distances the reference compares.
    auto nearest = [&](float y, float& d0, float& d1) -> int {
        int k = y >= 0.2451f ? 4 : 0;                          // c_4
        k += y >= (k ? 1.3439f : -0.7560f) ? 2 : 0;           // c_6 or c_2
        k += y >= s_cb[k + 1] ? 1 : 0;
        k = min(k, 6);                                        // c_k <= y < c_{k+1}, clamped at both ends
        d0 = fabsf(__fsub_rn(y, s_cb[k]));
        d1 = fabsf(__fsub_rn(y, s_cb[k + 1]));
        return k;
    };
    unsigned idx[EPL];
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
        float d0, d1;
        const int k = nearest(__fdiv_rn(v[j], s), d0, d1);
        idx[j] = (unsigned)(k + (d1 < d0 ? 1 : 0));
    }
    uint8_t* msb = p.msb[0] + b * p.ms_sb + h * p.ms_sh + (int64_t)t * p.ms_ss;
    uint8_t* lsb = p.lsb[0] + b * p.ls_sb + h * p.ls_sh + (int64_t)t * p.ls_ss;
    if constexpr (EPL == 4) {
        // lane = channels 4l..4l+3: exactly one byte of the 2-bit plane, half a byte of the 1-bit plane
        unsigned l8 = 0, m4 = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) { l8 |= (idx[j] & 3u) << (2 * j); m4 |= ((idx[j] >> 2) & 1u) << j; }
        const unsigned hi = __shfl_down_sync(0xffffffffu, m4, 1);
        if (4 * lane < D) lsb[lane] = (uint8_t)l8;
        if ((lane & 1) == 0 && 4 * lane < D) msb[lane >> 1] = (uint8_t)(m4 | (hi << 4));
    } else {
        uint8_t* si = s_idx[warp];
#pragma unroll
        for (int j = 0; j < EPL; ++j) {
            const int i = lane * EPL + j;
            if (i < D) si[i] = (uint8_t)idx[j];
        }
        __syncwarp();
        for (int k = lane; k < D / 8; k += 32) {
            unsigned m = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) m |= (unsigned)((si[8 * k + i] >> 2) & 1) << i;
            msb[k] = (uint8_t)m;
        }
        for (int k = lane; k < D / 4; k += 32) {
            unsigned m = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) m |= (unsigned)(si[4 * k + i] & 3) << (2 * i);
            lsb[k] = (uint8_t)m;
        }
    }
    if (lane == 0) p.scale[0][b * p.sc_sb + h * p.sc_sh + (int64_t)t * p.sc_ss] = f32_to_bf16_bits(s);
}

// The same coding for the shape that matters (head_dim 128, 16-bit values, 8-byte aligned rows); results are bit-identical
// to turbo_quant_kernel (the tests compare both with the reference's planes).  Issue bound, so the work per row is kept in
// packed 16-bit pairs and shared by four lanes: lane t of a row's quad holds channels 32j + 8t .. + 7, so four of the seven
// butterflies stay inside a lane and a warp codes eight tokens at a time.
//  * a butterfly with a partner lane is one shuffle and one packed fma(mine, +-1, other), which rounds once like the add;
//  * x / fp32(sqrt(128)) rounded to the dtype equals x * TURBO_RCD rounded to the dtype for every one of the 65 536 bit
//    patterns of either dtype (fq_exact_div.cuh);
//  * the sum of squares adds in turbo_quant_kernel's order: groups of four channels, then groups 16, 8, 4, 2, 1 apart;
//  * the code of v depends on the nearest entry of v / s, which is monotone in |v|.  So a token needs four 16-bit numbers:
//    the smallest |v| that reaches the second, third and fourth magnitude, and the smallest v > 0 that counts as positive
//    (tiny ones tie with the negative side).  Each lane of the quad finds one: the 16-bit neighbours around midpoint * s;
//    a value within 1e-6 of it (the fp32 roundings on either side reach 4e-7) goes through the reference's own arithmetic.
//    Then 2 values take four packed comparisons and five logic operations, bits land at their place by mask;
//  * a token whose two signs disagree at a threshold (an exact tie of the fp32 distances), or whose scale is not finite,
//    takes the value-by-value path.
// 32 768 tokens x 8 heads (67 MB of fp16): 77 us with a warp per token, 34 us so (2.3 TB/s).
// In an append K, V, the page extrema and the staged rows are one launch: 32 768 tokens 113 -> 75 us (three launches read K twice).

// The reference's own decision (kernel/kv_quant.py:253-279): fp32 quotient, fp32 distances, first index on ties.
// Out of line: it runs for a few values in 10^4 and should not lengthen the loop body.
__device__ __noinline__ unsigned turbo_idx_exact(float v, float s) {
    const float y = __fdiv_rn(v, s);
    int k = y >= 0.2451f ? 4 : 0;
    k += y >= (k ? 1.3439f : -0.7560f) ? 2 : 0;
    k += y >= c_turbo_codebook[k + 1] ? 1 : 0;
    k = min(k, 6);
    const float d0 = fabsf(__fsub_rn(y, c_turbo_codebook[k])), d1 = fabsf(__fsub_rn(y, c_turbo_codebook[k + 1]));
    return (unsigned)(k + (d1 < d0 ? 1 : 0));
}

// midpoints between neighbouring codebook magnitudes
constexpr float TURBO_M0 = 0.50055f, TURBO_M1 = 1.04995f, TURBO_M2 = 1.7479f;

// one value of the value-by-value path: |v| against the midpoints, the exact decision near them or near zero
__device__ __noinline__ unsigned turbo_idx_value(float v, float s) {
    constexpr float GUARD = 3e-5f;
    const float th0 = TURBO_M0 * s, th1 = TURBO_M1 * s, th2 = TURBO_M2 * s, av = fabsf(v);
    const int m = (av > th0 ? 1 : 0) + (av > th1 ? 1 : 0) + (av > th2 ? 1 : 0);
    const bool risky = fabsf(av - th0) < GUARD * th0 || fabsf(av - th1) < GUARD * th1 || fabsf(av - th2) < GUARD * th2 || av < GUARD * s;
    return risky ? turbo_idx_exact(v, s) : (unsigned)(v < 0.f ? 3 - m : 4 + m);
}

template <typename T> struct TurboT;
template <> struct TurboT<__half> {
    __device__ static uint32_t down(float f) { return __half_as_ushort(__float2half_rd(f)); }
    __device__ static uint32_t up(float f) { return __half_as_ushort(__float2half_ru(f)); }
    __device__ static float value(uint32_t b) { return __half2float(__ushort_as_half((unsigned short)b)); }
};
template <> struct TurboT<__nv_bfloat16> {
    __device__ static uint32_t down(float f) { return __bfloat16_as_ushort(__float2bfloat16_rd(f)); }
    __device__ static uint32_t up(float f) { return __bfloat16_as_ushort(__float2bfloat16_ru(f)); }
    __device__ static float value(uint32_t b) { return __bfloat162float(__ushort_as_bfloat16((unsigned short)b)); }
};

constexpr int TQ_WARPS = 4, TQ_TOK = 8;            // warps per CTA, tokens of a warp at a time

template <typename T>
__global__ void __launch_bounds__(TQ_WARPS * 32, 6) turbo_quant128_kernel(TurboParams p, int iters, int vec_in, int vec_out) {
    using P2 = typename Pk2<T>::type;
    constexpr bool IS_HALF = Dt<T>::code == FQ_F16;
    __shared__ __align__(16) uint8_t s_m[TQ_WARPS][TQ_TOK][16], s_l[TQ_WARPS][TQ_TOK][32];
    __shared__ uint32_t s_x[TQ_WARPS][16][32];     // the value-by-value path's copy of a warp's packed values
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = lane & 3, r = lane >> 2;
    const int which = p.n_streams == 2 ? blockIdx.z & 1 : 0, b = p.n_streams == 2 ? blockIdx.z >> 1 : blockIdx.z, h = blockIdx.y;
    const int t0 = (blockIdx.x * TQ_WARPS + warp) * TQ_TOK * iters;
    const T* head = static_cast<const T*>(p.head[which]) + b * p.hd_sb + h * p.hd_sh;
    const T* nw = static_cast<const T*>(p.nw[which]) + b * p.nw_sb + h * p.nw_sh;
    uint8_t* msb = p.msb[which] + b * p.ms_sb + h * p.ms_sh;
    uint8_t* lsb = p.lsb[which] + b * p.ls_sb + h * p.ls_sh;
    uint16_t* scale = p.scale[which] + b * p.sc_sb + h * p.sc_sh;

    auto row_of = [&](int tok) { return tok < p.n_head ? head + (int64_t)tok * p.hd_ss : nw + (int64_t)(tok - p.n_head) * p.nw_ss; };
    auto load_row = [&](int tok, uint4 (&raw)[4]) {
        tok = min(tok, p.n_quant - 1);
        const T* row = row_of(tok) + 8 * t;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (vec_in) raw[j] = __ldg(reinterpret_cast<const uint4*>(row + 32 * j));
            else {
                const uint2 lo = __ldg(reinterpret_cast<const uint2*>(row + 32 * j)), hi = __ldg(reinterpret_cast<const uint2*>(row + 32 * j + 4));
                raw[j] = make_uint4(lo.x, lo.y, hi.x, hi.y);
            }
        }
    };
    if (t0 >= p.n_quant) return;
    if (p.raw_scale != nullptr && which == 0 && t0 % 16 == 0) {
        // the page's extrema, as quant_pages_kernel computes them; these reads bring the rows in for the coding below
        const int half = lane >> 4, c = lane & 15;
        uint4 u[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) u[i] = __ldg(reinterpret_cast<const uint4*>(row_of(t0 + 2 * i + half)) + c);
        uint32_t mn[4] = {u[0].x, u[0].y, u[0].z, u[0].w}, mx[4] = {u[0].x, u[0].y, u[0].z, u[0].w};
#pragma unroll
        for (int i = 1; i < 8; ++i) {
            const uint32_t w[4] = {u[i].x, u[i].y, u[i].z, u[i].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) { mn[j] = Q2<T>::mn(mn[j], w[j]); mx[j] = Q2<T>::mx(mx[j], w[j]); }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            mn[j] = Q2<T>::mn(mn[j], __shfl_xor_sync(0xffffffffu, mn[j], 16));
            mx[j] = Q2<T>::mx(mx[j], __shfl_xor_sync(0xffffffffu, mx[j], 16));
        }
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {                              // lanes 0..15 the scales, 16..31 the minima
            const float2 lo = Q2<T>::f2(mn[j]), hi = Q2<T>::f2(mx[j]);
            const float eps = Dt<T>::rn(1e-6f);
            const float ox = half ? lo.x : page_scale<T>(hi.x, lo.x, 15.0f, 1.0f / 15.0f, eps);
            const float oy = half ? lo.y : page_scale<T>(hi.y, lo.y, 15.0f, 1.0f / 15.0f, eps);
            o[j] = f32_to_bf16_bits(ox) | ((uint32_t)f32_to_bf16_bits(oy) << 16);
        }
        const int64_t mo = b * p.km_sb + h * p.km_sh + (int64_t)(t0 >> 4) * p.km_sp + 8 * c;
        *reinterpret_cast<uint4*>((half ? p.raw_mn : p.raw_scale) + mo) = make_uint4(o[0], o[1], o[2], o[3]);
    }
    uint4 raw[4];
    load_row(t0 + r, raw);
    const uint32_t one = IS_HALF ? 0x3c003c00u : 0x3f803f80u;
    const P2 pm = p2_from<P2>(IS_HALF ? 0xbc003c00u : 0xbf803f80u);              // (+1, -1)
    const P2 sg0 = p2_from<P2>(one | (t & 1 ? 0x80008000u : 0u)), sg1 = p2_from<P2>(one | (t & 2 ? 0x80008000u : 0u));

#pragma unroll 1
    for (int it = 0; it < iters; ++it) {
        const int tok = t0 + it * TQ_TOK + r;
        if (t0 + it * TQ_TOK >= p.n_quant) break;
        P2 x[4][4];
        // stride 1: (a, b) -> (a + b, a - b)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t u[4] = {raw[j].x, raw[j].y, raw[j].z, raw[j].w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
                x[j][i] = __hfma2(p2_from<P2>(__byte_perm(u[i], u[i], 0x3232)), pm, p2_from<P2>(__byte_perm(u[i], u[i], 0x1010)));
        }
        if (it + 1 < iters) load_row(tok + TQ_TOK, raw);           // in flight while this tile is coded
        auto bfly = [](P2& a, P2& c) { const P2 u = a, v = c; a = __hadd2(u, v); c = __hsub2(u, v); };
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            bfly(x[j][0], x[j][1]); bfly(x[j][2], x[j][3]);        // stride 2
            bfly(x[j][0], x[j][2]); bfly(x[j][1], x[j][3]);        // stride 4
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) {                          // strides 8, 16: the quad
                x[j][i] = __hfma2(x[j][i], sg0, p2_from<P2>(__shfl_xor_sync(0xffffffffu, p2_bits(x[j][i]), 1)));
                x[j][i] = __hfma2(x[j][i], sg1, p2_from<P2>(__shfl_xor_sync(0xffffffffu, p2_bits(x[j][i]), 2)));
            }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            bfly(x[0][i], x[1][i]); bfly(x[2][i], x[3][i]);        // stride 32
            bfly(x[0][i], x[2][i]); bfly(x[1][i], x[3][i]);        // stride 64
        }
        // divide by sqrt(128), round to the dtype; sums of squares of each group of four channels
        float a[4][2];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 f = Pk2<T>::unpack(x[j][i]);
                x[j][i] = Pk2<T>::make(__fmul_rn(f.x, TURBO_RCD), __fmul_rn(f.y, TURBO_RCD));
                const float2 v = Pk2<T>::unpack(x[j][i]);
                a[j][i >> 1] = __fmaf_rn(v.y, v.y, __fmaf_rn(v.x, v.x, (i & 1) ? a[j][i >> 1] : 0.f));
            }
        float q[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            q[e] = __fadd_rn(__fadd_rn(a[0][e], a[2][e]), __fadd_rn(a[1][e], a[3][e]));
            q[e] = __fadd_rn(q[e], __shfl_xor_sync(0xffffffffu, q[e], 2));
            q[e] = __fadd_rn(q[e], __shfl_xor_sync(0xffffffffu, q[e], 1));
        }
        const float s = fmaxf(__fsqrt_rn(__fmul_rn(__fadd_rn(q[0], q[1]), 1.0f / 128)), 1e-6f);      // a / 128 is exact either way
        // this lane's threshold of the token
        const float th = s * (t == 0 ? TURBO_M0 : t == 1 ? TURBO_M1 : t == 2 ? TURBO_M2 : 7.450580596923828e-9f /* 2^-27 */);
        const uint32_t below = TurboT<T>::down(th * (1.0f - 1e-6f)), above = TurboT<T>::up(th * (1.0f + 1e-6f));
        uint32_t T16 = above;
        bool slow = !(s < 1e30f);
        if (below + 1 != above && !slow) {
            const float mid = TurboT<T>::value(below + 1);
            const unsigned ip = turbo_idx_exact(mid, s), in = turbo_idx_exact(-mid, s);
            const bool up = t == 3 ? ip >= 4u : ip >= 5u + t;
            slow = t != 3 && up != (in + t <= 2u);
            if (up) T16 = below + 1;
        }
        T16 |= T16 << 16;
        const P2 T0 = p2_from<P2>(__shfl_sync(0xffffffffu, T16, 0, 4)), T1 = p2_from<P2>(__shfl_sync(0xffffffffu, T16, 1, 4));
        const P2 T2 = p2_from<P2>(__shfl_sync(0xffffffffu, T16, 2, 4)), Tz = p2_from<P2>(__shfl_sync(0xffffffffu, T16, 3, 4));
        // bits of the 1-bit plane (z) and of the 2-bit plane: code 4 + m for positive values, 3 - m for the others
        uint32_t mw[2] = {0u, 0u}, lw[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const P2 ax = p2_from<P2>(p2_bits(x[j][i]) & 0x7fff7fffu);
                const uint32_t z = __hge2_mask(x[j][i], Tz), g0 = __hge2_mask(ax, T0), g1 = __hge2_mask(ax, T1), g2 = __hge2_mask(ax, T2);
                const uint32_t b1 = ~(g1 ^ z), b0 = g0 ^ g2 ^ b1;
                mw[j >> 1] |= z & (((1u << (2 * i)) | (0x20000u << (2 * i))) << (8 * (j & 1)));
                lw[j] |= b0 & ((1u << (4 * i)) | (0x40000u << (4 * i)));
                lw[j] |= b1 & ((2u << (4 * i)) | (0x80000u << (4 * i)));
            }
        const unsigned slow_lanes = __ballot_sync(0xffffffffu, slow);
        if ((slow_lanes >> (4 * r)) & 15u) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) s_x[warp][j * 4 + i][lane] = p2_bits(x[j][i]);
            mw[0] = mw[1] = 0u;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                lw[j] = 0u;
#pragma unroll 1
                for (int c = 0; c < 8; ++c) {
                    const unsigned idx = turbo_idx_value(TurboT<T>::value((s_x[warp][j * 4 + (c >> 1)][lane] >> (16 * (c & 1))) & 0xffffu), s);
                    mw[j >> 1] |= (idx >> 2) << (8 * (j & 1) + c);
                    lw[j] |= (idx & 3u) << (2 * c);
                }
            }
        }
        __syncwarp();                                              // the tile before has been stored
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t m = (mw[j >> 1] | (mw[j >> 1] >> 16)) >> (8 * (j & 1));
            s_m[warp][r][4 * j + t] = (uint8_t)m;
            *reinterpret_cast<uint16_t*>(&s_l[warp][r][2 * (4 * j + t)]) = (uint16_t)(lw[j] | (lw[j] >> 16));
        }
        if (t == 0 && tok < p.n_quant) scale[(int64_t)tok * p.sc_ss] = f32_to_bf16_bits(s);
        __syncwarp();
        // 8 rows of 16 bytes, 8 rows of 32 bytes: a 16-byte piece per lane
        if (lane < 24) {
            const int row = lane < 8 ? lane : (lane - 8) >> 1, wt = t0 + it * TQ_TOK + row;
            const uint8_t* src = lane < 8 ? s_m[warp][row] : s_l[warp][row] + 16 * (lane & 1);
            uint8_t* dst = lane < 8 ? msb + (int64_t)wt * p.ms_ss : lsb + (int64_t)wt * p.ls_ss + 16 * (lane & 1);
            if (wt < p.n_quant) {
                if (vec_out) *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(src);
                else {
#pragma unroll 1
                    for (int c = 0; c < 16; ++c) dst[c] = src[c];
                }
            }
        }
    }
    if (p.n_stage > 0 && blockIdx.x == 0 && warp < 2) {
        // the rows behind the last page become the staged ones, once the first page's warps have read those before
        if (iters == 1) asm volatile("bar.sync 1, 64;" ::: "memory");
        if (warp == 0) {
            T* st = const_cast<T*>(head);
            for (int i = lane >> 4; i < p.n_stage; i += 2)
                *(reinterpret_cast<uint4*>(st + (int64_t)i * p.hd_ss) + (lane & 15)) = *(reinterpret_cast<const uint4*>(nw + (int64_t)(p.n_quant - p.n_head + i) * p.nw_ss) + (lane & 15));
        }
    }
}

// The packed kernel, where it takes the rows: head_dim 128, 16-bit values, 8-byte aligned rows (16 bytes for the page
// extrema and the staging).  Returns false if it does not.
static bool turbo_launch128(const TurboParams& p, int dtype, int B, int H, cudaStream_t st) {
    auto vec = [](const void* q, int64_t m, int64_t n, int64_t a, int64_t b, int64_t c) { return q == nullptr || (aligned(q, m) && a % n == 0 && b % n == 0 && c % n == 0); };
    bool in8 = true, in16 = true, out16 = true;
    for (int i = 0; i < p.n_streams; ++i) {
        in8 = in8 && vec(p.head[i], 8, 4, p.hd_sb, p.hd_sh, p.hd_ss) && vec(p.nw[i], 8, 4, p.nw_sb, p.nw_sh, p.nw_ss);
        in16 = in16 && vec(p.head[i], 16, 8, p.hd_sb, p.hd_sh, p.hd_ss) && vec(p.nw[i], 16, 8, p.nw_sb, p.nw_sh, p.nw_ss);
        out16 = out16 && vec(p.msb[i], 16, 16, p.ms_sb, p.ms_sh, p.ms_ss) && vec(p.lsb[i], 16, 16, p.ls_sb, p.ls_sh, p.ls_ss);
    }
    const bool pages = p.raw_scale != nullptr || p.n_stage > 0;
    if (p.D != 128 || dtype == FQ_F32 || !in8 || (pages && !(in16 && vec(p.raw_scale, 16, 8, p.km_sb, p.km_sh, p.km_sp) && aligned(p.raw_mn, 16)))) return false;
    if ((int64_t)B * p.n_streams > 65535) return false;
    // tiles of 8 tokens per warp: one until every warp slot of the chip is taken, then two (the second one's rows are
    // in flight while the first is coded; with four the last wave costs more: 34.2 against 36.3 us at 262 144 rows)
    const int64_t tiles = (int64_t)((p.n_quant + TQ_TOK - 1) / TQ_TOK) * B * H * p.n_streams;
    const int iters = tiles > 148 * 24 ? 2 : 1;
    const int per_cta = TQ_WARPS * TQ_TOK * iters;
    dim3 grid((unsigned)((p.n_quant + per_cta - 1) / per_cta), (unsigned)H, (unsigned)(B * p.n_streams));
    count_launch();
    if (dtype == FQ_F16) turbo_quant128_kernel<__half><<<grid, TQ_WARPS * 32, 0, st>>>(p, iters, in16, out16);
    else turbo_quant128_kernel<__nv_bfloat16><<<grid, TQ_WARPS * 32, 0, st>>>(p, iters, in16, out16);
    return true;
}

// dequantize_k_turbo / dequantize_v_turbo (kernel/kv_quant.py:366-378, :408-420):
// codebook[idx] * scale in fp32, WHT in fp32, cast to bf16.
template <int EPL>
__global__ void __launch_bounds__(128) turbo_dequant_kernel(
    const uint8_t* __restrict__ msb, int64_t ms_sb, int64_t ms_sh, int64_t ms_ss,
    const uint8_t* __restrict__ lsb, int64_t ls_sb, int64_t ls_sh, int64_t ls_ss,
    const uint16_t* __restrict__ scale, int64_t sc_sb, int64_t sc_sh, int64_t sc_ss,
    int S, int D, uint16_t* __restrict__ out, int64_t o_sb, int64_t o_sh, int64_t o_ss) {
    const int lane = threadIdx.x & 31;
    const int b = blockIdx.z, h = blockIdx.y;
    const int t = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (t >= S) return;
    const uint8_t* mrow = msb + b * ms_sb + h * ms_sh + (int64_t)t * ms_ss;
    const uint8_t* lrow = lsb + b * ls_sb + h * ls_sh + (int64_t)t * ls_ss;
    const float s = bf16_lo(scale[b * sc_sb + h * sc_sh + (int64_t)t * sc_ss]);
    float v[EPL];
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
        const int i = lane * EPL + j;
        v[j] = 0.f;
        if (i < D) {
            const unsigned m = (mrow[i >> 3] >> (i & 7)) & 1u;
            const unsigned l2 = (lrow[i >> 2] >> (2 * (i & 3))) & 3u;
            v[j] = __fmul_rn(c_turbo_codebook[(m << 2) | l2], s);
        }
    }
    wht_lanes<float, EPL>(v, lane, D);
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
        const int i = lane * EPL + j;
        if (i < D) out[b * o_sb + h * o_sh + (int64_t)t * o_ss + i] = f32_to_bf16_bits(v[j]);
    }
}

template <typename T>
static int launch_wht(const void* x, void* out, int64_t n_rows, int D, cudaStream_t st) {
    const int epl = D >= 32 ? D / 32 : 1;
    const unsigned blocks = (unsigned)((n_rows + 3) / 4);
#define FQ_W(E) launch_k(PDL_QUANT, wht_kernel<T, E>, dim3(blocks), dim3(128), 0, st, static_cast<const T*>(x), static_cast<T*>(out), n_rows, D)
    switch (epl) {
        case 1: FQ_W(1); break;
        case 2: FQ_W(2); break;
        case 4: FQ_W(4); break;
        case 8: FQ_W(8); break;
        case 16: FQ_W(16); break;
        default: FQ_W(32); break;
    }
#undef FQ_W
    return FQ_OK;
}

template <typename T>
static void launch_turbo(const TurboParams& p, dim3 grid, cudaStream_t st) {
    const int epl = p.D >= 32 ? p.D / 32 : 1;
    count_launch();
#define FQ_T(E) turbo_quant_kernel<T, E><<<grid, 128, 0, st>>>(p)
    switch (epl) {
        case 1: FQ_T(1); break;
        case 2: FQ_T(2); break;
        case 4: FQ_T(4); break;
        case 8: FQ_T(8); break;
        case 16: FQ_T(16); break;
        default: FQ_T(32); break;
    }
#undef FQ_T
}

}  // namespace fq

extern "C" int fq_wht(const void* x, void* out, int dtype, int64_t n_rows, int D, void* stream) {
    using namespace fq;
    const char* fn = "fq_wht";
    FQ_CHECK_ARG(D > 0 && (D & (D - 1)) == 0, FQ_ERR_ARG, "%s: head_dim must be a positive power of 2, got %d", fn, D);
    FQ_CHECK_ARG(D <= 1024, FQ_ERR_UNSUPPORTED, "%s: head_dim %d above 1024", fn, D);
    FQ_CHECK_ARG(n_rows >= 0 && (n_rows == 0 || (x && out)), FQ_ERR_ARG, "%s: bad arguments", fn);
    if (n_rows == 0) return FQ_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (dtype == FQ_F32) launch_wht<float>(x, out, n_rows, D, st);
    else if (dtype == FQ_F16) launch_wht<__half>(x, out, n_rows, D, st);
    else if (dtype == FQ_BF16) launch_wht<__nv_bfloat16>(x, out, n_rows, D, st);
    else return fail(FQ_ERR_DTYPE, "%s: dtype code %d", fn, dtype);
    FQ_CHECK_LAUNCH(fn);
    return FQ_OK;
}

extern "C" int fq_quantize_turbo(
    const void* head, int64_t hd_sb, int64_t hd_sh, int64_t hd_ss, int n_head,
    const void* nw, int64_t nw_sb, int64_t nw_sh, int64_t nw_ss, int n_new,
    int dtype, int B, int H, int D, int n_quant,
    uint8_t* msb, int64_t ms_sb, int64_t ms_sh, int64_t ms_ss,
    uint8_t* lsb, int64_t ls_sb, int64_t ls_sh, int64_t ls_ss,
    void* scale, int64_t sc_sb, int64_t sc_sh, int64_t sc_ss, void* stream) {
    using namespace fq;
    const char* fn = "fq_quantize_turbo";
    FQ_CHECK_ARG(B > 0 && H > 0 && n_head >= 0 && n_new >= 0 && n_quant >= 0 && n_quant <= n_head + n_new, FQ_ERR_ARG, "%s: bad sizes", fn);
    FQ_CHECK_ARG(D % 8 == 0, FQ_ERR_ARG, "%s: requires head_dim multiple of 8; got %d", fn, D);
    FQ_CHECK_ARG(D > 0 && (D & (D - 1)) == 0, FQ_ERR_ARG, "%s: head_dim must be a positive power of 2, got %d", fn, D);
    FQ_CHECK_ARG(D <= 1024, FQ_ERR_UNSUPPORTED, "%s: head_dim %d above 1024", fn, D);
    FQ_CHECK_ARG(dtype == FQ_F32 || dtype == FQ_F16 || dtype == FQ_BF16, FQ_ERR_DTYPE, "%s: dtype code %d", fn, dtype);
    if (n_quant == 0) return FQ_OK;
    FQ_CHECK_ARG(msb && lsb && scale && (nw || n_new == 0) && (head || n_head == 0), FQ_ERR_ARG, "%s: null pointer", fn);
    FQ_CHECK_ARG(B <= 65535 && H <= 65535, FQ_ERR_ARG, "%s: B and H must be <= 65535", fn);
    TurboParams p{};
    p.n_streams = 1; p.head[0] = head; p.nw[0] = nw; p.hd_sb = hd_sb; p.hd_sh = hd_sh; p.hd_ss = hd_ss;
    p.nw_sb = nw_sb; p.nw_sh = nw_sh; p.nw_ss = nw_ss; p.n_head = n_head; p.n_quant = n_quant; p.D = D;
    p.msb[0] = msb; p.lsb[0] = lsb; p.ms_sb = ms_sb; p.ms_sh = ms_sh; p.ms_ss = ms_ss; p.ls_sb = ls_sb; p.ls_sh = ls_sh; p.ls_ss = ls_ss;
    p.scale[0] = static_cast<uint16_t*>(scale); p.sc_sb = sc_sb; p.sc_sh = sc_sh; p.sc_ss = sc_ss;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (turbo_launch128(p, dtype, B, H, st)) {
        FQ_CHECK_LAUNCH(fn);
        return FQ_OK;
    }
    dim3 grid((unsigned)((n_quant + 3) / 4), (unsigned)H, (unsigned)B);
    if (dtype == FQ_F32) launch_turbo<float>(p, grid, st);
    else if (dtype == FQ_F16) launch_turbo<__half>(p, grid, st);
    else launch_turbo<__nv_bfloat16>(p, grid, st);
    FQ_CHECK_LAUNCH(fn);
    return FQ_OK;
}

extern "C" int fq_append_kv_turbo(const fq_turbo_cache* c, int layer, int seen, const void* K_new, const void* V_new,
                                  int64_t nw_sb, int64_t nw_sh, int64_t nw_ss, int n_new, void* stream) {
    using namespace fq;
    const char* fn = "fq_append_kv_turbo";
    FQ_CHECK_ARG(c && K_new && V_new, FQ_ERR_ARG, "%s: null pointer", fn);
    FQ_CHECK_ARG(layer >= 0 && layer < c->L, FQ_ERR_ARG, "%s: layer_idx %d out of range [0, %d)", fn, layer, c->L);
    FQ_CHECK_ARG(seen >= 0 && n_new > 0 && seen + n_new <= c->max_seq_len, FQ_ERR_ARG, "%s: seen+new=%d exceeds max_seq_len=%d", fn, seen + n_new, c->max_seq_len);
    const int page = c->page, D = c->D, B = c->B, H = c->Hkv;
    const int partial = seen % page, n_quant = (partial + n_new) / page * page, tok0 = seen - partial;
    char* Kt = static_cast<char*>(c->K_partial) + layer * c->pt_sl * 2;
    char* Vt = static_cast<char*>(c->V_partial) + layer * c->pt_sl * 2;
    uint16_t* Ksr = static_cast<uint16_t*>(c->K_scale_raw) + layer * c->km_sl + (int64_t)(tok0 / page) * c->km_sp;
    uint16_t* Kmr = static_cast<uint16_t*>(c->K_mn_raw) + layer * c->km_sl + (int64_t)(tok0 / page) * c->km_sp;
    if (n_quant > 0) {
        TurboParams p{};
        p.n_streams = 2; p.head[0] = Kt; p.head[1] = Vt; p.nw[0] = K_new; p.nw[1] = V_new;
        p.hd_sb = c->pt_sb; p.hd_sh = c->pt_sh; p.hd_ss = c->pt_ss; p.nw_sb = nw_sb; p.nw_sh = nw_sh; p.nw_ss = nw_ss;
        p.n_head = partial; p.n_quant = n_quant; p.D = D;
        const int64_t mo = layer * c->ms_sl + (int64_t)tok0 * c->ms_ss, lo = layer * c->ls_sl + (int64_t)tok0 * c->ls_ss;
        p.msb[0] = c->K_msb + mo; p.msb[1] = c->V_msb + mo; p.ms_sb = c->ms_sb; p.ms_sh = c->ms_sh; p.ms_ss = c->ms_ss;
        p.lsb[0] = c->K_lsb + lo; p.lsb[1] = c->V_lsb + lo; p.ls_sb = c->ls_sb; p.ls_sh = c->ls_sh; p.ls_ss = c->ls_ss;
        p.scale[0] = static_cast<uint16_t*>(c->K_scale_turbo) + layer * c->st_sl + tok0;
        p.scale[1] = static_cast<uint16_t*>(c->V_scale_turbo) + layer * c->st_sl + tok0;
        p.sc_sb = c->st_sb; p.sc_sh = c->st_sh; p.sc_ss = 1;
        // One warp finds the extrema of 16 tokens, whose rows it brings in for the coding: a page of 16.  Larger pages would have
        // to join those of several warps, which is not built; their K is read again by the launch at the end.
        if (page == 16) {
            p.raw_scale = Ksr; p.raw_mn = Kmr; p.km_sb = c->km_sb; p.km_sh = c->km_sh; p.km_sp = c->km_sp;
            p.n_stage = partial + n_new - n_quant;
        }
        if (turbo_launch128(p, c->kv_dtype, B, H, static_cast<cudaStream_t>(stream))) {
            FQ_CHECK_LAUNCH(fn);
            if (page == 16) return FQ_OK;
        } else {
            for (int i = 0; i < 2; ++i) {
                const int rc = fq_quantize_turbo(p.head[i], c->pt_sb, c->pt_sh, c->pt_ss, partial, p.nw[i], nw_sb, nw_sh, nw_ss, n_new, c->kv_dtype, B, H, D, n_quant,
                                                 p.msb[i], c->ms_sb, c->ms_sh, c->ms_ss, p.lsb[i], c->ls_sb, c->ls_sh, c->ls_ss, p.scale[i], c->st_sb, c->st_sh, 1, stream);
                if (rc != FQ_OK) return rc;
            }
        }
    }
    // raw per-page K metadata (for scoring) + staging of the left-over tokens, after the launches
    // above have read the staged head
    return fq_quantize_kv_int4(Kt, Vt, c->pt_sb, c->pt_sh, c->pt_ss, partial, K_new, V_new, nw_sb, nw_sh, nw_ss, n_new,
                               c->kv_dtype, B, H, D, page, n_quant, nullptr, nullptr, 0, 0, 0, Ksr, Kmr, c->km_sb, c->km_sh, c->km_sp,
                               nullptr, nullptr, 0, 0, 0, Kt, Vt, c->pt_sb, c->pt_sh, c->pt_ss, stream);
}

extern "C" int fq_dequantize_turbo(
    const uint8_t* msb, int64_t ms_sb, int64_t ms_sh, int64_t ms_ss,
    const uint8_t* lsb, int64_t ls_sb, int64_t ls_sh, int64_t ls_ss,
    const void* scale, int64_t sc_sb, int64_t sc_sh, int64_t sc_ss,
    int B, int H, int S, int D, void* out, int64_t o_sb, int64_t o_sh, int64_t o_ss, void* stream) {
    using namespace fq;
    const char* fn = "fq_dequantize_turbo";
    FQ_CHECK_ARG(B > 0 && H > 0 && S >= 0, FQ_ERR_ARG, "%s: bad sizes", fn);
    FQ_CHECK_ARG(D >= 8 && (D & (D - 1)) == 0 && D <= 1024, FQ_ERR_UNSUPPORTED, "%s: head_dim %d must be a power of 2 in [8, 1024]", fn, D);
    if (S == 0) return FQ_OK;
    FQ_CHECK_ARG(msb && lsb && scale && out, FQ_ERR_ARG, "%s: null pointer", fn);
    FQ_CHECK_ARG(B <= 65535 && H <= 65535, FQ_ERR_ARG, "%s: B and H must be <= 65535", fn);
    dim3 grid((unsigned)((S + 3) / 4), (unsigned)H, (unsigned)B);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int epl = D >= 32 ? D / 32 : 1;
    count_launch();
#define FQ_D(E) turbo_dequant_kernel<E><<<grid, 128, 0, st>>>(msb, ms_sb, ms_sh, ms_ss, lsb, ls_sb, ls_sh, ls_ss, \
        static_cast<const uint16_t*>(scale), sc_sb, sc_sh, sc_ss, S, D, static_cast<uint16_t*>(out), o_sb, o_sh, o_ss)
    switch (epl) {
        case 1: FQ_D(1); break;
        case 2: FQ_D(2); break;
        case 4: FQ_D(4); break;
        case 8: FQ_D(8); break;
        case 16: FQ_D(16); break;
        default: FQ_D(32); break;
    }
#undef FQ_D
    FQ_CHECK_LAUNCH(fn);
    return FQ_OK;
}
