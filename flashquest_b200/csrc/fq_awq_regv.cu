// AWQ W4A16 linears for 1..8 rows of activations, group size 128: the decode step's projections.
//
// A launch moves 5-26 MB of weights (1-4 us of HBM time) in the middle of a chain of dependent launches, so what counts is
// that the weights are on their way before the input exists and that little happens after it does.  A warp owns ONE
// quantisation group (128 k) of 128 columns: 8 KiB of codes, requested by 32 8-byte loads per lane straight into registers
// BEFORE the dependency wait (weights never change) and used from there: no shared-memory ring, no barrier per stage.  The
// eight warps of a CTA are eight groups of the same columns, the CTAs of a cluster the remaining groups.
//   multiply: mma.m16n8k16, A = 16 columns x 16 k of codes, B = 16 k x 8 rows of x (fp16, exact).  Two words of neighbouring
//     k rows side by side (two byte permutes) give, masked in place, pairs of fp16 subnormals code * 2^-24 (odd nibbles
//     * 2^-20): 12 integer instructions per 16 codes, no conversion, exact products, fp32 sums.  One more MMA per step with
//     A = 1 sums x.
//   y += scale * (sum x*code - zero * sum x) once per group in fp32, then eight warps through shared memory, the cluster
//     through distributed shared memory, both in a fixed order; bias, fp16, rotary embedding and 16-byte stores by one CTA.
// Measured back to back in a graph, 28 layers of weights (before: shared-memory ring, lane-wise fp16 arithmetic), us for
// 3072 -> 5120 / 3072 -> 3072 / 3072 -> 16384 / 8192 -> 3072: 1 row 6.3 / 5.1 / 12.3 / 10.1 -> 5.4 / 5.2 / 12.6 / 7.6, 2 rows
// 8.7 / 6.2 / 15.2 / 12.4 -> 5.8 / 5.4 / 13.1 / 7.9, 8 rows 9.8 / 7.2 / 17.7 / 14.6 -> 7.6 / 7.0 / 15.2 / 9.5 (floors 1.3 / 0.8 / 4.1
// / 2.0).  Bound: 20-25 % by the fixed start, cluster exchange and finish (about 3.5 us), the rest by issue slots.
// The operator in front (add + RMSNorm, SwiGLU) is computed while x is staged, the rotary angles while the weights arrive.
#include "fq_awq_regv.cuh"

namespace fq {

constexpr int RV_THREADS = 256, RV_WARPS = 8, RV_TILE = 128, RV_GROUP = 128;
constexpr int RV_TOK = 164;             // floats per row of a warp's partial tile: 8 blocks of 16 + 4 columns, + 4: 16-byte stores hit all banks
constexpr int RV_XPAD = 16;             // halves behind a staged row: the fragment loads of 8 rows hit all banks

struct RvProj { const int32_t* qweight; const __half* scales; const int32_t* qzeros; const __half* bias; __half* y; int N, tile0, rope; };
struct RvParams {
    RvProj proj[RV_MAX_PROJ];
    const __half* x; int n_proj, M, K, n_groups, ks, passes, tiles_per_cta, tiles_total;
    int pro_kind; const __half* pro_b; const __half* pro_weight; float eps; __half* pro_out;
    const int* pos_dev; int pos; float theta; int head_dim;
};

__device__ __forceinline__ uint2 rv_ldg8(const void* p) {        // pinned in program order: requested before the dependency wait
    uint2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ uint4 rv_ldg16(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void rv_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// nibbles of two words (k rows a, b) as pairs (a, b) of fp16 subnormals; odd nibbles times 16
__device__ __forceinline__ void rv_pairs(uint32_t wa, uint32_t wb, uint32_t (&h)[8]) {
    const uint32_t x = __byte_perm(wa, wb, 0x5410), y = __byte_perm(wa, wb, 0x7632), x8 = x >> 8, y8 = y >> 8;
    h[0] = x & 0x000f000fu; h[1] = x & 0x00f000f0u; h[2] = x8 & 0x000f000fu; h[3] = x8 & 0x00f000f0u;
    h[4] = y & 0x000f000fu; h[5] = y & 0x00f000f0u; h[6] = y8 & 0x000f000fu; h[7] = y8 & 0x00f000f0u;
}

template <bool INTERLEAVED>
__global__ void __launch_bounds__(RV_THREADS, 2) awq_regv_kernel(const __grid_constant__ RvParams p) {
    extern __shared__ __align__(16) unsigned char rv_smem[];
    __shared__ float s_red[8][RV_WARPS];                        // sums of squares: CTA of the cluster, warp
    __shared__ __half2 s_cs[64];                                 // (cos, sin) of channel pair i
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int rank = blockIdx.x, tile_first = blockIdx.y * p.tiles_per_cta, n_tiles = min(p.tiles_per_cta, p.tiles_total - tile_first);
    const int M = p.M;
    const int range = RV_WARPS * p.passes * RV_GROUP;            // k positions of this CTA: groups rank*8*passes .. (contiguous)
    const int g_first = rank * RV_WARPS * p.passes, k_first = g_first * RV_GROUP;
    const int k_len = max(0, min(range, p.K - k_first));
    const int xstride = range + RV_XPAD;
    __half* s_x = reinterpret_cast<__half*>(rv_smem);            // [8][xstride]
    float* s_part = reinterpret_cast<float*>(rv_smem + (size_t)8 * xstride * 2);        // [8 warps][M][RV_TOK]
    float* s_recv = s_part + RV_WARPS * M * RV_TOK;              // [tile of the CTA][ks][M][128]
    __half* s_y = reinterpret_cast<__half*>(s_recv + p.tiles_per_cta * p.ks * M * RV_TILE);               // [M][128]
    if (p.ks > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");     // matched before the first remote store

    auto proj_of = [&](int tile) {
        int pj = 0;
#pragma unroll
        for (int i = 1; i < RV_MAX_PROJ; ++i)
            if (i < p.n_proj && tile >= p.proj[i].tile0) pj = i;
        return pj;
    };
    // ---- weights, scales and zeros of the first unit: on their way before the input exists ----
    uint2 w[8][4];
    uint4 sc[2];
    uint2 zw;
    // this lane's first word of a unit: k row 4t of the group, packs 2g and 2g + 1 of the tile
    auto unit_src = [&](int tile, int grp, int& npk) {
        const RvProj& P = p.proj[proj_of(tile)];
        npk = P.N >> 3;
        return P.qweight + (int64_t)(grp * RV_GROUP + 4 * t) * npk + (tile - P.tile0) * 16 + 2 * g;
    };
    auto load_meta = [&](int tile, int grp) {
        const RvProj& P = p.proj[proj_of(tile)];
        const int c0 = (tile - P.tile0) * RV_TILE + 16 * g;
        sc[0] = rv_ldg16(P.scales + (int64_t)grp * P.N + c0);
        sc[1] = rv_ldg16(P.scales + (int64_t)grp * P.N + c0 + 8);
        zw = rv_ldg8(P.qzeros + ((int64_t)grp * P.N + c0) / 8);
    };
    int grp = g_first + warp;
    if (grp < p.n_groups) {
        int npk;
        const int32_t* src = unit_src(tile_first, grp, npk);
#pragma unroll
        for (int s = 0; s < 8; ++s) {
#pragma unroll
            for (int j = 0; j < 4; ++j) w[s][j] = rv_ldg8(src + j * npk);
            src += 16 * npk;
        }
        load_meta(tile_first, grp);
    }
    // rows past the batch, and k positions past the end, multiply as zeros
    for (int i = tid; i < 8 * (range / 8); i += RV_THREADS) {
        const int m = i / (range / 8), k8 = (i - m * (range / 8)) * 8;
        if (m >= M || k8 >= k_len) *reinterpret_cast<uint4*>(s_x + m * xstride + k8) = make_uint4(0u, 0u, 0u, 0u);
    }
    pdl_wait();
    pdl_trigger();

    // ---- the CTA's k range of the input, through the operator in front of the linear ----
    union V8 { uint4 u; __half2 h[4]; };
    if (p.pro_kind == FQ_GEMV_ADD_RMSNORM) {
        // wr warps per row: h = x (+ b) of the CTA's own k range goes to shared memory; the sum of squares covers the whole
        // row.  From three rows on each CTA of the cluster sums its own range and they exchange the sums: reading whole rows
        // everywhere is 44 MB of L2 traffic per launch at 8 rows of 3072 (a batch-8 token 2497 -> 2406 us), while for one
        // row the exchange costs more than the 12 KB it saves (a single-row token 1983 -> 2020 us).
        const bool share = p.ks > 1 && M > 2;
        const int wr = M == 1 ? 8 : M == 2 ? 4 : M <= 4 ? 2 : 1, m = warp / wr, ws = warp - m * wr;
        const int k_lo = share ? k_first : 0, n8 = (share ? k_len : p.K) >> 3;
        float ss = 0.f;
        if (m < M) {
            const uint4* xa = reinterpret_cast<const uint4*>(p.x + (int64_t)m * p.K + k_lo);
            const uint4* xb = p.pro_b ? reinterpret_cast<const uint4*>(p.pro_b + (int64_t)m * p.K + k_lo) : nullptr;
#pragma unroll 4
            for (int k8 = ws * 32 + lane; k8 < n8; k8 += 32 * wr) {
                V8 a;
                a.u = __ldcg(xa + k8);
                if (xb) {
                    V8 b;
                    b.u = __ldcg(xb + k8);
#pragma unroll
                    for (int j = 0; j < 4; ++j) a.h[j] = __hadd2(a.h[j], b.h[j]);
                }
                const int kk = k_lo + 8 * k8 - k_first;
                if (kk >= 0 && kk < k_len) {
                    *reinterpret_cast<uint4*>(s_x + m * xstride + kk) = a.u;
                    if (p.pro_out && blockIdx.y == 0) *reinterpret_cast<uint4*>(p.pro_out + (int64_t)m * p.K + k_first + kk) = a.u;
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) { const float2 f = __half22float2(a.h[j]); ss = fmaf(f.x, f.x, ss); ss = fmaf(f.y, f.y, ss); }
            }
        }
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
        if (share) {
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");      // every CTA of the cluster runs
            if (lane < p.ks) {
                uint32_t at = (uint32_t)__cvta_generic_to_shared(&s_red[rank][warp]);
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(at), "r"(lane));
                asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(ss) : "memory");
            }
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        } else {
            if (lane == 0) s_red[0][warp] = ss;
            __syncthreads();
        }
        for (int i = tid; i < M * (k_len / 8); i += RV_THREADS) {
            const int r = i / (k_len / 8), k8 = i - r * (k_len / 8);
            float tot = 0.f;
            for (int c = 0; c < (share ? p.ks : 1); ++c)
                for (int j = 0; j < wr; ++j) tot += s_red[c][r * wr + j];
            const float inv = rsqrtf(tot / (float)p.K + p.eps);
            V8 a, wt;
            a.u = *reinterpret_cast<const uint4*>(s_x + r * xstride + 8 * k8);
            wt.u = __ldg(reinterpret_cast<const uint4*>(p.pro_weight + k_first) + k8);
#pragma unroll
            for (int j = 0; j < 4; ++j) { const float2 f = __half22float2(a.h[j]); a.h[j] = __hmul2(wt.h[j], __floats2half2_rn(f.x * inv, f.y * inv)); }
            *reinterpret_cast<uint4*>(s_x + r * xstride + 8 * k8) = a.u;
        }
    } else {
        for (int i = tid; i < M * (k_len / 8); i += RV_THREADS) {
            const int r = i / (k_len / 8), k8 = i - r * (k_len / 8);
            const int64_t o = (int64_t)r * p.K + k_first + 8 * k8;
            V8 a;
            a.u = __ldcg(reinterpret_cast<const uint4*>(p.x + o));
            if (p.pro_kind == FQ_GEMV_SWIGLU) {
                V8 b;
                b.u = __ldcg(reinterpret_cast<const uint4*>(p.pro_b + o));
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 f = __half22float2(a.h[j]);
                    a.h[j] = __hmul2(__floats2half2_rn(f.x / (1.0f + expf(-f.x)), f.y / (1.0f + expf(-f.y))), b.h[j]);
                }
                if (p.pro_out && blockIdx.y == 0) *reinterpret_cast<uint4*>(p.pro_out + o) = a.u;
            }
            *reinterpret_cast<uint4*>(s_x + r * xstride + 8 * k8) = a.u;
        }
    }
    if (p.head_dim) {
        // angles of the rotary embedding (Hugging Face's rotate_half convention), one position for all rows
        const int pos = p.pos_dev ? *p.pos_dev : p.pos, half = p.head_dim / 2;
        for (int i = tid; i < half; i += RV_THREADS) {
            const float inv_freq = 1.0f / powf(p.theta, (float)(2 * i) / (float)p.head_dim);
            const float ang = (float)pos * inv_freq;
            s_cs[i] = __floats2half2_rn(cosf(ang), sinf(ang));
        }
    }
    __syncthreads();
    if (p.ks > 1 && !(p.pro_kind == FQ_GEMV_ADD_RMSNORM && M > 2)) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");        // every CTA of the cluster runs

    float* part = s_part + (size_t)warp * M * RV_TOK;
    for (int u = 0; u < n_tiles; ++u) {
        const int tile = tile_first + u;
        for (int ps = 0; ps < p.passes; ++ps) {
            grp = g_first + ps * RV_WARPS + warp;
            // the unit behind this one: same tile, next pass, or the next tile
            const int ntile = ps + 1 < p.passes ? tile : tile + 1, ngrp = ps + 1 < p.passes ? grp + RV_WARPS : g_first + warp;
            const bool more = ngrp < p.n_groups && ntile < tile_first + n_tiles;
            int npk = 0;
            const int32_t* src = more ? unit_src(ntile, ngrp, npk) : nullptr;
            float acc[2][4][4], xs[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int f = 0; f < 4; ++f)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[m][f][e] = 0.f;
            const bool live = grp < p.n_groups;
            const __half* xrow = s_x + g * xstride + (ps * RV_WARPS + warp) * RV_GROUP + 4 * t;
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                if (live) {
                    const uint2 b = *reinterpret_cast<const uint2*>(xrow + 16 * s);
                    rv_mma(xs, 0x3c003c00u, 0x3c003c00u, 0x3c003c00u, 0x3c003c00u, b.x, b.y);
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        uint32_t h0[8], h1[8];
                        rv_pairs(m ? w[s][0].y : w[s][0].x, m ? w[s][1].y : w[s][1].x, h0);
                        rv_pairs(m ? w[s][2].y : w[s][2].x, m ? w[s][3].y : w[s][3].x, h1);
#pragma unroll
                        for (int f = 0; f < 4; ++f) rv_mma(acc[m][f], h0[f], h0[f + 4], h1[f], h1[f + 4], b.x, b.y);
                    }
                }
                if (more) {                                              // 16 k rows of the next unit into the registers just used
#pragma unroll
                    for (int j = 0; j < 4; ++j) w[s][j] = rv_ldg8(src + j * npk);
                    src += 16 * npk;
                }
            }
            // scale and zero once; columns in order, rows 2t and 2t + 1
            float y0[16], y1[16];
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                const uint32_t z = m ? zw.y : zw.x;
                const __half2* s2 = reinterpret_cast<const __half2*>(&sc[m]);
                float sf[8];
#pragma unroll
                for (int j = 0; j < 4; ++j) { const float2 f = __half22float2(s2[j]); sf[2 * j] = f.x; sf[2 * j + 1] = f.y; }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int col = INTERLEAVED ? (i & 3) * 2 + (i >> 2) : i;        // column of nibble i
                    const float s = live ? sf[col] : 0.f;
                    const float zero = __uint_as_float(((z >> (4 * i)) & 15u) | 0x4b000000u) - 8388608.0f;
                    const float sz = s * zero, sa = s * ((i & 1) ? 1048576.0f : 16777216.0f);        // 2^20, 2^24
                    y0[m * 8 + col] = fmaf(acc[m][i & 3][(i >> 2) * 2], sa, -sz * xs[0]);
                    y1[m * 8 + col] = fmaf(acc[m][i & 3][(i >> 2) * 2 + 1], sa, -sz * xs[1]);
                }
            }
            if (more) load_meta(ntile, ngrp);
            float4* d0 = reinterpret_cast<float4*>(part + (2 * t) * RV_TOK + g * 20);
            float4* d1 = reinterpret_cast<float4*>(part + (2 * t + 1) * RV_TOK + g * 20);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (2 * t < M) {
                    float4 v = make_float4(y0[4 * j], y0[4 * j + 1], y0[4 * j + 2], y0[4 * j + 3]);
                    if (ps > 0) { const float4 o = d0[j]; v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w; }
                    d0[j] = v;
                }
                if (2 * t + 1 < M) {
                    float4 v = make_float4(y1[4 * j], y1[4 * j + 1], y1[4 * j + 2], y1[4 * j + 3]);
                    if (ps > 0) { const float4 o = d1[j]; v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w; }
                    d1[j] = v;
                }
            }
        }
        __syncthreads();
        // ---- eight warps, then the cluster: CTA u % ks of the cluster finishes tile u ----
        const int owner = u % p.ks;
        for (int i = tid; i < M * 32; i += RV_THREADS) {
            const int m = i >> 5, c4 = i & 31;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int k = 0; k < RV_WARPS; ++k) {
                const float4 a = *reinterpret_cast<const float4*>(s_part + (k * M + m) * RV_TOK + (c4 >> 2) * 20 + (c4 & 3) * 4);
                v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
            }
            uint32_t at = (uint32_t)__cvta_generic_to_shared(s_recv + ((u * p.ks + rank) * M + m) * RV_TILE + c4 * 4);
            if (p.ks > 1) asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(at), "r"(owner));
            asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(at), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
        }
        if (u + 1 < n_tiles) __syncthreads();                            // s_part is used again
    }
    if (p.ks > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        __syncthreads();
    }
    for (int u = rank; u < n_tiles; u += p.ks) {
        const int tile = tile_first + u;
        const RvProj& P = p.proj[proj_of(tile)];
        const int c0 = (tile - P.tile0) * RV_TILE;
        if (P.rope && u != rank) __syncthreads();                        // s_y is used again
        for (int i = tid; i < M * 32; i += RV_THREADS) {
            const int m = i >> 5, c4 = (i & 31) * 4;
            float v[4] = {0.f, 0.f, 0.f, 0.f};
            for (int r = 0; r < p.ks; ++r) {
                const float4 a = *reinterpret_cast<const float4*>(s_recv + ((u * p.ks + r) * M + m) * RV_TILE + c4);
                v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
            }
            if (P.bias) {
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] += __half2float(P.bias[c0 + c4 + e]);
            }
            const __half2 h0 = __floats2half2_rn(v[0], v[1]), h1 = __floats2half2_rn(v[2], v[3]);
            const uint2 o = make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
            if (P.rope) *reinterpret_cast<uint2*>(s_y + m * RV_TILE + c4) = o;
            else *reinterpret_cast<uint2*>(P.y + (int64_t)m * P.N + c0 + c4) = o;
        }
        if (P.rope) {
            __syncthreads();
            const int half = p.head_dim / 2, hc = half / 4;              // 8-byte chunks per half head
            for (int i = tid; i < M * 16; i += RV_THREADS) {
                const int m = i >> 4, j = i & 15, lo = (j / hc) * 2 * hc + j % hc;
                union V4 { uint2 u; __half h[4]; } a, b;
                a.u = *reinterpret_cast<const uint2*>(s_y + m * RV_TILE + 4 * lo);
                b.u = *reinterpret_cast<const uint2*>(s_y + m * RV_TILE + 4 * (lo + hc));
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const __half2 cs = s_cs[(j % hc) * 4 + e];
                    const __half x1 = a.h[e], x2 = b.h[e];
                    a.h[e] = __hadd(__hmul(x1, __low2half(cs)), __hmul(__hneg(x2), __high2half(cs)));
                    b.h[e] = __hadd(__hmul(x2, __low2half(cs)), __hmul(x1, __high2half(cs)));
                }
                *reinterpret_cast<uint2*>(P.y + (int64_t)m * P.N + c0 + 4 * lo) = a.u;
                *reinterpret_cast<uint2*>(P.y + (int64_t)m * P.N + c0 + 4 * (lo + hc)) = b.u;
            }
        }
    }
}

static size_t rv_smem_bytes(int M, int passes, int ks, int tiles_per_cta) {
    const size_t range = (size_t)RV_WARPS * passes * RV_GROUP;
    return 8 * (range + RV_XPAD) * 2 + (size_t)RV_WARPS * M * RV_TOK * 4 + (size_t)tiles_per_cta * ks * M * RV_TILE * 4 + (size_t)M * RV_TILE * 2 + 16;
}

// K split: eight groups (one per warp) for each CTA of the cluster, several passes where eight CTAs are not enough
static void rv_shape(int n_groups, int* ks, int* passes) {
    int k = (n_groups + RV_WARPS - 1) / RV_WARPS;
    *passes = (k + 7) / 8;
    *ks = (n_groups + RV_WARPS * *passes - 1) / (RV_WARPS * *passes);
}

// Column tiles per CTA. One while all CTAs are resident at once (two per SM); two beyond that, so that the second
// tile's loads run under the first one's tensor-core work. 896 CTAs of one tile (4096 x 28672, one row) took 15.2 us,
// 448 of two 13.1, 300 of three 15.3, 224 of four 17.9: longer chains leave SMs idle at the end.
static int rv_tiles_per_cta(int tiles, int ks) { return tiles * ks > 2 * 148 ? 2 : 1; }

bool awq_regv_supported(const RegvCall& c) {
    if (c.group != RV_GROUP || c.K <= 0 || c.K % RV_GROUP || c.M < 1 || c.M > 8 || c.n_proj < 1 || c.n_proj > RV_MAX_PROJ || !aligned(c.x, 16)) return false;
    if (c.rope && c.rope->head_dim != 64 && c.rope->head_dim != 128) return false;
    for (int i = 0; i < c.n_proj; ++i)
        if (c.N[i] % RV_TILE || !aligned(c.qweight[i], 8) || !aligned(c.scales[i], 16) || !aligned(c.qzeros[i], 8) || !aligned(c.y[i], 16)) return false;
    int ks, passes, tiles = 0;
    rv_shape(c.K / RV_GROUP, &ks, &passes);
    for (int i = 0; i < c.n_proj; ++i) tiles += c.N[i] / RV_TILE;
    return rv_smem_bytes(c.M, passes, ks, rv_tiles_per_cta(tiles, ks)) <= 110 * 1024;
}

int awq_regv_launch(const RegvCall& c, void* stream, const char* fn) {
    RvParams p{};
    p.x = static_cast<const __half*>(c.x); p.n_proj = c.n_proj; p.M = c.M; p.K = c.K; p.n_groups = c.K / RV_GROUP;
    rv_shape(p.n_groups, &p.ks, &p.passes);
    p.pro_kind = FQ_GEMV_PLAIN;
    if (c.pro && c.pro->kind != FQ_GEMV_PLAIN) {
        p.pro_kind = c.pro->kind; p.pro_b = static_cast<const __half*>(c.pro->b); p.pro_weight = static_cast<const __half*>(c.pro->weight);
        p.eps = c.pro->eps; p.pro_out = static_cast<__half*>(c.pro->out);
    }
    if (c.rope) { p.pos_dev = c.rope->pos_dev; p.pos = c.rope->pos; p.theta = c.rope->theta; p.head_dim = c.rope->head_dim; }
    int tiles = 0;
    for (int i = 0; i < c.n_proj; ++i) {
        p.proj[i] = RvProj{c.qweight[i], static_cast<const __half*>(c.scales[i]), c.qzeros[i], static_cast<const __half*>(c.bias[i]), static_cast<__half*>(c.y[i]),
                           c.N[i], tiles, c.rope && ((c.rope->proj_mask >> i) & 1) ? 1 : 0};
        tiles += c.N[i] / RV_TILE;
    }
    for (int i = c.n_proj; i < RV_MAX_PROJ; ++i) p.proj[i] = RvProj{nullptr, nullptr, nullptr, nullptr, nullptr, 0, 1 << 30, 0};
    p.tiles_total = tiles;
    p.tiles_per_cta = rv_tiles_per_cta(tiles, p.ks);
    const size_t smem = rv_smem_bytes(c.M, p.passes, p.ks, p.tiles_per_cta);
    static std::atomic<uint64_t> reserved{0};                    // one bit per device
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (!(reserved.load(std::memory_order_relaxed) & bit)) {
        cudaError_t e = cudaFuncSetAttribute(awq_regv_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 110 * 1024);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(awq_regv_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 110 * 1024);
        if (e != cudaSuccess) return fail(FQ_ERR_CUDA, "%s: cannot reserve shared memory: %s", fn, cudaGetErrorString(e));
        reserved.fetch_or(bit, std::memory_order_relaxed);
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)p.ks, (unsigned)((tiles + p.tiles_per_cta - 1) / p.tiles_per_cta)); cfg.blockDim = dim3(RV_THREADS);
    cfg.dynamicSmemBytes = smem; cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute at[2]{};
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = p.ks; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = 2;
    cudaError_t e = c.interleaved ? cudaLaunchKernelEx(&cfg, awq_regv_kernel<true>, p) : cudaLaunchKernelEx(&cfg, awq_regv_kernel<false>, p);
    if (e != cudaSuccess) return fail(FQ_ERR_CUDA, "%s: launch failed: %s", fn, cudaGetErrorString(e));
    FQ_CHECK_LAUNCH(fn);
    return FQ_OK;
}

}  // namespace fq
