// AWQ W4A16 linears for 9 .. a few hundred rows on tcgen05: short prompts (up to one wave of tiles, or three while one tile
// holds all rows; beyond, the large GEMM in fq_awq_gemm.cu).
//
// y[M,N] = x[M,K] @ W with W in AutoAWQ's GEMM format.  The work is reading the weights (0.5 byte each) once; the grid of
// 256-column tiles of the large GEMM leaves most SMs idle at few rows (24 of 148 for 3072 columns) and its stages wait
// for the TMA latency.  Here a CTA owns 128 columns and up to 128 rows, and every kind of data has a ring as deep
// as its latency asks:
//   warp 0       raw weight tiles (128 k x 128 columns = 8 KiB) by TMA, the first ones before the dependency wait (weights
//                never change); scales and zeros by bulk copies
//   warp 2       x tiles by TMA (only the live rows are fetched; the MMA reads whatever lies behind them into rows that
//                nobody looks at, so stages of few rows overlap)
//   warp 1       tcgen05.mma M 128 (rows) x N 128 x K 16 into one TMEM accumulator
//   warps 4 ..   weights to fp16, (code - zero) * scale rounded once like the large GEMM: one shift, four three-input logic
//                operations, four exact subtractions (an odd nibble's factor of 16 goes with an fma) and four products per
//                8 weights; groups of four warps take turns.  Then the accumulator, bias, fp16, 16-byte stores.
// The K range is not split: one chain of products in k order gives the bits of the large GEMM, so a prompt's cache does not
// depend on which kernel its length picks (tests/test_gpu_awq_rows.py).  (Split over a cluster the 16-row linears took 48 us a
// layer instead of 82, but a last-bit difference moves 4-bit codes of the cache a few layers on.)  Bound by the chain itself: 8 MMAs of 64 cycles and their waits per block of 128 k.
// 3072 -> 5120 / 3072 / 16384 and 8192 -> 3072, 16 rows, us: large GEMM 41 / 41 / 42 / 100, here 13.5 / 13.4 / 17.7 / 33.4.
#include "fq_awq_skinny.cuh"

#include <cuda.h>

namespace fq {

constexpr int SK_BN = 128, SK_BK = 128;            // k block: the synchronisation of a block costs about 600 cycles whatever its length
constexpr int SK_RAW = SK_BK * SK_BN / 2;          // 8 KiB of codes per k block
constexpr int SK_A = SK_BK * SK_BN * 2;            // 32 KiB dequantised
constexpr int SK_MAX_RAW = 9;                     // ring depth limit
constexpr unsigned SK_SPIN_LIMIT = 1u << 26;

struct SkProj { const __half* scales; const int32_t* qzeros; const __half* bias; __half* y; int N, tile0; };
struct SkParams {
    SkProj proj[SK_MAX_PROJ];
    int n_proj, M, K, group, n_groups, raw_stages;
    int* status;
};

__device__ __forceinline__ uint32_t sk_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void sk_init(uint64_t* bar, unsigned count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sk_smem(bar)), "r"(count)); }
__device__ __forceinline__ void sk_expect(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sk_smem(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void sk_arrive(uint64_t* bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sk_smem(bar)) : "memory"); }
__device__ __forceinline__ bool sk_wait(uint64_t* bar, unsigned parity) {        // bounded; false = gave up
    for (unsigned spins = 0; spins <= SK_SPIN_LIMIT; ++spins) {
        unsigned ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(sk_smem(bar)), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}
__device__ __forceinline__ bool sk_any_timeout(uint64_t* bar, unsigned parity) { return __any_sync(0xffffffffu, !sk_wait(bar, parity)); }
__device__ __forceinline__ void sk_tma(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(sk_smem(dst)), "l"(map), "r"(sk_smem(bar)), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void sk_bulk(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(sk_smem(dst)), "l"(src), "r"(bytes), "r"(sk_smem(bar)) : "memory");
}
__device__ __forceinline__ void sk_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ bool sk_elect() {
    uint32_t pred;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(pred));
    return pred != 0;
}
__device__ __forceinline__ void sk_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(sk_smem(bar)) : "memory");
}
__device__ __forceinline__ uint64_t sk_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {      // 128-byte swizzle
    return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)((lbo >> 4) & 0x3fff) << 16) | ((uint64_t)((sbo >> 4) & 0x3fff) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void sk_ld8(uint32_t taddr, uint32_t* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(taddr));
}
// TN: rows of x per CTA (16 .. 128)
template <int TN> struct SkCfg {
    static constexpr int COLS = SK_BN / 2;                          // columns per epilogue thread
    static constexpr int STAGES = TN > 64 ? 2 : 3;                  // dequantised weights
    // Groups of four warps that dequantise, one k block each in turn: as many as stages.  With more, a group could come back to
    // a stage two of its phases ahead, which a parity wait cannot see; the raw ring is a multiple of it for the same reason.
    static constexpr int GROUPS = STAGES;
    static constexpr int THREADS = (4 + 4 * GROUPS) * 32;
    static constexpr int X_STAGES = 3;                              // an x tile arrives about 1 us after its request
    static constexpr int X_HALF = TN * 64 * 2;                      // bytes per 64 k (one 128-byte row per row of x)
    static constexpr int X_TILE = 2 * X_HALF;                       // bytes per k block
    static constexpr int X_BYTES = (2 * X_STAGES - 1) * X_HALF + 128 * 64 * 2;
    static constexpr int TMEM_COLS = SK_BN;
};
constexpr int SK_DEQ_GROUP = 4;                    // warps that dequantise one k block

template <bool INTERLEAVED, int TN>
__global__ void __launch_bounds__(SkCfg<TN>::THREADS, 1) awq_skinny_kernel(
    const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1,
    const __grid_constant__ CUtensorMap map_w2, const __grid_constant__ CUtensorMap map_w3, const __grid_constant__ SkParams p) {
    using C = SkCfg<TN>;
    constexpr int AS = C::STAGES, XS = C::X_STAGES;
    constexpr int DEQ0 = 4;
    extern __shared__ unsigned char sk_raw_smem[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(sk_raw_smem) + 1023) & ~(uintptr_t)1023);
    unsigned char* sW = base;
    unsigned char* sX = sW + AS * SK_A;
    unsigned char* sRaw = sX + C::X_BYTES;
    unsigned char* sMeta = sRaw + p.raw_stages * SK_RAW;            // per group: 128 scales fp16, 16 zero words
    float* sOut = reinterpret_cast<float*>(base);                   // [row][128] fp32, over the pipeline buffers at the end
    __shared__ uint64_t full_raw[SK_MAX_RAW], empty_raw[SK_MAX_RAW], a_ready[AS], a_empty[AS], x_full[XS], x_empty[XS], acc_ready, meta_full;
    __shared__ uint32_t tmem_slot;

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int row0 = blockIdx.y * TN;
    const int gpk = p.group / SK_BK;                                 // k blocks per group
    const int ng = p.n_groups, nkb = ng * gpk;
    int pj = 0;
#pragma unroll
    for (int i = 1; i < SK_MAX_PROJ; ++i)
        if (i < p.n_proj && (int)blockIdx.x >= p.proj[i].tile0) pj = i;
    const SkProj& P = p.proj[pj];
    const int n0 = ((int)blockIdx.x - P.tile0) * SK_BN;
    const int rows = min(TN, p.M - row0);                            // live rows of this tile
    bool failed = false;

    if (tid == 0) {
        for (int i = 0; i < p.raw_stages; ++i) { sk_init(&full_raw[i], 1); sk_init(&empty_raw[i], SK_DEQ_GROUP); }
        for (int i = 0; i < AS; ++i) { sk_init(&a_ready[i], SK_DEQ_GROUP); sk_init(&a_empty[i], 1); }
        for (int i = 0; i < XS; ++i) { sk_init(&x_full[i], 1); sk_init(&x_empty[i], 1); }
        sk_init(&acc_ready, 1);
        sk_init(&meta_full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sk_smem(&tmem_slot)), "r"(C::TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;

    if (warp == 0) {
        // =========================== weight producer ===========================
        const CUtensorMap* map_w = pj == 0 ? &map_w0 : (pj == 1 ? &map_w1 : (pj == 2 ? &map_w2 : &map_w3));
        const int nb = n0 / 8, depth = min(p.raw_stages, nkb);
        if (sk_elect()) {
            for (int kb = 0; kb < depth; ++kb) {
                sk_expect(&full_raw[kb], SK_RAW);
                sk_tma(sRaw + kb * SK_RAW, map_w, nb, kb * SK_BK, &full_raw[kb]);
            }
            sk_expect(&meta_full, (unsigned)ng * 320u);
        }
        __syncwarp();
        for (int g = lane; g < ng; g += 32) {
            sk_bulk(sMeta + g * 320, P.scales + (int64_t)g * P.N + n0, 256, &meta_full);
            sk_bulk(sMeta + g * 320 + 256, P.qzeros + ((int64_t)g * P.N + n0) / 8, 64, &meta_full);
        }
        __syncwarp();
        int s = 0;
        unsigned ph = 0u;
        for (int kb = depth; kb < nkb; ++kb) {
            if (sk_any_timeout(&empty_raw[s], ph)) {
                failed = true;
                for (int i = kb - p.raw_stages; i < kb; ++i) sk_wait(&full_raw[i % p.raw_stages], (unsigned)(i / p.raw_stages) & 1u);   // copies in flight
                break;
            }
            if (sk_elect()) {
                sk_expect(&full_raw[s], SK_RAW);
                sk_tma(sRaw + s * SK_RAW, map_w, nb, kb * SK_BK, &full_raw[s]);
            }
            __syncwarp();
            if (++s == p.raw_stages) { s = 0; ph ^= 1u; }
        }
    } else if (warp == 1) {
        // =========================== MMA issuer ===========================
        // The whole warp walks the loop and one elected lane issues: descriptors of warp-uniform values stay in uniform
        // registers.  Inside a branch on lane == 0 every operand went through vector registers and an issue took 90 cycles.
        // fp32 accumulators, fp16 A (x, K-major) and B (weights, MN-major), M = N = 128
        constexpr uint32_t idesc = (1u << 4) | (1u << 16) | ((uint32_t)(SK_BN >> 3) << 17) | (8u << 24);
        // A: 8 rows x 64 k per 1 KiB atom, 16 k = 32 B further inside the swizzled row; B: 64 columns x 8 k per 1 KiB atom, atoms
        // 1 KiB apart along k and BK * 128 B apart along the columns
        const uint64_t da0 = sk_desc(sk_smem(sX), 16, 1024), db0 = sk_desc(sk_smem(sW), SK_BK * 128, 1024);
        constexpr int XH = C::X_HALF >> 4;
        for (int kb = 0; kb < nkb; ++kb) {
            const int s = kb % AS, xs = kb % XS;
            if (sk_any_timeout(&a_ready[s], (unsigned)(kb / AS) & 1u) || sk_any_timeout(&x_full[xs], (unsigned)(kb / XS) & 1u)) { failed = true; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t da = da0 + (uint64_t)(xs * (C::X_TILE >> 4)), db = db0 + (uint64_t)(s * (SK_A >> 4));
            if (sk_elect()) {
#pragma unroll
                for (int k = 0; k < SK_BK / 16; ++k) sk_mma(tmem, da + (k >> 2) * XH + (k & 3) * (32 >> 4), db + k * (2048 >> 4), idesc, (kb | k) != 0 ? 1u : 0u);
                sk_commit(&a_empty[s]);
                sk_commit(&x_empty[xs]);
                if (kb + 1 == nkb) sk_commit(&acc_ready);
            }
            __syncwarp();
        }
    } else if (warp == 3) {
        // (fills the warpgroup)
    } else if (warp == 2) {
        // =========================== x producer ===========================
        pdl_wait();
        pdl_trigger();
        for (int kb = 0; kb < nkb; ++kb) {
            const int s = kb % XS;
            if (kb >= XS && sk_any_timeout(&x_empty[s], (unsigned)(kb / XS - 1) & 1u)) { failed = true; break; }
            if (sk_elect()) {
                sk_expect(&x_full[s], C::X_TILE);
                sk_tma(sX + s * C::X_TILE, &map_x, kb * SK_BK, row0, &x_full[s]);
                sk_tma(sX + s * C::X_TILE + C::X_HALF, &map_x, kb * SK_BK + 64, row0, &x_full[s]);
            }
            __syncwarp();
        }
    } else {
        // =========================== weights to fp16 ===========================
        const int grp = (warp - DEQ0) / SK_DEQ_GROUP, t = (tid - DEQ0 * 32) % (SK_DEQ_GROUP * 32);
        const int c = t & 15, kr0 = t >> 4;                           // pack of 8 columns; k rows kr0 + 8 i
        const int chunk = c & 7;
        if (sk_any_timeout(&meta_full, 0u)) failed = true;
        int r = grp % p.raw_stages;
        unsigned rph = (unsigned)(grp / p.raw_stages) & 1u;
        for (int kb = grp; kb < nkb && !failed; kb += C::GROUPS) {
            const int s = kb % AS;
            // per column pair: even nibbles h = 1024 + code, minus (1024 + zero); odd ones h = 1024 + 16 code, times 1/16 minus
            // (64 + zero): both exact; then the scale, rounded once
            __half2 zs[4], sc[4];
            {
                const unsigned char* meta = sMeta + (kb / gpk) * 320;
                const uint32_t zw = *reinterpret_cast<const uint32_t*>(meta + 256 + 4 * c);
                const uint4 s4 = *reinterpret_cast<const uint4*>(meta + 16 * c);
                const uint32_t sw[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const uint32_t z = ((zw >> (4 * q)) & 0x000f000fu) | 0x64006400u;
                    zs[q] = __hsub2((q & 1) ? __float2half2_rn(960.0f) : __float2half2_rn(0.0f), *reinterpret_cast<const __half2*>(&z));
                    if constexpr (INTERLEAVED) sc[q] = *reinterpret_cast<const __half2*>(&sw[q]);        // columns (2q, 2q + 1)
                    else {                                                                               // columns (q, q + 4)
                        const __half* h = reinterpret_cast<const __half*>(sw);
                        sc[q] = __halves2half2(h[q], h[q + 4]);
                    }
                }
            }
            const __half2 sixteenth = __float2half2_rn(0.0625f);
            if (sk_any_timeout(&full_raw[r], rph)) { failed = true; break; }
            const uint32_t* raw = reinterpret_cast<const uint32_t*>(sRaw + r * SK_RAW) + kr0 * 16 + c;
            uint32_t w[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) w[i] = raw[128 * i];
            if (kb >= AS && sk_any_timeout(&a_empty[s], (unsigned)(kb / AS - 1) & 1u)) { failed = true; break; }
            unsigned char* at = sW + s * SK_A + (c >> 3) * (SK_BK * 128);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int kr = kr0 + 8 * i;
                uint32_t o[4];
                const uint32_t w8 = w[i] >> 8;
                o[0] = (w[i] & 0x000f000fu) | 0x64006400u;
                o[1] = (w[i] & 0x00f000f0u) | 0x64006400u;
                o[2] = (w8 & 0x000f000fu) | 0x64006400u;
                o[3] = (w8 & 0x00f000f0u) | 0x64006400u;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const __half2 h = *reinterpret_cast<const __half2*>(&o[q]);
                    const __half2 d = __hmul2((q & 1) ? __hfma2(h, sixteenth, zs[q]) : __hadd2(h, zs[q]), sc[q]);
                    o[q] = *reinterpret_cast<const uint32_t*>(&d);
                }
                uint4 out;
                if constexpr (INTERLEAVED) out = make_uint4(o[0], o[1], o[2], o[3]);                 // columns (2q, 2q + 1)
                else out = make_uint4(__byte_perm(o[0], o[1], 0x5410), __byte_perm(o[2], o[3], 0x5410),   // pairs (q, q + 4)
                                      __byte_perm(o[0], o[1], 0x7632), __byte_perm(o[2], o[3], 0x7632));
                *reinterpret_cast<uint4*>(at + kr * 128 + ((chunk ^ (kr & 7)) << 4)) = out;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) { sk_arrive(&a_ready[s]); sk_arrive(&empty_raw[r]); }      // (the raw tile not before its values have been used)
            for (int i = 0; i < C::GROUPS; ++i)
                if (++r == p.raw_stages) { r = 0; rph ^= 1u; }
        }
        // ---- the accumulator ----
        if (warp < DEQ0 + 8) {
            if (sk_any_timeout(&acc_ready, 0u)) failed = true;       // every product is done, so the pipeline buffers are free
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int lq = warp & 3, part = (warp - DEQ0) >> 2, row = lq * 32 + lane;      // TMEM lane quarter (rows), half of the columns
            constexpr int RS = SK_BN + 4;                            // row stride (floats): 16-byte stores of 8 lanes hit all banks
            __syncwarp();
            if (lq * 32 < rows) {
                uint32_t acc[C::COLS];
#pragma unroll
                for (int c = 0; c < C::COLS / 8; ++c) sk_ld8(tmem + ((uint32_t)(lq * 32) << 16) + (uint32_t)(part * C::COLS + c * 8), acc + 8 * c);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (row < rows) {
#pragma unroll
                    for (int i = 0; i < C::COLS; i += 4)
                        *reinterpret_cast<uint4*>(sOut + row * RS + part * C::COLS + i) = make_uint4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
                }
            }
            __syncwarp();
            asm volatile("bar.sync 1, 256;" ::: "memory");
            __half* yb = P.y + (int64_t)row0 * P.N + n0;
            for (int i = tid - DEQ0 * 32; i < rows * 16; i += 256) {
                const int r = i >> 4, c8 = (i & 15) * 8;
                const float4 a = *reinterpret_cast<const float4*>(sOut + r * RS + c8), b = *reinterpret_cast<const float4*>(sOut + r * RS + c8 + 4);
                float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
                if (P.bias) {
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[e] += __half2float(P.bias[n0 + c8 + e]);
                }
                uint32_t o[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) { const __half2 h = __floats2half2_rn(v[2 * e], v[2 * e + 1]); o[e] = *reinterpret_cast<const uint32_t*>(&h); }
                *reinterpret_cast<uint4*>(yb + (int64_t)r * P.N + c8) = make_uint4(o[0], o[1], o[2], o[3]);
            }
        }
    }

    if (failed) atomicExch(p.status, FQ_ERR_TIMEOUT);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::TMEM_COLS) : "memory");
}

typedef CUresult (*SkEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                               const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static SkEncodeFn sk_encode_fn() {
    static std::atomic<void*> cached{nullptr};
    void* fn = cached.load(std::memory_order_relaxed);
    if (fn == nullptr) {
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess || qres != cudaDriverEntryPointSuccess) return nullptr;
        cached.store(fn, std::memory_order_relaxed);
    }
    return reinterpret_cast<SkEncodeFn>(fn);
}

bool awq_skinny_supported(const SkinnyCall& c) {
    if (!(c.group == 128 || c.group == 256) || c.K <= 0 || c.K % c.group || c.n_proj < 1 || c.n_proj > SK_MAX_PROJ || c.M < 1) return false;
    if (!aligned(c.x, 16) || (int64_t)(c.K / c.group) * 320 > 40 * 1024) return false;
    for (int i = 0; i < c.n_proj; ++i)
        if (c.N[i] % SK_BN || !aligned(c.qweight[i], 16) || !aligned(c.scales[i], 16) || !aligned(c.qzeros[i], 16) || !aligned(c.y[i], 16)) return false;
    return true;
}

template <bool IL, int TN>
static int sk_launch(const SkinnyCall& c, SkParams& p, const CUtensorMap* maps, int tiles, cudaStream_t st, const char* fn) {
    using C = SkCfg<TN>;
    const int m_tiles = (c.M + TN - 1) / TN;
    const int nkb = p.n_groups * (p.group / SK_BK), rows = c.M < TN ? c.M : TN;
    const int fixed = C::STAGES * SK_A + C::X_BYTES + p.n_groups * 320;
    int raw = (220 * 1024 - fixed) / SK_RAW;
    raw = (raw > SK_MAX_RAW ? SK_MAX_RAW : raw) / C::GROUPS * C::GROUPS;      // at least one per group: awq_skinny_supported bounds K
    p.raw_stages = raw > nkb ? nkb : raw;
    const int pipe = fixed + p.raw_stages * SK_RAW, out = rows * (SK_BN + 4) * 4;
    const int smem = (out > pipe ? out : pipe) + 1024;
    static std::atomic<uint64_t> reserved{0};                        // per instantiation, one bit per device
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (!(reserved.load(std::memory_order_relaxed) & bit)) {
        cudaError_t e = cudaFuncSetAttribute(awq_skinny_kernel<IL, TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024);
        if (e != cudaSuccess) return fail(FQ_ERR_CUDA, "%s: cannot reserve shared memory: %s", fn, cudaGetErrorString(e));
        reserved.fetch_or(bit, std::memory_order_relaxed);
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)tiles, (unsigned)m_tiles); cfg.blockDim = dim3(C::THREADS);
    cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at; cfg.numAttrs = 1;
    count_launch();
    cudaError_t e = cudaLaunchKernelEx(&cfg, awq_skinny_kernel<IL, TN>, maps[0], maps[1], maps[2], maps[3], maps[4], p);
    if (e != cudaSuccess) return fail(FQ_ERR_CUDA, "%s: launch failed: %s", fn, cudaGetErrorString(e));
    FQ_CHECK_LAUNCH(fn);
    return FQ_OK;
}

template <bool IL>
static int sk_launch_tn(const SkinnyCall& c, SkParams& p, const CUtensorMap* maps, int tn, int tiles, cudaStream_t st, const char* fn) {
    switch (tn) {
        case 16: return sk_launch<IL, 16>(c, p, maps, tiles, st, fn);
        case 32: return sk_launch<IL, 32>(c, p, maps, tiles, st, fn);
        case 64: return sk_launch<IL, 64>(c, p, maps, tiles, st, fn);
        default: return sk_launch<IL, 128>(c, p, maps, tiles, st, fn);
    }
}

int awq_skinny_launch(const SkinnyCall& c, void* stream, const char* fn) {
    SkEncodeFn encode = sk_encode_fn();
    if (!encode) return fail(FQ_ERR_CUDA, "%s: the driver does not export cuTensorMapEncodeTiled", fn);
    SkParams p{};
    p.n_proj = c.n_proj; p.M = c.M; p.K = c.K; p.group = c.group; p.n_groups = c.K / c.group;
    p.status = device_status_ptr();
    if (p.status == nullptr) return FQ_ERR_CUDA;
    const int tn = c.M <= 16 ? 16 : c.M <= 32 ? 32 : c.M <= 64 ? 64 : 128;
    CUtensorMap maps[1 + SK_MAX_PROJ];
    int tiles = 0;
    for (int i = 0; i < c.n_proj; ++i) {
        p.proj[i] = SkProj{static_cast<const __half*>(c.scales[i]), c.qzeros[i], static_cast<const __half*>(c.bias[i]), static_cast<__half*>(c.y[i]),
                           c.N[i], tiles};
        tiles += c.N[i] / SK_BN;
        const cuuint64_t dims[2] = {(cuuint64_t)(c.N[i] / 8), (cuuint64_t)c.K};
        const cuuint64_t strides[1] = {(cuuint64_t)(c.N[i] / 8) * 4};
        const cuuint32_t box[2] = {SK_BN / 8, SK_BK}, es[2] = {1, 1};
        const CUresult r = encode(&maps[1 + i], CU_TENSOR_MAP_DATA_TYPE_INT32, 2, const_cast<int32_t*>(c.qweight[i]), dims, strides, box, es,
                                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return fail(FQ_ERR_CUDA, "%s: tensor map for qweight[%d]: driver error %d", fn, i, (int)r);
    }
    for (int i = c.n_proj; i < SK_MAX_PROJ; ++i) { maps[1 + i] = maps[1]; p.proj[i] = SkProj{nullptr, nullptr, nullptr, nullptr, 0, 1 << 30}; }
    {
        const cuuint64_t dims[2] = {(cuuint64_t)c.K, (cuuint64_t)c.M};
        const cuuint64_t strides[1] = {(cuuint64_t)c.K * 2};
        const cuuint32_t box[2] = {64, (cuuint32_t)tn}, es[2] = {1, 1};
        const CUresult r = encode(&maps[0], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(c.x), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return fail(FQ_ERR_CUDA, "%s: tensor map for x: driver error %d", fn, (int)r);
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return c.interleaved ? sk_launch_tn<true>(c, p, maps, tn, tiles, st, fn) : sk_launch_tn<false>(c, p, maps, tn, tiles, st, fn);
}

}  // namespace fq
