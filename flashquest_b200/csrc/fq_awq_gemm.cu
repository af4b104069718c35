// AWQ W4A16 dequant-GEMM on the 5th-generation tensor cores (tcgen05) for prefill / batched
// shapes: y[M,N] = x[M,K] @ W, W in AutoAWQ's GEMM format (4-bit codes, group scales and zeros).
// The M <= 8 decode shapes stay with the GEMV (fq_awq_gemv.cu), short prompts with fq_awq_skinny.cu; this kernel is the
// dense contraction of the prefill branch (the q/k/v/o/gate/up/down linears over all prompt tokens).
//
// Two CTAs on neighbouring SMs (a cluster) multiply one 256 x 256 tile together (cta_group::2): each holds 128 rows of x,
// dequantises 128 of the 256 columns of W and accumulates its own 128 rows of all 256 columns in its tensor memory.  The
// pair reads what one CTA with a 256 x 256 tile of its own reads, but a tile is half the time of an SM, so that the last
// wave of tiles costs half, and two accumulator sets fit, so that a finished tile is drained while the next one is
// multiplied.  A CTA is persistent and walks K in steps of 64:
//   warp 0       : TMA producer: 128 rows x 64 k of x (fp16, 128-byte swizzle, K-major), counted on the first CTA's
//                  barrier, and the raw weight tile of 64 k x 16 int32;
//   warp 1       : in the first CTA, one lane issues tcgen05.mma (M 256, N 256, K 16, fp16 x fp16 -> fp32 in TMEM),
//                  four per step, commits the stages back to both producers and the accumulator set to both epilogues;
//                  in both, the warp owns the tensor-memory allocation (512 columns);
//   warps 2..13  : three groups that take turns dequantise the raw tile to fp16 in shared memory, (code - zero) * scale rounded
//                  once to fp16 like the reference's GEMM kernels, written N-contiguous in the
//                  canonical MN-major 128-byte-swizzle layout (AWQ's nibble order makes every
//                  masked word a pair of neighbouring columns, so a 32-bit word of codes becomes one
//                  16-byte store);
//   warps 14..17 : epilogue — drain an accumulator set (tcgen05.ld, lane quarter = warp id mod 4),
//                  add the bias, convert to fp16, store y, hand the set back.
// Stages and accumulator sets are handed over through mbarriers (TMA bytes -> dequantised ->
// consumed; multiplied -> drained), those the first CTA's MMA warp waits for with arrivals from both CTAs; every wait is
// bounded in time and reports through the device status word instead of spinning forever.
//
// Bound by the tensor pipe inside a tile and by the last wave of tiles.  With one CTA per 256 x 256 tile (one accumulator
// set, drained before the next tile began) the Llama-3.2-3B linears (q/k/v, o, gate/up, down) took 139 / 100 / 317 / 263 us at
// 4096 rows, in pairs 111 / 70 / 311 / 177 (1327 TFLOP/s for gate/up, of 1392 that cuBLAS holds under the power cap).  Three
// groups of four dequantising warps: with two (4 to 6 weight stages) the pair waited for them, 751 us for the four against 669;
// four groups are no faster (677).
#include <cuda.h>

#include "fq_awq_skinny.cuh"

namespace fq {

constexpr int GM_BM = 128;          // rows of x per CTA, 256 per pair
constexpr int GM_BN = 256;          // columns per pair
constexpr int GM_CN = 128;          // columns whose weights a CTA dequantises
constexpr int GM_BK = 64;
constexpr int GM_ACC_SETS = 2;      // of 256 fp32 columns: all of an SM's tensor memory
constexpr int GM_TMEM_COLS = 512;
constexpr int GM_DEQ_WARPS = 12;
constexpr int GM_DEQ_GROUP = 4;     // warps that convert one k block
constexpr int GM_EPI_WARPS = 4;
constexpr int GM_THREADS = (2 + GM_DEQ_WARPS + GM_EPI_WARPS) * 32;     // TMA warp, MMA warp, dequantise warps, epilogue warps

constexpr int GM_MAX_PROJ = 4;
constexpr int GM_X_BYTES = GM_BM * GM_BK * 2;             // 16 KiB
constexpr int GM_RAW_BYTES = GM_BK * (GM_CN / 8) * 4;     // 4 KiB
constexpr int GM_B_BYTES = GM_BK * GM_CN * 2;             // 16 KiB
// a ring for each kind of data, as deep as its latency asks: x tiles and raw codes come about 1 us after their request, four
// k blocks; a dequantised tile only has to bridge the MMAs of one block
constexpr int GM_X_STAGES = 5, GM_B_STAGES = 6, GM_RAW_STAGES = 9;
constexpr int GM_SMEM = GM_X_STAGES * GM_X_BYTES + GM_B_STAGES * GM_B_BYTES + GM_RAW_STAGES * GM_RAW_BYTES + 1024 /* alignment slack */ + 512 /* barriers, tmem address */;
static_assert((2 * (GM_X_STAGES + GM_B_STAGES + GM_RAW_STAGES) + 2 * GM_ACC_SETS) * 8 + 4 <= 512, "barrier block");
static_assert(GM_SMEM <= 227 * 1024, "shared memory");

struct GemmProj {
    const __half* scales; const int32_t* qzeros; const __half* bias; __half* y;
    int N, tile0;       // output columns; first N tile of this projection in the grid
};
struct GemmParams {
    GemmProj proj[GM_MAX_PROJ];
    int n_proj, M, K, group;
    int n_tiles, m_tiles;   // N tiles over all projections, M tiles of 256 rows
    int* status;
};

__device__ __forceinline__ uint32_t gm_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void gm_mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(gm_smem(bar)), "r"(count));
}
__device__ __forceinline__ void gm_mbar_expect_tx(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(gm_smem(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void gm_mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(gm_smem(bar)) : "memory");
}
// the address of the first CTA's copy of a barrier
__device__ __forceinline__ uint32_t gm_first(uint64_t* bar) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(gm_smem(bar)));
    return a;
}
__device__ __forceinline__ void gm_arrive_first(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(gm_first(bar)) : "memory");
}
__device__ __forceinline__ bool gm_mbar_try(uint64_t* bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(gm_smem(bar)), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t gm_now() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
// bounded wait (two seconds); false = gave up
__device__ __forceinline__ bool gm_wait(uint64_t* bar, unsigned parity) {
    if (gm_mbar_try(bar, parity)) return true;
    const uint64_t end = gm_now() + 2000000000ull;
    for (unsigned spins = 1; !gm_mbar_try(bar, parity); ++spins)
        if ((spins & 63u) == 0 && gm_now() > end) return false;
    return true;
}
// the same for a whole warp; true = gave up
__device__ __forceinline__ bool gm_timeout(uint64_t* bar, unsigned parity) { return __any_sync(0xffffffffu, !gm_wait(bar, parity)); }
__device__ __forceinline__ bool gm_elect() {
    uint32_t pred;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(pred));
    return pred != 0;
}
__device__ __forceinline__ void gm_tma_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(gm_smem(dst)), "l"(map), "r"(gm_smem(bar)), "r"(x), "r"(y) : "memory");
}
// into this CTA's shared memory, the bytes counted on a barrier of the pair's first CTA
__device__ __forceinline__ void gm_tma_2d_pair(void* dst, const CUtensorMap* map, int x, int y, uint32_t first_bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(gm_smem(dst)), "l"(map), "r"(first_bar), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void gm_mma(uint32_t tmem_c, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_c), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
// arrive on both CTAs' copies of the barrier when the MMAs issued so far have completed
__device__ __forceinline__ void gm_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(gm_smem(bar)), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void gm_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared-memory matrix descriptor, 128-byte swizzle, version 1 (sm_100); offsets in bytes
__device__ __forceinline__ uint64_t gm_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    return (uint64_t)((smem_addr >> 4) & 0x3fff) | ((uint64_t)((lbo_bytes >> 4) & 0x3fff) << 16) |
           ((uint64_t)((sbo_bytes >> 4) & 0x3fff) << 32) | (1ull << 46) | (2ull << 61);
}
// 32 fp32 columns of this warp's lane quarter
__device__ __forceinline__ void gm_tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
}

// SWIGLU: projection 0 is the gate, 1 the up projection of the same width, and y (of projection 0) becomes
// fp16(silu(gate)) * up of the fp16-rounded products, the arithmetic of fq_swiglu.  A tile is 128 columns of each: the first
// CTA dequantises the gate's, the second the up projection's, and every row of both lies in one CTA's accumulators.
template <bool INTERLEAVED, bool SWIGLU>
__global__ void __launch_bounds__(GM_THREADS, 1) awq_gemm_kernel(
    const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1,
    const __grid_constant__ CUtensorMap map_w2, const __grid_constant__ CUtensorMap map_w3, const GemmParams p) {
    constexpr int XS = GM_X_STAGES, BS = GM_B_STAGES, RS = GM_RAW_STAGES;
    extern __shared__ unsigned char gm_raw_smem[];
    // x tiles | dequantised weights | raw codes; every tile 1024-byte aligned (the same offsets in both CTAs)
    unsigned char* base = gm_raw_smem + ((1024u - (gm_smem(gm_raw_smem) & 1023u)) & 1023u);
    unsigned char* sX = base;
    unsigned char* sB = sX + XS * GM_X_BYTES;
    unsigned char* sRaw = sB + BS * GM_B_BYTES;
    uint64_t* x_full = reinterpret_cast<uint64_t*>(sRaw + RS * GM_RAW_BYTES);   // first CTA: both CTAs' x tiles have arrived
    uint64_t* x_empty = x_full + XS;                 // [x stages] the MMAs that read the tiles have completed
    uint64_t* raw_full = x_empty + XS;
    uint64_t* raw_empty = raw_full + RS;             // [raw stages] read by the four warps of its group
    uint64_t* b_ready = raw_empty + RS;              // [B stages] first CTA: dequantised tiles of both CTAs written
    uint64_t* b_empty = b_ready + BS;
    uint64_t* acc_ready = b_empty + BS;              // [sets] all MMAs of a tile have completed
    uint64_t* acc_empty = acc_ready + GM_ACC_SETS;   // [sets] first CTA: both epilogues have drained the set (an arrival per warp)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + GM_ACC_SETS);

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int rank = blockIdx.x & 1, pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;      // clusters of two along x
    const int num_kb = p.K / GM_BK;
    const int total_tiles = p.n_tiles * p.m_tiles;

    if (tid == 0) {
        for (int s = 0; s < XS; ++s) { gm_mbar_init(&x_full[s], 1); gm_mbar_init(&x_empty[s], 1); }
        for (int s = 0; s < RS; ++s) { gm_mbar_init(&raw_full[s], 1); gm_mbar_init(&raw_empty[s], GM_DEQ_GROUP); }
        for (int s = 0; s < BS; ++s) { gm_mbar_init(&b_ready[s], 2 * GM_DEQ_GROUP); gm_mbar_init(&b_empty[s], 1); }
        for (int a = 0; a < GM_ACC_SETS; ++a) {
            gm_mbar_init(&acc_ready[a], 1);
            gm_mbar_init(&acc_empty[a], 2 * GM_EPI_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {     // tensor memory: all 512 columns of both SMs
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(gm_smem(tmem_slot)), "r"(GM_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    gm_cluster_sync();       // the other CTA's barriers exist
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    bool failed = false;

    // tile index -> projection, first column inside it, first row (N tiles vary fastest: neighbouring pairs share x rows)
    auto locate = [&](int tile, int& pj, int& n0, int& m0) {
        const int nt = tile % p.n_tiles;
        m0 = (tile / p.n_tiles) * (2 * GM_BM);
        if constexpr (SWIGLU) {
            pj = rank;
            n0 = nt * GM_CN;
        } else {
            pj = 0;
#pragma unroll
            for (int i = 1; i < GM_MAX_PROJ; ++i)
                if (i < p.n_proj && nt >= p.proj[i].tile0) pj = i;
            n0 = (nt - p.proj[pj].tile0) * GM_BN;
        }
    };
    const int w_off = SWIGLU ? 0 : rank * GM_CN;      // this CTA's first column of W inside the tile

    // The producer and issuer warps walk their loops as whole warps and one elected lane issues: operands that are
    // uniform over the warp then stay in uniform registers (inside a branch on lane == 0 an MMA issue took 90 cycles).
    if (warp == 0) {
        // =========================== TMA producer ===========================
        // raw codes run RS blocks ahead of the dequantisation, x tiles XS blocks ahead of the MMAs
        const int my_tiles = total_tiles > pair ? (total_tiles - 1 - pair) / pairs + 1 : 0;
        const int blocks = my_tiles * num_kb;
        int rt = pair, rk = 0, xt = pair, xk = 0;       // tile and k block of the next raw / x request
        int rpj = 0, rn0 = 0, rm0 = 0, xpj = 0, xn0 = 0, xm0 = 0;
        int rs = 0, xs = 0;
        unsigned rph = 1u, xph = 1u;                                // the first pass finds every stage free
        for (int g = 0, r = 0; g < blocks && !failed; ++g) {
            for (; r < blocks && r < g + RS; ++r) {
                if (rk == 0) locate(rt, rpj, rn0, rm0);
                if (gm_timeout(&raw_empty[rs], rph)) { failed = true; break; }
                const CUtensorMap* map_w = rpj == 0 ? &map_w0 : (rpj == 1 ? &map_w1 : (rpj == 2 ? &map_w2 : &map_w3));
                if (gm_elect()) {
                    gm_mbar_expect_tx(&raw_full[rs], GM_RAW_BYTES);
                    gm_tma_2d(sRaw + rs * GM_RAW_BYTES, map_w, (rn0 + w_off) / 8, rk * GM_BK, &raw_full[rs]);
                }
                __syncwarp();
                if (++rs == RS) { rs = 0; rph ^= 1u; }
                if (++rk == num_kb) { rk = 0; rt += pairs; }
                if (r >= RS) { ++r; break; }                        // steady state: one raw request per x request
            }
            if (failed) break;
            if (g == 0) {          // x is the previous kernel's; the weights never change and are on their way
                pdl_wait();
                pdl_trigger();
            }
            if (xk == 0) locate(xt, xpj, xn0, xm0);
            if (gm_timeout(&x_empty[xs], xph)) { failed = true; break; }
            if (gm_elect()) {
                if (rank == 0) gm_mbar_expect_tx(&x_full[xs], 2 * GM_X_BYTES);      // the other CTA's bytes may come first: the phase still waits for this arrival
                gm_tma_2d_pair(sX + xs * GM_X_BYTES, &map_x, xk * GM_BK, xm0 + rank * GM_BM, gm_first(&x_full[xs]));
            }
            __syncwarp();
            if (++xs == XS) { xs = 0; xph ^= 1u; }
            if (++xk == num_kb) { xk = 0; xt += pairs; }
        }
        // the arrivals that the first CTA's commits send here have all come before this CTA may end
        for (int g = blocks > XS ? blocks - XS : 0; g < blocks && !failed; ++g) failed = gm_timeout(&x_empty[g % XS], (unsigned)(g / XS) & 1u);
        for (int g = blocks > BS ? blocks - BS : 0; g < blocks && !failed; ++g) failed = gm_timeout(&b_empty[g % BS], (unsigned)(g / BS) & 1u);
    } else if (warp == 1) {
        // =========================== MMA issuer (first CTA) ===========================
        // instruction descriptor: fp32 accumulate, fp16 A (K-major) and B (MN-major), N = 256, M = 256 over both CTAs
        constexpr uint32_t idesc = (1u << 4) | (0u << 7) | (0u << 10) | (0u << 15) | (1u << 16) | ((uint32_t)(GM_BN >> 3) << 17) |
                                   ((uint32_t)(2 * GM_BM >> 4) << 24);
        // A: K-major; 8 rows x 64 k = one 1 KiB atom; 16 k = 32 B further inside the swizzled row.  B: MN-major; 64 columns x
        // 8 k = one 1 KiB atom; atoms 1 KiB apart along K, BK*128 B apart along N (2 atoms per CTA).  Each CTA's tensor core
        // reads its own copy at these addresses
        const uint64_t da0 = gm_desc(gm_smem(sX), 16, 1024), db0 = gm_desc(gm_smem(sB), GM_BK * 128, 1024);
        int g = 0, it = 0;
        for (int tile = rank == 0 ? pair : total_tiles; tile < total_tiles && !failed; tile += pairs, ++it) {
            const int set = it % GM_ACC_SETS, use = it / GM_ACC_SETS;
            // the set must have been drained by the epilogues of the tile that used it last
            if (use >= 1 && gm_timeout(&acc_empty[set], (unsigned)(use - 1) & 1u)) { failed = true; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc = tmem_base + (uint32_t)(set * GM_BN);
            for (int kb = 0; kb < num_kb; ++kb, ++g) {
                const int xs = g % XS, bs = g % BS;
                if (gm_timeout(&x_full[xs], (unsigned)(g / XS) & 1u) || gm_timeout(&b_ready[bs], (unsigned)(g / BS) & 1u)) { failed = true; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t da = da0 + (uint64_t)(xs * (GM_X_BYTES >> 4)), db = db0 + (uint64_t)(bs * (GM_B_BYTES >> 4));
                if (gm_elect()) {
#pragma unroll
                    for (int k = 0; k < GM_BK / 16; ++k) gm_mma(acc, da + k * (32 >> 4), db + k * (2048 >> 4), idesc, (kb | k) != 0 ? 1u : 0u);
                    gm_commit(&x_empty[xs]);           // arrive when the MMAs issued so far have read their operands
                    gm_commit(&b_empty[bs]);
                    if (kb + 1 == num_kb) gm_commit(&acc_ready[set]);
                }
                __syncwarp();
            }
        }
    } else if (warp < 2 + GM_DEQ_WARPS) {
        // =========================== dequantise ===========================
        // three groups of four warps take turns: two blocks are converted while a third is multiplied
        const int grp = (warp - 2) / GM_DEQ_GROUP;
        const int t = (tid - 64) % (GM_DEQ_GROUP * 32);
        const int c = t & 15;                         // int32 column of the raw tile = 8 of this CTA's output columns
        const int kr0 = t >> 4;                       // first k row of this thread; it takes rows kr0 + 8 i
        const int gshift = p.group == 64 ? 0 : p.group == 128 ? 1 : 2;       // k blocks per quantisation group, as a shift
        const int a_n = c >> 3, chunk = c & 7;        // 64-column atom and 16-byte chunk inside its rows
        const __half2 sixteenth = __float2half2_rn(0.0625f);
        // block g of this CTA = k block kb of tile `tile`; the scale and zero words of this group's next block are requested one
        // block ahead, across tiles
        int tile = pair, kb = grp, width = 0;         // width: output columns of the tile's projection, 0 where this thread's are none
        const int32_t* zrow = nullptr;                // zeros and scales of this thread's columns, first quantisation group
        const __half* srow = nullptr;
        auto enter = [&]() {                          // divisions and look-ups once per tile
            while (kb >= num_kb && tile < total_tiles) { kb -= num_kb; tile += pairs; }
            width = 0;
            if (tile >= total_tiles) return;
            int pj, n0, m0;
            locate(tile, pj, n0, m0);
            const int n = n0 + w_off + 8 * c;
            if (n < p.proj[pj].N) {                   // a projection of 128 (mod 256) columns ends inside its last tile
                width = p.proj[pj].N;
                zrow = p.proj[pj].qzeros + n / 8;
                srow = p.proj[pj].scales + n;
            }
        };
        auto load_meta = [&](uint32_t& zw, uint4& s4) {
            zw = 0; s4 = make_uint4(0, 0, 0, 0);
            if (width != 0) {
                const int64_t at = (int64_t)(kb >> gshift) * width;
                zw = (uint32_t)__ldg(zrow + (at >> 3));
                s4 = __ldg(reinterpret_cast<const uint4*>(srow + at));
            }
        };
        uint32_t zw_nx;
        uint4 s4_nx;
        enter();
        load_meta(zw_nx, s4_nx);
        for (int g = grp, bs = grp, rs = grp; tile < total_tiles; g += GM_DEQ_WARPS / GM_DEQ_GROUP) {
            const uint32_t zw = zw_nx, sw[4] = {s4_nx.x, s4_nx.y, s4_nx.z, s4_nx.w};
            kb += GM_DEQ_WARPS / GM_DEQ_GROUP;
            if (kb >= num_kb) enter();
            load_meta(zw_nx, s4_nx);
            // per column pair: even nibbles h = 1024 + code, minus (1024 + zero); odd ones h = 1024 + 16 code, times 1/16 minus
            // (64 + zero): both exact; then the scale, rounded once
            __half2 zs[4], sc2[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t z = ((zw >> (4 * q)) & 0x000f000fu) | 0x64006400u;
                zs[q] = __hsub2((q & 1) ? __float2half2_rn(960.0f) : __float2half2_rn(0.0f), *reinterpret_cast<const __half2*>(&z));
                if constexpr (INTERLEAVED) sc2[q] = *reinterpret_cast<const __half2*>(&sw[q]);      // columns (2q, 2q+1)
                else {                                                                              // columns (q, q+4)
                    const __half* sh = reinterpret_cast<const __half*>(sw);
                    sc2[q] = __halves2half2(sh[q], sh[q + 4]);
                }
            }
            if (gm_timeout(&raw_full[rs], (unsigned)(g / RS) & 1u)) { failed = true; break; }
            const uint32_t* raw = reinterpret_cast<const uint32_t*>(sRaw + rs * GM_RAW_BYTES) + kr0 * (GM_CN / 8) + c;
            uint32_t w[GM_BK / 8];
#pragma unroll
            for (int i = 0; i < GM_BK / 8; ++i) w[i] = raw[8 * i * (GM_CN / 8)];
            if (g >= BS && gm_timeout(&b_empty[bs], (unsigned)(g / BS - 1) & 1u)) { failed = true; break; }
            unsigned char* bt = sB + bs * GM_B_BYTES + a_n * (GM_BK * 128);
#pragma unroll
            for (int i = 0; i < GM_BK / 8; ++i) {
                const int kr = kr0 + 8 * i;
                const uint32_t w8 = w[i] >> 8;
                uint32_t o[4] = {(w[i] & 0x000f000fu) | 0x64006400u, (w[i] & 0x00f000f0u) | 0x64006400u,
                                 (w8 & 0x000f000fu) | 0x64006400u, (w8 & 0x00f000f0u) | 0x64006400u};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const __half2 h = *reinterpret_cast<const __half2*>(&o[q]);
                    const __half2 r = __hmul2((q & 1) ? __hfma2(h, sixteenth, zs[q]) : __hadd2(h, zs[q]), sc2[q]);
                    o[q] = *reinterpret_cast<const uint32_t*>(&r);
                }
                uint4 out;
                if constexpr (INTERLEAVED) {
                    out = make_uint4(o[0], o[1], o[2], o[3]);
                } else {      // pairs (q, q+4) -> column order
                    out = make_uint4(__byte_perm(o[0], o[1], 0x5410), __byte_perm(o[2], o[3], 0x5410),
                                     __byte_perm(o[0], o[1], 0x7632), __byte_perm(o[2], o[3], 0x7632));
                }
                // row kr of the atom column a_n: 128 B per row, 16-byte chunks swizzled by the row index (kr mod 8 = kr0)
                *reinterpret_cast<uint4*>(bt + kr * 128 + ((chunk ^ kr0) << 4)) = out;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // generic-proxy stores -> visible to the tensor core
            __syncwarp();
            if (lane == 0) {
                gm_arrive_first(&b_ready[bs]);
                // not earlier: an arrival right behind the loads let the refill overtake them (wrong tiles, about 1 launch in 10)
                gm_mbar_arrive(&raw_empty[rs]);
            }
            bs = (bs + GM_DEQ_WARPS / GM_DEQ_GROUP) % BS; rs = (rs + GM_DEQ_WARPS / GM_DEQ_GROUP) % RS;
        }
    } else {
        // =========================== epilogue ===========================
        const int lq = warp & 3;                      // the TMEM lane quarter this warp may read
        pdl_wait();                                   // y may have been read by the kernel before
        int it = 0;
        for (int tile = pair; tile < total_tiles && !failed; tile += pairs, ++it) {
            int pj, n0, m0;
            locate(tile, pj, n0, m0);
            const GemmProj& P = p.proj[pj];
            const int set = it % GM_ACC_SETS, use = it / GM_ACC_SETS;
            if (gm_timeout(&acc_ready[set], (unsigned)use & 1u)) { failed = true; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int row = m0 + rank * GM_BM + lq * 32 + lane;
            if constexpr (SWIGLU) {
                const GemmProj &G = p.proj[0], &U = p.proj[1];
#pragma unroll 1
                for (int cb = 0; cb < GM_CN / 32; ++cb) {
                    uint32_t gv[32], uv[32];
                    const uint32_t taddr = tmem_base + ((uint32_t)(lq * 32) << 16) + (uint32_t)(set * GM_BN + cb * 32);
                    gm_tmem_ld32(taddr, gv);
                    gm_tmem_ld32(taddr + GM_CN, uv);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (row < p.M) {
                        const int n = n0 + cb * 32;
                        __half* yrow = G.y + (int64_t)row * G.N + n;
#pragma unroll
                        for (int j = 0; j < 32; j += 8) {
                            uint32_t pk[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const int i = j + 2 * e;
                                float g0 = __uint_as_float(gv[i]), g1 = __uint_as_float(gv[i + 1]), u0 = __uint_as_float(uv[i]), u1 = __uint_as_float(uv[i + 1]);
                                if (G.bias) { g0 += __half2float(G.bias[n + i]); g1 += __half2float(G.bias[n + i + 1]); }
                                if (U.bias) { u0 += __half2float(U.bias[n + i]); u1 += __half2float(U.bias[n + i + 1]); }
                                const float2 f = __half22float2(__floats2half2_rn(g0, g1));
                                const __half2 h = __hmul2(__floats2half2_rn(f.x / (1.0f + expf(-f.x)), f.y / (1.0f + expf(-f.y))), __floats2half2_rn(u0, u1));
                                pk[e] = *reinterpret_cast<const uint32_t*>(&h);
                            }
                            *reinterpret_cast<uint4*>(yrow + j) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                        }
                    }
                }
            } else {
#pragma unroll 1
            for (int cb = 0; cb < GM_BN / 32; ++cb) {
                uint32_t v[32];
                gm_tmem_ld32(tmem_base + ((uint32_t)(lq * 32) << 16) + (uint32_t)(set * GM_BN + cb * 32), v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (row < p.M && n0 + cb * 32 < P.N) {
                    __half* yrow = P.y + (int64_t)row * P.N + n0 + cb * 32;
#pragma unroll
                    for (int j = 0; j < 32; j += 8) {
                        uint32_t pk[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            float f0 = __uint_as_float(v[j + 2 * e]), f1 = __uint_as_float(v[j + 2 * e + 1]);
                            if (P.bias) {
                                f0 += __half2float(P.bias[n0 + cb * 32 + j + 2 * e]);
                                f1 += __half2float(P.bias[n0 + cb * 32 + j + 2 * e + 1]);
                            }
                            const __half2 h = __floats2half2_rn(f0, f1);
                            pk[e] = *reinterpret_cast<const uint32_t*>(&h);
                        }
                        *reinterpret_cast<uint4*>(yrow + j) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                    }
                }
            }
            }
            // the set's columns have been read: hand it back to the MMA warp
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) gm_arrive_first(&acc_empty[set]);
        }
    }
    if (failed) {
        atomicExch(p.status, FQ_ERR_TIMEOUT);
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);       // copies and MMAs in flight end before the memory is given back
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    gm_cluster_sync();       // the other CTA's arrivals here, and its tensor core's reads, are over
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(GM_TMEM_COLS) : "memory");
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled_fn() {
    static std::atomic<void*> cached{nullptr};
    void* fn = cached.load(std::memory_order_relaxed);
    if (fn == nullptr) {
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess || qres != cudaDriverEntryPointSuccess) return nullptr;
        cached.store(fn, std::memory_order_relaxed);
    }
    return reinterpret_cast<EncodeTiledFn>(fn);
}

// One wave of 128 x 128 tiles, up to three while the rows fit one tile, go to the few-row kernel, one chain of products per
// tile: same bits, shorter start.  From its second wave on a pair's tile of four times the size takes 1.3 of its time.
// Measured, few-row / this kernel, us:
//   3072 -> 5120:   18.8 / 26.0 at 384 rows (120 tiles), 35.7 / 26.1 at 512 (160), 54.9 / 43.2 at 1024 (320)
//   3072 -> 16384:  20.5 / 26.7 at 128 rows (128), 38.7 / 26.8 at 129 (256), 56.6 / 43.4 at 257 (384)
//   8192 -> 3072:   44.3 / 54.0 at 768 rows (144), 83.2 / 54.2 at 1024 (192);  4096 -> 6144: 24.7 / 31.1 at 384 (144), 45.5 / 31.2 at 512 (192)
//   4096 -> 28672:  42.6 / 54.3 at 16 rows, 49.7 / 56.0 at 128 (224 tiles, a half-empty row tile for the pair), 92.9 / 56.5 at 129 (448)
static bool few_rows(const SkinnyCall& c) {
    int64_t tiles128 = 0;
    for (int i = 0; i < c.n_proj; ++i) tiles128 += c.N[i] / 128;
    return tiles128 * ((c.M + 127) / 128) <= (int64_t)(c.M <= GM_BM ? 3 : 1) * sm_count() && awq_skinny_supported(c);
}

static int check_call(const SkinnyCall& c, const char* fn) {
    FQ_CHECK_ARG(c.M >= 1, FQ_ERR_ARG, "%s: M=%d", fn, c.M);
    FQ_CHECK_ARG(c.group == 64 || c.group == 128 || c.group == 256, FQ_ERR_UNSUPPORTED, "%s: group size %d; 64, 128 and 256 are built", fn, c.group);
    FQ_CHECK_ARG(c.K > 0 && c.K % c.group == 0, FQ_ERR_ARG, "%s: K=%d must be a multiple of the group size %d", fn, c.K, c.group);
    FQ_CHECK_ARG(aligned(c.x, 16), FQ_ERR_ALIGN, "%s: x must be 16-byte aligned", fn);
    for (int i = 0; i < c.n_proj; ++i) {
        FQ_CHECK_ARG(c.N[i] > 0 && c.N[i] % 128 == 0, FQ_ERR_UNSUPPORTED, "%s: N[%d]=%d must be a positive multiple of 128", fn, i, c.N[i]);
        FQ_CHECK_ARG(c.qweight[i] && c.scales[i] && c.qzeros[i] && c.y[i], FQ_ERR_ARG, "%s: null tensor in projection %d", fn, i);
        FQ_CHECK_ARG(aligned(c.y[i], 16) && aligned(c.scales[i], 16) && aligned(c.qweight[i], 16) && aligned(c.qzeros[i], 4), FQ_ERR_ALIGN,
                     "%s: y[%d], scales[%d] and qweight[%d] must be 16-byte aligned", fn, i, i, i);
    }
    return FQ_OK;
}

static SkinnyCall make_call(const void* x, int M, int K, int group, int n_proj, const int32_t* const* qweight, const void* const* scales,
                            const int32_t* const* qzeros, const void* const* bias, const int* N, void* const* y, int interleaved) {
    SkinnyCall c{};
    c.x = x; c.M = M; c.K = K; c.group = group; c.n_proj = n_proj; c.interleaved = interleaved ? 1 : 0;
    for (int i = 0; i < n_proj; ++i) {
        c.qweight[i] = qweight[i]; c.scales[i] = scales[i]; c.qzeros[i] = qzeros[i]; c.bias[i] = bias ? bias[i] : nullptr; c.N[i] = N[i]; c.y[i] = y[i];
    }
    return c;
}

// the pair kernel on a checked call
static int pairs_launch(const SkinnyCall& c, bool swiglu, void* stream, const char* fn) {
    EncodeTiledFn encode = encode_tiled_fn();
    if (!encode) return fail(FQ_ERR_CUDA, "%s: the driver does not export cuTensorMapEncodeTiled", fn);
    GemmParams p{};
    p.n_proj = c.n_proj; p.M = c.M; p.K = c.K; p.group = c.group;
    p.status = device_status_ptr();
    if (p.status == nullptr) return FQ_ERR_CUDA;
    CUtensorMap maps[1 + GM_MAX_PROJ];
    {
        const cuuint64_t dims[2] = {(cuuint64_t)c.K, (cuuint64_t)c.M};
        const cuuint64_t strides[1] = {(cuuint64_t)c.K * 2};
        const cuuint32_t box[2] = {(cuuint32_t)GM_BK, (cuuint32_t)GM_BM}, es[2] = {1, 1};
        CUresult r = encode(&maps[0], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(c.x), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return fail(FQ_ERR_CUDA, "%s: tensor map for x: driver error %d", fn, (int)r);
    }
    int tile0 = 0;
    for (int i = 0; i < c.n_proj; ++i) {
        p.proj[i] = GemmProj{static_cast<const __half*>(c.scales[i]), c.qzeros[i], static_cast<const __half*>(c.bias[i]), static_cast<__half*>(c.y[i]), c.N[i], tile0};
        tile0 += (c.N[i] + GM_BN - 1) / GM_BN;
        const cuuint64_t dims[2] = {(cuuint64_t)(c.N[i] / 8), (cuuint64_t)c.K};
        const cuuint64_t strides[1] = {(cuuint64_t)(c.N[i] / 8) * 4};
        const cuuint32_t box[2] = {(cuuint32_t)(GM_CN / 8), (cuuint32_t)GM_BK}, es[2] = {1, 1};
        CUresult r = encode(&maps[1 + i], CU_TENSOR_MAP_DATA_TYPE_INT32, 2, const_cast<int32_t*>(c.qweight[i]), dims, strides, box, es,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return fail(FQ_ERR_CUDA, "%s: tensor map for qweight[%d]: driver error %d", fn, i, (int)r);
    }
    for (int i = c.n_proj; i < GM_MAX_PROJ; ++i) { maps[1 + i] = maps[1]; p.proj[i] = GemmProj{nullptr, nullptr, nullptr, nullptr, 0, 1 << 30}; }
    if (swiglu) tile0 = c.N[0] / GM_CN;
    const int m_tiles = (c.M + 2 * GM_BM - 1) / (2 * GM_BM);
    FQ_CHECK_ARG((int64_t)m_tiles * tile0 <= 0x7fffffffLL, FQ_ERR_ARG, "%s: M=%d too large for one launch", fn, c.M);
    p.n_tiles = tile0; p.m_tiles = m_tiles;
    // one persistent pair of CTAs per pair of SMs (the shared memory of a CTA leaves room for no second one)
    const int total = m_tiles * tile0, sms = sm_count(), pairs = total < sms / 2 ? total : sms / 2;
    auto kern = swiglu ? (c.interleaved ? awq_gemm_kernel<true, true> : awq_gemm_kernel<false, true>)
                       : (c.interleaved ? awq_gemm_kernel<true, false> : awq_gemm_kernel<false, false>);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GM_SMEM);
    if (e != cudaSuccess) return fail(FQ_ERR_CUDA, "%s: cannot reserve %d B of shared memory: %s", fn, GM_SMEM, cudaGetErrorString(e));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(2 * pairs)); cfg.blockDim = dim3(GM_THREADS); cfg.dynamicSmemBytes = GM_SMEM; cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute at[2]{};
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = pdl_enabled(PDL_GEMV) ? 2 : 1;
    count_launch();
    e = cudaLaunchKernelEx(&cfg, kern, maps[0], maps[1], maps[2], maps[3], maps[4], p);
    if (e != cudaSuccess) return fail(FQ_ERR_CUDA, "%s: launch failed: %s", fn, cudaGetErrorString(e));
    FQ_CHECK_LAUNCH(fn);
    return FQ_OK;
}

}  // namespace fq

extern "C" int fq_awq_gemm(
    const void* x, int M, int K, int group, int n_proj,
    const int32_t* const* qweight, const void* const* scales, const int32_t* const* qzeros, const void* const* bias,
    const int* N, void* const* y, int interleaved, void* stream) {
    using namespace fq;
    const char* fn = "fq_awq_gemm";
    FQ_CHECK_ARG(n_proj >= 1 && n_proj <= GM_MAX_PROJ, FQ_ERR_ARG, "%s: 1..%d projections per call, got %d", fn, GM_MAX_PROJ, n_proj);
    FQ_CHECK_ARG(x && qweight && scales && qzeros && N && y, FQ_ERR_ARG, "%s: null pointer", fn);
    const SkinnyCall c = make_call(x, M, K, group, n_proj, qweight, scales, qzeros, bias, N, y, interleaved);
    const int rc = check_call(c, fn);
    if (rc != FQ_OK) return rc;
    return few_rows(c) ? awq_skinny_launch(c, stream, fn) : pairs_launch(c, false, stream, fn);
}

extern "C" int fq_awq_gate_up_swiglu(
    const void* x, int M, int K, int group, const int32_t* const* qweight, const void* const* scales, const int32_t* const* qzeros, const void* const* bias,
    int N, void* gate, void* up, void* y, int interleaved, void* stream) {
    using namespace fq;
    const char* fn = "fq_awq_gate_up_swiglu";
    FQ_CHECK_ARG(x && qweight && scales && qzeros && y, FQ_ERR_ARG, "%s: null pointer", fn);
    const int Ns[2] = {N, N};
    void* both[2] = {gate, up};
    void* ys[2] = {y, y};
    SkinnyCall c = make_call(x, M, K, group, 2, qweight, scales, qzeros, bias, Ns, ys, interleaved);
    int rc = check_call(c, fn);
    if (rc != FQ_OK) return rc;
    if (!few_rows(c)) return pairs_launch(c, true, stream, fn);
    for (int i = 0; i < 2; ++i) {
        c.y[i] = both[i];
        FQ_CHECK_ARG(both[i] && aligned(both[i], 16), FQ_ERR_ALIGN, "%s: gate and up must be 16-byte aligned", fn);
    }
    if ((rc = awq_skinny_launch(c, stream, fn)) != FQ_OK) return rc;
    return fq_swiglu(gate, up, (int64_t)M * N, y, stream);
}
