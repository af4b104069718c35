// Page scores read straight from the INT4 K metadata.
//
// score[b,hq,p] = sum_d q[d]*K_mn[p,d] + 15 * sum_d relu(q[d])*K_scale[p,d]
//
// HBM-bound: the only real traffic is the metadata, 2*D*2 bytes per (kv head, page), read
// exactly once and shared by all query heads of the GQA group.  Eight lanes (a quarter
// warp) own one page: each lane issues 16-byte loads of 8 channels, the eight lanes of a
// page read 128 contiguous bytes per instruction and the four quarter-warps read four
// consecutive pages, so every warp load is one contiguous 512-byte run.  Each lane keeps
// its slice of q for all NR query heads in registers; the per-page reduction is a 3-step
// xor shuffle inside the quarter warp.
#include "fq_append.cuh"
#include "fq_score_grid.cuh"
#include "fq_score_lane.cuh"

namespace fq {

constexpr int SCORE_THREADS = 128;            // 16 pages per CTA iteration
constexpr int SCORE_PAGES_PER_CTA = 32;       // 2 iterations per CTA

// What a decode step appends in the launch of its page scores, by one extra CTA per (batch, kv head).  A launch of its own for 4 KB
// per head took 1.9 to 2.5 us of every layer.  Two forms: rows to stage behind a known number of tokens, no page completed; and,
// with the position read on the device, whatever the position asks for.  There, pages completed before do not wait for the
// append, and the score of a page completed now is the same CTA's work.  That form is the Llama step's, in fp16 throughout.
struct NoAppend {};
struct StageAppend {
    const uint16_t *K_new, *V_new; int64_t nw_sb, nw_sh, nw_ss;
    uint16_t *K_stage, *V_stage; int64_t st_sb, st_sh, st_ss;      // row 0 of the new tokens, unless the position is read on the device
    int n;
};
struct DynAppend { StageAppend st; QuantParams q; };

// rows of n tokens, K and V, 16 bytes per thread and pass; before() runs between the loads and the stores and returns the first row
template <typename F>
__device__ __forceinline__ void stage_rows(const StageAppend& a, int b, int h, int chunks, F&& before) {
    const int i = threadIdx.x, per = a.n * chunks;
    auto src = [&](int j) {
        const int r = (j % per) / chunks, c = j % chunks;
        return reinterpret_cast<const uint4*>((j < per ? a.K_new : a.V_new) + b * a.nw_sb + h * a.nw_sh + r * a.nw_ss + 8 * c);
    };
    uint4 first_v = make_uint4(0, 0, 0, 0);
    if (i < 2 * per) first_v = *src(i);
    const int row0 = before();
    if (row0 < 0) return;
    for (int j = i; j < 2 * per; j += SCORE_THREADS) {
        const uint4 v = j == i ? first_v : *src(j);
        const int r = row0 + (j % per) / chunks, c = j % chunks;
        *reinterpret_cast<uint4*>((j < per ? a.K_stage : a.V_stage) + b * a.st_sb + h * a.st_sh + r * a.st_ss + 8 * c) = v;
    }
}

// the append that completes a page: one step in `page`
__device__ __noinline__ void append_page(const DynAppend& a, int b, int h) {
    QuantParams p = a.q;
    if (!quant_locate(p)) return;                              // full: nothing is written (the host checks its own count)
    quant_int4_cta<__half>(p, b, h, 0);
}

template <typename QT, int NR, int CH>
__device__ __forceinline__ void append_and_score(const DynAppend& a, const QT* __restrict__ Q, int64_t q_sb, int64_t q_sh, int b, int hkv, int n_rep, int head_off,
                                                 int P, int D, float* __restrict__ scores, int64_t sc_sb, int64_t sc_sh, float levels, const int* pos) {
    const int seen = __ldcg(pos);
    pdl_wait();
    pdl_trigger();
    const int page_len = a.q.page, partial = seen % page_len;
    const bool completes = partial + a.q.n_new >= page_len;
    stage_rows(a.st, b, hkv, D >> 3, [&]() { return completes || seen < 0 || seen + a.q.n_new > a.q.max_tokens ? -1 : partial; });
    if (!completes) return;
    append_page(a, b, hkv);
    const int page = seen / page_len;                          // completed by this append
    if (page >= P) return;
    __syncthreads();                                           // the metadata row is written; read it behind L1, which may hold older bytes
    if (threadIdx.x >= 32) return;
    const int l = threadIdx.x & 7, n_chunks = D >> 3, nr = min(NR, n_rep - head_off);
    uint4 m4[CH], s4[CH];
#pragma unroll
    for (int c = 0; c < CH; ++c) {
        const int chunk = l + 8 * c;
        m4[c] = s4[c] = make_uint4(0, 0, 0, 0);
        if (chunk < n_chunks) {
            const int64_t at = b * a.q.km_sb + hkv * a.q.km_sh + (int64_t)page * a.q.km_sp + 8 * chunk;
            m4[c] = __ldcg(reinterpret_cast<const uint4*>(a.q.K_mn + at));
            s4[c] = __ldcg(reinterpret_cast<const uint4*>(a.q.K_scale + at));
        }
    }
    float q[NR][CH][8];
    score_load_q<QT, NR, CH>(Q + b * q_sb, q_sh, hkv * n_rep + head_off, nr, l, n_chunks, q);
    const float v = score_page<NR, CH>(q, m4, s4, l, levels);
    if (threadIdx.x < nr) scores[b * sc_sb + (hkv * n_rep + head_off + l) * sc_sh + page] = v;
}

// NR = query heads handled per pass (<= 4), CH = 8-channel chunks per lane (D = 64*CH, or
// D = 32 with CH = 1 where lanes 4..7 hold no chunk).
template <typename QT, int NR, int CH, typename APPEND>
__global__ void __launch_bounds__(SCORE_THREADS) page_scores_kernel(
    const QT* __restrict__ Q, int64_t q_sb, int64_t q_sh,
    const uint16_t* __restrict__ K_scale, const uint16_t* __restrict__ K_mn,
    int64_t km_sb, int64_t km_sh, int64_t km_sp,
    int Hq, int Hkv, int P, int D, int head_off,
    float* __restrict__ scores, int64_t sc_sb, int64_t sc_sh, const int* __restrict__ pos, int pos_new, int pos_page, int pos_early, float levels,
    const __grid_constant__ APPEND app) {
    const int b = blockIdx.z, hkv = blockIdx.y;
    const int n_rep = Hq / Hkv;
    if constexpr (std::is_same_v<APPEND, StageAppend>) {
        if (blockIdx.x == gridDim.x - 1) {
            pdl_wait();
            pdl_trigger();
            stage_rows(app, b, hkv, D >> 3, []() { return 0; });
            return;
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int l = lane & 7, qw = lane >> 3;
    const int n_chunks = D >> 3;
    const int nr = min(NR, n_rep - head_off);   // heads actually present in this pass
    // A position on the device of either kind (DynPos); the decode steps take the kernel below for theirs.  Calls without one pass
    // both branches by, and the code in front of the wait and behind it stays apart: with neither branch the compiler lays the set-up
    // out behind the wait, and 28 layers of 2049 pages (scores, selection, attention) take 575 us instead of 563, with the second alone 573.
    int pos_v = 0;
    if (pos && pos_early) pos_v = __ldcg(pos);             // in flight during the wait
    pdl_wait();        // Q and the newest metadata row come from the kernels before this one
    pdl_trigger();
    if (pos) {
        if (!pos_early) pos_v = *pos;
        P = min(P, (pos_v + pos_new) / pos_page);          // completed pages after this step's append
    }

    // Metadata loads of every page this quarter warp will score are issued first, the q loads
    // after them, so the two global-memory latencies overlap instead of adding up.
    constexpr int ITERS = SCORE_PAGES_PER_CTA / 16;
    const int p_base = blockIdx.x * SCORE_PAGES_PER_CTA;
    const uint16_t* sc_base = K_scale + b * km_sb + hkv * km_sh;
    const uint16_t* mn_base = K_mn + b * km_sb + hkv * km_sh;
    uint4 m4[ITERS][CH], s4[ITERS][CH];
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
        const int p = p_base + it * 16 + warp * 4 + qw;
        score_load_meta<CH>(sc_base, mn_base, km_sp, p, p < P, l, n_chunks, m4[it], s4[it]);
    }
    float q[NR][CH][8];
    score_load_q<QT, NR, CH>(Q + b * q_sb, q_sh, hkv * n_rep + head_off, nr, l, n_chunks, q);
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
        const int p = p_base + it * 16 + warp * 4 + qw;
        const float v = score_page<NR, CH>(q, m4[it], s4[it], l, levels);
        if (p < P && l < nr) scores[b * sc_sb + (hkv * n_rep + head_off + l) * sc_sh + p] = v;
    }
}

// page_scores_kernel for the decode step, where the position may be read before the dependency wait
// (DynPos::early): the rows of the pages completed before this step -- nothing in flight writes them -- are
// requested before the wait as well, so the CTA spends the end of the previous kernel fetching instead of waiting.
template <typename QT, int NR, int CH, typename APPEND>
__global__ void __launch_bounds__(SCORE_THREADS) page_scores_early_kernel(
    const QT* __restrict__ Q, int64_t q_sb, int64_t q_sh,
    const uint16_t* __restrict__ K_scale, const uint16_t* __restrict__ K_mn,
    int64_t km_sb, int64_t km_sh, int64_t km_sp,
    int Hq, int Hkv, int P, int D, int head_off,
    float* __restrict__ scores, int64_t sc_sb, int64_t sc_sh, const int* __restrict__ pos, int pos_new, int pos_page, float levels,
    const __grid_constant__ APPEND app) {
    const int b = blockIdx.z, hkv = blockIdx.y;
    const int n_rep = Hq / Hkv;
    constexpr bool ALONG = std::is_same_v<APPEND, DynAppend>;
    if constexpr (ALONG) {
        if (blockIdx.x == gridDim.x - 1) {
            append_and_score<QT, NR, CH>(app, Q, q_sb, q_sh, b, hkv, n_rep, head_off, P, D, scores, sc_sb, sc_sh, levels, pos);
            return;
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int l = lane & 7, qw = lane >> 3;
    const int n_chunks = D >> 3;
    const int nr = min(NR, n_rep - head_off);   // heads actually present in this pass
    constexpr int ITERS = SCORE_PAGES_PER_CTA / 16;
    const int p_base = blockIdx.x * SCORE_PAGES_PER_CTA;
    const uint16_t* sc_base = K_scale + b * km_sb + hkv * km_sh;
    const uint16_t* mn_base = K_mn + b * km_sb + hkv * km_sh;
    uint4 m4[ITERS][CH], s4[ITERS][CH];
    const int pos_v = __ldcg(pos);
    const int P_old = min(P, pos_v / pos_page);
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
        const int p = p_base + it * 16 + warp * 4 + qw;
        if (p < P_old) score_load_meta<CH>(sc_base, mn_base, km_sp, p, true, l, n_chunks, m4[it], s4[it]);
    }
    pdl_wait();        // Q and the newest metadata row come from the kernels before this one
    pdl_trigger();
    P = ALONG ? P_old : min(P, (pos_v + pos_new) / pos_page);          // completed pages after this step's append; before it where that is made here
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
        const int p = p_base + it * 16 + warp * 4 + qw;
        if (p >= P_old) score_load_meta<CH>(sc_base, mn_base, km_sp, p, p < P, l, n_chunks, m4[it], s4[it]);
    }
    float q[NR][CH][8];
    score_load_q<QT, NR, CH>(Q + b * q_sb, q_sh, hkv * n_rep + head_off, nr, l, n_chunks, q);
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
        const int p = p_base + it * 16 + warp * 4 + qw;
        const float v = score_page<NR, CH>(q, m4[it], s4[it], l, levels);
        if (p < P && l < nr) scores[b * sc_sb + (hkv * n_rep + head_off + l) * sc_sh + p] = v;
    }
}

// page_scores_kernel for many pages (thousands per SM): CTAs stay and stream.  Each warp runs its own cp.async ring of
// SCORE_RING units of four pages (2 KiB at head_dim 128), so 16 warps keep 64 KiB and more per SM on the way while q stays
// in registers; the short-lived CTAs of the kernel above start with two latencies in a row (37 us against 20 of HBM time for 134 MB).
// 16 x 8 rows of 2048 pages 35.0 -> 24.6 us, of
// 8191 133.9 -> 88.0 (6.1 TB/s); a ring of 4 or 6 units is no faster (25.2, 26.2).
constexpr int SCORE_RING = 3;

template <typename QT, int NR, int CH>
__global__ void __launch_bounds__(SCORE_THREADS, score_stream_ctas_per_sm(NR, CH)) page_scores_stream_kernel(
    const QT* __restrict__ Q, int64_t q_sb, int64_t q_sh,
    const uint16_t* __restrict__ K_scale, const uint16_t* __restrict__ K_mn,
    int64_t km_sb, int64_t km_sh, int64_t km_sp,
    int Hq, int Hkv, int P, int head_off,
    float* __restrict__ scores, int64_t sc_sb, int64_t sc_sh, const int* __restrict__ pos, int pos_new, int pos_page, float levels) {
    constexpr int CHUNKS = 8 * CH;                         // 16-byte chunks per metadata row
    __shared__ __align__(16) uint4 ring[SCORE_THREADS / 32][SCORE_RING][4][2][CHUNKS];
    const int b = blockIdx.z, hkv = blockIdx.y;
    const int n_rep = Hq / Hkv;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int l = lane & 7, qw = lane >> 3;
    const int nr = min(NR, n_rep - head_off);
    pdl_wait();        // Q and the newest metadata row come from the kernels before this one
    pdl_trigger();
    if (pos) P = min(P, (*pos + pos_new) / pos_page);
    const int units = (P + 3) >> 2, per = (units + gridDim.x - 1) / gridDim.x;
    const int u_end = min(units, (int)(blockIdx.x + 1) * per);
    int u = blockIdx.x * per + warp;
    const uint16_t* sc_base = K_scale + b * km_sb + hkv * km_sh + 8 * l;
    const uint16_t* mn_base = K_mn + b * km_sb + hkv * km_sh + 8 * l;
    auto issue = [&](int unit, int slot) {
        const int p = 4 * unit + qw;
        if (unit < u_end && p < P) {
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(&ring[warp][slot][qw][0][l + 8 * c])), "l"(mn_base + (int64_t)p * km_sp + 64 * c) : "memory");
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(&ring[warp][slot][qw][1][l + 8 * c])), "l"(sc_base + (int64_t)p * km_sp + 64 * c) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int i = 0; i < SCORE_RING - 1; ++i) issue(u + 4 * i, i);
    float q[NR][CH][8];
    score_load_q<QT, NR, CH>(Q + b * q_sb, q_sh, hkv * n_rep + head_off, nr, l, CHUNKS, q);
    float* srow = scores + b * sc_sb + (hkv * n_rep + head_off + min(l, nr - 1)) * sc_sh;
    int slot = 0;
    for (; u < u_end; u += 4) {
        issue(u + 4 * (SCORE_RING - 1), (slot + SCORE_RING - 1) % SCORE_RING);
        asm volatile("cp.async.wait_group %0;" ::"n"(SCORE_RING - 1) : "memory");     // a lane reads only what it copied itself
        uint4 m4[CH], s4[CH];
#pragma unroll
        for (int c = 0; c < CH; ++c) { m4[c] = ring[warp][slot][qw][0][l + 8 * c]; s4[c] = ring[warp][slot][qw][1][l + 8 * c]; }
        const float v = score_page<NR, CH>(q, m4, s4, l, levels);
        const int p = 4 * u + qw;
        if (p < P && l < nr) srow[p] = v;
        slot = (slot + 1) % SCORE_RING;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

static int stream_ctas(int nr, int D, int rows, int P) {
    const int CH = D <= 64 ? 1 : D / 64, NR = nr > 4 ? 4 : nr;
    return D == 128 || D == 64 ? score_stream_ctas(rows, P, score_stream_ctas_per_sm(NR, CH) * sm_count()) : 0;
}

// Whether the launch of these scores can take the step's append along: the short-lived CTAs' kernels, 64 or 128 channels.  Streaming
// CTAs stay for as long as their pages last, and there the append is 1 to 2 % of the step.
bool page_scores_take_append(int q_dtype, int B, int Hq, int Hkv, int P, int D) {
    return (q_dtype == FQ_F16 || q_dtype == FQ_BF16) && (D == 64 || D == 128) && P > 0 && Hkv > 0 && Hq % Hkv == 0 && stream_ctas(Hq / Hkv, D, B * Hkv, P) == 0;
}

template <typename QT, int NR>
static void launch_scores(int CH, dim3 grid, cudaStream_t st, const void* Q, int64_t q_sb, int64_t q_sh,
                          const void* K_scale, const void* K_mn, int64_t km_sb, int64_t km_sh, int64_t km_sp,
                          int Hq, int Hkv, int P, int D, int head_off, float* scores, int64_t sc_sb, int64_t sc_sh, const DynPos& dp, float levels,
                          const DynAppend* app) {
    const int ctas = stream_ctas(NR, D, (int)(grid.y * grid.z), P);
    const NoAppend none{};
#define FQ_SC_ARGS static_cast<const QT*>(Q), q_sb, q_sh, static_cast<const uint16_t*>(K_scale), static_cast<const uint16_t*>(K_mn), km_sb, km_sh, km_sp, Hq, Hkv, P, D, \
                   head_off, scores, sc_sb, sc_sh, dp.pos, dp.n_new, dp.page
#define FQ_LAUNCH_SC(CHV)                                                                                                                                                  \
    do {                                                                                                                                                                   \
        if (ctas > 0)                                                                                                                                                      \
            launch_k(PDL_SCORES, page_scores_stream_kernel<QT, NR, (CHV > 2 ? 2 : CHV)>, dim3((unsigned)ctas, grid.y, grid.z), dim3(SCORE_THREADS), 0, st,                 \
                     static_cast<const QT*>(Q), q_sb, q_sh, static_cast<const uint16_t*>(K_scale), static_cast<const uint16_t*>(K_mn), km_sb, km_sh, km_sp, Hq, Hkv, P,    \
                     head_off, scores, sc_sb, sc_sh, dp.pos, dp.n_new, dp.page, levels);                                                                                   \
        else if (dp.pos && dp.early) launch_k(PDL_SCORES, page_scores_early_kernel<QT, NR, CHV, NoAppend>, grid, dim3(SCORE_THREADS), 0, st, FQ_SC_ARGS, levels, none);       \
        else launch_k(PDL_SCORES, page_scores_kernel<QT, NR, CHV, NoAppend>, grid, dim3(SCORE_THREADS), 0, st, FQ_SC_ARGS, dp.early ? 1 : 0, levels, none);                   \
    } while (0)
    if constexpr (sizeof(QT) == 2) {
        if (app) {
            ++grid.x;
            if constexpr (std::is_same_v<QT, __half>) {
                if (dp.pos) {
                    if (CH == 1) launch_k(PDL_SCORES, page_scores_early_kernel<QT, NR, 1, DynAppend>, grid, dim3(SCORE_THREADS), 0, st, FQ_SC_ARGS, levels, *app);
                    else launch_k(PDL_SCORES, page_scores_early_kernel<QT, NR, 2, DynAppend>, grid, dim3(SCORE_THREADS), 0, st, FQ_SC_ARGS, levels, *app);
                    return;
                }
            }
            if (CH == 1) launch_k(PDL_SCORES, page_scores_kernel<QT, NR, 1, StageAppend>, grid, dim3(SCORE_THREADS), 0, st, FQ_SC_ARGS, 0, levels, app->st);
            else launch_k(PDL_SCORES, page_scores_kernel<QT, NR, 2, StageAppend>, grid, dim3(SCORE_THREADS), 0, st, FQ_SC_ARGS, 0, levels, app->st);
            return;
        }
    }
    if (CH == 1) FQ_LAUNCH_SC(1);
    else if (CH == 2) FQ_LAUNCH_SC(2);
    else FQ_LAUNCH_SC(4);
#undef FQ_LAUNCH_SC
#undef FQ_SC_ARGS
}

template <typename QT>
static void launch_scores_nr(int nr, int CH, dim3 grid, cudaStream_t st, const void* Q, int64_t q_sb, int64_t q_sh,
                             const void* K_scale, const void* K_mn, int64_t km_sb, int64_t km_sh, int64_t km_sp,
                             int Hq, int Hkv, int P, int D, int head_off, float* scores, int64_t sc_sb, int64_t sc_sh, const DynPos& dp, float levels,
                             const DynAppend* app) {
#define FQ_ARGS CH, grid, st, Q, q_sb, q_sh, K_scale, K_mn, km_sb, km_sh, km_sp, Hq, Hkv, P, D, head_off, scores, sc_sb, sc_sh, dp, levels, app
    if (nr == 1) launch_scores<QT, 1>(FQ_ARGS);
    else if (nr == 2) launch_scores<QT, 2>(FQ_ARGS);
    else if (nr == 3) launch_scores<QT, 3>(FQ_ARGS);
    else launch_scores<QT, 4>(FQ_ARGS);
#undef FQ_ARGS
}

int page_scores_int4_launch(
    const void* Q, int q_dtype, int64_t q_sb, int64_t q_sh,
    const void* K_scale, const void* K_mn, int64_t km_sb, int64_t km_sh, int64_t km_sp,
    int B, int Hq, int Hkv, int P, int D,
    float* scores, int64_t sc_sb, int64_t sc_sh, void* stream, const DynPos& dp, float levels, const QuantParams* append, int append_dtype) {
    const char* fn = levels == 255.0f ? "fq_page_scores_int8" : "fq_page_scores_int4";
    FQ_CHECK_ARG(B > 0 && Hq > 0 && Hkv > 0 && P >= 0, FQ_ERR_ARG, "%s: bad sizes", fn);
    FQ_CHECK_ARG(Hq % Hkv == 0, FQ_ERR_ARG, "%s: H_q=%d must be divisible by H_kv=%d", fn, Hq, Hkv);
    FQ_CHECK_ARG(D == 32 || D == 64 || D == 128 || D == 256, FQ_ERR_UNSUPPORTED, "%s: head_dim %d not in {32,64,128,256}", fn, D);
    FQ_CHECK_ARG(q_dtype == FQ_F32 || q_dtype == FQ_F16 || q_dtype == FQ_BF16, FQ_ERR_DTYPE, "%s: dtype code %d", fn, q_dtype);
    if (P == 0) return FQ_OK;
    FQ_CHECK_ARG(Q && K_scale && K_mn && scores, FQ_ERR_ARG, "%s: null pointer", fn);
    const int64_t qa = q_dtype == FQ_F32 ? 4 : 8;
    FQ_CHECK_ARG(q_sb % qa == 0 && q_sh % qa == 0 && aligned(Q, 16), FQ_ERR_ALIGN, "%s: Q rows must be 16-byte aligned", fn);
    FQ_CHECK_ARG(km_sb % 8 == 0 && km_sh % 8 == 0 && km_sp % 8 == 0 && aligned(K_scale, 16) && aligned(K_mn, 16),
                 FQ_ERR_ALIGN, "%s: K metadata rows must be 16-byte aligned", fn);
    const int n_rep = Hq / Hkv;
    const int CH = D <= 64 ? 1 : D / 64;
    dim3 grid((unsigned)((P + SCORE_PAGES_PER_CTA - 1) / SCORE_PAGES_PER_CTA), (unsigned)Hkv, (unsigned)B);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    DynAppend app{};
    if (append) {
        FQ_CHECK_ARG(page_scores_take_append(q_dtype, B, Hq, Hkv, P, D) && (append_dtype == FQ_F16 || append_dtype == FQ_BF16) && append->n_layers == 1 &&
                     append->pos == dp.pos && (!dp.pos || (dp.early && q_dtype == FQ_F16 && append_dtype == FQ_F16)), FQ_ERR_ARG, "%s: an append that this launch does not take", fn);
        const QuantParams& q = *append;
        app.q = q;
        const int64_t first = q.pos ? 0 : q.n_head * q.st_ss;
        app.st = StageAppend{static_cast<const uint16_t*>(q.K_new), static_cast<const uint16_t*>(q.V_new), q.nw_sb, q.nw_sh, q.nw_ss,
                             static_cast<uint16_t*>(q.stage_K) + first, static_cast<uint16_t*>(q.stage_V) + first, q.st_sb, q.st_sh, q.st_ss, q.n_new};
    }
    // query heads of a group are served four at a time (one pass over the metadata per four); the first pass appends, the others
    // find the page completed
    for (int off = 0; off < n_rep; off += 4) {
        const int nr = n_rep - off < 4 ? n_rep - off : 4;
#define FQ_ARGS nr, CH, grid, st, Q, q_sb, q_sh, K_scale, K_mn, km_sb, km_sh, km_sp, Hq, Hkv, P, D, off, scores, sc_sb, sc_sh, dp, levels, append && off == 0 ? &app : nullptr
        if (q_dtype == FQ_F32) launch_scores_nr<float>(FQ_ARGS);
        else if (q_dtype == FQ_F16) launch_scores_nr<__half>(FQ_ARGS);
        else launch_scores_nr<__nv_bfloat16>(FQ_ARGS);
#undef FQ_ARGS
        FQ_CHECK_LAUNCH(fn);
    }
    return FQ_OK;
}

}  // namespace fq

extern "C" int fq_page_scores_int4(
    const void* Q, int q_dtype, int64_t q_sb, int64_t q_sh,
    const void* K_scale, const void* K_mn, int64_t km_sb, int64_t km_sh, int64_t km_sp,
    int B, int Hq, int Hkv, int P, int D,
    float* scores, int64_t sc_sb, int64_t sc_sh, void* stream) {
    return fq::page_scores_int4_launch(Q, q_dtype, q_sb, q_sh, K_scale, K_mn, km_sb, km_sh, km_sp, B, Hq, Hkv, P, D,
                                       scores, sc_sb, sc_sh, stream, fq::DynPos{}, 15.0f);
}

extern "C" int fq_page_scores_int8(
    const void* Q, int q_dtype, int64_t q_sb, int64_t q_sh,
    const void* K_scale, const void* K_mn, int64_t km_sb, int64_t km_sh, int64_t km_sp,
    int B, int Hq, int Hkv, int P, int D,
    float* scores, int64_t sc_sb, int64_t sc_sh, void* stream) {
    return fq::page_scores_int4_launch(Q, q_dtype, q_sb, q_sh, K_scale, K_mn, km_sb, km_sh, km_sp, B, Hq, Hkv, P, D,
                                       scores, sc_sb, sc_sh, stream, fq::DynPos{}, 255.0f);
}
